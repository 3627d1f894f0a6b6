// Host gate fusion for the executors: runs of gates whose qubits fit in k qubits are composed in
// FP64 into one dense k-qubit block.  The semantics are the reference's gate::merge
// (gate_merge.cpp:316-356: the later gate's matrix times the earlier one's, both expanded to the union
// of their qubits), computed with a plain dense product instead of Eigen.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>

#include "circuit.hpp"
#include "../../include/qulacs_b200.h"

namespace qs {

using cd = std::complex<double>;

static ITYPE qubit_mask(const GateRec& g) {
    ITYPE m = 0;
    for (UINT q : g.targets) m |= 1ULL << q;
    for (UINT q : g.controls) m |= 1ULL << q;
    return m;
}
// One more than the highest qubit of a gate list.
static UINT qubit_range(const std::vector<GateRec>& G) {
    ITYPE m = 0;
    for (const GateRec& g : G) m |= qubit_mask(g);
    return m ? 64u - (UINT)__builtin_clzll(m) : 0u;
}

void apply_gate_to_block(std::vector<cd>& U, int kb, const GateRec& g, const std::vector<int>& pos) {
    const int md = 1 << kb;
    const std::vector<cd> gm = g.dense_matrix();
    const int nt = (int)g.targets.size(), nc = (int)g.controls.size();
    const int gd = 1 << nt;
    int tmask = 0, cmask = 0, cval = 0;
    for (int j = 0; j < nt; ++j) tmask |= 1 << pos[j];
    for (int j = 0; j < nc; ++j) {
        cmask |= 1 << pos[nt + j];
        if (g.control_values[j]) cval |= 1 << pos[nt + j];
    }
    std::vector<int> off(gd, 0);
    for (int x = 0; x < gd; ++x)
        for (int j = 0; j < nt; ++j)
            if ((x >> j) & 1) off[x] |= 1 << pos[j];
    // plain real arithmetic: std::complex's operator* goes through the library's inf/nan-checking
    // routine, which dominated the cost of composing large blocks
    std::vector<double> tr(gd), ti(gd);
    for (int base = 0; base < md; ++base) {
        if ((base & tmask) || (base & cmask) != cval) continue;
        for (int col = 0; col < md; ++col) {
            for (int y = 0; y < gd; ++y) {
                double ar = 0., ai = 0.;
                for (int x = 0; x < gd; ++x) {
                    const cd m = gm[y * gd + x], u = U[(size_t)(base | off[x]) * md + col];
                    ar += m.real() * u.real() - m.imag() * u.imag();
                    ai += m.real() * u.imag() + m.imag() * u.real();
                }
                tr[y] = ar;
                ti[y] = ai;
            }
            for (int y = 0; y < gd; ++y) U[(size_t)(base | off[y]) * md + col] = cd(tr[y], ti[y]);
        }
    }
}

static bool fusable(const GateRec& g, int k) {
    return g.kind != QS_GATE_DEPOLARIZING && (int)g.qubits().size() <= k;
}

// One block -> one gate: the original gate when the block holds one, else a dense (or, when the
// product is diagonal on one qubit, a diagonal) gate on the block's qubits in ascending order.
static GateRec block_gate(const std::vector<GateRec>& G, ITYPE mask, const std::vector<int>& members) {
    if (members.size() == 1) return G[members[0]];
    std::vector<UINT> qs;
    for (UINT q = 0; q < 64; ++q)
        if ((mask >> q) & 1ULL) qs.push_back(q);
    const int kb = (int)qs.size(), md = 1 << kb;
    std::vector<cd> U((size_t)md * md, 0.);
    for (int i = 0; i < md; ++i) U[(size_t)i * md + i] = 1.;
    for (int gi : members) {
        std::vector<int> pos;
        for (UINT gq : G[gi].qubits()) pos.push_back((int)(std::find(qs.begin(), qs.end(), gq) - qs.begin()));
        apply_gate_to_block(U, kb, G[gi], pos);
    }
    GateRec r;
    r.targets = qs;
    bool diag = true;
    for (int y = 0; y < md && diag; ++y)
        for (int x = 0; x < md; ++x)
            if (x != y && U[(size_t)y * md + x] != cd(0.)) {
                diag = false;
                break;
            }
    if (diag && kb == 1) {
        r.kind = QS_GATE_DIAGONAL;
        r.matrix = {U[0], U[3]};
    } else {
        r.kind = QS_GATE_DENSE;
        r.matrix = U;
    }
    return r;
}

// *blocks (may be null): how many gates the fusion makes.  `keep` (may be null): whether a block stays one gate; its members go out one by one otherwise.
static std::vector<GateRec> fuse_blocks(const std::vector<GateRec>& G, int k,
    bool (*keep)(const std::vector<GateRec>&, ITYPE, const std::vector<int>&), size_t* blocks) {
    if (k <= 0) {
        if (blocks) *blocks = G.size();
        return G;
    }
    struct Block {
        ITYPE mask;
        std::vector<int> members;
    };
    std::vector<Block> open;  // pairwise disjoint qubit sets
    std::vector<GateRec> out;
    size_t count = 0;
    auto close = [&](const Block& b) {
        ++count;
        if (!keep || keep(G, b.mask, b.members)) out.push_back(block_gate(G, b.mask, b.members));
        else
            for (int i : b.members) out.push_back(G[i]);
    };
    for (int i = 0; i < (int)G.size(); ++i) {
        const ITYPE gm = qubit_mask(G[i]);
        ITYPE um = gm;
        std::vector<size_t> touch;
        for (size_t j = 0; j < open.size(); ++j)
            if (open[j].mask & gm) {
                touch.push_back(j);
                um |= open[j].mask;
            }
        const bool fits = fusable(G[i], k) && __builtin_popcountll(um) <= k;
        Block merged{um, {}};
        for (size_t j : touch) {
            if (fits) merged.members.insert(merged.members.end(), open[j].members.begin(), open[j].members.end());
            else close(open[j]);
        }
        for (size_t t = touch.size(); t-- > 0;) open.erase(open.begin() + (long)touch[t]);
        if (fits) {
            merged.members.push_back(i);
            open.push_back(merged);
        } else if (fusable(G[i], k)) {
            open.push_back({gm, {i}});
        } else {
            out.push_back(G[i]);
            ++count;
        }
    }
    for (const Block& b : open) close(b);
    if (blocks) *blocks = count;
    return out;
}

std::vector<GateRec> fuse_gates(const std::vector<GateRec>& G, int k) { return fuse_blocks(G, k, nullptr, nullptr); }

// ---------------------------------------------------------------- rotation form
using ld = long double;
using cl = std::complex<long double>;

static cl xmul(const cl& x, const cl& y) {
    return cl(x.real() * y.real() - x.imag() * y.imag(), x.real() * y.imag() + x.imag() * y.real());
}
static ld xnorm(const cl& z) { return z.real() * z.real() + z.imag() * z.imag(); }
static ld xabs(const cl& z) { return std::sqrt(xnorm(z)); }  // entries of unitaries: no overflow
static cl xdiv(const cl& x, const cl& y) {  // |y| near 1
    const ld n = xnorm(y);
    const cl z = xmul(x, std::conj(y));
    return cl(z.real() / n, z.imag() / n);
}

// What rounding leaves of the unitarity of a matrix computed in double precision (16 ulp: QR factors are off by up
// to 6, matrix exponentials by 11).  A matrix further off is applied as it is given.
constexpr ld kUnitTol = 0x1p-48L;
static bool is_unit(const cl& z) { return std::abs(xnorm(z) - 1.L) <= kUnitTol; }

// `gates`: how many matrices were multiplied.
static bool is_unitary2(const cl* u, int gates = 1) {
    const cl d = xmul(std::conj(u[0]), u[1]) + xmul(std::conj(u[2]), u[3]);
    const ld tol = kUnitTol * gates;
    return std::abs(xnorm(u[0]) + xnorm(u[2]) - 1.L) <= tol && std::abs(xnorm(u[1]) + xnorm(u[3]) - 1.L) <= tol &&
           xnorm(d) <= tol * tol;
}

// U = diag(1, q1) [[c, -s], [s, c]] diag(p0, p1), c, s >= 0, unit p0, p1, q1, of a unitary U.  Phases are
// quotients of entries (no angles), each taken where the entries are largest.
static void zyz(const cl* u, ld* c, ld* s, cl* q1, cl* p0, cl* p1) {
    const ld c0 = xabs(u[0]), c1 = xabs(u[3]), s0 = xabs(u[2]), s1 = xabs(u[1]), r = std::sqrt(c0 * c0 + s0 * s0);
    *c = c0 / r;
    *s = s0 / r;
    // e0, e1, f0, f1: phases of U00, U11, U10, -U01, with e0 e1 = f0 f1
    if (c0 >= s0) {
        const cl e0 = u[0] / c0, e1 = u[3] / c1;
        const cl f1 = s1 > 0.L ? -u[1] / s1 : e0;
        *p0 = e0;
        *p1 = f1;
        *q1 = xmul(e1, std::conj(f1));
    } else {
        const cl f0 = u[2] / s0, f1 = -u[1] / s1;
        const cl e0 = c0 > 0.L ? u[0] / c0 : cl(1.L);
        *p0 = e0;
        *p1 = f1;
        *q1 = xmul(f0, std::conj(e0));
    }
}

// A one-qubit gate's matrix in extended precision (rotations from their angle).
static void xmatrix(const GateRec& g, cl* m) {
    ld c = 1.L, s = 0.L;
    if (g.kind == QS_GATE_RX || g.kind == QS_GATE_RY || g.kind == QS_GATE_RZ) sincosl((ld)g.angle / 2, &s, &c);
    switch (g.kind) {
        case QS_GATE_RX: m[0] = m[3] = c; m[1] = m[2] = cl(0.L, s); return;
        case QS_GATE_RY: m[0] = m[3] = c; m[1] = s; m[2] = -s; return;
        case QS_GATE_RZ: m[0] = cl(c, s); m[3] = cl(c, -s); m[1] = m[2] = 0.L; return;
        case QS_GATE_DENSE:
            for (int i = 0; i < 4; ++i) m[i] = cl(g.matrix[i].real(), g.matrix[i].imag());
            return;
        default: break;
    }
    const std::vector<cd> d = g.dense_matrix();
    for (int i = 0; i < 4; ++i) m[i] = cl(d[i].real(), d[i].imag());
}

// The specialised pass kernels apply a real rotation in 2 FP64 instructions per amplitude, a 2 x 2 complex
// matrix in 8, and collect diagonals (phase_program.hpp).  So each run of one-qubit gates is multiplied
// out and written D1 R D2: R is emitted as RY with its (cosine, sine), D2 as a diagonal before it, and D1 is
// carried forward -- through controls, CZ and diagonals, which commute with it -- into the D2 of the next
// run on the qubit.  Only unitary diagonals are carried: a depolarizing channel does not commute with others,
// and their products have no bound.  Gates that do not commute with a carried diagonal (CNOT targets, dense
// blocks, ...) get it just before them.  Phases common to a whole state are multiplied up and emitted once at the end.
std::vector<GateRec> rotation_form(const std::vector<GateRec>& G, bool spec) {
    // A qubit's run of gates not emitted yet is diag(1, d), then a core, then diag(p0, p1).  The core is kept
    // as a rotation while it is one: which factors a run gets must not depend on the signs of its angles.
    enum Core { NONE, REAL, RX, MATRIX };
    struct Qubit {
        Core core = NONE;
        int len = 0;          // matrices in it
        ld c = 1.L, s = 0.L;  // REAL: {c, s; -s, c}; RX: {c, i s; i s, c}
        cl m[4];              // MATRIX
        bool post = false, post_free = false, post_unit = true;
        cl p0 = 1.L, p1 = 1.L;
        bool any = false, any_free = false;
        cl d = 1.L;           // carried; a product of quotients of unit entries
    };
    const UINT n = qubit_range(G);
    std::vector<Qubit> Q(n);
    std::vector<GateRec> out;
    out.reserve(2 * G.size() + 4);
    bool any_scalar = false;
    cl scalar = 1.L;
    auto diagonal = [&](UINT q, const cl& d0, const cl& d1, bool free_phase) {
        GateRec d;
        d.kind = QS_GATE_DIAGONAL;
        d.targets = {q};
        d.matrix = {cd((double)d0.real(), (double)d0.imag()), cd((double)d1.real(), (double)d1.imag())};
        d.extended = true;
        d.xd[0] = d0;
        d.xd[1] = d1;
        d.free_phase = free_phase;
        out.push_back(std::move(d));
    };
    auto carry = [&](UINT q, const cl& d0, const cl& d1, bool free_phase) {  // diag(d0, d1) after the carried one
        Qubit& k = Q[q];
        k.any = true;
        k.any_free = k.any_free || free_phase;
        if (free_phase || d0 != cl(1.L)) any_scalar = true;
        scalar = xmul(scalar, d0);
        // an exact sign or identity stays one
        k.d = xmul(k.d, d1 == d0 ? cl(1.L) : d1 == -d0 ? cl(-1.L) : xdiv(d1, d0));
    };
    auto flush = [&](UINT q) {  // the carried diagonal as a gate
        Qubit& k = Q[q];
        if (k.any) diagonal(q, 1.L, k.d, k.any_free);
        k.any = k.any_free = false;
        k.d = 1.L;
    };
    auto rotation = [&](UINT q, int kind, ld c, ld s) {
        GateRec r;
        r.kind = kind;
        r.targets = {q};
        r.extended = true;
        r.xc = c;
        r.xs = s;
        out.push_back(std::move(r));
    };
    auto core_matrix = [](const Qubit& k, cl* m) {
        if (k.core == MATRIX) std::copy(k.m, k.m + 4, m);
        else if (k.core == REAL) m[0] = m[3] = k.c, m[1] = k.s, m[2] = -k.s;
        else if (k.core == RX) m[0] = m[3] = k.c, m[1] = m[2] = cl(0.L, k.s);
        else m[0] = m[3] = 1.L, m[1] = m[2] = 0.L;
    };
    auto end_run = [&](UINT q) {  // emits the run's core; what may be carried further stays carried
        Qubit& k = Q[q];
        const bool post = k.post, post_free = k.post_free, post_unit = k.post_unit;
        const cl p0 = k.p0, p1 = k.p1;
        Core core = k.core;
        const int len = k.len;
        k.core = NONE;
        k.len = 0;
        k.post = k.post_free = false;
        k.post_unit = true;
        k.p0 = k.p1 = 1.L;
        const cl zero(0.L);
        if (core == RX && (k.any || !spec)) {
            const ld c = k.c, s = k.s;
            k.m[0] = k.m[3] = c;
            k.m[1] = k.m[2] = cl(0.L, s);
            core = MATRIX;
        }
        const cl* u = k.m;
        if (core == REAL) {
            flush(q);
            rotation(q, QS_GATE_RY, k.c, k.s);
        } else if (core == RX) {
            rotation(q, QS_GATE_RX, k.c, k.s);
        } else if (core == MATRIX) {
            if (u[0] == zero && u[3] == zero) {  // diag(u1, u2) X
                if (k.any) {  // X diag(1, d) = d diag(1, 1 / d) X
                    any_scalar = true;
                    scalar = xmul(scalar, k.d);
                    k.d = k.d == cl(-1.L) ? k.d : xdiv(cl(1.L), k.d);
                }
                GateRec x;
                x.kind = QS_GATE_DENSE;
                x.targets = {q};
                x.matrix = {0., 1., 1., 0.};
                out.push_back(x);
                if (is_unit(u[1]) && is_unit(u[2])) carry(q, u[1], u[2], false);
                else diagonal(q, u[1], u[2], false);
            } else if (is_unitary2(u, len)) {
                ld c, s;
                cl q1, e0, e1;
                zyz(u, &c, &s, &q1, &e0, &e1);
                carry(q, e0, e1, false);
                flush(q);
                rotation(q, QS_GATE_RY, c, -s);
                carry(q, 1.L, q1, false);
            } else {
                flush(q);
                GateRec r;
                r.kind = QS_GATE_DENSE;
                r.targets = {q};
                for (int i = 0; i < 4; ++i) r.matrix.push_back(cd((double)u[i].real(), (double)u[i].imag()));
                out.push_back(r);
            }
        }
        if (post) {
            if (post_unit) carry(q, p0, p1, post_free);
            else diagonal(q, p0, p1, false);  // commutes with the carried diagonal
        }
    };
    auto add_matrix = [&](UINT q, int kind, const cl* m) {
        Qubit& k = Q[q];
        const cl zero(0.L);
        ++k.len;
        if (m[1] == zero && m[2] == zero) {
            k.p0 = xmul(m[0], k.p0);
            k.p1 = xmul(m[3], k.p1);
            k.post = true;
            k.post_unit = k.post_unit && is_unit(m[0]) && is_unit(m[3]);
            k.post_free = k.post_free || kind == QS_GATE_RZ;
            if (k.core == NONE) end_run(q);
            return;
        }
        // a real rotation, or one after a sign of the |1> row
        bool real = true;
        for (int i = 0; i < 4; ++i) real = real && m[i].imag() == 0.L;
        real = real && m[0] != zero && is_unitary2(m);
        if (real && !k.post && (k.core == NONE || k.core == REAL)) {
            const ld c = m[0].real(), s = m[1].real();
            const bool det = m[0].real() * m[3].real() - m[1].real() * m[2].real() > 0.L;
            const ld c0 = k.core == REAL ? k.c : 1.L, s0 = k.core == REAL ? k.s : 0.L;
            k.core = REAL;
            k.c = c * c0 - s * s0;
            k.s = c * s0 + s * c0;
            if (!det) {
                k.p1 = -1.L;
                k.post = true;
            }
            return;
        }
        if (kind == QS_GATE_RX && !k.post && (k.core == NONE || k.core == RX)) {
            const ld c = m[0].real(), s = m[1].imag();
            const ld c0 = k.core == RX ? k.c : 1.L, s0 = k.core == RX ? k.s : 0.L;
            k.core = RX;
            k.c = c * c0 - s * s0;
            k.s = c * s0 + s * c0;
            return;
        }
        cl a[4];
        core_matrix(k, a);
        for (int x = 0; x < 2; ++x) {
            a[x] = xmul(k.p0, a[x]);
            a[2 + x] = xmul(k.p1, a[2 + x]);
        }
        for (int y = 0; y < 2; ++y)
            for (int x = 0; x < 2; ++x) k.m[y * 2 + x] = xmul(m[y * 2], a[x]) + xmul(m[y * 2 + 1], a[2 + x]);
        k.core = MATRIX;
        k.post = k.post_free = false;
        k.post_unit = true;
        k.p0 = k.p1 = 1.L;
    };
    for (const GateRec& g : G) {
        if (g.targets.size() == 1 && g.controls.empty() && g.kind != QS_GATE_DEPOLARIZING) {
            cl m[4];
            xmatrix(g, m);
            add_matrix(g.targets[0], g.kind, m);
            continue;
        }
        for (UINT q : g.targets) end_run(q);
        for (UINT q : g.controls) end_run(q);
        switch (g.kind) {
            case QS_GATE_CZ:
            case QS_GATE_DIAGONAL: break;
            case QS_GATE_CNOT: flush(g.targets[1]); break;
            case QS_GATE_SWAP: {
                Qubit &a = Q[g.targets[0]], &b = Q[g.targets[1]];
                std::swap(a.any, b.any);
                std::swap(a.any_free, b.any_free);
                std::swap(a.d, b.d);
                break;
            }
            default:
                if (g.depol == 1) {
                    // a channel commutes with a unitary U on the row bit and conj(U) on the column bit together
                    const Qubit &c = Q[g.targets[0]], &r = Q[g.targets[1]];
                    if (c.any && r.any && c.d == std::conj(r.d)) break;
                }
                for (UINT t : g.targets) flush(t);  // controls commute
        }
        out.push_back(g);
    }
    for (UINT q = 0; q < n; ++q) {
        end_run(q);
        flush(q);
    }
    if (any_scalar && n) diagonal(0, scalar, scalar, true);
    return out;
}

// Fused blocks on up to two qubits cost 16 FP64 instructions per amplitude as a matrix; their gates apart,
// in rotation form, cost about 4 per run of one-qubit gates (2 for the rotation and a share of the
// diagonals), nothing per CNOT, CZ or SWAP and 16 per two-qubit matrix.  The cheaper of the two is kept.
static bool dense_pays(const std::vector<GateRec>& G, ITYPE mask, const std::vector<int>& members) {
    if (__builtin_popcountll(mask) > 2) return true;
    int cost = 0;
    ITYPE run = 0;  // qubits with a run of one-qubit gates open
    for (int i : members) {
        const GateRec& g = G[i];
        const ITYPE q = qubit_mask(g);
        if (g.targets.size() == 1 && g.controls.empty()) {
            if (!(run & q)) cost += 4;
            run |= q;
        } else {
            run &= ~q;
            if (g.depol) cost += 2;
            else if (g.kind == QS_GATE_DENSE && g.controls.empty()) cost += 16;
            else if (g.kind != QS_GATE_CNOT && g.kind != QS_GATE_CZ && g.kind != QS_GATE_SWAP)
                return true;  // apart, it would need a pass of its own
        }
    }
    return cost > 16;
}

std::vector<GateRec> executor_gates(const std::vector<GateRec>& G, int k, bool spec, size_t* blocks) {
    return rotation_form(fuse_blocks(G, k, dense_pays, blocks), spec);
}

// A one-qubit depolarizing channel commutes with every unitary on its qubit, and channels of strengths
// q1, q2 compose to 1 - (1 - q1)(1 - q2), so runs of (gate, channel) pairs on a qubit become the gates and
// one channel.
std::vector<GateRec> merge_depolarizing(const std::vector<GateRec>& G) {
    const UINT n = qubit_range(G);
    std::vector<ld> keep(n, 1.L);  // 1 - strength carried on each qubit
    std::vector<GateRec> out;
    auto flush = [&](UINT q) {
        if (keep[q] == 1.L) return;
        GateRec d;
        d.kind = QS_GATE_DEPOLARIZING;
        d.targets = {q};
        d.prob = (double)(0.75L * (1.L - keep[q]));
        out.push_back(d);
        keep[q] = 1.L;
    };
    for (const GateRec& g : G) {
        const bool one = g.targets.size() == 1 && g.controls.empty();
        if (one && g.kind == QS_GATE_DEPOLARIZING) {
            keep[g.targets[0]] *= 1.L - 4.L / 3.L * g.prob;
            continue;
        }
        cl m[4];
        if (one) xmatrix(g, m);
        if (!one || !is_unitary2(m))
            for (UINT q : g.qubits()) flush(q);
        out.push_back(g);
    }
    for (UINT q = 0; q < n; ++q) flush(q);
    return out;
}

}  // namespace qs
