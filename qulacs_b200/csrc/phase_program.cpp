// Builds phase programs (phase_program.hpp) from a pass's ops.
#include "phase_program.hpp"

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>

namespace qs {

// Parameters are multiplied up in extended precision and rounded once.
using ld = long double;
using cl = std::complex<long double>;

namespace {

cl mulc(const cl& x, const cl& y) {
    return cl(x.real() * y.real() - x.imag() * y.imag(), x.real() * y.imag() + x.imag() * y.real());
}
double2 rounded(const cl& z) { return make_double2((double)z.real(), (double)z.imag()); }
// hi + lo of a parameter pair
cl joined(const double2& hi, const double2& lo) { return cl((ld)hi.x + lo.x, (ld)hi.y + lo.y); }

struct Node {
    bool diag = false;
    // diagonal factors: functionals of the register index (1 or 2 of them) and the 16 values
    int nf = 0;
    uint8_t g[2] = {};
    bool sign = false;  // values +-1
    bool free = false;  // one functional, free phase: counts as a factor whatever its value
    cl lo = 1., hi = 1.;  // value where the factor's bits (its mask) are 0 and 1
    uint16_t on = 0;
    ProgStep step;      // other nodes: in the algebra of X^v (v in vs) and Z^f (f in fs)
    int nv = 0, ns = 0;
    uint8_t vs[4], fs[4];
    bool rot = false;
    int waits = 0;      // earlier nodes that do not commute with this one and have not run
    bool done = false;
};

int par4(unsigned x) { return __builtin_popcount(x & 15u) & 1; }

// Sets of functionals (or of vectors) as bits of a 16-bit word: odd[v] holds the functionals that are 1 at v.
struct Odd {
    uint16_t at[16];
    Odd() {
        for (int v = 0; v < 16; ++v) {
            at[v] = 0;
            for (int f = 0; f < 16; ++f) at[v] |= (uint16_t)(par4(f & v) << f);
        }
    }
};
const Odd kOdd;

// A node as the commutation test sees it: its functionals (a diagonal's, or a step's Z^f), and those that are 1
// at one of its vectors (a step's X^v).
struct Sets {
    uint16_t f = 0, odd = 0;
    bool diag = false, rot = false;
    explicit Sets(const Node& n) : diag(n.diag), rot(n.rot) {
        if (diag) {
            for (int i = 0; i < n.nf; ++i) f |= (uint16_t)(1u << n.g[i]);
            return;
        }
        for (int i = 0; i < n.ns; ++i) f |= (uint16_t)(1u << n.fs[i]);
        for (int i = 0; i < n.nv; ++i) odd |= kOdd.at[n.vs[i]];
    }
};

bool commute(const Sets& a, const Sets& b) {
    if (a.diag && b.diag) return true;
    const bool ab = a.f & b.odd, ba = b.f & a.odd;
    if (a.rot && b.rot) return ab == ba;  // two strings X^v Z^f: RY is X^v Z^f, RX is X^v
    return !ab && !ba;
}

struct PassScalar {
    cl value = 1.;
    bool any = false;      // something was deferred (whatever its value: the kernel depends on structure only)
    bool complex = false;
    double bits = 0.;      // log2 of the growth deferred so far
};

struct Builder {
    // each qubit's functional, vector and constant over the register's index
    uint8_t F[4], V[4], A[4] = {};
    std::vector<Node> nodes;
    PassScalar& S;
    const bool move;  // CNOT, SWAP and X are steps; the map stays the identity
    Builder(PassScalar& s, bool m, size_t gates, const uint8_t* in) : S(s), move(m) {
        nodes.reserve(gates);
        for (int b = 0; b < 4; ++b) {
            F[b] = 0;
            for (int k = 0; k < 4; ++k) F[b] |= (uint8_t)(((in[k] >> b) & 1) << k);
        }
        for (int j = 0; j < 16; ++j) {
            int i = 0;
            for (int k = 0; k < 4; ++k)
                if ((j >> k) & 1) i ^= in[k];
            if (i && !(i & (i - 1))) V[__builtin_ctz(i)] = (uint8_t)j;
        }
    }

    // qubit i of the node's step is register bit b; x, z: whether the node moves and reads it
    void set_qubit(Node& n, int i, int b, bool x = true, bool z = true) {
        ProgStep& p = n.step;
        p.v[i] = V[b];
        p.f[i] = F[b];
        p.a[i] = A[b];
        p.nq = (uint8_t)std::max<int>(p.nq, i + 1);
        if (x) n.vs[n.nv++] = V[b];
        if (z) n.fs[n.ns++] = F[b];
    }
    void push(Node n) { nodes.push_back(std::move(n)); }

    // `free`: the phases are parameters, so the step is the same whatever their values
    void diag1(int b, cl d0, cl d1, bool free = false) {
        Node n;
        n.diag = true;
        n.nf = 1;
        n.g[0] = F[b];
        n.free = free;
        // the factor of bit value 0 joins the pass's scalar if it is 1 in modulus (others have no bound)
        const bool ok = free || std::abs(std::norm(d0) - 1.L) <= 0x1p-49L;
        if (d0 == d1 && ok && (!free || d0 != cl(1.))) {  // a scalar
            if (d0 != cl(1.)) scalar(d0, free);
            return;
        }
        if (ok) {
            if (d0 != cl(1.)) scalar(d0, free);
            const cl r = d1 == -d0 ? cl(-1.) : d0 == cl(1.) ? d1 : mulc(d1, std::conj(d0)) / std::norm(d0);
            n.sign = !free && r == cl(-1.);
            n.hi = r;
        } else {
            n.lo = d0;
            n.hi = d1;
        }
        for (int j = 0; j < 16; ++j) n.on |= (uint16_t)((par4(F[b] & j) ^ A[b]) << j);
        push(std::move(n));
    }
    void scalar(cl z, bool free = false) {
        S.any = true;
        S.complex = S.complex || free || z.imag() != 0.;
        S.value = mulc(S.value, z);
    }
    void cz(int a, int b) {
        Node n;
        n.diag = n.sign = true;
        n.nf = 2;
        n.g[0] = F[a];
        n.g[1] = F[b];
        n.hi = -1.;
        for (int j = 0; j < 16; ++j) n.on |= (uint16_t)(((par4(F[a] & j) ^ A[a]) & (par4(F[b] & j) ^ A[b])) << j);
        push(std::move(n));
    }
    // csim's RY {c, s; -s, c} (x = false) or RX {c, i s; i s, c}
    void rot(int b, ld c, ld s, bool x) {
        Node n;
        n.rot = true;
        n.step.kind = SP_ROT;
        set_qubit(n, 0, b, true, !x);
        const double bits = -std::log2(std::max((double)std::abs(c), 1e-300));
        const uint8_t base = x ? RF_X_TAN : RF_Y_TAN;
        if (bits <= 20. && S.bits + bits <= kMaxDeferredBits) {
            n.step.form = base;
            n.step.par.push_back(make_double2((double)(s / c), 0.));
            scalar(c);
            S.bits += bits;
        } else if (S.bits + 1. <= kMaxDeferredBits) {  // nearly a flip: the sine is near 1
            n.step.form = base + 1;
            n.step.par.push_back(make_double2((double)(c / s), 0.));
            scalar(s);
            S.bits += 1.;
        } else {
            n.step.form = base + 2;
            n.step.par.push_back(make_double2((double)c, (double)s));
        }
        push(std::move(n));
    }
    void flip(int b) {
        if (move) return perm(SP_X, b, -1);
        A[b] ^= 1;
    }
    void perm(StepKind kind, int a, int b) {
        Node n;
        n.step.kind = kind;
        set_qubit(n, 0, a, kind != SP_CNOT, kind != SP_X);
        if (b >= 0) set_qubit(n, 1, b, true, kind == SP_SWAP);
        push(std::move(n));
    }
    void cnot(int c, int t) {
        if (move) return perm(SP_CNOT, c, t);
        F[t] ^= F[c];
        A[t] ^= A[c];
        V[c] ^= V[t];
    }
    void swap(int a, int b) {
        if (move) return perm(SP_SWAP, a, b);
        std::swap(F[a], F[b]);
        std::swap(V[a], V[b]);
        std::swap(A[a], A[b]);
    }
    void dense1(int b, const double2* m) {
        cl u[4];
        for (int i = 0; i < 4; ++i) u[i] = cl(m[i].x, m[i].y);
        if (u[1] == cl(0.) && u[2] == cl(0.)) return diag1(b, u[0], u[3]);
        if (u[0] == cl(0.) && u[3] == cl(0.)) {
            flip(b);
            return diag1(b, u[1], u[2]);
        }
        Node n;
        n.step.kind = SP_DENSE1;
        set_qubit(n, 0, b);
        n.step.par.assign(m, m + 4);
        push(std::move(n));
    }
    void dense2(int a, int b, const double2* m) {
        Node n;
        n.step.kind = SP_DENSE2;
        set_qubit(n, 0, a);
        set_qubit(n, 1, b);
        n.step.par.assign(m, m + 16);
        push(std::move(n));
    }
    // depolarizing channel of strength q (rho -> (1 - q) rho + q I / 2^k tr): column bits, then row bits
    void depol(const int* bits, int k, ld q) {
        Node n;
        n.step.kind = k == 1 ? SP_DEPOL1 : SP_DEPOL2;
        for (int i = 0; i < 2 * k; ++i) set_qubit(n, i, bits[i]);
        const ld d = k == 1 ? 1.L - q / 2 : 1.L - q;  // what the scaled form leaves out
        const double grow = -std::log2(std::max((double)std::abs(d), 1e-300));
        const bool scaled = grow <= 10. && S.bits + grow <= kMaxDeferredBits;  // one qubit: d >= 1/3
        if (scaled) {
            scalar(d);
            S.bits += grow;
        }
        n.step.form = !scaled;
        if (k == 1) {
            n.step.par.push_back(make_double2((double)(q / 2 / d), (double)((1.L - q) / (scaled ? d : 1.L))));
            if (!scaled) n.step.par.push_back(make_double2((double)d, 0.));
        } else {
            n.step.par.push_back(scaled ? make_double2((double)(q / 4 / d), 0.) : make_double2((double)(q / 4), (double)d));
        }
        push(std::move(n));
    }

    void schedule(PhaseProgram* P) {
        const int N = (int)nodes.size();
        std::vector<Sets> sets;
        sets.reserve(N);
        for (const Node& n : nodes) sets.emplace_back(n);
        std::vector<std::vector<int>> after(N);
        for (int j = 0; j < N; ++j)
            for (int i = 0; i < j; ++i)
                if (!commute(sets[i], sets[j])) {
                    after[i].push_back(j);
                    ++nodes[j].waits;
                }
        int left = N;
        auto finish = [&](int i) {
            nodes[i].done = true;
            --left;
            for (int j : after[i]) --nodes[j].waits;
        };
        std::vector<int> ready;
        auto others = [&]() {  // every ready step that is no diagonal, rotations by register bit
            bool any = false;
            while (true) {
                ready.clear();
                for (int i = 0; i < N; ++i)
                    if (!nodes[i].done && !nodes[i].diag && nodes[i].waits == 0) ready.push_back(i);
                if (ready.empty()) return any;
                std::stable_sort(ready.begin(), ready.end(),
                    [&](int x, int y) { return (nodes[x].rot ? nodes[x].step.v[0] : 0) < (nodes[y].rot ? nodes[y].step.v[0] : 0); });
                for (int i : ready) {
                    P->steps.push_back(std::move(nodes[i].step));
                    finish(i);
                }
                any = true;
            }
        };
        auto diagonals = [&](bool signs_only) {
            ProgStep s;
            bool any = false, sign = true;
            cl val[16];
            bool touched[16] = {};
            for (int j = 0; j < 16; ++j) val[j] = 1.;
            for (int i = 0; i < N; ++i) {
                Node& n = nodes[i];
                if (n.done || !n.diag || n.waits || (signs_only && !n.sign)) continue;
                const bool lo = n.lo != cl(1.), hi = n.hi != cl(1.) || n.free;
                for (int j = 0; j < 16; ++j) {
                    const bool on = (n.on >> j) & 1;
                    if (!(on ? hi : lo)) continue;
                    touched[j] = true;
                    val[j] = mulc(val[j], on ? n.hi : n.lo);
                }
                any = true;
                sign = sign && n.sign;
                finish(i);
            }
            if (!any) return;
            if (sign) {
                s.kind = SP_SIGN;
                for (int j = 0; j < 16; ++j)
                    if (val[j] != cl(1.)) s.mask |= (uint16_t)(1u << j);
                if (!s.mask) return;
            } else {
                s.kind = SP_DIAG;
                for (int j = 0; j < 16; ++j) {
                    s.par.push_back(rounded(val[j]));
                    s.xpar.push_back(val[j]);
                    if (touched[j]) s.mask |= (uint16_t)(1u << j);
                }
            }
            P->steps.push_back(std::move(s));
        };
        while (left) {
            others();
            if (!left) break;
            diagonals(true);  // sign flips cost nothing: first
            if (others()) continue;
            diagonals(false);
        }
        // register j holds coset index out[j] holds coset index i(j)
        for (int j = 0; j < 16; ++j) {
            int i = 0;
            for (int b = 0; b < 4; ++b) i |= (par4(F[b] & j) ^ A[b]) << b;
            P->out[j] = (uint8_t)i;
        }
    }
};

}  // namespace

std::vector<PhaseProgram> build_pass_program(const StPhase* phases, size_t count, const StOp* ops, const double2* pool) {
    std::vector<PhaseProgram> out(count);
    PassScalar S;
    for (size_t ph = 0; ph < count; ++ph) {
        const StOp *begin = ops + phases[ph].op_begin, *end = begin + phases[ph].op_count;
        bool move = false;
        for (const StOp* o = begin; o != end; ++o) {
            const double2* m = pool + o->param;
            const bool one = o->kind == ST_DENSE1;  // an X or a diagonal is no matrix
            const bool flip = one && m[0].x == 0. && m[0].y == 0. && m[3].x == 0. && m[3].y == 0.;
            const bool diag = one && m[1].x == 0. && m[1].y == 0. && m[2].x == 0. && m[2].y == 0.;
            move = move || o->kind == ST_DENSE2 || o->kind == ST_DEPOL1 || o->kind == ST_DEPOL2 || (one && !flip && !diag);
        }
        Builder B(S, move, (size_t)(end - begin), phases[ph].in);
        for (const StOp* op = begin; op != end; ++op) {
            const StOp& o = *op;
            const double2* p = pool + o.param;
            switch (o.kind) {
                case ST_RX:
                case ST_RY: B.rot(o.a, (ld)p[0].x + p[1].x, (ld)p[0].y + p[1].y, o.kind == ST_RX); break;
                case ST_DIAG1: B.diag1(o.a, joined(p[0], p[2]), joined(p[1], p[3]), o.aux != 0); break;
                case ST_CNOT: B.cnot(o.a, o.b); break;
                case ST_CZ: B.cz(o.a, o.b); break;
                case ST_SWAP: B.swap(o.a, o.b); break;
                case ST_DENSE1: B.dense1(o.a, p); break;
                case ST_DENSE2: B.dense2(o.a, o.b, p); break;
                case ST_DEPOL1: {
                    const int bits[2] = {o.a, o.b};
                    B.depol(bits, 1, (ld)p[0].x * 4 / 3);
                    break;
                }
                case ST_DEPOL2: {
                    const int bits[4] = {o.a, o.b, o.aux & 3, (o.aux >> 2) & 3};
                    B.depol(bits, 2, (ld)p[0].x * 16 / 15);
                    break;
                }
                default: break;
            }
        }
        B.schedule(&out[ph]);
    }
    if (S.any) {
        // the pass's scalar joins the fullest set of diagonal factors, else it is a step of its own
        ProgStep* best = nullptr;
        for (PhaseProgram& P : out)
            for (ProgStep& s : P.steps)
                if (s.kind == SP_DIAG && (!best || __builtin_popcount(s.mask) > __builtin_popcount(best->mask))) best = &s;
        if (best) {
            best->mask = 0xffff;
            for (int j = 0; j < 16; ++j) best->par[j] = rounded(mulc(S.value, best->xpar[j]));
        } else {
            ProgStep s;
            s.kind = SP_SCALE;
            s.form = S.complex;
            s.par.push_back(rounded(S.value));
            out.back().steps.push_back(s);
        }
    }
    return out;
}

// The program as rounds, if it holds nothing else than signs, diagonals and scaled RY (on register bits: the
// planner starts a new phase where a CNOT has relabelled a register that turns again).
static bool encode_rounds(const PhaseProgram& P, StPhase* phase, std::vector<double2>* pool) {
    for (const ProgStep& s : P.steps) {
        const bool ry = s.kind == SP_ROT && s.form == RF_Y_TAN;
        if (!ry && s.kind != SP_DIAG && s.kind != SP_SIGN && s.kind != SP_SCALE) return false;
    }
    // turns (4 tangents) and factors in the order in which they run
    struct Part {
        bool turns;
        double2 v[16];
    };
    std::vector<Part> parts;
    auto open = [&](bool turns) {
        parts.emplace_back();
        parts.back().turns = turns;
        for (double2& v : parts.back().v) v = turns ? make_double2(0., 0.) : make_double2(1., 0.);
    };
    int used = 0;  // register bits that the open turns have
    for (const ProgStep& s : P.steps) {
        if (s.kind == SP_ROT) {
            const int b = __builtin_ctz(s.v[0]);
            if (parts.empty() || !parts.back().turns || used >> b) {  // ascending: the order in which they run
                open(true);
                used = 0;
            }
            used |= 1 << b;
            double2& t = parts.back().v[b / 2];
            (b & 1 ? t.y : t.x) = s.a[0] ? -s.par[0].x : s.par[0].x;
            continue;
        }
        if (parts.empty() || parts.back().turns) open(false);
        for (int j = 0; j < 16; ++j) {
            if (s.kind != SP_SCALE && !((s.mask >> j) & 1)) continue;
            const double2 z = s.kind == SP_SIGN ? make_double2(-1., 0.) : s.par[s.kind == SP_SCALE ? 0 : j];
            double2& d = parts.back().v[j];
            // signs next to factors stay exact
            d = make_double2(z.x * d.x - z.y * d.y, z.x * d.y + z.y * d.x);
        }
    }
    phase->param = (uint32_t)pool->size();
    phase->rounds = 0;
    if (parts.empty()) return true;
    // the order of a round that leaves fewer sets of factors 1
    const bool turns_first = parts.front().turns && !parts.back().turns;
    bool turns = turns_first;  // the kind of the next part of a round
    auto put = [&](const Part* q) {
        for (int j = 0; j < (turns ? 2 : 16); ++j)
            pool->push_back(q ? q->v[j] : turns ? make_double2(0., 0.) : make_double2(1., 0.));
        if (turns) ++phase->rounds;
        turns = !turns;
    };
    for (const Part& q : parts) {
        if (q.turns != turns) put(nullptr);
        put(&q);
    }
    if (turns_first) phase->flags |= PH_TURNS_FIRST;
    else if (turns) phase->flags |= PH_TAIL;
    return true;
}

// Codes: run_step in csrc/staged.cu.
void encode_program(const PhaseProgram& P, std::vector<StStep>* steps, std::vector<double2>* pool, StPhase* phase) {
    auto bit = [](uint8_t v) { return __builtin_ctz(v); };
    phase->step_begin = (uint32_t)steps->size();
    phase->out0 = P.out[0];
    for (int k = 0; k < 4; ++k) phase->out[k] = P.out[1 << k] ^ P.out[0];
    phase->step_count = 0;
    if (encode_rounds(P, phase, pool)) return;
    phase->rounds = 0;
    for (const ProgStep& s : P.steps) {
        StStep t{};
        t.param = (uint32_t)pool->size();
        t.mask = s.mask;
        const int a = s.nq > 0 ? bit(s.v[0]) : 0, b = s.nq > 1 ? bit(s.v[1]) : 0;
        switch (s.kind) {
            case SP_DIAG: t.code = 0; break;
            case SP_SIGN: t.code = 1; break;
            case SP_SCALE: t.code = s.form ? 3 : 2; break;
            case SP_CNOT: t.code = (uint8_t)(16 + a * 4 + b); break;
            case SP_X: t.code = (uint8_t)(16 + a * 5); break;
            case SP_SWAP: t.code = (uint8_t)(32 + std::min(a, b) * 4 + std::max(a, b)); break;
            case SP_DENSE1: t.code = (uint8_t)(32 + a * 5); break;
            case SP_DEPOL1: t.code = (uint8_t)((s.form ? 80 : 32) + std::max(a, b) * 4 + std::min(a, b)); break;
            case SP_DENSE2: t.code = (uint8_t)(48 + a * 4 + b); break;
            case SP_DEPOL2: {  // by the partner of register bit 0: 1, 2 or 3
                const int c = bit(s.v[2]), d = bit(s.v[3]);
                const int mate = a == 0 ? c : b == 0 ? d : c == 0 ? a : b;
                t.code = (uint8_t)(48 + (mate - 1) * 5);
                t.mask = s.form;
                break;
            }
            case SP_ROT: t.code = (uint8_t)(64 + (s.form == RF_Y_TAN ? 0 : 4) + a); break;
        }
        if (s.kind == SP_ROT) {  // rotation_form leaves RY alone; a relabelled bit turns the other way
            const double sign = s.a[0] ? -1. : 1.;
            if (s.form == RF_Y_TAN) pool->push_back(make_double2(sign * s.par[0].x, 0.));
            else if (s.form == RF_Y_COT) pool->push_back(make_double2(s.par[0].x, sign));  // cosine and sine over the sine
            else pool->push_back(make_double2(s.par[0].x, sign * s.par[0].y));
        } else {
            pool->insert(pool->end(), s.par.begin(), s.par.end());
        }
        steps->push_back(t);
    }
    phase->step_count = (uint32_t)(steps->size() - phase->step_begin);
}

}  // namespace qs
