// Runs a circuit's staged schedule on a host state: the same passes, phases and programs that the device
// executors run, step by step in double precision.  It checks the planning without a GPU; nothing else
// calls it.
#include <cmath>
#include <complex>
#include <vector>

#include "../../include/qulacs_b200.h"
#include "circuit.hpp"
#include "host_plan.hpp"
#include "phase_program.hpp"

namespace qs {

int set_error(int code, const std::string& msg);

namespace {

using cd = std::complex<double>;

cd mul(const cd& a, const cd& b) {  // cmul of the kernels
    return cd(std::fma(a.real(), b.real(), -a.imag() * b.imag()), std::fma(a.real(), b.imag(), a.imag() * b.real()));
}
cd mul_add(const cd& a, const cd& b, const cd& acc) {  // cfma of the kernels
    return cd(std::fma(-a.imag(), b.imag(), std::fma(a.real(), b.real(), acc.real())),
        std::fma(a.imag(), b.real(), std::fma(a.real(), b.imag(), acc.imag())));
}
cd axpy(double t, const cd& y, const cd& x) { return cd(std::fma(t, y.real(), x.real()), std::fma(t, y.imag(), x.imag())); }
cd at(const double2& v) { return cd(v.x, v.y); }

// x' = c x + s y, y' = c y - s x; with i (RX): x' = c x + i s y, y' = c y + i s x.
void rotate(cd& x, cd& y, double c, double s, bool rx) {
    const cd X = x, sy = rx ? cd(-s * y.imag(), s * y.real()) : s * y, sx = rx ? cd(-s * X.imag(), s * X.real()) : -s * X;
    x = axpy(c, X, sy);
    y = axpy(c, y, sx);
}
void scaled_rotation(cd& x, cd& y, double t, bool rx) {
    const cd X = x;
    if (rx) {
        x = cd(std::fma(-t, y.imag(), X.real()), std::fma(t, y.real(), X.imag()));
        y = cd(std::fma(-t, X.imag(), y.real()), std::fma(t, X.real(), y.imag()));
    } else {
        x = axpy(t, y, X);
        y = axpy(-t, X, y);
    }
}

void dense(cd* r, const int* idx, int k, const double2* m) {
    cd v[4], o[4];
    for (int x = 0; x < k; ++x) v[x] = r[idx[x]];
    for (int y = 0; y < k; ++y) {
        o[y] = mul(at(m[y * k]), v[0]);
        for (int x = 1; x < k; ++x) o[y] = mul_add(at(m[y * k + x]), v[x], o[y]);
    }
    for (int y = 0; y < k; ++y) r[idx[y]] = o[y];
}
void channel1(cd& x, cd& y, cd& a, cd& b, double t, double k, const double2* full) {
    if (full) {
        x *= full->x;
        y *= full->x;
    }
    const cd X = x;
    x = axpy(t, y, X);
    y = axpy(t, X, y);
    a *= k;
    b *= k;
}
void channel2(cd* r, const int* pop, double t, double k, bool full) {
    const cd S = (r[pop[0]] + r[pop[1]]) + (r[pop[2]] + r[pop[3]]);
    if (full)
        for (int j = 0; j < 16; ++j) r[j] *= k;
    for (int i = 0; i < 4; ++i) r[pop[i]] = axpy(t, S, r[pop[i]]);
}

// A step as pass_codegen.cpp emits it.
void run_spec(const ProgStep& s, cd* r) {
    auto coset = [&](int b, int k) {
        int j = b;
        for (int i = 0; i < s.nq; ++i)
            if (((k >> i) & 1) != step_bit(s, i, j)) j ^= s.v[i];
        return j;
    };
    for (int j = 0; j < 16; ++j) {
        if (s.kind == SP_DIAG && ((s.mask >> j) & 1)) r[j] = mul(at(s.par[j]), r[j]);
        if (s.kind == SP_SIGN && ((s.mask >> j) & 1)) r[j] = -r[j];
        if (s.kind == SP_SCALE) r[j] = s.form ? mul(at(s.par[0]), r[j]) : s.par[0].x * r[j];
    }
    if (s.kind == SP_DIAG || s.kind == SP_SIGN || s.kind == SP_SCALE) return;
    for (int j = 0; j < 16; ++j) {
        bool base = true;
        for (int i = 0; i < s.nq; ++i) base = base && !step_bit(s, i, j);
        if (!base) continue;
        const int o[4] = {j, coset(j, 1), coset(j, 2), coset(j, 3)};
        switch (s.kind) {
            case SP_X: std::swap(r[j], r[o[1]]); break;
            case SP_CNOT: std::swap(r[o[1]], r[o[3]]); break;
            case SP_SWAP: std::swap(r[o[1]], r[o[2]]); break;
            case SP_ROT: {
                const bool rx = s.form >= RF_X_TAN;
                const double t = s.par[0].x;
                if (s.form == RF_Y_TAN || s.form == RF_X_TAN) scaled_rotation(r[j], r[o[1]], t, rx);
                else if (s.form == RF_Y_COT || s.form == RF_X_COT) rotate(r[j], r[o[1]], t, 1., rx);
                else rotate(r[j], r[o[1]], t, s.par[0].y, rx);
                break;
            }
            case SP_DENSE1: dense(r, o, 2, s.par.data()); break;
            case SP_DENSE2: dense(r, o, 4, s.par.data()); break;
            case SP_DEPOL1: channel1(r[j], r[o[3]], r[o[1]], r[o[2]], s.par[0].x, s.par[0].y, s.form ? &s.par[1] : nullptr); break;
            case SP_DEPOL2: {
                const int pop[4] = {j, coset(j, 5), coset(j, 10), coset(j, 15)};
                channel2(r, pop, s.par[0].x, s.form ? s.par[0].y : 1., s.form != 0);
                break;
            }
            default: break;
        }
    }
}

// A step as run_step in csrc/staged.cu decodes it.
void run_code(const StStep& s, const double2* p, cd* r) {
    const int kind = s.code >> 4, V = s.code & 15, A = V >> 2, B = V & 3, a = 1 << A, b = 1 << B;
    for (int j = 0; j < 16; ++j) {
        const int o[4] = {j, j | a, j | b, j | a | b};
        const bool base1 = !(j & a), base1b = !(j & b), base2 = base1 && base1b;
        if (s.code == 0) {
            if ((s.mask >> j) & 1) r[j] = mul(at(p[j]), r[j]);
        } else if (s.code == 1) {
            if ((s.mask >> j) & 1) r[j] = -r[j];
        } else if (s.code == 2) r[j] *= p[0].x;
        else if (s.code == 3) r[j] = mul(at(p[0]), r[j]);
        else if (kind == 1 && A != B) {
            if (base2) std::swap(r[o[1]], r[o[3]]);
        } else if (kind == 1) {
            if (base1) std::swap(r[j], r[o[1]]);
        } else if (kind == 2 && A < B) {
            if (base2) std::swap(r[o[1]], r[o[2]]);
        } else if (kind == 2 && A == B) {
            if (base1) dense(r, o, 2, p);
        } else if (kind == 2) {
            if (base2) channel1(r[j], r[o[3]], r[o[1]], r[o[2]], p[0].x, p[0].y, nullptr);
        } else if (kind == 5) {
            if (base2) channel1(r[j], r[o[3]], r[o[1]], r[o[2]], p[0].x, p[0].y, p + 1);
        } else if (kind == 3 && A != B) {
            if (base2) dense(r, o, 4, p);
        } else if (kind == 3) {
            const int mate = 1 | (1 << (A + 1)), pop[4] = {0, mate, 15 ^ mate, 15};
            if (j == 0) channel2(r, pop, p[0].x, p[0].y, s.mask != 0);
        } else if (base1b) {
            if (A == 0) scaled_rotation(r[j], r[j | b], p[0].x, false);
            else rotate(r[j], r[j | b], p[0].x, p[0].y, false);
        }
    }
}

void run_generic(const StPhase& P, const HostPlan& H, cd* r) {
    for (uint32_t o = 0; o < P.step_count; ++o) {
        const StStep& s = H.steps[P.step_begin + o];
        run_code(s, H.params.data() + s.param, r);
    }
    if (P.step_count) return;
    const double2* p = H.params.data() + P.param;
    auto factors = [&]() {
        for (int j = 0; j < 16; ++j) r[j] = mul(at(p[j]), r[j]);
        p += 16;
    };
    for (uint32_t o = 0; o < P.rounds; ++o) {
        if (!(P.flags & PH_TURNS_FIRST)) factors();
        const double t[4] = {p[0].x, p[0].y, p[1].x, p[1].y};
        for (int b = 0; b < 4; ++b)
            for (int j = 0; j < 16; ++j)
                if (!((j >> b) & 1)) scaled_rotation(r[j], r[j | (1 << b)], t[b], false);
        p += 2;
        if (P.flags & PH_TURNS_FIRST) factors();
    }
    if (P.flags & PH_TAIL) factors();
}

void apply_single(const GateRec& g, cd* state, ITYPE dim) {
    const std::vector<cd> m = g.dense_matrix();
    const size_t md = size_t(1) << g.targets.size();
    ITYPE tmask = 0, cmask = 0, cval = 0;
    for (UINT t : g.targets) tmask |= 1ULL << t;
    for (size_t j = 0; j < g.controls.size(); ++j) {
        cmask |= 1ULL << g.controls[j];
        if (g.control_values[j]) cval |= 1ULL << g.controls[j];
    }
    std::vector<cd> v(md);
    for (ITYPE base = 0; base < dim; ++base) {
        if ((base & tmask) || (base & cmask) != cval) continue;
        auto index = [&](size_t x) {
            ITYPE i = base;
            for (size_t j = 0; j < g.targets.size(); ++j)
                if ((x >> j) & 1) i |= 1ULL << g.targets[j];
            return i;
        };
        for (size_t x = 0; x < md; ++x) v[x] = state[index(x)];
        for (size_t y = 0; y < md; ++y) {
            cd acc = 0.;
            for (size_t x = 0; x < md; ++x) acc += m[y * md + x] * v[x];
            state[index(y)] = acc;
        }
    }
}

void run_pass(const HostPlan& H, size_t pass, bool spec, cd* state, ITYPE dim) {
    const std::vector<UINT>& q = H.passes[pass].q;
    const int m = (int)q.size();
    ITYPE tile = 0;
    for (UINT b : q) tile |= 1ULL << b;
    auto global = [&](ITYPE base, UINT u) {
        for (int j = 0; j < m; ++j)
            if ((u >> j) & 1) base |= 1ULL << q[j];
        return base;
    };
    for (ITYPE base = 0; base < dim; ++base) {
        if (base & tile) continue;
        for (size_t ph = 0; ph < H.pp[pass].nphases; ++ph) {
            const size_t at = H.pp[pass].phase_begin + ph;
            const StPhase& P = H.phases[at];
            UINT bits = 0;
            for (int b = 0; b < kPhaseBits; ++b) bits |= 1u << P.bits[b];
            for (UINT u = 0; u < (1u << m); ++u) {
                if (u & bits) continue;
                auto index = [&](UINT i) {
                    UINT v = u;
                    for (int b = 0; b < kPhaseBits; ++b)
                        if ((i >> b) & 1) v |= 1u << P.bits[b];
                    return global(base, v);
                };
                cd r[16];
                for (UINT j = 0; j < 16; ++j) {
                    UINT i = 0;
                    for (int b = 0; b < kPhaseBits; ++b)
                        if ((j >> b) & 1) i ^= P.in[b];
                    r[j] = state[index(i)];
                }
                if (spec)
                    for (const ProgStep& s : H.programs[at].steps) run_spec(s, r);
                else
                    run_generic(P, H, r);
                for (UINT j = 0; j < 16; ++j) {
                    UINT i = spec ? H.programs[at].out[j] : P.out0;
                    if (!spec)
                        for (int b = 0; b < kPhaseBits; ++b)
                            if ((j >> b) & 1) i ^= P.out[b];
                    state[index(i)] = r[j];
                }
            }
        }
    }
}

}  // namespace
}  // namespace qs

// `circuit` on a host state vector of `dim` amplitudes, or with `density_matrix` on the row-major host
// matrix of dim x dim, as the staged executors plan it: block size k (0: no fusion), tiles of 2^tile_bits
// amplitudes, the specialised kernels' programs or the generic kernels'.
extern "C" QS_API int qs_debug_staged_replay(qs_circuit_t circuit, int density_matrix, int k, int specialized,
    QS_UINT tile_bits, double* state, QS_ITYPE dim) {
    const qs::Circuit* c = reinterpret_cast<const qs::Circuit*>(circuit);
    if (!c || !state) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    if (dim != (1ULL << c->n)) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "dim differs from 2^qubit_count");
    const UINT n = density_matrix ? 2 * c->n : c->n;
    if (n < (UINT)qs::kPhaseBits || n > 20) return qs::set_error(QS_ERR_NOT_SUPPORTED, "replay: 4..20 vector qubits");
    if (k < 0 || k > 6 || tile_bits < (QS_UINT)qs::kLowFixed || tile_bits > (QS_UINT)qs::kTileBits)
        return qs::set_error(QS_ERR_INVALID_ARGUMENT, "replay: block size 0..6, tile bits 4..12");
    const std::vector<qs::GateRec> gates = qs::executor_gates(
        density_matrix ? qs::dm_vector_gates(qs::merge_depolarizing(c->gates), c->n) : c->gates, k, specialized != 0);
    qs::HostPlan H;
    qs::make_host_plan(gates, n, &H, (int)tile_bits, specialized != 0);
    std::complex<double>* s = reinterpret_cast<std::complex<double>*>(state);
    for (size_t p = 0; p < H.passes.size(); ++p) {
        if (H.passes[p].single) {
            const qs::GateRec& g = gates[H.passes[p].gate];
            if (g.kind == QS_GATE_DEPOLARIZING)
                return qs::set_error(QS_ERR_NOT_SUPPORTED, "depolarizing noise needs a density matrix");
            qs::apply_single(g, s, 1ULL << n);
        } else {
            qs::run_pass(H, p, specialized != 0, s, 1ULL << n);
        }
    }
    return QS_OK;
}
