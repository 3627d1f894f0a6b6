// Staged executor: many gates per HBM pass.
//
// A pass owns a set Q of m "tile qubits" (always including qubits 0..3, so every HBM access is a
// run of >= 16 contiguous amplitudes = 256 B).  Each CTA loads one tile -- the 2^m amplitudes that
// share the values of the other n - m qubits -- into shared memory, applies every gate of the pass
// (all of whose qubits lie in Q), and writes the tile back: one read and one write of the state per
// pass instead of one per gate.  Inside the tile, gates are grouped into "phases" of at most 4 tile
// qubits: each thread gathers the 16 amplitudes of its 4-qubit coset into registers, applies all the
// phase's gates there, and scatters them back, so shared memory is touched once per phase, not once
// per gate.  A phase's gates run as a program of rotations, collected diagonals and register relabellings
// (phase_program.hpp), which the kernels here interpret step by step; the specialised pass kernels
// (pass_codegen.cpp) run the same programs as straight-line code.  The host scheduler (below) builds passes
// and phases greedily from the gate list in rotation form (fusion.cpp).  The scheduler moves a gate only past
// gates on disjoint qubits; rotation form carries unitary diagonals past controls, CZ, SWAP, diagonals and
// depolarizing channels, with which they commute, and a phase's program reorders steps that commute.  So the
// result equals gate-by-gate application up to rounding (~1e-16), and exactly where gates only permute.  Gates
// the pass kernel does not cover (more than 2 targets, controls, Pauli strings, multi-qubit diagonals) run
// between passes with the gate-by-gate kernels.
//
// What bounds the generic kernel on small states is the chain of rounds in a CTA: one coset per thread (256
// threads for a 2^12-amplitude tile, where 128 threads took two in turn), rotations in place of matrices and
// rounds (run_rounds) brought the layered circuit on 16 qubits from 0.43 to 0.20 ms; CNOTs as relabellings of the
// coset's addresses (relabel_segments; H CZ H on the target before, 42 phases with 197 rounds against 87 with 81)
// to 0.151, with the record of a phase read as four words (some forty loads field by field: 0.157).  20 layers of
// U3 + CZ on 26 qubits took 46.9 ms step by step and 26.5 in rounds (specialised: 16.0).
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstring>
#include <memory>
#include <string>
#include <mutex>
#include <thread>
#include <vector>

#include "circuit.hpp"
#include "host_plan.hpp"
#include "qs_internal.cuh"
#include "phase_program.hpp"
#include "staged.hpp"

namespace qs {

struct StPassArgs {
    int m;                 // tile bits (<= kTileBits)
    int nphases;
    int io;                // bit 0: the first phase gathers from HBM; bit 1: the last phase scatters to HBM
    UINT q[kTileBits];     // global qubit of tile bit j, ascending, q[j] = j for j < kLowFixed
    const StPhase* phases;
    const StStep* steps;
    const double2* pool;   // the steps' parameters
};

// ---------------------------------------------------------------- register steps
// The steps of a phase program (phase_program.hpp) on a thread's 16 amplitudes; the arithmetic of each is
// that of the specialised kernels' (csrc/pass_codegen.cpp), in the same order.
// A parameter read at its use (volatile: a whole matrix is not held in registers).
__device__ __forceinline__ double2 ld_par(const double2* p) {
    double2 v;
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double flipped(double t, unsigned odd) {  // -t where odd is 1
    return __hiloint2double(__double2hiint(t) ^ (int)(odd << 31), __double2loint(t));
}
template <int B>
__device__ __forceinline__ void r_ry_tan(double2 (&r)[16], double t) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << B))) {
            double2 &x = r[j], &y = r[j | (1 << B)];
            const double2 X = x;
            x = make_double2(fma(t, y.x, X.x), fma(t, y.y, X.y));
            y = make_double2(fma(-t, X.x, y.x), fma(-t, X.y, y.y));
        }
}
template <int B>
__device__ __forceinline__ void r_ry_full(double2 (&r)[16], double c, double s) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << B))) {
            double2 &x = r[j], &y = r[j | (1 << B)];
            const double2 X = x;
            x = make_double2(fma(c, X.x, s * y.x), fma(c, X.y, s * y.y));
            y = make_double2(fma(c, y.x, -s * X.x), fma(c, y.y, -s * X.y));
        }
}
__device__ __forceinline__ void r_diag(double2 (&r)[16], const double2* __restrict__ p, unsigned mask) {
#pragma unroll
    for (int h = 0; h < 16; h += 4) {
        double2 d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] = ld_par(p + h + j);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((mask >> (h + j)) & 1u) r[h + j] = cmul(d[j], r[h + j]);
    }
}
__device__ __forceinline__ void r_sign(double2 (&r)[16], unsigned mask) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        r[j] = make_double2(flipped(r[j].x, (mask >> j) & 1u), flipped(r[j].y, (mask >> j) & 1u));
}
template <int B>
__device__ __forceinline__ void r_dense1(double2 (&r)[16], const double2* __restrict__ p) {
    const double2 m0 = p[0], m1 = p[1], m2 = p[2], m3 = p[3];
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << B))) {
            const double2 x = r[j], y = r[j | (1 << B)];
            r[j] = cfma(m1, y, cmul(m0, x));
            r[j | (1 << B)] = cfma(m3, y, cmul(m2, x));
        }
}
// matrix-index bit 0 <-> register bit A (first target), bit 1 <-> B
template <int A, int B>
__device__ __forceinline__ void r_dense2(double2 (&r)[16], const double2* __restrict__ p) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << A)) && !(j & (1 << B))) {
            const int o[4] = {j, j | (1 << A), j | (1 << B), j | (1 << A) | (1 << B)};
            double2 v[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) v[x] = r[o[x]];
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                double2 acc = cmul(ld_par(p + y * 4), v[0]);
#pragma unroll
                for (int x = 1; x < 4; ++x) acc = cfma(ld_par(p + y * 4 + x), v[x], acc);
                r[o[y]] = acc;
            }
        }
}
template <int C, int T>
__device__ __forceinline__ void r_cnot(double2 (&r)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if ((j & (1 << C)) && !(j & (1 << T))) {
            const double2 t = r[j];
            r[j] = r[j | (1 << T)];
            r[j | (1 << T)] = t;
        }
}
template <int A>
__device__ __forceinline__ void r_x(double2 (&r)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << A))) {
            const double2 t = r[j];
            r[j] = r[j | (1 << A)];
            r[j | (1 << A)] = t;
        }
}
template <int A, int B>
__device__ __forceinline__ void r_swap(double2 (&r)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if ((j & (1 << A)) && !(j & (1 << B))) {
            const int k = j ^ (1 << A) ^ (1 << B);
            const double2 t = r[j];
            r[j] = r[k];
            r[k] = t;
        }
}
// One-qubit depolarizing channel, scaled (column and row bit A, B): populations mix, coherences shrink.
template <int A, int B>
__device__ __forceinline__ void r_depol1(double2 (&r)[16], double t, double k) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << A)) && !(j & (1 << B))) {
            double2 &x = r[j], &y = r[j | (1 << A) | (1 << B)];
            const double2 X = x;
            x = make_double2(fma(t, y.x, X.x), fma(t, y.y, X.y));
            y = make_double2(fma(t, X.x, y.x), fma(t, X.y, y.y));
            r[j | (1 << A)] = make_double2(k * r[j | (1 << A)].x, k * r[j | (1 << A)].y);
            r[j | (1 << B)] = make_double2(k * r[j | (1 << B)].x, k * r[j | (1 << B)].y);
        }
}
// The channel itself: the populations shrink by d before they mix.
template <int A, int B>
__device__ __forceinline__ void r_depol1_full(double2 (&r)[16], double t, double k, double d) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (!(j & (1 << A)) == !(j & (1 << B))) r[j] = make_double2(d * r[j].x, d * r[j].y);
    r_depol1<A, B>(r, t, k);
}
// Two-qubit depolarizing channel on pairs of register bits (0, MATE) and the other two: the four populations
// have equal bits in each pair.
template <int MATE>
__device__ __forceinline__ void r_depol2(double2 (&r)[16], double t, double k, bool full) {
    constexpr int p = 1 | (1 << MATE), q = 15 ^ p;
    const double2 S = make_double2((r[0].x + r[p].x) + (r[q].x + r[15].x), (r[0].y + r[p].y) + (r[q].y + r[15].y));
    if (full) {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = make_double2(k * r[j].x, k * r[j].y);
    }
    for (int j : {0, p, q, 15}) r[j] = make_double2(fma(t, S.x, r[j].x), fma(t, S.y, r[j].y));
}

// One indirect branch per step: the host's code (encode_program) selects fully specialised register code.
//   0 diagonal, 1 signs, 2 real and 3 complex scale;  16..31 CNOT a * 4 + b, X at a = b;
//   32..47 SWAP (a < b), one-qubit matrix (a = b), one-qubit channel (a > b);
//   48..63 two-qubit matrix, two-qubit channel at a = b (register bit 0's partner a + 1);
//   64..67 RY scaled, 68..71 RY with cosine and sine;  80.. one-qubit channel unscaled (a > b).
template <int CODE>
__device__ __forceinline__ void run_step(double2 (&r)[16], const double2* __restrict__ p, unsigned mask) {
    constexpr int kind = CODE >> 4, V = CODE & 15, A = V >> 2, B = V & 3;
    if constexpr (CODE == 0) r_diag(r, p, mask);
    else if constexpr (CODE == 1) r_sign(r, mask);
    else if constexpr (CODE == 2) {
        const double k = p[0].x;
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = make_double2(k * r[j].x, k * r[j].y);
    } else if constexpr (CODE == 3) {
        const double2 z = p[0];
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = cmul(z, r[j]);
    } else if constexpr (kind == 1 && A != B) r_cnot<A, B>(r);
    else if constexpr (kind == 1) r_x<A>(r);
    else if constexpr (kind == 2 && A < B) r_swap<A, B>(r);
    else if constexpr (kind == 2 && A == B) r_dense1<A>(r, p);
    else if constexpr (kind == 2) r_depol1<A, B>(r, p[0].x, p[0].y);
    else if constexpr (kind == 3 && A != B) r_dense2<A, B>(r, p);
    else if constexpr (kind == 3 && A < 3) r_depol2<A + 1>(r, p[0].x, p[0].y, mask != 0);
    else if constexpr (kind == 4 && A == 0) r_ry_tan<B>(r, p[0].x);
    else if constexpr (kind == 4 && A == 1) r_ry_full<B>(r, p[0].x, p[0].y);
    else if constexpr (kind == 5 && A > B) r_depol1_full<A, B>(r, p[0].x, p[0].y, p[1].x);
}
#define QS_CODE1(c) \
    case c: run_step<c>(r, p, s.mask); break;
#define QS_CODE4(c) QS_CODE1(c) QS_CODE1(c + 1) QS_CODE1(c + 2) QS_CODE1(c + 3)
#define QS_CODE16(c) QS_CODE4(c) QS_CODE4(c + 4) QS_CODE4(c + 8) QS_CODE4(c + 12)
__device__ __forceinline__ void apply_step(const StStep& s, double2 (&r)[16], const double2* __restrict__ pool) {
    const double2* p = pool + s.param;
    switch (s.code) {
        QS_CODE4(0)
        QS_CODE16(16)
        QS_CODE16(32)
        QS_CODE16(48)
        QS_CODE4(64)
        QS_CODE4(68)
        QS_CODE16(80)
        default: break;
    }
}
#undef QS_CODE16
#undef QS_CODE4
#undef QS_CODE1

// Rounds of 16 diagonal factors and a scaled rotation on each register bit, in either order (factor 1, tangent 0
// where there is none): straight-line code on fixed registers.  Conditions around the parts, or the switch over
// step kinds, cost moves of the whole coset at every join: the FP64 pipe was 15 % busy at 63 % issue with the
// switch, 20 % with conditions, 35 % (46 % in the fullest passes) with rounds.  A condition between rotations and
// factors, in place of the two orders, cost 20 % of a 10-qubit circuit: the factors' loads waited behind it.
// Reading factors ahead across rounds gained 3 % at 14 qubits and lost 3 % at 26, and was not kept.
__device__ __forceinline__ void r_turns(double2 (&r)[16], const double2* __restrict__ p) {
    const double2 t01 = ld_par(p), t23 = ld_par(p + 1);
    r_ry_tan<0>(r, t01.x);
    r_ry_tan<1>(r, t01.y);
    r_ry_tan<2>(r, t23.x);
    r_ry_tan<3>(r, t23.y);
}
__device__ __forceinline__ void run_rounds(const StPhase& P, double2 (&r)[16], const double2* __restrict__ p) {
    if (P.flags & PH_TURNS_FIRST) {
#pragma unroll 1
        for (UINT o = 0; o < P.rounds; ++o, p += 18) {
            r_turns(r, p);
            r_diag(r, p + 2, 0xffffu);
        }
        return;
    }
#pragma unroll 1
    for (UINT o = 0; o < P.rounds; ++o, p += 18) {
        r_diag(r, p, 0xffffu);
        r_turns(r, p + 16);
    }
    if (P.flags & PH_TAIL) r_diag(r, p, 0xffffu);
}

__device__ __forceinline__ UINT swz(UINT u) { return QS_SWZ(u); }

// Tile index u = tid + k * threads has global offset base | lo_off | hi_off[k]: lo_off takes tid's bits to
// the lowest tile qubits, hi_off[k] takes k's bits to the others.

// Global rows of 16 amplitudes per thread from the swizzled tile to HBM.
template <UINT threads, class T>
__device__ __forceinline__ void tile_rows_store(T* __restrict__ s, const double2* tile, ITYPE off,
    const ITYPE* hi_off, UINT tsize) {
    const UINT tid = threadIdx.x;
    double2 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (tid + (UINT)k * threads < tsize) v[k] = tile[swz(tid + (UINT)k * threads)];
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (tid + (UINT)k * threads < tsize) st_amp(s + (off | hi_off[k]), v[k]);
}

// One tile of one pass: load, apply every phase, store.  Shared by the per-pass kernel and the
// persistent multi-circuit kernel.  `tile` holds 2^m amplitudes (m <= MAX_BITS) in FP64 whatever the
// state's type E (complex128, or complex64 widened on load and rounded on store).  One 16-amplitude coset per
// thread and phase, for the cosets of the largest tile.  Ends with a CTA barrier so the shared buffers can be
// reused immediately.
// STEPS: whether a phase may be a list of steps; without, every phase is rounds.
template <int MAX_BITS, bool STEPS, class E>
__device__ __forceinline__ void staged_tile(E* __restrict__ s, const StPassArgs& a, ITYPE T, double2* tile,
    ITYPE* hi_off) {
    constexpr int tb = MAX_BITS - kPhaseBits;
    constexpr UINT threads = 1u << tb;
    const int m = a.m;
    const UINT tsize = 1u << m;
    // base: insert zeros at the tile qubits into the tile index
    ITYPE base = T;
    for (int j = 0; j < m; ++j) base = insert0(base, a.q[j]);
    const int tid = threadIdx.x;
    const bool hbm_first = a.io & 1, hbm_last = (a.io >> 1) & 1;
    ITYPE lo_off = 0;
    if (!hbm_first || !hbm_last) {
        if (tid < 16) {
            ITYPE o = 0;
            for (int j = tb; j < m; ++j)
                if ((tid >> (j - tb)) & 1) o |= 1ULL << a.q[j];
            hi_off[tid] = o;
        }
        for (int j = 0; j < tb && j < m; ++j)
            if ((tid >> j) & 1) lo_off |= 1ULL << a.q[j];
        __syncthreads();
    }
    if (!hbm_first) {
        const ITYPE off = base | lo_off;
        if constexpr (sizeof(E) == sizeof(double2)) {
            // 16-byte cp.async copies straight into the swizzled tile: every copy of a thread in flight at
            // once, without holding registers
#pragma unroll
            for (int k = 0; k < 16; ++k)
                if ((UINT)tid + (UINT)k * threads < tsize) {
                    const unsigned dst =
                        (unsigned)__cvta_generic_to_shared(tile + swz((UINT)tid + (UINT)k * threads));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(s + (off | hi_off[k]))
                                 : "memory");
                }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        } else {
            // complex64: widened in registers, 8 loads in flight per thread before their stores
#pragma unroll
            for (int k0 = 0; k0 < 16; k0 += 8) {
                double2 v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if ((UINT)tid + (UINT)(k0 + k) * threads < tsize) v[k] = ld_amp(s + (off | hi_off[k0 + k]));
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if ((UINT)tid + (UINT)(k0 + k) * threads < tsize)
                        tile[swz((UINT)tid + (UINT)(k0 + k) * threads)] = v[k];
            }
        }
        __syncthreads();
    }
    const UINT ncos = tsize >> kPhaseBits;  // cosets per phase
    char* tile_bytes = reinterpret_cast<char*>(tile);
    for (int ph = 0; ph < a.nphases; ++ph) {
        StPhase P;
        {  // whole words: field by field it is some forty loads
            uint4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = reinterpret_cast<const uint4*>(a.phases + ph)[i];
            memcpy(&P, w, sizeof(P));
        }
        // The first phase may gather its cosets straight from HBM and the last scatter them straight to
        // HBM (the host sets this when the phase's bits are all >= 4, so that a coset's lanes 0..15 cover
        // 16 consecutive amplitudes): no tile load or store round through shared memory.
        const bool from_hbm = hbm_first && ph == 0, to_hbm = hbm_last && ph == a.nphases - 1;
        if ((UINT)tid < ncos) {
            UINT u0 = 0;
#pragma unroll
            for (int k = 0; k < tb; ++k) u0 |= ((tid >> k) & 1u) << P.order[k];
            ITYPE g0 = base;  // global index of the coset's first amplitude (only for HBM phases)
            if (from_hbm || to_hbm)
                for (int j = 0; j < m; ++j)
                    if ((u0 >> j) & 1) g0 |= 1ULL << a.q[j];
            auto global_bits = [&](UINT i) {  // qubits of coset index i
                ITYPE u = 0;
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if ((i >> p) & 1u) u |= 1ULL << a.q[P.bits[p]];
                return u;
            };
            double2 r[16];
            // Offset of register j from the coset's first amplitude: the XOR of one offset per set bit of j (the
            // relabelling and the swizzle are XOR-linear).  The 16 amplitudes are visited in Gray-code order, so
            // that each address is the previous one with one offset XORed in.
            if (from_hbm) {
                ITYPE gb[4], gi = g0;
#pragma unroll
                for (int p = 0; p < 4; ++p) gb[p] = global_bits(P.in[p]);
#pragma unroll
                for (int g = 0; g < 16; ++g) {
                    if (g) gi ^= gb[(g & 1) ? 0 : (g & 2) ? 1 : (g & 4) ? 2 : 3];
                    r[g ^ (g >> 1)] = ld_amp(s + gi);
                }
            } else {
                UINT addr = swz(u0) << 4;
#pragma unroll
                for (int g = 0; g < 16; ++g) {
                    if (g) addr ^= P.in_at[(g & 1) ? 0 : (g & 2) ? 1 : (g & 4) ? 2 : 3];
                    r[g ^ (g >> 1)] = *reinterpret_cast<const double2*>(tile_bytes + addr);
                }
            }
            if constexpr (STEPS) {
                if (P.step_count == 0) {
                    run_rounds(P, r, a.pool + P.param);
                } else {
                    for (UINT o = 0; o < P.step_count; ++o) apply_step(a.steps[P.step_begin + o], r, a.pool);
                }
            } else {
                run_rounds(P, r, a.pool + P.param);
            }
            // register j goes to coset index out0 ^ (XOR of out[k] over the bits k of j)
            if (to_hbm) {
                ITYPE gb[4], gi = g0 | global_bits(P.out0);
#pragma unroll
                for (int p = 0; p < 4; ++p) gb[p] = global_bits(P.out[p]);
#pragma unroll
                for (int g = 0; g < 16; ++g) {
                    if (g) gi ^= gb[(g & 1) ? 0 : (g & 2) ? 1 : (g & 4) ? 2 : 3];
                    st_amp(s + gi, r[g ^ (g >> 1)]);
                }
            } else {
                UINT addr = (swz(u0) << 4) ^ P.out0_at;
#pragma unroll
                for (int g = 0; g < 16; ++g) {
                    if (g) addr ^= P.out_at[(g & 1) ? 0 : (g & 2) ? 1 : (g & 4) ? 2 : 3];
                    *reinterpret_cast<double2*>(tile_bytes + addr) = r[g ^ (g >> 1)];
                }
            }
        }
        if (!to_hbm && !(P.flags & PH_SAME_NEXT)) __syncthreads();  // the next phase's cosets are these: each thread's own
    }
    if (!hbm_last) tile_rows_store<threads>(s, tile, base | lo_off, hi_off, tsize);
    __syncthreads();
}

// One CTA per tile; the tile (2^m x 16 bytes, up to 64 KiB) is dynamic shared memory.  CTAS: per SM.
template <class E, bool STEPS, int CTAS>
__global__ void __launch_bounds__(kStThreads, CTAS) k_staged_pass(E* __restrict__ s, const __grid_constant__ StPassArgs a) {
    extern __shared__ double2 st_tile[];
    __shared__ ITYPE hi_off[16];
    staged_tile<kTileBits, STEPS>(s, a, blockIdx.x, st_tile, hi_off);
}
template <class E>
using PassKernel = void (*)(E* __restrict__, StPassArgs);
// Two CTAs of 256 threads per SM leave 128 registers: enough for rounds, not for lists of steps (1.2 KB of spill).
// A state of no more tiles than SMs has one CTA on each either way: without the bound its kernels need 184 to 190
// registers and read further ahead.  In us with one bound for all, and so: 10 qubits, layered 65 48, U3 + CZ 75 56;
// 32 two-qubit matrices at 8 qubits 44 36, 64 at 16 qubits 124 110.
template <class E>
static PassKernel<E> pass_kernel(bool steps, ITYPE tiles) {
    const bool few = tiles <= (ITYPE)sm_count();
    return steps ? (few ? k_staged_pass<E, true, 1> : k_staged_pass<E, true, 2>)
                 : (few ? k_staged_pass<E, false, 1> : k_staged_pass<E, false, 2>);
}

// Opt k_staged_pass in to 64 KiB of dynamic shared memory, once per device.
static int staged_allow_smem() {
    static std::mutex mu;
    static std::vector<char> done;
    int dev = 0;
    QS_CUDA_CHECK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if ((int)done.size() <= dev) done.resize(dev + 1, 0);
    if (!done[dev]) {
        for (const void* f : {(const void*)k_staged_pass<double2, false, 1>, (const void*)k_staged_pass<double2, false, 2>,
                 (const void*)k_staged_pass<double2, true, 1>, (const void*)k_staged_pass<double2, true, 2>,
                 (const void*)k_staged_pass<float2, false, 1>, (const void*)k_staged_pass<float2, false, 2>,
                 (const void*)k_staged_pass<float2, true, 1>, (const void*)k_staged_pass<float2, true, 2>})
            QS_CUDA_CHECK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                (int)(sizeof(double2) << kTileBits)));
        done[dev] = 1;
    }
    return QS_OK;
}


// ---------------------------------------------------------------- host scheduler
using cd = std::complex<double>;

static bool stageable(const GateRec& g) {
    if (!g.controls.empty()) return false;
    if (g.depol) return true;
    switch (g.kind) {
        case QS_GATE_RX:
        case QS_GATE_RY:
        case QS_GATE_RZ:
        case QS_GATE_CNOT:
        case QS_GATE_CZ:
        case QS_GATE_SWAP: return true;
        case QS_GATE_DENSE: return g.targets.size() <= 2;
        case QS_GATE_DIAGONAL: return g.targets.size() == 1;
        default: return false;
    }
}

// Whether a gate acts on a phase's registers as a matrix or a channel (build_pass_program's `move`): one that
// flips, or is diagonal, does not.
static bool mixes_registers(const GateRec& g) {
    if (g.depol) return true;
    if (g.kind != QS_GATE_DENSE) return false;
    const cd zero(0.);
    return g.targets.size() > 1 || !((g.matrix[0] == zero && g.matrix[3] == zero) || (g.matrix[1] == zero && g.matrix[2] == zero));
}

// A gate as the scheduler sees it.
struct GateMask {
    ITYPE q;    // its qubits
    bool stage;  // runs inside passes
};

// Absorb greedily in program order with a fixed tile set; returns the absorbed gate indices.
static void absorb(const std::vector<GateMask>& G, const std::vector<int>& pending, ITYPE Q, UINT n,
    std::vector<int>* got) {
    std::vector<int>& out = *got;
    out.clear();
    ITYPE blocked = 0;
    const ITYPE all = (n >= 64) ? ~0ULL : ((1ULL << n) - 1);
    for (int gi : pending) {
        const ITYPE gm = G[gi].q;
        if ((gm & blocked) || !G[gi].stage || (gm & ~Q)) {
            blocked |= gm;
            if ((blocked & all) == all) break;
            continue;
        }
        out.push_back(gi);
    }
}

// Grow Q greedily in program order (capacity m), absorbing as we go.
static ITYPE greedy_q(const std::vector<GateMask>& G, const std::vector<int>& pending, ITYPE Q, int m) {
    ITYPE blocked = 0;
    for (int gi : pending) {
        const ITYPE gm = G[gi].q;
        if ((gm & blocked) || !G[gi].stage) {
            blocked |= gm;
            continue;
        }
        if ((gm & ~Q) == 0) continue;
        if (__builtin_popcountll(Q | gm) <= m) Q |= gm;
        else blocked |= gm;
    }
    return Q;
}

static std::vector<PassPlan> plan_passes(const std::vector<GateRec>& gates, UINT n, int tile_bits) {
    std::vector<PassPlan> plan;
    std::vector<GateMask> G(gates.size());
    for (size_t i = 0; i < G.size(); ++i) {
        G[i] = {0, stageable(gates[i])};
        for (UINT q : gates[i].targets) G[i].q |= 1ULL << q;
        for (UINT q : gates[i].controls) G[i].q |= 1ULL << q;
    }
    std::vector<char> taken(G.size(), 0);
    std::vector<int> got, best;
    std::vector<int> pending(G.size());
    for (size_t i = 0; i < G.size(); ++i) pending[i] = (int)i;
    const int m = (int)std::min<UINT>((UINT)tile_bits, n);
    const int low = std::min(kLowFixed, m);
    const ITYPE lowmask = (1ULL << low) - 1;
    while (!pending.empty()) {
        if (!G[pending[0]].stage) {
            PassPlan p;
            p.single = true;
            p.gate = pending[0];
            plan.push_back(p);
            pending.erase(pending.begin());
            continue;
        }
        // candidate tile sets: greedy in program order, and windows of consecutive high qubits
        std::vector<ITYPE> cands;
        cands.push_back(greedy_q(G, pending, lowmask, m));
        for (int a = low; a + (m - low) <= (int)n; ++a) {
            ITYPE Q = lowmask;
            for (int j = 0; j < m - low; ++j) Q |= 1ULL << (a + j);
            cands.push_back(Q);
        }
        best.clear();
        ITYPE bestQ = 0;
        for (ITYPE Q : cands) {
            absorb(G, pending, Q, n, &got);
            if (got.size() > best.size()) {
                best.swap(got);
                bestQ = Q;
            }
        }
        if (best.empty()) {  // cannot happen for a stageable front gate; keep progress anyway
            PassPlan p;
            p.single = true;
            p.gate = pending[0];
            plan.push_back(p);
            pending.erase(pending.begin());
            continue;
        }
        // pad Q to m qubits with the lowest unused ones
        for (UINT q = 0; q < n && __builtin_popcountll(bestQ) < m; ++q) bestQ |= 1ULL << q;
        PassPlan p;
        for (UINT q = 0; q < n; ++q)
            if (bestQ >> q & 1ULL) p.q.push_back(q);
        p.gates = best;
        plan.push_back(p);
        for (int gi : best) taken[gi] = 1;
        pending.erase(std::remove_if(pending.begin(), pending.end(), [&](int gi) { return taken[gi] != 0; }), pending.end());
    }
    return plan;
}

struct DevPass {
    bool single;
    int gate;
    StPassArgs args;
    size_t phase_begin = 0;  // the pass's phases in StagedPlan::phases
    bool steps = false;      // a phase is a list of steps
    void* spec = nullptr;    // specialised kernel of this pass (pass_codegen.cpp), if compiled
    std::vector<double2> spec_params;  // its parameter block
};

template <class E>
static void launch_pass(E* state, const DevPass& d, ITYPE tiles, cudaStream_t st) {
    const size_t smem = sizeof(double2) << d.args.m;  // the tile is FP64 for either state type
    pass_kernel<E>(d.steps, tiles)<<<(unsigned)tiles, kStThreads, smem, st>>>(state, d.args);
}

struct StagedPlan {
    ITYPE dim = 0;
    std::vector<DevPass> passes;
    void* dev = nullptr;  // phases | steps | parameters
    // host copies of the schedule (for specialised pass kernels)
    std::vector<StPhase> phases;
    std::vector<PhaseProgram> programs;
    bool generic = true;       // the generic kernels' programs are on the device
    bool specialized = false;  // every pass has its specialised kernel
    double compile_ms = 0.;    // wall time of compiling them
    ~StagedPlan() {
        if (dev) cudaFree(dev);
    }
};

// The tile bits outside a phase, in the order in which the coset number's bits run over them: three with
// independent swizzle vectors first (the lowest such triple, for conflict-free accesses), the others ascending.
static void lane_order(StPhase* P, int m) {
    std::vector<uint8_t> rest;
    for (int b = 0; b < m; ++b)
        if (b != P->bits[0] && b != P->bits[1] && b != P->bits[2] && b != P->bits[3]) rest.push_back((uint8_t)b);
    const int k = (int)rest.size();
    auto vec = [](UINT b) { return QS_SWZ(1u << b) & 7u; };
    auto pick = [&]() {
        for (int x = 0; x < k; ++x)
            for (int y = x + 1; y < k; ++y)
                for (int z = y + 1; z < k; ++z) {
                    const UINT a = vec(rest[x]), b = vec(rest[y]), c = vec(rest[z]);
                    if (!a || !b || a == b || !c || c == a || c == b || c == (a ^ b)) continue;
                    std::vector<uint8_t> out = {rest[x], rest[y], rest[z]};
                    for (int i = 0; i < k; ++i)
                        if (i != x && i != y && i != z) out.push_back(rest[i]);
                    rest.swap(out);
                    return;
                }
    };
    pick();
    for (int i = 0; i < 8; ++i) P->order[i] = i < k ? rest[i] : 0;
}

// A phase's gates for the generic kernels, which rotate along register bits only.  A CNOT relabels registers (for
// nothing: the coset is read or written under another order), so a rotation must come after those relabellings
// that the phase can start with and before the others; where it cannot, a new phase starts on the same tile bits
// (the coset goes through shared memory).  Phases with matrices or channels stay whole: their CNOTs are steps.
struct Segment {
    std::vector<int> gates;
    uint8_t in[4] = {1, 2, 4, 8};  // StPhase::in
};
template <class F>
static std::vector<Segment> relabel_segments(const std::vector<GateRec>& gates, const std::vector<int>& phase, F reg) {
    std::vector<Segment> out;
    for (int gi : phase)
        if (mixes_registers(gates[gi])) {
            out.emplace_back();
            out.back().gates = phase;
            return out;
        }
    struct Labels {  // functional and vector of each qubit over the register's index
        UINT f[4] = {1, 2, 4, 8}, v[4] = {1, 2, 4, 8};
        void relabel(int kind, int a, int b) {
            if (kind == QS_GATE_CNOT) {
                f[b] ^= f[a];
                v[a] ^= v[b];
            } else if (kind == QS_GATE_SWAP) {
                std::swap(f[a], f[b]);
                std::swap(v[a], v[b]);
            }
        }
    };
    struct Item {
        int gate, kind, a, b;
    };
    std::vector<Item> todo, left;
    for (int gi : phase) {
        const GateRec& g = gates[gi];
        const int a = reg(g.targets[0]);
        todo.push_back({gi, g.kind, a, g.targets.size() > 1 ? reg(g.targets[1]) : a});
    }
    while (!todo.empty()) {
        // relabellings before any rotation of their qubits: the phase starts with them undone, so that they end
        // on register bits
        Labels L;
        UINT turned = 0;
        std::vector<const Item*> lead;
        for (const Item& i : todo) {
            const UINT bits = (1u << i.a) | (1u << i.b);
            const bool moves = i.kind == QS_GATE_CNOT || i.kind == QS_GATE_SWAP;
            if (i.kind == QS_GATE_RX || i.kind == QS_GATE_RY || (bits & turned)) turned |= bits;
            else if (moves) lead.push_back(&i);
        }
        for (size_t k = lead.size(); k-- > 0;) L.relabel(lead[k]->kind, lead[k]->a, lead[k]->b);
        out.emplace_back();
        Segment& S = out.back();
        for (int k = 0; k < 4; ++k) {
            S.in[k] = 0;
            for (int b = 0; b < 4; ++b) S.in[k] |= (uint8_t)(((L.f[b] >> k) & 1u) << b);
        }
        UINT blocked = 0;
        left.clear();
        for (const Item& i : todo) {
            const UINT bits = (1u << i.a) | (1u << i.b);
            const bool rotation = i.kind == QS_GATE_RX || i.kind == QS_GATE_RY;
            if ((bits & blocked) || (rotation && (L.f[i.a] != L.v[i.a] || (L.v[i.a] & (L.v[i.a] - 1))))) {
                blocked |= bits;
                left.push_back(i);
                continue;
            }
            S.gates.push_back(i.gate);
            L.relabel(i.kind, i.a, i.b);
        }
        todo.swap(left);
    }
    return out;
}

void make_host_plan(const std::vector<GateRec>& gates, UINT n, HostPlan* H, int tile_bits, bool spec) {
    H->passes = plan_passes(gates, n, tile_bits);
    const std::vector<PassPlan>& passes = H->passes;
    std::vector<StPhase>& phases = H->phases;
    std::vector<StOp>& ops = H->ops;
    std::vector<double2>& pool = H->pool;
    std::vector<HostPlan::Range>& pp = H->pp;
    for (const PassPlan& p : passes) {
        if (p.single) {
            pp.push_back({0, 0});
            continue;
        }
        const size_t ph0 = phases.size();
        // phases: greedy over the pass's gates (program order) with 4 register bits each
        struct Todo {
            int gate;
            UINT bits;  // its tile-local bits
        };
        std::vector<Todo> todo;
        int local[64];
        for (size_t j = 0; j < p.q.size(); ++j) local[p.q[j]] = (int)j;
        for (int gi : p.gates) {
            UINT bm = 0;
            for (UINT g : gates[gi].targets) bm |= 1u << local[g];
            todo.push_back({gi, bm});
        }
        std::vector<int> got, best;
        const int m = (int)p.q.size();
        while (!todo.empty()) {
            // candidates: greedy in order, and windows of 4 consecutive tile bits
            auto take = [&](UINT R) {
                got.clear();
                UINT blocked = 0;
                for (const Todo& t : todo) {
                    const UINT bm = t.bits;
                    if ((bm & blocked) || (bm & ~R)) {
                        blocked |= bm;
                        continue;
                    }
                    got.push_back(t.gate);
                }
            };
            std::vector<UINT> cands;
            {
                UINT R = 0, blocked = 0;
                for (const Todo& t : todo) {
                    const UINT bm = t.bits;
                    if (bm & blocked) {
                        blocked |= bm;
                        continue;
                    }
                    if (__builtin_popcount(R | bm) <= kPhaseBits) R |= bm;
                    else blocked |= bm;
                }
                cands.push_back(R);
            }
            for (int a0 = 0; a0 + kPhaseBits <= m; ++a0) cands.push_back(((1u << kPhaseBits) - 1) << a0);
            best.clear();
            UINT bestR = 0;
            for (UINT R : cands) {
                take(R);
                if (got.size() > best.size()) {
                    best.swap(got);
                    bestR = R;
                }
            }
            for (int b = 0; b < m && __builtin_popcount(bestR) < kPhaseBits; ++b) bestR |= 1u << b;
            StPhase ph{};
            int nb = 0;
            int regbit[64];
            for (int b = 0; b < m; ++b)
                if (bestR >> b & 1u) {
                    regbit[b] = nb;
                    ph.bits[nb++] = (uint8_t)b;
                }
            lane_order(&ph, m);
            auto rb = [&](UINT gq) { return (uint8_t)regbit[local[gq]]; };
            std::vector<Segment> segments(1);
            if (spec) segments[0].gates = best;
            else segments = relabel_segments(gates, best, rb);
            for (const Segment& segment : segments) {
            std::copy(segment.in, segment.in + 4, ph.in);
            ph.op_begin = (uint32_t)ops.size();
            for (int gi : segment.gates) {
                const GateRec& g = gates[gi];
                StOp op{};
                op.param = (uint32_t)pool.size();
                if (g.depol) {
                    op.kind = g.depol == 1 ? ST_DEPOL1 : ST_DEPOL2;
                    op.a = rb(g.targets[0]);
                    op.b = rb(g.targets[1]);
                    if (g.depol == 2) op.aux = (uint8_t)(rb(g.targets[2]) | rb(g.targets[3]) << 2);
                    pool.push_back(make_double2(g.prob, 0.));
                    ops.push_back(op);
                    continue;
                }
                if (g.extended) {  // parameters as hi + lo
                    op.a = op.b = rb(g.targets[0]);
                    auto split = [&](long double x0, long double y0, long double x1, long double y1, int pairs) {
                        const long double v[2][2] = {{x0, y0}, {x1, y1}};
                        for (int i = 0; i < pairs; ++i) pool.push_back(make_double2((double)v[i][0], (double)v[i][1]));
                        for (int i = 0; i < pairs; ++i)
                            pool.push_back(make_double2((double)(v[i][0] - (double)v[i][0]), (double)(v[i][1] - (double)v[i][1])));
                    };
                    if (g.kind == QS_GATE_DIAGONAL) {
                        op.kind = ST_DIAG1;
                        op.aux = g.free_phase;
                        split(g.xd[0].real(), g.xd[0].imag(), g.xd[1].real(), g.xd[1].imag(), 2);
                    } else {
                        op.kind = g.kind == QS_GATE_RX ? ST_RX : ST_RY;
                        split(g.xc, g.xs, 0.L, 0.L, 1);
                    }
                    ops.push_back(op);
                    continue;
                }
                switch (g.kind) {
                    case QS_GATE_CNOT:
                    case QS_GATE_CZ:
                    case QS_GATE_SWAP:
                        op.kind = g.kind == QS_GATE_CNOT ? ST_CNOT : g.kind == QS_GATE_CZ ? ST_CZ : ST_SWAP;
                        op.a = rb(g.targets[0]);
                        op.b = rb(g.targets[1]);
                        break;
                    default:  // dense 1 or 2 targets
                        if (g.targets.size() == 1) {
                            op.kind = ST_DENSE1;
                            op.a = rb(g.targets[0]);
                            for (int i = 0; i < 4; ++i) pool.push_back(make_double2(g.matrix[i].real(), g.matrix[i].imag()));
                        } else {
                            op.kind = ST_DENSE2;
                            op.a = rb(g.targets[0]);
                            op.b = rb(g.targets[1]);
                            for (int i = 0; i < 16; ++i) pool.push_back(make_double2(g.matrix[i].real(), g.matrix[i].imag()));
                        }
                        break;
                }
                ops.push_back(op);
            }
            ph.op_count = (uint32_t)(ops.size() - ph.op_begin);
            ph.flags = &segment != &segments.back() ? PH_SAME_NEXT : 0;
            phases.push_back(ph);
            }
            size_t at = 0;  // best lists todo's gates in order
            todo.erase(std::remove_if(todo.begin(), todo.end(),
                           [&](const Todo& t) { return at < best.size() && best[at] == t.gate && (++at, true); }),
                todo.end());
        }
        std::vector<PhaseProgram> prog = build_pass_program(phases.data() + ph0, phases.size() - ph0, ops.data(), pool.data());
        for (size_t i = 0; i < prog.size(); ++i) {
            if (spec) {
                H->programs.push_back(std::move(prog[i]));
                continue;
            }
            StPhase& ph = phases[ph0 + i];
            encode_program(prog[i], &H->steps, &H->params, &ph);
            auto at = [&](UINT index) {  // QS_SWZ is linear: the offset of an index is the XOR of its bits' offsets
                UINT u = 0;
                for (int b = 0; b < kPhaseBits; ++b) u |= ((index >> b) & 1u) << ph.bits[b];
                return (uint16_t)(QS_SWZ(u) << 4);
            };
            for (int k = 0; k < 4; ++k) {
                ph.in_at[k] = at(ph.in[k]);
                ph.out_at[k] = at(ph.out[k]);
            }
            ph.out0_at = at(ph.out0);
        }
        pp.push_back({ph0, phases.size() - ph0});
    }
}

static int upload_plan(const HostPlan& H, ITYPE dim, std::shared_ptr<StagedPlan>* out);

static int build_plan(const std::vector<GateRec>& gates, UINT n, ITYPE dim, std::shared_ptr<StagedPlan>* out,
    int tile_bits = kTileBits, bool spec = false) {
    HostPlan H;
    make_host_plan(gates, n, &H, tile_bits, spec);
    return upload_plan(H, dim, out);
}

// Device copy of a host plan (phases | steps | parameters in one allocation) and its launch args.
static int upload_plan(const HostPlan& H, ITYPE dim, std::shared_ptr<StagedPlan>* out) {
    auto P = std::make_shared<StagedPlan>();
    P->dim = dim;
    P->phases = H.phases;
    P->programs = H.programs;
    P->generic = H.programs.empty();
    const std::vector<PassPlan>& passes = H.passes;
    const std::vector<StPhase>& phases = H.phases;
    const std::vector<HostPlan::Range>& pp = H.pp;
    // upload
    const size_t bph = sizeof(StPhase) * phases.size(), bst = sizeof(StStep) * H.steps.size(),
                 bpa = sizeof(double2) * H.params.size();
    const size_t o_steps = (bph + 255) / 256 * 256, o_params = o_steps + (bst + 255) / 256 * 256;
    const size_t total = o_params + bpa + 256;
    QS_CUDA_CHECK(cudaMalloc(&P->dev, total));
    std::vector<char> host(total, 0);
    if (bph) memcpy(host.data(), phases.data(), bph);
    if (bst) memcpy(host.data() + o_steps, H.steps.data(), bst);
    if (bpa) memcpy(host.data() + o_params, H.params.data(), bpa);
    QS_CUDA_CHECK(cudaMemcpy(P->dev, host.data(), total, cudaMemcpyHostToDevice));
    const StPhase* dph = (const StPhase*)P->dev;
    const StStep* dst = (const StStep*)((char*)P->dev + o_steps);
    const double2* dpa = (const double2*)((char*)P->dev + o_params);
    for (size_t i = 0; i < passes.size(); ++i) {
        DevPass d{};
        d.single = passes[i].single;
        d.gate = passes[i].gate;
        if (!d.single) {
            d.args.m = (int)passes[i].q.size();
            for (int j = 0; j < d.args.m; ++j) d.args.q[j] = passes[i].q[j];
            d.args.nphases = (int)pp[i].nphases;
            auto high_bits = [&](const StPhase& ph) {  // all of the phase's tile bits >= 4
                for (int p = 0; p < 4; ++p)
                    if (ph.bits[p] < kLowFixed) return false;
                return true;
            };
            if (pp[i].nphases) {
                if (high_bits(phases[pp[i].phase_begin])) d.args.io |= 1;
                if (high_bits(phases[pp[i].phase_begin + pp[i].nphases - 1])) d.args.io |= 2;
            }
            d.args.phases = dph + pp[i].phase_begin;
            d.phase_begin = pp[i].phase_begin;
            for (size_t ph = 0; ph < pp[i].nphases; ++ph) d.steps = d.steps || phases[d.phase_begin + ph].step_count;
            d.args.steps = dst;
            d.args.pool = dpa;
        }
        P->passes.push_back(d);
    }
    *out = P;
    return QS_OK;
}

static int run_plan(const std::vector<GateRec>& gates, const StagedPlan& P, void* state, ITYPE dim, cudaStream_t st) {
    QS_TRY(staged_allow_smem());
    for (const DevPass& d : P.passes) {
        if (d.single) {
            QS_TRY(apply_gate_by_gate(gates[d.gate], state, dim, st));
            continue;
        }
        const ITYPE tiles = dim >> d.args.m;
        if (d.spec) {
            QS_TRY(launch_specialized_pass(d.spec, (double2*)state, d.spec_params.empty() ? nullptr : d.spec_params.data(),
                tiles, d.args.m, st));
            continue;
        }
        if (!P.generic) return set_error(QS_ERR_CUDA, "staged schedule without its specialised kernels");
        launch_pass((double2*)state, d, tiles, st);
        QS_TRY(check_launch("k_staged_pass"));
    }
    return QS_OK;
}

// The pass as the code generator sees it.
static PassDesc pass_desc(const StagedPlan& P, const DevPass& d) {
    PassDesc pd;
    pd.m = d.args.m;
    pd.io = d.args.io;
    for (int j = 0; j < d.args.m; ++j) pd.q[j] = d.args.q[j];
    pd.nphases = d.args.nphases;
    pd.phases = P.phases.data() + d.phase_begin;
    pd.programs = P.programs.data() + d.phase_begin;
    return pd;
}

// Specialised kernels for every pass of a plan, compiled on host threads in parallel.  On failure the
// error is returned and the plan cannot run: it holds no programs for the generic kernel.
static int specialize_plan(StagedPlan& P) {
    if (P.specialized) return QS_OK;
    std::vector<size_t> todo;
    for (size_t i = 0; i < P.passes.size(); ++i)
        if (!P.passes[i].single && P.passes[i].args.nphases > 0) todo.push_back(i);
    std::vector<void*> handles(P.passes.size(), nullptr);
    std::vector<std::vector<double2>> params(P.passes.size());
    std::vector<int> rcs(P.passes.size(), QS_OK);
    std::vector<std::string> errs(P.passes.size());
    std::atomic<size_t> next{0};
    const auto t0 = std::chrono::steady_clock::now();
    const unsigned nt = std::max(1u, std::min<unsigned>((unsigned)todo.size(), std::thread::hardware_concurrency()));
    std::vector<std::thread> pool;
    for (unsigned t = 0; t < nt; ++t)
        pool.emplace_back([&] {
            for (size_t j; (j = next.fetch_add(1)) < todo.size();) {
                const size_t i = todo[j];
                rcs[i] = specialized_pass_kernel(pass_desc(P, P.passes[i]), &handles[i], &params[i], nullptr);
                if (rcs[i] != QS_OK) errs[i] = qs_get_last_error();
            }
        });
    for (std::thread& t : pool) t.join();
    for (size_t i : todo)
        if (rcs[i] != QS_OK) return set_error(rcs[i], errs[i]);
    for (size_t i : todo) {
        P.passes[i].spec = handles[i];
        P.passes[i].spec_params = std::move(params[i]);
    }
    P.specialized = true;
    P.compile_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return QS_OK;
}

// Whether a circuit's single-state passes use specialised kernels: forced on or off per circuit, else
// for states of at least 2^kSpecializeMinQubits amplitudes (where a pass runs long enough to repay its
// compile time).
constexpr UINT kSpecializeMinQubits = 22;
static bool want_specialized(const Circuit& c, ITYPE dim) {
    if (c.specialize >= 0) return c.specialize == 1;
    return dim >= (1ULL << kSpecializeMinQubits);
}

// Tile size of the generic kernel for a circuit alone.  From 13 to 18 qubits there are at most 64 tiles of 2^12
// amplitudes for 148 SMs: 2^11 spreads each pass over twice the SMs, at about a third more passes.  U3 + CZ (20
// layers), HEA (8), layered (10), U3 + random CNOT and CZ (10), in us by 2^12 and 2^11: 13 qubits 145 129 121 132, 118
// 111 95 106; 16 qubits 218 171 147 203, 190 136 151 187; 18 qubits 282 194 181 225, 231 157 172 202; from 19 on
// there are tiles enough: 273 202 192 277, 308 203 260 321.  Up to 12 qubits one tile of the whole state needs one
// pass.
static int generic_tile_bits(UINT n) { return n >= 13 && n <= 18 ? kTileBits - 1 : kTileBits; }

// The unfused schedule of a circuit, host part: its gates in rotation form and their plan.
static void staged_host_plan(const Circuit& c, ITYPE dim, std::vector<GateRec>* gates, HostPlan* H) {
    const bool spec = want_specialized(c, dim);
    *gates = rotation_form(c.gates, spec);
    make_host_plan(*gates, c.n, H, spec ? kTileBits : generic_tile_bits(c.n), spec);
}

static int ensure_plan(Circuit& c, ITYPE dim) {
    if (c.plan && c.plan->dim == dim) return QS_OK;
    std::shared_ptr<StagedPlan> P;
    std::vector<GateRec> g;
    HostPlan H;
    staged_host_plan(c, dim, &g, &H);
    QS_TRY(upload_plan(H, dim, &P));
    if (want_specialized(c, dim)) QS_TRY(specialize_plan(*P));
    c.rgates.swap(g);
    c.plan = P;
    return QS_OK;
}

int run_staged(Circuit& c, void* state, ITYPE dim, cudaStream_t st) {
    if (c.n < kPhaseBits) {  // too small for a 4-qubit register phase
        for (const GateRec& g : c.gates) QS_TRY(apply_gate_by_gate(g, state, dim, st));
        return QS_OK;
    }
    QS_TRY(ensure_plan(c, dim));
    return run_plan(c.rgates, *c.plan, state, dim, st);
}

// ---- FP64 gate fusion + staged passes, block size and tile shape chosen by measurement.
// The autotuner fuses the gate list for each candidate block size k = 0..6 (0 = unfused), builds its
// staged schedule with 2^12-amplitude tiles, and times every pass's kernel -- the specialised kernel
// when the circuit runs specialised passes, else the generic one -- on a scratch buffer of whole tiles
// (the pass's ops only see tile-local bits, so its tile qubits are remapped to 0..m-1); a pass costs at
// least its HBM time, and gates left outside passes cost one HBM pass each (dense 5- and 6-qubit
// kernels more), or their launch.  The best k is then also tried with 2^11-amplitude tiles (the tile shape).
constexpr int kTuneMaxK = 6;
constexpr int kTuneSlots = kTuneMaxK + 2;  // k = 0..6 at 2^12 tiles, then the best k at 2^11 tiles
constexpr double kTuneHbmBytesPerSec = 6.5e12;  // B200 streaming copy bandwidth

// A gate outside the passes: HBM passes, but at least what its launch and arithmetic take on a state in the L2
// cache (8 to 18 qubits: 3 to 4.2 us up to three targets, 6.2 to 7.8 for four, 10 to 13 for five, 26 to 27 for
// six).  By the HBM time alone 30 five-qubit blocks at 14 qubits cost nothing: 412 us were chosen over 122.
static double single_gate_ms(const GateRec& g, double hbm_ms) {
    const size_t k = g.targets.size() + g.controls.size();
    const bool dense = g.kind == QS_GATE_DENSE;
    if (dense && k == 5) return std::max(0.012, 2.0 * hbm_ms);
    if (dense && k >= 6) return std::max(0.026, 6.5 * hbm_ms);  // k_denseK_blk: 33 ms against a 5.3 ms pass at 30 qubits
    return std::max(dense && k == 4 ? 0.0065 : 0.0042, hbm_ms);
}

static int estimate_plan_ms(const std::vector<GateRec>& gates, const StagedPlan& P, ITYPE dim, cudaStream_t st,
    bool specialized, double* out_ms) {
    const double hbm_ms = 2.0 * 16.0 * (double)dim / kTuneHbmBytesPerSec * 1e3;
    QS_TRY(staged_allow_smem());
    // specialised kernels of the remapped passes, compiled on host threads in parallel
    std::vector<void*> spec(P.passes.size(), nullptr);
    std::vector<std::vector<double2>> sparams(P.passes.size());
    if (specialized) {
        std::vector<size_t> todo;
        for (size_t i = 0; i < P.passes.size(); ++i)
            if (!P.passes[i].single && P.passes[i].args.nphases > 0) todo.push_back(i);
        std::vector<int> rcs(P.passes.size(), QS_OK);
        std::vector<std::string> errs(P.passes.size());
        std::atomic<size_t> next{0};
        const unsigned nt =
            std::max(1u, std::min<unsigned>((unsigned)todo.size(), std::thread::hardware_concurrency()));
        std::vector<std::thread> pool;
        for (unsigned t = 0; t < nt; ++t)
            pool.emplace_back([&] {
                for (size_t j; (j = next.fetch_add(1)) < todo.size();) {
                    const size_t i = todo[j];
                    PassDesc pd = pass_desc(P, P.passes[i]);
                    for (int b = 0; b < pd.m; ++b) pd.q[b] = (UINT)b;
                    rcs[i] = specialized_pass_kernel(pd, &spec[i], &sparams[i], nullptr);
                    if (rcs[i] != QS_OK) errs[i] = qs_get_last_error();
                }
            });
        for (std::thread& t : pool) t.join();
        for (size_t i : todo)
            if (rcs[i] != QS_OK) return set_error(rcs[i], errs[i]);
    }
    double total = 0.;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    QS_CUDA_CHECK(cudaEventCreate(&e0));
    QS_CUDA_CHECK(cudaEventCreate(&e1));
    int rc = QS_OK;
    for (size_t i = 0; i < P.passes.size(); ++i) {
        const DevPass& d = P.passes[i];
        if (d.single) {
            total += single_gate_ms(gates[d.gate], hbm_ms);
            continue;
        }
        const ITYPE tiles = dim >> d.args.m;
        const ITYPE tt = std::min<ITYPE>(tiles, (ITYPE)sm_count() * 3 * 4);
        void* buf = nullptr;
        rc = scratch(st, (size_t)(tt << d.args.m) * sizeof(double2), &buf);
        if (rc != QS_OK) break;
        StPassArgs a = d.args;
        for (int j = 0; j < a.m; ++j) a.q[j] = (UINT)j;
        DevPass dt = d;
        dt.args = a;
        auto launch = [&]() -> int {
            if (spec[i])
                return launch_specialized_pass(spec[i], (double2*)buf, sparams[i].empty() ? nullptr : sparams[i].data(),
                    tt, a.m, st);
            launch_pass((double2*)buf, dt, tt, st);
            return check_launch("k_staged_pass");
        };
        rc = launch();  // warm-up
        if (rc != QS_OK) break;
        cudaEventRecord(e0, st);
        rc = launch();
        cudaEventRecord(e1, st);
        if (rc != QS_OK) break;
        if (cudaEventSynchronize(e1) != cudaSuccess) {
            rc = set_error(QS_ERR_CUDA, "autotune: event synchronize failed");
            break;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        total += std::max((double)ms * (double)tiles / (double)tt, hbm_ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *out_ms = total;
    return rc;
}

static int ensure_fused_plan(Circuit& c, ITYPE dim, cudaStream_t st) {
    if (c.fplan && c.fplan->dim == dim) return QS_OK;
    const bool spec = want_specialized(c, dim);
    // the circuit gets a schedule once it can run: a failing candidate leaves none behind
    struct Candidate {
        std::vector<GateRec> gates;
        size_t count = 0;
        std::shared_ptr<StagedPlan> plan;
        int k = -1, tile_bits = kTileBits;
    };
    auto make = [&](int k, int tile_bits, Candidate* F) -> int {
        F->k = k;
        F->tile_bits = tile_bits;
        F->gates = executor_gates(c.gates, k, spec, &F->count);
        return build_plan(F->gates, c.n, dim, &F->plan, tile_bits, spec);
    };
    Candidate chosen;
    std::vector<double> ms;
    if (c.fusion_k >= 0) {
        QS_TRY(make(c.fusion_k, kTileBits, &chosen));
    } else {
        ms.assign(kTuneSlots, -1.);
        double best = 0.;
        auto consider = [&](int k, int tile_bits, int slot) -> int {
            Candidate F;
            QS_TRY(make(k, tile_bits, &F));
            QS_TRY(estimate_plan_ms(F.gates, *F.plan, dim, st, spec, &ms[slot]));
            if (!chosen.plan || ms[slot] < best) {
                best = ms[slot];
                chosen = std::move(F);
            }
            return QS_OK;
        };
        for (int k = 0; k <= kTuneMaxK; ++k) QS_TRY(consider(k, kTileBits, k));
        if (c.n > (UINT)kTileBits - 1) QS_TRY(consider(chosen.k, kTileBits - 1, kTuneMaxK + 1));
    }
    if (spec) QS_TRY(specialize_plan(*chosen.plan));
    c.tune_ms.swap(ms);
    c.fgates.swap(chosen.gates);
    c.fused_count = chosen.count;
    c.fused_k = chosen.k;
    c.fused_tile_bits = chosen.tile_bits;
    c.fplan = chosen.plan;
    return QS_OK;
}

int run_staged_fused(Circuit& c, void* state, ITYPE dim, cudaStream_t st) {
    if (c.n < kPhaseBits) {
        for (const GateRec& g : c.gates) QS_TRY(apply_gate_by_gate(g, state, dim, st));
        return QS_OK;
    }
    QS_TRY(ensure_fused_plan(c, dim, st));
    return run_plan(c.fgates, *c.fplan, state, dim, st);
}

// ---------------------------------------------------------------- complex64 states, FP64 passes
// The staged schedule over a complex64 state: each tile is widened to FP64 in shared memory, every
// phase runs in FP64 (the generic pass kernel's code), and the tile is rounded back on the store, so a
// pass moves half the bytes of the complex128 pass.  Gates are fused into blocks of at most 2 qubits
// (a forced QS_EXEC_STAGED_FUSED size of 0..2 is kept) so that every block is a pass op.  The same
// schedule (it does not depend on the state type) runs the large circuits of a batch.
static int c64_block_size(const Circuit& c) { return (c.fusion_k >= 0 && c.fusion_k <= 2) ? c.fusion_k : 2; }

static int ensure_c64_plan(Circuit& c, ITYPE dim) {
    const int k = c64_block_size(c);
    if (c.cplan && c.cplan->dim == dim && c.ck == k) return QS_OK;
    c.cgates = executor_gates(c.gates, k, false);
    c.ck = k;
    QS_TRY(build_plan(c.cgates, c.n, dim, &c.cplan));
    for (const DevPass& d : c.cplan->passes)
        if (d.single) {
            c.cplan.reset();
            return set_error(QS_ERR_NOT_SUPPORTED,
                "complex64 FP64 passes: every gate must be stageable (<= 2 targets and controls together)");
        }
    return QS_OK;
}

int run_staged_c64(Circuit& c, void* state, ITYPE dim, cudaStream_t st) {
    if (c.n < kPhaseBits) return set_error(QS_ERR_NOT_SUPPORTED, "complex64 FP64 passes need at least 4 qubits");
    QS_TRY(ensure_c64_plan(c, dim));
    QS_TRY(staged_allow_smem());
    for (const DevPass& d : c.cplan->passes) {
        launch_pass((float2*)state, d, dim >> d.args.m, st);
        QS_TRY(check_launch("k_staged_pass"));
    }
    return QS_OK;
}

int staged_pass_count(Circuit& c, ITYPE dim, UINT* out) {
    if (c.n < kPhaseBits) {
        *out = (UINT)c.gates.size();
        return QS_OK;
    }
    HostPlan H;
    std::vector<GateRec> g;
    staged_host_plan(c, dim, &g, &H);
    *out = (UINT)H.passes.size();
    return QS_OK;
}

}  // namespace qs

// Host-only statistics of the QS_EXEC_STAGED schedule that runs at 2^n amplitudes (the specialised kernels' or
// the generic one's): HBM passes, register phases, operations in phases, and gates run by the gate-by-gate
// kernels between passes.
extern "C" QS_API int qs_circuit_staged_stats(qs_circuit_t circuit, QS_UINT* passes, QS_UINT* phases, QS_UINT* ops,
    QS_UINT* single_gates) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c || !passes || !phases || !ops || !single_gates) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    if (c->n < (UINT)qs::kPhaseBits) {  // gate by gate
        *passes = *single_gates = (QS_UINT)c->gates.size();
        *phases = *ops = 0;
        return QS_OK;
    }
    qs::HostPlan H;
    std::vector<qs::GateRec> gates;
    qs::staged_host_plan(*c, 1ULL << c->n, &gates, &H);
    UINT single = 0;
    for (const qs::PassPlan& p : H.passes) single += p.single ? 1 : 0;
    *passes = (QS_UINT)H.passes.size();
    *phases = (QS_UINT)H.phases.size();
    *ops = (QS_UINT)H.ops.size();
    *single_gates = single;
    return QS_OK;
}

// Block size, gate count and HBM passes of the FP64-fused schedule last built for QS_EXEC_STAGED_FUSED
// (k = -1 before the first run), and the autotuner's estimates (ms; < 0 when not tried, e.g. with a
// forced k): estimates_ms[k] for k = 0..6 with 2^12-amplitude tiles, estimates_ms[7] for the best k
// with 2^11-amplitude tiles (the schedule uses those tiles when that estimate is the smallest).
extern "C" QS_API int qs_circuit_fusion_info(qs_circuit_t circuit, int* k, QS_UINT* gate_count, QS_UINT* passes,
    double* estimates_ms) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c || !k || !gate_count || !passes) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    *k = c->fplan ? c->fused_k : -1;
    *gate_count = c->fplan ? (QS_UINT)c->fused_count : 0;
    *passes = c->fplan ? (QS_UINT)c->fplan->passes.size() : 0;
    if (estimates_ms)
        for (int i = 0; i < qs::kTuneSlots; ++i)
            estimates_ms[i] = i < (int)c->tune_ms.size() ? c->tune_ms[i] : -1.;
    return QS_OK;
}

// Specialised pass kernels for this circuit's single-state staged modes: 1 = always, 0 = never (the
// generic pass kernel), -1 = for states of at least 2^22 amplitudes (default).
extern "C" QS_API int qs_circuit_set_specialized(qs_circuit_t circuit, int mode) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null circuit");
    if (mode < -1 || mode > 1) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "specialised mode must be -1, 0 or 1");
    c->specialize = mode;
    c->plan.reset();
    c->fplan.reset();
    c->fgates.clear();
    c->fused_k = -1;
    c->tune_ms.clear();
    return QS_OK;
}

// Whether the last-built QS_EXEC_STAGED and QS_EXEC_STAGED_FUSED schedules run specialised kernels, and
// the wall time their compilation took (ms, both schedules; 0 when served from the kernel cache).
extern "C" QS_API int qs_circuit_specialized_info(qs_circuit_t circuit, int* staged, int* staged_fused,
    double* compile_ms) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c || !staged || !staged_fused) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    *staged = c->plan && c->plan->specialized;
    *staged_fused = c->fplan && c->fplan->specialized;
    if (compile_ms)
        *compile_ms = (c->plan ? c->plan->compile_ms : 0.) + (c->fplan ? c->fplan->compile_ms : 0.);
    return QS_OK;
}

// CUDA C source of the specialised kernel of pass `pass` of the circuit's QS_EXEC_STAGED schedule at
// `dim` amplitudes (host only).  With buf == NULL, *size receives the length + 1; otherwise up to *size
// bytes are written, NUL-terminated.
extern "C" QS_API int qs_circuit_specialized_source(qs_circuit_t circuit, QS_ITYPE dim, QS_UINT pass, char* buf,
    QS_ITYPE* size) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c || !size) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    if (dim != (1ULL << c->n)) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "dim differs from 2^qubit_count");
    if (c->n < (UINT)qs::kPhaseBits + 3) return qs::set_error(QS_ERR_NOT_SUPPORTED, "fewer than 7 qubits");
    qs::HostPlan H;
    qs::make_host_plan(qs::rotation_form(c->gates, true), c->n, &H, qs::kTileBits, true);
    if (pass >= H.passes.size() || H.passes[pass].single)
        return qs::set_error(QS_ERR_INVALID_ARGUMENT, "no such staged pass");
    qs::StagedPlan P;
    P.phases = H.phases;
    P.programs = H.programs;
    qs::DevPass d{};
    d.args.m = (int)H.passes[pass].q.size();
    for (int j = 0; j < d.args.m; ++j) d.args.q[j] = H.passes[pass].q[j];
    d.args.nphases = (int)H.pp[pass].nphases;
    d.phase_begin = H.pp[pass].phase_begin;
    if (d.args.nphases) {
        auto high_bits = [&](const qs::StPhase& ph) {
            for (int p = 0; p < 4; ++p)
                if (ph.bits[p] < qs::kLowFixed) return false;
            return true;
        };
        if (high_bits(H.phases[d.phase_begin])) d.args.io |= 1;
        if (high_bits(H.phases[d.phase_begin + d.args.nphases - 1])) d.args.io |= 2;
    }
    const std::string src = qs::specialized_pass_source(qs::pass_desc(P, d));
    if (!buf) {
        *size = src.size() + 1;
        return QS_OK;
    }
    if (*size == 0) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "zero-size buffer");
    const size_t n = std::min<size_t>(src.size(), (size_t)*size - 1);
    memcpy(buf, src.data(), n);
    buf[n] = '\0';
    return QS_OK;
}

// Force the FP64 fusion block size of QS_EXEC_STAGED_FUSED (0..6; 0 = no fusion) or, with -1, let
// the autotuner choose on the next run.
extern "C" QS_API int qs_circuit_set_fusion(qs_circuit_t circuit, int k) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null circuit");
    if (k < -1 || k > 6) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "fusion block size must be -1..6");
    c->fusion_k = k;
    c->dm_vec.reset();
    c->fplan.reset();
    c->fgates.clear();
    c->fused_k = -1;
    c->tune_ms.clear();
    return QS_OK;
}

// ---------------------------------------------------------------- batched execution
// Many circuits (each on its own state, of any size >= 4 qubits) in ONE persistent launch.  Work
// items are (circuit, pass, tile); the queue lists every circuit's pass 0, then every circuit's
// pass 1, and so on.  A CTA takes the next item with an atomic counter and, for pass p > 0, waits
// until all tiles of pass p - 1 of the same circuit are done (acquire load of a per-pass counter).
// Dependencies only point to earlier queue items, which resident CTAs already hold, so the wait
// always ends; it is still bounded (a %globaltimer deadline, 2 s) and reports QS_ERR_TIMEOUT through an
// error flag, after which the CTA leaves without touching the item.
namespace qs {

struct BatchRec {
    StPassArgs args;
    void* state;  // complex128 or complex64 (one type per launch)
    ITYPE tiles;
    ITYPE prefix;  // first work item of this record
    int dep;       // record of the previous pass of the same circuit, -1 for pass 0
};


__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

template <class E, bool STEPS>
__global__ void __launch_bounds__(kBatchThreads, 3) k_batch_staged(const BatchRec* __restrict__ recs, int nrec,
    ITYPE total, unsigned long long* head, unsigned* done, int* err, unsigned long long wait_ns) {
    __shared__ double2 tile[1 << kBatchTileBits];
    __shared__ ITYPE hi_off[16];
    __shared__ ITYPE s_item;
    __shared__ int s_rec, s_abort;
    __shared__ StPassArgs s_args;  // the record's pass, copied so the tile code indexes shared memory
    __shared__ E* s_state;
    const int tid = threadIdx.x;
    while (true) {
        if (tid == 0) {
            s_abort = 0;
            s_item = atomicAdd(head, 1ULL);
            if (s_item < total) {
                int lo = 0, hi = nrec - 1;  // last record with prefix <= item
                while (lo < hi) {
                    const int mid = (lo + hi + 1) / 2;
                    if (recs[mid].prefix <= s_item) lo = mid;
                    else hi = mid - 1;
                }
                s_rec = lo;
                const int dep = recs[lo].dep;
                if (dep >= 0) {
                    const unsigned need = (unsigned)recs[dep].tiles;
                    const unsigned long long t0 = global_ns();
                    while (ld_acquire_u32(done + dep) < need) {
                        if (global_ns() - t0 > wait_ns) {
                            atomicExch(err, 1);
                            s_abort = 1;
                            break;
                        }
                        __nanosleep(64);
                    }
                }
            }
        }
        __syncthreads();
        if (s_item >= total || s_abort) break;
        if (tid == 0) {
            s_args = recs[s_rec].args;
            s_state = (E*)recs[s_rec].state;
        }
        __syncthreads();
        staged_tile<kBatchTileBits, STEPS>(s_state, s_args, s_item - recs[s_rec].prefix, tile, hi_off);
        if (tid == 0) {
            __threadfence();
            atomicAdd(done + s_rec, 1u);
        }
    }
}

// Block size of batched execution: the circuit's forced QS_EXEC_STAGED_FUSED size when it is at most 2,
// else 2 (autotuning each circuit of a batch would cost more than it saves; k <= 2 keeps every fused
// block a pass op).
static int batch_block_size(const Circuit& c) { return (c.fusion_k >= 0 && c.fusion_k <= 2) ? c.fusion_k : 2; }

static int ensure_batch_plan(Circuit& c, ITYPE dim) {
    const int k = batch_block_size(c);
    if (c.bplan && c.bplan->dim == dim && c.bk == k) return QS_OK;
    c.bgates = executor_gates(c.gates, k, false);
    c.bk = k;
    return build_plan(c.bgates, c.n, dim, &c.bplan, kBatchTileBits);
}

// `wait_ns`: the dependency wait limit; `self_dep` >= 0 makes that work record depend on itself (a
// counter nothing can complete), which only the wait-expiry check below uses.
// The work records of a batch (plans missing from the circuits' caches built first: FP64 fusion and
// host planning on host threads in parallel, uploads afterwards), the number of work items, and whether any
// of their phases is a list of steps.
static int batch_records(Circuit* const* cs, void* const* states, UINT count, std::vector<BatchRec>* recs,
    ITYPE* total_out, bool* steps) {
    for (UINT i = 0; i < count; ++i)
        if (cs[i]->n < kPhaseBits) return set_error(QS_ERR_NOT_SUPPORTED, "batch: circuits need at least 4 qubits");
    {
        std::vector<char> need(count, 0);
        for (UINT i = 0; i < count; ++i) {
            const Circuit& c = *cs[i];
            need[i] = !(c.bplan && c.bplan->dim == (1ULL << c.n) && c.bk == batch_block_size(c));
            for (UINT j = 0; j < i && need[i]; ++j)
                if (cs[j] == cs[i]) need[i] = 0;
        }
        std::vector<std::vector<GateRec>> fg(count);
        std::vector<HostPlan> hp(count);
        std::atomic<UINT> next{0};
        const unsigned nt = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
        std::vector<std::thread> pool;
        for (unsigned t = 0; t < nt; ++t)
            pool.emplace_back([&] {
                for (UINT i; (i = next.fetch_add(1)) < count;)
                    if (need[i]) {
                        fg[i] = executor_gates(cs[i]->gates, batch_block_size(*cs[i]), false);
                        make_host_plan(fg[i], cs[i]->n, &hp[i], kBatchTileBits);
                    }
            });
        for (std::thread& t : pool) t.join();
        for (UINT i = 0; i < count; ++i)
            if (need[i]) {
                Circuit& c = *cs[i];
                c.bgates = std::move(fg[i]);
                c.bk = batch_block_size(c);
                QS_TRY(upload_plan(hp[i], 1ULL << c.n, &c.bplan));
            }
    }
    std::vector<std::vector<const DevPass*>> passes(count);
    size_t maxp = 0;
    for (UINT i = 0; i < count; ++i) {
        Circuit& c = *cs[i];
        QS_TRY(ensure_batch_plan(c, 1ULL << c.n));
        for (const DevPass& d : c.bplan->passes) {
            if (d.single)
                return set_error(QS_ERR_NOT_SUPPORTED,
                    "batch: every gate must be stageable (<= 2 targets, no controls, no Pauli strings)");
            passes[i].push_back(&d);
        }
        maxp = std::max(maxp, passes[i].size());
    }
    recs->clear();
    std::vector<int> last(count, -1);
    ITYPE total = 0;
    for (size_t p = 0; p < maxp; ++p)
        for (UINT i = 0; i < count; ++i) {
            if (p >= passes[i].size()) continue;
            BatchRec r{};
            r.args = passes[i][p]->args;
            r.state = states[i];
            r.tiles = (1ULL << cs[i]->n) >> r.args.m;
            r.prefix = total;
            r.dep = last[i];
            last[i] = (int)recs->size();
            total += r.tiles;
            *steps = *steps || passes[i][p]->steps;
            recs->push_back(r);
        }
    *total_out = total;
    return QS_OK;
}

// Device buffer of a batch launch: records | per-record done counters | (16-byte aligned) work head |
// error flag.  Everything after the records must be zero before a launch.
struct BatchLayout {
    size_t brec, zero_bytes, bytes;
    explicit BatchLayout(size_t nrec) {
        brec = sizeof(BatchRec) * nrec;
        const size_t bdone = sizeof(unsigned) * nrec;
        bytes = brec + bdone + 256;
        zero_bytes = bytes - brec;
    }
    unsigned* done(void* b) const { return (unsigned*)((char*)b + brec); }
    unsigned long long* head(void* b) const {
        return (unsigned long long*)((char*)b + ((brec + (bytes - 256 - brec) + 15) / 16 * 16));
    }
    int* err(void* b) const { return (int*)(head(b) + 1); }
};

static int batch_kernel(void* buf, const BatchLayout& L, int nrec, ITYPE total, bool steps, unsigned long long wait_ns,
    bool c64, cudaStream_t st) {
    auto kernel = c64 ? (steps ? (const void*)k_batch_staged<float2, true> : (const void*)k_batch_staged<float2, false>)
                      : (steps ? (const void*)k_batch_staged<double2, true> : (const void*)k_batch_staged<double2, false>);
    int per_sm = 0;
    QS_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBatchThreads, 0));
    const ITYPE resident = (ITYPE)std::max(1, per_sm) * sm_count();
    const unsigned grid = (unsigned)std::min<ITYPE>(resident, total);
    const BatchRec* drec = (const BatchRec*)buf;
    unsigned long long* head = L.head(buf);
    unsigned* done = L.done(buf);
    int* err = L.err(buf);
    void* args[] = {&drec, &nrec, &total, &head, &done, &err, &wait_ns};
    QS_CUDA_CHECK(cudaLaunchKernel(kernel, dim3(grid), dim3(kBatchThreads), args, 0, st));
    return check_launch("k_batch_staged");
}

// Circuits of at least this many qubits leave the persistent launch: a pass of theirs has >= 1024
// tiles of 2^11 amplitudes, enough to fill the device alone, so they run as their own staged passes
// with 2^12-amplitude tiles (fewer passes, no dependency waits), on the same stream.
constexpr UINT kBatchSoloQubits = 21;

int batch_update(Circuit* const* cs, void* const* states, UINT count, cudaStream_t st, unsigned long long wait_ns,
    int self_dep, bool c64) {
    if (count == 0) return QS_OK;
    std::vector<Circuit*> shared_cs, solo_cs;
    std::vector<void*> shared_st, solo_st;
    for (UINT i = 0; i < count; ++i) {
        const bool solo = self_dep < 0 && cs[i]->n >= kBatchSoloQubits;
        (solo ? solo_cs : shared_cs).push_back(cs[i]);
        (solo ? solo_st : shared_st).push_back(states[i]);
    }
    // every plan first (a refusal comes before any launch)
    for (size_t i = 0; i < solo_cs.size(); ++i) QS_TRY(ensure_c64_plan(*solo_cs[i], 1ULL << solo_cs[i]->n));
    std::vector<BatchRec> recs;
    ITYPE total = 0;
    bool steps = false;
    if (!shared_cs.empty())
        QS_TRY(batch_records(shared_cs.data(), shared_st.data(), (UINT)shared_cs.size(), &recs, &total, &steps));
    if (!solo_cs.empty()) QS_TRY(staged_allow_smem());
    for (size_t i = 0; i < solo_cs.size(); ++i) {
        const ITYPE dim = 1ULL << solo_cs[i]->n;
        for (const DevPass& d : solo_cs[i]->cplan->passes) {
            if (c64) launch_pass((float2*)solo_st[i], d, dim >> d.args.m, st);
            else launch_pass((double2*)solo_st[i], d, dim >> d.args.m, st);
            QS_TRY(check_launch("k_staged_pass"));
        }
    }
    if (recs.empty()) {
        QS_CUDA_CHECK(cudaStreamSynchronize(st));
        return QS_OK;
    }
    if (self_dep >= 0) {
        if (self_dep >= (int)recs.size()) return set_error(QS_ERR_INVALID_ARGUMENT, "batch: no such work record");
        recs[self_dep].dep = self_dep;
    }
    const BatchLayout L(recs.size());
    void* buf = nullptr;
    QS_TRY(scratch(st, L.bytes, &buf));
    QS_CUDA_CHECK(cudaMemcpyAsync(buf, recs.data(), L.brec, cudaMemcpyHostToDevice, st));
    QS_CUDA_CHECK(cudaMemsetAsync(L.done(buf), 0, L.zero_bytes, st));
    QS_TRY(batch_kernel(buf, L, (int)recs.size(), total, steps, wait_ns, c64, st));
    int err = 0;
    QS_CUDA_CHECK(cudaMemcpyAsync(&err, L.err(buf), sizeof(int), cudaMemcpyDeviceToHost, st));
    QS_CUDA_CHECK(cudaStreamSynchronize(st));
    if (err) return set_error(QS_ERR_TIMEOUT, "batch: dependency wait expired");
    return QS_OK;
}

// ---------------------------------------------------------------- captured CUDA graphs
// A circuit (or a batch) applied to fixed device states, recorded once as a CUDA graph and replayed
// with one cudaGraphLaunch: the host planning, parameter uploads and per-pass launches of a call are
// paid once.  Plans (and the autotuner, and specialised kernels) are prepared before the capture;
// the capture records only stream work.  Work that copies from pageable host memory during a run (a
// dense gate of >= 6 qubits left outside the staged passes, a multi-qubit diagonal) refuses to be
// recorded: creation then fails with QS_ERR_NOT_SUPPORTED.
struct GraphExec {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    void* dev = nullptr;       // batch graphs: work records and counters
    int* host_err = nullptr;   // batch graphs: the wait-expiry flag, copied back by the graph (pinned)
    long long kernels = 0;     // kernel launches one replay performs
    ~GraphExec() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (dev) cudaFree(dev);
        if (host_err) cudaFreeHost(host_err);
    }
};

// Records `work` on a capturing stream (the caller's, or a private one for the legacy default stream)
// into G.  Capture is thread-local, so other threads' unrelated CUDA calls are not affected.
template <class F>
static int capture_graph(cudaStream_t user, GraphExec* G, F work) {
    cudaStream_t st = user;
    cudaStream_t own = nullptr;
    if (!st) {  // the legacy default stream cannot capture
        QS_TRY(qs_stream_create((void**)&own));
        st = own;
    }
    const unsigned long long l0 = qs_launch_count();
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        if (own) qs_stream_destroy(own);
        return check_cuda(e, "cudaStreamBeginCapture");
    }
    set_capturing(true);
    int rc = work(st);
    set_capturing(false);
    std::string msg = rc == QS_OK ? std::string() : std::string(qs_get_last_error());
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(st, &g);
    G->kernels = (long long)(qs_launch_count() - l0);
    count_launches(-G->kernels);  // recorded, not run
    if (own) qs_stream_destroy(own);  // with any scratch the capture allocated for it
    if (rc != QS_OK || e != cudaSuccess || !g) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();  // clear the capture error
        return set_error(QS_ERR_NOT_SUPPORTED,
            "graph capture: this work cannot be recorded (" + (msg.empty() ? std::string(cudaGetErrorString(e)) : msg) +
            ")");
    }
    G->graph = g;
    e = cudaGraphInstantiate(&G->exec, g, 0);
    if (e != cudaSuccess) return check_cuda(e, "cudaGraphInstantiate");
    return QS_OK;
}

}  // namespace qs

extern "C" QS_API int qs_circuit_graph_create(qs_circuit_t circuit, void* state, QS_ITYPE dim, int mode, int reset_state,
    void* stream, qs_graph_t* out) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c || !state || !out) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    if (dim != (1ULL << c->n)) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "dim differs from 2^qubit_count");
    if (mode != QS_EXEC_GATE_BY_GATE && mode != QS_EXEC_STAGED && mode != QS_EXEC_STAGED_FUSED)
        return qs::set_error(QS_ERR_INVALID_ARGUMENT, "unknown execution mode");
    cudaStream_t st = (cudaStream_t)stream;
    // plans, autotuning and specialised kernels first: they synchronise and allocate
    if (c->n >= (UINT)qs::kPhaseBits) {
        if (mode == QS_EXEC_STAGED) QS_TRY(qs::ensure_plan(*c, dim));
        if (mode == QS_EXEC_STAGED_FUSED) QS_TRY(qs::ensure_fused_plan(*c, dim, st));
    }
    QS_TRY(qs::staged_allow_smem());
    auto G = std::make_unique<qs::GraphExec>();
    QS_TRY(qs::capture_graph(st, G.get(), [&](cudaStream_t cs) -> int {
        if (reset_state) QS_TRY(qs_initialize_quantum_state(state, dim, cs));
        if (mode == QS_EXEC_STAGED) return qs::run_staged(*c, state, dim, cs);
        if (mode == QS_EXEC_STAGED_FUSED) return qs::run_staged_fused(*c, state, dim, cs);
        for (const qs::GateRec& g : c->gates) QS_TRY(qs::apply_gate_by_gate(g, state, dim, cs));
        return QS_OK;
    }));
    *out = reinterpret_cast<qs_graph_t>(G.release());
    return QS_OK;
}

extern "C" QS_API int qs_batch_graph_create(const qs_circuit_t* circuits, void* const* states, QS_UINT count, int c64,
    int reset_states, void* stream, qs_graph_t* out) {
    if (!circuits || !states || !out || count == 0) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    std::vector<qs::Circuit*> cs(count);
    for (QS_UINT i = 0; i < count; ++i) {
        cs[i] = reinterpret_cast<qs::Circuit*>(circuits[i]);
        if (!cs[i] || !states[i]) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null circuit or state");
    }
    std::vector<qs::BatchRec> recs;
    ITYPE total = 0;
    bool steps = false;
    QS_TRY(qs::batch_records(cs.data(), states, count, &recs, &total, &steps));
    if (recs.empty()) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "batch graph: no passes to run");
    auto G = std::make_unique<qs::GraphExec>();
    const qs::BatchLayout L(recs.size());
    QS_CUDA_CHECK(cudaMalloc(&G->dev, L.bytes));
    QS_CUDA_CHECK(cudaMemcpy(G->dev, recs.data(), L.brec, cudaMemcpyHostToDevice));
    QS_CUDA_CHECK(cudaMallocHost((void**)&G->host_err, sizeof(int)));
    *G->host_err = 0;
    void* dev = G->dev;
    int* host_err = G->host_err;
    QS_TRY(qs::capture_graph((cudaStream_t)stream, G.get(), [&](cudaStream_t st) -> int {
        if (reset_states)
            for (QS_UINT i = 0; i < count; ++i) {
                const QS_ITYPE dim = 1ULL << cs[i]->n;
                QS_TRY(c64 ? qs_initialize_quantum_state_c64(states[i], dim, st)
                           : qs_initialize_quantum_state(states[i], dim, st));
            }
        QS_CUDA_CHECK(cudaMemsetAsync(L.done(dev), 0, L.zero_bytes, st));
        QS_TRY(qs::batch_kernel(dev, L, (int)recs.size(), total, steps, qs::kBatchWaitNs, c64 != 0, st));
        QS_CUDA_CHECK(cudaMemcpyAsync(host_err, L.err(dev), sizeof(int), cudaMemcpyDeviceToHost, st));
        return QS_OK;
    }));
    *out = reinterpret_cast<qs_graph_t>(G.release());
    return QS_OK;
}

extern "C" QS_API int qs_graph_launch(qs_graph_t graph, void* stream) {
    qs::GraphExec* G = reinterpret_cast<qs::GraphExec*>(graph);
    if (!G || !G->exec) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null graph");
    cudaStream_t st = (cudaStream_t)stream;
    QS_CUDA_CHECK(cudaGraphLaunch(G->exec, st));
    qs::count_launches(G->kernels);
    if (G->host_err) {  // a batch graph: its wait-expiry flag arrives with the graph's last node
        QS_CUDA_CHECK(cudaStreamSynchronize(st));
        if (*G->host_err) return qs::set_error(QS_ERR_TIMEOUT, "batch graph: dependency wait expired");
    }
    return QS_OK;
}

extern "C" QS_API int qs_graph_kernel_count(qs_graph_t graph, QS_ITYPE* kernels) {
    qs::GraphExec* G = reinterpret_cast<qs::GraphExec*>(graph);
    if (!G || !kernels) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    *kernels = (QS_ITYPE)G->kernels;
    return QS_OK;
}

extern "C" QS_API int qs_graph_destroy(qs_graph_t graph) {
    delete reinterpret_cast<qs::GraphExec*>(graph);
    return QS_OK;
}

namespace qs {
}  // namespace qs

extern "C" QS_API int qs_batch_update_quantum_states(const qs_circuit_t* circuits, void* const* states, QS_UINT count,
    void* stream) {
    if (!circuits || !states) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null argument");
    std::vector<qs::Circuit*> cs(count);
    for (QS_UINT i = 0; i < count; ++i) {
        cs[i] = reinterpret_cast<qs::Circuit*>(circuits[i]);
        if (!cs[i] || !states[i]) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null circuit or state");
    }
    return qs::batch_update(cs.data(), states, count, (cudaStream_t)stream, qs::kBatchWaitNs, -1, false);
}

// Failure-path check of the batch executor's bounded dependency wait: runs `circuit` on `state` as a
// one-circuit batch whose last pass waits on its own completion counter, which never completes, with
// a wait limit of `wait_limit_us`.  Every CTA that takes a tile of that pass gives up after the limit,
// sets the error flag and leaves, so the call returns QS_ERR_TIMEOUT and the context stays usable; the
// state is left with all passes but the last applied.
extern "C" QS_API int qs_debug_batch_wait_expiry(qs_circuit_t circuit, void* state, QS_UINT wait_limit_us,
    void* stream) {
    qs::Circuit* c = reinterpret_cast<qs::Circuit*>(circuit);
    if (!c || !state) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "null circuit or state");
    if (wait_limit_us == 0 || wait_limit_us > 2000000u)
        return qs::set_error(QS_ERR_INVALID_ARGUMENT, "wait limit must be 1 us .. 2 s");
    qs::Circuit* cs[1] = {c};
    void* ss[1] = {state};
    // the last record of a one-circuit batch is its last pass
    UINT passes = 0;
    {
        qs::HostPlan H;
        std::vector<qs::GateRec> fg = qs::executor_gates(c->gates, qs::batch_block_size(*c), false);
        qs::make_host_plan(fg, c->n, &H, qs::kBatchTileBits);
        passes = (UINT)H.passes.size();
    }
    if (passes == 0) return qs::set_error(QS_ERR_INVALID_ARGUMENT, "circuit has no passes");
    return qs::batch_update(cs, ss, 1, (cudaStream_t)stream, 1000ULL * wait_limit_us, (int)passes - 1, false);
}

