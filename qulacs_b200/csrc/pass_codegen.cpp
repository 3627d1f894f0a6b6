// Specialised staged-pass kernels: one kernel per pass, generated as CUDA C from the pass's schedule and
// compiled for sm_100a with NVRTC at plan time.
//
// The generic pass kernel (k_staged_pass, staged.cu) reads each phase's program from memory: rounds in which a
// rotation or factor that is not there costs as much as one that is, or, with matrices and channels, steps
// behind a switch that returns the 16 amplitudes to fixed registers.  Here every tile qubit, phase bit, address
// offset and register index is a compile-time constant: a phase is the straight-line code of its program
// (phase_program.hpp), and gate parameters are constant-bank operands.
//
// What bounds it: a pass needs one read and one write of the state, 16 bytes through shared memory each
// way per amplitude and inner phase, and the program's FP64 instructions.  The layered circuit at 30 qubits
// (16 passes, 77 phases, 1296 FP64 instructions per amplitude) has 84 ms of HBM, ~60 ms of shared memory
// and 75 ms of FP64 time and runs in 139 ms; with one matrix per gate (2400 instructions) it took 212 ms.
//  * One 16-amplitude coset per thread, so 256 threads and 2 CTAs per SM for a 2^12-amplitude tile
//    (128 registers): 141 ms, against 159 ms for 128 threads with two cosets each and 3 CTAs per SM
//    (12 warps, and the coset loop turned parameters into separate constant loads).
//  * Lanes run over tile bits whose swizzle vectors are independent (lane_order): the density-matrix
//    circuit of 12 qubits went from 3.6 to 3.1 ms.
//  * Plain loads and stores: with streaming hints (.cs) the layered circuit took 141 ms, without them 137.
//
// NVRTC is opened at run time (libnvrtc.so.12); the compiled cubin is loaded with cudaLibraryLoadData,
// which makes it available to every device context.  Kernels are cached by source text for the life of
// the process.
#include <dlfcn.h>

#include <chrono>
#include <cinttypes>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <sstream>
#include <string>
#include <vector>

#include "../../include/qulacs_b200.h"
#include "codegen.hpp"
#include "phase_program.hpp"
#include "staged.hpp"

namespace qs {

int set_error(int code, const std::string& msg);
int check_cuda(cudaError_t e, const char* what);
int check_launch(const char* kernel);

namespace {

// ---------------------------------------------------------------- NVRTC, opened at run time
typedef int nvrtcResult_t;
typedef struct _nvrtcProgram* nvrtcProgram_t;
struct Nvrtc {
    void* h = nullptr;
    nvrtcResult_t (*create)(nvrtcProgram_t*, const char*, const char*, int, const char* const*, const char* const*) =
        nullptr;
    nvrtcResult_t (*compile)(nvrtcProgram_t, int, const char* const*) = nullptr;
    nvrtcResult_t (*cubin_size)(nvrtcProgram_t, size_t*) = nullptr;
    nvrtcResult_t (*cubin)(nvrtcProgram_t, char*) = nullptr;
    nvrtcResult_t (*log_size)(nvrtcProgram_t, size_t*) = nullptr;
    nvrtcResult_t (*log)(nvrtcProgram_t, char*) = nullptr;
    nvrtcResult_t (*destroy)(nvrtcProgram_t*) = nullptr;
    std::string error;
};

Nvrtc* nvrtc() {
    static Nvrtc N;
    static std::once_flag once;
    std::call_once(once, [] {
        std::vector<std::string> names;
        for (const char* env : {"CUDA_HOME", "CUDA_PATH"})
            if (const char* p = std::getenv(env)) names.push_back(std::string(p) + "/lib64/libnvrtc.so.12");
        names.push_back("libnvrtc.so.12");
        names.push_back("libnvrtc.so");
        for (const std::string& nm : names) {
            N.h = dlopen(nm.c_str(), RTLD_NOW | RTLD_LOCAL);
            if (N.h) break;
        }
        if (!N.h) {
            N.error = "NVRTC (libnvrtc.so.12) not found";
            return;
        }
        auto sym = [&](const char* s) { return dlsym(N.h, s); };
        N.create = (decltype(N.create))sym("nvrtcCreateProgram");
        N.compile = (decltype(N.compile))sym("nvrtcCompileProgram");
        N.cubin_size = (decltype(N.cubin_size))sym("nvrtcGetCUBINSize");
        N.cubin = (decltype(N.cubin))sym("nvrtcGetCUBIN");
        N.log_size = (decltype(N.log_size))sym("nvrtcGetProgramLogSize");
        N.log = (decltype(N.log))sym("nvrtcGetProgramLog");
        N.destroy = (decltype(N.destroy))sym("nvrtcDestroyProgram");
        if (!N.create || !N.compile || !N.cubin_size || !N.cubin || !N.log_size || !N.log || !N.destroy) {
            N.error = "NVRTC lacks the CUBIN entry points";
            N.h = nullptr;
        }
    });
    return &N;
}

// ---------------------------------------------------------------- kernel source
// The device helpers every generated kernel shares.  The register ops mirror staged.cu's r_* ops, with
// the matrix entries passed by value so that literal arguments become constants.
const char* kPrelude = R"(
typedef unsigned long long u64;
struct __align__(16) D2 { double x, y; };
__device__ __forceinline__ D2 mk(double x, double y) { D2 v; v.x = x; v.y = y; return v; }
__device__ __forceinline__ D2 cmul(D2 a, D2 b) { return mk(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)); }
__device__ __forceinline__ D2 cfma(D2 a, D2 b, D2 acc) {
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
    return acc;
}
__device__ __forceinline__ D2 ldg(const D2* p) {
    D2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void stg(D2* p, D2 v) {
    asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
// A parameter read at its use (volatile: not hoisted out of the coset loop, where every parameter of
// the pass would stay live in registers).
__device__ __forceinline__ D2 ldp(const D2* p) {
    D2 v;
    asm volatile("ld.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned swz(unsigned u) { return u ^ (((u >> 3) ^ (u >> 5) ^ (u >> 6) ^ (u >> 8)) & 7u); }
__device__ __forceinline__ u64 ins0(u64 i, unsigned q) { return ((i >> q) << (q + 1)) | (i & ((1ULL << q) - 1ULL)); }

// Register steps (phase_program.hpp).  A pair (x, y): the amplitudes where the step's qubit is 0 and 1.
__device__ __forceinline__ void ry_tan(D2& x, D2& y, double t) {
    const D2 X = x;
    x = mk(fma(t, y.x, X.x), fma(t, y.y, X.y));
    y = mk(fma(-t, X.x, y.x), fma(-t, X.y, y.y));
}
__device__ __forceinline__ void ry_cot(D2& x, D2& y, double u) {
    const D2 X = x;
    x = mk(fma(u, X.x, y.x), fma(u, X.y, y.y));
    y = mk(fma(u, y.x, -X.x), fma(u, y.y, -X.y));
}
__device__ __forceinline__ void ry_full(D2& x, D2& y, double c, double s) {
    const D2 X = x;
    x = mk(fma(c, X.x, s * y.x), fma(c, X.y, s * y.y));
    y = mk(fma(c, y.x, -s * X.x), fma(c, y.y, -s * X.y));
}
__device__ __forceinline__ void rx_tan(D2& x, D2& y, double t) {
    const D2 X = x;
    x = mk(fma(-t, y.y, X.x), fma(t, y.x, X.y));
    y = mk(fma(-t, X.y, y.x), fma(t, X.x, y.y));
}
__device__ __forceinline__ void rx_cot(D2& x, D2& y, double u) {
    const D2 X = x;
    x = mk(fma(u, X.x, -y.y), fma(u, X.y, y.x));
    y = mk(fma(u, y.x, -X.y), fma(u, y.y, X.x));
}
__device__ __forceinline__ void rx_full(D2& x, D2& y, double c, double s) {
    const D2 X = x;
    x = mk(fma(c, X.x, -s * y.y), fma(c, X.y, s * y.x));
    y = mk(fma(c, y.x, -s * X.y), fma(c, y.y, s * X.x));
}
__device__ __forceinline__ void dense1(D2& x, D2& y, D2 m0, D2 m1, D2 m2, D2 m3) {
    const D2 X = x;
    x = cfma(m1, y, cmul(m0, X));
    y = cfma(m3, y, cmul(m2, X));
}
// One row of a 4 x 4 matrix; the entries are read at their use (volatile), so one row's are live at a time.
__device__ __forceinline__ D2 row4(const D2* p, D2 a, D2 b, D2 c, D2 d) {
    return cfma(ldp(p + 3), d, cfma(ldp(p + 2), c, cfma(ldp(p + 1), b, cmul(ldp(p), a))));
}
__device__ __forceinline__ void dense2(D2& a, D2& b, D2& c, D2& d, const D2* p) {
    const D2 A = row4(p, a, b, c, d), B = row4(p + 4, a, b, c, d), C = row4(p + 8, a, b, c, d);
    d = row4(p + 12, a, b, c, d);
    a = A; b = B; c = C;
}
// Populations (x, y) of a one-qubit depolarizing channel mix.
__device__ __forceinline__ void mix2(D2& x, D2& y, double t) {
    const D2 X = x;
    x = mk(fma(t, y.x, X.x), fma(t, y.y, X.y));
    y = mk(fma(t, X.x, y.x), fma(t, X.y, y.y));
}
__device__ __forceinline__ void rscale(D2& x, double k) { x = mk(k * x.x, k * x.y); }
__device__ __forceinline__ D2 sum4(D2 a, D2 b, D2 c, D2 d) { return mk((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y)); }
__device__ __forceinline__ void axpy(D2& x, double t, D2 s) { x = mk(fma(t, s.x, x.x), fma(t, s.y, x.y)); }
)";

// An exact C++17 hexadecimal literal of a double.
std::string lit(double v) {
    char buf[64];
    std::snprintf(buf, sizeof(buf), "%a", v);
    return buf;
}
// Gate parameters of a generated kernel: written into the source as literals, or (when `bank` is set)
// referenced as P.v[i] of the kernel's __grid_constant__ parameter block and collected into `bank`, so
// the kernel depends only on the pass's structure and is shared by circuits that differ in angles.  A
// reference is a constant-bank operand of the instruction that uses it.
struct ParamSink {
    std::vector<double2>* bank = nullptr;
    long half = -1;  // entry whose second double is free
    std::string d2(const double2& v) {
        if (!bank) return "mk(" + lit(v.x) + ", " + lit(v.y) + ")";
        bank->push_back(v);
        return "P.v[z + " + std::to_string(bank->size() - 1) + "]";
    }
    std::string d1(double v) {
        if (!bank) return lit(v);
        if (half >= 0) {
            (*bank)[half].y = v;
            const std::string r = "P.v[z + " + std::to_string(half) + "].y";
            half = -1;
            return r;
        }
        half = (long)bank->size();
        bank->push_back(make_double2(v, 0.));
        return "P.v[z + " + std::to_string(half) + "].x";
    }
};

std::string u64hex(ITYPE v) {
    char buf[40];
    std::snprintf(buf, sizeof(buf), "0x%llxULL", (unsigned long long)v);
    return buf;
}

int gray_bit(int g) { return (g & 1) ? 0 : (g & 2) ? 1 : (g & 4) ? 2 : 3; }

unsigned swz_host(unsigned u) { return QS_SWZ(u); }

// One step of a phase program on the registers r0..r15.
void emit_step(std::ostringstream& o, const ProgStep& s, ParamSink& ps) {
    auto reg = [](int j) { return "r[" + std::to_string(j) + "]"; };
    // registers by the values of the step's qubits: at(k) for base register b, k = packed qubit values
    auto coset = [&](int b, int k) {
        int j = b;
        for (int i = 0; i < s.nq; ++i)
            if (((k >> i) & 1) != step_bit(s, i, j)) j ^= s.v[i];
        return j;
    };
    auto bases = [&]() {  // one register of each coset of the step's qubits: all its qubits 0
        std::vector<int> out;
        for (int j = 0; j < 16; ++j) {
            bool zero = true;
            for (int i = 0; i < s.nq; ++i) zero = zero && !step_bit(s, i, j);
            if (zero) out.push_back(j);
        }
        return out;
    };
    switch (s.kind) {
        case SP_DIAG:
            for (int j = 0; j < 16; ++j)
                if ((s.mask >> j) & 1) o << "      " << reg(j) << " = cmul(" << ps.d2(s.par[j]) << ", " << reg(j) << ");\n";
            break;
        case SP_SIGN:
            for (int j = 0; j < 16; ++j)
                if ((s.mask >> j) & 1) o << "      " << reg(j) << " = mk(-" << reg(j) << ".x, -" << reg(j) << ".y);\n";
            break;
        case SP_CNOT:
        case SP_SWAP:
        case SP_X:  // moves between registers: names, once the compiler has unrolled them
            for (int j = 0; j < 16; ++j) {
                const int b0 = step_bit(s, 0, j), b1 = s.nq > 1 ? step_bit(s, 1, j) : 0;
                const bool first = s.kind == SP_CNOT ? b0 && !b1 : s.kind == SP_SWAP ? b0 && !b1 : !b0;
                const int k = s.kind == SP_CNOT ? j ^ s.v[1] : s.kind == SP_SWAP ? j ^ s.v[0] ^ s.v[1] : j ^ s.v[0];
                if (first) o << "      { const D2 t = " << reg(j) << "; " << reg(j) << " = " << reg(k) << "; " << reg(k) << " = t; }\n";
            }
            break;
        case SP_SCALE: {
            const std::string z = s.form ? ps.d2(s.par[0]) : ps.d1(s.par[0].x);
            for (int j = 0; j < 16; ++j) {
                if (s.form) o << "      " << reg(j) << " = cmul(" << z << ", " << reg(j) << ");\n";
                else o << "      rscale(" << reg(j) << ", " << z << ");\n";
            }
            break;
        }
        case SP_ROT: {
            static const char* names[] = {"ry_tan", "ry_cot", "ry_full", "rx_tan", "rx_cot", "rx_full"};
            const bool full = s.form == RF_Y_FULL || s.form == RF_X_FULL;
            std::string args = ps.d1(s.par[0].x);
            if (full) args += ", " + ps.d1(s.par[0].y);
            for (int j : bases())
                o << "      " << names[s.form] << "(" << reg(j) << ", " << reg(coset(j, 1)) << ", " << args << ");\n";
            break;
        }
        case SP_DENSE1: {
            std::string args;
            for (int i = 0; i < 4; ++i) args += ", " + ps.d2(s.par[i]);
            for (int j : bases()) o << "      dense1(" << reg(j) << ", " << reg(coset(j, 1)) << args << ");\n";
            break;
        }
        case SP_DENSE2: {
            std::string m;
            if (ps.bank) {  // one run of the parameter block
                m = "&P.v[" + std::to_string(ps.bank->size()) + "]";
                for (int i = 0; i < 16; ++i) ps.bank->push_back(s.par[i]);
            } else {
                o << "      { const D2 m[16] = {";
                for (int i = 0; i < 16; ++i) o << (i ? ", " : "") << ps.d2(s.par[i]);
                o << "};\n";
                m = "m";
            }
            for (int j : bases())
                o << "      dense2(" << reg(j) << ", " << reg(coset(j, 1)) << ", " << reg(coset(j, 2)) << ", "
                  << reg(coset(j, 3)) << ", " << m << ");\n";
            if (!ps.bank) o << "      }\n";
            break;
        }
        case SP_DEPOL1: {  // qubits: column, row
            const std::string t = ps.d1(s.par[0].x), k = ps.d1(s.par[0].y), d = s.form ? ps.d1(s.par[1].x) : std::string();
            for (int j : bases()) {
                if (s.form) o << "      rscale(" << reg(j) << ", " << d << "); rscale(" << reg(coset(j, 3)) << ", " << d << ");\n";
                o << "      mix2(" << reg(j) << ", " << reg(coset(j, 3)) << ", " << t << "); rscale(" << reg(coset(j, 1))
                  << ", " << k << "); rscale(" << reg(coset(j, 2)) << ", " << k << ");\n";
            }
            break;
        }
        case SP_DEPOL2: {  // qubits: columns 0, 1, rows 0, 1; populations: equal column and row
            const int b = bases()[0];
            const std::string t = ps.d1(s.par[0].x), k = s.form ? ps.d1(s.par[0].y) : std::string();
            const int pop[4] = {coset(b, 0), coset(b, 5), coset(b, 10), coset(b, 15)};
            o << "      { const D2 S = sum4(" << reg(pop[0]) << ", " << reg(pop[1]) << ", " << reg(pop[2]) << ", "
              << reg(pop[3]) << ");\n";
            if (s.form)
                for (int j = 0; j < 16; ++j) o << "      rscale(" << reg(j) << ", " << k << ");\n";
            for (int j : pop) o << "      axpy(" << reg(j) << ", " << t << ", S);\n";
            o << "      }\n";
            break;
        }
    }
}

// Largest parameter block passed to a kernel (the kernel-parameter space is 32764 bytes; the state
// pointer is in it too); a pass with more parameters gets them as literals instead.
constexpr size_t kMaxParamBytes = 32000;

// One coset per thread (up to 256 threads); two where a pass holds a two-qubit matrix, whose 16 products
// per output do not fit beside the coset in 128 registers (184 bytes of spill).
int spec_threads(const PassDesc& d) {
    for (int ph = 0; ph < d.nphases; ++ph)
        for (const ProgStep& s : d.programs[ph].steps)
            if (s.kind == SP_DENSE2) return 128;
    return d.m >= 12 ? 256 : 128;
}

// CUDA C of one pass; mirrors staged_tile (staged.cu) with every schedule quantity a constant.  With
// `params`, gate parameters come from the kernel's parameter block (their values appended to *params);
// without, they are literals.
std::string pass_source(const PassDesc& d, std::vector<double2>* params) {
    const int m = d.m;
    const unsigned tsize = 1u << m, ncos = tsize >> kPhaseBits;
    const bool hbm_first = d.io & 1, hbm_last = (d.io >> 1) & 1;
    const int threads = spec_threads(d), tb = __builtin_ctz(threads);
    const int rows = 1 << (m - tb);  // tile rows of `threads` amplitudes
    ParamSink ps;
    ps.bank = params;
    std::ostringstream o;  // kernel body (the parameter block's size is known once it is written)
    o << ") {\n";
    o << "  extern __shared__ D2 tile[];\n  char* tb = reinterpret_cast<char*>(tile);\n";
    o << "  const unsigned tid = threadIdx.x;\n  u64 base = blockIdx.x;\n";
    // Parameters are read at P.v[z + i] with z zero but different, to the compiler, in each round of the coset
    // loop: they stay inside it (hoisted, all of a phase's would be live at once) and uniform over the warp.
    if (params) o << "  const unsigned zero = blockDim.z - 1u;\n";
    for (int j = 0; j < m; ++j) o << "  base = ins0(base, " << d.q[j] << "u);\n";
    if (!hbm_first || !hbm_last) {
        o << "  u64 lo = 0;\n";
        for (int j = 0; j < tb && j < m; ++j) o << "  lo |= (u64)((tid >> " << j << ") & 1u) << " << d.q[j] << ";\n";
    }
    if (!hbm_first) {
        o << "  {\n";
        for (int k = 0; k < rows; ++k) {
            ITYPE hi = 0;
            for (int j = tb; j < m; ++j)
                if ((k >> (j - tb)) & 1) hi |= 1ULL << d.q[j];
            o << "    asm volatile(\"cp.async.cg.shared.global [%0], [%1], 16;\" :: \"r\"((unsigned)__cvta_generic_to_shared("
              << "tile + swz(tid + " << k * threads << "u))), \"l\"(s + (base | lo | " << u64hex(hi) << ")) : \"memory\");\n";
        }
        o << "    asm volatile(\"cp.async.commit_group;\\ncp.async.wait_group 0;\" ::: \"memory\");\n    __syncthreads();\n  }\n";
    }
    const int np = d.nphases;
    for (int ph = 0; ph < np; ++ph) {
        const StPhase& P = d.phases[ph];
        const bool from_hbm = hbm_first && ph == 0, to_hbm = hbm_last && ph == np - 1;
        o << "  // phase " << ph << ": tile bits " << (int)P.bits[0] << "," << (int)P.bits[1] << "," << (int)P.bits[2] << ","
          << (int)P.bits[3] << ", " << d.programs[ph].steps.size() << " steps\n";
        const unsigned rounds = (ncos + threads - 1) / threads;
        o << "#pragma unroll 1\n  for (unsigned it = 0; it < " << rounds << "u; ++it) {\n    const unsigned c = tid + it * "
          << threads << "u;\n";
        if (ncos < (unsigned)threads) o << "    if (c >= " << ncos << "u) break;\n";
        const std::vector<int> order(P.order, P.order + (m - kPhaseBits));
        o << "    const unsigned u0 = 0u";
        for (size_t k = 0; k < order.size();) {  // runs of consecutive bits
            size_t e = k + 1;
            while (e < order.size() && order[e] == order[e - 1] + 1) ++e;
            o << " | ((c >> " << k << ") & " << ((1u << (e - k)) - 1u) << "u) << " << order[k];
            k = e;
        }
        o << ";\n";
        o << "    D2 r[16];\n";
        if (params) o << "    const unsigned z = zero & it;\n";
        if (from_hbm || to_hbm) {
            o << "    u64 g0 = base;\n";
            for (int j = 0; j < m; ++j) o << "    g0 |= (u64)((u0 >> " << j << ") & 1u) << " << d.q[j] << ";\n";
        }
        if (from_hbm) {
            o << "    { u64 gi = g0;\n";
            for (int g = 0; g < 16; ++g) {
                if (g) o << "      gi ^= " << u64hex(1ULL << d.q[P.bits[gray_bit(g)]]) << ";\n";
                o << "      r[" << (g ^ (g >> 1)) << "] = ldg(s + gi);\n";
            }
            o << "    }\n";
        } else {
            o << "    { unsigned a = swz(u0) << 4;\n";
            for (int g = 0; g < 16; ++g) {
                if (g) o << "      a ^= " << (swz_host(1u << P.bits[gray_bit(g)]) << 4) << "u;\n";
                o << "      r[" << (g ^ (g >> 1)) << "] = *reinterpret_cast<const D2*>(tb + a);\n";
            }
            o << "    }\n";
        }
        for (const ProgStep& s : d.programs[ph].steps) emit_step(o, s, ps);
        int at[16];  // the register that holds coset index i
        for (int j = 0; j < 16; ++j) at[d.programs[ph].out[j]] = j;
        if (to_hbm) {
            o << "    { u64 gi = g0;\n";
            for (int g = 0; g < 16; ++g) {
                if (g) o << "      gi ^= " << u64hex(1ULL << d.q[P.bits[gray_bit(g)]]) << ";\n";
                o << "      stg(s + gi, r[" << at[g ^ (g >> 1)] << "]);\n";
            }
            o << "    }\n";
        } else {
            o << "    { unsigned a = swz(u0) << 4;\n";
            for (int g = 0; g < 16; ++g) {
                if (g) o << "      a ^= " << (swz_host(1u << P.bits[gray_bit(g)]) << 4) << "u;\n";
                o << "      *reinterpret_cast<D2*>(tb + a) = r[" << at[g ^ (g >> 1)] << "];\n";
            }
            o << "    }\n";
        }
        o << "  }\n";
        if (!to_hbm) o << "  __syncthreads();\n";
    }
    if (!hbm_last) {
        // batches of 16 rows per thread: the batch's shared-memory loads first, then its stores; row k's
        // global offset takes k's bits to the tile qubits q[tb..]
        const int batch = rows < 16 ? rows : 16;
        o << "#pragma unroll 1\n  for (unsigned k0 = 0; k0 < " << rows << "u; k0 += " << batch << "u) {\n";
        o << "    D2 v[" << batch << "];\n#pragma unroll\n    for (unsigned k = 0; k < " << batch
          << "u; ++k) v[k] = tile[swz(tid + (k0 + k) * " << threads << "u)];\n";
        o << "#pragma unroll\n    for (unsigned k = 0; k < " << batch << "u; ++k) {\n      const unsigned row = k0 + k;\n"
          << "      u64 hi = 0;\n";
        for (int j = tb; j < m; ++j) o << "      hi |= (u64)((row >> " << j - tb << ") & 1u) << " << d.q[j] << ";\n";
        o << "      stg(s + (base | lo | hi), v[k]);\n    }\n  }\n";
    }
    o << "}\n";
    std::ostringstream h;
    h << kPrelude;
    if (params) h << "struct PassParams { D2 v[" << std::max<size_t>(1, params->size()) << "]; };\n";
    h << "extern \"C\" __global__ void __launch_bounds__(" << threads << ", " << (threads == 256 ? 2 : m >= 12 ? 3 : 4) << ") k_pass_spec(D2* __restrict__ s";
    if (params) h << ", const __grid_constant__ PassParams P";
    return h.str() + o.str();
}

struct Compiled {
    cudaLibrary_t lib = nullptr;
    cudaKernel_t kernel = nullptr;
    bool has_params = false;  // takes a parameter block after the state pointer
    int threads = 256;
    std::set<int> smem_set;  // devices on which the dynamic shared-memory limit is raised
};

std::mutex g_mu;
std::map<std::string, std::shared_ptr<Compiled>> g_cache;
std::map<std::string, std::shared_ptr<std::mutex>> g_building;  // one compile per source at a time

int compile(const std::string& src, const char* name, std::vector<char>* cubin) {
    Nvrtc* N = nvrtc();
    if (!N->h) return set_error(QS_ERR_NOT_SUPPORTED, "specialised kernels: " + N->error);
    nvrtcProgram_t prog = nullptr;
    const std::string file = std::string(name) + ".cu";
    if (N->create(&prog, src.c_str(), file.c_str(), 0, nullptr, nullptr) != 0)
        return set_error(QS_ERR_CUDA, "specialised kernels: nvrtcCreateProgram failed");
    const char* opts[] = {"--gpu-architecture=sm_100a", "--std=c++17"};
    const int rc = N->compile(prog, 2, opts);
    if (rc != 0) {
        size_t n = 0;
        N->log_size(prog, &n);
        std::string log(n, '\0');
        if (n) N->log(prog, &log[0]);
        N->destroy(&prog);
        return set_error(QS_ERR_CUDA, std::string(name) + ": NVRTC compile failed: " + log.substr(0, 2000));
    }
    size_t n = 0;
    N->cubin_size(prog, &n);
    cubin->resize(n);
    N->cubin(prog, cubin->data());
    N->destroy(&prog);
    return QS_OK;
}

}  // namespace

int nvrtc_kernel(const std::string& src, const char* name, void** kernel, double* compile_ms) {
    std::shared_ptr<std::mutex> build_mu;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        auto it = g_cache.find(src);
        if (it != g_cache.end()) {
            *kernel = it->second.get();
            if (compile_ms) *compile_ms = 0.;
            return QS_OK;
        }
        auto& b = g_building[src];
        if (!b) b = std::make_shared<std::mutex>();
        build_mu = b;
    }
    std::lock_guard<std::mutex> blk(*build_mu);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        auto it = g_cache.find(src);
        if (it != g_cache.end()) {
            *kernel = it->second.get();
            if (compile_ms) *compile_ms = 0.;
            return QS_OK;
        }
    }
    const auto t0 = std::chrono::steady_clock::now();
    std::vector<char> cubin;
    int rc = compile(src, name, &cubin);
    if (rc != QS_OK) return rc;
    auto C = std::make_shared<Compiled>();
    cudaError_t e = cudaLibraryLoadData(&C->lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
    if (e != cudaSuccess) return check_cuda(e, "cudaLibraryLoadData (specialised kernel)");
    e = cudaLibraryGetKernel(&C->kernel, C->lib, name);
    if (e != cudaSuccess) return check_cuda(e, "cudaLibraryGetKernel (specialised kernel)");
    if (compile_ms)
        *compile_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    std::lock_guard<std::mutex> lk(g_mu);
    g_cache[src] = C;  // entries live for the process, so the handle stays valid
    g_building.erase(src);
    *kernel = C.get();
    return QS_OK;
}

int launch_nvrtc_kernel(void* handle, dim3 grid, dim3 block, void** args, size_t smem, size_t smem_limit,
    cudaStream_t st, const char* what) {
    Compiled* C = static_cast<Compiled*>(handle);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return check_cuda(e, "cudaGetDevice");
    {
        // raise the kernel's dynamic shared-memory limit once per device
        std::lock_guard<std::mutex> lk(g_mu);
        if (!C->smem_set.count(dev)) {
            e = cudaFuncSetAttribute((const void*)C->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                (int)smem_limit);
            if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute (specialised kernel)");
            C->smem_set.insert(dev);
        }
    }
    e = cudaLaunchKernel((const void*)C->kernel, grid, block, args, smem, st);
    if (e != cudaSuccess) return check_cuda(e, what);
    return check_launch(what);
}

int specialized_pass_kernel(const PassDesc& d, void** kernel, std::vector<double2>* params, double* compile_ms) {
    if (d.m < 7 || d.m > kTileBits || d.nphases == 0)
        return set_error(QS_ERR_NOT_SUPPORTED, "specialised passes need 7..12 tile qubits and a phase");
    params->clear();
    std::string src = pass_source(d, params);
    if (params->empty() || params->size() * sizeof(double2) > kMaxParamBytes) {
        // no parameters (the kernel takes only the state), or too many for a parameter block: literals
        params->clear();
        src = pass_source(d, nullptr);
    }
    const int rc = nvrtc_kernel(src, "k_pass_spec", kernel, compile_ms);
    if (rc != QS_OK) return rc;
    static_cast<Compiled*>(*kernel)->has_params = !params->empty();  // properties of the source
    static_cast<Compiled*>(*kernel)->threads = spec_threads(d);
    return QS_OK;
}

int launch_specialized_pass(void* handle, double2* state, const double2* params, ITYPE tiles, int m, cudaStream_t st) {
    Compiled* C = static_cast<Compiled*>(handle);
    if (C->has_params && !params) return set_error(QS_ERR_INVALID_ARGUMENT, "specialised pass: no parameter block");
    void* args[] = {&state, const_cast<double2*>(params)};  // the parameter block is copied at launch
    return launch_nvrtc_kernel(handle, dim3((unsigned)tiles), dim3(C->threads), args, sizeof(double2) << m,
        sizeof(double2) << kTileBits, st, "k_pass_spec");
}

std::string specialized_pass_source(const PassDesc& d) {
    std::vector<double2> params;
    return pass_source(d, &params);
}

}  // namespace qs
