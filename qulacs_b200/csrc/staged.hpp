// Host-visible description of a staged pass (csrc/staged.cu builds it; csrc/pass_codegen.cpp turns one
// pass into a specialised kernel).  A pass owns m tile qubits q[0..m-1] (ascending, q[j] = j for
// j < kLowFixed); its gates run in phases of 4 tile bits, each phase a list of register ops on a
// thread's 16-amplitude coset, run as a program of register steps.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

typedef unsigned long long ITYPE;
typedef unsigned int UINT;

namespace qs {

constexpr int kLowFixed = 4;        // qubits 0..3 always belong to a tile
constexpr int kTileBits = 12;       // pass kernel: 2^12 amplitudes = 64 KiB of shared memory per CTA
constexpr int kBatchTileBits = 11;  // multi-circuit kernel: 2^11 amplitudes = 32 KiB
constexpr int kPhaseBits = 4;       // 16 amplitudes (a coset) in registers per thread
constexpr int kStThreads = 256;     // pass kernel: one coset per thread of a 2^12-amplitude tile
constexpr int kBatchThreads = 128;  // multi-circuit kernel: one per thread of a 2^11-amplitude tile

// XOR swizzle of the tile index.  A quarter warp's eight 16-byte accesses are conflict-free when the
// low three bits of swz() differ, that is when the swizzle vectors of the three tile bits that its lanes
// run over are independent.  With these shifts every set of 4 phase bits out of 11 or 12 tile bits leaves
// such a triple, which lane_order puts first.  Linear over XOR: swz(a | b) = swz(a) ^ swz(b) for disjoint bits.
#define QS_SWZ(u) ((u) ^ ((((u) >> 3) ^ ((u) >> 5) ^ ((u) >> 6) ^ ((u) >> 8)) & 7u))

// Gates of a phase, from which its program (phase_program.hpp) is built.
enum StKind : uint8_t {
    ST_DENSE1 = 0, ST_DIAG1, ST_RX, ST_RY, ST_CNOT, ST_CZ, ST_SWAP, ST_DENSE2,
    // depolarizing channels of a density matrix seen as a vector; parameter: the channel's probability.
    // a, b: column and row bit (one qubit), or the two column bits with the row bits in aux (two qubits)
    ST_DEPOL1, ST_DEPOL2
};

struct StOp {
    uint8_t kind, a, b, aux;  // a, b: register-bit indices 0..3 within the phase; aux: ST_DIAG1 1 = its phase is
                              // a parameter, ST_DEPOL2 the row bits
    uint32_t param;           // index into the parameter pool (double2); the parameters of ST_RX, ST_RY and
                              // ST_DIAG1 are followed by their low parts (hi + lo)
};
// A step of a phase's program for the generic kernels.
struct StStep {
    uint8_t code, pad;
    uint16_t mask;   // registers of a diagonal or of signs; a channel's form
    uint32_t param;  // index into the steps' parameter pool
};
// Bits of StPhase::flags.
enum PhaseFlag : uint8_t {
    PH_TURNS_FIRST = 1,  // rounds of tangents, then factors
    PH_TAIL = 2,         // factors after the last round
    PH_SAME_NEXT = 4     // the next phase has the same tile bits (relabel_segments)
};
// Four 16-byte words, as the kernels read them.
struct alignas(16) StPhase {
    uint8_t bits[4];   // tile-local bit positions, ascending
    uint8_t order[8];  // tile bit of bit k of the coset number
    uint8_t in[4];     // register j starts with coset index XOR of in[k] over the bits k of j (specialised: j)
    uint8_t out0, out[4];  // after the steps it holds coset index out0 ^ (XOR of out[k] over the bits k of j)
    uint8_t flags;
    uint16_t out0_at, in_at[4], out_at[4];  // in, out0 and out as swizzled byte offsets into the tile
    // Its program for the generic kernels, from `param` of the parameter pool: `rounds` of 16 diagonal factors and 4
    // tangents (16 + 2 entries), then 16 more factors (PH_TAIL); or rounds of 4 tangents and 16 factors
    // (PH_TURNS_FIRST); or, where it needs other steps, those.
    uint32_t rounds, param;
    uint32_t step_begin, step_count;
    uint32_t op_begin, op_count;  // its gates (host)
};
static_assert(sizeof(StPhase) == 64, "four words");

// One pass as the code generator sees it: tile qubits, the HBM-direct first/last phase flags, and the
// programs of its phases.
struct PhaseProgram;
struct PassDesc {
    int m = 0;
    int io = 0;  // bit 0: the first phase gathers from HBM; bit 1: the last phase scatters to HBM
    UINT q[kTileBits] = {};
    const StPhase* phases = nullptr;
    const PhaseProgram* programs = nullptr;
    int nphases = 0;
};

// csrc/pass_codegen.cpp: a kernel for one pass with its tile qubits, phase bits and programs compiled
// in (NVRTC, sm_100a), cached by source for the life of the process.  `handle` receives the
// cache entry (valid until exit), launched over dim >> m CTAs with 16 << m bytes of dynamic shared memory.  QS_ERR_NOT_SUPPORTED when NVRTC cannot be loaded.
// The kernel depends only on the pass's structure: its gate parameters are a kernel-parameter block
// whose values `params` receives (empty when the pass has too many and they are literals instead), to
// be passed at every launch.
int specialized_pass_kernel(const PassDesc& d, void** handle, std::vector<double2>* params, double* compile_ms);
int launch_specialized_pass(void* handle, double2* state, const double2* params, ITYPE tiles, int m, cudaStream_t st);
std::string specialized_pass_source(const PassDesc& d);

}  // namespace qs
