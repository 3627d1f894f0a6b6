// A staged phase (a thread's 16-amplitude coset and the gates applied to it) as a short list of register
// steps in which each gate costs the fewest FP64 instructions.  csrc/phase_program.cpp builds it on the
// host; the generic pass kernels (csrc/staged.cu) interpret it and csrc/pass_codegen.cpp turns it into
// CUDA C, with the same arithmetic step by step.
//
// What bounds a pass is FP64 issue (64 lanes per SM and clock): a 2 x 2 complex matrix costs 8 FP64
// instructions per amplitude.  Here a unitary U is written D1 R D2 with unit diagonals and a real rotation:
//  * rotations run scaled: x + t y, y - t x with t = tan of the half angle, one fma per real number (2 per
//    amplitude), and the cosine joins one scalar of the whole pass;
//  * diagonal factors (D1, D2, RZ, CZ, phase gates) are collected and applied together, 16 complex
//    factors per coset (4 per amplitude) for every diagonal that can meet there, or sign flips alone (0);
//  * CNOT, SWAP and X only relabel registers (an affine map over GF(2) of the register index), 0.  In a
//    phase with dense matrices or channels they are steps that move registers, so that those act on
//    register bits.  The generic kernels rotate along register bits only (relabel_segments, csrc/staged.cu).
#pragma once

#include <complex>
#include <vector>

#include "staged.hpp"

namespace qs {

enum StepKind : uint8_t {
    SP_DIAG, SP_SIGN, SP_ROT, SP_DENSE1, SP_DENSE2, SP_DEPOL1, SP_DEPOL2, SP_SCALE, SP_CNOT, SP_SWAP, SP_X
};
// Rotation forms; (x, y) are the pair's amplitudes where the qubit is 0 and 1.
//   tan: par t, x + t y, y - t x (cosine deferred);  cot: par u, u x + y, u y - x (sine deferred);
//   full: par c, s.  RX likewise with i: x + i t y, y + i t x.
enum RotForm : uint8_t { RF_Y_TAN, RF_Y_COT, RF_Y_FULL, RF_X_TAN, RF_X_COT, RF_X_FULL };

// Register j and register j ^ v[i] differ in the qubit i of the step; the qubit's value in register j is
// parity(f[i] & j) ^ a[i].
struct ProgStep {
    StepKind kind = SP_DIAG;
    uint8_t form = 0;       // SP_ROT: RotForm; SP_DEPOL1, SP_DEPOL2: 0 scaled, 1 full; SP_SCALE: 1 complex
    uint8_t nq = 0;
    uint8_t v[4] = {}, f[4] = {}, a[4] = {};
    uint16_t mask = 0;      // SP_DIAG: registers with a factor; SP_SIGN: registers negated
    std::vector<double2> par;  // SP_DIAG: 16 factors; SP_ROT: (t, 0) or (c, s); dense: the matrix; ...
    std::vector<std::complex<long double>> xpar;  // SP_DIAG: the factors before rounding
};

struct PhaseProgram {
    std::vector<ProgStep> steps;
    uint8_t out[16];        // the coset index whose amplitude register j holds after the steps
};

// Whether a real scale deferred over a pass may grow this much (log2): far inside the FP64 range.
constexpr double kMaxDeferredBits = 400.;

// The programs of a pass's phases, from its ops.
std::vector<PhaseProgram> build_pass_program(const StPhase* phases, size_t count, const StOp* ops, const double2* pool);

// A phase's program as the generic kernels read it: rounds or steps and their parameters appended, and the
// phase's map from register bits to tile bits after them filled in.
void encode_program(const PhaseProgram& P, std::vector<StStep>* steps, std::vector<double2>* pool, StPhase* phase);

// Value of a step's qubit i in register j.
inline int step_bit(const ProgStep& s, int i, int j) { return (__builtin_popcount(s.f[i] & j) & 1) ^ s.a[i]; }

}  // namespace qs
