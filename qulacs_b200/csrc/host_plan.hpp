// A staged schedule as the host plans it: passes, their phases and the phases' programs (csrc/staged.cu
// builds and uploads it; csrc/staged_replay.cpp runs it on a host state).
#pragma once

#include <vector>

#include "circuit.hpp"
#include "phase_program.hpp"
#include "staged.hpp"

namespace qs {

struct PassPlan {
    bool single = false;  // a gate run by the gate-by-gate kernels
    int gate = -1;
    std::vector<UINT> q;  // tile qubits (ascending)
    std::vector<int> gates;
};

struct HostPlan {
    std::vector<PassPlan> passes;
    std::vector<StPhase> phases;
    std::vector<StOp> ops;      // the phases' gates and their parameters
    std::vector<double2> pool;
    std::vector<PhaseProgram> programs;  // one per phase
    std::vector<StStep> steps;  // the programs as the generic kernels read them
    std::vector<double2> params;
    struct Range {
        size_t phase_begin, nphases;
    };
    std::vector<Range> pp;
};

// Host-only part of planning: passes, phases and their programs (no device calls).  The gates are in
// rotation form.  `spec`: the passes will run specialised kernels.
void make_host_plan(const std::vector<GateRec>& gates, UINT n, HostPlan* H, int tile_bits = kTileBits, bool spec = false);

}  // namespace qs
