// tiles.h -- plain gate lists in shared-memory tiles (tiles.cu).
#pragma once

#include <vector>

#include "qcs_cuda.h"

struct qcs_cuda_state;

namespace qcs {

// Consecutive gates ops[first .. last) run in one pass over the state, on the
// tile qubits `qubits` (a bit mask).  A group applies `gates` in order, whose
// non-diagonal targets lie on at most `regs` qubits (its mask), then `moves` (X,
// CNOT).
struct TileStretch {
  struct Group {
    unsigned long long qubits = 0;
    std::vector<int> gates, moves;
  };
  int first = 0, last = 0;
  unsigned long long qubits = 0;
  std::vector<Group> groups;
};

// The passes of a gate list on n qubits with tiles of 2^nt amplitudes that
// always hold the `low` lowest qubits.  The gates keep their order (but for
// moves that commute exactly).
std::vector<TileStretch> tile_stretches(const qcs_cuda_op *ops, int count, int n, int nt, int low,
                                        bool reference, int regs);

// Applies a list of gates (no phase flips or diffusions) in place.
int run_tiles(qcs_cuda_state *s, const qcs_cuda_op *ops, int count);
bool tiles_supported(const qcs_cuda_state *s);

}  // namespace qcs
