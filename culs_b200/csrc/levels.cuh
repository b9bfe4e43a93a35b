// Levels of one graph in the shared memory of one block (levels.cu).
#pragma once

#include "rw_work.cuh"

namespace culs {

// Node i of an order of n nodes has fanin literals 2 * (order index) +
// complement in a0[i] and a1[i]; a0[i] = kLevelZero for the constant and the
// PIs, kLevelSkip for a node to leave out.  With pre, a node of pre[i] != -1
// is a constant or PI whatever a0 says.
constexpr int kLevelZero = -1, kLevelSkip = -2;
struct LevelsArgs {
    int64_t n = 0;
    const int *a0 = nullptr, *a1 = nullptr;
    const int *pre = nullptr;
    const int *posOf = nullptr;       // where node i's results go (null: i)
    int *level = nullptr;             // level, or
    int *levelPhase = nullptr;        //   2 * level + phase
    const uint8_t *counted = nullptr; // by posOf: the nodes that count towards the depth (null: all)
    int *depth0 = nullptr, *depth1 = nullptr;  // raised to the largest level
    int *unsettled = nullptr;         // raised by the nodes left without a level
    int *status = nullptr;
};

constexpr int64_t kLevelsBlockMax = 57000;  // nodes whose words fit a block's shared memory
// Runs the pass on one block; n <= kLevelsBlockMax.
cudaError_t levels_block(const LevelsArgs &A, cudaStream_t s);

}  // namespace culs
