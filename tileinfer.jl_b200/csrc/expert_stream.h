// The form of the grouped products in which every (token, choice) pair finds its unit by itself (csrc/expert_stream.cu).
#pragma once
#include "common.cuh"

#define ES_ACT_NONE 0
#define ES_ACT_RELU2 1

// A unit's matrix is [out, in], or with `gated` [2 * out, in]: gate rows and then up rows, with `limits` [units], slope and shift of the
// clamped gated unit. y [pairs, out]; pair p reads row p / per_row of x (the choices of a token, or 1 where x has a row per pair), times
// scores[p], rounded, where `scores` is given. `ids` null: pair p is row p % units of token p / units and takes unit p % units. `pair_row` (or
// null) receives the pairs' rows in y, -1 for a choice without a unit (ids < 0). `ahead`: the kernel right before this one on the stream has
// not written `ids` (an earlier one has), so they and the first weights may be read while it still runs.
struct ExpertStream {
    const int* ids;
    const float* scores;
    int* pair_row;
    const float* limits;
    int pairs, per_row, gated, act, ahead;
    float slope, shift;
};

int expert_stream(void* y, const void* x, const void* W, const ExpertStream& e, int units, int out, int in, cudaStream_t stream);
