// Which barrier and which of its phases belongs to which tile of the prefill attention (attention_umma.cu).  Plain arithmetic, so that the host can walk it too.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define MK_PHASES __host__ __device__ __forceinline__
#else
#define MK_PHASES inline
#endif

namespace mk {

// Scores, weights and output products of tile t are told of by barrier `at` of a pair, in its phase of this parity.  A pair, because a parity only tells neighbouring
// phases apart: whoever waits for tile t's must know that the same barrier's phase before, tile t - 2's, is over.  For output products that holds
// without a wait for every tile's: the scores of tile t + 1 are there, and they were asked for behind the product of tile t - 1.
struct TilePhase {
    int at;
    uint32_t parity;
};
MK_PHASES TilePhase tile_phase(int t) { return TilePhase{t & 1, (uint32_t)(t >> 1 & 1)}; }

}  // namespace mk

#undef MK_PHASES
