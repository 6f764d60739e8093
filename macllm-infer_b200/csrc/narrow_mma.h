// Matmul of the narrowest ticks: a handful of rows against a 16-bit image or against Q4_K / Q6_K units (see narrow_mma.cu).
#pragma once
#include "common.cuh"
#include "device_util.h"
#include "row_types.cuh"

namespace mk {

constexpr int kNarrowImageRows = 16, kNarrowBlockRows = 8;   // most activation rows of a call: on a 16-bit image, on Q4_K / Q6_K units

// RG row tiles of 16 are a CTA's work at a time, 8 / RG of its warps share the K of each; `shares` CTAs share K besides and leave partial sums.
struct NarrowPlan {
    int RG = 1, shares = 1, ctas = 0;
    size_t smem = 0, partial_floats = 0;
    double us = 0.0;                    // what the plan is expected to take, to compare plans with
    bool ok = false;                    // there is a plan within the scratch and the shared memory
};
enum class NarrowFormat : int { F16 = 0, BF16 = 1, Blocks = 2 };  // Blocks: Q4_K / Q6_K units
// The cut of a call that is better off here than on the tcgen05 kernels; not ok: it is theirs.  Launches and the host's query go by it alike.  q6: a
// matrix of the call is in Q6_K.
NarrowPlan narrow_plan(NarrowFormat format, bool q6, int64_t rows, int64_t cols, int T, bool gated, int max_shares, size_t scratch_floats, int n_inputs, int sms);

struct NarrowCall {
    NarrowFormat format = NarrowFormat::F16;
    const void* w = nullptr;            // image [rows][cols], or the units of the first matrix
    const void* w2 = nullptr;           // units of the second matrix, whose rows follow
    int64_t rows = 0, rows_first = 0, cols = 0;
    bool q6 = false, q6_2 = false;      // Blocks: the matrices' formats
    int n_inputs = 1;                   // image: stacked projections with inputs of their own (see HalfWeight)
    int input_end[kMaxRowGroups] = {};  // in 128-row tiles
    int input_tiles = 0;
    const __half* x = nullptr;          // [n_inputs][T][cols], 16-bit values of the image's kind
    int T = 0;
    // the result: rows y[t][n], or partial sums partial[(share * T + t) * rows + n] where there are shares, or f16 / bf16 (as the image) gated
    // rows yh[t][n / 2], or `scatter`
    float* y = nullptr;
    int ldy = 0;
    float out_scale = 1.f, softcap = 0.f;
    float* partial = nullptr;
    int32_t* status = nullptr;          // non-zero after a bounded wait gave up
    const GatedAct* act = nullptr;
    __half* yh = nullptr;
    int ldyh = 0;
    const MatmulScatter* scatter = nullptr;
};
// The plan is narrow_plan's for the same call.
void launch_narrow_mma(const NarrowCall& c, const NarrowPlan& plan, cudaStream_t s);

}  // namespace mk
