// A warp's ring of asynchronous copies in narrow_mma.cu: which stage and which barrier phase belongs to which copy.  Plain arithmetic, so that the host can
// walk it too.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define MK_RING __host__ __device__ __forceinline__
#else
#define MK_RING inline
#endif

namespace mk {

// Copies are asked for and waited for in the same order, at most `stages` of them at a time, one barrier per stage.
struct NarrowRing {
    int stages, to_load;           // copies that are still to be asked for
    int load_stage = 0, stage = 0; // of the next copy, of the next wait
    uint32_t phase = 0;            // parity of the next wait

    MK_RING NarrowRing(int n_stages, int copies) : stages(n_stages), to_load(copies) {}
    MK_RING bool more() const { return to_load != 0; }
    MK_RING void loaded() {
        --to_load;
        load_stage = load_stage + 1 == stages ? 0 : load_stage + 1;
    }
    MK_RING void used() {
        if (stage + 1 == stages) {
            stage = 0;
            phase ^= 1;
        } else {
            ++stage;
        }
    }
    // The wait for the present stage was in vain, `left` copies (that one included, the later ones asked for or not) before the last: nothing more is asked
    // for.  Returns what drain() is to be given, never 0.
    MK_RING uint32_t give_up(int left) {
        to_load = 0;
        return (uint32_t)(left < stages ? left : stages) | (uint32_t)stage << 8 | phase << 16;
    }
    // wait(stage, parity) for every copy that was under way when the ring was given up.  Only those: a stage that was not asked for again has a phase that
    // never completes.
    template <typename Wait>
    static MK_RING void drain(int stages, uint32_t given_up, Wait wait) {
#pragma unroll 1
        for (int j = 0; j < (int)(given_up & 255); ++j) {
            const int at = (int)(given_up >> 8 & 255) + j;
            wait(at < stages ? at : at - stages, given_up >> 16 ^ (at < stages ? 0u : 1u));
        }
    }
};

// Row groups i0 .. i1 - 1 of (1 << rg_shift) 16-row tiles: how many hold a tile at place `sub_tile` of a matrix of `tiles` (the last groups may reach past it).
MK_RING int narrow_live_groups(int i0, int i1, int rg_shift, int sub_tile, int tiles) {
    const int end = tiles > sub_tile ? (tiles - sub_tile + (1 << rg_shift) - 1) >> rg_shift : 0;
    return (end < i1 ? end : i1) > i0 ? (end < i1 ? end : i1) - i0 : 0;
}

}  // namespace mk

#undef MK_RING
