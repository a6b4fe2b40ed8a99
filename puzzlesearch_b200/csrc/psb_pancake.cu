// Kernel table for the pancake puzzle (Puzzles/PancakeSimple.cpp), one
// instantiation per size: sizes 2..16 (PancakeSimple.cpp:26).
#include "psb_kernels.cuh"
#include "psb_pancake_windows.cuh"
#include "psb_small.cuh"

namespace psb {

namespace {
template <int N>
PuzzleKernels pancake_table() {
    PuzzleKernels k = make_kernels<PancakeK<N>>();
    if constexpr (N >= kPancakeWindowsMin) {
        k.level[kThreeBit] = k.level_shape[0][kThreeBit] = &launch_pancake_level<N, kThreeBit>;
        k.level[kClassic] = &launch_pancake_level<N, kClassic>;
        k.level[kTwoBit] = k.level_shape[0][kTwoBit] = &launch_pancake_level<N, kTwoBit>;
        k.level_shape[1][kThreeBit] = &launch_pancake_level<N, kThreeBit, 1>;
        k.level_shape[1][kTwoBit] = &launch_pancake_level<N, kTwoBit, 1>;
        k.level_shape[2][kThreeBit] = &launch_pancake_level<N, kThreeBit, 2>;
        k.level_shape[2][kTwoBit] = &launch_pancake_level<N, kTwoBit, 2>;
    } else {
        k.small = &launch_small_search<PancakeK<N>>;
    }
    return k;
}
}  // namespace

bool pancake_kernels(int n, PuzzleKernels* out) {
    switch (n) {
#define PSB_CASE(N) case N: *out = pancake_table<N>(); return true;
        PSB_CASE(2) PSB_CASE(3) PSB_CASE(4) PSB_CASE(5) PSB_CASE(6) PSB_CASE(7) PSB_CASE(8) PSB_CASE(9)
        PSB_CASE(10) PSB_CASE(11) PSB_CASE(12) PSB_CASE(13) PSB_CASE(14) PSB_CASE(15) PSB_CASE(16)
#undef PSB_CASE
    }
    return false;
}

}  // namespace psb
