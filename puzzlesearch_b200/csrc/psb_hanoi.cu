// Kernel table for four-peg Towers of Hanoi (Puzzles/FourPegHanoiSimple.cpp);
// the disk count and the symmetry flag are runtime arguments.
#include <algorithm>

#include "psb_hanoi_words.cuh"
#include "psb_kernels.cuh"
#include "psb_small.cuh"

namespace psb {

// Top-down level, 64 states at a time.  A fixed number of blocks walks the
// windows: each looks up the flags of blockDim.x of its windows at once, so a
// thin level of a large search reads its flags instead of launching a block
// per window (17 disks: 131,072 windows).
template <int MODE, int T>
__global__ void __launch_bounds__(T, 1024 / T) hanoi_level_kernel(LevelArgs a, uint32_t n_windows) {
    extern __shared__ __align__(16) unsigned long long smem64[];
    __shared__ WindowShared sh;
    __shared__ uint32_t active[T / 32];
    HanoiCounts cnt;
    hanoi_begin<MODE, T>(a, smem64, sh);
    for (uint64_t g = blockIdx.x; g < n_windows; g += uint64_t(gridDim.x) * T) {
        const uint64_t mine = g + uint64_t(threadIdx.x) * gridDim.x;
        const bool on = mine < n_windows && (!a.wflag_cur || a.wflag_cur[mine]);
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
        if ((threadIdx.x & 31) == 0) active[threadIdx.x >> 5] = bal;
        __syncthreads();
        for (int i = 0; i < T / 32; ++i) {
            uint32_t m = active[i];
            while (m) {
                const uint32_t j = __ffs(m) - 1;
                m &= m - 1;
                hanoi_window<MODE, T>(a, g + uint64_t(32 * i + j) * gridDim.x, smem64, sh, cnt);
            }
        }
        __syncthreads();  // every thread has read active[]
    }
    hanoi_end<MODE>(a, cnt, sh);
}

template <int MODE, int V = 0>
cudaError_t launch_hanoi_level(const LevelArgs& a, unsigned grid, size_t smem, cudaStream_t s) {
    if (!hanoi_words_ok(a.pz)) return launch_level<HanoiK, MODE, false, V>(a, grid, smem, s);
    constexpr int T = variant_threads(V);
    const size_t bytes = hanoi_smem_bytes(MODE, size_t(1) << a.window_bits, T);
    constexpr size_t limit = hanoi_smem_bytes(MODE, size_t(1) << window_bits_max(MODE), T);  // as launch_level's
    cudaError_t e = cudaFuncSetAttribute(hanoi_level_kernel<MODE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(limit));
    if (e != cudaSuccess) return e;
    // As many blocks as 148 SMs hold at once by threads; where shared memory
    // holds fewer, the rest queue up (no block waits for another).
    const unsigned blocks = std::min(grid, 148u * (1024 / T));
    hanoi_level_kernel<MODE, T><<<blocks, T, bytes, s>>>(a, grid);
    return cudaGetLastError();
}

bool hanoi_kernels(PuzzleKernels* out) {
    *out = make_kernels<HanoiK>();
    out->level[kThreeBit] = out->level_shape[0][kThreeBit] = &launch_hanoi_level<kThreeBit>;
    out->level[kClassic] = &launch_hanoi_level<kClassic>;
    out->level[kTwoBit] = out->level_shape[0][kTwoBit] = &launch_hanoi_level<kTwoBit>;
    out->level[kFrontier] = &launch_hanoi_level<kFrontier>;
    out->level_shape[1][kThreeBit] = &launch_hanoi_level<kThreeBit, 1>;
    out->level_shape[1][kTwoBit] = &launch_hanoi_level<kTwoBit, 1>;
    out->level_shape[2][kThreeBit] = &launch_hanoi_level<kThreeBit, 2>;
    out->level_shape[2][kTwoBit] = &launch_hanoi_level<kTwoBit, 2>;
    out->small = &launch_small_search<HanoiK>;
    return true;
}

}  // namespace psb
