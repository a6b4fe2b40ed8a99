// psb_pancake_windows.cuh -- top-down pancake levels in windows of 8! states.
//
// A flip of m values only changes the last m Lehmer digits, so it stays
// inside its aligned block of m! indexes.  level_window's windows of 2^16
// states cut those blocks anywhere: every flip of 4 and more had to test
// whether its child is in the window, and a warp then ran both the
// shared-memory mark and the long-range mark for almost every flip (62% of
// the lanes active, 13-pancake).  An aligned window of 8! states holds every
// flip of up to 8 of its parents: those are marked in shared memory with no
// test, and the larger flips are always marked in global memory (29 of 32
// lanes active).  8! = 40,320 is a multiple of 64, so windows begin on array
// words, and the eight unranking prefixes of its blocks of 7! are made once.
// B200, whole searches against the windows of 2^16: 13-pancake two-bit
// 154 -> 138 ms, three-bit 162 -> 152 ms, 12-pancake three-bit 9.0 -> 7.7 ms.
// Windows of 9! keep one flip more on chip but spread the long-range marks in
// flight over nine times the states, which costs more in L2 than it saves
// (13-pancake two-bit 163 ms).
//
// The window flags keep their 2^window_bits states each; a window looks at
// all it overlaps and sweeps only the units of flagged ones.
#pragma once

#include "psb_kernels.cuh"

namespace psb {

constexpr int kPancakeK = 8;
constexpr uint32_t kPancakeWindow = uint32_t(fact(kPancakeK));
// 11 pancakes make 990 windows; smaller searches keep level_window, whose
// smaller windows give every SM some.
constexpr int kPancakeWindowsMin = 11;
constexpr uint32_t kPancakeUnit = 32;  // states per lane and chunk, in every mode

// Marks, each warp's list of a chunk's states, the unranking prefixes of the
// window's blocks of 7! indexes.
template <int N>
__host__ __device__ constexpr size_t pancake_smem_bytes(int threads) {
    return size_t(kPancakeWindow / 8) + size_t(threads / 32) * (32 * kPancakeUnit * 2) +
           size_t(kPancakeWindow / PancakeK<N>::kBlock) * sizeof(typename PancakeK<N>::Prefix);
}

template <int MODE>
struct PancakeEmitter {
    const LevelArgs& a;
    uint32_t* smarks;
    uint32_t parent_off = 0;  // the parent's offset in the window
    uint32_t marked = 0, bad = 0;

    __device__ __forceinline__ uint64_t next_code() const { return a.cur_code == 2 ? 3u : 1u; }
    __device__ __forceinline__ void flag(uint64_t c) {
        if (!a.wflag_next) return;
        uint8_t* f = a.wflag_next + (c >> a.window_bits);
        if (!*f) *f = 1;
    }
    template <bool kFar>
    __device__ __forceinline__ void remote(uint64_t c) {
        if (c >= a.n_states) { bad = 1; return; }  // never expected: keeps a bad index off the memory system
        if constexpr (MODE == kTwoBit) {
            if (a.far && (!kFar || a.far_all)) {
                flag(c);
                if constexpr (kFar) red_or_far(a.far + (c >> 5), 1u << (uint32_t(c) & 31u));
                else atomicOr(a.far + (c >> 5), 1u << (uint32_t(c) & 31u));
                return;
            }
            const unsigned long long* w = reinterpret_cast<unsigned long long*>(a.marks) + (c >> 5);
            complete(c, kFar ? ld_cg_far(w) : __ldcg(w));
        } else {
            flag(c);
            unsigned int* w = reinterpret_cast<unsigned int*>(a.marks) + (c >> 5);
            if constexpr (kFar) red_or_far(w, 1u << (uint32_t(c) & 31u));
            else atomicOr(w, 1u << (uint32_t(c) & 31u));
        }
    }
    // Two-bit: UNVISITED -> NEXT, given the target's code word.
    __device__ __forceinline__ void complete(uint64_t c, uint64_t word) {
        const uint32_t sh = 2u * (uint32_t(c) & 31u);
        if ((word >> sh) & 3u) return;
        flag(c);
        atomicOr(reinterpret_cast<unsigned long long*>(a.marks) + (c >> 5), (unsigned long long)next_code() << sh);
        ++marked;
    }
    // Flip of op + 2 <= 12 values; op is a constant after unrolling.
    __device__ __forceinline__ void rel(uint64_t parent, int32_t delta, uint32_t op) {
        if (op + 2 <= uint32_t(kPancakeK)) {
            const uint32_t o = parent_off + uint32_t(delta);
            atomicOr(&smarks[o >> 5], 1u << (o & 31u));
        } else {
            remote<false>(parent + int64_t(delta));
        }
    }
    __device__ __forceinline__ void operator()(uint64_t c, uint32_t) { remote<false>(c); }
    // Flips of 13 and more (see EmitFar, EmitSplitFar).
    __device__ __forceinline__ void far(uint64_t c, uint32_t) { remote<true>(c); }
    __device__ __forceinline__ FarTicket far_issue(uint64_t c, uint32_t) {
        if constexpr (MODE == kTwoBit) {
            if (c < a.n_states && !(a.far && a.far_all))
                return FarTicket{ld_cg_far(reinterpret_cast<const unsigned long long*>(a.marks) + (c >> 5)), true};
        }
        remote<true>(c);
        return FarTicket{0, false};
    }
    __device__ __forceinline__ void far_finish(uint64_t c, uint32_t, const FarTicket& t) {
        if constexpr (MODE == kTwoBit) {
            if (t.pending) complete(c, t.word);
        }
    }
};

// Window `window` (8! states) of one top-down level.
template <int N, int MODE, int T>
__device__ __forceinline__ void pancake_window(const LevelArgs& a, uint64_t window, unsigned long long* smem64,
                                               WindowShared& sh) {
    using PZ = PancakeK<N>;
    using Prefix = typename PZ::Prefix;
    constexpr int kWarps = T / 32;
    constexpr uint32_t W = kPancakeWindow, kUnits = W / kPancakeUnit;
    static_assert(W % 128 == 0 && W % PZ::kBlock == 0 && N > kPancakeK, "windows of whole words and blocks");
    constexpr uint32_t kChunks = (kUnits + 31) / 32, kChunk = 32 * kPancakeUnit;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t base = window * W;
    const uint32_t f0 = uint32_t(base >> a.window_bits);
    if (a.wflag_cur) {  // no frontier state unless a flagged window overlaps this one
        const uint32_t f1 = uint32_t((base + W - 1) >> a.window_bits);
        int any = 0;
        for (uint32_t f = f0 + tid; f <= f1; f += T) any |= a.wflag_cur[f];
        if (!__syncthreads_or(any)) return;
    }
    uint32_t* smarks = reinterpret_cast<uint32_t*>(smem64);
    char* scratch = reinterpret_cast<char*>(smem64) + W / 8;
    uint16_t* wlist = reinterpret_cast<uint16_t*>(scratch) + size_t(warp) * kChunk;
    Prefix* pref = reinterpret_cast<Prefix*>(scratch + size_t(kWarps) * kChunk * 2);
    constexpr uint32_t kBlocks = W / PZ::kBlock;
    for (uint32_t i = tid; i < kBlocks; i += T) PZ::make_prefix(uint32_t(base / PZ::kBlock) + i, pref[i]);

    for (uint32_t i = tid; i < W / 128; i += T) reinterpret_cast<uint4*>(smem64)[i] = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        sh.any = 0;
        sh.next_chunk = kWarps;  // chunks 0 .. kWarps-1 go to warps 0 .. kWarps-1
        for (int i = 0; i < 8; ++i) sh.cnt[i] = 0;
    }
    __syncthreads();

    PancakeEmitter<MODE> em{a, smarks};
    uint32_t found = 0;
    // Lane's unit of chunk ch: its array word (two-bit: 32 codes, else 32 bits).
    using Word = typename std::conditional<MODE == kTwoBit, uint64_t, uint32_t>::type;
    Word* front = reinterpret_cast<Word*>(a.front) + base / kPancakeUnit;
    auto load = [&](uint32_t ch) -> Word {
        const uint32_t u = ch * 32 + uint32_t(lane);
        if (ch >= kChunks || u >= kUnits) return 0;
        if (a.wflag_cur && !a.wflag_cur[(base + u * kPancakeUnit) >> a.window_bits]) return 0;
        return front[u];
    };
    uint32_t ch = uint32_t(warp);
    Word cw = load(ch);
    while (ch < kChunks) {  // uniform within the warp
        uint32_t nch = 0;
        if (lane == 0) nch = atomicAdd(&sh.next_chunk, 1u);
        nch = __shfl_sync(0xFFFFFFFFu, nch, 0);
        const Word nw = load(nch);
        const uint32_t u = ch * 32 + uint32_t(lane);
        uint32_t F = 0;  // the unit's frontier states
        if constexpr (MODE == kTwoBit) {
            const uint64_t hi = cw & kEven, lo = (cw >> 1) & kEven;
            const uint64_t cur = hi & (a.cur_code == 3 ? lo : ~lo);
            if (cur) {  // CUR -> OLD (code 1); only this block changes this window's CUR codes
                atomicXor(reinterpret_cast<unsigned long long*>(front) + u,
                          (unsigned long long)(cur | (a.cur_code == 2 ? (cur << 1) : 0)));
                F = gather_even(cur);
            }
        } else {
            F = cw;
            if (MODE == kClassic && F) front[u] = 0;  // BitArray::ScanBitsAndClear
        }
        const uint32_t cnt = __popc(F);
        found += cnt;
        // Flips of 2 and 3, all of the unit's at once; both stay in the window.
        if (F) {
            uint64_t pv, own, nx;
            flip3_push<32>(F, base / kPancakeUnit + u, pv, own, nx);
            own |= ((F & 0x55555555u) << 1) | ((F >> 1) & 0x55555555u);
            atomicOr(&smarks[u], uint32_t(own));
            if (pv) atomicOr(&smarks[u - 1], uint32_t(pv));
            if (nx) atomicOr(&smarks[u + 1], uint32_t(nx));
        }
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (total) {
            uint32_t at = incl - cnt;
            while (F) {
                const uint32_t j = __ffs(F) - 1;
                F &= F - 1;
                wlist[at++] = uint16_t(uint32_t(lane) * 32 + j);
            }
            const uint32_t coff = ch * kChunk;  // the chunk's first state in the window
            __syncwarp();
            for (uint32_t e = uint32_t(lane); e < total; e += 32) {
                const uint32_t o = coff + wlist[e];
                const uint32_t q = o / PZ::kBlock;
                em.parent_off = o;
                PZ::template expand_from_prefixed<2>(base + o, pref[q], o - q * PZ::kBlock, em);
            }
            __syncwarp();
        }
        cw = nw;
        ch = nch;
    }
    if (found) sh.any = 1;
    __syncthreads();

    uint32_t fresh = 0;
    if (sh.any) {
        if constexpr (MODE == kTwoBit) {
            unsigned long long* codes = reinterpret_cast<unsigned long long*>(front);
            const uint64_t lo = a.cur_code == 2 ? ~uint64_t(0) : 0;  // NEXT = 3: both bits
            for (uint32_t i0 = tid; i0 < kUnits; i0 += 4 * T) {  // four reads in flight
                uint32_t v[4];
                uint64_t w[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t i = i0 + q * T;
                    v[q] = i < kUnits ? smarks[i] : 0;
                    if (v[q]) w[q] = __ldcg(codes + i);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!v[q]) continue;
                    const uint32_t i = i0 + q * T;
                    const uint64_t m = spread_even(v[q]) & ~(w[q] | (w[q] >> 1));
                    if (!m) continue;
                    em.flag(base + uint64_t(i) * kPancakeUnit);
                    atomicOr(codes + i, (unsigned long long)(m | ((m << 1) & lo)));
                    fresh += __popcll(m);
                }
            }
        } else {
            unsigned long long* g = reinterpret_cast<unsigned long long*>(a.marks) + base / 64;
            for (uint32_t i = tid; i < W / 64; i += T) {
                const unsigned long long v = smem64[i];
                if (!v) continue;
                em.flag(base + uint64_t(i) * 64);
                atomicOr(g + i, v);
            }
        }
    }

    // Every parent has N - 1 children, those of flips up to 8 in the window and the
    // others long-range (in the far bitmap: those of flips up to 12, or all).
    const uint32_t c0 = __reduce_add_sync(0xFFFFFFFFu, found);
    const uint32_t c3 = __reduce_or_sync(0xFFFFFFFFu, em.bad);
    uint32_t c5 = 0;
    if constexpr (MODE == kTwoBit) c5 = __reduce_add_sync(0xFFFFFFFFu, em.marked + fresh);
    if (lane == 0) {
        if (c0) atomicAdd(&sh.cnt[0], (unsigned long long)c0);
        if (c3) atomicOr(&sh.cnt[3], 1ull);
        if (c5) atomicAdd(&sh.cnt[5], (unsigned long long)c5);
    }
    __syncthreads();  // the shared marks and lists may be reused for another window
    if (tid == 0 && sh.cnt[0]) {
        const unsigned long long n = sh.cnt[0];
        atomicAdd(&a.stats[0], n);
        atomicAdd(&a.stats[1], n * (N - 1));
        atomicAdd(&a.stats[2], n * (kPancakeK - 1));
        if (sh.cnt[3]) atomicOr(&a.stats[3], 1ull);
        if (MODE == kTwoBit && sh.cnt[5]) atomicAdd(&a.stats[5], sh.cnt[5]);
        const int in_far = (a.far_all || N < 12 ? N : 12) - kPancakeK;
        if (MODE == kTwoBit && a.far && in_far > 0) atomicAdd(&a.stats[6], n * in_far);
    }
}

// Blocks per SM: 64 to 73 registers per thread.
template <int T>
__host__ __device__ constexpr int pancake_blocks() { return T == 128 ? 7 : T == 256 ? 4 : 2; }

template <int N, int MODE, int T>
__global__ void __launch_bounds__(T, pancake_blocks<T>()) pancake_level_kernel(LevelArgs a) {
    extern __shared__ __align__(16) unsigned long long smem64[];
    __shared__ WindowShared sh;
    pancake_window<N, MODE, T>(a, blockIdx.x, smem64, sh);
}

template <int N, int MODE, int V = 0>
cudaError_t launch_pancake_level(const LevelArgs& a, unsigned grid, size_t smem, cudaStream_t s) {
    if (!a.own_windows) return launch_level<PancakeK<N>, MODE, false, V>(a, grid, smem, s);
    constexpr int T = variant_threads(V);
    constexpr size_t bytes = pancake_smem_bytes<N>(T);
    constexpr uint64_t windows = fact(N) / kPancakeWindow;
    static_assert(windows < (uint64_t(1) << 31), "grid");
    cudaError_t e = cudaFuncSetAttribute(pancake_level_kernel<N, MODE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(bytes));
    if (e != cudaSuccess) return e;
    pancake_level_kernel<N, MODE, T><<<unsigned(windows), T, bytes, s>>>(a);
    return cudaGetLastError();
}

}  // namespace psb
