// psb_small.cuh -- a whole search (two-bit, three-bit or classic) of a small
// puzzle in one launch.
//
// A level of a small search (3x3 board: at most 24,047 states) is a few
// microseconds of work, and launching it, clearing its counters, reading them
// back and waiting cost 28 us on the host, level after level.  Here one
// cluster of 16 blocks runs all levels.  Each block owns a sixteenth of the
// states as three bitmaps in its shared memory (visited, frontier, marks);
// children are marked in their owner's shared memory, the cluster's hardware
// barrier separates the levels, and every block takes psb_bfs's decisions
// (direction, end of the search) from counts the blocks exchange.  Global
// memory sees the final codes and the counts only.  B200, whole calls: 3x3 board
// 950 -> 232 us (32 levels, 6 us each), 8 pancakes 342 -> 96 us, 8-disk Hanoi
// 922 -> 149 us.
#pragma once

#include <cooperative_groups.h>

#include "psb_hanoi_words.cuh"
#include "psb_kernels.cuh"

namespace psb {

// One block's share of a level's counters, written into every block.
struct SmallCounts {
    unsigned long long next, children, local, bad;
};

// Children of the frontier: marked in their owner's bitmap.
struct SmallMarker {
    uint32_t* marks;  // this block's
    uint64_t n_states;
    uint32_t rank;
    int bits;
    uint32_t children = 0, local = 0, bad = 0;
    __device__ __forceinline__ void operator()(uint64_t c, uint32_t) {
        if (c >= n_states) { bad = 1; return; }  // never expected: keeps a bad index off the memory system
        ++children;
        const uint32_t owner = uint32_t(c >> bits), o = uint32_t(c) & ((1u << bits) - 1u);
        uint32_t* word = marks + (o >> 5);
        if (owner == rank) ++local;
        else word = cooperative_groups::this_cluster().map_shared_rank(word, owner);
        atomicOr(word, 1u << (o & 31u));
    }
};

// Hanoi without symmetry, 64 states at a time (psb_hanoi_words.cuh): the
// children of frontier states F of the block's unit u.  An 8-disk search took
// 306 us state by state: the warps whose 32 words hold most of a level's states
// expanded them alone; 149 us.
__device__ __forceinline__ void small_hanoi_unit(SmallMarker& em, const PuzzleArgs& pz, uint32_t u, uint64_t F) {
    const uint32_t U = (em.rank << (em.bits - 6)) + u;
    const uint32_t E = 0x55555555u & ((1u << (2 * (pz.disks - 3))) - 1u);  // a small search has few disks
    auto mark = [&](uint32_t T, uint64_t m) {
        const uint32_t owner = T >> (em.bits - 6);
        uint32_t* word = em.marks + 2 * (T & ((1u << (em.bits - 6)) - 1u));
        if (owner != em.rank) word = cooperative_groups::this_cluster().map_shared_rank(word, owner);
        if (uint32_t(m)) atomicOr(word, uint32_t(m));
        if (uint32_t(m >> 32)) atomicOr(word + 1, uint32_t(m >> 32));
    };
    mark(U, unit_moves<kThreeBit, 0>(F) | unit_moves<kThreeBit, 1>(F) | unit_moves<kThreeBit, 2>(F));
    uint32_t none = 0, elsewhere = 0;  // pairs with both pegs empty; children in other blocks
#pragma unroll
    for (uint32_t i = 0; i < 6; ++i) {
        const uint32_t x = 1 + (i >> 1), v = i & 1;
        const uint64_t S = F & unit_free_mask<kThreeBit>(int(x), int(v));
        if (!S) continue;
        const uint32_t g = x == 1 ? U >> 1 : x == 2 ? U : U ^ (U >> 1);
        const uint32_t e = (v ? g : ~g) & E, k = e & (0u - e);
        const uint32_t c = __popcll(S);
        if (!k) {
            none += c;
            continue;
        }
        const uint32_t T = U ^ (k * x);
        if (T >> (em.bits - 6) != em.rank) elsewhere += c;
        mark(T, S);
    }
    const uint32_t children = 6 * __popcll(F) - none;
    em.children += children;
    em.local += children - elsewhere;
}

// Neighbours of an unvisited state: is one of them in the frontier?
struct SmallProbe {
    uint32_t* front;  // this block's
    uint64_t n_states;
    uint32_t rank;
    int bits;
    uint32_t probes = 0, hit = 0, bad = 0;
    __device__ __forceinline__ void operator()(uint64_t c, uint32_t) {
        if (c >= n_states) { bad = 1; return; }
        ++probes;
        const uint32_t owner = uint32_t(c >> bits), o = uint32_t(c) & ((1u << bits) - 1u);
        uint32_t* word = front + (o >> 5);
        if (owner != rank) word = cooperative_groups::this_cluster().map_shared_rank(word, owner);
        hit |= (*word >> (o & 31u)) & 1u;
    }
};

template <class PZ>
__global__ void __launch_bounds__(kSmallThreads, 1) small_search_kernel(SmallArgs a) {
    extern __shared__ __align__(16) uint32_t small_mem[];
    __shared__ SmallCounts parts[2][kSmallBlocks];  // of levels l and l + 1
    __shared__ unsigned long long own[4];
    constexpr int T = kSmallThreads;
    auto cluster = cooperative_groups::this_cluster();
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t units = 1u << (a.bits - 5);  // 32 states each
    uint32_t *visited = small_mem, *front = visited + units, *marks = front + units;
    // Three-bit's final arrays hold the last two depths.
    const bool keep = a.mode == kThreeBit && a.arrays[0];
    uint32_t *prev = marks + units, *before = prev + (keep ? units : 0);
    uint16_t* list = reinterpret_cast<uint16_t*>(before + (keep ? units : 0)) + warp * 1024;
    const uint64_t n = a.n_states, base = uint64_t(rank) << a.bits;

    for (uint32_t u = tid; u < (keep ? 5 : 3) * units; u += T) small_mem[u] = 0;
    if (tid < 4) own[tid] = 0;
    __syncthreads();
    if (tid == 0 && (a.initial >> a.bits) == rank) {
        const uint32_t o = uint32_t(a.initial - base);
        visited[o >> 5] = front[o >> 5] = 1u << (o & 31u);
    }
    cluster.sync();

    uint32_t level = 0, status = 0, bu_levels = 0;
    uint64_t seen = 0, frontier = 1, expanded = 0, children = 0, local = 0;
    while (level < a.max_levels) {
        if (level >= kSmallDepths) { status = 2; break; }
        const uint64_t unvisited = n - (seen + frontier < n ? seen + frontier : n);
        const bool bu = a.can_bu && (a.direction == kSmallBottomUp ||
                                     (a.direction == 0 && frontier >= n / 64 && double(unvisited) < a.ratio * double(frontier)));
        SmallMarker mark{marks, n, rank, a.bits};
        SmallProbe probe{front, n, rank, a.bits};
        bool by_unit = false;
        if constexpr (PZ::kSymMult) {
            by_unit = !bu && hanoi_words_ok(a.pz);
            for (uint32_t u = tid; by_unit && u < units / 2; u += T) {
                const uint64_t F = front[2 * u] | (uint64_t(front[2 * u + 1]) << 32);
                if (F) small_hanoi_unit(mark, a.pz, u, F);
            }
        }
        // A warp lists the states of 32 words and expands them 32 at a time.
        for (uint32_t u0 = warp * 32; !by_unit && u0 < units; u0 += T) {
            const uint32_t u = u0 + lane;
            uint32_t m = bu ? ~visited[u] : front[u];
            if (bu) {  // states below n_states only
                const uint64_t first = base + 32ull * u;
                if (first + 32 > n) m &= first < n ? (1u << uint32_t(n - first)) - 1u : 0u;
            }
            uint32_t incl = __popc(m);
            const uint32_t c = incl;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= uint32_t(o)) incl += y;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            uint32_t at = incl - c;
            while (m) {
                list[at++] = uint16_t(lane * 32 + __ffs(m) - 1);
                m &= m - 1;
            }
            __syncwarp();
            for (uint32_t e = lane; e < total; e += 32) {
                const uint32_t o = u0 * 32 + list[e];
                if (bu) {
                    probe.hit = 0;
                    PZ::template expand<false>(base + o, 0u, a.pz, probe);
                    if (probe.hit) atomicOr(&marks[o >> 5], 1u << (o & 31u));
                } else {
                    PZ::template expand<false>(base + o, 0u, a.pz, mark);
                }
            }
            __syncwarp();
        }
        cluster.sync();  // every mark is made, every probe has read
        // The marked states not visited yet are the next frontier.
        uint32_t found = 0;
        for (uint32_t u = tid; u < units; u += T) {
            const uint32_t v = visited[u], f = marks[u] & ~v;
            if (marks[u]) marks[u] = 0;
            if (keep) {
                before[u] = prev[u];
                prev[u] = front[u];
            }
            front[u] = f;
            if (f) visited[u] = v | f;
            found += __popc(f);
        }
        const uint32_t sum[4] = {found, bu ? probe.probes : mark.children, bu ? 0u : mark.local,
                                 bu ? probe.bad : mark.bad};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t t = __reduce_add_sync(0xFFFFFFFFu, sum[i]);
            if (lane == 0 && t) atomicAdd(&own[i], (unsigned long long)t);
        }
        __syncthreads();
        // Into every block: thread i writes block i's copy.
        if (tid < kSmallBlocks)
            *cluster.map_shared_rank(&parts[level & 1][rank], tid) = SmallCounts{own[0], own[1], own[2], own[3]};
        cluster.sync();
        if (tid < 4) own[tid] = 0;
        SmallCounts all{0, 0, 0, 0};
        for (int i = 0; i < kSmallBlocks; ++i) {
            const SmallCounts& p = parts[level & 1][i];
            all.next += p.next;
            all.children += p.children;
            all.local += bu ? p.next : p.local;
            all.bad += p.bad;
        }
        if (rank == 0 && tid == 0) {
            a.out[kSmallHeader + 2 * level] = frontier;
            a.out[kSmallHeader + 2 * level + 1] = all.children;
        }
        expanded += bu ? unvisited : frontier;
        children += all.children;
        local += all.local;
        bu_levels += bu ? 1 : 0;
        if (all.bad) { status = 1; break; }
        ++level;
        seen += frontier;
        frontier = all.next;
        if (frontier == 0) break;
    }
    if (rank == 0 && tid == 0) {
        const uint64_t head[kSmallHeader] = {status, level, bu_levels, expanded, children, local, frontier};
        for (int i = 0; i < kSmallHeader; ++i) a.out[i] = head[i];
    }
    // The arrays as the level-by-level search leaves them.
    for (uint32_t u = tid; a.arrays[0] && u < units; u += T) {
        const uint64_t w = (base >> 5) + u;
        if (w >= a.units) break;
        uint32_t* const one[3] = {reinterpret_cast<uint32_t*>(a.arrays[0]), reinterpret_cast<uint32_t*>(a.arrays[1]),
                                  reinterpret_cast<uint32_t*>(a.arrays[2])};
        if (a.mode == kTwoBit) {
            // Codes: visited states OLD (1), the depth that no level expanded
            // CUR, 2 at even depths and 3 at odd ones (bit 2i = code / 2, bit 2i + 1 = code % 2).
            const uint64_t f = spread_even(front[u]), old = spread_even(visited[u] & ~front[u]);
            a.arrays[0][w] = f | ((old | ((level & 1) ? f : 0)) << 1);
        } else if (a.mode == kThreeBit) {  // old, cur: the last two depths; new: empty
            one[0][w] = frontier ? prev[u] : before[u];
            one[1][w] = frontier ? front[u] : prev[u];
            one[2][w] = 0;
        } else {  // closed, open: the depth that no level expanded, newOpen: empty
            one[0][w] = visited[u];
            one[1][w] = front[u];
            one[2][w] = 0;
        }
    }
    cluster.sync();  // no block leaves while others may still reach into it
}

// Dynamic shared memory of a block: its bitmaps and its warps' lists.
__host__ __device__ constexpr size_t small_smem_bytes(size_t bitmaps, int bits) {
    return bitmaps * (size_t(1) << bits) / 8 + kSmallThreads / 32 * 1024 * 2;
}

// The kernel's limit is the largest use, whatever this search takes: set to
// each call's size, a smaller search on another thread could lower it between
// this one's setting it and its launch.
template <class PZ>
cudaError_t launch_small_search(const SmallArgs& a, cudaStream_t s) {
    const size_t smem = small_smem_bytes(a.mode == kThreeBit && a.arrays[0] ? 5 : 3, a.bits);
    constexpr size_t limit = small_smem_bytes(5, kSmallBitsMax);
    cudaError_t e = cudaFuncSetAttribute(small_search_kernel<PZ>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(small_search_kernel<PZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(limit));
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kSmallBlocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kSmallBlocks);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, small_search_kernel<PZ>, a);
}

}  // namespace psb
