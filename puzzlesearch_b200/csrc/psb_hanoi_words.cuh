// psb_hanoi_words.cuh -- level pass of 4-peg Hanoi without symmetry, 64
// states at a time.
//
// A unit is the 64 states that differ in the three smallest disks only; all
// of them share the disks above, U = index >> 6.  Whether a disk may move
// depends on the smaller disks alone, so every move of a whole unit is a mask
// and a fixed bit permutation:
//   * disks 0..2 move inside the unit: peg p -> p ^ x (x = 1, 2, 3) is an
//     exchange of fixed bit groups under a constant mask of the states where
//     no smaller disk sits on either peg;
//   * for each of the six peg pairs, the states whose three small disks sit
//     on the two other pegs (8 of the 64) move the smallest of the larger
//     disks on the pair, which is the same disk for the whole unit: the
//     masked word goes to unit U ^ (x << 2k).
// With g_1 = high bit, g_2 = low bit and g_3 = high ^ low of a disk's peg, a
// pair is {pegs with g_x == v}; x names the exchange, v the pair.
//
// The per-state kernel (level_window<HanoiK>) spent about 100 instructions on
// each state and was ALU-bound (76% of the ALU pipe, DRAM at 5%); a unit
// takes about 250 here whatever number of its states is in the frontier.
// Units holding frontier states are queued per warp and expanded 32 at a
// time, so sparse chunks do not leave lanes idle.  17 disks, two-bit, whole
// search on B200: 444 -> 102 ms; a dense level of 15 disks 757 -> 197 us, the
// ALU pipe at 53%, DRAM at 19%, an eighth of the stalls at window barriers.
//
// Marks of a unit are one 64-bit mask in shared memory (four for frontier
// search, one per operator) in the unit's bit order, which is the order its
// array words come apart in without packing:
//   1-bit arrays : bit = p0 + 4 p1 + 16 p2, the word itself
//   2-bit codes  : word 0 (p2 = 0, 1) at even bits, word 1 (p2 = 2, 3) at odd
//                  bits: bit 0 = p2 high, 1-2 = p0, 3-4 = p1, 5 = p2 low
//   4-bit arrays : word p2's nibble j at bit 4 j + p2: bits 0-1 = p2,
//                  2-3 = p0, 4-5 = p1
#pragma once

#include "psb_kernels.cuh"

namespace psb {

// Bit positions of the low and high peg bit of disk d (0..2) in a unit.
template <int MODE>
struct UnitOrder {
    __host__ __device__ static constexpr int lo(int d) {
        return MODE == kTwoBit ? 2 * d + 1 : MODE == kFrontier ? (2 * d + 2) % 6 : 2 * d;
    }
    __host__ __device__ static constexpr int hi(int d) {
        return MODE == kTwoBit ? (2 * d + 2) % 6 : MODE == kFrontier ? (2 * d + 3) % 6 : 2 * d + 1;
    }
};

// g_x of disk d at unit position pos.
template <int MODE>
__host__ __device__ constexpr int unit_g(int pos, int d, int x) {
    using O = UnitOrder<MODE>;
    const int l = (pos >> O::lo(d)) & 1, h = (pos >> O::hi(d)) & 1;
    return x == 1 ? h : x == 2 ? l : (h ^ l);
}
// Positions where disk d may move p -> p ^ x: every smaller disk is off the pair.
template <int MODE>
__host__ __device__ constexpr uint64_t unit_move_mask(int d, int x) {
    uint64_t m = 0;
    for (int pos = 0; pos < 64; ++pos) {
        bool ok = true;
        for (int s = 0; s < d; ++s) ok = ok && unit_g<MODE>(pos, s, x) != unit_g<MODE>(pos, d, x);
        if (ok) m |= uint64_t(1) << pos;
    }
    return m;
}
// Positions whose three disks are all off the pair (x, v).
template <int MODE>
__host__ __device__ constexpr uint64_t unit_free_mask(int x, int v) {
    uint64_t m = 0;
    for (int pos = 0; pos < 64; ++pos)
        if (unit_g<MODE>(pos, 0, x) != v && unit_g<MODE>(pos, 1, x) != v && unit_g<MODE>(pos, 2, x) != v)
            m |= uint64_t(1) << pos;
    return m;
}
// Positions with disk d on peg p.
template <int MODE>
__host__ __device__ constexpr uint64_t unit_peg_mask(int d, int p) {
    uint64_t m = 0;
    for (int pos = 0; pos < 64; ++pos)
        if (unit_g<MODE>(pos, d, 2) == (p & 1) && unit_g<MODE>(pos, d, 1) == (p >> 1)) m |= uint64_t(1) << pos;
    return m;
}

// Exchanges the positions that differ in bit B of their number.
template <int B>
__device__ __forceinline__ uint64_t unit_swap(uint64_t v) {
    const uint32_t l = uint32_t(v), h = uint32_t(v >> 32);
    if constexpr (B == 5) {
        return (uint64_t(l) << 32) | h;
    } else if constexpr (B >= 3) {
        constexpr uint32_t sel = B == 4 ? 0x1032 : 0x2301;
        return (uint64_t(__byte_perm(h, 0, sel)) << 32) | __byte_perm(l, 0, sel);
    } else {
        constexpr uint32_t m = B == 0 ? 0x55555555u : B == 1 ? 0x33333333u : 0x0F0F0F0Fu;
        auto half = [](uint32_t w) -> uint32_t { return ((w & m) << (1 << B)) | ((w >> (1 << B)) & m); };
        return (uint64_t(half(h)) << 32) | half(l);
    }
}

// Children of A by moves of disk D inside the unit (x = 1: low peg bit
// flips, 2: high, 3: both).
template <int MODE, int D>
__device__ __forceinline__ uint64_t unit_moves(uint64_t A) {
    using O = UnitOrder<MODE>;
    constexpr uint64_t m1 = unit_move_mask<MODE>(D, 1), m2 = unit_move_mask<MODE>(D, 2),
                       m3 = unit_move_mask<MODE>(D, 3);
    return unit_swap<O::lo(D)>((A & m1) | unit_swap<O::hi(D)>(A & m3)) | unit_swap<O::hi(D)>(A & m2);
}

// The search's disks this pass takes: three in the unit, the others' pegs in
// 32 bits of unit number.
__host__ __device__ constexpr bool hanoi_words_ok(const PuzzleArgs& p) {
    return p.sym == 0 && p.disks >= 3 && p.disks <= 19;
}

// Chunks of 32 units that a warp sweeps at a time.
__host__ __device__ constexpr int hanoi_group(int mode) { return mode == kFrontier ? 2 : 4; }
// Shared memory of a window pass: the marks, then each warp's queue of units
// (mask and unit number; at most 31 and a whole group wait).
__host__ __device__ constexpr uint32_t hanoi_queue(int mode) { return 32u * (1 + hanoi_group(mode)); }
__host__ __device__ constexpr size_t hanoi_queue_bytes(int mode) {
    return hanoi_queue(mode) * (8 * (mode == kFrontier ? 4 : 1) + 2);
}
__host__ __device__ constexpr size_t hanoi_smem_bytes(int mode, size_t window_states, int threads) {
    return mark_bytes(mode, window_states) + size_t(threads / 32) * hanoi_queue_bytes(mode);
}

// A thread's share of the level's counters (LevelArgs::stats).
struct HanoiCounts {
    uint32_t found = 0, children = 0, remote = 0, next = 0, farmarks = 0;
};

// Clears the marks before a block's first window; hanoi_window leaves them
// clear for the next.
template <int MODE, int KTHREADS>
__device__ __forceinline__ void hanoi_begin(const LevelArgs& a, unsigned long long* smem64, WindowShared& sh) {
    const uint32_t mbytes = uint32_t(mark_bytes(MODE, size_t(1) << a.window_bits));
    for (uint32_t i = threadIdx.x; i < mbytes / 16; i += KTHREADS)
        reinterpret_cast<uint4*>(smem64)[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) {
        sh.next_chunk = KTHREADS / 32;  // warp w's first group is group w
        for (int i = 0; i < 8; ++i) sh.cnt[i] = 0;
    }
    __syncthreads();
}

// Adds the block's counters to the level's: one global atomic per block and counter.
template <int MODE>
__device__ __forceinline__ void hanoi_end(const LevelArgs& a, const HanoiCounts& c, WindowShared& sh) {
    // signed: a unit's states are counted by the lane that sweeps it, its
    // missing moves and remote children by the lane that expands it
    const int32_t children = int32_t(c.children + (MODE != kFrontier ? 6 * c.found : 0));
    const int32_t v[5] = {int32_t(c.found), children, children - int32_t(c.remote), int32_t(c.next),
                          int32_t(c.farmarks)};
    constexpr int kCounters = MODE == kTwoBit ? 5 : 3;
#pragma unroll
    for (int i = 0; i < kCounters; ++i) {
        long long t = v[i];  // a block's windows can hold more than 2^32 children
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
        if ((threadIdx.x & 31) == 0 && t) atomicAdd(&sh.cnt[i < 3 ? i : i + 2], (unsigned long long)t);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < 8; ++i)
            if (sh.cnt[i]) atomicAdd(&a.stats[i], sh.cnt[i]);
    }
}

// One window of a top-down level: level_window's contract between
// hanoi_begin and hanoi_end, for searches with hanoi_words_ok and a window
// that exists and is flagged (the caller looks).
template <int MODE, int KTHREADS>
__device__ __forceinline__ void hanoi_window(const LevelArgs& a, uint64_t window, unsigned long long* smem64,
                                             WindowShared& sh, HanoiCounts& cnt) {
    constexpr int kWarps = KTHREADS / 32;
    constexpr int kPlanes = MODE == kFrontier ? 4 : 1;
    constexpr uint32_t kQueue = hanoi_queue(MODE);
    constexpr size_t kWarpBytes = hanoi_queue_bytes(MODE);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t W = 1u << a.window_bits;
    const uint64_t base = window << a.window_bits;
    const uint64_t remaining = a.n_states - base;  // both multiples of 64
    const uint32_t units = (remaining < W ? uint32_t(remaining) : W) / 64;
    const uint32_t chunks = (units + 31) / 32;
    const uint32_t mbytes = uint32_t(mark_bytes(MODE, W));
    uint32_t* smarks = reinterpret_cast<uint32_t*>(smem64);
    uint64_t* qmask = reinterpret_cast<uint64_t*>(reinterpret_cast<char*>(smem64) + mbytes + warp * kWarpBytes);
    uint16_t* qunit = reinterpret_cast<uint16_t*>(qmask + kQueue * kPlanes);
    const uint32_t U0 = uint32_t(base >> 6);  // the window's first unit
    const uint32_t E = a.pz.disks == 19 ? 0x55555555u : 0x55555555u & ((1u << (2 * (a.pz.disks - 3))) - 1u);

    uint32_t found = 0, children = 0, remote = 0, marked = 0, farmarks = 0;
    const uint32_t next_pat = 1u | (a.cur_code == 2 ? 2u : 0u);

    auto flag_window = [&](uint32_t unit) {
        if (!a.wflag_next) return;
        uint8_t* f = a.wflag_next + (unit >> (a.window_bits - 6));
        if (!*f) *f = 1;
    };
    auto mark_local = [&](uint32_t word, uint64_t m) {  // word: 64-bit mark word in the window
        if (uint32_t(m)) atomicOr(&smarks[2 * word], uint32_t(m));
        if (uint32_t(m >> 32)) atomicOr(&smarks[2 * word + 1], uint32_t(m >> 32));
    };
    // Marks the states m of unit T outside the window (plane: operator).
    auto mark_remote = [&](uint32_t T, uint64_t m, uint32_t plane) {
        remote += __popcll(m);
        if constexpr (MODE == kTwoBit) {
            unsigned long long* codes = reinterpret_cast<unsigned long long*>(a.marks) + 2ull * T;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint64_t s = (m >> h) & kEven;
                if (!s) continue;
                if (a.far) {  // long-range bitmap, folded into the codes after the level
                    flag_window(T);
                    farmarks += __popcll(s);
                    atomicOr(a.far + 2ull * T + h, gather_even(s));
                    continue;
                }
                const uint64_t w = __ldcg(codes + h);
                s &= ~(w | (w >> 1));  // UNVISITED -> NEXT
                if (s) {
                    flag_window(T);
                    atomicOr(codes + h, (unsigned long long)(s | ((next_pat & 2u) ? (s << 1) : 0)));
                    marked += __popcll(s);
                }
            }
        } else if constexpr (MODE == kFrontier) {
            flag_window(T);
            unsigned long long* g = reinterpret_cast<unsigned long long*>(a.marks) + 4ull * T;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const uint64_t s = (m >> w) & 0x1111111111111111ull;
                if (s) atomicOr(g + w, (unsigned long long)(s << plane));
            }
        } else {
            flag_window(T);
            atomicOr(reinterpret_cast<unsigned long long*>(a.marks) + T, (unsigned long long)m);
        }
    };

    // Expands one queued unit: its frontier states (F), and for frontier
    // search the used operators (used[p]: states whose moves from peg p are skipped).
    auto expand = [&](uint32_t u, uint64_t F, const uint64_t (&used)[kPlanes]) {
        const uint32_t U = U0 + u;
        // moves inside the unit
        if constexpr (MODE == kFrontier) {
            uint64_t out[4] = {0, 0, 0, 0};
            auto low = [&](auto disk) {
                constexpr int D = decltype(disk)::value;
                uint64_t A = F;
#pragma unroll
                for (int p = 0; p < 4; ++p) A &= ~(used[p] & unit_peg_mask<MODE>(D, p));
                const uint64_t y = unit_moves<MODE, D>(A);
#pragma unroll
                for (int p = 0; p < 4; ++p) out[p] |= y & unit_peg_mask<MODE>(D, p);
#pragma unroll
                for (int x = 1; x < 4; ++x) children += __popcll(A & unit_move_mask<MODE>(D, x));
            };
            low(std::integral_constant<int, 0>{});
            low(std::integral_constant<int, 1>{});
            low(std::integral_constant<int, 2>{});
#pragma unroll
            for (int p = 0; p < 4; ++p) mark_local(4 * u + p, out[p]);
        } else {
            mark_local(u, unit_moves<MODE, 0>(F) | unit_moves<MODE, 1>(F) | unit_moves<MODE, 2>(F));
            // children: 6 per state, less the pairs with both pegs empty (below)
        }
        // Larger disks, one per peg pair (x, v): the states S of the unit that
        // move one, to unit T (frontier search: as operator `plane`).
        auto pair = [&](uint32_t x, uint32_t v, uint64_t& S, uint32_t& T, uint32_t& plane) {
            const uint32_t g = x == 1 ? U >> 1 : x == 2 ? U : U ^ (U >> 1);
            const uint32_t e = (v ? g : ~g) & E;  // larger disks on the pair
            const uint32_t k = e & (0u - e);      // the smallest of them
            if (!k) {  // both pegs empty: no move
                if constexpr (MODE != kFrontier) children -= __popcll(S);
                S = 0;
            }
            if constexpr (MODE == kFrontier) {
                // its peg: g_x == v, and the other peg of the pair is peg ^ x
                const uint32_t src = ((U & k) ? 1u : 0u) | (((U >> 1) & k) ? 2u : 0u);
                S &= ~(src == 0 ? used[0] : src == 1 ? used[1] : src == 2 ? used[2] : used[3]);
                plane = src ^ x;
            }
            T = U ^ (k * x);
        };
        uint32_t far_pairs = 0;
#pragma unroll
        for (uint32_t i = 0; i < 6; ++i) {
            uint64_t S = F & unit_free_mask<MODE>(1 + int(i >> 1), int(i & 1));
            if (!S) continue;
            uint32_t T, plane = 0;
            pair(1 + (i >> 1), i & 1, S, T, plane);
            if (!S) continue;
            if constexpr (MODE == kFrontier) children += __popcll(S);
            const uint32_t t = T - U0;
            if (t < units) mark_local(MODE == kFrontier ? 4 * t + plane : t, S);
            else far_pairs |= 1u << i;
        }
        // Moves that leave the window (under 1%), worked out again here: one
        // copy of the long-range code instead of six.
        while (far_pairs) {
            const uint32_t i = __ffs(far_pairs) - 1;
            far_pairs &= far_pairs - 1;
            uint64_t S = F;
#pragma unroll
            for (uint32_t j = 0; j < 6; ++j)
                if (j == i) S &= unit_free_mask<MODE>(1 + int(j >> 1), int(j & 1));
            uint32_t T, plane = 0;
            pair(1 + (i >> 1), i & 1, S, T, plane);
            mark_remote(T, S, plane);
        }
    };
    auto expand_queued = [&](uint32_t i) {
        uint64_t F = 0, used[kPlanes];
#pragma unroll
        for (int p = 0; p < kPlanes; ++p) {
            used[p] = qmask[i * kPlanes + p];
            F |= used[p];
        }
        expand(qunit[i], F, used);
    };

    constexpr int kWords = MODE == kTwoBit ? 2 : MODE == kFrontier ? 4 : 1;  // array words per unit
    // A warp sweeps groups of kGroup chunks (32 units each), all of whose
    // words it loads at once; groups come from a shared counter.
    constexpr int kGroup = hanoi_group(MODE);
    uint32_t grp = uint32_t(warp), queued = 0;
    for (bool more = grp * kGroup < chunks; more;) {  // uniform within the warp
        uint64_t cw[kGroup][kWords];
#pragma unroll
        for (int c = 0; c < kGroup; ++c) {
            const uint32_t u = (grp * kGroup + c) * 32 + uint32_t(lane);
#pragma unroll
            for (int q = 0; q < kWords; ++q) cw[c][q] = 0;
            if (u >= units) continue;
            const uint64_t* p = a.front + uint64_t(U0 + u) * kWords;
            if constexpr (kWords == 1) {
                cw[c][0] = *p;
            } else {
#pragma unroll
                for (int q = 0; q < kWords; q += 2) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + q);
                    cw[c][q] = v.x;
                    cw[c][q + 1] = v.y;
                }
            }
        }
        uint32_t next = 0;
        if (lane == 0) next = atomicAdd(&sh.next_chunk, 1u);
#pragma unroll
        for (int c = 0; c < kGroup; ++c) {
            const uint32_t u = (grp * kGroup + c) * 32 + uint32_t(lane);
            uint64_t F[kPlanes] = {};
            if constexpr (MODE == kTwoBit) {
                const uint64_t flip = a.cur_code == 3 ? 0 : ~uint64_t(0);
                const uint64_t c0 = cw[c][0] & ((cw[c][0] >> 1) ^ flip) & kEven;
                const uint64_t c1 = cw[c][1] & ((cw[c][1] >> 1) ^ flip) & kEven;
                F[0] = c0 | (c1 << 1);
            } else {
                F[0] = cw[c][0];
                if constexpr (MODE == kFrontier) F[0] |= cw[c][1] | cw[c][2] | cw[c][3];
            }
            if (!__any_sync(0xFFFFFFFFu, F[0] != 0)) continue;  // nothing in these 32 units
            if (F[0]) {
                if constexpr (MODE == kTwoBit) {
                    // CUR -> OLD (code 1); only this block changes this window's CUR codes
                    unsigned long long* g = reinterpret_cast<unsigned long long*>(a.front) + 2ull * (U0 + u);
                    const uint64_t c0 = F[0] & kEven, c1 = (F[0] >> 1) & kEven;
                    if (c0) atomicXor(g, (unsigned long long)(c0 | (a.cur_code == 2 ? (c0 << 1) : 0)));
                    if (c1) atomicXor(g + 1, (unsigned long long)(c1 | (a.cur_code == 2 ? (c1 << 1) : 0)));
                } else if constexpr (MODE == kClassic) {
                    a.front[U0 + u] = 0;  // BitArray::ScanBitsAndClear
                } else if constexpr (MODE == kFrontier) {
                    uint64_t keep = 0;  // in index order
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (cw[c][q]) a.front[4ull * (U0 + u) + q] = 0;  // FourBitArray::ScanAndClear
                        keep |= uint64_t(nibble_flags(cw[c][q])) << (16 * q);
                    }
                    if (a.odd) {
                        keep &= ~a.excl_cur[U0 + u];
                        if (keep) a.excl_next[U0 + u] = keep;  // excl_next is clear before the level
                    }
                    found += __popcll(keep);
#pragma unroll
                    for (int p = 0; p < kPlanes; ++p) F[p] = 0;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        // nibbles of the kept states of word q
                        uint64_t k = (keep >> (16 * q)) & 0xFFFFull;
                        k = (k | (k << 24)) & 0x000000FF000000FFull;
                        k = (k | (k << 12)) & 0x000F000F000F000Full;
                        k = (k | (k << 6)) & 0x0303030303030303ull;
                        k = (k | (k << 3)) & 0x1111111111111111ull;
#pragma unroll
                        for (int p = 0; p < kPlanes; ++p) F[p] |= ((cw[c][q] >> p) & k) << q;
                    }
                }
                if constexpr (MODE != kFrontier) found += __popcll(F[0]);
            }
            uint64_t any = F[0];
#pragma unroll
            for (int p = 1; p < kPlanes; ++p) any |= F[p];
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, any != 0);
            if (any) {
                const uint32_t at = queued + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
                for (int p = 0; p < kPlanes; ++p) qmask[at * kPlanes + p] = F[p];
                qunit[at] = uint16_t(u);
            }
            queued += __popc(bal);
        }
        grp = __shfl_sync(0xFFFFFFFFu, next, 0);
        more = grp * kGroup < chunks;
        __syncwarp();
        // 32 units at a time; after the last group what is left.  The one
        // place that expands: inlined twice it outgrows the instruction cache
        // (17 disks two-bit: 250 ms with four copies, 140 ms with two).
        while (queued >= (more ? 32u : 1u)) {
            const uint32_t n = queued < 32 ? queued : 32u;
            queued -= n;
            if (uint32_t(lane) < n) expand_queued(queued + uint32_t(lane));
        }
        __syncwarp();
    }
    const bool any = __syncthreads_or(found != 0);
    if (tid == 0) sh.next_chunk = kWarps;
    uint32_t fresh = 0;
    if (any) {  // flush the marks and clear them
        if (a.wflag_next && tid == 0) a.wflag_next[window] = 1;
        if constexpr (MODE == kTwoBit) {
            // The codes were read by the sweep and mostly still sit in L1.  A
            // stale word only lacks NEXT codes that other blocks set since,
            // and setting those again changes nothing (`fresh` is an upper
            // estimate).  Four units a turn keep four reads in flight.
            ulonglong2* codes = reinterpret_cast<ulonglong2*>(a.marks) + U0;
            for (uint32_t u0 = tid; u0 < units; u0 += 4 * KTHREADS) {
                uint64_t v[4];
                ulonglong2 w[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t u = u0 + q * KTHREADS;
                    v[q] = u < units ? smem64[u] : 0;
                    if (v[q]) {
                        w[q] = codes[u];
                        smem64[u] = 0;
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!v[q]) continue;
                    unsigned long long* c = reinterpret_cast<unsigned long long*>(codes + u0 + q * KTHREADS);
                    const uint64_t m0 = v[q] & ~(w[q].x | (w[q].x >> 1)) & kEven;
                    const uint64_t m1 = (v[q] >> 1) & ~(w[q].y | (w[q].y >> 1)) & kEven;
                    if (m0) atomicOr(c, (unsigned long long)(m0 | ((next_pat & 2u) ? (m0 << 1) : 0)));
                    if (m1) atomicOr(c + 1, (unsigned long long)(m1 | ((next_pat & 2u) ? (m1 << 1) : 0)));
                    fresh += __popcll(m0 | (m1 << 1));
                }
            }
        }
        for (uint32_t u = tid; MODE != kTwoBit && u < units; u += KTHREADS) {
            if constexpr (MODE == kFrontier) {
                uint64_t v[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) v[p] = smem64[4 * u + p];
                if (!(v[0] | v[1] | v[2] | v[3])) continue;
#pragma unroll
                for (int p = 0; p < 4; ++p) smem64[4 * u + p] = 0;
                unsigned long long* g = reinterpret_cast<unsigned long long*>(a.marks) + 4ull * (U0 + u);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint64_t w = 0;
#pragma unroll
                    for (int p = 0; p < 4; ++p) w |= ((v[p] >> q) & 0x1111111111111111ull) << p;
                    if (w) atomicOr(g + q, (unsigned long long)w);
                }
            } else {
                const unsigned long long v = smem64[u];
                if (!v) continue;
                smem64[u] = 0;
                atomicOr(reinterpret_cast<unsigned long long*>(a.marks) + U0 + u, v);
            }
        }
    }

    __syncthreads();  // the marks are clear and the queues free
    cnt.found += found;
    cnt.children += children;
    cnt.remote += remote;
    cnt.next += marked + fresh;
    cnt.farmarks += farmarks;
}

}  // namespace psb
