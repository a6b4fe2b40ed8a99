// psb_puzzles.cuh -- device-side state codecs and expanders for the three
// puzzles of the reference (lightln2/PuzzleSearch), in the index spaces of its
// *Simple classes, so that every index, child and operator code is identical
// to the reference's CPU path.
//
//   sliding tile : Puzzles/SlidingTilePuzzleSimple.cpp  (n! permutation index)
//   pancake      : Puzzles/PancakeSimple.cpp            (n! permutation index, suffix reversal)
//   4-peg Hanoi  : Puzzles/FourPegHanoiSimple.cpp       (2 bits per disk)
//
// Permutation index (Puzzles/PermutationMap.cpp:39-58): position 0 is the
// most significant digit; digit i equals the number of later values smaller
// than the value at i; index = sum_i d_i * (n-1-i)!.  Everything is
// templated on n so all radices and factorial weights are compile-time
// constants: divisions become multiply-high sequences and the value arrays
// stay in registers.
#pragma once

#include <cstdint>
#include <type_traits>

namespace psb {

constexpr uint64_t kInvalidIndex = ~uint64_t(0);  // Common/Puzzle.h:19

// Emitters with a member rel(parent, delta, op) take a child given as its
// parent's index plus a signed 32-bit delta (see Pancake); others get the
// child's index.
template <class E, class = void>
struct EmitRel : std::false_type {};
template <class E>
struct EmitRel<E, decltype(void(&E::rel))> : std::true_type {};

// Emitters with a member far(child, op) take children that can land anywhere
// in a large index space (pancake flips of more than 12) there, so they can
// mark them without displacing cached data that nearer children reuse.
template <class E, class = void>
struct EmitFar : std::false_type {};
template <class E>
struct EmitFar<E, decltype(void(&E::far))> : std::true_type {};

// Emitters with members far_issue(child, op) and far_finish(child, op, ticket)
// take the far children in two steps: the first starts whatever the mark
// has to read and returns a ticket, the second completes the mark.  The
// expander issues the far children first and finishes them after the near
// ones, so the reads overlap the near children's arithmetic.
template <class E, class = void>
struct EmitSplitFar : std::false_type {};
template <class E>
struct EmitSplitFar<E, decltype(void(&E::far_issue))> : std::true_type {};

struct FarTicket {
    uint64_t word;  // the target's code word, when `pending`
    bool pending;
};

// k!, 0 <= k <= 16.  A chain of selects, which the compiler folds for every
// constant k of an unrolled loop.  Written as a recursion it was left as a
// loop of 64-bit multiplications at run time in the rank sums, over half of
// their instructions: 13-pancake two-bit 208 -> 154 ms on B200, its bottom-up
// depth 12 57 -> 27 ms.
__host__ __device__ constexpr uint64_t fact(int k) {
    return k <= 1    ? 1ull
           : k == 2  ? 2ull
           : k == 3  ? 6ull
           : k == 4  ? 24ull
           : k == 5  ? 120ull
           : k == 6  ? 720ull
           : k == 7  ? 5040ull
           : k == 8  ? 40320ull
           : k == 9  ? 362880ull
           : k == 10 ? 3628800ull
           : k == 11 ? 39916800ull
           : k == 12 ? 479001600ull
           : k == 13 ? 6227020800ull
           : k == 14 ? 87178291200ull
           : k == 15 ? 1307674368000ull
                     : 20922789888000ull;
}
constexpr uint32_t kF12 = 479001600u;  // 12!

// Lehmer digits of a permutation index below 2^32.
template <int N>
__device__ __forceinline__ void perm_digits(uint32_t index, uint32_t (&d)[N]) {
#pragma unroll
    for (int i = N - 1; i >= 0; --i) {
        d[i] = index % uint32_t(N - i);
        index /= uint32_t(N - i);
    }
}

// PermutationUncompact (PermutationMap.cpp:21-37): digit k picks the k-th
// unused value from a nibble list.
template <int N>
__device__ __forceinline__ void perm_values(const uint32_t (&d)[N], uint32_t (&v)[N]) {
    uint64_t tiles = 0xFEDCBA9876543210ull;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t s = 4u * d[i];
        v[i] = uint32_t(tiles >> s) & 15u;
        const uint64_t lo = tiles & ((uint64_t(1) << s) - 1);
        const uint64_t hi = ((tiles >> s) >> 4) << s;
        tiles = hi | lo;
    }
}

// --------------------------------------------------------------------------
// Pancake (PancakeSimple.cpp:12-20,62-73): operator k reverses the LAST k+2
// values; the child's operator code is k.  Only the last m = k+2 Lehmer
// digits change, so child = parent - low_m(parent) + low_m(child), where
// low_m(child) = sum_{q<m} q! * #(earlier values of the parent suffix that
// are smaller than the parent value at position n-m+q).
// --------------------------------------------------------------------------

// n > 7.  The first kL = n-7 positions of an index depend on index / 7! only
// (digit i has weight (n-1-i)!): every index of a block of 7! = 5040 shares
// them, and their part of each larger flip's rank is a constant of the block.
// A Prefix holds those constants; a state unranks its last seven values from
// index % 7! and adds their terms: 60 popcounts a parent at 13 pancakes
// instead of 75, no digits or masks of the other positions, and 70 registers
// instead of 96 to 128.
// (A table of the 5040 arrangements, with or without the small flips'
// deltas, instead of the unranking: no faster, 132.8 to 134.0 against
// 135.0 ms; its loads queue behind the marks.)
template <int N>
struct PancakeLarge {
    static constexpr int kBranch = N - 1;
    static constexpr int kOps = N - 1;
    static constexpr int kL = N - 7;
    static constexpr uint32_t kBlock = 5040;  // 7!
    static constexpr int kNear = (N < 12 ? N : 12) - 7;  // flips of 8 .. 12
    static constexpr int kFar = N > 12 ? N - 12 : 1;     // flips of 13 ..
    struct Prefix {
        uint32_t acc;     // values at positions < kL, one bit each
        uint32_t tiles7;  // the other 7 values, ascending, one nibble each
        struct {
            uint32_t base;  // of flip m: (terms of the positions < kL) - (their parent digits), mod 2^32
            uint32_t keep;  // values not left of the flip
        } near[kNear];
        uint32_t far_keep[kFar];
        uint64_t far_base[kFar];
    };

    // Prefix of the indexes in [q*7!, (q+1)*7!); q < n!/7! <= 16!/7! < 2^32.
    __device__ __forceinline__ static void make_prefix(uint32_t q, Prefix& P) {
        uint32_t d[kL], pre[kL], pb[kL];  // digits; values left of the position; those smaller than its own
#pragma unroll
        for (int i = kL - 1; i >= 0; --i) {
            d[i] = q % uint32_t(N - i);
            q /= uint32_t(N - i);
        }
        uint64_t tiles = 0xFEDCBA9876543210ull;
        uint32_t acc = 0;
#pragma unroll
        for (int i = 0; i < kL; ++i) {
            const uint32_t s = 4u * d[i];
            const uint32_t v = uint32_t(tiles >> s) & 15u;
            tiles = (((tiles >> s) >> 4) << s) | (tiles & ((uint64_t(1) << s) - 1));
            pre[i] = acc;
            pb[i] = acc & ((1u << v) - 1u);
            acc |= 1u << v;
        }
        P.acc = acc;
        P.tiles7 = uint32_t(tiles) & 0x0FFFFFFFu;
#pragma unroll
        for (int m = 8; m <= N; ++m) {
            const int i = N - m;
            uint64_t base = 0;
#pragma unroll
            for (int j = i; j < kL; ++j) {
                const uint32_t c = j > i ? __popc(pb[j] & ~pre[i]) : 0;
                if (m <= 12) base = uint32_t(base) + uint32_t(fact(j - i)) * c - d[j] * uint32_t(fact(N - 1 - j));
                else base += fact(j - i) * c - uint64_t(d[j]) * fact(N - 1 - j);
            }
            if (m <= 12) {
                P.near[m - 8].base = uint32_t(base);
                P.near[m - 8].keep = ~pre[i];
            } else {
                P.far_base[m - 13 < kFar ? m - 13 : 0] = base;
                P.far_keep[m - 13 < kFar ? m - 13 : 0] = ~pre[i];
            }
        }
    }

    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand(uint64_t index, uint32_t opbits, Emit& emit) {
        expand_range<kOpBits>(index, opbits, 0, N - 1, emit);
    }

    // Only the children with operator in [first, last) (bottom-up probe rounds).
    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand_range(uint64_t index, uint32_t opbits, int first, int last,
                                                        Emit& emit) {
        const uint32_t q = uint32_t(index / kBlock);
        Prefix P;
        make_prefix(q, P);
        expand_prefixed<kOpBits>(index, P, uint32_t(index - uint64_t(q) * kBlock), opbits, first, last, emit);
    }

    // expand_range for index = q*7! + r, with P = make_prefix(q).  For m <= 12
    // every quantity is below 12! < 2^31, so the child is passed to emitters
    // that take it (EmitRel) as the parent plus a 32-bit signed delta.
    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand_prefixed(uint64_t index, const Prefix& prefix, uint32_t r,
                                                           uint32_t opbits, int first, int last, Emit& emit) {
        const Prefix P = prefix;  // in registers: marks may alias a prefix in shared memory
        // pb[t]: the values left of the t-th of the last seven that are smaller
        // and pre[t] those left of it at all
        uint32_t d[7], pb[7], pre[7], low[7], acc = P.acc, tiles7 = P.tiles7;
        uint32_t x = r;
#pragma unroll
        for (int t = 6; t >= 0; --t) {
            d[t] = x % uint32_t(7 - t);
            x /= uint32_t(7 - t);
            low[t] = r - x * uint32_t(fact(7 - t));  // r mod (7-t)!
        }
#pragma unroll
        for (int t = 0; t < 7; ++t) {
            const uint32_t s = 4u * d[t];
            const uint32_t bit = 1u << ((tiles7 >> s) & 15u);
            tiles7 = ((tiles7 >> s) >> 4 << s) | (tiles7 & ((1u << s) - 1u));
            pre[t] = acc;
            pb[t] = acc & (bit - 1u);
            acc |= bit;
        }
        auto skip = [&](int op) { return op < first || op >= last || (kOpBits && ((opbits >> op) & 1u)); };
        auto far_child = [&](int m) -> uint64_t {  // m >= 13
            const uint32_t keep = P.far_keep[m - 13 < kFar ? m - 13 : 0];
            uint32_t s32 = 0, hi = 0;
#pragma unroll
            for (int t = 0; t < 7; ++t) {
                const uint32_t c = __popc(pb[t] & keep);
                if (m - 7 + t < 12) s32 += uint32_t(fact(m - 7 + t)) * c;
                else hi += uint32_t(fact(m - 7 + t) / kF12) * c;
            }
            return index + P.far_base[m - 13 < kFar ? m - 13 : 0] - r + (uint64_t(hi) * kF12 + s32);
        };
        // Far children first, for emitters that take them in two steps.
        constexpr bool kSplit = EmitSplitFar<Emit>::value && (N > 12);
        uint64_t far[kFar];
        FarTicket ticket[kFar];
        if constexpr (kSplit) {
#pragma unroll
            for (int m = 13; m <= N; ++m) {
                far[m - 13] = kInvalidIndex;
                if (skip(m - 2)) continue;
                far[m - 13] = far_child(m);
                ticket[m - 13] = emit.far_issue(far[m - 13], uint32_t(m - 2));
            }
        }
#pragma unroll
        for (int m = 2; m <= N; ++m) {
            if (skip(m - 2)) continue;
            if (m <= 12) {  // m is a compile-time constant after unrolling
                int32_t delta;
                if (m <= 7) {
                    const int t0 = 7 - m;
                    uint32_t s32 = 0;
#pragma unroll
                    for (int t = t0 + 1; t < 7; ++t) s32 += uint32_t(fact(t - t0)) * __popc(pb[t] & ~pre[t0]);
                    delta = int32_t(s32 - low[t0]);
                } else {
                    const auto f = P.near[m - 8 < kNear ? m - 8 : 0];
                    uint32_t s32 = f.base - r;
#pragma unroll
                    for (int t = 0; t < 7; ++t) s32 += uint32_t(fact(m - 7 + t)) * __popc(pb[t] & f.keep);
                    delta = int32_t(s32);
                }
                if constexpr (EmitRel<Emit>::value) emit.rel(index, delta, uint32_t(m - 2));
                else emit(index + int64_t(delta), uint32_t(m - 2));
            } else if (!kSplit) {
                const uint64_t child = far_child(m);
                if constexpr (EmitFar<Emit>::value) emit.far(child, uint32_t(m - 2));
                else emit(child, uint32_t(m - 2));
            }
        }
        if constexpr (kSplit) {
#pragma unroll
            for (int k = 0; k < N - 12; ++k)
                if (far[k] != kInvalidIndex) emit.far_finish(far[k], uint32_t(k + 11), ticket[k]);
        }
    }
};

// n <= 7: one block of at most 7! indexes.
template <int N>
struct PancakeSmall {
    static constexpr int kBranch = N - 1;
    static constexpr int kOps = N - 1;
    static constexpr uint32_t kBlock = 5040;
    struct Prefix { uint32_t unused; };
    __device__ __forceinline__ static void make_prefix(uint32_t, Prefix&) {}

    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand(uint64_t index, uint32_t opbits, Emit& emit) {
        expand_range<kOpBits>(index, opbits, 0, N - 1, emit);
    }
    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand_prefixed(uint64_t index, const Prefix&, uint32_t, uint32_t opbits,
                                                           int first, int last, Emit& emit) {
        expand_range<kOpBits>(index, opbits, first, last, emit);
    }
    // Rank of the child of flip m: with pre = the values left of the suffix
    // (positions < n-m) and pb[j] = the values left of position j that are
    // smaller than v[j], the count above is popc(pb[j] & ~pre).
    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand_range(uint64_t index, uint32_t opbits, int first, int last,
                                                        Emit& emit) {
        uint32_t d[N], v[N], pre[N], pb[N];
        perm_digits<N>(uint32_t(index), d);
        perm_values<N>(d, v);
        uint32_t acc = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            pre[i] = acc;
            pb[i] = acc & ((1u << v[i]) - 1u);
            acc |= 1u << v[i];
        }
        uint32_t low = 0;  // low_m (d[n-1] is always 0)
#pragma unroll
        for (int m = 2; m <= N; ++m) {
            low += d[N - m] * uint32_t(fact(m - 1));
            const int op = m - 2;
            if (op < first || op >= last || (kOpBits && ((opbits >> op) & 1u))) continue;
            uint32_t s = 0;
#pragma unroll
            for (int q = 1; q < m; ++q) s += uint32_t(fact(q)) * __popc(pb[N - m + q] & ~pre[N - m]);
            const int32_t delta = int32_t(s - low);
            if constexpr (EmitRel<Emit>::value) emit.rel(index, delta, uint32_t(op));
            else emit(index + int64_t(delta), uint32_t(op));
        }
    }
};
template <int N>
using Pancake = typename std::conditional<(N > 7), PancakeLarge<(N > 7 ? N : 8)>, PancakeSmall<(N > 7 ? 7 : N)>>::type;

// --------------------------------------------------------------------------
// Sliding tile (SlidingTilePuzzleSimple.cpp:8,61-99): operators UP=0, LEFT=1,
// RIGHT=2, DOWN=3; children in the order up, down, left, right; each child
// carries the operator that moves the blank back.
//
// The children come from the parent's Lehmer digits alone.  The blank is
// value 0, so it is the first position whose digit is 0 (every position left
// of it counts it).  Moving a tile t from position c to the blank's place b < c
// changes the digits of b .. c only: with s_j = [v_j < t] for b < j < c, the
// digits become d_t + sum s_j + 1 at b, d_j + s_j between and 0 at c; s_j is
// [d_j <= r], r running from d_t up by each s_j right to left.  Moving it the
// other way undoes that (s_j = [d_j <= R], R running from d_a - 1 down left
// to right).  A full unrank and a rerank per child took 115 warp instructions
// a parent on the 3x4 board (compute 80%, DRAM 1%); its two-bit search went
// from 42 to 12 ms on B200.
// --------------------------------------------------------------------------
static __device__ const uint64_t kFactorials[16] = {fact(0),  fact(1),  fact(2),  fact(3), fact(4),  fact(5),
                                                    fact(6),  fact(7),  fact(8),  fact(9), fact(10), fact(11),
                                                    fact(12), fact(13), fact(14), fact(15)};

template <int N>
struct Sliding {
    static constexpr int kBranch = 4;
    static constexpr int kOps = 4;
    // Index deltas: below 12! for up to 12 cells (32 bits, taken mod 2^32).
    using Delta = typename std::conditional<N <= 12, uint32_t, uint64_t>::type;

    // Lehmer digits as nibbles, digit i at bits 4 i, in two independent chains
    // (the last seven digits and the others).
    __device__ __forceinline__ static uint64_t digits(uint64_t index) {
        constexpr int kTail = N < 7 ? N : 7;
        uint32_t q = 0, r = uint32_t(index);
        if constexpr (N > 7) {
            if constexpr (N <= 12) q = uint32_t(index) / 5040u;
            else q = uint32_t(index / 5040u);  // below 16! / 7! < 2^32
            r = uint32_t(index) - q * 5040u;
        }
        uint64_t D = 0;
#pragma unroll
        for (int i = N - 2; i >= N - kTail; --i) {
            D |= uint64_t(r % uint32_t(N - i)) << (4 * i);
            r /= uint32_t(N - i);
        }
#pragma unroll
        for (int i = N - kTail - 1; i >= 0; --i) {
            D |= uint64_t(q % uint32_t(N - i)) << (4 * i);
            q /= uint32_t(N - i);
        }
        return D;
    }

    // inv_width = ceil(256 / width), so b / width = b * inv_width >> 8 for b < 16.
    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand(uint64_t index, uint32_t opbits, int width, int inv_width,
                                                  Emit& emit) {
        const uint64_t D = digits(index);
        // first zero digit (the last digit is always 0): the lowest nibble
        // flag is exact, borrows only reach nibbles above a zero one
        constexpr uint64_t kOnes = 0x1111111111111111ull;
        const int b = (__ffsll((long long)((D - kOnes) & ~D & (kOnes << 3))) - 1) >> 2;
        const int col = b - width * ((b * inv_width) >> 8);
        auto from = [&](int i) -> uint32_t { return uint32_t(D >> (4 * i)); };  // eight digits, i first
        auto weight = [&](int i) -> Delta { return Delta(__ldg(&kFactorials[N - 1 - i])); };
        auto child = [&](Delta delta, uint32_t op) {
            if constexpr (N <= 12 && EmitRel<Emit>::value) emit.rel(index, int32_t(delta), op);
            else if constexpr (N <= 12) emit(index + int64_t(int32_t(delta)), op);
            else emit(index + delta, op);
        };
        const Delta wb = weight(b);
        const uint32_t right = from(b + 1 < 16 ? b + 1 : 15);  // the digits right of the blank
        if (b >= width && !(kOpBits && (opbits & 1u))) {
            const int a = b - width;
            uint32_t left = from(a), R = (left & 15u) - 1;
            Delta t = left & 15u;  // Horner sum of the digit changes at a .. j
            for (int j = a + 1; j < b; ++j) {
                left >>= 4;
                const uint32_t s = (left & 15u) <= R ? 1u : 0u;
                R -= s;
                t = t * Delta(N - j) + s;
            }
            child(-((t * Delta(N - b) - R) * wb), 3u);
        }
        if (b < N - width && !(kOpBits && (opbits & 8u))) {
            const int c = b + width;
            uint32_t r = (right >> (4 * (width - 1))) & 15u;
            Delta w = weight(c), sum = -(Delta(r) * w);
            for (int j = c - 1; j > b; --j) {
                w *= Delta(N - 1 - j);
                const uint32_t s = ((right >> (4 * (j - b - 1))) & 15u) <= r ? 1u : 0u;
                r += s;
                sum += s ? w : Delta(0);
            }
            child(sum + Delta(r + 1) * wb, 0u);
        }
        if (col > 0 && !(kOpBits && (opbits & 2u))) {
            const Delta d = from(b - 1) & 15u;
            child(-((d * Delta(N - b) - (d - 1)) * wb), 2u);
        }
        if (col < width - 1 && !(kOpBits && (opbits & 4u))) {
            const Delta d = right & 15u;
            child((d + 1) * wb - d * weight(b + 1), 1u);
        }
    }
};

// --------------------------------------------------------------------------
// Sliding tile in SlidingTilePuzzleOptimized's index
// (Puzzles/SlidingTilePuzzleOptimized.cpp:99-236; GPU expand
// kernel_sliding_tile_optimized, Puzzles/SlidingPuzzleGpu.cu:211-269).  The
// board's T = N-1 tiles in board order, the blank left out; digit i of tile
// i (i >= 2) = how many earlier tiles are smaller.  Digit 0 is always 0 and
// digit 1 follows from the parity rule (:79-97), so neither is stored.  Low
// 32 bits: blank + 16 * sum_{i=2..11} d_i * i!/2; bits 32 and up (14..16
// cells): d_12 | d_13 << 4 | d_14 << 8.  Moving the blank up or down rotates
// the tiles between the two blank positions by one place; moving it left or
// right only changes the blank digit (index -+ 1).
// --------------------------------------------------------------------------
template <int N>
struct SlidingOpt {
    static constexpr int kBranch = 4;
    static constexpr int kOps = 4;
    static constexpr int T = N - 1;                    // tiles
    static constexpr int kTop = T - 1 < 11 ? T - 1 : 11;  // last digit of the low word
    static_assert(N >= 4 && N <= 16, "2x2 .. 4x4 boards");

    // The tiles (values 0..T-1, list position i in nibble i) and blank of an
    // index; false when the index names no board.
    __device__ __forceinline__ static bool board(uint64_t index, int width, uint64_t& tiles, uint32_t& blank) {
        blank = uint32_t(index) & 15u;
        if (blank >= uint32_t(N)) return false;
        uint32_t d[16];
        uint32_t low = uint32_t(index) >> 4;
#pragma unroll
        for (int i = 2; i <= kTop; ++i) {
            d[i] = low % uint32_t(i + 1);
            low /= uint32_t(i + 1);
        }
        if (low) return false;
        uint64_t seg = index >> 32;
#pragma unroll
        for (int i = 12; i < T; ++i) {
            d[i] = uint32_t(seg) & 15u;
            seg >>= 4;
            if (d[i] > uint32_t(i)) return false;
        }
        if (seg) return false;
        // Values, last tile first: d_i picks among the values still unused
        // (ascending in a nibble list; the first i+1 entries are the unused ones).
        uint64_t left = 0xFEDCBA9876543210ull;
        uint32_t odd = 1;  // inversions of the tile list with d_1 = 0: sum (i - d_i) + 1
        tiles = 0;
#pragma unroll
        for (int i = T - 1; i >= 2; --i) {
            const uint32_t s = 4u * d[i];
            tiles |= ((left >> s) & 15u) << (4 * i);
            left = (((left >> s) >> 4) << s) | (left & ((uint64_t(1) << s) - 1));
            odd += uint32_t(i) - d[i];
        }
        const uint32_t lo = uint32_t(left) & 15u, hi = (uint32_t(left) >> 4) & 15u;
        if (width % 2 == 0) odd += blank / uint32_t(width);
        // d_1 = 0 puts the larger of the last two values first; the other
        // parity class swaps them (Unpack, :133-137)
        tiles |= (odd & 1u) ? uint64_t(lo | (hi << 4)) : uint64_t(hi | (lo << 4));
        return true;
    }

    // Index of tiles / blank (Pack + GetIndex, :99-158).
    __device__ __forceinline__ static uint64_t index_of(uint64_t tiles, uint32_t blank) {
        uint32_t seen = (1u << (tiles & 15u)) | (1u << ((tiles >> 4) & 15u));
        uint32_t low = 0;
        uint64_t seg = 0;
#pragma unroll
        for (int i = 2; i < T; ++i) {
            const uint32_t v = uint32_t(tiles >> (4 * i)) & 15u;
            const uint32_t d = __popc(seen & ((1u << v) - 1u));
            seen |= 1u << v;
            if (i <= 11) low += d * uint32_t(fact(i) / 2);
            else seg |= uint64_t(d) << (4 * (i - 12));
        }
        return (seg << 32) | (uint64_t(low) * 16u + blank);
    }

    template <bool kOpBits, class Emit>
    __device__ __forceinline__ static void expand(uint64_t index, uint32_t opbits, int width, Emit& emit) {
        uint64_t tiles;
        uint32_t z;
        if (!board(index, width, tiles, z)) return;
        const uint32_t w = uint32_t(width);
        const uint64_t mask = (uint64_t(1) << (4 * w)) - 1;  // w <= 8 tiles
        if (z >= w && !(kOpBits && (opbits & 1u))) {  // blank up: tiles z-w .. z-1 rotate left
            const uint32_t a = 4u * (z - w);
            const uint64_t seg = (tiles >> a) & mask;
            const uint64_t rot = (seg >> 4) | ((seg & 15u) << (4 * (w - 1)));
            emit(index_of((tiles & ~(mask << a)) | (rot << a), z - w), 3u);
        }
        if (z + w < uint32_t(N) && !(kOpBits && (opbits & 8u))) {  // blank down: tiles z .. z+w-1 rotate right
            const uint32_t a = 4u * z;
            const uint64_t seg = (tiles >> a) & mask;
            const uint64_t rot = ((seg << 4) & mask) | (seg >> (4 * (w - 1)));
            emit(index_of((tiles & ~(mask << a)) | (rot << a), z + w), 0u);
        }
        if (z % w > 0 && !(kOpBits && (opbits & 2u))) emit(index - 1, 2u);
        if (z % w < w - 1 && !(kOpBits && (opbits & 4u))) emit(index + 1, 1u);
    }
};

// --------------------------------------------------------------------------
// Four-peg Towers of Hanoi (FourPegHanoiSimple.cpp:104-124,156-174): disk d
// (0 = smallest) sits on peg (index >> 2d) & 3.  For each peg pair a<b the
// smaller of the two top disks moves; the operator bit tested is the source
// peg and the child's operator is the destination peg.  With symmetry on,
// pegs 1..3 are relabelled after the move so that their bottom disks are in
// descending order, using the compare-exchange sequence (2,3),(1,2),(2,3)
// of FourPegHanoiSimple.cpp:51-69, and the child's operator is the
// destination's new label.
// --------------------------------------------------------------------------
struct Hanoi {
    static constexpr int kBranch = 6;
    static constexpr int kOps = 4;

    template <bool kOpBits, class Emit>
    // sym: 0 none; 1 FourPegHanoiSimple (restore after every move); 2
    // FourPegHanoiOptimized (restore only when the move empties the source
    // peg or lands on an empty one, FourPegHanoiOptimized.cpp:190-197; the
    // same children for canonical states, different ones for the others).
    __device__ __forceinline__ static void expand(uint64_t index, uint32_t opbits, int disks, int sym,
                                                  Emit& emit) {
        const uint64_t even = disks >= 32 ? 0x5555555555555555ull
                                          : (0x5555555555555555ull & ((uint64_t(1) << (2 * disks)) - 1));
        const uint64_t L = index & even, H = (index >> 1) & even;
        uint64_t m[4];
        m[0] = ~H & ~L & even;
        m[1] = ~H & L;
        m[2] = H & ~L;
        m[3] = H & L;
        int top[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) top[p] = m[p] ? __ffsll((long long)m[p]) - 1 : 64;  // even bit position
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int b = a + 1; b < 4; ++b) {
                if (top[a] == 64 && top[b] == 64) continue;
                const bool a_src = top[a] < top[b];
                const int src = a_src ? a : b, dst = a_src ? b : a;
                const int pos = a_src ? top[a] : top[b];
                if (kOpBits && ((opbits >> src) & 1u)) continue;
                uint64_t child = index ^ (uint64_t(src ^ dst) << pos);
                uint32_t op = uint32_t(dst);
                if (sym == 1 || (sym == 2 && (top[dst] == 64 || m[src] == (uint64_t(1) << pos)))) {
                    const uint64_t bitpos = uint64_t(1) << pos;
                    uint64_t mm[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) mm[q] = m[q] ^ ((q == src || q == dst) ? bitpos : 0);
                    int bottom[4], lab[4] = {0, 1, 2, 3};
#pragma unroll
                    for (int p = 0; p < 4; ++p) bottom[p] = mm[p] ? 63 - __clzll((long long)mm[p]) : -1;
                    // compare-exchange (2,3), (1,2), (2,3): swap when bottom[i] < bottom[j]
                    auto cx = [&](int i, int j) {
                        if (bottom[i] < bottom[j]) {
                            int t = bottom[i]; bottom[i] = bottom[j]; bottom[j] = t;
                            uint64_t u = mm[i]; mm[i] = mm[j]; mm[j] = u;
                            t = lab[i]; lab[i] = lab[j]; lab[j] = t;
                        }
                    };
                    cx(2, 3); cx(1, 2); cx(2, 3);
                    // position k now holds original peg lab[k]: index bits of disks on it = k
                    const uint64_t nl = mm[1] | mm[3], nh = mm[2] | mm[3];
                    child = nl | (nh << 1);
                    uint32_t inv = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) if (lab[k] == dst) inv = uint32_t(k);
                    op = inv;
                }
                emit(child, op);
            }
        }
    }
};

}  // namespace psb
