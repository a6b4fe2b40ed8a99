// psb_codec.cu -- frontier compression on the GPU, byte-exact with the
// reference's segment stream:
//   FrontierCompression::Encode / Decode   Common/FrontierCompression.cpp:36-125
//   StreamVInt::Encode / Decode            Common/StreamVInt.cpp:116-251
//   CompressedSegmentWriter framing        Common/CompressedFrontier.cpp:103-140
//
// A segment's frontier (the set bits of a bitmap range of at most 2^32
// states, as u32 offsets in ascending order) is cut into blocks of 262,144
// offsets (StreamVInt::MAX_INDEXES_COUNT).  Each block becomes either
//   * a bitmap block: [u32 words | 0x80000000][u32 first][bitmap of v - first - 1],
//     chosen when count > 128 and the bitmap's bits < 10*count - 8; or
//   * a StreamVInt block: [u32 count], then the deltas (first value raw),
//     zero-padded to a multiple of 8 values, as tuples of four values:
//     one descriptor byte (2 bits per value = bytes - 1), then each value's
//     1..4 little-endian bytes.
// The blocks are concatenated.  Decoding needs each block's start; the
// encoder returns that as a side table (psb_codec_block), and
// psb_frontier_index builds it on the host for a stream from elsewhere.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <new>
#include <string>
#include <memory>
#include <vector>

#include "../../include/psb200.h"
#include "psb_internal.h"

namespace {

constexpr uint32_t kBlock = 256 * 1024;  // StreamVInt::MAX_INDEXES_COUNT (Common/StreamVInt.h:9)
constexpr uint32_t kMap = 0x80000000u;   // CODEC_MAP (Common/FrontierCompression.cpp:6)
constexpr int kT = 256;
constexpr int kCW = 4;                      // words per thread of a chunk
constexpr uint32_t kChunkWords = kT * kCW;  // bitmap words whose popcounts are summed together

#define CD_CUDA(call)                                                                           \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return psb_set_error(e_ == cudaErrorMemoryAllocation ? PSB_ERR_NOMEM : PSB_ERR_CUDA, \
                                 (std::string(#call) + ": " + cudaGetErrorString(e_)).c_str());  \
    } while (0)

__device__ __forceinline__ uint64_t masked_word(const uint64_t* bits, uint64_t w, uint64_t n_words, uint64_t n_bits) {
    uint64_t v = bits[w];
    if (w == n_words - 1 && (n_bits & 63)) v &= (uint64_t(1) << (n_bits & 63)) - 1;
    return v;
}

// Popcount of each chunk of kChunkWords words.
__global__ void k_block_sums(const uint64_t* bits, uint64_t n_words, uint64_t n_bits, unsigned long long* bsum) {
    const uint64_t base = uint64_t(blockIdx.x) * kChunkWords;
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < kCW; ++k) {
        const uint64_t w = base + uint64_t(k) * kT + threadIdx.x;
        if (w < n_words) c += __popcll(masked_word(bits, w, n_words, n_bits));
    }
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    __shared__ uint32_t s[kT / 32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < kT / 32; ++i) t += s[i];
        bsum[blockIdx.x] = t;
    }
}

// Exclusive scan of n u64 values in place by one CTA of kScanT threads
// (chunk sums, tuple-group sums: at most a few hundred thousand values), in
// tiles of kScanT * 16 values: thread t sums values 16 t .. 16 t + 15 of a
// tile, warp shuffles and one pass over the warp totals rank them.
constexpr int kScanT = 1024;
__global__ void __launch_bounds__(kScanT) k_scan_small(unsigned long long* v, uint64_t n, unsigned long long* total) {
    __shared__ unsigned long long warp_tot[kScanT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (uint64_t base = 0; base < n; base += uint64_t(kScanT) * 16) {
        const uint64_t i0 = base + uint64_t(threadIdx.x) * 16;
        unsigned long long x[16], c = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            x[k] = i0 + k < n ? v[i0 + k] : 0;
            c += x[k];
        }
        unsigned long long inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) warp_tot[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            unsigned long long t = warp_tot[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane] = t;  // inclusive over warps
        }
        __syncthreads();
        unsigned long long run = carry + (warp ? warp_tot[warp - 1] : 0) + inc - c;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            if (i0 + k < n) v[i0 + k] = run;
            run += x[k];
        }
        carry += warp_tot[kScanT / 32 - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// Inclusive block-wide sum scan of one value per thread (kT threads).
__device__ __forceinline__ uint32_t block_inclusive_scan(uint32_t v, uint32_t* warp_tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += warp_tot[w];
    __syncthreads();
    return before + v;
}

// Sum of one value per thread over the CTA, written by thread 0.
__device__ __forceinline__ void chunk_total(uint32_t c, unsigned long long* out) {
    __shared__ uint32_t warp_tot[kT / 32];
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < kT / 32; ++i) t += warp_tot[i];
        *out = t;
    }
}

__device__ __forceinline__ uint32_t vbytes(uint32_t x) { return x >> 24 ? 4 : x >> 16 ? 3 : x >> 8 ? 2 : 1; }

// A block of up to kBlock offsets.
struct BlockInfo {
    unsigned long long out_off;  // byte offset of the block in the segment's stream
    unsigned long long bytes;
    uint32_t count, first, last, is_bitmap;
    uint32_t svi, pad;  // StreamVInt blocks: which one (its place in the offset list)
};

// One segment's result, on the device (EncTotals) and read by the host.
using psb::EncTotals;

// StreamVInt blocks are worked on in parts of kPartTuples tuples.
constexpr uint32_t kPartTuples = 1024, kParts = kBlock / 4 / kPartTuples;
// Bitmap blocks in parts of kPartWords words: a bitmap block's bitmap is
// smaller than 10 bits per offset, so 40 parts hold any.
constexpr uint32_t kPartWords = 1024, kBitmapParts = 40;
static_assert(uint64_t(kBitmapParts) * kPartWords * 64 >= uint64_t(kBlock) * 10, "every bitmap block's words have a part");

// Writes the ascending offsets of the set bits that fall in StreamVInt
// blocks into their block's place of the offset list (bitmap blocks need no
// list: their words are copied from the bitmap).  One CTA per chunk; warp w
// takes words 128 w .. 128 w + 127 of it, lane l words l, 32 + l, .. of those
// (a dense stretch is spread over the lanes), and two scans of paired counts
// rank all of the warp's offsets.  The lanes put them into shared memory at
// their ranks and the warp stores them in order; a warp with more than
// kStaged offsets stores each where it goes.
// (A rank-ordered search per 32 words took 52 us where this takes 6: its
// chain of shuffles, on chunks four times as large.)
constexpr uint32_t kStaged = 1024;
__global__ void __launch_bounds__(kT) k_compact(const uint64_t* bits, uint64_t n_words, uint64_t n_bits,
                                                const unsigned long long* bsum, uint64_t nbs, const EncTotals* totals,
                                                const BlockInfo* blocks, uint32_t cap_refs, uint32_t* idx) {
    __shared__ uint32_t warp_tot[kT / 32];
    __shared__ uint16_t staged[kT / 32][kStaged];
    if (totals->n_refs == 0 || totals->n_refs > cap_refs) return;
    // Chunks with no offsets, or whose offsets all fall in bitmap blocks,
    // have nothing to list (uniform over the CTA).  A chunk has at most 65,536
    // offsets, so they fall in at most two blocks.
    const unsigned long long r_lo = bsum[blockIdx.x];
    const unsigned long long r_hi = blockIdx.x + 1 < nbs ? bsum[blockIdx.x + 1] : totals->count;
    if (r_hi == r_lo) return;
    const uint64_t b0 = r_lo / kBlock, b1 = (r_hi - 1) / kBlock;
    const bool list0 = !blocks[b0].is_bitmap, list1 = !blocks[b1].is_bitmap;
    if (!list0 && !list1) return;
    uint32_t* const to0 = idx + uint64_t(blocks[b0].svi) * kBlock;
    uint32_t* const to1 = idx + uint64_t(blocks[b1].svi) * kBlock;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t w0 = uint64_t(blockIdx.x) * kChunkWords + warp * (32 * kCW);  // the warp's first word
    static_assert(kCW == 4, "two pairs of words per lane");
    uint64_t v[kCW];
    uint32_t at[kCW];  // rank of the word's first offset in the warp
    uint32_t before = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t c = 0;  // counts of words 2h (low half) and 2h + 1; a word row has at most 2048
#pragma unroll
        for (int k = 2 * h; k < 2 * h + 2; ++k) {
            const uint64_t w = w0 + 32 * k + lane;
            v[k] = w < n_words ? masked_word(bits, w, n_words, n_bits) : 0;
            c |= uint32_t(__popcll(v[k])) << (16 * (k & 1));
        }
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        const uint32_t rows = __shfl_sync(0xFFFFFFFFu, incl, 31);
        at[2 * h] = before + (incl & 0xFFFFu) - (c & 0xFFFFu);
        at[2 * h + 1] = before + (rows & 0xFFFFu) + (incl >> 16) - (c >> 16);
        before += (rows & 0xFFFFu) + (rows >> 16);
    }
    if (lane == 31) warp_tot[warp] = before;
    __syncthreads();
    const uint32_t total = warp_tot[warp];
    unsigned long long r = r_lo;  // rank of the warp's first offset
    for (uint32_t k = 0; k < warp; ++k) r += warp_tot[k];
    auto put = [&](uint32_t k, uint32_t offset) {  // the warp's k-th offset
        const unsigned long long rank = r + k;
        const bool second = rank / kBlock != b0;
        if (second ? list1 : list0) (second ? to1 : to0)[rank % kBlock] = offset;
    };
    const uint32_t first = uint32_t(w0 * 64);  // offsets fit 32 bits
#pragma unroll
    for (int k = 0; k < kCW; ++k) {
        uint64_t m = v[k];
        while (m) {
            const uint32_t o = (32 * k + lane) * 64 + uint32_t(__ffsll((long long)m) - 1);
            m &= m - 1;
            if (total <= kStaged) staged[warp][at[k]] = uint16_t(o);
            else put(at[k], first + o);
            ++at[k];
        }
    }
    if (total <= kStaged) {
        __syncwarp();
        for (uint32_t k = lane; k < total; k += 32) put(k, first + staged[warp][k]);
    }
}

// First and last offset of every block (ranks b * kBlock and the block's
// last rank), by select: the chunk holding the rank from the chunk prefix
// sums (a search with one probe per thread a turn), then a block scan of that
// chunk's per-thread counts (thread t: words kCW t .. kCW t + kCW - 1).  Items
// 2b and 2b + 1 serve block b.
__global__ void __launch_bounds__(kT) k_select_blocks(const uint64_t* bits, uint64_t n_words, uint64_t n_bits,
                                                      const unsigned long long* bsum, uint64_t nbs,
                                                      const EncTotals* totals, BlockInfo* blocks) {
    __shared__ uint32_t warp_tot[kT / 32];
    const uint64_t count = totals->count, nb = (count + kBlock - 1) / kBlock;
    for (uint64_t item = blockIdx.x; item < 2 * nb; item += gridDim.x) {
        const uint64_t b = item / 2;
        const bool last = item & 1;
        const uint64_t end = (b + 1) * kBlock < count ? (b + 1) * kBlock : count;
        const uint64_t r = last ? end - 1 : b * kBlock;
        uint64_t lo = 0, n = nbs;  // the largest chunk with bsum <= r is in [lo, lo + n) (bsum[0] = 0)
        while (n > 1) {
            const uint64_t step = (n + kT - 1) / kT, at = threadIdx.x * step;
            const uint32_t k = __syncthreads_count(at < n && bsum[lo + at] <= r);
            lo += (k - 1) * step;
            n = n - (k - 1) * step < step ? n - (k - 1) * step : step;
        }
        const uint64_t rem = r - bsum[lo];
        const uint64_t w0 = lo * kChunkWords + uint64_t(threadIdx.x) * kCW;
        uint64_t v[kCW];
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < kCW; ++k) {
            v[k] = w0 + k < n_words ? masked_word(bits, w0 + k, n_words, n_bits) : 0;
            c += __popcll(v[k]);
        }
        const uint32_t inc = block_inclusive_scan(c, warp_tot);  // ends with a barrier
        const uint32_t exc = inc - c;
        if (rem < exc || rem >= inc) continue;  // exactly one thread holds the rank
        uint32_t left = uint32_t(rem - exc);
#pragma unroll
        for (int k = 0; k < kCW; ++k) {
            const uint32_t ck = __popcll(v[k]);
            if (left < ck) {
                const uint32_t pos = uint32_t((w0 + k) * 64 + psb::select_bit(v[k], left));
                if (last) blocks[b].last = pos; else blocks[b].first = pos;
                left = 0xFFFFFFFFu;  // found
            } else if (left != 0xFFFFFFFFu) {
                left -= ck;
            }
        }
    }
}

// Inclusive scan of one value per thread over a CTA of kScanT threads.
__device__ __forceinline__ unsigned long long scan_cta(unsigned long long v, unsigned long long* warp_tot,
                                                       unsigned long long* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    unsigned long long before = 0, all = 0;
    for (int w = 0; w < kScanT / 32; ++w) {
        if (w < warp) before += warp_tot[w];
        all += warp_tot[w];
    }
    __syncthreads();
    *total = all;
    return before + v;
}

// FrontierCompression::Encode (FrontierCompression.cpp:92-102): a block is a
// bitmap block when it holds more than 128 offsets and its bitmap is smaller
// than 10 bits per offset.  With operator bits (force_svi) every block is a
// StreamVInt block, as CompressedFrontierWriter writes them
// (Common/CompressedFrontier.cpp:63-70).  One CTA; the StreamVInt blocks are
// numbered in order.
__global__ void __launch_bounds__(kScanT) k_decide(EncTotals* totals, BlockInfo* blocks, uint32_t* refs,
                                                   int force_svi) {
    __shared__ unsigned long long warp_tot[kScanT / 32];
    const uint64_t count = totals->count, nb = (count + kBlock - 1) / kBlock;
    unsigned long long n_refs = 0;
    for (uint64_t b0 = 0; b0 < nb; b0 += kScanT) {
        const uint64_t b = b0 + threadIdx.x;
        uint32_t svi = 0;
        if (b < nb) {
            BlockInfo& bi = blocks[b];
            const uint64_t r0 = b * kBlock;
            const uint32_t n = uint32_t(count - r0 < kBlock ? count - r0 : kBlock);
            bi.count = n;
            const uint64_t bm_bytes = (uint64_t(bi.last) - bi.first + 63) / 64 * 8 + 8;
            bi.is_bitmap = (!force_svi && n > 128 && bm_bytes * 8 < uint64_t(n) * 10 - 8) ? 1 : 0;
            bi.bytes = bm_bytes;  // of a bitmap block; k_layout fills in the others
            svi = !bi.is_bitmap;
        }
        unsigned long long total;
        const unsigned long long at = n_refs + scan_cta(svi, warp_tot, &total) - svi;
        if (svi) {
            blocks[b].svi = uint32_t(at);
            refs[at] = uint32_t(b);
        }
        n_refs += total;
    }
    if (threadIdx.x == 0) {
        totals->nb = uint32_t(nb);
        totals->n_refs = uint32_t(n_refs);
    }
}

// The four deltas of tuple t of a block (0 past its count; the first value
// of a block is itself) and the tuple's length: 1 descriptor byte and 1..4
// bytes per value.
__device__ __forceinline__ uint32_t tuple_of(const uint32_t* v, uint32_t count, uint32_t t, uint32_t (&x)[4]) {
    const uint32_t k = 4 * t;
    const uint4 q = *reinterpret_cast<const uint4*>(v + k);
    const uint32_t prev = k ? v[k - 1] : 0;
    x[0] = k < count ? q.x - prev : 0;
    x[1] = k + 1 < count ? q.y - q.x : 0;
    x[2] = k + 2 < count ? q.z - q.y : 0;
    x[3] = k + 3 < count ? q.w - q.z : 0;
    return 1 + vbytes(x[0]) + vbytes(x[1]) + vbytes(x[2]) + vbytes(x[3]);
}

__device__ __forceinline__ uint32_t tuples_of(uint32_t count) { return uint32_t((uint64_t(count) + 7) / 8 * 2); }

// psum[ref * kParts + p] = bytes of the tuples of part p of StreamVInt block `ref`.
__global__ void __launch_bounds__(kT) k_part_bytes(const uint32_t* idx, const EncTotals* totals,
                                                   const BlockInfo* blocks, const uint32_t* refs, uint32_t cap_refs,
                                                   unsigned long long* psum) {
    if (totals->n_refs > cap_refs) return;
    const uint32_t items = totals->n_refs * kParts;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t ref = item / kParts, count = blocks[refs[ref]].count, tuples = tuples_of(count);
        const uint32_t t0 = (item % kParts) * kPartTuples;
        uint32_t c = 0;
        for (uint32_t t = t0 + threadIdx.x; t < t0 + kPartTuples && t < tuples; t += kT) {
            uint32_t x[4];
            c += tuple_of(idx + uint64_t(ref) * kBlock, count, t, x);
        }
        chunk_total(c, psum + item);
        __syncthreads();
    }
}

// Places the blocks: each StreamVInt block's bytes (header, tuples and, with
// operator bits, one nibble per padded value, StreamVInt.cpp:253-275), its
// parts' first bytes (psum becomes their exclusive prefix), each block's
// offset in the stream and the segment's place: at `first_off`, or after the
// segment before it.  One CTA.
__global__ void __launch_bounds__(kScanT) k_layout(EncTotals* totals, BlockInfo* blocks, const uint32_t* refs,
                                                   unsigned long long* psum, uint32_t cap_refs, int with_ops, int first,
                                                   unsigned long long first_off) {
    __shared__ unsigned long long warp_tot[kScanT / 32];
    const uint64_t nb = totals->nb;
    const uint32_t n_refs = totals->n_refs <= cap_refs ? totals->n_refs : 0;  // the listed ones
    // A warp per StreamVInt block: its parts' bytes, two per lane.
    static_assert(kParts == 64, "two parts per lane");
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t ref = threadIdx.x >> 5; ref < n_refs; ref += kScanT / 32) {
        ulonglong2* parts = reinterpret_cast<ulonglong2*>(psum + uint64_t(ref) * kParts) + lane;
        const ulonglong2 own = *parts;
        unsigned long long incl = own.x + own.y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        *parts = make_ulonglong2(incl - own.x - own.y, incl - own.y);
        if (lane == 31) {
            BlockInfo& bi = blocks[refs[ref]];
            bi.bytes = 4 + incl + (with_ops ? (uint64_t(bi.count) + 7) / 8 * 4 : 0);
        }
    }
    __syncthreads();
    unsigned long long off = 0;
    for (uint64_t b0 = 0; b0 < nb; b0 += kScanT) {
        const uint64_t b = b0 + threadIdx.x;
        const unsigned long long bytes = b < nb ? blocks[b].bytes : 0;
        unsigned long long total;
        const unsigned long long incl = scan_cta(bytes, warp_tot, &total);
        if (b < nb) blocks[b].out_off = off + incl - bytes;
        off += total;
    }
    if (threadIdx.x == 0) {
        totals->bytes = off;
        totals->off = first ? first_off : totals[-1].off + totals[-1].bytes;
    }
}

// The segment's stream, or NULL when it was not planned whole or does not fit.
__device__ __forceinline__ uint8_t* stream_place(const EncTotals* totals, uint32_t cap_refs, uint8_t* out,
                                                 unsigned long long out_cap) {
    if (totals->n_refs > cap_refs || totals->off + totals->bytes > out_cap) return nullptr;
    return out + totals->off;
}

// The CTA's threads write n bytes of shared memory (from a 4-byte boundary,
// readable 4 bytes past n) to dst (any alignment): whole aligned words, and
// the few bytes at the ends.
__device__ __forceinline__ void store_bytes(uint8_t* dst, const uint32_t* src, uint32_t n) {
    const uint8_t* sb = reinterpret_cast<const uint8_t*>(src);
    const uint32_t to_word = uint32_t(0 - reinterpret_cast<uintptr_t>(dst)) & 3u;
    const uint32_t head = to_word < n ? to_word : n, words = (n - head) / 4, tail = head + 4 * words;
    if (threadIdx.x < head) dst[threadIdx.x] = sb[threadIdx.x];
    for (uint32_t j = threadIdx.x; j < words; j += kT)
        *reinterpret_cast<uint32_t*>(dst + head + 4 * j) = __funnelshift_r(src[j], src[j + 1], 8 * head);
    if (threadIdx.x < n - tail) dst[tail + threadIdx.x] = sb[tail + threadIdx.x];
}

// The tuples of the StreamVInt blocks, part by part, kT tuples at a time
// through shared memory, so that the stores are whole words.
__global__ void __launch_bounds__(kT) k_write_svi(const uint32_t* idx, const EncTotals* totals,
                                                  const BlockInfo* blocks, const uint32_t* refs, uint32_t cap_refs,
                                                  const unsigned long long* psum, uint8_t* out,
                                                  unsigned long long out_cap) {
    __shared__ uint32_t buf[kT * 17 / 4 + 2];
    __shared__ uint32_t warp_tot[kT / 32], round_bytes;
    uint8_t* place = stream_place(totals, cap_refs, out, out_cap);
    if (!place) return;
    uint8_t* sb = reinterpret_cast<uint8_t*>(buf);
    const uint32_t items = totals->n_refs * kParts;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t ref = item / kParts, part = item % kParts;
        const BlockInfo bi = blocks[refs[ref]];
        const uint32_t tuples = tuples_of(bi.count), t0 = part * kPartTuples;
        if (t0 >= tuples) continue;
        uint8_t* p = place + bi.out_off;
        if (part == 0 && threadIdx.x < 4) p[threadIdx.x] = uint8_t(bi.count >> (8 * threadIdx.x));
        p += 4 + psum[item];
        for (uint32_t r = t0; r < t0 + kPartTuples && r < tuples; r += kT) {
            const uint32_t t = r + threadIdx.x;
            uint32_t x[4], len = 0;
            if (t < tuples) len = tuple_of(idx + uint64_t(ref) * kBlock, bi.count, t, x);
            const uint32_t incl = block_inclusive_scan(len, warp_tot);
            if (threadIdx.x == kT - 1) round_bytes = incl;
            if (len) {
                uint32_t at = incl - len, desc = 0, pos = at + 1;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t nbytes = vbytes(x[q]);
                    desc |= (nbytes - 1) << (2 * q);
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i)
                        if (i < nbytes) sb[pos + i] = uint8_t(x[q] >> (8 * i));
                    pos += nbytes;
                }
                sb[at] = uint8_t(desc);
            }
            __syncthreads();
            const uint32_t n = round_bytes;
            store_bytes(p, buf, n);
            p += n;
            __syncthreads();
        }
    }
}

// Bounds of the StreamVInt blocks (StreamVInt::EncodeBounds,
// StreamVInt.cpp:139-147,193-198): the operator nibble of each value, 8 per
// group packed as bytes b_q | b_(q+4) << 4, after the block's tuples.  The
// nibble of offset v is state nib_first + v of the 4-bit array `nib` (NULL:
// every nibble is 0); values past the count have nibble 0.
__global__ void __launch_bounds__(kT) k_write_bounds(const uint32_t* idx, const EncTotals* totals,
                                                     const BlockInfo* blocks, const uint32_t* refs, uint32_t cap_refs,
                                                     const uint64_t* nib, uint64_t nib_first, uint8_t* out,
                                                     unsigned long long out_cap) {
    uint8_t* place = stream_place(totals, cap_refs, out, out_cap);
    if (!place) return;
    const uint32_t items = totals->n_refs * kParts;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t ref = item / kParts, part = item % kParts;
        const BlockInfo bi = blocks[refs[ref]];
        const uint32_t groups = tuples_of(bi.count) / 2, g0 = part * (kPartTuples / 2);
        const uint32_t* v = idx + uint64_t(ref) * kBlock;
        uint8_t* bounds = place + bi.out_off + bi.bytes - uint64_t(groups) * 4;
        for (uint32_t g = g0 + threadIdx.x; g < g0 + kPartTuples / 2 && g < groups; g += kT) {
            uint32_t b[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                b[j] = 0;
                if (nib && 8 * g + j < bi.count) {
                    const uint64_t state = nib_first + v[8 * g + j];
                    b[j] = uint32_t(nib[state >> 4] >> (4 * (state & 15))) & 15u;
                }
            }
            uint8_t* p = bounds + 4ull * g;
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] = uint8_t(b[q] | (b[q + 4] << 4));
        }
    }
}

// Bitmap block: bit j of output word i is state first + 1 + 64 i + j (<= last).
// A chunk with no set bits; its words may be stale scratch
// (an extraction skips chunks of windows that hold no frontier state).
__device__ __forceinline__ bool chunk_empty(const unsigned long long* bsum, uint64_t nbs, uint64_t count,
                                            uint64_t w) {
    const uint64_t k = w / kChunkWords;
    return (k + 1 < nbs ? bsum[k + 1] : count) == bsum[k];
}

__device__ __forceinline__ uint64_t live_word(const uint64_t* bits, uint64_t w, uint64_t n_words, uint64_t n_bits,
                                              const unsigned long long* bsum, uint64_t nbs, uint64_t count) {
    return chunk_empty(bsum, nbs, count, w) ? 0 : masked_word(bits, w, n_words, n_bits);
}

__global__ void __launch_bounds__(kT) k_write_bitmap(const uint64_t* bits, uint64_t n_words, uint64_t n_bits,
                                                     const EncTotals* totals, const BlockInfo* blocks,
                                                     const unsigned long long* bsum, uint64_t nbs, uint32_t cap_refs,
                                                     uint8_t* out, unsigned long long out_cap) {
    __shared__ uint64_t buf[kPartWords + 1];
    uint8_t* place = stream_place(totals, cap_refs, out, out_cap);
    if (!place || totals->n_refs == totals->nb) return;
    const uint64_t count = totals->count, items = uint64_t(totals->nb) * kBitmapParts;
    for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t part = uint32_t(item % kBitmapParts);
        const BlockInfo bi = blocks[item / kBitmapParts];
        const uint32_t words = uint32_t((uint64_t(bi.last) - bi.first + 63) / 64), i0 = part * kPartWords;
        if (!bi.is_bitmap || (i0 >= words && part)) continue;
        uint8_t* p = place + bi.out_off;
        if (part == 0 && threadIdx.x < 8) {
            const uint64_t h = (words | kMap) | (uint64_t(bi.first) << 32);
            p[threadIdx.x] = uint8_t(h >> (8 * threadIdx.x));
        }
        const uint32_t n = i0 >= words ? 0 : words - i0 < kPartWords ? words - i0 : kPartWords;
        for (uint32_t i = threadIdx.x; i < n; i += kT) {
            const uint64_t start = uint64_t(bi.first) + 1 + 64ull * (i0 + i);  // first state of this output word
            const uint64_t w0 = start >> 6, sh = start & 63;
            uint64_t v = live_word(bits, w0, n_words, n_bits, bsum, nbs, count) >> sh;
            if (sh && w0 + 1 < n_words) v |= live_word(bits, w0 + 1, n_words, n_bits, bsum, nbs, count) << (64 - sh);
            if (start + 63 > bi.last) {  // last state this word covers
                const uint64_t keep = uint64_t(bi.last) - start + 1;  // 0..63
                v &= (uint64_t(1) << keep) - 1;
            }
            buf[i] = v;
        }
        __syncthreads();
        store_bytes(p + 8 + 8ull * i0, reinterpret_cast<const uint32_t*>(buf), 8 * n);
        __syncthreads();
    }
}

}  // namespace

namespace psb {

// Encodes segments in stream order without host round trips: every size
// that depends on the segment (offsets, blocks, tuples, bytes) stays in its
// EncTotals on the device, and the launches cover whatever it turns out to
// be.  Only the offset list of the StreamVInt blocks has a capacity
// (cap_refs blocks); a segment that needs more, or does not fit the output,
// is planned but not written, and its totals say so.  (With four round
// trips a segment, 81 depths of 13-disk Hanoi took 16 ms to encode.)
struct SegmentEncoder {
    uint8_t *fixed = nullptr, *lists = nullptr;  // sized by the segment / by cap_refs
    size_t cap_fixed = 0;
    EncTotals* totals = nullptr;
    uint32_t cap_totals = 0;
    // parts of the buffers
    unsigned long long *bsum = nullptr, *psum = nullptr;
    BlockInfo* blocks = nullptr;
    uint32_t *refs = nullptr, *idx = nullptr;
    uint32_t cap_refs = 0;
    uint64_t launches = 0;  // kernels launched since the last encoder_take_launches
    // Operator bits (set_ops): every block StreamVInt with bounds, the nibble
    // of offset v being state ops_first + v of ops_nib (NULL: all zero).
    bool with_ops = false;
    const uint64_t* ops_nib = nullptr;
    uint64_t ops_first = 0;

    // The buffers come from the device's pool in stream order; earlier
    // segments on other streams have been waited for by their callers.
    template <class T>
    static int replace(T** p, size_t bytes, cudaStream_t s) {
        cudaMemPool_t pool = nullptr;
        if (int rc = scratch_pool(&pool)) return rc;
        if (*p) CD_CUDA(cudaFreeAsync(*p, s));
        *p = nullptr;
        CD_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(p), bytes, pool, s));
        return PSB_OK;
    }
    void release(cudaStream_t s) {
        if (fixed) cudaFreeAsync(fixed, s);
        if (lists) cudaFreeAsync(lists, s);
        if (totals) cudaFreeAsync(totals, s);
        fixed = lists = nullptr;
        totals = nullptr;
    }
    ~SegmentEncoder() {
        if (fixed) cudaFree(fixed);
        if (lists) cudaFree(lists);
        if (totals) cudaFree(totals);
    }

    static uint64_t chunks(uint64_t n) { return ((n + 63) / 64 + kChunkWords - 1) / kChunkWords; }
    static uint32_t max_blocks(uint64_t n) { return uint32_t((n + kBlock - 1) / kBlock); }

    int reserve_totals(uint32_t slots, cudaStream_t s) {
        if (slots <= cap_totals) return PSB_OK;
        cap_totals = 0;
        if (int rc = replace(&totals, slots * sizeof(EncTotals), s)) return rc;
        cap_totals = slots;
        return PSB_OK;
    }
    // Room for segments of n bits.
    int reserve(uint64_t n, cudaStream_t s) {
        const size_t at_blocks = ((chunks(n) + 1) * 8 + 255) / 256 * 256;
        const size_t at_refs = at_blocks + (max_blocks(n) * sizeof(BlockInfo) + 255) / 256 * 256;
        const size_t need = at_refs + size_t(max_blocks(n)) * 4;
        if (need > cap_fixed) {
            cap_fixed = 0;
            if (int rc = replace(&fixed, need, s)) return rc;
            cap_fixed = need;
        }
        bsum = reinterpret_cast<unsigned long long*>(fixed);
        blocks = reinterpret_cast<BlockInfo*>(fixed + at_blocks);
        refs = reinterpret_cast<uint32_t*>(fixed + at_refs);
        return PSB_OK;
    }
    // Room for the offsets of n_refs StreamVInt blocks.
    int reserve_lists(uint32_t n_refs, cudaStream_t s) {
        if (n_refs <= cap_refs) return PSB_OK;
        cap_refs = 0;
        const size_t at_psum = size_t(n_refs) * kBlock * 4;
        if (int rc = replace(&lists, at_psum + size_t(n_refs) * kParts * 8, s)) return rc;
        idx = reinterpret_cast<uint32_t*>(lists);
        psum = reinterpret_cast<unsigned long long*>(lists + at_psum);
        cap_refs = n_refs;
        return PSB_OK;
    }

    // Counts, cuts and decides the blocks of an n-bit segment (totals[slot]:
    // count, nb, n_refs).  sums_ready: the chunk popcounts are in bsum.
    int plan(const uint64_t* bits, uint64_t n, bool sums_ready, uint32_t slot, cudaStream_t s) {
        const uint64_t n_words = (n + 63) / 64, nbs = chunks(n);
        EncTotals* t = totals + slot;
        if (!sums_ready) {
            k_block_sums<<<unsigned(nbs), kT, 0, s>>>(bits, n_words, n, bsum);
            launches++;
        }
        k_scan_small<<<1, kScanT, 0, s>>>(bsum, nbs, &t->count);
        k_select_blocks<<<std::min(2 * max_blocks(n), kGrid), kT, 0, s>>>(bits, n_words, n, bsum, nbs, t, blocks);
        k_decide<<<1, kScanT, 0, s>>>(t, blocks, refs, with_ops ? 1 : 0);
        launches += 3;
        CD_CUDA(cudaGetLastError());
        return PSB_OK;
    }
    // Lists the StreamVInt blocks' offsets and places the blocks (totals:
    // bytes, off); `first`: the stream starts at first_off, else after slot - 1's.
    int layout(const uint64_t* bits, uint64_t n, uint32_t slot, bool first, uint64_t first_off, cudaStream_t s) {
        EncTotals* t = totals + slot;
        if (cap_refs) {
            k_compact<<<unsigned(chunks(n)), kT, 0, s>>>(bits, (n + 63) / 64, n, bsum, chunks(n), t, blocks, cap_refs,
                                                         idx);
            k_part_bytes<<<part_grid(n), kT, 0, s>>>(idx, t, blocks, refs, cap_refs, psum);
            launches += 2;
        }
        k_layout<<<1, kScanT, 0, s>>>(t, blocks, refs, psum, cap_refs, with_ops ? 1 : 0, first ? 1 : 0, first_off);
        launches++;
        CD_CUDA(cudaGetLastError());
        return PSB_OK;
    }
    // Writes the stream at out + off if it ends within out_cap bytes of out.
    int write(const uint64_t* bits, uint64_t n, uint32_t slot, uint8_t* out, uint64_t out_cap, cudaStream_t s) {
        const EncTotals* t = totals + slot;
        if (cap_refs) {
            k_write_svi<<<part_grid(n), kT, 0, s>>>(idx, t, blocks, refs, cap_refs, psum, out, out_cap);
            launches++;
            if (with_ops) {
                k_write_bounds<<<part_grid(n), kT, 0, s>>>(idx, t, blocks, refs, cap_refs, ops_nib, ops_first, out,
                                                           out_cap);
                launches++;
            }
        }
        if (!with_ops) {
            const unsigned grid = unsigned(std::min<uint64_t>(uint64_t(max_blocks(n)) * kBitmapParts, kGrid));
            k_write_bitmap<<<grid, kT, 0, s>>>(bits, (n + 63) / 64, n, t, blocks, bsum, chunks(n), cap_refs, out,
                                               out_cap);
            launches++;
        }
        CD_CUDA(cudaGetLastError());
        return PSB_OK;
    }

private:
    static constexpr unsigned kGrid = 148 * 8;  // grids of kernels that loop over items
    unsigned part_grid(uint64_t n) const {
        return unsigned(std::min<uint64_t>(uint64_t(std::min(cap_refs, max_blocks(n))) * kParts, kGrid));
    }
};

// Bit t of the result = bit 2t of x (t < 32): the even bits, packed.
__device__ __forceinline__ uint64_t even_bits(uint64_t x) {
    x &= 0x5555555555555555ull;
    x = (x | (x >> 1)) & 0x3333333333333333ull;
    x = (x | (x >> 2)) & 0x0F0F0F0F0F0F0F0Full;
    x = (x | (x >> 4)) & 0x00FF00FF00FF00FFull;
    x = (x | (x >> 8)) & 0x0000FFFF0000FFFFull;
    return (x | (x >> 16)) & 0x00000000FFFFFFFFull;
}

// Bit t of the result = bit 4t of x (t < 16).
__device__ __forceinline__ uint64_t every_fourth_bit(uint64_t x) {
    x &= 0x1111111111111111ull;
    x = (x | (x >> 3)) & 0x0303030303030303ull;
    x = (x | (x >> 6)) & 0x000F000F000F000Full;
    x = (x | (x >> 12)) & 0x000000FF000000FFull;
    return (x | (x >> 24)) & 0x000000000000FFFFull;
}

// Frontier bitmap of a two-bit array segment: states whose code is `code`
// (InMemoryTwoBitBFS.cpp:6-20 layout: bit 2i = code / 2, bit 2i+1 = code % 2).
// Out word j covers states first + 64 j .. + 63, i.e. code words
// 2 (first/64 + j) + {0, 1}.  One CTA per chunk of kChunkWords out words, whose
// popcount goes to sums[chunk] (the encoder's chunk sums); codes past the
// last state are 0 and never match.
// With active-window flags (one byte per 2^wb states, a superset of the
// windows holding the depth's states), a chunk none of whose windows is
// flagged is empty: it counts 0 and its words are left unwritten.
__device__ __forceinline__ bool chunk_flagged(const uint8_t* flags, int wb, uint64_t n_windows, uint64_t first,
                                              uint64_t n_out, uint64_t base) {
    if (!flags) return true;
    const uint64_t s0 = first + base * 64;
    const uint64_t end_out = base + kChunkWords < n_out ? base + kChunkWords : n_out;
    const uint64_t s1 = first + end_out * 64 - 1;
    const uint64_t w0 = s0 >> wb, w1 = (s1 >> wb) < n_windows ? (s1 >> wb) : n_windows - 1;
    int any = 0;
    for (uint64_t w = w0 + threadIdx.x; w <= w1; w += kT) any |= flags[w];
    return __syncthreads_or(any) != 0;
}

__global__ void __launch_bounds__(kT) k_frontier_two_bit(const uint64_t* __restrict__ codes, uint64_t first,
                                                          uint64_t n_out, uint32_t code, uint64_t* __restrict__ out,
                                                          unsigned long long* __restrict__ sums,
                                                          const uint8_t* __restrict__ flags, int wb,
                                                          uint64_t n_windows) {
    const uint64_t hi_sel = (code & 2) ? 0 : ~uint64_t(0), lo_sel = (code & 1) ? 0 : ~uint64_t(0);
    const uint64_t base = uint64_t(blockIdx.x) * kChunkWords;
    if (!chunk_flagged(flags, wb, n_windows, first, n_out, base)) {
        if (threadIdx.x == 0) sums[blockIdx.x] = 0;
        return;
    }
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < kCW; ++k) {
        const uint64_t j = base + uint64_t(k) * kT + threadIdx.x;
        if (j < n_out) {
            const uint64_t w = 2 * (first / 64 + j);
            const uint64_t a = codes[w], b = codes[w + 1];
            const uint64_t ma = (a ^ hi_sel) & ((a >> 1) ^ lo_sel);
            const uint64_t mb = (b ^ hi_sel) & ((b >> 1) ^ lo_sel);
            const uint64_t v = even_bits(ma) | (even_bits(mb) << 32);
            out[j] = v;
            c += __popcll(v);
        }
    }
    chunk_total(c, sums + blockIdx.x);
}

// Frontier bitmap of a frontier-search segment: states whose four operator
// bits are not all zero (InMemoryFrontierSearch.cpp:57-112), less the states
// of `excl` (the previous level's, on puzzles with odd cycles; may be NULL).
// Same CTA layout and chunk sums as k_frontier_two_bit.
__global__ void __launch_bounds__(kT) k_frontier_nibbles(const uint64_t* __restrict__ nib,
                                                          const uint64_t* __restrict__ excl, uint64_t first,
                                                          uint64_t n_out, uint64_t* __restrict__ out,
                                                          unsigned long long* __restrict__ sums) {
    const uint64_t base = uint64_t(blockIdx.x) * kChunkWords;
    uint32_t c = 0;
    for (int k = 0; k < kCW; ++k) {
        const uint64_t j = base + uint64_t(k) * kT + threadIdx.x;
        if (j < n_out) {
            const uint64_t w = 4 * (first / 64 + j);
            uint64_t v = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t x = nib[w + q];
                v |= every_fourth_bit(x | (x >> 1) | (x >> 2) | (x >> 3)) << (16 * q);
            }
            if (excl) v &= ~excl[first / 64 + j];
            out[j] = v;
            c += __popcll(v);
        }
    }
    chunk_total(c, sums + blockIdx.x);
}

unsigned chunks_of(uint64_t n_out) { return unsigned((n_out + kChunkWords - 1) / kChunkWords); }

int frontier_bits_two_bit(const uint64_t* codes, uint64_t first_state, uint64_t n_states, uint32_t code,
                          uint64_t* out, unsigned long long* sums, const uint8_t* flags, int window_bits,
                          uint64_t n_windows, cudaStream_t s) {
    const uint64_t n_out = (n_states + 63) / 64;
    k_frontier_two_bit<<<chunks_of(n_out), kT, 0, s>>>(codes, first_state, n_out, code, out, sums, flags,
                                                        window_bits, n_windows);
    CD_CUDA(cudaGetLastError());
    return PSB_OK;
}

int frontier_bits_nibbles(const uint64_t* nibbles, const uint64_t* excl, uint64_t first_state, uint64_t n_states,
                          uint64_t* out, unsigned long long* sums, cudaStream_t s) {
    const uint64_t n_out = (n_states + 63) / 64;
    k_frontier_nibbles<<<chunks_of(n_out), kT, 0, s>>>(nibbles, excl, first_state, n_out, out, sums);
    CD_CUDA(cudaGetLastError());
    return PSB_OK;
}

// OpBitsCompression<BITS> (Common/OpBitsCompression.cpp:10-76): each group of
// 8 op-bit bytes (a little-endian u64 `all`) packs into BITS bytes,
//   BITS 2: u16 (all | all >> 14 | all >> 28 | all >> 42)
//   BITS 4: u32 (all | all >> 28)   (also StreamVInt's bounds, StreamVInt.cpp:139-147)
//   BITS 8: unchanged.
// One thread per group: one 8-byte load, one BITS-byte store.
template <int BITS>
__global__ void k_opbits_encode(const uint64_t* __restrict__ in, uint64_t groups, uint8_t* __restrict__ out) {
    for (uint64_t g = blockIdx.x * uint64_t(kT) + threadIdx.x; g < groups; g += uint64_t(gridDim.x) * kT) {
        const uint64_t all = in[g];
        if constexpr (BITS == 2) reinterpret_cast<uint16_t*>(out)[g] = uint16_t(all | (all >> 14) | (all >> 28) | (all >> 42));
        else if constexpr (BITS == 4) reinterpret_cast<uint32_t*>(out)[g] = uint32_t(all | (all >> 28));
        else reinterpret_cast<uint64_t*>(out)[g] = all;
    }
}
template <int BITS>
__global__ void k_opbits_decode(const uint8_t* __restrict__ in, uint64_t groups, uint64_t* __restrict__ out) {
    for (uint64_t g = blockIdx.x * uint64_t(kT) + threadIdx.x; g < groups; g += uint64_t(gridDim.x) * kT) {
        uint64_t all;
        if constexpr (BITS == 2) {
            const uint64_t st = reinterpret_cast<const uint16_t*>(in)[g];
            all = (st & 0x0303ull) | ((st & 0x0C0Cull) << 14) | ((st & 0x3030ull) << 28) | ((st & 0xC0C0ull) << 42);
        } else if constexpr (BITS == 4) {
            const uint64_t st = reinterpret_cast<const uint32_t*>(in)[g];
            all = (st & 0x0F0F0F0Full) | ((st & 0xF0F0F0F0ull) << 28);
        } else {
            all = reinterpret_cast<const uint64_t*>(in)[g];
        }
        out[g] = all;
    }
}

SegmentEncoder* encoder_create() { return new (std::nothrow) SegmentEncoder(); }
void encoder_destroy(SegmentEncoder* e) { delete e; }

int encoder_begin(SegmentEncoder* e, uint64_t n_bits, uint32_t slots, cudaStream_t s, unsigned long long** sums) {
    if (int rc = e->reserve(n_bits, s)) return rc;
    if (int rc = e->reserve_totals(slots, s)) return rc;
    *sums = e->bsum;
    return PSB_OK;
}

int encoder_segment(SegmentEncoder* e, const uint64_t* d_bits, uint64_t n_bits, bool sums_ready, uint32_t slot,
                    uint64_t first_off, uint8_t* out, uint64_t out_cap, cudaStream_t s) {
    if (int rc = e->plan(d_bits, n_bits, sums_ready, slot, s)) return rc;
    if (int rc = e->layout(d_bits, n_bits, slot, slot == 0, first_off, s)) return rc;
    return e->write(d_bits, n_bits, slot, out, out_cap, s);
}

int encoder_totals(SegmentEncoder* e, uint32_t slots, EncTotals* host, bool* complete, cudaStream_t s) {
    CD_CUDA(cudaMemcpyAsync(host, e->totals, slots * sizeof(EncTotals), cudaMemcpyDeviceToHost, s));
    CD_CUDA(cudaStreamSynchronize(s));
    uint32_t most = 0;
    for (uint32_t i = 0; i < slots; ++i) most = std::max(most, host[i].n_refs);
    *complete = most <= e->cap_refs;
    return *complete ? PSB_OK : e->reserve_lists(most + most / 4, s);
}

void encoder_set_ops(SegmentEncoder* e, bool on, const uint64_t* nibbles, uint64_t first_state) {
    e->with_ops = on;
    e->ops_nib = nibbles;
    e->ops_first = first_state;
}

uint64_t encoder_take_launches(SegmentEncoder* e) {
    const uint64_t n = e->launches;
    e->launches = 0;
    return n;
}

}  // namespace psb

extern "C" int psb_frontier_encode(const uint64_t* d_bits, uint64_t first_bit, uint64_t n_bits, uint8_t* d_out,
                                   uint64_t out_cap, uint64_t* out_bytes, psb_codec_block* blocks,
                                   uint32_t blocks_cap, uint32_t* n_blocks, void* stream) {
    if (!d_bits || !out_bytes || !n_blocks) return psb_set_error(PSB_ERR_ARG, "bad argument");
    if (first_bit & 63) return psb_set_error(PSB_ERR_ARG, "first_bit must be a multiple of 64");
    if (n_bits > (uint64_t(1) << 32)) return psb_set_error(PSB_ERR_ARG, "a segment holds at most 2^32 states");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    *out_bytes = 0;
    *n_blocks = 0;
    if (n_bits == 0) return PSB_OK;
    const uint64_t* bits = d_bits + first_bit / 64;
    psb::SegmentEncoder E;
    // Scratch goes back to the pool in stream order, whatever the outcome.
    struct Release { psb::SegmentEncoder& e; cudaStream_t s; ~Release() { e.release(s); } } release{E, s};
    if (int rc = E.reserve(n_bits, s)) return rc;
    if (int rc = E.reserve_totals(1, s)) return rc;
    if (int rc = E.plan(bits, n_bits, false, 0, s)) return rc;
    EncTotals t{};
    CD_CUDA(cudaMemcpyAsync(&t, E.totals, sizeof t, cudaMemcpyDeviceToHost, s));
    CD_CUDA(cudaStreamSynchronize(s));
    if (t.count == 0) return PSB_OK;  // an empty segment writes nothing (CompressedSegmentWriter)
    // The offset list has its exact size now.
    if (int rc = E.reserve_lists(t.n_refs, s)) return rc;
    if (int rc = E.layout(bits, n_bits, 0, true, 0, s)) return rc;
    const bool table = blocks && blocks_cap >= t.nb;
    if (d_out && (!blocks || table))  // written only if it fits
        if (int rc = E.write(bits, n_bits, 0, d_out, out_cap, s)) return rc;
    std::vector<BlockInfo> hb(table ? t.nb : 0);
    if (table)
        CD_CUDA(cudaMemcpyAsync(hb.data(), E.blocks, hb.size() * sizeof(BlockInfo), cudaMemcpyDeviceToHost, s));
    CD_CUDA(cudaMemcpyAsync(&t, E.totals, sizeof t, cudaMemcpyDeviceToHost, s));
    CD_CUDA(cudaStreamSynchronize(s));
    *out_bytes = t.bytes;
    *n_blocks = t.nb;
    if (blocks && !table) return psb_set_error(PSB_ERR_CAPACITY, "blocks table too small");
    for (size_t b = 0; b < hb.size(); b++)
        blocks[b] = psb_codec_block{hb[b].out_off, hb[b].count, uint32_t(hb[b].bytes), hb[b].first, hb[b].is_bitmap};
    if (!d_out || out_cap < t.bytes) return psb_set_error(PSB_ERR_CAPACITY, "output needs more bytes (see *out_bytes)");
    return PSB_OK;
}

extern "C" int psb_frontier_index(const uint8_t* in, uint64_t in_bytes, psb_codec_block* blocks, uint32_t cap,
                                  uint32_t* n) {
    if (!n || (!in && in_bytes)) return psb_set_error(PSB_ERR_ARG, "bad argument");
    uint64_t pos = 0;
    uint32_t k = 0;
    auto u32 = [&](uint64_t at) {
        return uint32_t(in[at]) | (uint32_t(in[at + 1]) << 8) | (uint32_t(in[at + 2]) << 16) | (uint32_t(in[at + 3]) << 24);
    };
    while (pos < in_bytes) {
        if (pos + 4 > in_bytes) return psb_set_error(PSB_ERR_ARG, "truncated block header");
        const uint32_t h = u32(pos);
        psb_codec_block b{};
        b.offset = pos;
        if (h & kMap) {
            if (pos + 8 > in_bytes) return psb_set_error(PSB_ERR_ARG, "truncated bitmap header");
            const uint64_t words = h & ~kMap;
            b.is_bitmap = 1;
            b.first = u32(pos + 4);
            const uint64_t size = 8 + words * 8;
            if (pos + size > in_bytes) return psb_set_error(PSB_ERR_ARG, "truncated bitmap block");
            uint32_t c = 1;
            for (uint64_t i = 0; i < words * 8; i++) c += __builtin_popcount(in[pos + 8 + i]);
            b.count = c;
            b.bytes = uint32_t(size);
        } else {
            b.count = h;
            const uint64_t tuples = (uint64_t(h) + 7) / 8 * 2;
            uint64_t q = pos + 4;
            for (uint64_t t = 0; t < tuples; t++) {
                if (q >= in_bytes) return psb_set_error(PSB_ERR_ARG, "truncated StreamVInt block");
                const uint8_t d = in[q];
                q += 1 + 4 + (d & 3) + ((d >> 2) & 3) + ((d >> 4) & 3) + ((d >> 6) & 3);
            }
            if (q > in_bytes) return psb_set_error(PSB_ERR_ARG, "truncated StreamVInt block");
            if (h) {  // first value: the first delta of the first tuple
                const uint8_t d = in[pos + 4];
                uint32_t v = 0;
                for (int i = 0; i <= (d & 3); i++) v |= uint32_t(in[pos + 5 + i]) << (8 * i);
                b.first = v;
            }
            b.bytes = uint32_t(q - pos);
        }
        if (blocks) {
            if (k >= cap) return psb_set_error(PSB_ERR_CAPACITY, "blocks table too small");
            blocks[k] = b;
        }
        k++;
        pos += b.bytes;
    }
    *n = k;
    return PSB_OK;
}

namespace {
int opbits_check(int bits, const void* in, uint64_t count, const void* out) {
    if (bits != 2 && bits != 4 && bits != 8) return psb_set_error(PSB_ERR_ARG, "bits must be 2, 4 or 8");
    if (count & 7) return psb_set_error(PSB_ERR_ARG, "count must be a multiple of 8");
    if (count && (!in || !out)) return psb_set_error(PSB_ERR_ARG, "bad argument");
    return PSB_OK;
}
unsigned opbits_grid(uint64_t groups) {
    return unsigned(std::min<uint64_t>((groups + kT - 1) / kT, 148ull * 16));
}
}  // namespace

extern "C" int psb_opbits_encode(int bits, const uint8_t* d_op_bits, uint64_t count, uint8_t* d_out, void* stream) {
    if (int rc = opbits_check(bits, d_op_bits, count, d_out)) return rc;
    if (reinterpret_cast<uintptr_t>(d_op_bits) % 8 || reinterpret_cast<uintptr_t>(d_out) % bits)
        return psb_set_error(PSB_ERR_ARG, "op bits must be 8-byte aligned and the output aligned to `bits` bytes");
    const uint64_t groups = count / 8;
    if (!groups) return PSB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint64_t* in = reinterpret_cast<const uint64_t*>(d_op_bits);
    if (bits == 2) psb::k_opbits_encode<2><<<opbits_grid(groups), kT, 0, s>>>(in, groups, d_out);
    else if (bits == 4) psb::k_opbits_encode<4><<<opbits_grid(groups), kT, 0, s>>>(in, groups, d_out);
    else psb::k_opbits_encode<8><<<opbits_grid(groups), kT, 0, s>>>(in, groups, d_out);
    CD_CUDA(cudaGetLastError());
    return PSB_OK;
}

extern "C" int psb_opbits_decode(int bits, const uint8_t* d_in, uint64_t count, uint8_t* d_op_bits, void* stream) {
    if (int rc = opbits_check(bits, d_in, count, d_op_bits)) return rc;
    if (reinterpret_cast<uintptr_t>(d_op_bits) % 8 || reinterpret_cast<uintptr_t>(d_in) % bits)
        return psb_set_error(PSB_ERR_ARG, "op bits must be 8-byte aligned and the input aligned to `bits` bytes");
    const uint64_t groups = count / 8;
    if (!groups) return PSB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint64_t* out = reinterpret_cast<uint64_t*>(d_op_bits);
    if (bits == 2) psb::k_opbits_decode<2><<<opbits_grid(groups), kT, 0, s>>>(d_in, groups, out);
    else if (bits == 4) psb::k_opbits_decode<4><<<opbits_grid(groups), kT, 0, s>>>(d_in, groups, out);
    else psb::k_opbits_decode<8><<<opbits_grid(groups), kT, 0, s>>>(d_in, groups, out);
    CD_CUDA(cudaGetLastError());
    return PSB_OK;
}
