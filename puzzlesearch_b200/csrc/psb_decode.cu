// psb_decode.cu -- frontier streams back into bitmaps (the formats are
// described in psb_codec.cu):
//   FrontierCompression::Decode   Common/FrontierCompression.cpp:60-125
//   StreamVInt::Decode            Common/StreamVInt.cpp:132-145
//
// A StreamVInt block is a chain: each descriptor byte gives its tuple's
// length (5..17 bytes), so where a tuple starts depends on every tuple
// before it.  Walking a block's descriptors on one thread took 22 ms for a
// 2^28-state segment of 5.4 M offsets (65,536 dependent loads per block of
// 262,144 offsets).  Here the bytes of a block are cut into tiles of 16 KB
// and pieces of 64 bytes.  A tuple that begins before a piece's end reaches
// at most 16 bytes past it, so what a piece does to the chain is a map from
// 17 entry offsets to 17 exit offsets; it is found for all entries at once
// by one backward pass over the piece's bytes (the exit from byte p is the
// exit from p + length(p)).  Maps compose, so:
//   k_tile_maps    every tile's map, 64 bytes per thread;
//   k_tile_entries each block's tiles in order: their entries (a lookup per 16 KB);
//   k_tile_sums    every piece's entry, its tuples and the sum of its deltas;
//   k_tile_bases   each block's tiles in order: first tuple and value of each;
//   k_tile_marks   every piece's values, set in the bitmap.
// All launches cover the stream's bytes, whatever the number of blocks.
// Bitmap blocks are tiles of the last launch only.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "../../include/psb200.h"
#include "psb_internal.h"

namespace {

constexpr uint32_t kPiece = 64;                  // bytes per thread
constexpr uint32_t kDT = 256;                    // threads per tile
constexpr uint32_t kTile = kPiece * kDT;         // bytes per tile
constexpr uint32_t kEntries = 17;                // entry offsets 0 .. 16
constexpr uint32_t kMapStride = 32;              // bytes per tile map
constexpr uint32_t kStageWords = kTile / 4 + 5;  // a tuple reaches 16 bytes past its tile

#define DC_CUDA(call)                                                                           \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return psb_set_error(e_ == cudaErrorMemoryAllocation ? PSB_ERR_NOMEM : PSB_ERR_CUDA, \
                                 (std::string(#call) + ": " + cudaGetErrorString(e_)).c_str());  \
    } while (0)

// Where a piece's chain enters, and the tuples and delta sum before it in its tile.
struct PieceInfo {
    uint32_t sum;
    uint16_t tuples;
    uint16_t entry;
};
struct TileInfo {
    uint32_t sum, tuples;  // of the tile, then (k_tile_bases) before it in its block
};

// Staged bytes are padded by 4 per 64, so that the pieces of a warp's threads
// start in different banks.
__device__ __forceinline__ uint32_t staged(uint32_t x) { return x + ((x >> 6) << 2); }
constexpr uint32_t kStageBytes = kStageWords * 4 + (kStageWords * 4 / 64 + 1) * 4;

// The aligned word at w, bytes outside [lo, hi) as 0 and not read.
__device__ __forceinline__ uint32_t word_in(const uint8_t* w, const uint8_t* lo, const uint8_t* hi) {
    if (w >= lo && w + 4 <= hi) return __ldg(reinterpret_cast<const uint32_t*>(w));
    uint32_t v = 0;
    for (int q = 0; q < 4; ++q)
        if (w + q >= lo && w + q < hi) v |= uint32_t(w[q]) << (8 * q);
    return v;
}

// Stages kStageWords words of stream bytes from src (any alignment) on;
// bytes at or past hi are 0.
__device__ __forceinline__ void stage(uint32_t* sw, const uint8_t* src, const uint8_t* hi) {
    const uint32_t mis = uint32_t(reinterpret_cast<uintptr_t>(src) & 3u);
    const uint8_t* base = src - mis;
    for (uint32_t j = threadIdx.x; j < kStageWords; j += kDT) {
        const uint32_t w0 = word_in(base + 4ull * j, src, hi);
        const uint32_t w1 = mis ? word_in(base + 4ull * j + 4, src, hi) : 0;
        sw[j + (j >> 4)] = __funnelshift_r(w0, w1, 8 * mis);
    }
}

__device__ __forceinline__ uint32_t tuple_bytes(uint32_t desc) {
    const uint32_t t = (desc & 0x33u) + ((desc >> 2) & 0x33u);
    return 5u + (t & 15u) + (t >> 4);
}

// The block of tile t: the last b with first[b] <= t (blocks without tiles
// share their successor's first tile and are passed over).
__device__ __forceinline__ uint32_t block_of(const uint32_t* first, uint32_t n_blocks, uint32_t t) {
    uint32_t lo = 0, hi = n_blocks;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (first[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// A tile's bytes of a StreamVInt block's tuples: [begin, end) is what is left
// of the block from the tile on.
struct TileBytes {
    const uint8_t *begin, *end;
    __device__ __forceinline__ TileBytes(const uint8_t* in, const psb_codec_block& bk, uint32_t tile_in_block)
        : begin(in + bk.offset + 4 + uint64_t(tile_in_block) * kTile), end(in + bk.offset + bk.bytes) {}
    __device__ __forceinline__ uint32_t left() const {
        return uint32_t(min((unsigned long long)(end - begin), (unsigned long long)(kTile + 32)));
    }
};

// exits[staged(p)] = where the chain through byte p leaves p's piece (0 .. 16).
__device__ __forceinline__ void piece_exits(const uint32_t* sw, uint8_t* exits) {
    uint8_t* ex = exits + threadIdx.x * (kPiece + 4);
    const uint32_t* w = sw + threadIdx.x * (kPiece / 4 + 1);
    for (int k = int(kPiece / 4) - 1; k >= 0; --k) {
        const uint32_t v = w[k];
#pragma unroll
        for (int q = 3; q >= 0; --q) {
            const uint32_t p = 4u * k + q, nx = p + tuple_bytes((v >> (8 * q)) & 255u);
            ex[p] = nx >= kPiece ? uint8_t(nx - kPiece) : ex[nx];
        }
    }
}

// Lanes 0 .. 16 of each warp: the exit of the warp's 32 pieces for entry `lane`.
__device__ __forceinline__ void warp_map(const uint8_t* exits, uint8_t (*maps)[kMapStride]) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    __syncwarp();
    if (lane < kEntries) {
        uint32_t e = lane;
        for (uint32_t t = 0; t < 32; ++t) e = exits[(warp * 32 + t) * (kPiece + 4) + e];
        maps[warp][lane] = uint8_t(e);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kDT) k_tile_maps(const uint8_t* __restrict__ in, const psb_codec_block* blocks,
                                                   uint32_t n_blocks, const uint32_t* first, uint8_t* tile_maps) {
    __shared__ uint32_t sw[kStageBytes / 4];
    __shared__ uint8_t exits[kDT * (kPiece + 4)];
    __shared__ uint8_t maps[kDT / 32][kMapStride];
    const uint32_t b = block_of(first, n_blocks, blockIdx.x);
    const psb_codec_block bk = blocks[b];
    if (bk.is_bitmap) return;
    const TileBytes tb(in, bk, blockIdx.x - first[b]);
    stage(sw, tb.begin, tb.end);
    __syncthreads();
    piece_exits(sw, exits);
    warp_map(exits, maps);
    if (threadIdx.x < kEntries) {
        uint32_t e = threadIdx.x;
        for (uint32_t w = 0; w < kDT / 32; ++w) e = maps[w][e];
        tile_maps[uint64_t(blockIdx.x) * kMapStride + threadIdx.x] = uint8_t(e);
    }
}

// One warp per block: entries[t] = the entry offset of each of its tiles.
__global__ void __launch_bounds__(32) k_tile_entries(const psb_codec_block* blocks, const uint32_t* first,
                                                     const uint8_t* tile_maps, uint8_t* entries) {
    __shared__ uint4 maps[32 * kMapStride / 16];
    if (blocks[blockIdx.x].is_bitmap) return;
    const uint32_t t0 = first[blockIdx.x], t1 = first[blockIdx.x + 1];
    uint32_t e = 0;
    for (uint32_t t = t0; t < t1; t += 32) {
        const uint32_t n = t1 - t < 32 ? t1 - t : 32;
        for (uint32_t i = threadIdx.x; i < n * kMapStride / 16; i += 32)
            maps[i] = reinterpret_cast<const uint4*>(tile_maps)[uint64_t(t) * (kMapStride / 16) + i];
        __syncwarp();
        if (threadIdx.x == 0) {
            for (uint32_t i = 0; i < n; ++i) {
                entries[t + i] = uint8_t(e);
                e = reinterpret_cast<const uint8_t*>(maps)[i * kMapStride + e];
            }
        }
        __syncwarp();
    }
}

// Little-endian value of n (1..4) staged bytes at x.
__device__ __forceinline__ uint32_t staged_value(const uint8_t* sb, uint32_t x, uint32_t n) {
    uint32_t v = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
        if (i < n) v |= uint32_t(sb[staged(x + i)]) << (8 * i);
    return v;
}

__global__ void __launch_bounds__(kDT) k_tile_sums(const uint8_t* __restrict__ in, const psb_codec_block* blocks,
                                                   uint32_t n_blocks, const uint32_t* first, const uint8_t* entries,
                                                   PieceInfo* pieces, TileInfo* tiles) {
    __shared__ uint32_t sw[kStageBytes / 4];
    __shared__ uint8_t exits[kDT * (kPiece + 4)];
    __shared__ uint8_t maps[kDT / 32][kMapStride];
    __shared__ uint8_t enter[kDT], warp_enter[kDT / 32];
    __shared__ uint32_t warp_sum[kDT / 32], warp_tuples[kDT / 32];
    const uint32_t b = block_of(first, n_blocks, blockIdx.x);
    const psb_codec_block bk = blocks[b];
    if (bk.is_bitmap) return;
    const TileBytes tb(in, bk, blockIdx.x - first[b]);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    stage(sw, tb.begin, tb.end);
    __syncthreads();
    piece_exits(sw, exits);
    warp_map(exits, maps);
    if (threadIdx.x == 0) {
        uint32_t e = entries[blockIdx.x];
        for (uint32_t w = 0; w < kDT / 32; ++w) {
            warp_enter[w] = uint8_t(e);
            e = maps[w][e];
        }
    }
    __syncthreads();
    if (lane == 0) {
        uint32_t e = warp_enter[warp];
        for (uint32_t t = 0; t < 32; ++t) {
            enter[warp * 32 + t] = uint8_t(e);
            e = exits[(warp * 32 + t) * (kPiece + 4) + e];
        }
    }
    __syncwarp();
    // This piece's tuples and the sum of their deltas; a tuple that the
    // block's bytes cut short ends the chain.
    const uint8_t* sb = reinterpret_cast<const uint8_t*>(sw);
    const uint32_t p0 = threadIdx.x * kPiece, p1 = p0 + kPiece, left = tb.left();
    uint32_t sum = 0, n = 0;
    for (uint32_t p = p0 + enter[threadIdx.x]; p < p1 && p < left;) {
        const uint32_t desc = sb[staged(p)], len = tuple_bytes(desc);
        if (p + len > left) break;
        uint32_t x = p + 1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t nb = 1u + ((desc >> (2 * q)) & 3u);
            sum += staged_value(sb, x, nb);
            x += nb;
        }
        ++n;
        p += len;
    }
    // Exclusive scan over the tile's pieces.
    uint32_t isum = sum, in_ = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t s = __shfl_up_sync(0xFFFFFFFFu, isum, o), t = __shfl_up_sync(0xFFFFFFFFu, in_, o);
        if (lane >= uint32_t(o)) {
            isum += s;
            in_ += t;
        }
    }
    if (lane == 31) {
        warp_sum[warp] = isum;
        warp_tuples[warp] = in_;
    }
    __syncthreads();
    uint32_t bsum = 0, btuples = 0;
    for (uint32_t w = 0; w < warp; ++w) {
        bsum += warp_sum[w];
        btuples += warp_tuples[w];
    }
    pieces[uint64_t(blockIdx.x) * kDT + threadIdx.x] =
        PieceInfo{bsum + isum - sum, uint16_t(btuples + in_ - n), uint16_t(enter[threadIdx.x])};
    if (threadIdx.x == kDT - 1) tiles[blockIdx.x] = TileInfo{bsum + isum, btuples + in_};
}

// One warp per block: tiles[t] becomes the sums of the block's tiles before
// t.  A chain of fewer tuples than the block's count is a stream shorter
// than its block table.
__global__ void __launch_bounds__(32) k_tile_bases(const psb_codec_block* blocks, const uint32_t* first,
                                                   TileInfo* tiles, unsigned long long* err) {
    const psb_codec_block bk = blocks[blockIdx.x];
    if (bk.is_bitmap) return;
    const uint32_t t0 = first[blockIdx.x], t1 = first[blockIdx.x + 1], lane = threadIdx.x;
    uint32_t sum = 0, tuples = 0;
    for (uint32_t t = t0; t < t1; t += 32) {
        const TileInfo own = t + lane < t1 ? tiles[t + lane] : TileInfo{0, 0};
        uint32_t s = own.sum, n = own.tuples;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o), z = __shfl_up_sync(0xFFFFFFFFu, n, o);
            if (lane >= uint32_t(o)) {
                s += y;
                n += z;
            }
        }
        if (t + lane < t1) tiles[t + lane] = TileInfo{sum + s - own.sum, tuples + n - own.tuples};
        sum += __shfl_sync(0xFFFFFFFFu, s, 31);
        tuples += __shfl_sync(0xFFFFFFFFu, n, 31);
    }
    if (lane == 0 && tuples < uint32_t((uint64_t(bk.count) + 7) / 8 * 2)) atomicOr(err, 1ull);
}

// Sets the values of a tile: a StreamVInt piece's running sums, which mostly
// fall in one or two words at a time, or the words of a bitmap block
// (kTile / 8 per tile), shifted to the segment's words.
__global__ void __launch_bounds__(kDT) k_tile_marks(const uint8_t* __restrict__ in, const psb_codec_block* blocks,
                                                    uint32_t n_blocks, const uint32_t* first,
                                                    const PieceInfo* pieces, const TileInfo* tiles, uint64_t* bits,
                                                    uint64_t n_bits, unsigned long long* err) {
    __shared__ uint32_t sw[kStageBytes / 4];
    const uint8_t* sb = reinterpret_cast<const uint8_t*>(sw);
    const uint32_t b = block_of(first, n_blocks, blockIdx.x);
    const psb_codec_block bk = blocks[b];
    const uint32_t tile = blockIdx.x - first[b];
    auto set_word = [&](uint64_t w, uint64_t m) {
        if (m) atomicOr(reinterpret_cast<unsigned long long*>(bits) + w, (unsigned long long)m);
    };
    if (bk.is_bitmap) {
        const uint8_t* p = in + bk.offset;
        if (bk.bytes < 8) {
            if (threadIdx.x == 0) atomicOr(err, 1ull);
            return;
        }
        auto u32 = [&](uint32_t at) {
            return uint32_t(p[at]) | (uint32_t(p[at + 1]) << 8) | (uint32_t(p[at + 2]) << 16) | (uint32_t(p[at + 3]) << 24);
        };
        const uint64_t words = u32(0) & 0x7FFFFFFFu;
        const uint64_t base = uint64_t(u32(4));
        if (8 + 8 * words > bk.bytes) {  // a stream shorter than its block table
            if (threadIdx.x == 0) atomicOr(err, 1ull);
            return;
        }
        if (tile == 0 && threadIdx.x == 0) {
            if (base < n_bits) set_word(base >> 6, uint64_t(1) << (base & 63));
            else atomicOr(err, 1ull);
        }
        stage(sw, p + 8 + uint64_t(tile) * kTile, p + 8 + 8 * words);
        __syncthreads();
        const uint64_t w0 = uint64_t(tile) * (kTile / 8);
        for (uint32_t i = threadIdx.x; i < kTile / 8 && w0 + i < words; i += kDT) {
            uint64_t v = sw[2 * i + (i >> 3)] | (uint64_t(sw[2 * i + 1 + (i >> 3)]) << 32);
            if (!v) continue;
            const uint64_t s0 = base + 1 + 64 * (w0 + i);  // state of bit 0
            if (s0 + 63 >= n_bits) {
                const uint64_t keep = s0 < n_bits ? ((uint64_t(1) << (n_bits - s0)) - 1) : 0;
                if (v & ~keep) atomicOr(err, 1ull);
                v &= keep;
            }
            const uint32_t sh = uint32_t(s0 & 63);
            set_word(s0 >> 6, v << sh);
            if (sh) set_word((s0 >> 6) + 1, v >> (64 - sh));
        }
        return;
    }
    const TileBytes tb(in, bk, tile);
    const TileInfo base = tiles[blockIdx.x];
    const PieceInfo pi = pieces[uint64_t(blockIdx.x) * kDT + threadIdx.x];
    stage(sw, tb.begin, tb.end);
    __syncthreads();
    const uint32_t p0 = threadIdx.x * kPiece, p1 = p0 + kPiece, left = tb.left();
    uint32_t cur = base.sum + pi.sum;
    uint64_t k = 4 * (uint64_t(base.tuples) + pi.tuples);
    uint64_t word = 0, mask = 0;
    bool bad = false;
    for (uint32_t p = p0 + pi.entry; p < p1 && p < left && k < bk.count;) {
        const uint32_t desc = sb[staged(p)], len = tuple_bytes(desc);
        if (p + len > left) break;
        uint32_t x = p + 1;
#pragma unroll
        for (int q = 0; q < 4; ++q, ++k) {
            const uint32_t nb = 1u + ((desc >> (2 * q)) & 3u);
            cur += staged_value(sb, x, nb);
            x += nb;
            if (k >= bk.count) continue;
            if (cur >= n_bits) {
                bad = true;
                continue;
            }
            if ((cur >> 6) != word) {
                set_word(word, mask);
                word = cur >> 6;
                mask = 0;
            }
            mask |= uint64_t(1) << (cur & 63);
        }
        p += len;
    }
    set_word(word, mask);
    if (bad) atomicOr(err, 1ull);
}

}  // namespace

namespace psb {

// Device scratch of the decoder, grown on demand and kept for the next call:
// one allocation of the device's pool, in stream order.
struct DecodeScratch {
    uint8_t* buf = nullptr;
    size_t cap = 0;
    cudaStream_t stream = nullptr;
    std::vector<uint8_t> h_table;  // the blocks, then each one's first tile

    int reserve(size_t need, cudaStream_t s) {
        if (need <= cap) return PSB_OK;
        cudaMemPool_t pool = nullptr;
        if (int rc = scratch_pool(&pool)) return rc;
        if (buf) DC_CUDA(cudaFreeAsync(buf, stream));
        buf = nullptr;
        cap = 0;
        stream = s;
        DC_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&buf), need + need / 4, pool, s));
        cap = need + need / 4;
        return PSB_OK;
    }
    ~DecodeScratch() { if (buf) cudaFreeAsync(buf, stream); }
};
DecodeScratch* decoder_create() { return new (std::nothrow) DecodeScratch(); }
void decoder_destroy(DecodeScratch* d) { delete d; }

int frontier_decode_async(const uint8_t* d_in, const psb_codec_block* h_blocks, uint32_t n_blocks, uint64_t* d_bits,
                          uint64_t n_bits, unsigned long long* d_err, DecodeScratch* x, cudaStream_t s) {
    if (n_blocks == 0) return PSB_OK;
    // Tiles per block (none for a StreamVInt block without tuples).
    size_t need = 0;
    auto part = [&](size_t bytes) {
        const size_t at = need;
        need += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t at_blocks = part(size_t(n_blocks) * sizeof(psb_codec_block));
    const size_t at_first = part((size_t(n_blocks) + 1) * 4);
    const size_t table = need;
    x->h_table.resize(table);
    std::memcpy(x->h_table.data() + at_blocks, h_blocks, size_t(n_blocks) * sizeof(psb_codec_block));
    uint32_t* const h_first = reinterpret_cast<uint32_t*>(x->h_table.data() + at_first);
    uint64_t n_tiles = 0;
    bool any_svi = false;
    for (uint32_t b = 0; b < n_blocks; ++b) {
        h_first[b] = uint32_t(n_tiles);
        const uint64_t head = h_blocks[b].is_bitmap ? 8 : 4;
        const uint64_t left = h_blocks[b].bytes > head ? h_blocks[b].bytes - head : 0;
        uint64_t tiles = (left + kTile - 1) / kTile;
        if (h_blocks[b].is_bitmap) tiles = std::max<uint64_t>(tiles, 1);  // the first offset is in the header
        else any_svi = true;
        n_tiles += tiles;
        if (n_tiles > 0x7FFFFFFFull) return psb_set_error(PSB_ERR_ARG, "stream too large");
    }
    h_first[n_blocks] = uint32_t(n_tiles);
    const size_t at_maps = part(n_tiles * kMapStride), at_entries = part(n_tiles);
    const size_t at_pieces = part(n_tiles * kDT * sizeof(PieceInfo)), at_tiles = part(n_tiles * sizeof(TileInfo));
    if (int rc = x->reserve(need, s)) return rc;
    auto* blocks = reinterpret_cast<psb_codec_block*>(x->buf + at_blocks);
    auto* first = reinterpret_cast<uint32_t*>(x->buf + at_first);
    auto* maps = x->buf + at_maps;
    auto* entries = x->buf + at_entries;
    auto* pieces = reinterpret_cast<PieceInfo*>(x->buf + at_pieces);
    auto* tiles = reinterpret_cast<TileInfo*>(x->buf + at_tiles);
    // Pageable source: the copy has left host memory when the call returns.
    DC_CUDA(cudaMemcpyAsync(x->buf, x->h_table.data(), table, cudaMemcpyHostToDevice, s));
    const unsigned grid = unsigned(n_tiles);
    if (any_svi) {
        if (grid) k_tile_maps<<<grid, kDT, 0, s>>>(d_in, blocks, n_blocks, first, maps);
        k_tile_entries<<<n_blocks, 32, 0, s>>>(blocks, first, maps, entries);
        if (grid) k_tile_sums<<<grid, kDT, 0, s>>>(d_in, blocks, n_blocks, first, entries, pieces, tiles);
        k_tile_bases<<<n_blocks, 32, 0, s>>>(blocks, first, tiles, d_err);
    }
    if (grid) k_tile_marks<<<grid, kDT, 0, s>>>(d_in, blocks, n_blocks, first, pieces, tiles, d_bits, n_bits, d_err);
    DC_CUDA(cudaGetLastError());
    return PSB_OK;
}
}  // namespace psb

extern "C" int psb_frontier_decode(const uint8_t* d_in, const psb_codec_block* blocks, uint32_t n_blocks,
                                   uint64_t* d_bits, uint64_t first_bit, uint64_t n_bits, void* stream) {
    if (!d_bits || (n_blocks && (!d_in || !blocks))) return psb_set_error(PSB_ERR_ARG, "bad argument");
    if (first_bit & 63) return psb_set_error(PSB_ERR_ARG, "first_bit must be a multiple of 64");
    if (n_blocks == 0) return PSB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    std::unique_ptr<psb::DecodeScratch> x(psb::decoder_create());
    if (!x) return psb_set_error(PSB_ERR_NOMEM, "decoder scratch");
    cudaMemPool_t pool = nullptr;
    if (int rc = psb::scratch_pool(&pool)) return rc;
    unsigned long long* d_err = nullptr;
    DC_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&d_err), 8, pool, s));
    unsigned long long err = 0;
    int rc = PSB_OK;
    cudaError_t e = cudaMemsetAsync(d_err, 0, 8, s);
    if (e == cudaSuccess)
        rc = psb::frontier_decode_async(d_in, blocks, n_blocks, d_bits + first_bit / 64, n_bits, d_err, x.get(), s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&err, d_err, 8, cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(d_err, s);
    x.reset();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    DC_CUDA(e);
    if (rc) return rc;
    if (err) return psb_set_error(PSB_ERR_ARG, "a decoded offset lies outside the segment");
    return PSB_OK;
}
