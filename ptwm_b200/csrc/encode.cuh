// Device code of the encode path: forward bit reorder + plane split, per-chunk
// histograms, per-chunk table build, per-stream rANS / Huffman encoding and
// the gather that lays chunk frames out in the container.
//
// Byte-exact targets under crates/ptwm-core/src of the reference:
//   split      transforms/fusion.rs:35-122,207-262,329-371,431-473
//   rANS       entropy/rans/compress.rs:35-259
//   Huffman    entropy/huffman/{compress.rs:9-103, bitstream.rs:3-51, weights.rs:8-32}
//   tANS       entropy/tans/mod.rs:199-339
//   O1SAC      codecs/order1_scale_ac.rs:620-663,963-1025, quantize.rs:13-45, range_coder.rs:16-113
//   framing    compressor.rs:316-381, codecs/{huffman,rans,tans}.rs encode
#pragma once
#include <cooperative_groups.h>

#include "encode_tables.cuh"
#include "kernels.cuh"

namespace ptwm {

constexpr uint64_t ENC_PAD = 64;  // bytes behind the planes and the slots that a 16-byte access may reach

struct EncChunk {
    uint64_t plane_off;  // this chunk's bytes in the planes buffer
    uint64_t slot_off;   // four stream slots of slot_cap bytes each in the slot buffer (tANS / O1SAC: one stream over all four)
    uint64_t table_off;  // this chunk's area in the table buffer (size by codec, see below)
    uint32_t n;
    uint32_t slot_cap;
    uint32_t plane;      // global plane index
    uint32_t row_len;    // O1SAC: symbols per row (context resets at row starts); 0 = one row spanning the chunk
};
struct EncResult {       // per chunk, read back by the host
    uint32_t stream_len[4];  // tANS: [0] bytes of bits, [1..2] total bits (lo, hi); O1SAC: [0] payload bytes, [1] state bytes
    uint32_t hdr_n;      // rANS: max_sym; Huffman: number of weights; tANS: present symbols; O1SAC: context rows
    uint32_t coded;      // 0: no table could be built, store raw
};
// One plane as the host lays it out; chunk k of it starts k * chunk bytes into the plane.
struct EncPlane {
    uint64_t buf_off;    // the plane's bytes in the planes buffer
    uint64_t len, chunk;
    uint64_t slot_off, slot_stride, table_off;  // areas of the first chunk, distance between chunks
    uint32_t first_chunk, n_chunks;
    uint32_t table_bytes, row_len;
    uint32_t codec;
    uint32_t shared;     // Order1ScaleAC against a shared state: no state of its own
    uint32_t list_off;   // where the plane's chunks go in the encoders' lists, ENC_NO_LIST for nowhere
    uint32_t reserved;
};
constexpr uint32_t ENC_NO_LIST = 0xFFFFFFFFu;
__host__ __device__ inline uint32_t enc_slot_cap(uint64_t n) { return uint32_t((((n + 3) / 4) * 3 / 2 + 16 + 15) / 16 * 16); }  // <= 12 bits per symbol plus the rANS state
struct ChunkPlace {
    uint64_t frame;      // offset of the chunk frame from the plane's first
    uint32_t entry;      // offset of the chunk's entry in the plane's chunk table
    uint32_t mode;       // 0 identity (bare bytes), 1 raw-tagged, 2 rANS, 3 Huffman, 4 tANS, 5 Order1ScaleAC (state inside the frame);
                         // + GATHER_BARE: the payload alone, no chunk frame header (and no state)
};
struct PlaneSizes { uint64_t frames; uint32_t entries, state_len; };  // bytes of all frames / of the chunk table / of an unchunked Order1ScaleAC plane's state
struct PlaneDst { uint64_t frames, table; };                         // where they go in the container; frames = ENC_NOWHERE: the plane is not written
constexpr uint64_t ENC_NOWHERE = ~0ull;
constexpr uint32_t GATHER_BARE = 0x100;
constexpr uint32_t GATHER_NOFRAME = 0x200;  // an unchunked plane: inline state (if the codec has one) and payload, no frame header

// layout of the table area of a chunk (what the gather and the encoder need of it; the rest is rebuilt in shared memory)
//   rANS:    freqs u16[256]
//   Huffman: lengths u8[256] | codes u32[256]: reversed code | length << 16                 (1280 bytes)
//   tANS:    norm u16[256]
//   O1SAC:   joint counts u32[256][256] | row-start counts u32[256] | present u8[256] | rank u16[256] |
//            pmf u16[257][256] (row 0 marginal, row 1 + c for context c) | cum u16[257][256]
constexpr uint32_t ENC_FREQ_TABLE_BYTES = 512;
constexpr uint32_t ENC_HUFF_TABLE_BYTES = 256 + 1024;
constexpr uint32_t O1E_JOINT = 0, O1E_MARG = 262144, O1E_PRESENT = O1E_MARG + 1024, O1E_RANK = O1E_PRESENT + 256, O1E_PMF = O1E_RANK + 512,
                   O1E_CUM = O1E_PMF + 257 * 512, ENC_O1SAC_TABLE_BYTES = O1E_CUM + 257 * 512;
constexpr uint32_t O1SAC_TOTAL = 4096;
__host__ __device__ inline uint32_t enc_table_bytes(int codec) {
    return codec == C_HUFFMAN ? ENC_HUFF_TABLE_BYTES : codec == C_O1SAC ? ENC_O1SAC_TABLE_BYTES : ENC_FREQ_TABLE_BYTES;
}

__device__ __forceinline__ uint32_t warp_prefix(uint32_t v, uint32_t lane) {  // exclusive
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d); if (lane >= uint32_t(d)) incl += t; }
    return incl - v;
}

// Forward bit reorder and byte split, with the histogram of every plane taken on the way: a block owns a chunk of a tensor (or
// SPLIT_TILE elements of a longer one), reads its elements once and writes the planes' bytes.  Sixteen elements per thread and
// step where the source is 16-byte aligned: 128-bit loads, one 128-bit store per plane.  (Plane offsets are multiples of 16;
// the groups start at multiples of 16 elements of the tensor, what lies outside them at either end of the block's range goes
// element by element.)  Sixteen 16-bit elements are one 256-bit load where the source is 32-byte aligned: 203 -> 194 us for 0.44 GB of bf16, of
// which the bytes alone are 133 at the copy bandwidth.  Stores that take no place in the L1 would save 2 us more of that, but where the
// planes fit the L2 those who read them next lose more (bf16, 27 MB: rANS streams 613 -> 639 us, gather 15.5 -> 21.3).
//
// COPIES histograms per plane, laid out [symbol][copy], lane l counting in copy l mod COPIES: with 32 a lane has a bank of its
// own and no atomic waits for another lane's (eight copies took three passes: the lanes that share a copy mostly meet in the
// same few symbols of an exponent plane, or in the same bank).  Clearing and adding up 32 copies costs as much as counting
// 16 Ki symbols, so chunks below SPLIT_WIDE_FROM keep eight.  COPIES = 0: no counts.
struct SplitItem {
    const uint8_t* src;     // raw tensor bytes (device)
    uint64_t plane_off[4];  // where each plane starts in the planes buffer
    uint64_t n;             // elements (= bytes per plane)
    uint64_t chunk;         // elements per chunk
    uint32_t kind;
    uint32_t first_tile;
    uint32_t first_chunk[4];  // of each plane
};
constexpr uint32_t SPLIT_TILE = 32768, SPLIT_WIDE_FROM = 8192, SPLIT_THREADS = 512;
__host__ __device__ inline uint32_t split_tiles_per_chunk(uint64_t n, uint64_t chunk) { return uint32_t(((n < chunk ? n : chunk) + SPLIT_TILE - 1) / SPLIT_TILE); }
inline uint64_t split_tiles(uint64_t n, uint64_t chunk) { return (n + chunk - 1) / chunk * split_tiles_per_chunk(n, chunk); }
inline uint32_t split_smem_bytes(uint32_t planes, uint32_t copies) { return planes * copies * 1024; }

template <int COPIES>
__global__ void __launch_bounds__(SPLIT_THREADS) split_kernel(const SplitItem* __restrict__ items, uint32_t n_items, uint8_t* __restrict__ planes, uint32_t* __restrict__ hist) {
    extern __shared__ uint32_t counts[];
    uint32_t first = 0, after = n_items;
    while (first + 1 < after) { const uint32_t mid = (first + after) >> 1; if (items[mid].first_tile <= blockIdx.x) first = mid; else after = mid; }
    const SplitItem it = items[first];
    const uint32_t tile = blockIdx.x - it.first_tile, per_chunk = split_tiles_per_chunk(it.n, it.chunk), chunk = tile / per_chunk;
    const uint64_t chunk_at = uint64_t(chunk) * it.chunk, chunk_end = chunk_at + it.chunk < it.n ? chunk_at + it.chunk : it.n;
    const uint64_t begin = chunk_at + uint64_t(tile % per_chunk) * SPLIT_TILE;
    if (begin >= chunk_end) return;  // the last chunk of a tensor can have fewer tiles
    const uint64_t end = begin + SPLIT_TILE < chunk_end ? begin + SPLIT_TILE : chunk_end;
    const int np = kind_planes(int(it.kind)), eb = kind_elem_bytes(int(it.kind));
    if (COPIES) {
        for (uint32_t i = threadIdx.x; i < uint32_t(np) * 64 * COPIES; i += SPLIT_THREADS) reinterpret_cast<uint4*>(counts)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
    }
    auto count = [&](int p, uint32_t byte) { if (COPIES) atomicAdd(&counts[(uint32_t(p) * 256 + byte) * COPIES + (threadIdx.x & (COPIES - 1))], 1u); };
    auto count_words = [&](int p, const uint32_t w[4]) {
        if (COPIES) {
#pragma unroll
            for (int k = 0; k < 16; ++k) count(p, (w[k >> 2] >> (8 * (k & 3))) & 0xFFu);
        }
    };
    auto put = [&](int p, uint64_t at, const uint32_t w[4]) {
        *reinterpret_cast<uint4*>(planes + it.plane_off[p] + at) = make_uint4(w[0], w[1], w[2], w[3]);
        count_words(p, w);
    };
    auto one = [&](uint64_t i) {
        uint32_t r;
        switch (it.kind) {
            case K_PASS: r = it.src[i]; break;
            case K_M16: {
                const uint32_t v = uint32_t(it.src[2 * i]) | uint32_t(it.src[2 * i + 1]) << 8;
                r = ((v << 1) & 0xFF00u) | ((v >> 8) & 0x0080u) | (v & 0x007Fu);
                break;
            }
            case K_M32: {
                const uint32_t v = ld_u32_unaligned(it.src + 4 * i);
                r = ((v << 1) & 0xFF000000u) | ((v >> 8) & 0x00800000u) | (v & 0x007FFFFFu);
                break;
            }
            default: {  // plane 0 holds the high nibble
                const uint32_t v = it.src[i];
                const uint32_t x = it.kind == K_E4M3 ? (((v & 0x78) << 1) | ((v & 0x80) >> 4) | (v & 0x07)) : (((v & 0x7C) << 1) | ((v & 0x80) >> 5) | (v & 0x03));
                r = x >> 4 | (x & 0x0Fu) << 8;
                break;
            }
        }
        for (int p = 0; p < np; ++p) { planes[it.plane_off[p] + i] = uint8_t(r >> (8 * p)); count(p, (r >> (8 * p)) & 0xFFu); }
    };
    uint64_t lo = end, hi = end;  // whole groups of sixteen: [lo, hi)
    if ((reinterpret_cast<uintptr_t>(it.src) & 15) == 0) {
        lo = (begin + 15) & ~uint64_t(15); hi = end & ~uint64_t(15);
        if (lo >= hi) lo = hi = end;
    }
    for (uint64_t i = begin + threadIdx.x; i < lo; i += SPLIT_THREADS) one(i);
    for (uint64_t i = hi + threadIdx.x; i < end; i += SPLIT_THREADS) one(i);
    const uint32_t groups = uint32_t((hi - lo) >> 4);
    const uint4* src = reinterpret_cast<const uint4*>(it.src + lo * uint64_t(eb));
    const bool whole = (reinterpret_cast<uintptr_t>(src) & 31) == 0;  // a thread's sixteen 16-bit elements are one sector
    if (it.kind == K_M16) {
        for (uint32_t g = threadIdx.x; g < groups; g += SPLIT_THREADS) {
            uint32_t w[8];
            if (whole) {
                const Block32 b = ldg256(src + 2 * g);
#pragma unroll
                for (int k = 0; k < 8; ++k) w[k] = b.w[k];
            } else {
                const uint4 a = src[2 * g], b = src[2 * g + 1];
                w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
            }
            uint32_t l[4], h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // two words = four elements -> one word per plane
                const uint32_t r0 = ((w[2 * k] << 1) & 0xFF00FF00u) | ((w[2 * k] >> 8) & 0x00800080u) | (w[2 * k] & 0x007F007Fu);
                const uint32_t r1 = ((w[2 * k + 1] << 1) & 0xFF00FF00u) | ((w[2 * k + 1] >> 8) & 0x00800080u) | (w[2 * k + 1] & 0x007F007Fu);
                l[k] = __byte_perm(r0, r1, 0x6420);
                h[k] = __byte_perm(r0, r1, 0x7531);
            }
            put(0, lo + 16 * uint64_t(g), l);
            put(1, lo + 16 * uint64_t(g), h);
        }
    } else if (it.kind == K_M32) {
        for (uint32_t g = threadIdx.x; g < groups; g += SPLIT_THREADS) {
            uint32_t pl[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // four elements -> one word per plane
                const uint4 v = src[4 * g + q];
                const uint32_t e[4] = {v.x, v.y, v.z, v.w};
                uint32_t r[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) r[k] = ((e[k] << 1) & 0xFF000000u) | ((e[k] >> 8) & 0x00800000u) | (e[k] & 0x007FFFFFu);
                const uint32_t t0 = __byte_perm(r[0], r[1], 0x5140), t1 = __byte_perm(r[2], r[3], 0x5140);  // bytes 0,1 of the pairs
                const uint32_t t2 = __byte_perm(r[0], r[1], 0x7362), t3 = __byte_perm(r[2], r[3], 0x7362);  // bytes 2,3
                pl[0][q] = __byte_perm(t0, t1, 0x5410); pl[1][q] = __byte_perm(t0, t1, 0x7632);
                pl[2][q] = __byte_perm(t2, t3, 0x5410); pl[3][q] = __byte_perm(t2, t3, 0x7632);
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) put(p, lo + 16 * uint64_t(g), pl[p]);
        }
    } else if (it.kind == K_PASS) {
        for (uint32_t g = threadIdx.x; g < groups; g += SPLIT_THREADS) {
            const uint4 v = src[g];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            put(0, lo + 16 * uint64_t(g), w);
        }
    } else {
        for (uint32_t g = threadIdx.x; g < groups; g += SPLIT_THREADS) {
            const uint4 v = src[g];
            const uint32_t e[4] = {v.x, v.y, v.z, v.w};
            uint32_t h[4], l[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t r = it.kind == K_E4M3 ? (((e[k] & 0x78787878u) << 1) | ((e[k] & 0x80808080u) >> 4) | (e[k] & 0x07070707u))
                                                    : (((e[k] & 0x7C7C7C7Cu) << 1) | ((e[k] & 0x80808080u) >> 5) | (e[k] & 0x03030303u));
                h[k] = (r >> 4) & 0x0F0F0F0Fu; l[k] = r & 0x0F0F0F0Fu;
            }
            put(0, lo + 16 * uint64_t(g), h);
            put(1, lo + 16 * uint64_t(g), l);
        }
    }
    if (!COPIES) return;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < uint32_t(np) * 256; i += SPLIT_THREADS) {
        uint32_t total = 0;
#pragma unroll
        for (uint32_t k = 0; k < uint32_t(COPIES); ++k) total += counts[i * COPIES + ((k + i) & (COPIES - 1))];  // rotated: the threads of a warp in different banks
        uint32_t* out = hist + uint64_t(it.first_chunk[i >> 8] + chunk) * 256 + (i & 255);
        if (per_chunk == 1) *out = total; else if (total) atomicAdd(out, total);
    }
}

// Counts of every plane from those of its chunks: blocks of 64 chunks, one thread per symbol.
__global__ void __launch_bounds__(256) plane_hist_kernel(const EncPlane* __restrict__ enc_planes, const uint32_t* __restrict__ hist, unsigned long long* __restrict__ plane_hist) {
    const EncPlane& p = enc_planes[blockIdx.y];
    const uint32_t first = blockIdx.x * 64;
    if (first >= p.n_chunks) return;
    const uint32_t last = first + 64 < p.n_chunks ? first + 64 : p.n_chunks;
    unsigned long long total = 0;
    for (uint32_t k = first; k < last; ++k) total += hist[uint64_t(p.first_chunk + k) * 256 + threadIdx.x];
    if (total) atomicAdd(&plane_hist[uint64_t(blockIdx.y) * 256 + threadIdx.x], total);
}
// Counts of bytes that are already there (the IntDelta planes, a single plane): the blocks of a chunk (the grid's second
// dimension) take SPLIT_TILE bytes at a time.  The count areas were cleared.
inline uint32_t hist_blocks(uint64_t n) { const uint64_t t = (n + SPLIT_TILE - 1) / SPLIT_TILE; return uint32_t(t < 1024 ? t : 1024); }
__global__ void __launch_bounds__(256) hist_kernel(const EncChunk* __restrict__ chunks, const uint8_t* __restrict__ planes, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[256 * 8];
    const EncChunk c = chunks[blockIdx.x];
    for (uint32_t i = threadIdx.x; i < 256 * 8; i += blockDim.x) h[i] = 0;
    __syncthreads();
    uint32_t* mine = h + (threadIdx.x & 7);
    const uintptr_t start = reinterpret_cast<uintptr_t>(planes + c.plane_off);
    for (uint64_t begin = uint64_t(blockIdx.y) * SPLIT_TILE; begin < c.n; begin += uint64_t(gridDim.y) * SPLIT_TILE) {
        const uintptr_t lo = start + begin, hi = start + (begin + SPLIT_TILE < c.n ? begin + SPLIT_TILE : c.n);
        const uintptr_t first_block = (lo + 15) & ~uintptr_t(15), last_block = hi & ~uintptr_t(15);
        if (first_block >= last_block) {
            for (uintptr_t a = lo + threadIdx.x; a < hi; a += blockDim.x) atomicAdd(&mine[uint32_t(*reinterpret_cast<const uint8_t*>(a)) * 8], 1u);
            continue;
        }
        if (lo + threadIdx.x < first_block) atomicAdd(&mine[uint32_t(*reinterpret_cast<const uint8_t*>(lo + threadIdx.x)) * 8], 1u);
        if (last_block + threadIdx.x < hi) atomicAdd(&mine[uint32_t(*reinterpret_cast<const uint8_t*>(last_block + threadIdx.x)) * 8], 1u);
        for (uintptr_t b = first_block + 16 * uintptr_t(threadIdx.x); b < last_block; b += 16 * uintptr_t(blockDim.x)) {
            const uint4 v = *reinterpret_cast<const uint4*>(b);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 16; ++k) atomicAdd(&mine[((w[k >> 2] >> (8 * (k & 3))) & 0xFFu) * 8], 1u);
        }
    }
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) total += h[threadIdx.x * 8 + k];
    if (total) atomicAdd(&hist[uint64_t(blockIdx.x) * 256 + threadIdx.x], total);
}

// The chunk descriptors of all planes, and the lists of chunks the stream encoders walk.
__global__ void __launch_bounds__(256) expand_chunks_kernel(const EncPlane* __restrict__ enc_planes, uint32_t n_planes, uint32_t n_chunks, EncChunk* __restrict__ chunks, uint32_t* __restrict__ lists) {
    const uint32_t ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= n_chunks) return;
    uint32_t lo = 0, hi = n_planes;  // the last plane that starts at or before the chunk (planes without chunks start where the next one does)
    while (lo + 1 < hi) { const uint32_t mid = (lo + hi) >> 1; if (enc_planes[mid].first_chunk <= ci) lo = mid; else hi = mid; }
    const EncPlane& p = enc_planes[lo];
    const uint32_t k = ci - p.first_chunk;
    const uint64_t at = uint64_t(k) * p.chunk;
    const uint32_t n = uint32_t(p.len - at < p.chunk ? p.len - at : p.chunk);
    chunks[ci] = EncChunk{p.buf_off + at, p.slot_off + uint64_t(k) * p.slot_stride, p.table_off + uint64_t(k) * p.table_bytes, n, enc_slot_cap(n), lo, p.row_len};
    if (p.list_off != ENC_NO_LIST) lists[p.list_off + k] = ci;
}

// ---- layout --------------------------------------------------------------------------------------------
// Frame size and form of every chunk, running offsets over a plane's chunks, and the bytes of the plane's chunk table (a varint
// offset and a varint length per chunk).  One block per plane; what the host needs for the records is one PlaneSizes each.
__host__ __device__ inline uint32_t varint_bytes(uint64_t v) { uint32_t n = 1; while (v >= 0x80) { v >>= 7; ++n; } return n; }
__device__ __forceinline__ uint32_t put_varint_dev(uint8_t* d, uint64_t v) {
    uint32_t n = 0;
    while (v >= 0x80) { d[n++] = uint8_t(v) | 0x80; v >>= 7; }
    d[n++] = uint8_t(v);
    return n;
}
// Payload bytes (without a chunk frame header) and the gather's form of one chunk.
__host__ __device__ inline uint64_t enc_payload(int codec, bool shared, uint32_t n, const EncResult& r, uint32_t& mode) {
    if (codec == C_IDENTITY) { mode = 0; return n; }
    if (codec == C_O1SAC) { mode = shared ? (5 | GATHER_BARE) : 5; return (shared ? 0 : r.stream_len[1]) + uint64_t(r.stream_len[0]); }  // a plane's own state sits in front of the coder's bytes
    uint64_t blob;
    if (codec == C_TANS) blob = 3 + 3 * uint64_t(r.hdr_n) + 8 + r.stream_len[0];
    else {
        const uint64_t hdr = codec == C_RANS ? 1 + 2 * (uint64_t(r.hdr_n) + 1) : (r.hdr_n <= 127 ? 1 : 2) + (uint64_t(r.hdr_n) + 1) / 2;
        blob = hdr + 16 + uint64_t(r.stream_len[0]) + r.stream_len[1] + r.stream_len[2] + r.stream_len[3];
    }
    // stored raw when coding does not shrink the chunk (compress.rs NotBeneficial) or the length rule refuses it (length_prefix.rs:29-33)
    const bool coded = r.coded && blob < n && (codec == C_HUFFMAN || n <= (1u << 30) || n <= blob * 64);
    mode = coded ? (codec == C_RANS ? 2 : codec == C_HUFFMAN ? 3 : 4) : 1;
    return coded ? 5 + blob : 1 + uint64_t(n);
}
__global__ void __launch_bounds__(256) layout_kernel(const EncPlane* __restrict__ enc_planes, const EncChunk* __restrict__ chunks, const EncResult* __restrict__ results, uint32_t framed,
                                                     ChunkPlace* __restrict__ places, PlaneSizes* __restrict__ sizes) {
    __shared__ uint64_t warp_frames[8];
    __shared__ uint32_t warp_entries[8];
    const EncPlane& p = enc_planes[blockIdx.x];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t frames = 0;   // bytes of the chunks before the current 256
    uint32_t entries = 0;  // bytes of their table entries
    for (uint32_t base = 0; base < p.n_chunks; base += 256) {
        const uint32_t k = base + threadIdx.x, ci = p.first_chunk + k;
        uint64_t size = 0;
        uint32_t mode = 0, n = 0;
        if (k < p.n_chunks) {
            n = chunks[ci].n;
            size = enc_payload(int(p.codec), p.shared != 0, n, results[ci], mode) + (framed ? 5 : 0);
        }
        uint64_t incl = size;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint64_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d); if (lane >= uint32_t(d)) incl += t; }
        __syncthreads();
        if (lane == 31) warp_frames[warp] = incl;
        __syncthreads();
        uint64_t before = frames + incl - size, all = 0;
        for (uint32_t w = 0; w < 8; ++w) { if (w < warp) before += warp_frames[w]; all += warp_frames[w]; }
        const uint32_t e = k < p.n_chunks ? varint_bytes(before) + varint_bytes(n) : 0u;
        const uint32_t e_excl = warp_prefix(e, lane);
        if (lane == 31) warp_entries[warp] = e_excl + e;
        __syncthreads();
        uint32_t e_before = entries + e_excl, e_all = 0;
        for (uint32_t w = 0; w < 8; ++w) { if (w < warp) e_before += warp_entries[w]; e_all += warp_entries[w]; }
        if (k < p.n_chunks) places[ci] = ChunkPlace{before, e_before, mode | (framed ? 0u : GATHER_NOFRAME)};
        frames += all; entries += e_all;
    }
    if (threadIdx.x == 0) sizes[blockIdx.x] = PlaneSizes{frames, entries, p.codec == C_O1SAC && p.n_chunks == 1 && !p.shared ? results[p.first_chunk].stream_len[1] : 0u};
}

// ---- tables --------------------------------------------------------------------------------------------
// One warp per chunk turns its histogram into the table of the codec its plane uses; lane l owns the symbols 8 l .. 8 l + 7.
// The same choices as rans_normalize, tans_normalize, huffman_lengths of encode_tables.cuh, made by all
// lanes together: with one thread per chunk the 256-step loops and the Huffman tree took 0.6 - 1.1 ms however few chunks
// there were.
// The first index at which the largest of all values stands.
__device__ __forceinline__ uint32_t warp_first_argmax(const uint32_t v[8], uint32_t lane, uint32_t& best) {
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) m = max(m, v[k]);
    best = __reduce_max_sync(0xFFFFFFFFu, m);
    uint32_t at = 0xFFFFFFFFu;
#pragma unroll
    for (int k = 7; k >= 0; --k) if (v[k] == best) at = lane * 8 + k;
    return __reduce_min_sync(0xFFFFFFFFu, at);
}
// floor(c * 2048 / n), at least one where c is not zero; returns the sum over all symbols
__device__ __forceinline__ uint32_t warp_scale_counts(const uint32_t c[8], uint32_t n, uint32_t f[8]) {
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        f[k] = 0;
        if (c[k]) { f[k] = uint32_t(uint64_t(c[k]) * 2048u / n); if (f[k] == 0) f[k] = 1; }
        sum += f[k];
    }
    return __reduce_add_sync(0xFFFFFFFFu, sum);
}
__device__ __forceinline__ void warp_add_at(uint32_t f[8], uint32_t lane, uint32_t at, uint32_t d) {
#pragma unroll
    for (int k = 0; k < 8; ++k) if (lane * 8 + k == at) f[k] += d;
}
__device__ __forceinline__ void warp_store_freqs(uint8_t* tab, uint32_t lane, const uint32_t f[8]) {
    *reinterpret_cast<uint4*>(tab + 16 * lane) = make_uint4(f[0] | f[1] << 16, f[2] | f[3] << 16, f[4] | f[5] << 16, f[6] | f[7] << 16);
}
__device__ __forceinline__ void warp_load_freqs(const uint8_t* tab, uint32_t lane, uint32_t f[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(tab + 16 * lane);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = (w[k >> 1] >> (16 * (k & 1))) & 0xFFFFu;
}

struct HuffWork {             // shared memory of one warp while it builds a Huffman code
    uint32_t leaf_f[256];     // count of leaf i (leaves numbered in symbol order)
    uint32_t sorted_f[257];   // counts in increasing (count, leaf) order
    uint32_t node_f[256];     // internal nodes in the order they are made; later their depth
    uint16_t leaf_parent[256], node_parent[256];  // by place in sorted order / by node
    uint8_t leaf_sym[256], sorted_leaf[256], len[256];
};
// Code lengths: the two smallest nodes under the (count, node id) order are merged again and again.  With the leaves sorted
// that is the two-queue method: merged nodes come out in increasing count order, and on equal counts a leaf goes first
// because its id is smaller.  Returns the number of weights to store; the lengths end up in w.len.
__device__ __forceinline__ uint32_t warp_huffman_lengths(const uint32_t c[8], uint32_t lane, HuffWork& w) {
    uint32_t mine = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) mine += c[k] != 0;
    uint32_t at = warp_prefix(mine, lane), last = 0;
    const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, mine);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        w.len[lane * 8 + k] = 0;
        if (c[k]) { w.leaf_f[at] = c[k]; w.leaf_sym[at] = uint8_t(lane * 8 + k); ++at; last = lane * 8 + k; }
    }
    last = __reduce_max_sync(0xFFFFFFFFu, last);
    if (n == 0) return 0;
    __syncwarp();
    if (n == 1) { if (lane == 0) w.len[w.leaf_sym[0]] = 1; __syncwarp(); return last + 1; }
    for (uint32_t i = lane; i < n; i += 32) {
        const uint32_t f = w.leaf_f[i];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < n; ++j) { const uint32_t g = w.leaf_f[j]; rank += (g < f) || (g == f && j < i); }
        w.sorted_f[rank] = f; w.sorted_leaf[rank] = uint8_t(i);
    }
    __syncwarp();
    if (lane == 0) {
        uint32_t i = 0, j = 0, made = 0;  // next leaf, next merged node, merged nodes made
        uint32_t fi = w.sorted_f[0], fj = 0;
        while (made < n - 1) {
            uint32_t sum = 0;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (i < n && (j >= made || fi <= fj)) { sum += fi; w.leaf_parent[i] = uint16_t(made); ++i; fi = i < n ? w.sorted_f[i] : 0u; }
                else { sum += fj; w.node_parent[j] = uint16_t(made); ++j; fj = j < made ? w.node_f[j] : 0u; }
            }
            w.node_f[made] = sum;
            if (j == made) fj = sum;
            ++made;
        }
        w.node_f[n - 2] = 0;  // depths, from the root down: a parent is always made after its children
        for (uint32_t k = n - 2; k-- > 0;) w.node_f[k] = w.node_f[w.node_parent[k]] + 1;
    }
    __syncwarp();
    bool clamped = false;
    for (uint32_t r = lane; r < n; r += 32) {
        uint32_t d = w.node_f[w.leaf_parent[r]] + 1;
        if (d > 11) { d = 11; clamped = true; }
        w.len[w.leaf_sym[w.sorted_leaf[r]]] = uint8_t(d);
    }
    __syncwarp();
    if (__any_sync(0xFFFFFFFFu, clamped)) {  // lengthen the first of the shortest codes until the lengths fit a prefix code
        uint32_t len[8], kraft = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) { len[k] = w.len[lane * 8 + k]; kraft += len[k] ? 1u << (11 - len[k]) : 0u; }
        kraft = __reduce_add_sync(0xFFFFFFFFu, kraft);
        while (kraft > 2048) {
            uint32_t key = 0xFFFFFFFFu;
#pragma unroll
            for (int k = 0; k < 8; ++k) if (len[k] && len[k] < 11) key = min(key, len[k] << 8 | (lane * 8 + k));
            key = __reduce_min_sync(0xFFFFFFFFu, key);
            if (key == 0xFFFFFFFFu) break;
#pragma unroll
            for (int k = 0; k < 8; ++k) if (lane * 8 + k == (key & 0xFFu)) ++len[k];
            kraft -= 1u << (10 - (key >> 8));  // 2^(11 - len) becomes half of that
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) w.len[lane * 8 + k] = uint8_t(len[k]);
        __syncwarp();
    }
    return last + 1;
}

__global__ void __launch_bounds__(128) table_kernel(const EncPlane* __restrict__ enc_planes, const EncChunk* __restrict__ chunks, uint32_t n_chunks,
                                                    const uint32_t* __restrict__ hist, uint8_t* __restrict__ tables, EncResult* __restrict__ results) {
    __shared__ HuffWork huff[4];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ci = blockIdx.x * 4 + warp;
    if (ci >= n_chunks) return;
    const EncChunk c = chunks[ci];
    const int codec = int(enc_planes[c.plane].codec);
    if (codec == C_O1SAC) return;  // fitted by its own kernels
    EncResult r{{0, 0, 0, 0}, 0, 0};
    if (codec != C_IDENTITY && c.n) {
        uint8_t* tab = tables + c.table_off;
        const uint4* raw = reinterpret_cast<const uint4*>(hist + uint64_t(ci) * 256) + 2 * lane;
        const uint4 a = raw[0], b = raw[1];
        const uint32_t cnt[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (codec == C_HUFFMAN) {
            HuffWork& w = huff[warp];
            const uint32_t nw = warp_huffman_lengths(cnt, lane, w);
            if (nw) {
                // canonical codes: first code of every length, then symbols in order (tree.rs:119-170), bit-reversed for the LSB-first stream
                uint32_t len[8], code[8] = {0, 0, 0, 0, 0, 0, 0, 0}, next = 0, bits = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) { len[k] = w.len[lane * 8 + k]; bits += cnt[k] * len[k]; }
                for (uint32_t l = 1; l < 12; ++l) {
                    uint32_t mine = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) mine += len[k] == l;
                    uint32_t at = next + warp_prefix(mine, lane);
#pragma unroll
                    for (int k = 0; k < 8; ++k) if (len[k] == l) code[k] = __brev(at++) >> (32 - l);
                    next = (next + __reduce_add_sync(0xFFFFFFFFu, mine)) << 1;
                }
                *reinterpret_cast<uint2*>(tab + 8 * lane) = make_uint2(len[0] | len[1] << 8 | len[2] << 16 | len[3] << 24, len[4] | len[5] << 8 | len[6] << 16 | len[7] << 24);
                uint4* out = reinterpret_cast<uint4*>(tab + 256) + 2 * lane;
                out[0] = make_uint4(code[0] | len[0] << 16, code[1] | len[1] << 16, code[2] | len[2] << 16, code[3] | len[3] << 16);
                out[1] = make_uint4(code[4] | len[4] << 16, code[5] | len[5] << 16, code[6] | len[6] << 16, code[7] | len[7] << 16);
                r.hdr_n = nw; r.coded = 1;
                // the four streams together hold at least ceil(total bits / 8) bytes: no encoding pass for a chunk that cannot shrink
                uint64_t total_bits = bits;  // a lane's share stays below 2^32 only for chunks below 2^28 symbols
                if (c.n >= (1u << 28)) { total_bits = 0; for (int k = 0; k < 8; ++k) total_bits += uint64_t(cnt[k]) * len[k]; }
#pragma unroll
                for (int d = 16; d; d >>= 1) total_bits += __shfl_xor_sync(0xFFFFFFFFu, total_bits, d);
                if ((total_bits + 7) / 8 + (nw <= 127 ? 1 : 2) + (nw + 1) / 2 + 16 >= c.n) r.coded = 0;
            }
        } else {
            uint32_t f[8], best, present = 0;
            const uint32_t sum = warp_scale_counts(cnt, c.n, f), top = warp_first_argmax(cnt, lane, best);
#pragma unroll
            for (int k = 0; k < 8; ++k) present |= uint32_t(cnt[k] != 0) << k;
            if (codec == C_RANS) {
                bool ok = true;
                if (sum > 2048) {  // the excess comes off the most frequent symbol, or the chunk stays raw
                    uint32_t ft = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) if (lane * 8 + k == top) ft = f[k];
                    ft = __reduce_max_sync(0xFFFFFFFFu, ft);
                    ok = ft > sum - 2048;
                }
                if (ok) {
                    warp_add_at(f, lane, top, 2048 - sum);
                    warp_store_freqs(tab, lane, f);
                    const uint32_t ms = __reduce_max_sync(0xFFFFFFFFu, present ? lane * 8 + 31 - __clz(present) : 0u);
                    r.hdr_n = ms; r.coded = 1;
                    // A chunk that cannot come out smaller than it is gets no encoding pass: the coder's output is at least the
                    // information content of the chunk under its table, less the four initial states, so when that alone (with a
                    // margin for the float logarithm) reaches the chunk's size the result would be discarded anyway
                    // (compress.rs: NotBeneficial).  Sign / mantissa planes are the usual case.
                    float bits = 0.f;
#pragma unroll
                    for (int k = 0; k < 8; ++k) if (cnt[k]) bits += float(cnt[k]) * (11.f - log2f(float(f[k])));
#pragma unroll
                    for (int d = 16; d; d >>= 1) bits += __shfl_xor_sync(0xFFFFFFFFu, bits, d);
                    const float lower = bits * (1.f - 1e-4f) / 8.f - 16.f + float(1 + 2 * (ms + 1) + 16);
                    if (lower >= float(c.n) + 64.f) r.coded = 0;
                }
            } else {  // tANS (entropy/tans/mod.rs:153-194)
                uint32_t left = sum;
                while (left > 2048) {  // one at a time from the first largest entry above one
                    uint32_t most;
                    const uint32_t at = warp_first_argmax(f, lane, most);
                    if (most <= 1) break;
                    warp_add_at(f, lane, at, 0xFFFFFFFFu);
                    --left;
                }
                if (left < 2048) warp_add_at(f, lane, top, 2048 - left);
                const uint32_t nsym = __reduce_add_sync(0xFFFFFFFFu, __popc(present));
                warp_store_freqs(tab, lane, f);
                if (nsym >= 2) { r.hdr_n = nsym; r.coded = 1; }
            }
        }
    }
    if (lane == 0) results[ci] = r;
}

// ---- streams -------------------------------------------------------------------------------------------
// The bytes of rANS and Huffman streams are made last to first.  They are appended upward from the start of the stream's slot
// in the order they are made, and the gather turns them around.
// f(sym) for the bytes of [lo, hi), last to first, out of aligned 16-byte blocks, each requested while the one above it is
// worked on; `block` gets the sixteen bytes of a whole block, highest first.
template <class Byte, class Block>
__device__ __forceinline__ void walk_down(uintptr_t lo, uintptr_t hi, Byte&& byte, Block&& block) {
    const uintptr_t first_block = (lo + 15) & ~uintptr_t(15), last_block = hi & ~uintptr_t(15);
    if (first_block >= last_block) {
        for (uintptr_t a = hi; a-- > lo;) byte(uint32_t(*reinterpret_cast<const uint8_t*>(a)));
        return;
    }
    for (uintptr_t a = hi; a-- > last_block;) byte(uint32_t(*reinterpret_cast<const uint8_t*>(a)));
    uintptr_t b = last_block - 16;
    uint4 ahead = *reinterpret_cast<const uint4*>(b);
    for (;;) {
        const uint4 v = ahead;
        const bool more = b > first_block;
        if (more) ahead = *reinterpret_cast<const uint4*>(b - 16);
        block(v);
        if (!more) break;
        b -= 16;
    }
    for (uintptr_t a = first_block; a-- > lo;) byte(uint32_t(*reinterpret_cast<const uint8_t*>(a)));
}

// rANS: one lane per stream, eight chunks per warp.  A symbol is a serial step of the coder's state: its chain is kept short
// (what the symbol's step needs sits in shared memory, 16 bytes per symbol, read ahead of use because it depends on the data
// alone; the number of bytes that leave is 0, 1 or 2 by two compares) and so is the number of instructions, because the
// integer pipe is what bounds a launch that fills the GPU: the bytes that leave are shifted into a register pair from above,
// and every two symbols the oldest word of the pair is put into a ring in shared memory whether it is full or not (only the
// write position moves on a full word), from where sixteen bytes at a time go out.  A branch with a store per full word was
// taken by some lane in nearly every step.  The rows cover `range` symbols: the chunk's lowest one first, whatever its distance (an
// exact zero lies far below the other exponents), then all values from its second lowest on.  The host knows the span of a
// plane's alphabet and sends planes of similar span together, so that exponent planes (some 30 values) keep 24 blocks on an SM.
// 26,640 chunks of 32 Ki symbols, with and without zeros in them: 1170 + 335 us in one launch of 12 and one of 20 blocks per SM,
// 1190 in one of 24, 1121 with a row's entries of the eight chunks side by side, where a quarter of a warp reads eight chunks' entries
// from banks of their own.  That is 12 cycles per warp and symbol with the integer pipe 73 % busy.  With 16-byte entries in global
// memory and a loop per byte a symbol took 330 ns.
// x' = x + bias + floor(x / f) * (2048 - f) with the quotient from a rounded-up reciprocal: exact for every state below 2^31,
// i.e. identical to (x / f) * 2048 + x % f + start (entropy/rans/compress.rs:140-185).
constexpr uint32_t RENC_RING = 16;  // words per lane: up to 3 waiting, up to 8 more in sixteen symbols, one being filled
__host__ __device__ inline uint32_t renc_smem_bytes(uint32_t range) { return RANS_WARP_CHUNKS * range * 16 + RENC_RING * 32 * 4; }
__global__ void __launch_bounds__(32) rans_encode_kernel(const EncChunk* __restrict__ chunks, const uint32_t* __restrict__ list, uint32_t n_list, uint32_t range,
                                                         const uint8_t* __restrict__ planes, const uint8_t* __restrict__ tables, uint8_t* __restrict__ slots,
                                                         EncResult* __restrict__ results) {
    extern __shared__ __align__(16) uint8_t renc_smem[];
    uint4* entries = reinterpret_cast<uint4*>(renc_smem);
    uint32_t* ring_all = reinterpret_cast<uint32_t*>(renc_smem + RANS_WARP_CHUNKS * range * 16);
    const uint32_t lane = threadIdx.x, c8 = lane & 7, s = lane >> 3, li = blockIdx.x * RANS_WARP_CHUNKS + c8;
    const uint32_t ci = li < n_list ? list[li] : 0xFFFFFFFFu;
    EncChunk c{};
    if (li < n_list) c = chunks[ci];
    const bool live = li < n_list && c.n && results[ci].coded;
    uint32_t first_sym = 0;
    for (uint32_t k = 0; k < RANS_WARP_CHUNKS; ++k) {  // entry: reciprocal, bias << 8 | reciprocal shift, 2048 - frequency, frequency << 20
        if (!__shfl_sync(0xFFFFFFFFu, uint32_t(live), k)) continue;
        uint32_t f[8], sum = 0, lowest = 0xFFFFFFFFu, second = 0xFFFFFFFFu;
        warp_load_freqs(tables + __shfl_sync(0xFFFFFFFFu, c.table_off, k), lane, f);
#pragma unroll
        for (int j = 7; j >= 0; --j) { sum += f[j]; if (f[j]) lowest = lane * 8 + j; }
        lowest = __reduce_min_sync(0xFFFFFFFFu, lowest);
#pragma unroll
        for (int j = 7; j >= 0; --j) if (f[j] && lane * 8 + j > lowest) second = lane * 8 + j;
        second = __reduce_min_sync(0xFFFFFFFFu, second);
        const uint32_t base = second == 0xFFFFFFFFu ? lowest : second - 1;  // the value of the first row
        if (c8 == k) first_sym = base;
        uint32_t start = warp_prefix(sum, lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t sym = lane * 8 + j, at = sym == lowest ? 0u : sym - base;  // (wraps for symbols below the second, which have no count)
            uint4 e = make_uint4(0xFFFFFFFFu, (start + 2047u) << 8, 2047u, 1u << 20);  // f = 1: the quotient comes out one short of x
            if (f[j] > 1) {
                const uint32_t shift = 32 - __clz(f[j] - 1);  // smallest with f <= 2^shift
                e = make_uint4(uint32_t(((1ull << (shift + 31)) + f[j] - 1) / f[j]), start << 8 | (shift - 1), 2048u - f[j], f[j] << 20);
            }
            if (f[j] && at < range) entries[at * RANS_WARP_CHUNKS + k] = e;
            start += f[j];
        }
    }
    __syncwarp();
    if (!live) return;
    uint32_t start, len;
    split_four_dev(c.n, s, start, len);
    uint8_t* slot = slots + c.slot_off + uint64_t(s) * c.slot_cap;
    const uint4* rows = entries + c8 - first_sym * RANS_WARP_CHUNKS;
    auto row = [&](uint32_t sym) -> const uint4& { return rows[(sym > first_sym ? sym : first_sym) * RANS_WARP_CHUNKS]; };
    uint32_t* ring = ring_all + lane;
    uint32_t x = 1u << 23;
    uint32_t b_lo = 0, b_hi = 0, have = 0;  // the youngest `have` bits wait at the top of b_hi:b_lo; below 32 between pairs of symbols
    uint32_t put = 0, sent = 0;             // words made / stored
    auto step = [&](const uint4& e) {
        // bytes leave while x >= f << 20 (= ((L >> 11) << 8) * f): at most two, the state being below 2^31
        uint32_t sh = x >= e.w ? 8u : 0u;
        sh = (x >> 8) >= e.w ? 16u : sh;
        b_lo = __funnelshift_r(b_lo, b_hi, sh);
        b_hi = __funnelshift_r(b_hi, x, sh);
        have += sh;
        x >>= sh;
        x = x + (e.y >> 8) + __funnelshift_r(__umulhi(x, e.x), 0u, e.y) * e.z;  // shift by the low five bits of e.y
    };
    auto settle = [&]() {
        ring[(put & (RENC_RING - 1)) * 32] = __funnelshift_rc(b_lo, b_hi, 64 - have);  // the oldest word when there is one
        const bool full = have >= 32;
        put += full; have -= full ? 32u : 0u;
    };
    auto drain = [&]() {  // sixteen bytes out for every lane that has them, when any has
        if (__any_sync(__activemask(), put - sent >= 4)) {
            if (put - sent >= 4) {
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) w[k] = ring[((sent + k) & (RENC_RING - 1)) * 32];
                *reinterpret_cast<uint4*>(slot + 4 * size_t(sent)) = make_uint4(w[0], w[1], w[2], w[3]);
                sent += 4;
            }
        }
    };
    const uintptr_t lo = reinterpret_cast<uintptr_t>(planes + c.plane_off) + start;
    walk_down(lo, lo + len, [&](uint32_t b) { step(row(b)); settle(); drain(); },
              [&](const uint4& v) {
                  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                  for (int h = 3; h >= 0; --h) {
                      uint4 e[4];
#pragma unroll
                      for (int k = 0; k < 4; ++k) e[k] = row((w[h] >> (8 * k)) & 0xFFu);
                      step(e[3]); step(e[2]); settle();
                      step(e[1]); step(e[0]); settle();
                  }
                  drain();
                  drain();
              });
    // the final state, little-endian once the bytes are turned around, then what waits
    for (int k = 3; k >= 0; --k) {
        b_lo = __funnelshift_r(b_lo, b_hi, 8);
        b_hi = __funnelshift_r(b_hi, x >> (8 * k), 8);
        have += 8;
        settle();
    }
    for (; sent < put; ++sent) *reinterpret_cast<uint32_t*>(slot + 4 * size_t(sent)) = ring[(sent & (RENC_RING - 1)) * 32];
    if (have) *reinterpret_cast<uint32_t*>(slot + 4 * size_t(put)) = b_hi >> (32 - have);
    results[ci].stream_len[s] = 4 * put + (have + 7) / 8;
}

// Huffman: the place of a symbol's bits follows from the lengths before it, so a warp codes a stream 512 symbols at a time:
// every lane strings its sixteen codes together, a prefix sum over the lanes gives the bit each string starts at, and the
// strings are put together in shared memory.  (One thread per stream took 107 ns per symbol.)
// WARPS > 1, for launches that do not fill the GPU: that many warps to a stream in each block of a cluster, every warp with a share of the
// stream's rounds.  They first count the bits of their shares, which all blocks read of one another; a word that shares meet in
// is kept by all of them and put together at the end by the one that fills it.  It asks the shares before it one after the other, in other
// blocks' shared memory, so a stream has no more shares than rounds: with empty ones 1000 symbols took 25.4 us, without 8.5.
constexpr uint32_t HENC_LANE = 16, HENC_WORDS = (32 * HENC_LANE * 11 + 31) / 32 + 2, HENC_ROUND = 32 * HENC_LANE;
template <int WARPS>
__global__ void __launch_bounds__(128 * WARPS) huffman_encode_kernel(const EncChunk* __restrict__ chunks, const uint32_t* __restrict__ list, uint32_t n_list,
                                                                     const uint8_t* __restrict__ planes, const uint8_t* __restrict__ tables, uint8_t* __restrict__ slots,
                                                                     EncResult* __restrict__ results) {
    struct Shared {
        uint32_t codes[256];
        uint32_t words[4 * WARPS][HENC_WORDS];
        uint64_t bits[4][WARPS];
        uint32_t head_at[4][WARPS], head[4][WARPS], tail_at[4][WARPS], tail[4][WARPS];  // the words a share meets its neighbours in
    };
    __shared__ Shared sh;
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const uint32_t blocks = WARPS > 1 ? cluster.num_blocks() : 1, rank = WARPS > 1 ? cluster.block_rank() : 0;
    const uint32_t ci = list[blockIdx.x / blocks], lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s = warp / WARPS, mine = warp % WARPS;
    const uint32_t part = rank * WARPS + mine;
    auto of = [&](uint32_t q) -> const Shared* { return cluster.map_shared_rank(&sh, q / WARPS); };  // where share q is kept, at place q % WARPS
    const EncChunk c = chunks[ci];
    if (!c.n || !results[ci].coded) return;
    const uint32_t* g_codes = reinterpret_cast<const uint32_t*>(tables + c.table_off + 256);
    for (uint32_t i = threadIdx.x; i < 256; i += 128 * WARPS) sh.codes[i] = g_codes[i];
    uint32_t* words = sh.words[warp];
    for (uint32_t i = lane; i < HENC_WORDS; i += 32) words[i] = 0;
    __syncthreads();
    uint32_t start, len;
    split_four_dev(c.n, s, start, len);
    const uint8_t* src = planes + c.plane_off + start;
    uint8_t* slot = slots + c.slot_off + uint64_t(s) * c.slot_cap;
    uint32_t* out = reinterpret_cast<uint32_t*>(slot);
    const uint32_t rounds = (len + HENC_ROUND - 1) / HENC_ROUND;
    const uint32_t parts = min(blocks * WARPS, max(rounds, 1u));  // shares, a round or more each; the warps behind them have none
    const uint32_t from = part < parts ? uint32_t(uint64_t(rounds) * part / parts) * HENC_ROUND : len;
    const uint32_t to = part + 1 < parts ? uint32_t(uint64_t(rounds) * (part + 1) / parts) * HENC_ROUND : len;
    auto fetch = [&](uint32_t at, uint32_t n, uint64_t& a, uint64_t& b) {  // up to sixteen bytes from src + at
        a = b = 0;
        if (n == HENC_LANE) { a = ld8_unaligned(src + at); b = ld8_unaligned(src + at + 8); }
        else { a = ld_bytes(src + at, n < 8 ? n : 8); if (n > 8) b = ld_bytes(src + at + 8, n - 8); }
    };
    auto count_at = [&](uint32_t base) -> uint32_t { const uint32_t at = base + lane * HENC_LANE; return at >= to ? 0u : to - at < HENC_LANE ? to - at : HENC_LANE; };
    auto code_of = [&](uint64_t a, uint64_t b, uint32_t k) { return sh.codes[uint32_t((k < 8 ? a : b) >> (8 * (k & 7))) & 0xFFu]; };
    uint64_t na, nb, before_us = 0;
    if (WARPS > 1) {
        uint64_t sum = 0;
        fetch(from + lane * HENC_LANE, count_at(from), na, nb);
        for (uint32_t base = from; base < to; base += HENC_ROUND) {
            const uint32_t n = count_at(base);
            const uint64_t ca = na, cb = nb;
            if (base + HENC_ROUND < to) fetch(base + HENC_ROUND + lane * HENC_LANE, count_at(base + HENC_ROUND), na, nb);
#pragma unroll
            for (uint32_t k = 0; k < HENC_LANE; ++k) sum += k < n ? code_of(ca, cb, k) >> 16 : 0u;
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
        if (lane == 0) sh.bits[s][mine] = sum;
        cluster.sync();
        if (part < parts) for (uint32_t q = lane; q < part; q += 32) before_us += of(q)->bits[s][q % WARPS];
#pragma unroll
        for (int d = 16; d; d >>= 1) before_us += __shfl_xor_sync(0xFFFFFFFFu, before_us, d);
    }
    uint32_t have = uint32_t(before_us) & 31;  // bits of the word that is not full yet, which stays in words[0]
    out += before_us >> 5;
    bool meets = have != 0;  // words[0] is the last one of the share before
    if (WARPS > 1 && lane == 0) sh.head_at[s][mine] = sh.tail_at[s][mine] = 0xFFFFFFFFu;
    fetch(from + lane * HENC_LANE, count_at(from), na, nb);
    for (uint32_t base = from; base < to; base += HENC_ROUND) {
        const uint32_t n = count_at(base);
        const uint64_t ca = na, cb = nb;
        if (base + HENC_ROUND < to) fetch(base + HENC_ROUND + lane * HENC_LANE, count_at(base + HENC_ROUND), na, nb);  // the next round's symbols
        uint32_t e[HENC_LANE], bits = 0;
#pragma unroll
        for (uint32_t k = 0; k < HENC_LANE; ++k) {
            e[k] = k < n ? code_of(ca, cb, k) : 0u;
            bits += e[k] >> 16;
        }
        const uint32_t before = warp_prefix(bits, lane), total = __shfl_sync(0xFFFFFFFFu, before + bits, 31);
        const uint32_t at = have + before;
        uint32_t w = at >> 5, fill = at & 31, lo = 0;
        bool first = true;  // the word the lane before this one may also write into
#pragma unroll
        for (uint32_t k = 0; k < HENC_LANE; ++k) {
            const uint32_t cd = e[k] & 0xFFFFu, l = e[k] >> 16;
            lo |= cd << fill;
            fill += l;
            if (fill >= 32) {
                if (first) atomicOr(&words[w], lo); else words[w] = lo;
                first = false;
                ++w; fill -= 32;
                lo = fill ? cd >> (l - fill) : 0u;
            }
        }
        if (fill && lo) atomicOr(&words[w], lo);
        __syncwarp();
        const uint32_t full = (have + total) >> 5;
        have = (have + total) & 31;
        const uint32_t rest = words[full];
        if (WARPS > 1 && meets && full) {
            if (lane == 0) { sh.head_at[s][mine] = uint32_t(out - reinterpret_cast<uint32_t*>(slot)); sh.head[s][mine] = words[0]; }
            for (uint32_t i = lane; i < full; i += 32) if (i) out[i] = words[i];
            meets = false;
        } else {
            for (uint32_t i = lane; i < full; i += 32) out[i] = words[i];
        }
        __syncwarp();
        for (uint32_t i = lane; i <= full; i += 32) words[i] = i == 0 ? rest : 0u;
        out += full;
        __syncwarp();
    }
    if (WARPS == 1) {
        if (lane == 0) {
            if (have) *out = words[0];
            results[ci].stream_len[s] = uint32_t(reinterpret_cast<uint8_t*>(out) - slot) + (have + 7) / 8;
        }
        return;
    }
    if (lane == 0 && have) { sh.tail_at[s][mine] = uint32_t(out - reinterpret_cast<uint32_t*>(slot)); sh.tail[s][mine] = words[0]; }
    cluster.sync();
    if (lane == 0) {
        auto with_tails = [&](uint32_t w, uint32_t v) {  // and the bits of the shares before this one that end in word w
            for (uint32_t q = part; q-- > 0;) {
                const Shared* o = of(q);
                if (o->tail_at[s][q % WARPS] == w) v |= o->tail[s][q % WARPS];
                else if (o->bits[s][q % WARPS] != 0) break;
            }
            reinterpret_cast<uint32_t*>(slot)[w] = v;
        };
        if (sh.head_at[s][mine] != 0xFFFFFFFFu) with_tails(sh.head_at[s][mine], sh.head[s][mine]);
        if (part + 1 == parts) {
            const uint64_t all = before_us + sh.bits[s][mine];
            if (all & 31) with_tails(uint32_t(all >> 5), sh.tail_at[s][mine] == uint32_t(all >> 5) ? sh.tail[s][mine] : 0u);
            results[ci].stream_len[s] = uint32_t((all + 7) / 8);
        }
    }
    cluster.sync();  // the other blocks' shared memory is read until here
}
// Chunks of a launch up to which eight warps and more take a stream.  us of a whole compress_model with one / eight warps: 64 Ki symbols, 1 chunk 194 /
// 165, 148: 198 / 162, 592: 246 / 253; 16 Ki, 148: 158 / 146, 592: 174 / 185; 4 Ki, 148: 147 / 149, 296: 147 / 161.  Launches that leave SMs
// idle get two, four or eight blocks to a chunk: 200,003 symbols in a call of their own 65 -> 16 us, the call 139 -> 90, and 77 with the payload
// gathered by several blocks that see for themselves whether it fits.
constexpr uint32_t HENC_WIDE_CHUNKS = 148;
inline cudaError_t huffman_encode_launch(const EncChunk* chunks, const uint32_t* list, uint32_t n, const uint8_t* planes, const uint8_t* tables, uint8_t* slots, EncResult* results,
                                         cudaStream_t st) {
    if (n > HENC_WIDE_CHUNKS) {
        huffman_encode_kernel<1><<<n, 128, 0, st>>>(chunks, list, n, planes, tables, slots, results);
        return cudaGetLastError();
    }
    uint32_t blocks = 8;
    while (blocks > 1 && n * blocks > HENC_WIDE_CHUNKS) blocks /= 2;
    cudaLaunchAttribute cluster{};
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = blocks; cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(n * blocks); config.blockDim = dim3(1024); config.stream = st;
    config.attrs = &cluster; config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, huffman_encode_kernel<8>, chunks, list, n, planes, tables, slots, results);
}

// tANS (entropy/tans/mod.rs:268-318): one serial stream per chunk, its symbols walked last to first, its bits going upward.
// One warp per chunk all the same: the chunk is cut into 32 runs of symbols and every lane codes its run from a guessed state.
// Two coders with different states that see the same symbols meet after a while (both states of a pair fall into the few
// states of a rare symbol; about 1,100 symbols on an exponent plane) and then stay together, so most lanes leave their run in
// the state the serial coder has there.  The state a lane leaves in is where the lane below must start: lanes whose start
// was not that go again until nobody's changes.  Each round settles at least one more lane, so the worst case is the serial
// chain.  A last pass writes the bits at the places the runs' bit counts give.
__global__ void __launch_bounds__(32) tans_encode_kernel(const EncChunk* __restrict__ chunks, const uint32_t* __restrict__ list, uint32_t n_list,
                                                         const uint8_t* __restrict__ planes, const uint8_t* __restrict__ tables, uint8_t* __restrict__ slots,
                                                         EncResult* __restrict__ results) {
    __shared__ uint16_t next_state[2048];
    __shared__ uint2 sym[256];        // bit-count term, offset into next_state
    __shared__ uint16_t fill[256];
    __shared__ uint8_t spread[2048];
    const uint32_t lane = threadIdx.x, ci = list[blockIdx.x];
    const EncChunk c = chunks[ci];
    if (!results[ci].coded || !c.n) return;
    {
        uint32_t f[8], sum = 0;
        warp_load_freqs(tables + c.table_off, lane, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += f[k];
        uint32_t run = warp_prefix(sum, lane);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint2 e = make_uint2(0, 0);
            if (f[k] == 1) e = make_uint2((11u << 16) - 2048u, run - 1);
            else if (f[k] > 1) {
                const uint32_t max_bits = 11u - (31u - uint32_t(__clz(f[k] - 1)));
                e = make_uint2((max_bits << 16) - (f[k] << max_bits), run - f[k]);
            }
            sym[lane * 8 + k] = e;
            fill[lane * 8 + k] = uint16_t(run);
            run += f[k];
        }
        __syncwarp();
        // position k of the symbols in order goes to state 1283 k mod 2048; lane l places positions 64 l .. 64 l + 63
        uint32_t sy = 0;
        for (uint32_t d = 128; d; d >>= 1) if (sy + d < 256 && fill[sy + d] <= 64 * lane) sy += d;  // the last symbol that starts at or below 64 l
        for (uint32_t k = 64 * lane; k < 64 * lane + 64; ++k) {
            while (sy < 255 && fill[sy + 1] <= k) ++sy;
            spread[(k * 1283u) & 2047u] = uint8_t(sy);
        }
        __syncwarp();
        for (uint32_t u0 = 0; u0 < 2048; u0 += 32) {  // the states of a symbol, in increasing order
            const uint32_t t = spread[u0 + lane], same = __match_any_sync(0xFFFFFFFFu, t), before = same & ((1u << lane) - 1u), at = fill[t];
            __syncwarp();
            next_state[at + __popc(before)] = uint16_t(2048u + u0 + lane);
            if (!before) fill[t] = uint16_t(at + __popc(same));
            __syncwarp();
        }
    }
    const uintptr_t base = reinterpret_cast<uintptr_t>(planes + c.plane_off);
    const uint32_t per = tans_encode_run(c.n);
    const uint64_t first = uint64_t(lane) * per;
    const uint32_t r_lo = first < c.n ? uint32_t(first) : c.n, r_hi = first + per < c.n ? uint32_t(first + per) : c.n;
    auto entry = [&](uint32_t b) { return sym[b]; };
    // the run from `state`: state at its end; emit(bits, count) for every symbol
    auto code_run = [&](uint32_t value, auto&& emit) -> uint32_t {
        auto step = [&](uint2 e) {
            const uint32_t nb = (value + e.x) >> 16;
            emit(value & ((1u << nb) - 1u), nb);
            value = next_state[(value >> nb) + e.y];
        };
        walk_down(base + r_lo, base + r_hi, [&](uint32_t b) { step(entry(b)); },
                  [&](const uint4& v) {
                      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                      for (int h = 3; h >= 0; --h) {
                          uint2 e[4];
#pragma unroll
                          for (int k = 0; k < 4; ++k) e[k] = entry((w[h] >> (8 * k)) & 0xFFu);
#pragma unroll
                          for (int k = 3; k >= 0; --k) step(e[k]);
                      }
                  });
        return value;
    };
    const uint32_t last = (c.n - 1) / per;  // the lane that starts the chain, in state 2048
    uint32_t from = 2048, end = 0;
    uint64_t bits = 0;
    bool go = lane <= last;
    for (;;) {
        if (go) { bits = 0; end = code_run(from, [&](uint32_t, uint32_t nb) { bits += nb; }); }
        uint32_t want = __shfl_down_sync(0xFFFFFFFFu, end, 1);
        if (lane >= last) want = 2048;
        go = lane <= last && want != from;
        from = want;
        if (!__any_sync(0xFFFFFFFFu, go)) break;
    }
    // bits go upward from the run that is coded first, i.e. the highest lane's
    uint64_t incl = bits;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const uint64_t t = __shfl_down_sync(0xFFFFFFFFu, incl, d); if (lane + d < 32) incl += t; }
    const uint64_t at = incl - bits, all = __shfl_sync(0xFFFFFFFFu, incl, 0);
    uint32_t* out = reinterpret_cast<uint32_t*>(slots + c.slot_off);  // slot areas start on 16-byte boundaries
    // the words where two runs meet are put together with atomics, from zero
    uint32_t* w = out + (at >> 5);
    if (lane <= last) { *w = 0; out[(at + bits) >> 5] = 0; }
    if (lane == 0) { out[all >> 5] = 0; out[(all + 11) >> 5] = 0; }
    __threadfence_block();
    __syncwarp();
    if (lane <= last) {
        uint32_t lo = 0, hi = 0, have = uint32_t(at & 31);
        bool shared_word = true;
        auto flush = [&]() { if (shared_word) atomicOr(w, lo); else *w = lo; shared_word = false; ++w; lo = hi; hi = 0; have -= 32; };
        const uint32_t value = code_run(from, [&](uint32_t v, uint32_t nb) {
            lo |= v << have;
            hi |= __funnelshift_l(v, 0u, have);
            have += nb;
            if (have >= 32) flush();
        });
        if (lane == 0) {
            const uint32_t v = value & 2047u;
            lo |= v << have; hi |= __funnelshift_l(v, 0u, have);
            have += 11;
            if (have >= 32) flush();
        }
        if (have) atomicOr(w, lo);
    }
    if (lane == 0) {
        const uint64_t total = all + 11;
        results[ci].stream_len[0] = uint32_t((total + 7) / 8);
        results[ci].stream_len[1] = uint32_t(total);
        results[ci].stream_len[2] = uint32_t(total >> 32);
    }
}

// n bytes from s to d by the threads of a block.  d is brought to a 16-byte boundary, then every thread stores 16 bytes at a
// time, taken from the two aligned blocks that hold them (a block that holds a needed byte is read whole: the planes and slot
// buffers are padded for that).
__device__ __forceinline__ void block_copy(uint8_t* d, const uint8_t* s, uint32_t n, uint32_t t, uint32_t nt) {
    uint32_t head = uint32_t((16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15);
    if (head > n) head = n;
    if (t < head) d[t] = s[t];
    d += head; s += head; n -= head;
    const uint32_t blocks = n >> 4, off = uint32_t(reinterpret_cast<uintptr_t>(s) & 15);
    const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<uintptr_t>(s) & ~uintptr_t(15));
    for (uint32_t b = t; b < blocks; b += nt) {
        uint4 v = q[b];
        if (off) { uint32_t w[4]; extract16(v, q[b + 1], off, w); v = make_uint4(w[0], w[1], w[2], w[3]); }
        *reinterpret_cast<uint4*>(d + 16 * size_t(b)) = v;
    }
    const uint32_t i = blocks * 16 + t;
    if (i < n) d[i] = s[i];
}
// The same with the bytes in opposite order: d[i] = s[n - 1 - i].
__device__ __forceinline__ void block_copy_reversed(uint8_t* d, const uint8_t* s, uint32_t n, uint32_t t, uint32_t nt) {
    uint32_t head = uint32_t((16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15);
    if (head > n) head = n;
    if (t < head) d[t] = s[n - 1 - t];
    d += head; n -= head;
    const uint32_t blocks = n >> 4;
    if (t < blocks) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(s) + n - 16;  // the source bytes of block 0; block b sits 16 b below
        const uint32_t off = uint32_t(a & 15);
        const uint4* q = reinterpret_cast<const uint4*>(a & ~uintptr_t(15));
        for (uint32_t b = t; b < blocks; b += nt) {
            const uint4 v = *(q - b);
            uint32_t w[4] = {v.x, v.y, v.z, v.w};
            if (off) extract16(v, *(q - b + 1), off, w);
            *reinterpret_cast<uint4*>(d + 16 * size_t(b)) =
                make_uint4(__byte_perm(w[3], 0, 0x0123), __byte_perm(w[2], 0, 0x0123), __byte_perm(w[1], 0, 0x0123), __byte_perm(w[0], 0, 0x0123));
        }
    }
    const uint32_t i = blocks * 16 + t;
    if (i < n) d[i] = s[n - 1 - i];
}
// One chunk frame by `nt` threads of whole warps, of which this is the `t`-th: [state_version 0][state_len 0 u32] then the codec payload, at its final place.
__device__ __forceinline__ void gather_frame(uint8_t* d, const EncChunk& c, const EncResult& r, uint32_t form, const uint8_t* __restrict__ planes, const uint8_t* __restrict__ tables,
                                             const uint8_t* __restrict__ slots, uint32_t t, uint32_t nt) {
    const uint32_t mode = form & 0xFFu;
    const bool framed = !(form & (GATHER_BARE | GATHER_NOFRAME));
    if (framed) {
        if (t < 5 && mode != 5) d[t] = 0;
        d += 5;
    }
    if (mode <= 1) {
        if (mode == 1) { if (t == 0) d[0] = 0; d += 1; }
        const uint8_t* p = planes + c.plane_off;
        block_copy(d, p, c.n, t, nt);
        return;
    }
    const uint8_t* tab = tables + c.table_off;
    if (mode == 5) {  // Order1ScaleAC: inline state [bitmap 32][marginal 512][rows 512 each, contexts in increasing order], then the coder's bytes
        const uint8_t* present = tab + O1E_PRESENT;
        const uint16_t* rank = reinterpret_cast<const uint16_t*>(tab + O1E_RANK);
        const uint16_t* pmf = reinterpret_cast<const uint16_t*>(tab + O1E_PMF);
        if (!(form & GATHER_BARE)) {
            const uint32_t state_len = r.stream_len[1];
            if (framed && t == 0) {  // frame header: state_version 1, state length
                uint8_t* fh = d - 5;
                fh[0] = 1; fh[1] = uint8_t(state_len); fh[2] = uint8_t(state_len >> 8); fh[3] = uint8_t(state_len >> 16); fh[4] = uint8_t(state_len >> 24);
            }
            if (t < 32) { uint32_t bits = 0; for (int k = 0; k < 8; ++k) bits |= uint32_t(present[8 * t + k] != 0) << k; d[t] = uint8_t(bits); }
            for (uint32_t i = t; i < 256; i += nt) { d[32 + 2 * i] = uint8_t(pmf[i]); d[33 + 2 * i] = uint8_t(pmf[i] >> 8); }
            for (uint32_t ctx = 0; ctx < 256; ++ctx) {
                if (!present[ctx]) continue;
                uint8_t* row = d + 32 + 512 + 512 * uint32_t(rank[ctx]);
                const uint16_t* pr = pmf + 256 * (1 + ctx);
                for (uint32_t i = t; i < 256; i += nt) { row[2 * i] = uint8_t(pr[i]); row[2 * i + 1] = uint8_t(pr[i] >> 8); }
            }
            d += state_len;
        }
        const uint8_t* sp = slots + c.slot_off;
        block_copy(d, sp, r.stream_len[0], t, nt);
        return;
    }
    if (t == 0) { d[0] = 1; d[1] = uint8_t(c.n); d[2] = uint8_t(c.n >> 8); d[3] = uint8_t(c.n >> 16); d[4] = uint8_t(c.n >> 24); }
    d += 5;
    if (mode == 4) {  // tANS blob: [11][nsym u16][(symbol, freq u16) per present symbol][total bits u64][bits]
        if (t < 32) {
            if (t == 0) {
                d[0] = 11; d[1] = uint8_t(r.hdr_n); d[2] = uint8_t(r.hdr_n >> 8);
                uint8_t* q = d + 3 + 3 * r.hdr_n;
                for (int k = 0; k < 4; ++k) { q[k] = uint8_t(r.stream_len[1] >> (8 * k)); q[4 + k] = uint8_t(r.stream_len[2] >> (8 * k)); }
            }
            uint32_t f[8], present = 0;
            warp_load_freqs(tab, t, f);
#pragma unroll
            for (int k = 0; k < 8; ++k) present += f[k] != 0;
            uint8_t* q = d + 3 + 3 * warp_prefix(present, t);
#pragma unroll
            for (int k = 0; k < 8; ++k) if (f[k]) { q[0] = uint8_t(8 * t + k); q[1] = uint8_t(f[k]); q[2] = uint8_t(f[k] >> 8); q += 3; }
        }
        d += 3 + 3 * r.hdr_n + 8;
        const uint8_t* sp = slots + c.slot_off;
        block_copy(d, sp, r.stream_len[0], t, nt);
        return;
    }
    uint32_t hdr;
    if (mode == 2) {
        const uint16_t* freqs = reinterpret_cast<const uint16_t*>(tab);
        hdr = 1 + 2 * (r.hdr_n + 1);
        if (t == 0) d[0] = uint8_t(r.hdr_n);
        for (uint32_t i = t; i <= r.hdr_n; i += nt) { d[1 + 2 * i] = uint8_t(freqs[i]); d[2 + 2 * i] = uint8_t(freqs[i] >> 8); }
    } else {
        const uint32_t nw = r.hdr_n;
        uint32_t hb = nw <= 127 ? 1 : 2;
        hdr = hb + (nw + 1) / 2;
        if (t == 0) { if (nw <= 127) d[0] = uint8_t(0x80 | nw); else { d[0] = 0x80; d[1] = uint8_t(nw); } }
        for (uint32_t i = t; i < (nw + 1) / 2; i += nt) {
            uint32_t lo = tab[2 * i] & 0x0F, hi = (2 * i + 1 < nw ? tab[2 * i + 1] : 0) & 0x0F;
            d[hb + i] = uint8_t(lo | (hi << 4));
        }
    }
    d += hdr;
    if (t < 16) d[t] = uint8_t(r.stream_len[t >> 2] >> (8 * (t & 3)));
    d += 16;
    for (uint32_t s = 0; s < 4; ++s) {
        block_copy_reversed(d, slots + c.slot_off + uint64_t(s) * c.slot_cap, r.stream_len[s], t, nt);
        d += r.stream_len[s];
    }
}

__global__ void __launch_bounds__(128) gather_kernel(const EncChunk* __restrict__ chunks, const EncResult* __restrict__ results, const ChunkPlace* __restrict__ places,
                                                     const PlaneDst* __restrict__ dsts, const uint8_t* __restrict__ planes, const uint8_t* __restrict__ tables,
                                                     const uint8_t* __restrict__ slots, uint8_t* __restrict__ out) {
    const EncChunk c = chunks[blockIdx.x];
    const PlaneDst dst = dsts[c.plane];
    if (dst.frames == ENC_NOWHERE) return;
    const ChunkPlace place = places[blockIdx.x];
    if (dst.table != ENC_NOWHERE && threadIdx.x == 127) {  // the chunk's entry in the plane's table: frame offset, decoded length
        uint8_t* e = out + dst.table + place.entry;
        e += put_varint_dev(e, place.frame);
        put_varint_dev(e, c.n);
    }
    gather_frame(out + dst.frames + place.frame, c, results[blockIdx.x], place.mode, planes, tables, slots, threadIdx.x, blockDim.x);
}
// The payload of one plane, in the form its coded size calls for and without a frame, by all blocks; nothing where it does not fit.
__global__ void __launch_bounds__(512) gather_one_kernel(const EncChunk* __restrict__ chunk, const EncResult* __restrict__ result, uint32_t codec, const uint8_t* __restrict__ planes,
                                                         const uint8_t* __restrict__ tables, const uint8_t* __restrict__ slots, uint8_t* __restrict__ out, uint64_t out_cap) {
    const EncChunk c = *chunk;
    const EncResult r = *result;
    uint32_t mode;
    if (enc_payload(int(codec), false, c.n, r, mode) > out_cap) return;
    gather_frame(out, c, r, mode | GATHER_BARE, planes, tables, slots, blockIdx.x * 512 + threadIdx.x, gridDim.x * 512);
}

// ---- ops between a byte split and a terminal (transforms/int_delta.rs:36-44, transforms/mantissa_zero.rs) ------
// IntDelta forward, byte width: every byte minus the one before it, modulo 256, over the whole plane (out of place).
__global__ void __launch_bounds__(256) delta_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, uint64_t n) {
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        dst[i] = uint8_t(src[i] - (i ? src[i - 1] : 0));
}
// OR of all bytes of a plane: MantissaZeroStrip(k) applies when the low k bits of that are clear.
__global__ void __launch_bounds__(256) or_bytes_kernel(const uint8_t* __restrict__ src, uint64_t n, uint32_t* __restrict__ out) {
    uint32_t v = 0;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) v |= src[i];
    v = __reduce_or_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicOr(out, v);
}
__global__ void __launch_bounds__(256) shift_right_kernel(uint8_t* __restrict__ p, uint64_t n, uint32_t k) {
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) p[i] = uint8_t(p[i] >> k);
}
// The chunk histograms of a plane whose bytes were just shifted right by k (all with k clear low bits): count v moves to v >> k.
__global__ void __launch_bounds__(256) relabel_hist_kernel(uint32_t* __restrict__ hist, uint32_t first_chunk, uint32_t k) {
    uint32_t* h = hist + uint64_t(first_chunk + blockIdx.x) * 256;
    const uint32_t v = threadIdx.x, c = h[v];
    __syncthreads();
    h[v] = 0;
    __syncthreads();
    if (c) h[v >> k] = c;
}

// ---- Order1ScaleAC encode (codecs/order1_scale_ac.rs:620-663, 963-1025) -------------------------------------
// Lag-1 counts of one chunk: the first symbol of a row counts toward the marginal, every other symbol toward the row
// of the symbol before it.  One CTA per listed chunk; the count areas were cleared beforehand.
__global__ void __launch_bounds__(256) o1sac_count_kernel(const EncChunk* __restrict__ chunks, const uint32_t* __restrict__ list, const uint8_t* __restrict__ planes,
                                                          uint8_t* __restrict__ tables) {
    const EncChunk c = chunks[list[blockIdx.x]];
    uint32_t* joint = reinterpret_cast<uint32_t*>(tables + c.table_off + O1E_JOINT);
    uint32_t* marg = reinterpret_cast<uint32_t*>(tables + c.table_off + O1E_MARG);
    const uint8_t* p = planes + c.plane_off;
    const uint32_t row_len = c.row_len ? c.row_len : (c.n ? c.n : 1);
    for (uint32_t i = threadIdx.x; i < c.n; i += blockDim.x) {
        if (i % row_len == 0) atomicAdd(&marg[p[i]], 1u);
        else atomicAdd(&joint[uint32_t(p[i - 1]) * 256 + p[i]], 1u);
    }
}
// Probability rows from the counts (a context gets a row when it was seen at all), their cumulative sums for the coder,
// and the rank of every present context (its place among the rows of the serialized state).  One CTA of 288 threads per chunk:
// thread c < 256 owns context c, thread 256 the marginal.
__global__ void __launch_bounds__(288) o1sac_fit_kernel(const EncChunk* __restrict__ chunks, const uint32_t* __restrict__ list, uint8_t* __restrict__ tables,
                                                        EncResult* __restrict__ results) {
    const uint32_t ci = list[blockIdx.x];
    uint8_t* tab = tables + chunks[ci].table_off;
    const uint32_t* joint = reinterpret_cast<const uint32_t*>(tab + O1E_JOINT);
    const uint32_t* marg = reinterpret_cast<const uint32_t*>(tab + O1E_MARG);
    uint8_t* present = tab + O1E_PRESENT;
    uint16_t* rank = reinterpret_cast<uint16_t*>(tab + O1E_RANK);
    uint16_t* pmf = reinterpret_cast<uint16_t*>(tab + O1E_PMF);
    uint16_t* cum = reinterpret_cast<uint16_t*>(tab + O1E_CUM);
    const uint32_t t = threadIdx.x;
    __shared__ uint32_t seen[256];
    if (t <= 256) {
        const uint32_t* raw = t < 256 ? joint + 256 * t : marg;
        const uint32_t row = t < 256 ? 1 + t : 0;
        bool use = true;
        if (t < 256) {
            uint64_t total = 0;
            for (int i = 0; i < 256; ++i) total += raw[i];
            use = total != 0;
            present[t] = use;
            seen[t] = use;
        }
        if (use) {
            uint16_t* out = pmf + 256 * row;
            quantize_pmf256(raw, O1SAC_TOTAL, out);
            uint32_t acc = 0;
            for (int i = 0; i < 256; ++i) { cum[256 * row + i] = uint16_t(acc); acc += out[i]; }
        }
    }
    __syncthreads();
    if (t == 0) {
        uint32_t k = 0;
        for (int ctx = 0; ctx < 256; ++ctx) { rank[ctx] = uint16_t(k); k += seen[ctx]; }
        results[ci].hdr_n = k;
        results[ci].stream_len[1] = 32 + 512 + 512 * k;
        results[ci].coded = 1;
    }
}
// The range coder over one chunk (range_coder.rs:16-113): 64-bit low, 32-bit range, carry held back in a cache byte and
// a run of 0xFF bytes; total 4096 makes range / total a shift.  One thread per listed chunk, bytes upward from the
// start of the chunk's slot area.
__global__ void __launch_bounds__(64) o1sac_encode_kernel(const EncChunk* __restrict__ chunks, const uint32_t* __restrict__ list, uint32_t n_list,
                                                          const uint8_t* __restrict__ planes, const uint8_t* __restrict__ tables, uint8_t* __restrict__ slots,
                                                          EncResult* __restrict__ results) {
    const uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= n_list) return;
    const uint32_t ci = list[li];
    const EncChunk c = chunks[ci];
    const uint8_t* tab = tables + c.table_off;
    const uint8_t* present = tab + O1E_PRESENT;
    const uint16_t* pmf = reinterpret_cast<const uint16_t*>(tab + O1E_PMF);
    const uint16_t* cum = reinterpret_cast<const uint16_t*>(tab + O1E_CUM);
    const uint8_t* p = planes + c.plane_off;
    uint8_t* out = slots + c.slot_off;
    uint32_t written = 0;
    uint64_t low = 0, range = 0xFFFFFFFFull;
    uint32_t cache = 0, cache_size = 0;
    auto shift_low = [&]() {
        const uint32_t carry = uint32_t(low >> 32) & 0xFFu, top = uint32_t(low >> 24) & 0xFFu;
        if (top == 0xFF && carry == 0) ++cache_size;
        else {
            out[written++] = uint8_t(cache + carry);
            const uint8_t fill = carry ? 0x00 : 0xFF;
            for (uint32_t i = 0; i < cache_size; ++i) out[written++] = fill;
            cache_size = 0;
            cache = top;
        }
        low = (low & 0x00FFFFFFull) << 8;
    };
    const uint32_t row_len = c.row_len ? c.row_len : (c.n ? c.n : 1);
    uint32_t in_row = 0, row = 0;
    for (uint32_t i = 0; i < c.n; ++i) {
        const uint32_t sym = p[i];
        const uint32_t cu = cum[256 * row + sym], pr = pmf[256 * row + sym];
        const uint64_t rpt = range >> 12;
        low += uint64_t(cu) * rpt;
        range = uint64_t(pr) * rpt;
        while (range < (1ull << 24)) { shift_low(); range <<= 8; }
        if (++in_row == row_len) { in_row = 0; row = 0; }
        else row = present[sym] ? 1 + sym : 0;
    }
    for (int i = 0; i < 5; ++i) shift_low();
    out[written++] = uint8_t(cache);
    for (uint32_t i = 0; i < cache_size; ++i) out[written++] = 0xFF;
    results[ci].stream_len[0] = written;
}

// Scatter host-built byte pieces (record headers, index, footer) into the container.
__global__ void __launch_bounds__(128) scatter_kernel(const uint8_t* __restrict__ staged, const uint64_t* __restrict__ triples, uint8_t* __restrict__ out) {
    uint64_t dst = triples[3 * blockIdx.x], src = triples[3 * blockIdx.x + 1], len = triples[3 * blockIdx.x + 2];
    for (uint64_t i = threadIdx.x; i < len; i += blockDim.x) out[dst + i] = staged[src + i];
}

}  // namespace ptwm
