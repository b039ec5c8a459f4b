// Code/table construction of the encoders, usable from host and device code.
// They must make the same choices as the reference's encoders so that the
// bytes written equal what ptwm-core would write for the same plane:
//   rANS     entropy/rans/compress.rs:72-122 (normalize_freqs)
//   Huffman  entropy/huffman/tree.rs:19-85 (from_frequencies), :212-242
//            (enforce_max_code_length)
//   tANS     entropy/tans/mod.rs:153-194 (normalize)
//   O1SAC    quantize.rs:13-45 (quantize_pmf)
#pragma once
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <utility>

namespace ptwm {

// Normalised rANS frequencies (sum 2048, every present symbol >= 1; the
// rounding excess or deficit goes to the first most frequent symbol).
// Returns max_sym, or -1 when the plane must be stored raw.
__host__ __device__ inline int rans_normalize(const uint32_t* raw, uint64_t total, uint16_t* freqs) {
    if (total == 0) return -1;
    uint32_t assigned = 0;
    int max_sym = 0, max_freq_sym = 0;
    for (int i = 0; i < 256; ++i) {
        freqs[i] = 0;
        if (raw[i] > 0) {
            uint64_t f = uint64_t(raw[i]) * 2048u / total;
            if (f < 1) f = 1;
            freqs[i] = uint16_t(f);
            assigned += uint32_t(f);
            max_sym = i;
            if (raw[i] > raw[max_freq_sym]) max_freq_sym = i;
        }
    }
    if (assigned > 2048) {
        uint32_t excess = assigned - 2048;
        if (freqs[max_freq_sym] > excess) freqs[max_freq_sym] = uint16_t(freqs[max_freq_sym] - excess);
        else return -1;
    } else if (assigned < 2048) {
        freqs[max_freq_sym] = uint16_t(freqs[max_freq_sym] + (2048 - assigned));
    }
    return max_sym;
}

// Normalised tANS frequencies (sum 2048): floor(c * 2048 / total) with a floor
// of one; an excess is taken one at a time from the first largest entry above
// one, a deficit goes to the first most frequent symbol.  Returns the number
// of present symbols.
__host__ __device__ inline int tans_normalize(const uint32_t* counts, uint64_t total, uint16_t* norm) {
    uint32_t sum = 0, max_count = 0;
    int max_sym = 0, nsym = 0;
    for (int s = 0; s < 256; ++s) {
        norm[s] = 0;
        const uint32_t c = counts[s];
        if (c == 0) continue;
        uint32_t v = uint32_t(uint64_t(c) * 2048u / total);
        if (v == 0) v = 1;
        norm[s] = uint16_t(v); sum += v; ++nsym;
        if (c > max_count) { max_count = c; max_sym = s; }
    }
    while (sum > 2048) {
        int bi = -1; uint32_t bv = 1;
        for (int s = 0; s < 256; ++s) if (norm[s] > bv) { bv = norm[s]; bi = s; }
        if (bi < 0) break;
        norm[bi]--; sum--;
    }
    if (sum < 2048) norm[max_sym] = uint16_t(norm[max_sym] + (2048 - sum));
    return nsym;
}

// Probability row of the Order1ScaleAC state from raw counts: Laplace +1,
// scaled to `total` and rounded half away from zero in double precision, at
// least one each; then the last largest entry is shaved, or the first smallest
// grown, until the row sums to `total`.
__host__ __device__ inline void quantize_pmf256(const uint32_t* raw, uint32_t total, uint16_t* out) {
    double sum = 0;
    for (int i = 0; i < 256; ++i) sum += double(raw[i] + 1);
    uint32_t current = 0;
    for (int i = 0; i < 256; ++i) {
        double v = round((double(raw[i] + 1) / sum) * double(total));
        if (v < 1.0) v = 1.0;
        out[i] = uint16_t(v);
        current += out[i];
    }
    while (current > total) {
        int am = 0;
        for (int i = 0; i < 256; ++i) if (out[i] >= out[am]) am = i;
        if (out[am] > 1) { out[am]--; current--; } else break;
    }
    while (current < total) {
        int am = 0;
        for (int i = 0; i < 256; ++i) if (out[i] < out[am]) am = i;
        out[am]++; current++;
    }
}

// Huffman code lengths for a histogram: repeated merge of the two smallest
// nodes under the (frequency, node id) order, leaves numbered in symbol order
// and internal nodes after them; depth clamp to 11 with the reference's Kraft
// repair.  Merged nodes come out in increasing frequency order, so with sorted
// leaves two queues replace the heap (a leaf first on equal frequencies: its
// id is smaller).  Returns the number of weights to store (last used symbol +
// 1), or 0 when there is no symbol.  (The device code's own version is
// warp_huffman_lengths.)
inline int huffman_lengths(const unsigned long long* raw, uint8_t* lengths) {
    std::pair<unsigned long long, int> leaf[256];
    int n = 0, last = -1;
    for (int i = 0; i < 256; ++i) { lengths[i] = 0; if (raw[i]) { leaf[n++] = {raw[i], i}; last = i; } }
    if (n == 0) return 0;
    if (n == 1) { lengths[last] = 1; return last + 1; }
    std::sort(leaf, leaf + n);
    unsigned long long node[256];
    int leaf_parent[256], node_parent[256], depth[256];
    for (int made = 0, i = 0, j = 0; made < n - 1; ++made) {
        unsigned long long sum = 0;
        for (int k = 0; k < 2; ++k) {
            if (i < n && (j >= made || leaf[i].first <= node[j])) { sum += leaf[i].first; leaf_parent[i++] = made; }
            else { sum += node[j]; node_parent[j++] = made; }
        }
        node[made] = sum;
    }
    depth[n - 2] = 0;
    for (int k = n - 3; k >= 0; --k) depth[k] = depth[node_parent[k]] + 1;
    uint32_t kraft = 0;
    for (int i = 0; i < n; ++i) {
        const int d = depth[leaf_parent[i]] + 1;
        lengths[leaf[i].second] = uint8_t(d > 11 ? 11 : d);
        kraft += 1u << (11 - lengths[leaf[i].second]);
    }
    while (kraft > 2048) {
        int victim = -1;
        for (int s = 0; s < 256; ++s) if (lengths[s] > 0 && lengths[s] < 11 && (victim < 0 || lengths[s] < lengths[victim])) victim = s;
        if (victim < 0) break;
        lengths[victim]++;
        kraft -= 1u << (11 - lengths[victim]);
    }
    return last + 1;
}

// A single plane of n bytes through the plane call: bytes of one of its four stream slots (a symbol takes at most 12 bits in any of the
// codecs; slots start on 16-byte boundaries and are written in aligned words), and whether the call takes planes that long.
__host__ __device__ inline uint64_t plane_slot_bytes(uint64_t n) { return ((n / 4 + 1) * 12 + 7) / 8 + 64; }
__host__ __device__ inline uint64_t plane_slot_cap(uint64_t n) { return (plane_slot_bytes(n) + 15) / 16 * 16; }
__host__ __device__ inline bool plane_codable(uint64_t n) { return plane_slot_bytes(n) <= 0x3FFFFFFFull; }

// tANS: symbols per lane when a warp codes a chunk of n.  Any 32-bit n: the lanes' runs cover it.
constexpr uint32_t TENC_MIN_RUN = 256;  // shorter runs would hardly ever end in the right state
__host__ __device__ inline uint32_t tans_encode_run(uint32_t n) {
    const uint32_t per = n / 32 + (n % 32 != 0);
    return per < TENC_MIN_RUN ? TENC_MIN_RUN : per;
}

}  // namespace ptwm
