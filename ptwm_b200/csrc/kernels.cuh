// Device code of the PTWM decode path for sm_100a: chunk-parallel rANS /
// canonical-Huffman / tANS / Order1ScaleAC decoders with the plane merge and
// inverse bit reorder fused into their epilogue, the stand-alone merge kernel
// and the integrity kernels (CRC-32 of the re-split planes, XXH64).
//
// Bit-exact targets, all under crates/ptwm-core/src of the reference:
//   rANS        entropy/rans/decompress.rs:24-164
//   Huffman     entropy/huffman/{weights.rs:34-85, tree.rs:103-177, bitstream.rs:54-187, decompress.rs:8-211}
//   tANS        entropy/tans/mod.rs:199-211,346-451
//   O1SAC       range_coder.rs:122-198, codecs/order1_scale_ac.rs:85-151,474-486,665-706
//   merges      transforms/fusion.rs:124-193,264-315,373-417,475-519
//
// All of this is integer / byte work bounded by instruction issue, shared
// memory capacity and HBM; nothing here is GEMM-shaped, so no tensor cores.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "plan.h"

namespace ptwm {

__device__ __forceinline__ const uint8_t* rd(const Bases& b, Ref r) {
    uint64_t off = r & ((1ull << 62) - 1);
    uint32_t sp = uint32_t(r >> 62);
    return sp == SP_BLOB ? b.blob + off : sp == SP_SCRATCH ? b.scratch + off : b.out + off;
}
__device__ __forceinline__ uint8_t* wr(const Bases& b, Ref r) {
    uint64_t off = r & ((1ull << 62) - 1);
    return (uint32_t(r >> 62) == SP_SCRATCH ? b.scratch : b.out) + off;
}

// A failed item: its own status word, and the word before the first one, which is all the host looks at when nothing failed.
__device__ __forceinline__ void report(uint32_t* status, uint32_t id, uint32_t err) {
    atomicMax(&status[id], err);
    atomicMax(status - 1, err);
}

__device__ __forceinline__ uint32_t ld_u32_unaligned(const uint8_t* p) {
    return uint32_t(p[0]) | uint32_t(p[1]) << 8 | uint32_t(p[2]) << 16 | uint32_t(p[3]) << 24;
}

// Eight bytes from any address.  The two aligned words both overlap the
// requested range, so nothing outside the 8-byte-aligned span of the source
// is touched.
__device__ __forceinline__ uint64_t ld8_unaligned(const uint8_t* p) {
    uintptr_t a = reinterpret_cast<uintptr_t>(p);
    uint32_t sh = uint32_t(a & 7) * 8;
    const uint64_t* q = reinterpret_cast<const uint64_t*>(a & ~uintptr_t(7));
    uint64_t lo = __ldg(q);
    if (sh == 0) return lo;
    uint64_t hi = __ldg(q + 1);
    return (lo >> sh) | (hi << (64 - sh));
}
__device__ __forceinline__ uint64_t ld_bytes(const uint8_t* p, uint32_t count) {
    uint64_t v = 0;
    for (uint32_t i = 0; i < count; ++i) v |= uint64_t(p[i]) << (8 * i);
    return v;
}

__device__ __forceinline__ void stg256(void* p, uint4 a, uint4 b);

// ---- element composition ---------------------------------------------------
__device__ __forceinline__ uint32_t revert16x2(uint32_t r) {  // split/dtype16.rs:20-25
    return ((r << 8) & 0x80008000u) | ((r >> 1) & 0x7F807F80u) | (r & 0x007F007Fu);
}
// Four 16-bit elements from four bytes of the low plane ([S M7]) and four of
// the high plane (E8): the bit reorder done on the packed planes, then the
// interleave.  Same result as revert16x2 on the interleaved words.
__device__ __forceinline__ void compose16x4(uint32_t lo, uint32_t hi, uint32_t& v0, uint32_t& v1) {
    uint32_t oh = (lo & 0x80808080u) | ((hi >> 1) & 0x7F7F7F7Fu);
    uint32_t ol = ((hi << 7) & 0x80808080u) | (lo & 0x7F7F7F7Fu);
    v0 = __byte_perm(ol, oh, 0x5140);
    v1 = __byte_perm(ol, oh, 0x7362);
}
__device__ __forceinline__ uint32_t revert32(uint32_t r) {  // transforms/fusion.rs:287-292
    return ((r << 8) & 0x80000000u) | ((r >> 1) & 0x7F800000u) | (r & 0x007FFFFFu);
}
__device__ __forceinline__ uint64_t revert_fp8x8(uint64_t h, uint64_t l, bool e4m3) {  // split/dtype8.rs:39-44,57-62
    uint64_t r = ((h & 0x0F0F0F0F0F0F0F0Full) << 4) | (l & 0x0F0F0F0F0F0F0F0Full);
    return e4m3 ? ((r & 0xF0F0F0F0F0F0F0F0ull) >> 1) | ((r & 0x0808080808080808ull) << 4) | (r & 0x0707070707070707ull)
                : ((r & 0xF8F8F8F8F8F8F8F8ull) >> 1) | ((r & 0x0404040404040404ull) << 5) | (r & 0x0303030303030303ull);
}

// Store `count` (<= 8) elements starting at element `pos` of a tensor whose
// planes' bytes for those elements are b[0..np).  Full groups on aligned
// addresses go out as 128-bit (or 64-bit) stores.
__device__ __forceinline__ void compose_store(int kind, uint8_t* dst, uint64_t pos, uint32_t count, const uint64_t b[4]) {
    switch (kind) {
        case K_PASS: {
            uint8_t* p = dst + pos;
            if (count == 8 && (reinterpret_cast<uintptr_t>(p) & 7) == 0) *reinterpret_cast<uint64_t*>(p) = b[0];
            else for (uint32_t i = 0; i < count; ++i) p[i] = uint8_t(b[0] >> (8 * i));
            break;
        }
        case K_E4M3:
        case K_E5M2: {
            uint64_t v = revert_fp8x8(b[0], b[1], kind == K_E4M3);
            uint8_t* p = dst + pos;
            if (count == 8 && (reinterpret_cast<uintptr_t>(p) & 7) == 0) *reinterpret_cast<uint64_t*>(p) = v;
            else for (uint32_t i = 0; i < count; ++i) p[i] = uint8_t(v >> (8 * i));
            break;
        }
        case K_M16: {
            uint32_t l0 = uint32_t(b[0]), l1 = uint32_t(b[0] >> 32), h0 = uint32_t(b[1]), h1 = uint32_t(b[1] >> 32);
            uint4 v;
            compose16x4(l0, h0, v.x, v.y);
            compose16x4(l1, h1, v.z, v.w);
            uint8_t* p = dst + pos * 2;
            if (count == 8 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) *reinterpret_cast<uint4*>(p) = v;
            else {
                uint32_t w[4] = {v.x, v.y, v.z, v.w};
                for (uint32_t i = 0; i < count; ++i) {
                    uint32_t e = (w[i >> 1] >> (16 * (i & 1))) & 0xFFFF;
                    p[2 * i] = uint8_t(e); p[2 * i + 1] = uint8_t(e >> 8);
                }
            }
            break;
        }
        case K_M32: {
            uint32_t w[8];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t p0 = uint32_t(b[0] >> (32 * half)), p1 = uint32_t(b[1] >> (32 * half)), p2 = uint32_t(b[2] >> (32 * half)),
                         p3 = uint32_t(b[3] >> (32 * half));
                uint32_t t0 = __byte_perm(p0, p1, 0x5140), t1 = __byte_perm(p2, p3, 0x5140);
                uint32_t t2 = __byte_perm(p0, p1, 0x7362), t3 = __byte_perm(p2, p3, 0x7362);
                w[4 * half + 0] = revert32(__byte_perm(t0, t1, 0x5410));
                w[4 * half + 1] = revert32(__byte_perm(t0, t1, 0x7632));
                w[4 * half + 2] = revert32(__byte_perm(t2, t3, 0x5410));
                w[4 * half + 3] = revert32(__byte_perm(t2, t3, 0x7632));
            }
            uint8_t* p = dst + pos * 4;
            if (count == 8 && (reinterpret_cast<uintptr_t>(p) & 31) == 0) {
                stg256(p, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));  // one sector per lane and instruction
            } else if (count == 8 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
                reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
            } else {
                for (uint32_t i = 0; i < count; ++i) {
                    p[4 * i] = uint8_t(w[i]); p[4 * i + 1] = uint8_t(w[i] >> 8); p[4 * i + 2] = uint8_t(w[i] >> 16); p[4 * i + 3] = uint8_t(w[i] >> 24);
                }
            }
            break;
        }
    }
}

// Epilogue of a decoding lane: where its symbols go.
struct Epilogue {
    uint8_t* dst;
    const uint8_t* partner[3];
    int kind, slot, fused;
};
__device__ __forceinline__ Epilogue make_epilogue(const Bases& bases, const DecodeItem& it) {
    Epilogue e;
    e.dst = wr(bases, it.dst);
    e.kind = it.kind; e.slot = it.slot; e.fused = it.fused;
    int np = it.fused ? kind_planes(it.kind) : 1;
    for (int j = 0; j < 3; ++j) e.partner[j] = (j < np - 1) ? rd(bases, it.partner[j]) : nullptr;
    return e;
}
// Bytes of the other planes for `count` elements at `pos` (fused lanes only).
// Issued before the group's symbols are decoded so the loads overlap the decode.
__device__ __forceinline__ void gather_partners(const Epilogue& e, uint64_t pos, uint32_t count, uint64_t b[4]) {
    b[0] = b[1] = b[2] = b[3] = 0;
    if (!e.fused) return;
    int np = kind_planes(e.kind);
    int j = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        if (p >= np) break;
        if (p == e.slot) continue;
        const uint8_t* q = e.partner[j++] + pos;
        b[p] = count == 8 ? ld8_unaligned(q) : ld_bytes(q, count);
    }
}
// `pos` is the symbol index inside the chunk, `syms` holds `count` symbols,
// b[] the partner bytes from gather_partners.
__device__ __forceinline__ void emit_with(const Epilogue& e, uint64_t pos, uint32_t count, uint64_t syms, uint64_t b[4]) {
    if (!e.fused) { b[0] = syms; compose_store(K_PASS, e.dst, pos, count, b); return; }
#pragma unroll
    for (int p = 0; p < 4; ++p) if (p == e.slot) b[p] = syms;
    compose_store(e.kind, e.dst, pos, count, b);
}
__device__ __forceinline__ void emit(const Epilogue& e, uint64_t pos, uint32_t count, uint64_t syms) {
    uint64_t b[4];
    gather_partners(e, pos, count, b);
    emit_with(e, pos, count, syms, b);
}
// The other planes' bytes of a fused lane, read as a stream of aligned 8-byte
// words one group ahead of their use: a group of eight elements needs the
// words w0 and w1, the word after them is requested while the group's symbols
// are still being decoded, so its DRAM latency hides behind the decode.
struct PartnerStream {
    const uint64_t* q[3];    // word that holds the first byte of the current group
    const uint64_t* lim[3];  // first word that must not be read
    uint64_t w0[3], w1[3], w2[3];
    uint32_t sh[3];
    int n;                   // partners (planes - 1), 0 for a plain lane
    __device__ __forceinline__ void start(const Epilogue& e, uint64_t pos, uint32_t chunk_n) {
        n = e.fused ? kind_planes(e.kind) - 1 : 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j >= n) break;
            uintptr_t a = reinterpret_cast<uintptr_t>(e.partner[j]) + pos;
            q[j] = reinterpret_cast<const uint64_t*>(a & ~uintptr_t(7));
            sh[j] = uint32_t(a & 7) * 8;
            lim[j] = reinterpret_cast<const uint64_t*>((reinterpret_cast<uintptr_t>(e.partner[j]) + chunk_n + 7) & ~uintptr_t(7));
            w0[j] = q[j] < lim[j] ? __ldg(q[j]) : 0;
            w1[j] = q[j] + 1 < lim[j] ? __ldg(q[j] + 1) : 0;
        }
    }
    __device__ __forceinline__ void prefetch() {
#pragma unroll
        for (int j = 0; j < 3; ++j) { if (j >= n) break; w2[j] = q[j] + 2 < lim[j] ? __ldg(q[j] + 2) : 0; }
    }
    // plane bytes of the current group into b[] (slot = the plane the lane itself decodes), then step to the next group
    __device__ __forceinline__ void take(int slot, uint64_t b[4]) {
        int p = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j >= n) break;
            if (p == slot) ++p;
            b[p++] = sh[j] ? (w0[j] >> sh[j]) | (w1[j] << (64 - sh[j])) : w0[j];
            w0[j] = w1[j]; w1[j] = w2[j]; q[j] += 1;
        }
    }
};

// Length of the first group so that later groups start on an 8-element
// boundary of the destination.
__device__ __forceinline__ uint32_t first_group(const Epilogue& e, uint64_t pos, uint32_t remaining) {
    uintptr_t a = reinterpret_cast<uintptr_t>(e.dst) / uint32_t(e.fused ? kind_elem_bytes(e.kind) : 1) + pos;
    uint32_t g = 8 - uint32_t(a & 7);
    return g < remaining ? g : remaining;
}

__device__ __forceinline__ void split_four_dev(uint32_t n, uint32_t s, uint32_t& start, uint32_t& len) {  // entropy/stream_frame.rs:27-41
    uint32_t base = n >> 2, rem = n & 3;
    len = base + (s < rem ? 1u : 0u);
    start = s * base + (s < rem ? s : rem);
}

// 256-bit global accesses (sm_100): a lane that walks its own stream touches
// one 32-byte sector per instruction instead of half of one, which halves the
// load/store-pipe cost of these scattered accesses.  Nothing in such a sector is touched twice, and with the tables taking the shared memory
// little is left of the L1 that so many lanes' lines would go through: without a place there the six-layer bf16 rANS model takes 4103 instead of
// 4775 us (loads alone 8 % less, stores alone 9 %).  The 16-byte blocks of a stream do come from a sector twice and are kept.
struct Block32 { uint32_t w[8]; };
__device__ __forceinline__ Block32 ldg256(const void* p) {
    Block32 b;
    asm("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(b.w[0]), "=r"(b.w[1]), "=r"(b.w[2]), "=r"(b.w[3]), "=r"(b.w[4]), "=r"(b.w[5]), "=r"(b.w[6]), "=r"(b.w[7])
        : "l"(p));
    return b;
}
__device__ __forceinline__ void stg256(void* p, uint4 a, uint4 b) {
    asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
// The same for bytes that the block reads again.
__device__ __forceinline__ void stg256_kept(void* p, uint4 a, uint4 b) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
// Aligned 32-byte block at `a`; bytes outside [lo, hi) read as zero and are not touched.
__device__ __forceinline__ Block32 load_block_guarded(uintptr_t a, uintptr_t lo, uintptr_t hi) {
    if (a >= lo && a + 32 <= hi) return ldg256(reinterpret_cast<const void*>(a));
    Block32 b;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        uint32_t v = 0;
        for (int i = 0; i < 4; ++i) {
            uintptr_t q = a + 4 * k + i;
            if (q >= lo && q < hi) v |= uint32_t(__ldg(reinterpret_cast<const uint8_t*>(q))) << (8 * i);
        }
        b.w[k] = v;
    }
    return b;
}
// The 32 bytes that start `off` (0..31) bytes into the 64 bytes (cur, nxt), as eight words.
__device__ __forceinline__ void extract32(const Block32& cur, const Block32& nxt, uint32_t off, uint32_t out[8]) {
    uint32_t a[16], b[12], c[10], d[9];
#pragma unroll
    for (int i = 0; i < 8; ++i) { a[i] = cur.w[i]; a[8 + i] = nxt.w[i]; }
    const bool j4 = off & 16, j2 = off & 8, j1 = off & 4;
#pragma unroll
    for (int i = 0; i < 12; ++i) b[i] = j4 ? a[i + 4] : a[i];
#pragma unroll
    for (int i = 0; i < 10; ++i) c[i] = j2 ? b[i + 2] : b[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) d[i] = j1 ? c[i + 1] : c[i];
    const uint32_t sel = 0x3210u + 0x1111u * (off & 3u);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = __byte_perm(d[i], d[i + 1], sel);
}

// ---- fast output loops of a decoding lane -----------------------------------
// `dec8(s_lo, s_hi)` decodes the lane's next eight symbols (symbol j in byte
// j & 3 of s_lo for j < 4, of s_hi above); the loops below place them.
//
// Fused lane, 16-bit elements, one partner plane.  Rounds of 32 elements: the
// partner bytes come as aligned 32-byte blocks two rounds ahead of their use
// (cur, nxt, and one in flight), the composed elements leave as two 32-byte
// stores.  Blocks that are not wholly inside the partner's chunk are never read
// whole, so nothing outside the caller's buffers is touched.  What does not
// fill a round is left to the caller.
template <class Dec8>
__device__ __forceinline__ void fused16_rounds(const Epilogue& ep, uint32_t chunk_n, uint32_t& pos, uint32_t& remaining, Dec8&& dec8) {
    if (remaining >= 8 && ((reinterpret_cast<uintptr_t>(ep.dst) + size_t(pos) * 2) & 31) != 0) {
        uint32_t s_lo, s_hi;  // one more group of eight brings the destination to a 32-byte boundary
        dec8(s_lo, s_hi);
        emit(ep, pos, 8, uint64_t(s_lo) | uint64_t(s_hi) << 32);
        pos += 8; remaining -= 8;
    }
    const uintptr_t p_lo = reinterpret_cast<uintptr_t>(ep.partner[0]), p_hi = p_lo + chunk_n;
    const uintptr_t pa = p_lo + pos;
    uintptr_t q = pa & ~uintptr_t(31);
    uint8_t* out = ep.dst + size_t(pos) * 2;
    // round r reads the block at q + 32 (r + 2): it must end inside the chunk
    uint32_t rounds = 0;
    if ((reinterpret_cast<uintptr_t>(out) & 31) == 0 && q + 96 <= p_hi) {
        rounds = uint32_t((p_hi - q - 96) >> 5) + 1;
        if (rounds > (remaining >> 5)) rounds = remaining >> 5;
    }
    if (!rounds) return;
    const uint32_t off = uint32_t(pa & 31);
    const bool low_plane = ep.slot == 0;  // the lane decodes the low bytes, the partner holds the high bytes
    Block32 cur = load_block_guarded(q, p_lo, p_hi), nxt = ldg256(reinterpret_cast<const void*>(q + 32));
    for (uint32_t r = 0; r < rounds; ++r) {
        const Block32 ahead = ldg256(reinterpret_cast<const void*>(q + 64));
        uint32_t pw[8];
        uint4 v[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint32_t s_lo, s_hi;
            dec8(s_lo, s_hi);
            if (g == 0) extract32(cur, nxt, off, pw);
            if (low_plane) { compose16x4(s_lo, pw[2 * g], v[g].x, v[g].y); compose16x4(s_hi, pw[2 * g + 1], v[g].z, v[g].w); }
            else { compose16x4(pw[2 * g], s_lo, v[g].x, v[g].y); compose16x4(pw[2 * g + 1], s_hi, v[g].z, v[g].w); }
        }
        stg256(out, v[0], v[1]);
        stg256(out + 32, v[2], v[3]);
        out += 64; q += 32;
        cur = nxt; nxt = ahead;
    }
    pos += rounds * 32; remaining -= rounds * 32;
}
// Fused lane, fp8 elements: the two nibble planes (one nibble per byte) of 32 elements become one 32-byte store.
__device__ __forceinline__ uint32_t compose_fp8x4(uint32_t hi, uint32_t lo, bool e4m3) {  // split/dtype8.rs:39-44,57-62 on four elements
    uint32_t r = ((hi & 0x0F0F0F0Fu) << 4) | (lo & 0x0F0F0F0Fu);
    return e4m3 ? ((r & 0xF0F0F0F0u) >> 1) | ((r & 0x08080808u) << 4) | (r & 0x07070707u)
                : ((r & 0xF8F8F8F8u) >> 1) | ((r & 0x04040404u) << 5) | (r & 0x03030303u);
}
template <class Dec8>
__device__ __forceinline__ void fused8_rounds(const Epilogue& ep, uint32_t chunk_n, uint32_t& pos, uint32_t& remaining, Dec8&& dec8) {
    while (remaining >= 8 && ((reinterpret_cast<uintptr_t>(ep.dst) + pos) & 31) != 0) {
        uint32_t s_lo, s_hi;  // groups of eight up to a 32-byte boundary of the destination
        dec8(s_lo, s_hi);
        emit(ep, pos, 8, uint64_t(s_lo) | uint64_t(s_hi) << 32);
        pos += 8; remaining -= 8;
    }
    const uintptr_t p_lo = reinterpret_cast<uintptr_t>(ep.partner[0]), p_hi = p_lo + chunk_n;
    const uintptr_t pa = p_lo + pos;
    uintptr_t q = pa & ~uintptr_t(31);
    uint8_t* out = ep.dst + pos;
    uint32_t rounds = 0;
    if ((reinterpret_cast<uintptr_t>(out) & 31) == 0 && q + 96 <= p_hi) {
        rounds = uint32_t((p_hi - q - 96) >> 5) + 1;
        if (rounds > (remaining >> 5)) rounds = remaining >> 5;
    }
    if (!rounds) return;
    const uint32_t off = uint32_t(pa & 31);
    const bool high_plane = ep.slot == 0, e4m3 = ep.kind == K_E4M3;  // plane 0 holds the high nibbles
    Block32 cur = load_block_guarded(q, p_lo, p_hi), nxt = ldg256(reinterpret_cast<const void*>(q + 32));
    for (uint32_t r = 0; r < rounds; ++r) {
        const Block32 ahead = ldg256(reinterpret_cast<const void*>(q + 64));
        uint32_t pw[8], v[8];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint32_t s_lo, s_hi;
            dec8(s_lo, s_hi);
            if (g == 0) extract32(cur, nxt, off, pw);
            v[2 * g] = high_plane ? compose_fp8x4(s_lo, pw[2 * g], e4m3) : compose_fp8x4(pw[2 * g], s_lo, e4m3);
            v[2 * g + 1] = high_plane ? compose_fp8x4(s_hi, pw[2 * g + 1], e4m3) : compose_fp8x4(pw[2 * g + 1], s_hi, e4m3);
        }
        stg256(out, make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]));
        out += 32; q += 32;
        cur = nxt; nxt = ahead;
    }
    pos += rounds * 32; remaining -= rounds * 32;
}
// Fused lane, 32-bit elements, the lane decoding plane 3 (the exponent byte, the usual case: the three mantissa
// planes are stored raw or were decoded before).  Rounds of 16 elements: each of the three partner planes arrives as
// aligned 16-byte blocks one round ahead, the composed elements leave as two 32-byte stores.
__device__ __forceinline__ uint4 load_block16_guarded(uintptr_t a, uintptr_t lo, uintptr_t hi) {
    if (a >= lo && a + 16 <= hi) return __ldg(reinterpret_cast<const uint4*>(a));
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint32_t v = 0;
        for (int i = 0; i < 4; ++i) {
            uintptr_t q = a + 4 * k + i;
            if (q >= lo && q < hi) v |= uint32_t(__ldg(reinterpret_cast<const uint8_t*>(q))) << (8 * i);
        }
        w[k] = v;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// The 16 bytes that start `off` (0..15) bytes into the 32 bytes (cur, nxt), as four words.
__device__ __forceinline__ void extract16(const uint4& cur, const uint4& nxt, uint32_t off, uint32_t out[4]) {
    const uint32_t a[8] = {cur.x, cur.y, cur.z, cur.w, nxt.x, nxt.y, nxt.z, nxt.w};
    uint32_t b[6], c[5];
    const bool j2 = off & 8, j1 = off & 4;
#pragma unroll
    for (int i = 0; i < 6; ++i) b[i] = j2 ? a[i + 2] : a[i];
#pragma unroll
    for (int i = 0; i < 5; ++i) c[i] = j1 ? b[i + 1] : b[i];
    const uint32_t sel = 0x3210u + 0x1111u * (off & 3u);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = __byte_perm(c[i], c[i + 1], sel);
}
// ---- sixteen elements of a merge --------------------------------------------
// Sixteen elements to `out`, which lies on a boundary of their size, from 16 bytes of every plane.
__device__ __forceinline__ void merge_store16(int kind, uint8_t* out, const uint32_t pw[4][4]) {
    switch (kind) {
        case K_PASS: *reinterpret_cast<uint4*>(out) = make_uint4(pw[0][0], pw[0][1], pw[0][2], pw[0][3]); break;
        case K_E4M3:
        case K_E5M2: {
            const bool e4m3 = kind == K_E4M3;
            *reinterpret_cast<uint4*>(out) = make_uint4(compose_fp8x4(pw[0][0], pw[1][0], e4m3), compose_fp8x4(pw[0][1], pw[1][1], e4m3),
                                                        compose_fp8x4(pw[0][2], pw[1][2], e4m3), compose_fp8x4(pw[0][3], pw[1][3], e4m3));
            break;
        }
        case K_M16: {
            uint4 v[2];
            compose16x4(pw[0][0], pw[1][0], v[0].x, v[0].y); compose16x4(pw[0][1], pw[1][1], v[0].z, v[0].w);
            compose16x4(pw[0][2], pw[1][2], v[1].x, v[1].y); compose16x4(pw[0][3], pw[1][3], v[1].z, v[1].w);
            stg256(out, v[0], v[1]);
            break;
        }
        default: {  // K_M32 (transforms/fusion.rs:287-292)
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
                uint32_t w[8];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t t0 = __byte_perm(pw[0][k + h], pw[1][k + h], 0x5140), t1 = __byte_perm(pw[2][k + h], pw[3][k + h], 0x5140);
                    const uint32_t t2 = __byte_perm(pw[0][k + h], pw[1][k + h], 0x7362), t3 = __byte_perm(pw[2][k + h], pw[3][k + h], 0x7362);
                    w[4 * h + 0] = revert32(__byte_perm(t0, t1, 0x5410));
                    w[4 * h + 1] = revert32(__byte_perm(t0, t1, 0x7632));
                    w[4 * h + 2] = revert32(__byte_perm(t2, t3, 0x5410));
                    w[4 * h + 3] = revert32(__byte_perm(t2, t3, 0x7632));
                }
                stg256(out + 16 * k, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
            }
            break;
        }
    }
}

template <class Dec8>
__device__ __forceinline__ void fused32_rounds(const Epilogue& ep, uint32_t chunk_n, uint32_t& pos, uint32_t& remaining, Dec8&& dec8) {
    uint8_t* out = ep.dst + size_t(pos) * 4;
    uintptr_t q[3], lo[3], hi[3];
    uint32_t off[3], rounds = remaining >> 4;
    if (reinterpret_cast<uintptr_t>(out) & 31) rounds = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        lo[j] = reinterpret_cast<uintptr_t>(ep.partner[j]); hi[j] = lo[j] + chunk_n;
        const uintptr_t pa = lo[j] + pos;
        q[j] = pa & ~uintptr_t(15); off[j] = uint32_t(pa & 15);
        // round r reads the block at q + 16 (r + 2): it must end inside the chunk
        const uint32_t fit = q[j] + 48 <= hi[j] ? uint32_t((hi[j] - q[j] - 48) >> 4) + 1 : 0;
        rounds = fit < rounds ? fit : rounds;
    }
    if (!rounds) return;
    uint4 cur[3], nxt[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) { cur[j] = load_block16_guarded(q[j], lo[j], hi[j]); nxt[j] = __ldg(reinterpret_cast<const uint4*>(q[j] + 16)); }
    for (uint32_t r = 0; r < rounds; ++r) {
        uint4 ahead[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) ahead[j] = __ldg(reinterpret_cast<const uint4*>(q[j] + 32));
        uint32_t sy[4], pw[3][4], w[16];
        dec8(sy[0], sy[1]);
        dec8(sy[2], sy[3]);
#pragma unroll
        for (int j = 0; j < 3; ++j) extract16(cur[j], nxt[j], off[j], pw[j]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // four elements: bytes 0..2 from the partner planes, byte 3 from this lane (transforms/fusion.rs:287-292)
            const uint32_t t0 = __byte_perm(pw[0][k], pw[1][k], 0x5140), t1 = __byte_perm(pw[2][k], sy[k], 0x5140);
            const uint32_t t2 = __byte_perm(pw[0][k], pw[1][k], 0x7362), t3 = __byte_perm(pw[2][k], sy[k], 0x7362);
            w[4 * k + 0] = revert32(__byte_perm(t0, t1, 0x5410));
            w[4 * k + 1] = revert32(__byte_perm(t0, t1, 0x7632));
            w[4 * k + 2] = revert32(__byte_perm(t2, t3, 0x5410));
            w[4 * k + 3] = revert32(__byte_perm(t2, t3, 0x7632));
        }
        stg256(out, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
        stg256(out + 32, make_uint4(w[8], w[9], w[10], w[11]), make_uint4(w[12], w[13], w[14], w[15]));
        out += 64;
#pragma unroll
        for (int j = 0; j < 3; ++j) { cur[j] = nxt[j]; nxt[j] = ahead[j]; q[j] += 16; }
    }
    pos += rounds * 16; remaining -= rounds * 16;
}
// Plain lane: eight symbols are eight bytes of the plane; 32 bytes per store.
template <class Dec8>
__device__ __forceinline__ void plain_rounds(const Epilogue& ep, uint32_t& pos, uint32_t& remaining, Dec8&& dec8) {
    uint8_t* out = ep.dst + pos;
    if (reinterpret_cast<uintptr_t>(out) & 7) return;
    while (remaining >= 8 && (reinterpret_cast<uintptr_t>(out) & 31) != 0) {
        uint32_t s_lo, s_hi;
        dec8(s_lo, s_hi);
        *reinterpret_cast<uint2*>(out) = make_uint2(s_lo, s_hi);
        out += 8; pos += 8; remaining -= 8;
    }
    const uint32_t rounds = remaining >> 5;
    for (uint32_t r = 0; r < rounds; ++r) {
        uint4 a, b;
        dec8(a.x, a.y); dec8(a.z, a.w); dec8(b.x, b.y); dec8(b.z, b.w);
        stg256(out, a, b);
        out += 32;
    }
    pos += rounds * 32; remaining -= rounds * 32;
}
// Other fused kinds: partner words streamed one group ahead, 128-bit stores.
template <class Dec8>
__device__ __forceinline__ void fused_groups(const Epilogue& ep, uint32_t chunk_n, uint32_t& pos, uint32_t& remaining, Dec8&& dec8) {
    if (remaining < 8) return;
    PartnerStream ps;
    ps.start(ep, pos, chunk_n);
    while (remaining >= 8) {
        uint32_t s_lo, s_hi;
        uint64_t pb[4] = {0, 0, 0, 0};
        ps.prefetch();
        dec8(s_lo, s_hi);
        ps.take(ep.slot, pb);
        emit_with(ep, pos, 8, uint64_t(s_lo) | uint64_t(s_hi) << 32, pb);
        pos += 8; remaining -= 8;
    }
}
template <class Dec8>
__device__ __forceinline__ void fast_groups(const Epilogue& ep, uint32_t chunk_n, uint32_t& pos, uint32_t& remaining, Dec8&& dec8) {
    if (!ep.fused) plain_rounds(ep, pos, remaining, dec8);
    else if (ep.kind == K_M16) fused16_rounds(ep, chunk_n, pos, remaining, dec8);
    else if (ep.kind == K_E4M3 || ep.kind == K_E5M2) fused8_rounds(ep, chunk_n, pos, remaining, dec8);
    else {
        if (ep.kind == K_M32 && ep.slot == 3) fused32_rounds(ep, chunk_n, pos, remaining, dec8);
        fused_groups(ep, chunk_n, pos, remaining, dec8);  // the other plane orders, and what the rounds left
    }
}

// ---- per-lane byte window over a stream ------------------------------------
// A lane reads its stream one byte (rANS, forward) or one aligned word
// (Huffman, backward) at a time.  Global memory is fetched in aligned 16-byte
// blocks one step ahead of use and parked in a 64-byte ring per lane in shared
// memory, laid out [ring word][lane] so that any mix of positions across the
// warp is bank-conflict free.
struct Ring {
    uint32_t* base;  // &ring[0][lane]
    __device__ __forceinline__ uint32_t& word(uintptr_t addr) { return base[((addr >> 2) & 15) * 32]; }
    __device__ __forceinline__ uint8_t byte(uintptr_t addr) { return reinterpret_cast<uint8_t*>(&word(addr))[addr & 3]; }
    __device__ __forceinline__ void put(uintptr_t addr16, uint4 v) {
        word(addr16) = v.x; word(addr16 + 4) = v.y; word(addr16 + 8) = v.z; word(addr16 + 12) = v.w;
    }
};
// Aligned 16-byte block, zero outside [lo16, hi16) (the 16-byte hull of the blob).
__device__ __forceinline__ uint4 fetch16(uintptr_t a, uintptr_t lo16, uintptr_t hi16) {
    if (a < lo16 || a >= hi16) return make_uint4(0, 0, 0, 0);
    return __ldg(reinterpret_cast<const uint4*>(a));
}

// ---- rANS ------------------------------------------------------------------
constexpr uint32_t RANS_L = 1u << 23;
constexpr int RANS_WARP_CHUNKS = 8;
constexpr int RING_SMEM = 16 * 32 * 4;
// How many distinct symbols a chunk may hold for the kernel that keeps a copy
// of the symbol list per lane (two pad entries come on top).
constexpr uint32_t RANS_NARROW_SYMBOLS = 38;
// From this many distinct symbols on a chunk counts as nearly incompressible (packed fp4 values, mantissa-like bytes).
constexpr uint32_t RANS_DENSE_SYMBOLS = 96;
// Shared memory per chunk:
//  * a rank table over the 2048 slots: 128 words of (16-bit boundary bitmap,
//    boundaries before the word << 16).  Bit i of a bitmap is set when slot
//    16 w + i is the first slot of a symbol, so the symbol covering a slot is
//    number count + popc(bits up to the slot) among the present symbols: 512
//    bytes instead of a byte per slot, and shared memory per chunk is what
//    bounds the number of streams an SM keeps in flight;
//  * one word per present symbol (symbol | freq << 8 | start << 20), entry 0 a
//    pad so that the count above indexes it directly.  Two layouts:
//    shared by the four lanes of a chunk, `l_entries` words per chunk (alphabet
//    bound + 2), any alphabet; or one copy per lane (PER_LANE), entry k of lane
//    l in word k * 32 + l, a bank of its own, so the read is conflict free.
//    `l_entries` is then the number of rows and bounds the distinct symbols of
//    a chunk; the host sends only chunks that fit.
constexpr int RANS_RANK_BYTES = 512;
// The kernel for narrow alphabets takes another table where all eight chunks of a warp allow it: an entry of two words for 32 slots,
// the symbol that covers the first of them and the one that covers the last, so one read instead of two that wait for one another.
// Exponent planes have their rare symbols at the ends of the slots, a few slots each, so the first 64 and the last 16 slots have an
// entry each; elsewhere two symbols to 32 slots are all there are (normal, Laplace and Student-t weights, one sigma or one per row: every
// chunk of some hundred; a plane half of zeros has more and keeps the rank table).  The number of a slot's entry is
// max(min(slot, 62 + slot / 32), slot - 1906).  1136 bytes per chunk, 19 blocks per SM.
constexpr uint32_t RANS_PAIR_LOW = 64, RANS_PAIR_HIGH = 16, RANS_PAIR_COARSE = RANS_PAIR_LOW - RANS_PAIR_LOW / 32;
constexpr uint32_t RANS_PAIR_TOP = 2048 - RANS_PAIR_HIGH - (RANS_PAIR_COARSE + 64);  // slot minus entry, last slots
constexpr uint32_t RANS_PAIR_ENTRIES = 2048 - RANS_PAIR_TOP;
constexpr uint32_t RANS_PAIR_SMEM = RANS_WARP_CHUNKS * RANS_PAIR_ENTRIES * 8;
__host__ __device__ inline uint32_t rans_l_entries(uint32_t max_sym) { return (max_sym + 3 + 3) & ~3u; }
__host__ __device__ inline uint32_t rans_smem_bytes(uint32_t l_entries, bool per_lane = false) {
    const uint32_t rank = RANS_WARP_CHUNKS * RANS_RANK_BYTES + (per_lane ? 128 * l_entries : RANS_WARP_CHUNKS * 4 * l_entries);
    return (per_lane && rank < RANS_PAIR_SMEM ? RANS_PAIR_SMEM : rank) + RING_SMEM;
}

// Four kernels have a table entry per slot.  Launches of up to 592 chunks, one to a block: entries of four words, and the chunk's streams in shared
// memory beside them where they fit, else through the rings.  Above that four chunks to a block, a word to an entry.  us of one chunk of 32 Ki
// symbols / 64 Ki in a call of its own, bf16: a word to an entry 479 / 762, four words 460 / 725, streams in shared memory 412 / 630 (73 cycles per
// symbol; the way from state to state alone is 47).  Tried: both byte counts from the table and one move chosen by them 415 / 652.
// Chunks of few symbols, one to a block, take a word to an entry too: the larger table, with a division for each slot, takes longer to build than
// so few gain.  Word / four words and streams, us, 100 chunks: 512 symbols of 32 values 34.0 / 34.4, 800 34.8 / 37.5, 1200 42.3 / 42.4, 2000 46.4 /
// 46.6; bf16 512 40.7 / 44.4, 1200 46.4 / 54.3, 2000 58.5 / 57.2, 3000 68.9 / 66.5.
constexpr uint32_t RANS_FEW = 1500;
// Chunks of a launch up to which the kernel with a table entry per slot is the faster one: what the GPU holds of it at once (six
// blocks of four chunks per SM).  Chunks of 32 Ki symbols, us of a bf16 tensor, table per slot against tables of pairs: 1 to 592 chunks
// 420 / 681, 2368 518 / 709, 3552 619 / 694, and beyond that a second wave (start of it, 4144: 832 / 694).  fp32: 445 / 739, 592 chunks 547 / 752,
// 2368 667 / 758, 3552 855 / 780; fp16 (rank tables) 483 / 876, 3552 645 / 928.
constexpr uint32_t RANS_DIRECT_CHUNKS = 6 * 4 * 148;
constexpr uint32_t RANS_DIRECT_BYTES = 2048 * 4;  // per chunk
constexpr uint32_t RANS_WIDE_BYTES = 2048 * 16;   // with four words to an entry
__host__ __device__ inline uint32_t rans_direct_smem(bool wide, uint32_t warp_chunks) { return (wide ? RANS_WIDE_BYTES : warp_chunks * RANS_DIRECT_BYTES) + RING_SMEM; }
// The same with a chunk's streams beside the table: up to fifteen bytes on either side of them, and 64 that a group may read too far.
constexpr uint32_t RANS_STREAM_PAD = 64;
__host__ __device__ inline uint32_t rans_resident_smem(uint32_t src_len) { return RANS_WIDE_BYTES + RING_SMEM + ((src_len + 32 + 15) & ~15u) + RANS_STREAM_PAD; }
constexpr uint32_t RANS_RESIDENT_MOST = 220 * 1024;  // of a block; the blocks of an SM have 227 KiB, one of which each takes beside its own

// Ring addressing: byte q of a lane's ring lives in word (q >> 2) & 15 of the
// [word][lane] array, `rw` points at the lane's column.
__device__ __forceinline__ uint32_t ring_byte(const uint32_t* rw, uint32_t q) {
    return reinterpret_cast<const uint8_t*>(rw)[((q & 60u) << 5) | (q & 3u)];
}
// The eight ring bytes from q on, big-endian: byte q is the top byte of `wh`.
__device__ __forceinline__ void ring_window_be(const uint32_t* rw, uint32_t q, uint32_t& wh, uint32_t& wl) {
    const uint8_t* rb = reinterpret_cast<const uint8_t*>(rw);
    const uint32_t t = q << 5;  // word k of the ring sits at byte (k & 15) * 128 of the lane's column
    uint32_t w0 = *reinterpret_cast<const uint32_t*>(rb + (t & 0x780u));
    uint32_t w1 = *reinterpret_cast<const uint32_t*>(rb + ((t + 0x80u) & 0x780u));
    uint32_t w2 = *reinterpret_cast<const uint32_t*>(rb + ((t + 0x100u) & 0x780u));
    uint32_t sel = 0x0123u + 0x1111u * (q & 3u);
    wh = __byte_perm(w0, w1, sel);
    wl = __byte_perm(w1, w2, sel);
}
// One symbol (decompress.rs:118-139): slot -> number of the covering symbol ->
// (symbol | freq << 8 | start << 20), state update.  `e` is returned whole; its
// low byte is the symbol.  LS = distance in words between list entries.
template <int LS>
__device__ __forceinline__ uint32_t rans_lookup(const uint32_t* tab, const uint32_t* lst, uint32_t& x) {
    uint32_t idx = x & 2047u;
    uint32_t w = tab[idx >> 4];
    uint32_t k = (w >> 16) + __popc(w << ((~idx & 15u) | 16u));  // boundaries at or below the slot: the count above the bitmap, the bitmap's bits up to the slot
    uint32_t e = lst[k * LS];
    x = ((e >> 8) & 0xFFFu) * (x >> 11) + (idx - (e >> 20));
    return e;
}
// Up to eight symbols, renormalising a byte at a time straight from the ring.
template <int LS>
__device__ __forceinline__ void rans_short_group(const uint32_t* tab, const uint32_t* lst, const uint32_t* rw, uint32_t& x, uint32_t& rq, uint32_t g,
                                                 uint32_t& s_lo, uint32_t& s_hi) {
    s_lo = 0; s_hi = 0;
    for (uint32_t j = 0; j < g; ++j) {
        uint32_t sym = rans_lookup<LS>(tab, lst, x) & 0xFFu;
        if (j < 4) s_lo |= sym << (8 * j); else s_hi |= sym << (8 * (j - 4));
        for (int k = 0; k < 3 && x < RANS_L; ++k) { x = (x << 8) | ring_byte(rw, rq); ++rq; }
    }
}
// The same for the group decoder's second try, out of line and by value (state, read position, symbols 0-3, symbols 4-7 come
// back in registers): one copy of the loop instead of one in every instance of the group decoder, which the instruction
// cache repays (14.28 -> 14.20 ms per pass of the benchmark container).
template <int LS>
__device__ __noinline__ uint4 rans_short_group8(const uint32_t* tab, const uint32_t* lst, const uint32_t* rw, uint32_t x, uint32_t rq) {
    uint32_t s_lo, s_hi;
    rans_short_group<LS>(tab, lst, rw, x, rq, 8, s_lo, s_hi);
    return make_uint4(x, rq, s_lo, s_hi);
}
// Exactly eight symbols, without a branch per symbol.  The next eight stream
// bytes sit big-endian in two registers behind the state; renormalising by
// 0..3 bytes (the count follows from the leading zeros of the state) is a
// funnel shift of state and window.  Eight bytes cover a group unless its
// symbols average more than one byte each; the total is checked once per group
// and a group that needed more is decoded again byte-wise.  On a plane of
// nearly incompressible bytes (many symbols, close to a byte each) that would
// happen in every other group, so a lane whose chunk has many distinct symbols
// (`dense`, only where DENSE_OK) reloads the window after four symbols.
// The byte count is ((leading zeros - 1) & 24) / 8, which holds for every state
// below 2^31.  An update never takes a state from below 2^31 to above it
// (freq <= 2^11, x >> 11 < 2^20), so only a stream whose stored initial state
// has the top bit set can get there: such a lane passes `slow` and takes the
// byte-wise path for every group.
template <int LS, bool DENSE_OK>
__device__ __forceinline__ void rans_group8(const uint32_t* tab, const uint32_t* lst, const uint32_t* rw, uint32_t& x, uint32_t& rq, uint32_t& s_lo,
                                            uint32_t& s_hi, bool dense, bool slow) {
    uint32_t wh, wl, used = 0, over = 0;
    const uint32_t x0 = x, rq0 = rq;
    ring_window_be(rw, rq, wh, wl);
    s_lo = 0; s_hi = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (DENSE_OK && j == 4 && dense) {
            over = used;  // the first half must have fit its window too
            rq += used >> 3; used = 0;
            ring_window_be(rw, rq, wh, wl);
        }
        uint32_t e = rans_lookup<LS>(tab, lst, x);
        const uint32_t ins = (0x3210u & ~(0xFu << (4 * (j & 3)))) | (4u << (4 * (j & 3)));  // low byte of e into byte j & 3
        if (j < 4) s_lo = __byte_perm(s_lo, e, ins); else s_hi = __byte_perm(s_hi, e, ins);
        // bytes until x >= 2^23, at most three: 0 for clz <= 8, 1 for 9..16, 2 for 17..24, 3 above
        uint32_t sh = (uint32_t(__clz(x)) - 1u) & 0x18u;
        x = __funnelshift_l(wh, x, sh);
        wh = __funnelshift_l(wl, wh, sh);
        wl <<= sh;
        used += sh;
    }
    if (used > 64 || over > 64 || slow) {
        const uint4 again = rans_short_group8<LS>(tab, lst, rw, x0, rq0);
        x = again.x; rq = again.y; s_lo = again.z; s_hi = again.w;
    } else {
        rq += used >> 3;
    }
}

// The same on the table of pairs.  The state is kept doubled with the next bit of the stream below it, so that the bits it wants are
// its leading zeros without their low three bits, and a slot is twelve bits: twice its number and that bit.  A word of an entry added to the
// slot (on top, ones below) is the slot's distance from the symbol's first, doubled, << 20 | symbol << 12 | frequency * 2: all that
// the update takes.  A symbol that starts behind the slot gives a distance that wraps, so the right one of two is the smaller sum.
// The integer pipe (half an instruction per cycle and scheduler) is as busy as anything here, so what can be is a multiply-add with a
// power of two that the compiler does not know, or a float multiply-add with truncation (2^23 + 2 * slot, divided by 64).
// 8192 symbols of a stream: 830 -> 695 us up to four blocks per SM; the six-layer bf16 model, 3.2 rounds of 19 blocks, 4103 -> 3670 us:
// POPC and a read less in the chain, 10.8 -> 9.0 passes of the load/store pipe per warp and symbol, 23 -> 20 integer instructions.
// Tried: entries laid out so that the chunks of a read have banks of their own (6.3 -> 5.3 passes) 3822; byte count by comparisons 3982; the
// window's second word left alone for four symbols 3668; sixteen symbols to a look at the ring 3913; streams in 32-byte blocks 3977.
constexpr uint32_t RANS_PAIR_ONE = 0x4B000000u;   // 2^23
struct RansPair { uint32_t base, two20, one, four, eight; };  // shared address of the chunk's first entry, for the float's bits; powers of two
// `one` is 1 and not a constant.  Called when the table is complete and changes no more: the reads name neither memory nor each other, so that the
// compiler may order them as it likes, but none of them can come before the address, which is not known before all stores have been made.
__device__ __forceinline__ RansPair rans_pair_at(const void* table, uint32_t one) {
    uint32_t at = uint32_t(__cvta_generic_to_shared(table)) - 4 * RANS_PAIR_ONE;
    asm volatile("" : "+r"(at) : : "memory");
    return {at, one << 20, one, one * 4, one * 8};
}
__device__ __forceinline__ uint32_t mad_u32(uint32_t a, uint32_t b, uint32_t c) { uint32_t d; asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d; }
// One symbol of a state `xx` (doubled, see above): the sum; the symbol is in bits 12 to 19.
__device__ __forceinline__ uint32_t rans_pair_lookup(const RansPair& p, uint32_t& xx) {
    uint32_t m, q, first, second;
    asm("lop3.b32 %0, %1, 0xFFE, 0x4B000000, 0xEA;" : "=r"(m) : "r"(xx));  // (xx & 0xFFE) | 2^23
    const uint32_t c = __float_as_uint(__fmaf_rz(__uint_as_float(m), 0x1p-6f, 8388608.0f - 131072.0f));
    const int low = int(mad_u32(m, p.four, p.base)), coarse = int(mad_u32(c, p.eight, p.base + 8 * RANS_PAIR_COARSE - 4 * RANS_PAIR_ONE));
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(first), "=r"(second) : "r"(max(min(low, coarse), low - int(8 * RANS_PAIR_TOP))));
    const uint32_t slot = mad_u32(xx, p.two20, 0xFFFFFu);
    asm("mul.hi.u32 %0, %1, %2;" : "=r"(q) : "r"(xx), "r"(p.two20));
    const uint32_t d = min(mad_u32(first, p.one, slot), slot + second);
    xx = (d & 0xFFFu) * q + (d >> 20);
    return d;
}
// Up to eight symbols, byte by byte: `x` as in rans_short_group.
__device__ __forceinline__ void rans_pair_short(const RansPair& p, const uint32_t* rw, uint32_t& x, uint32_t& rq, uint32_t g, uint32_t& s_lo, uint32_t& s_hi) {
    s_lo = 0; s_hi = 0;
    for (uint32_t j = 0; j < g; ++j) {
        uint32_t xx = x << 1;
        const uint32_t sym = (rans_pair_lookup(p, xx) >> 12) & 0xFFu;
        x = xx >> 1;
        if (j < 4) s_lo |= sym << (8 * j); else s_hi |= sym << (8 * (j - 4));
        for (int k = 0; k < 3 && x < RANS_L; ++k) { x = (x << 8) | ring_byte(rw, rq); ++rq; }
    }
}
__device__ __noinline__ uint4 rans_pair_short8(uint32_t base, const uint32_t* rw, uint32_t x, uint32_t rq) {
    uint32_t s_lo, s_hi;
    rans_pair_short(RansPair{base, 1u << 20, 1, 4, 8}, rw, x, rq, 8, s_lo, s_hi);
    return make_uint4(x, rq, s_lo, s_hi);
}
__device__ __forceinline__ void rans_pair_group8(const RansPair& p, const uint32_t* rw, uint32_t& x, uint32_t& rq, uint32_t& s_lo, uint32_t& s_hi) {
    uint32_t wh, wl, used = 0;
    ring_window_be(rw, rq, wh, wl);
    uint32_t xx = __funnelshift_l(wh, x, 1);
    wh = __funnelshift_l(wl, wh, 1);
    wl <<= 1;
    s_lo = 0; s_hi = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t e = rans_pair_lookup(p, xx) * 16;  // the symbol in the third byte
        const uint32_t ins = (0x3210u & ~(0xFu << (4 * (j & 3)))) | (6u << (4 * (j & 3)));
        if (j < 4) s_lo = __byte_perm(s_lo, e, ins); else s_hi = __byte_perm(s_hi, e, ins);
        uint32_t zeros;
        asm("bfind.shiftamt.u32 %0, %1;" : "=r"(zeros) : "r"(xx));
        const uint32_t sh = zeros & 0x18u;
        xx = __funnelshift_l(wh, xx, sh);
        wh = __funnelshift_l(wl, wh, sh);
        wl <<= sh;
        used += sh;
    }
    if (used > 64) {
        const uint4 again = rans_pair_short8(p.base, rw, x, rq);
        x = again.x; rq = again.y; s_lo = again.z; s_hi = again.w;
    } else {
        x = xx >> 1;
        rq += used >> 3;
    }
}

// The same on a table with an entry per slot: slot's distance from the symbol's first << 20 | symbol << 12 | frequency, so that
// both factors of the update are one step away.  From one state to the next it is a mask, one shared-memory read, a shift and a
// multiply-add; renormalising moves the state shifted by one or two bytes over the state, two moves that hang on the comparisons
// alone.  A state that has been normalised once
// never needs more than two bytes (an update leaves at least 2^12), so eight bytes of stream last for four symbols and nothing
// is decoded twice.  A stream whose stored initial state is not normalised goes byte by byte.
__device__ __forceinline__ uint32_t rans_direct_lookup(const uint32_t* tab, uint32_t& x) {
    const uint32_t e = tab[x & 2047u];
    x = (e & 0xFFFu) * (x >> 11) + (e >> 20);
    return e >> 12;
}
// The ring's words are kept with their first byte on top here.
template <bool WIDE>
__device__ __forceinline__ void rans_direct_short(const uint32_t* tab, const uint32_t* rw, uint32_t& x, uint32_t& rq, uint32_t g, uint32_t& s_lo, uint32_t& s_hi) {
    s_lo = 0; s_hi = 0;
    for (uint32_t j = 0; j < g; ++j) {
        uint32_t sym;
        if (WIDE) {
            const uint4 e = reinterpret_cast<const uint4*>(tab)[x & 2047u];
            x = e.x * (x >> 11) + e.y; sym = e.w;
        } else sym = rans_direct_lookup(tab, x) & 0xFFu;
        if (j < 4) s_lo |= sym << (8 * j); else s_hi |= sym << (8 * (j - 4));
        for (int k = 0; k < 3 && x < RANS_L; ++k) { x = (x << 8) | ring_byte(rw, rq ^ 3u); ++rq; }
    }
}
__device__ __forceinline__ void rans_direct_words(const uint32_t* rw, uint32_t rq, uint32_t v[5]) {  // five ring words from the one that holds byte rq on
#pragma unroll
    for (uint32_t k = 0; k < 5; ++k) v[k] = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(rw) + (((rq << 5) + 0x80u * k) & 0x780u));
}
// One symbol with an entry of four words: frequency, slot's distance from the symbol's first, from which value of x >> 11 on the next state is
// normalised, symbol.  The third is there so that the first byte need not wait for the state.
__device__ __forceinline__ void rans_direct_step(const uint4& e, uint32_t wh, uint32_t& x, uint32_t& bits) {
    asm("{\n\t.reg .pred some, more;\n\t.reg .u32 q, y;\n\t"
        "shr.u32 q, %0, 11;\n\tsetp.lt.u32 some, q, %5;\n\t"
        "mad.lo.u32 y, %3, q, %4;\n\tsetp.lt.u32 more, y, 0x8000;\n\t"
        "mov.u32 %0, y;\n\tmov.u32 %1, 0;\n\t"
        "@some prmt.b32 %0, y, %2, 0x2107;\n\t@some mov.u32 %1, 8;\n\t"
        "@more prmt.b32 %0, y, %2, 0x1076;\n\t@more mov.u32 %1, 16;\n\t}"
        : "+r"(x), "=&r"(bits) : "r"(wh), "r"(e.x), "r"(e.y), "r"(e.z));
}
// Four symbols.  `v` are five ring words read before the last four symbols were decoded, `skip` the bits of them that are used
// up by now (88 at most).  The five words for the next four are requested here.  WIDE: an entry of four words.
template <bool WIDE>
__device__ __forceinline__ uint32_t rans_direct_four(const uint32_t* tab, const uint32_t* rw, uint32_t& x, uint32_t& rq, uint32_t v[5], uint32_t& skip) {
    const bool one_off = skip >= 32, two_off = skip >= 64;
    const uint32_t a = two_off ? v[2] : one_off ? v[1] : v[0], b = two_off ? v[3] : one_off ? v[2] : v[1], c = two_off ? v[4] : one_off ? v[3] : v[2];
    uint32_t wh = __funnelshift_l(b, a, skip), wl = __funnelshift_l(c, b, skip), used = 0, sy = 0;  // a funnel shift takes the amount mod 32
    rans_direct_words(rw, rq, v);
    skip = (rq & 3u) * 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t ins = (0x3210u & ~(0xFu << (4 * j))) | (4u << (4 * j));
        uint32_t bits;
        if (WIDE) {
            const uint4 e = reinterpret_cast<const uint4*>(tab)[x & 2047u];
            rans_direct_step(e, wh, x, bits);
            sy = __byte_perm(sy, e.w, ins);
        } else {
            const uint32_t e = rans_direct_lookup(tab, x);
            sy = __byte_perm(sy, e, ins);
            asm("{\n\t.reg .pred some, more;\n\t.reg .u32 y;\n\t"
                "setp.lt.u32 some, %0, 0x800000;\n\tsetp.lt.u32 more, %0, 0x8000;\n\t"
                "mov.u32 y, %0;\n\tmov.u32 %1, 0;\n\t"
                "@some prmt.b32 y, %0, %2, 0x2107;\n\t@some mov.u32 %1, 8;\n\t"
                "@more prmt.b32 y, %0, %2, 0x1076;\n\t@more mov.u32 %1, 16;\n\t"
                "mov.u32 %0, y;\n\t}"
                : "+r"(x), "=&r"(bits) : "r"(wh));
        }
        wh = __funnelshift_l(wl, wh, bits);
        wl <<= bits;
        used += bits;
    }
    skip += used;
    rq += used >> 3;
    return sy;
}

// The same on streams that lie in shared memory whole, words with their first byte on top: nothing to fill up and no ring to go round, so the
// next words are four reads from one address.  `at` is a position in bits from `words` on, `last` the last word whose three successors
// may be read (a damaged stream can lead anywhere).
__device__ __forceinline__ void rans_resident_words(const uint32_t* words, uint32_t at, uint32_t last, uint32_t v[4]) {
    const uint32_t k = min(at >> 5, last);
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) v[j] = words[k + j];
}
__device__ __forceinline__ void rans_resident_short(const uint4* tab, const uint32_t* words, uint32_t last, uint32_t& x, uint32_t& at, uint32_t g, uint32_t& s_lo, uint32_t& s_hi) {
    s_lo = 0; s_hi = 0;
    for (uint32_t j = 0; j < g; ++j) {
        const uint4 e = tab[x & 2047u];
        x = e.x * (x >> 11) + e.y;
        if (j < 4) s_lo |= e.w << (8 * j); else s_hi |= e.w << (8 * (j - 4));
        for (int k = 0; k < 3 && x < RANS_L; ++k) { x = (x << 8) | ((words[min(at >> 5, last)] >> (24 - (at & 24u))) & 0xFFu); at += 8; }
    }
}
// Four symbols.  `v` are words read when the last four were half done, `skip` the bits of them that are used up by now (below 64).
__device__ __forceinline__ uint32_t rans_resident_four(const uint4* tab, const uint32_t* words, uint32_t last, uint32_t& x, uint32_t& at, uint32_t v[4], uint32_t& skip) {
    const bool one_off = skip >= 32;
    const uint32_t a = one_off ? v[1] : v[0], b = one_off ? v[2] : v[1], c = one_off ? v[3] : v[2];
    uint32_t wh = __funnelshift_l(b, a, skip), wl = __funnelshift_l(c, b, skip), used = 0, sy = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j == 2) {
            at += used;
            rans_resident_words(words, at, last, v);
            skip = at & 31u;
            used = 0;
        }
        const uint4 e = tab[x & 2047u];
        uint32_t bits;
        rans_direct_step(e, wh, x, bits);
        sy = __byte_perm(sy, e.w, (0x3210u & ~(0xFu << (4 * j))) | (4u << (4 * j)));
        wh = __funnelshift_l(wl, wh, bits);
        wl <<= bits;
        used += bits;
    }
    at += used;
    skip += used;
    return sy;
}

// The bound of 20 blocks per SM lets the compiler use 96 registers, which the 32-bit rounds need to stay out of local memory; shared memory allows 19,
// also where a warp that could not have tables of pairs takes rank tables after all.  Those had 22 before there were tables of pairs, and no less time
// for it: 32 Ki, half of the weights zero, 3600 chunks 1543 us then and now, 7104: 1654 / 1641, 20,000: 3007 / 2894.
//
// DIRECT: 0 the tables above; otherwise a table entry per slot, for launches that do not fill the GPU, where the time from one symbol to the
// next is all that counts: 4 chunks per warp with a word to an entry (rans_direct_four), 3 one chunk, 1 one chunk with four words to an entry, 2 the
// same with the chunk's streams in shared memory (rans_resident_four).
template <bool PER_LANE, int DIRECT = 0>
__global__ void __launch_bounds__(32, DIRECT ? 1 : 20) rans_decode_kernel_t(const DecodeItem* __restrict__ items, uint32_t n_items, Bases bases, uint32_t* __restrict__ status,
                                                           uint32_t l_entries) {
    constexpr int LS = PER_LANE ? 32 : 1;
    constexpr bool RESIDENT = DIRECT == 2, WIDE = DIRECT == 1 || RESIDENT;
    constexpr uint32_t CHUNKS = DIRECT == 0 ? RANS_WARP_CHUNKS : DIRECT == 4 ? 4 : 1;
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = threadIdx.x, c = lane >> 2, s = lane & 3;
    // DIRECT: the rings come first, and in their place, while the tables are built, one chunk's rank table and symbol list
    uint32_t* slots = reinterpret_cast<uint32_t*>(smem + RING_SMEM);                                  // DIRECT: [chunk][2048]
    uint32_t* ranktab = reinterpret_cast<uint32_t*>(smem);                                            // [8][128]
    uint32_t* symlist = reinterpret_cast<uint32_t*>(smem + (DIRECT ? 1 : CHUNKS) * RANS_RANK_BYTES);  // entry 0 of every list is a pad
    Ring ring{reinterpret_cast<uint32_t*>(DIRECT ? smem : smem + rans_smem_bytes(l_entries, PER_LANE) - RING_SMEM) + lane};

    const uint32_t item_idx = blockIdx.x * CHUNKS + c;
    const bool valid = c < CHUNKS && item_idx < n_items;
    DecodeItem it;
    if (valid) it = items[item_idx];
    const uint8_t* src = valid ? rd(bases, it.src) : nullptr;
    uint32_t err = ST_OK;

    // header: [max_sym][freq u16 x (max_sym+1)][4 x u32 stream lengths]
    uint32_t max_sym = 0, hdr = 0, my_off = 0, my_len = 0;
    if (valid) {
        if (it.src_len < 1) err = ST_BAD_HEADER;
        else {
            max_sym = src[0];
            hdr = 1 + 2 * (max_sym + 1);
            if (it.src_len < hdr + 16) err = ST_BAD_HEADER;
            else {
                uint64_t total = 0;
                uint32_t off = hdr + 16;
                for (uint32_t k = 0; k < 4; ++k) {
                    uint32_t l = ld_u32_unaligned(src + hdr + 4 * k);
                    if (k == s) { my_off = off + uint32_t(total); my_len = l; }
                    total += l;
                }
                if (total != uint64_t(it.src_len - hdr - 16)) err = ST_BAD_HEADER;
            }
        }
    }

    // tables: the whole warp builds one chunk's tables at a time
    bool dense = false;  // this lane's chunk is close to incompressible (see rans_group8)
    // The narrow kernel tries the tables of pairs first, with a chunk's rank table and symbol list in the place of the rings meanwhile.
    bool pairs = PER_LANE;
    if (PER_LANE) {  // states that rans_pair_group8 cannot take: see rans_group8, rans_direct_four
        const uint32_t x = valid && !err && my_len >= 4 ? ld_u32_unaligned(src + my_off) : RANS_L;
        pairs = !__any_sync(0xFFFFFFFFu, x >> 31 || x < RANS_L);
    }
    for (uint32_t pass = 0; pass < (PER_LANE ? 2u : 1u); ++pass) {  // 0: tables of pairs; 1: the others, also when a chunk does not fit the former
        if (PER_LANE && (pass == 0) != pairs) continue;
        for (uint32_t c2 = 0; c2 < CHUNKS; ++c2) {
            const uint32_t leader = c2 * 4;
            uintptr_t psrc = __shfl_sync(0xFFFFFFFFu, reinterpret_cast<uintptr_t>(src), leader);
            uint32_t pms = __shfl_sync(0xFFFFFFFFu, max_sym, leader);
            uint32_t perr = __shfl_sync(0xFFFFFFFFu, err, leader);
            uint32_t pvalid = __shfl_sync(0xFFFFFFFFu, uint32_t(valid), leader);
            if (!pvalid || perr) continue;
            const uint8_t* ps = reinterpret_cast<const uint8_t*>(psrc);
            uint32_t f[8], sum = 0, present = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                uint32_t sym = lane * 8 + k;
                f[k] = sym <= pms ? uint32_t(ps[1 + 2 * sym]) | uint32_t(ps[2 + 2 * sym]) << 8 : 0u;
                sum += f[k];
                present += f[k] != 0;
            }
            uint32_t incl = sum, rincl = present;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d), r = __shfl_up_sync(0xFFFFFFFFu, rincl, d);
                if (lane >= d) { incl += t; rincl += r; }
            }
            uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31), distinct = __shfl_sync(0xFFFFFFFFu, rincl, 31);
            bool bad = total != 2048;  // decompress.rs:49-55
            if (!PER_LANE && c == c2) dense = distinct >= RANS_DENSE_SYMBOLS;
            if (distinct + 2 > l_entries) bad = true;  // the host sizes the list from the planned bytes; a blob that differs from them may not fit
            if (bad) { if (c == c2) err = ST_BAD_HEADER; continue; }
            uint32_t start = incl - sum, rank = rincl - present;
            uint32_t* tab = pairs ? ring.base - lane : DIRECT ? ranktab : ranktab + c2 * 128;
            uint32_t* lst = pairs ? tab + 128 : DIRECT ? symlist : PER_LANE ? symlist + c2 * 4 : symlist + c2 * l_entries;
            if (lane == 0) {
                if (PER_LANE && !pairs) *reinterpret_cast<uint4*>(lst) = make_uint4(0, 0, 0, 0); else lst[0] = 0;
            }
            *reinterpret_cast<uint4*>(tab + 4 * lane) = make_uint4(0, 0, 0, 0);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                uint32_t sym = lane * 8 + k, fr = f[k];
                if (!fr) continue;
                uint32_t entry = sym | (fr << 8) | (start << 20);
                if (PER_LANE && !pairs) *reinterpret_cast<uint4*>(lst + (rank + 1) * 32) = make_uint4(entry, entry, entry, entry);  // the four lanes of the chunk
                else lst[rank + 1] = entry;
                atomicOr(&tab[start >> 4], 1u << (start & 15));
                start += fr; ++rank;
            }
            __syncwarp();
            // boundaries before each word: lane l owns words 4l .. 4l+3
            uint4 bm = *reinterpret_cast<uint4*>(tab + 4 * lane);
            uint32_t p0 = __popc(bm.x), p1 = __popc(bm.y), p2 = __popc(bm.z), p3 = __popc(bm.w), scan = p0 + p1 + p2 + p3;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                uint32_t t = __shfl_up_sync(0xFFFFFFFFu, scan, d);
                if (lane >= d) scan += t;
            }
            uint32_t before = scan - (p0 + p1 + p2 + p3);
            bm.x |= before << 16; before += p0;
            bm.y |= before << 16; before += p1;
            bm.z |= before << 16; before += p2;
            bm.w |= before << 16;
            *reinterpret_cast<uint4*>(tab + 4 * lane) = bm;
            if (pairs) {
                __syncwarp();
                auto number = [&](uint32_t u) { const uint32_t w = tab[u >> 4]; return (w >> 16) + __popc(w << ((~u & 15u) | 16u)); };
                auto entry = [&](uint32_t k) { const uint32_t e = lst[k]; return ((e & 0xFFu) << 12 | ((e >> 8) & 0xFFFu) * 2) - 0xFFFFFu - ((e >> 20) << 21); };
                bool fits = distinct > 1;  // (a frequency of 2048 is one bit too long)
                for (uint32_t k = lane; k < RANS_PAIR_ENTRIES; k += 32) {
                    const bool coarse = k >= RANS_PAIR_LOW && k < RANS_PAIR_COARSE + 64;
                    const uint32_t u = k < RANS_PAIR_LOW ? k : coarse ? (k - RANS_PAIR_COARSE) * 32 : k + RANS_PAIR_TOP;
                    const uint32_t last = coarse ? (u + 31 < 2047 - RANS_PAIR_HIGH ? u + 31 : 2047 - RANS_PAIR_HIGH) : u;
                    const uint32_t a = number(u), b = number(last);
                    fits = fits && b - a <= 1;
                    reinterpret_cast<uint2*>(smem)[c2 * RANS_PAIR_ENTRIES + k] = make_uint2(entry(a), entry(b));
                }
                pairs = __all_sync(0xFFFFFFFFu, fits);
                __syncwarp();
                if (!pairs) break;
            }
            if (DIRECT) {
                __syncwarp();
#pragma unroll 8
                for (uint32_t u = lane; u < 2048; u += 32) {
                    const uint32_t w = tab[u >> 4], e = lst[(w >> 16) + __popc(w << ((~u & 15u) | 16u))];
                    const uint32_t f = (e >> 8) & 0xFFFu, d = u - (e >> 20);
                    if (WIDE) reinterpret_cast<uint4*>(slots)[u] = make_uint4(f, d, (RANS_L - 1 - d) / f + 1, e & 0xFFu);
                    else slots[c2 * 2048 + u] = d << 20 | (e & 0xFFu) << 12 | f;
                }
                __syncwarp();
            }
        }
    }
    uint32_t* const words = slots + RANS_WIDE_BYTES / 4;  // RESIDENT: the chunk's streams, from the aligned 16 bytes on that hold their first one
    uintptr_t words_from = 0;
    uint32_t last_word = 0;
    if (RESIDENT) {
        const uintptr_t first = reinterpret_cast<uintptr_t>(rd(bases, items[blockIdx.x].src)) + __shfl_sync(0xFFFFFFFFu, hdr, 0) + 16;
        const uintptr_t end = reinterpret_cast<uintptr_t>(rd(bases, items[blockIdx.x].src)) + items[blockIdx.x].src_len;
        words_from = first & ~uintptr_t(15);
        if (__shfl_sync(0xFFFFFFFFu, err, 0) == ST_OK) {  // the header fits, so first <= end
            const uintptr_t lo16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_first) & ~uintptr_t(15);
            const uintptr_t hi16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_end + 15) & ~uintptr_t(15);
            const uint32_t blocks = uint32_t((end - words_from + 15) >> 4);
            last_word = 4 * blocks + RANS_STREAM_PAD / 4 - 4;
            uint4* out = reinterpret_cast<uint4*>(words);
            for (uint32_t b0 = 0; b0 < blocks; b0 += 8 * 32) {
                uint4 v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = fetch16(words_from + 16 * uintptr_t(b0 + 32 * k + lane), lo16, hi16);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t b = b0 + 32 * k + lane;
                    if (b < blocks) out[b] = make_uint4(__byte_perm(v[k].x, 0, 0x0123), __byte_perm(v[k].y, 0, 0x0123), __byte_perm(v[k].z, 0, 0x0123), __byte_perm(v[k].w, 0, 0x0123));
                }
            }
            if (lane < RANS_STREAM_PAD / 16) out[blocks + lane] = make_uint4(0, 0, 0, 0);
        }
    }
    __syncwarp();

    uint32_t seg_start = 0, seg_len = 0;
    if (valid) split_four_dev(it.n, s, seg_start, seg_len);
    if (valid && !err && seg_len > 0) {
        if (my_len < 4) err = ST_STREAM_UNDERRUN;  // decompress.rs:82-86
        else {
            const uint32_t* tab = DIRECT && CHUNKS == 1 ? slots : DIRECT ? slots + c * 2048 : ranktab + c * 128;
            const uint32_t* lst = PER_LANE ? symlist + lane : symlist + c * l_entries;
            const RansPair pair = PER_LANE ? rans_pair_at(smem + c * RANS_PAIR_ENTRIES * 8, n_items ? 1u : 0u) : RansPair{};
            const uint32_t* rw = ring.base;
            Epilogue ep = make_epilogue(bases, it);
            const uint8_t* st = src + my_off;
            uint32_t x = ld_u32_unaligned(st);
            const bool slow = x >> 31 || (DIRECT && x < RANS_L);  // see rans_group8, rans_direct_four
            if (RESIDENT) {
                const uint4* wide = reinterpret_cast<const uint4*>(slots);
                uint32_t at = 8 * uint32_t(reinterpret_cast<uintptr_t>(st) + 4 - words_from), pos = seg_start, remaining = seg_len, s_lo, s_hi;
                const uint32_t end_at = 8 * uint32_t(reinterpret_cast<uintptr_t>(st) + my_len - words_from);
                const uint32_t g = first_group(ep, pos, remaining);
                if (g < 8 || remaining < 16) {
                    rans_resident_short(wide, words, last_word, x, at, g, s_lo, s_hi);
                    emit(ep, pos, g, uint64_t(s_lo) | uint64_t(s_hi) << 32);
                    pos += g; remaining -= g;
                }
                if (!slow) {
                    uint32_t v[4], skip = at & 31u;
                    rans_resident_words(words, at, last_word, v);
                    fast_groups(ep, it.n, pos, remaining, [&](uint32_t& lo, uint32_t& hi) {
                        lo = rans_resident_four(wide, words, last_word, x, at, v, skip);
                        hi = rans_resident_four(wide, words, last_word, x, at, v, skip);
                    });
                }
                while (remaining) {
                    const uint32_t t = remaining < 8 ? remaining : 8;
                    rans_resident_short(wide, words, last_word, x, at, t, s_lo, s_hi);
                    emit(ep, pos, t, uint64_t(s_lo) | uint64_t(s_hi) << 32);
                    pos += t; remaining -= t;
                }
                if (at > end_at) report(status, it.id, ST_STREAM_UNDERRUN);  // decompress.rs:99-104
                return;
            }
            // ring cursor as a 32-bit offset from the 16-byte aligned block that holds the first renorm byte
            const uintptr_t g0 = (reinterpret_cast<uintptr_t>(st) + 4) & ~uintptr_t(15);
            uint32_t rq = uint32_t(reinterpret_cast<uintptr_t>(st) + 4 - g0);
            const uint32_t end_q = uint32_t(reinterpret_cast<uintptr_t>(st) + my_len - g0);
            const uintptr_t lo16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_first) & ~uintptr_t(15);
            const uintptr_t hi16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_end + 15) & ~uintptr_t(15);
            uint32_t fq = 0;
            auto park = [&](uint4 v) {
                if (DIRECT) v = make_uint4(__byte_perm(v.x, 0, 0x0123), __byte_perm(v.y, 0, 0x0123), __byte_perm(v.z, 0, 0x0123), __byte_perm(v.w, 0, 0x0123));
                ring.put(fq, v);
                fq += 16;
            };
            for (int k = 0; k < 3; ++k) park(fetch16(g0 + fq, lo16, hi16));
            uint4 pending = fetch16(g0 + fq, lo16, hi16);
            // A group consumes at most 24 bytes; 32 valid bytes at its start always suffice.
            // The lanes of a warp drain their rings at similar rates: when any active lane runs low,
            // every lane with room for a block takes one, so the refill code runs once per several groups.
            auto top_up_at = [&](uint32_t q, uint32_t low) {
                if (__any_sync(__activemask(), fq - q < low)) {
                    if (fq - q <= 48) { park(pending); pending = fetch16(g0 + fq, lo16, hi16); }
                }
            };
            auto top_up = [&]() { top_up_at(rq, 32); };

            uint32_t pos = seg_start, remaining = seg_len;
            auto short_group = [&](uint32_t g, uint32_t& s_lo, uint32_t& s_hi) {
                if (DIRECT) rans_direct_short<WIDE>(tab, rw, x, rq, g, s_lo, s_hi);
                else if (PER_LANE && pairs) rans_pair_short(pair, rw, x, rq, g, s_lo, s_hi);
                else rans_short_group<LS>(tab, lst, rw, x, rq, g, s_lo, s_hi);
            };
            // head: a short group up to the next 8-element boundary of the destination
            {
                uint32_t g = first_group(ep, pos, remaining);
                if (g < 8 || remaining < 16) {
                    uint32_t s_lo, s_hi;
                    top_up();
                    short_group(g, s_lo, s_hi);
                    emit(ep, pos, g, uint64_t(s_lo) | uint64_t(s_hi) << 32);
                    pos += g; remaining -= g;
                }
            }
            if (DIRECT && !slow) {
                // A read of the ring takes as long as half a symbol, so words are read four symbols before they are used, and the
                // ring is topped up by where the group began: that position has been known for long, and no wait hangs on it.
                // Four symbols take eight bytes at most and words are read for eight: from a group's beginning on 24 bytes are
                // there, and 40 after the top-up, which is 24 behind a group's end.
                uint32_t v[5], skip = (rq & 3u) * 8;
                top_up();
                rans_direct_words(rw, rq, v);
                fast_groups(ep, it.n, pos, remaining, [&](uint32_t& s_lo, uint32_t& s_hi) {
                    const uint32_t began = rq;
                    s_lo = rans_direct_four<WIDE>(tab, rw, x, rq, v, skip);
                    top_up_at(began, 40);
                    s_hi = rans_direct_four<WIDE>(tab, rw, x, rq, v, skip);
                });
            } else if (PER_LANE && pairs) {
                fast_groups(ep, it.n, pos, remaining, [&](uint32_t& s_lo, uint32_t& s_hi) {
                    top_up();
                    rans_pair_group8(pair, rw, x, rq, s_lo, s_hi);
                });
            } else {
                fast_groups(ep, it.n, pos, remaining, [&](uint32_t& s_lo, uint32_t& s_hi) {
                    top_up();
                    if (DIRECT) rans_direct_short<WIDE>(tab, rw, x, rq, 8, s_lo, s_hi);
                    else rans_group8<LS, !PER_LANE>(tab, lst, rw, x, rq, s_lo, s_hi, dense, slow);
                });
            }
            // tail: whatever the fast loops left
            while (remaining) {
                uint32_t g = remaining < 8 ? remaining : 8, s_lo, s_hi;
                top_up();
                short_group(g, s_lo, s_hi);
                emit(ep, pos, g, uint64_t(s_lo) | uint64_t(s_hi) << 32);
                pos += g; remaining -= g;
            }
            if (rq > end_q) err = ST_STREAM_UNDERRUN;  // decompress.rs:99-104
        }
    }
    if (err) report(status, it.id, err);
}

// `direct`: the launch takes a kernel with a table entry per slot, and `size` is the largest rans_direct_size.  Else `size` is the rows of the
// symbol lists (`narrow`) or the most distinct symbols of a chunk.
inline uint32_t rans_direct_size(const DecodeItem& it) { return it.n < RANS_FEW ? 0 : it.n < 1u << 29 ? it.src_len : ~0u; }  // (positions in shared memory are 32-bit, in bits)
// What blocks of rans_launch may take of an SM's shared memory, all together.
struct RansRoom { uint32_t resident, wide; };
inline RansRoom rans_room_alone() { return {RANS_RESIDENT_MOST, RANS_RESIDENT_MOST}; }
// Beside other codecs' decoders, whose blocks on an SM have `huffman` and `tans` bytes of shared memory: blocks that find no room wait until some of
// the others have ended, and their streams are behind then.  Huffman's blocks stay for as long as their launch takes, so theirs is not to be had.
// tANS blocks come and go, but too many large blocks keep them out in turn.  us by streams in shared memory / four words / four chunks to a block, u8
// of 32 values in chunks of 64 Ki: 200 chunks beside 400 tANS chunks 671 / 764 / 819, 1776: 1082 / 1159 / 1206, 8000 Huffman chunks 1355 / 1306 / 1260;
// 300 chunks 795 / 764 / 818, 1098 / 1171 / 1194, 1361 / 1310 / 1265; 444 chunks 905 / 770 / 822, 1610 / 1293 / 1211, 1847 / 1311 / 1268; 592 chunks (no
// room for streams) - / 1009 / 826, - / 1328 / 1211, - / 1532 / 1269.  32 Ki, 300 chunks: 362 / 414 / 441, 642 / 684 / 704, 703 / 678 / 655; 370 beside 400: 450 / 416 / 441; 444: 469 / 418 /
// 445, 666 / 762 / 706, 707 / 679 / 657.  256 Ki, 592 beside 100 tANS chunks, which leave room for all: - / 2796 / 3002.  A word to an entry and a chunk to
// a block are the slower ones nearly everywhere (64 Ki, 592: 818, 1380, 1335).
inline RansRoom rans_room_beside(uint32_t chunks, uint32_t huffman, uint32_t tans) {
    auto without = [](uint32_t taken) { return taken < RANS_RESIDENT_MOST ? RANS_RESIDENT_MOST - taken : 0u; };
    const uint32_t room = without(huffman) > 80u << 10 ? without(huffman) : 80u << 10;
    return {chunks > 340 ? 0u : room, chunks <= 3 * 148 ? room : huffman ? 0u : without(tans)};
}
inline void rans_launch(const DecodeItem* items, uint32_t n, const Bases& bases, uint32_t* status, bool direct, bool narrow, uint32_t size, RansRoom room, cudaStream_t st) {
    auto blocks = [n](uint32_t per) { return (n + per - 1) / per; };
    const uint32_t per_sm = blocks(148);
    if (direct && n <= 4 * 148 && size == 0) rans_decode_kernel_t<false, 3><<<n, 32, rans_direct_smem(false, 1), st>>>(items, n, bases, status, rans_l_entries(255));
    else if (direct && n <= 4 * 148 && size < room.resident && per_sm * rans_resident_smem(size) <= room.resident)
        rans_decode_kernel_t<false, 2><<<n, 32, rans_resident_smem(size), st>>>(items, n, bases, status, rans_l_entries(255));
    else if (direct && n <= 4 * 148 && per_sm * rans_direct_smem(true, 1) <= room.wide)
        rans_decode_kernel_t<false, 1><<<n, 32, rans_direct_smem(true, 1), st>>>(items, n, bases, status, rans_l_entries(255));
    else if (direct) rans_decode_kernel_t<false, 4><<<blocks(4), 32, rans_direct_smem(false, 4), st>>>(items, n, bases, status, rans_l_entries(255));
    else if (narrow) rans_decode_kernel_t<true><<<blocks(RANS_WARP_CHUNKS), 32, rans_smem_bytes(size + 2, true), st>>>(items, n, bases, status, size + 2);
    else {
        const uint32_t le = (size + 2 + 3) & ~3u;
        rans_decode_kernel_t<false><<<blocks(RANS_WARP_CHUNKS), 32, rans_smem_bytes(le), st>>>(items, n, bases, status, le);
    }
}
inline cudaError_t rans_direct_allow_shared() {
    cudaError_t e = cudaFuncSetAttribute(rans_decode_kernel_t<false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(RANS_RESIDENT_MOST));
    for (auto k : {rans_decode_kernel_t<false, 1>, rans_decode_kernel_t<false, 2>, rans_decode_kernel_t<false, 3>, rans_decode_kernel_t<false, 4>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e;
}

// ---- canonical Huffman -----------------------------------------------------
// Shared memory per chunk:
//  * a one-symbol table over the next HUF_LUT_BITS stream bits, (length << 8) |
//    symbol, 0 when the code is longer than the window: 1 KiB instead of the
//    4 KiB of a table over all eleven bits, and shared memory per chunk is what
//    bounds the streams an SM keeps in flight;
//  * the canonical description (first code, count and list offset per length,
//    the symbols in canonical order): codes longer than the window (the rarest
//    symbols) and windows that no code covers are decoded from it.
constexpr int HUF_WARP_CHUNKS = 8;
constexpr int HUF_LUT_BITS = 9;
constexpr int HUF_LUT_BYTES = 2 << HUF_LUT_BITS;
constexpr int HUF_CANON_BYTES = 256 + 3 * 16 * 2;  // symbols in canonical order; u16 first[16], count[16], offs[16]
constexpr int HUF_SMEM = HUF_WARP_CHUNKS * (HUF_LUT_BYTES + HUF_CANON_BYTES) + RING_SMEM;

struct HuffCanon {
    const uint8_t* syms;
    const uint16_t* first;  // first[0] = max_bits
    const uint16_t* count;  // count[0] = 1 when the tables are usable
    const uint16_t* offs;
};
// One symbol from the low `max_bits` bits of `window` (stream order, first bit lowest): (length << 8) | symbol.
// A window that no code covers reads as symbol 0 of full length, like an unassigned slot of the reference's table
// (huffman/tree.rs:128-177).  Kept out of line: the decode loops meet a code longer than the table's window once in a
// few hundred symbols, and eight inlined copies of this loop per group of eight symbols, in every instance of the
// group decoder, made the kernel wait for its own instructions.  Four scalar arguments travel in registers; the
// canonical description (symbols, then first code / count / list offset per length) is addressed from its base.
__device__ __noinline__ uint32_t huff_canon_decode(const uint8_t* canon, uint32_t max_bits, uint32_t window, uint32_t shortest) {
    const uint16_t* first = reinterpret_cast<const uint16_t*>(canon + 256);
    const uint16_t* count = reinterpret_cast<const uint16_t*>(canon + 256 + 32);
    const uint16_t* offs = reinterpret_cast<const uint16_t*>(canon + 256 + 64);
    const uint32_t v = __brev(window) >> (32 - max_bits);  // code bits, first bit highest
    for (uint32_t len = shortest; len <= max_bits; ++len) {
        uint32_t d = (v >> (max_bits - len)) - first[len];
        if (d < count[len]) return (len << 8) | canon[offs[len] + d];
    }
    return max_bits << 8;
}

__global__ void __launch_bounds__(32) huffman_decode_kernel(const DecodeItem* __restrict__ items, uint32_t n_items, Bases bases, uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = threadIdx.x, c = lane >> 2, s = lane & 3;
    uint16_t* lut_all = reinterpret_cast<uint16_t*>(smem);                                  // [8][512]
    uint8_t* canon_all = smem + HUF_WARP_CHUNKS * HUF_LUT_BYTES;                            // [8][HUF_CANON_BYTES]
    Ring ring{reinterpret_cast<uint32_t*>(smem + HUF_WARP_CHUNKS * (HUF_LUT_BYTES + HUF_CANON_BYTES)) + lane};
    auto canon_of = [&](uint32_t chunk) {
        uint8_t* base = canon_all + chunk * HUF_CANON_BYTES;
        return HuffCanon{base, reinterpret_cast<uint16_t*>(base + 256), reinterpret_cast<uint16_t*>(base + 256 + 32), reinterpret_cast<uint16_t*>(base + 256 + 64)};
    };

    const uint32_t item_idx = blockIdx.x * HUF_WARP_CHUNKS + c;
    const bool valid = item_idx < n_items;
    DecodeItem it;
    if (valid) it = items[item_idx];
    const uint8_t* src = valid ? rd(bases, it.src) : nullptr;
    uint32_t err = ST_OK;
    uint32_t max_bits = 1, my_off = 0, my_len = 0;

    // weights header (weights.rs:34-85)
    uint32_t nsym = 0, hb = 0, hdr = 0;
    if (valid) {
        if (it.src_len < 1 || (src[0] & 0x80) == 0) err = ST_BAD_HEADER;
        else if (src[0] == 0x80) {
            if (it.src_len < 2) err = ST_BAD_HEADER;
            else { nsym = src[1] == 0 ? 256u : src[1]; hb = 2; if (nsym < 128) err = ST_BAD_HEADER; }
        } else { nsym = src[0] & 0x7F; hb = 1; }
        if (!err) {
            hdr = hb + (nsym + 1) / 2;
            if (it.src_len < hdr + 16) err = ST_BAD_HEADER;
        }
        if (!err) {
            uint64_t total = 0;
            uint32_t off = hdr + 16;
            for (uint32_t k = 0; k < 4; ++k) {
                uint32_t l = ld_u32_unaligned(src + hdr + 4 * k);
                if (k == s) { my_off = off + uint32_t(total); my_len = l; }
                total += l;
            }
            if (total != uint64_t(it.src_len - hdr - 16)) err = ST_BAD_HEADER;
        }
    }
    auto weight = [&](uint32_t i) -> uint32_t { uint8_t b = src[hb + (i >> 1)]; return (i & 1) ? (b >> 4) : (b & 0x0F); };

    // canonical description: lane s == 0 of each chunk (tree.rs:103-177); code assignment is sequential per length
    if (s == 0) {
        HuffCanon hc = canon_of(c);
        uint16_t* first = const_cast<uint16_t*>(hc.first);
        uint16_t* count = const_cast<uint16_t*>(hc.count);
        uint16_t* offs = const_cast<uint16_t*>(hc.offs);
        uint8_t* syms = const_cast<uint8_t*>(hc.syms);
        uint32_t next_code[12];
        if (valid && !err) {
            uint32_t counts[12];
#pragma unroll
            for (int k = 0; k < 12; ++k) counts[k] = 0;
            uint32_t mb = 0, tot = 0;
            for (uint32_t i = 0; i < nsym; ++i) {
                uint32_t w = weight(i);
                if (w > 11) { err = ST_BAD_HEADER; break; }
                if (w) {
                    tot++;
                    mb = w > mb ? w : mb;
#pragma unroll
                    for (int k = 1; k < 12; ++k) counts[k] += (w == uint32_t(k));
                }
            }
            if (tot == 0) err = ST_BAD_HEADER;
            max_bits = mb < 1 ? 1 : mb;
            uint32_t code = 0, before = 0;
#pragma unroll
            for (int bits = 1; bits < 12; ++bits) {
                next_code[bits] = 0;
                if (uint32_t(bits) <= max_bits) {
                    code = (code + counts[bits - 1]) << 1;
                    if (code > (1u << bits)) err = ST_BAD_HEADER;
                    next_code[bits] = code;
                }
                first[bits] = uint16_t(code); count[bits] = uint16_t(counts[bits]); offs[bits] = uint16_t(before);
                before += counts[bits];
            }
        }
        if (valid && !err) {
            uint32_t placed[12];
#pragma unroll
            for (int k = 0; k < 12; ++k) placed[k] = 0;
            for (uint32_t sym = 0; sym < nsym; ++sym) {
                uint32_t len = weight(sym);
                if (!len) continue;
                uint32_t cde = 0, at = 0;
#pragma unroll
                for (int k = 1; k < 12; ++k) if (len == uint32_t(k)) { cde = next_code[k]; next_code[k] = cde + 1; at = offs[k] + placed[k]; placed[k]++; }
                if (cde >= (1u << len)) { err = ST_BAD_HEADER; break; }
                syms[at] = uint8_t(sym);
            }
        }
        first[0] = uint16_t(max_bits);
        count[0] = uint16_t(valid && !err);
    }
    { uint32_t be = __shfl_sync(0xFFFFFFFFu, err, c * 4); err = be > err ? be : err; }  // table errors of the builder lane reach its chunk
    max_bits = __shfl_sync(0xFFFFFFFFu, max_bits, c * 4);
    __syncwarp();

    // table: the four lanes of a chunk fill it, one symbol of the canonical list at a time
    {
        const HuffCanon hc = canon_of(c);
        const bool build = valid && !err;
        uint16_t* lut = lut_all + c * (1 << HUF_LUT_BITS);
        if (build) {
            const uint16_t fill = max_bits <= HUF_LUT_BITS ? uint16_t(max_bits << 8) : uint16_t(0);  // a slot no code covers; with longer codes the canonical decoder decides
            for (uint32_t i = s; i < (1u << HUF_LUT_BITS); i += 4) lut[i] = fill;
        }
        __syncwarp();
        if (build) {
            const uint32_t total = uint32_t(hc.offs[11]) + hc.count[11];
            for (uint32_t k = s; k < total; k += 4) {
                uint32_t len = 1;
                while (len < 11 && k >= uint32_t(hc.offs[len]) + hc.count[len]) ++len;
                if (len > HUF_LUT_BITS) continue;
                const uint32_t code = hc.first[len] + (k - hc.offs[len]);
                const uint32_t rev = __brev(code) >> (32 - len);
                const uint16_t entry = uint16_t((len << 8) | hc.syms[k]);
                for (uint32_t idx = rev; idx < (1u << HUF_LUT_BITS); idx += (1u << len)) lut[idx] = entry;
            }
        }
        __syncwarp();
    }

    uint32_t seg_start = 0, seg_len = 0;
    if (valid) split_four_dev(it.n, s, seg_start, seg_len);
    if (valid && !err) {
        const uint16_t* lut = lut_all + c * (1 << HUF_LUT_BITS);
        const HuffCanon hc = canon_of(c);
        Epilogue ep = make_epilogue(bases, it);
        // Stream positions are 32-bit offsets from `org`, a 16-byte aligned address two blocks below the stream's
        // first byte (the look-ahead fetch reaches one block below the stream), so that the compares and steps of
        // the loop are single instructions.
        const uintptr_t org = (reinterpret_cast<uintptr_t>(src + my_off) & ~uintptr_t(15)) - 32;
        const uint32_t start = uint32_t(reinterpret_cast<uintptr_t>(src + my_off) - org);
        uint32_t rp = start + my_len;  // one past the next byte to read (moves down)
        const uintptr_t lo16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_first) & ~uintptr_t(15);
        const uintptr_t hi16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_end + 15) & ~uintptr_t(15);
        // ring holds [fetched, ...): blocks are fetched downward
        uint32_t fetched = (rp + 15) & ~15u;
        for (int k = 0; k < 3; ++k) { fetched -= 16; ring.put(fetched, fetch16(org + fetched, lo16, hi16)); }
        uint4 pending = fetch16(org + fetched - 16, lo16, hi16);

        // bit container: 64 bits kept as two words so that every shift is one funnel shift (a code has at most 11 bits)
        uint32_t c_lo = 0, c_hi = 0;
        int32_t cnt = 0;  // bits in the container
        auto push = [&](uint32_t w) {  // w's bits go above the cnt (<= 32) bits held
            c_lo |= __funnelshift_lc(0u, w, uint32_t(cnt));
            c_hi |= __funnelshift_lc(w, 0u, uint32_t(cnt));
        };
        auto drop = [&](uint32_t nb) { c_lo = __funnelshift_r(c_lo, c_hi, nb); c_hi >>= nb; };
        // byte steps until the read position is word aligned
        while ((rp & 3) && rp > start) { --rp; push(ring.byte(rp)); cnt += 8; }
        const uint32_t mask = (1u << max_bits) - 1;
        uint32_t pos = seg_start, remaining = seg_len;
        // The lanes of a warp drain at similar rates: when any active lane runs low, every lane with room refills,
        // so the refill code runs once per several groups instead of (for some lane) in every one.
        auto ring_top_up = [&]() {
            if (__any_sync(__activemask(), rp - fetched < 32 && fetched > start)) {
                if (rp - fetched <= 48 && fetched > start) { fetched -= 16; ring.put(fetched, pending); pending = fetch16(org + fetched - 16, lo16, hi16); }
            }
        };
        // one aligned word (or the last partial one) into the bit container when it holds at most 32 bits
        auto take_word = [&]() {
            if (cnt <= 32 && rp > start) {
                uint32_t w = __byte_perm(ring.word(rp - 4), 0, 0x0123);  // byte rp-1 becomes the lowest
                uint32_t take = rp - start >= 4 ? 4u : uint32_t(rp - start);
                if (take < 4) w &= (1u << (8 * take)) - 1;
                push(w);
                cnt += 8 * int32_t(take);
                rp -= take;
            }
        };
        // (length << 8) | symbol of the next code, without consuming it
        auto peek = [&]() -> uint32_t {
            uint32_t e = lut[c_lo & ((1u << HUF_LUT_BITS) - 1)];
            if (e == 0) e = huff_canon_decode(hc.syms, max_bits, c_lo & mask, HUF_LUT_BITS + 1);  // the rarest symbols, or a window no code covers
            return e;
        };
        // one symbol with the reference's checks (decompress.rs:176-196)
        auto one_symbol = [&]() -> uint32_t {
            take_word();
            uint32_t e = peek();
            int32_t nb = int32_t(e >> 8);
            if (nb > cnt) { err = ST_STREAM_UNDERRUN; nb = cnt; }
            drop(uint32_t(nb)); cnt -= nb;
            return e;
        };
        // Eight symbols in two halves.  After a refill the container holds more than 32 bits (unless the stream is
        // at its end); four symbols take 44 bits at most and around ten on an exponent plane, so the halves run
        // without a check per symbol: the lowest bit count seen is tested once, and a group that ran out of bits is
        // decoded again one symbol at a time.
        auto dec8 = [&](uint32_t& s_lo, uint32_t& s_hi) {
            ring_top_up();
            const uint32_t lo0 = c_lo, hi0 = c_hi;
            const int32_t cnt0 = cnt;
            const uint32_t rp0 = rp;
            // With eight or more stream bytes left both refills of the group are whole aligned words: one conditional
            // word each, no partial-word handling.  Otherwise the group starts with a negative `lowest` and goes down
            // the checked path.
            int32_t lowest = rp - start >= 8 ? 0 : -1;
            s_lo = 0; s_hi = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if ((j & 3) == 0 && cnt <= 32) {
                    push(__byte_perm(ring.word(rp - 4), 0, 0x0123));  // byte rp-1 becomes the lowest
                    cnt += 32; rp -= 4;
                }
                uint32_t e = peek();
                const uint32_t nb = e >> 8;
                drop(nb); cnt -= int32_t(nb);
                if ((j & 3) == 3) lowest |= cnt;  // the count only falls between two refills
                const uint32_t ins = (0x3210u & ~(0xFu << (4 * (j & 3)))) | (4u << (4 * (j & 3)));  // low byte of e into byte j & 3
                if (j < 4) s_lo = __byte_perm(s_lo, e, ins); else s_hi = __byte_perm(s_hi, e, ins);
            }
            if (lowest < 0) {
                c_lo = lo0; c_hi = hi0; cnt = cnt0; rp = rp0;
                s_lo = 0; s_hi = 0;
                for (uint32_t j = 0; j < 8; ++j) {
                    uint32_t sym = one_symbol() & 0xFFu;
                    if (j < 4) s_lo |= sym << (8 * j); else s_hi |= sym << (8 * (j - 4));
                }
            }
        };
        auto short_group = [&](uint32_t g) {
            uint64_t syms = 0;
            ring_top_up();
            for (uint32_t j = 0; j < g; ++j) syms |= uint64_t(one_symbol() & 0xFFu) << (8 * j);
            emit(ep, pos, g, syms);
            pos += g; remaining -= g;
        };
        if (remaining) {
            uint32_t g = first_group(ep, pos, remaining);
            if (g < 8 || remaining < 16) short_group(g);
        }
        fast_groups(ep, it.n, pos, remaining, dec8);
        while (remaining) short_group(remaining < 8 ? remaining : 8);
        // every stream must end with no unread byte and only zero bits left
        // (decompress.rs:140-144, bitstream.rs:184-186)
        while (rp > start && !err) {
            if (rp - fetched < 32 && fetched > start) { fetched -= 16; ring.put(fetched, pending); pending = fetch16(org + fetched - 16, lo16, hi16); }
            --rp;
            if (ring.byte(rp)) err = ST_NOT_CONSUMED;
        }
        if (!err && (c_lo | c_hi) != 0) err = ST_NOT_CONSUMED;
    }
    if (err) report(status, it.id, err);
}

// ---- tANS ------------------------------------------------------------------
// One serial stream per chunk: a symbol is a table look-up by the state and the
// next state needs the bits the entry says.  Many lanes decode a chunk all the
// same.  The stream's bits are cut into equal runs, one per lane, and every
// lane decodes from its cut on in a guessed state.  Two decoders of one stream
// fall in with one another after a while (same bit, same state; about 1,400
// symbols on an exponent plane of normal weights, 200 - 700 on flatter planes)
// and stay together, so it is enough to know where each of them meets a path
// that another lane walks anyway:
//
// * The stream has nodes at fixed bits, TansShape::SEGS to a run.  A lane that
//   comes past one enters (bit, state) of its first symbol boundary there, with
//   the symbols it has met so far.  A lane that finds its own pair entered
//   already stops: from here on its path is the other lane's.  Lanes do not stop
//   at the end of their run but when they have met another path, or at the
//   start of the last run.
// * Nobody waits for anybody while this goes on; which of two lanes enters a
//   pair first does not change what is decoded from it.
// * Lane 0 starts in the right state.  Its path, then that of the lane it met,
//   and so on is the right one; along it the state at every cut and the number
//   of symbols before it are known.  It is followed by jumps of doubling length
//   (one by one it was 85 steps of 280 cycles with 256 lanes), and once it
//   reaches the last run the walks that still go on are none of it and end:
//   two tANS chunks of 4096 symbols 204 -> 150 us, 256 of 64 Ki 282 -> 258,
//   4049 of 64 Ki 1375 -> 1326.
// * Before it falls in, a lane can take many more symbols out of the same bits
//   than the right path does (codes of rare symbols read out of step are mostly
//   the frequent one).  So a lane that has met as many symbols as the chunk
//   holds is only set aside; where the right path has come to it, one lane
//   takes it up with the number of symbols the right path has left.
// * A last pass decodes every run from its right start and puts the symbols to
//   their places.
//
// A path may meet any other that passes the same node, so with short runs they
// meet sooner: 64 Ki symbols, steps until the last of all lanes has met one:
// 6900 with 32 lanes, 5500 with 64, 4500 with 128, 3400 with 256 (8200 with 128
// lanes that each walked its run again from its neighbour's end until no start
// changed).  Walks that have ended leave their lanes idle, so the ones that go
// on are gathered into fewer warps.  What bounds it: in launches of few chunks
// the latency of a step (54 cycles: the table read, two shifts, an add) times
// those steps; in large ones shared memory (a look-up of 32 lanes takes 3.4
// passes) and the issue slots, 2.7 to 4.3 look-ups per symbol.  A 4096 x 4096
// bf16 tensor in 256 chunks: 607 -> 258 us.  A step is 45 cycles where nothing
// but the group of eight goes on, 60 with the looks at the ring, more with many
// warps.  Tried: loops without a branch that depends on a lane, the group at a
// node decoded twice (317 against 282 us), the look at the ring in the middle
// of every group (313).
//
// Table: one word per state, bit count (low five bits: what a funnel shift
// takes of it) | symbol << 8 | byte offset of the baseline's entry << 16.
constexpr uint32_t TANS_SHORT = 3000;          // chunks below this many symbols are mostly serial
constexpr uint32_t TANS_FEW = 10240;           // chunks below this many have fewer runs than 32 or 64 lanes (tans_runs)
constexpr uint32_t TANS_GATHER = 512;          // symbols between two looks at how many walks are left
constexpr uint32_t TANS_GROUP_BITS = 8 * 11;  // a group of eight symbols takes at most this many

// SEGS: nodes per run; SLOTS: paths a node can hold when every lane has a run (a power of two; what finds no room is met later);
// BLOCKS: per SM.
template <int LANES> struct TansShape;
template <> struct TansShape<32> { static constexpr uint32_t SEGS = 2, SLOTS = 2, BLOCKS = 16; };
template <> struct TansShape<64> { static constexpr uint32_t SEGS = 1, SLOTS = 4, BLOCKS = 12; };
template <> struct TansShape<128> { static constexpr uint32_t SEGS = 1, SLOTS = 8, BLOCKS = 6; };
template <> struct TansShape<256> { static constexpr uint32_t SEGS = 1, SLOTS = 8, BLOCKS = 2; };  // launches of two chunks per SM at most: room for its registers

// Runs of a chunk.  32 and 64 lanes serve launches whose walks fill the GPU: there many walks of a short chunk cost more than they save, and
// nodes that hold few paths each let them pass one another unmet.  us of 1184 chunks, bf16, 32 lanes with up to 32 / 16 / 8 runs: 2700
// symbols 188 / 189 / 151; 4096: 395 / 258 / 189; 6000: 486 / 271 / 245; 8192: 482 / 278 / 310; 64 lanes with up to 64 / 32 / 16: 4096 417 / 180 /
// 204; 8192: 344 / 227 / 287.
template <int LANES>
__device__ __forceinline__ uint32_t tans_runs(uint32_t n) {
    const uint32_t runs = n / (LANES == 32 ? 256 : LANES == 64 ? 128 : n < TANS_SHORT ? 256 : 64);
    const uint32_t most = n >= TANS_FEW || LANES > 64 ? LANES : LANES == 64 ? 32 : n < 5500 ? 8 : 16;
    return runs > most ? most : runs;
}

template <int LANES>
struct TansShared {
    static constexpr uint32_t NODES = LANES * TansShape<LANES>::SEGS, SLOTS = TansShape<LANES>::SLOTS;
    uint32_t table[2048];
    uint32_t ring[20 * LANES];      // 64 bytes of stream per lane, the last 16 twice; while the table is built: work space
    uint32_t key[NODES * SLOTS];   // 0 or 1 << 31 | lane << 16 | bits below the node << 11 | state
    uint32_t count[NODES * SLOTS]; // symbols of that lane so far
    uint32_t link[LANES];          // the entry the lane met, a TANS_ value, or TANS_ASIDE | node << 15 | bits below it << 11 | state
    uint32_t met[LANES];           // its symbols up to there
    uint32_t from[LANES];          // node from which its path is the right one
    uint32_t base[LANES];          // symbols of the chunk minus symbols of the lane, on its right part
    uint32_t start[LANES];         // bits below the cut << 11 | state: the right start of the run
    uint32_t at[LANES];            // symbols before it
    uint32_t tally[LANES / 32];    // walks of each warp
};
constexpr uint32_t TANS_FINISHED = 0xFFFFFFFFu, TANS_DEAD = 0xFFFFFFFEu, TANS_ASIDE = 0x80000000u, TANS_WALKING = 0xFFFFFFFDu, TANS_NONE = 0xFFFFFFFFu;

// All lanes of a chunk.
template <int LANES>
__device__ __forceinline__ void tans_sync() {
    if (LANES == 32) __syncwarp();
    else __syncthreads();
}

// Builds one chunk's table (mod.rs:199-211,346-369); false on a bad header.  `work` holds 384 words and 128 for every warp.
template <int LANES>
__device__ __forceinline__ bool tans_build(const uint8_t* src, uint32_t nsym, uint32_t* table, uint32_t* work) {
    constexpr uint32_t WARPS = LANES / 32, ROWS = 64 / WARPS;  // rows of 32 states to a warp
    const uint32_t l = threadIdx.x, lane = l % 32, warp = l / 32;
    uint32_t* count = work;  // per symbol
    uint16_t* first = reinterpret_cast<uint16_t*>(work + 256);  // its place among the symbols in order
    uint16_t* next = reinterpret_cast<uint16_t*>(work + 384) + 256 * warp;  // the number of its next occurrence in the warp's rows
    for (uint32_t i = l; i < 256; i += LANES) count[i] = 0;
    tans_sync<LANES>();
    if (warp == 0) {
        uint32_t sum = 0;
        bool bad = false;
        for (uint32_t i = lane; i < nsym; i += 32) {
            const uint32_t sy = src[3 + 3 * i], fr = uint32_t(src[4 + 3 * i]) | uint32_t(src[5 + 3 * i]) << 8;
            bad |= fr == 0 || fr > 2048;             // mod.rs:404-411 (above 2048 the sum cannot come out right)
            bad |= atomicExch(&count[sy], fr) != 0;  // a symbol listed twice
            sum += fr;
        }
        sum = __reduce_add_sync(0xFFFFFFFFu, sum);
        if (__any_sync(0xFFFFFFFFu, bad) || sum != 2048) { if (lane == 0) count[0] = ~0u; }
        __syncwarp();
        uint32_t mine = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) mine += count[lane * 8 + k];
        uint32_t run = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, run, d); if (lane >= uint32_t(d)) run += t; }
        run -= mine;
#pragma unroll
        for (int k = 0; k < 8; ++k) { first[lane * 8 + k] = uint16_t(run); run += count[lane * 8 + k]; }
    }
    tans_sync<LANES>();
    if (count[0] == ~0u) return false;
    // position k of the symbols in order goes to state 1283 k mod 2048
    constexpr uint32_t EACH = 2048 / LANES;
    uint32_t sy = 0;
    for (uint32_t d = 128; d; d >>= 1) if (sy + d < 256 && first[sy + d] <= EACH * l) sy += d;
    for (uint32_t k = EACH * l; k < EACH * l + EACH; ++k) {
        while (sy < 255 && first[sy + 1] <= k) ++sy;
        table[(k * 1283u) & 2047u] = sy;
    }
    tans_sync<LANES>();
    // The states of a symbol are numbered in increasing order, from its frequency on: every warp counts the symbols of its rows,
    // the counts are summed over the warps before it, and the rows are gone through once more.
    uint32_t* rows = table + warp * ROWS * 32 + lane;
    if (WARPS > 1) {
        for (uint32_t i = lane; i < 128; i += 32) reinterpret_cast<uint32_t*>(next)[i] = 0;
        __syncwarp();
#pragma unroll 4
        for (uint32_t r = 0; r < ROWS; ++r) {
            const uint32_t s = rows[32 * r], same = __match_any_sync(0xFFFFFFFFu, s);
            if ((same & ((1u << lane) - 1u)) == 0) next[s] += uint16_t(__popc(same));
            __syncwarp();
        }
        tans_sync<LANES>();
    }
    for (uint32_t s = l; s < 256; s += LANES) {
        uint32_t run = count[s];
        uint16_t* q = reinterpret_cast<uint16_t*>(work + 384) + s;
        for (uint32_t w = 0; w < WARPS; ++w, q += 256) { const uint32_t t = *q; *q = uint16_t(run); run += t; }
    }
    tans_sync<LANES>();
    constexpr uint32_t UNROLL = ROWS < 8 ? ROWS : 8;
    for (uint32_t r0 = 0; r0 < ROWS; r0 += UNROLL) {
        uint32_t s[UNROLL], same[UNROLL];
#pragma unroll
        for (uint32_t k = 0; k < UNROLL; ++k) s[k] = rows[32 * (r0 + k)];
#pragma unroll
        for (uint32_t k = 0; k < UNROLL; ++k) same[k] = __match_any_sync(0xFFFFFFFFu, s[k]);
#pragma unroll
        for (uint32_t k = 0; k < UNROLL; ++k) {
            const uint32_t before = same[k] & ((1u << lane) - 1u);
            const uint32_t x = next[s[k]] + __popc(before), nb = 11 - (31 - __clz(x));
            __syncwarp();
            rows[32 * (r0 + k)] = nb | s[k] << 8 | ((x << nb) - 2048u) << 18;
            if (!before) next[s[k]] = uint16_t(x + __popc(same[k]));
            __syncwarp();
        }
    }
    tans_sync<LANES>();
    return true;
}

// Merges a chunk in the block that decoded one of its planes: that plane's bytes lie at `stage`, the end of the chunk's own output
// [dst, dst + n * element size).  Elements go to their places in tiles of ascending position, each read whole before any of it is
// written: a tile's elements end at or below the bytes of the next one's symbols.
template <int LANES, int NP>
__device__ __forceinline__ void merge_in_place(const Bases& bases, const DecodeItem& it, uint8_t* dst, const uint8_t* stage) {
    constexpr int U = NP == 2 ? 2 : 1;  // groups of sixteen elements per thread and tile, all their loads in flight together
    const int kind = it.kind;
    const uint32_t eb = uint32_t(kind_elem_bytes(kind)), n = it.n;
    const uint8_t* src[NP];
    int j = 0;
#pragma unroll
    for (int p = 0; p < NP; ++p) src[p] = p == it.slot ? stage : rd(bases, it.partner[j++]);
    auto slow = [&](uint32_t begin, uint32_t end) {
        for (; begin < end; begin += 8 * LANES) {
            const uint32_t pos = begin + 8 * threadIdx.x, count = pos >= end ? 0 : end - pos < 8 ? end - pos : 8;
            uint64_t b[4] = {0, 0, 0, 0};
#pragma unroll
            for (int p = 0; p < NP; ++p) b[p] = ld_bytes(src[p] + pos, count);
            tans_sync<LANES>();
            if (count) compose_store(kind, dst, pos, count, b);
        }
    };
    // the groups whose aligned blocks lie inside the planes whatever their alignment: not the first and not the last two
    uint32_t head = uint32_t((16 - ((reinterpret_cast<uintptr_t>(dst) / eb) & 15)) & 15) + 16;
    if (head > n) head = n;
    const uint32_t full = n - head < 48 ? 0 : (n - head - 32) >> 4;
    slow(0, head);
    for (uint32_t g0 = 0; g0 < full; g0 += LANES * U) {
        uint4 cur[U][NP], nxt[U][NP];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t g = g0 + u * LANES + threadIdx.x;
            if (g < full) {
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const uintptr_t at = reinterpret_cast<uintptr_t>(src[p]) + head + g * 16;
                    const uint4* q = reinterpret_cast<const uint4*>(at & ~uintptr_t(15));
                    cur[u][p] = *q;
                    if (at & 15) nxt[u][p] = q[1];
                }
            }
        }
        tans_sync<LANES>();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t g = g0 + u * LANES + threadIdx.x;
            if (g < full) {
                uint32_t pw[4][4];
#pragma unroll
                for (int p = 0; p < NP; ++p) extract16(cur[u][p], nxt[u][p], uint32_t(reinterpret_cast<uintptr_t>(src[p]) + head) & 15u, pw[p]);
                merge_store16(kind, dst + size_t(head + g * 16) * eb, pw);
            }
        }
    }
    slow(head + full * 16, n);
}

template <int LANES>
__global__ void __launch_bounds__(LANES, TansShape<LANES>::BLOCKS) tans_decode_kernel(const DecodeItem* __restrict__ items, Bases bases, uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t tans_smem[];
    typedef TansShared<LANES> Shared;
    constexpr uint32_t SEGS = TansShape<LANES>::SEGS, SLOTS = TansShape<LANES>::SLOTS;
    constexpr uint32_t WORD = LANES * 4;  // bytes between two words of a lane's ring
    Shared& sh = *reinterpret_cast<Shared*>(tans_smem);
    const uint32_t l = threadIdx.x;
    const DecodeItem it = items[blockIdx.x];
    const uint8_t* src = rd(bases, it.src);

    // ---- header (mod.rs:388-425) and table ----
    uint32_t nsym = 0;
    bool bad = it.src_len < 3 || src[0] != 11;
    if (!bad) {
        nsym = uint32_t(src[1]) | uint32_t(src[2]) << 8;
        bad = nsym < 2 || nsym > 256 || 3 + nsym * 3 + 8 > it.src_len;
    }
    const uint8_t* bs = src + 3 + nsym * 3 + 8;
    uint64_t total_bits = 0;
    if (!bad) {
        total_bits = uint64_t(ld_u32_unaligned(bs - 8)) | uint64_t(ld_u32_unaligned(bs - 4)) << 32;
        bad = total_bits > uint64_t(it.src_len - (3 + nsym * 3 + 8)) * 8;
    }
    for (uint32_t i = l; i < Shared::NODES * SLOTS; i += LANES) sh.key[i] = 0;
    sh.start[l] = TANS_NONE;
    bad = bad || !tans_build<LANES>(src, nsym, sh.table, sh.ring);
    // A symbol takes at most eleven bits, and so does the first state: what is longer cannot be used up.
    uint32_t err = bad ? uint32_t(ST_BAD_HEADER) : total_bits < 11 ? uint32_t(ST_STREAM_UNDERRUN)
                 : total_bits > 11 * (uint64_t(it.n) + 1) ? uint32_t(ST_NOT_CONSUMED) : uint32_t(ST_OK);
    if (err) { if (l == 0) report(status, it.id, err); return; }

    // ---- runs ----
    // LIFO reader (mod.rs:118-147): the stream is read from its last bit down.
    uint32_t runs = tans_runs<LANES>(it.n);
    if (uint64_t(runs) * (32 * SEGS) > total_bits) runs = uint32_t(total_bits) / (32 * SEGS);  // nodes at least 32 bits apart
    if (runs < 1) runs = 1;
    const uint64_t apart = total_bits / (runs * SEGS);
    uint32_t slot_bits = SLOTS == 8 ? 3 : SLOTS == 4 ? 2 : 1;  // short runs leave more paths to a node, and fewer nodes
    while (slot_bits < 5 && (2u << slot_bits) * runs <= SLOTS * LANES) ++slot_bits;
    const uint32_t slots = 1u << slot_bits;
    const uint32_t last_node = (runs - 1) * SEGS;  // start of the last run, whose symbols are what is left of the chunk's
    const uint64_t floor_bit = uint64_t(reinterpret_cast<uintptr_t>(bs)) * 8;  // bit address of the stream's first bit
    const uint64_t top_bit = floor_bit + total_bits;
    const uintptr_t lo16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_first) & ~uintptr_t(15);
    const uintptr_t hi16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_end + 15) & ~uintptr_t(15);

    // The decoder: bits left (32-bit offset from `org`), byte offset of its state's table entry, and a window on the stream: a 64-byte
    // ring in shared memory, filled downward in aligned 16-byte blocks one step ahead of use.  Word w of the lane's column is row
    // 4 + w; rows 0 to 3 repeat the last four, so that the words below any word are at fixed distances.  The lanes drain at
    // similar rates: when any lane of the warp runs low every one with room takes a block.  `org` lies on a 64-byte boundary, at
    // least 128 bytes below what the lane is on its way to, and moves along (the stream may be longer than 2^32 bits).
    uintptr_t org = 0;
    uint32_t at = 0, entry = 0, fetched = 0;
    uint4 pending;
    uint8_t* ring = reinterpret_cast<uint8_t*>(sh.ring) + l * 4;
    auto park = [&](uint32_t off, const uint4& v) {
        const uint32_t row = (off >> 2) & 12u;
        uint8_t* r = ring + (row + 4) * WORD;
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint32_t*>(r + k * WORD) = w[k];
        if (row == 12) {
#pragma unroll
            for (int k = 0; k < 4; ++k) *reinterpret_cast<uint32_t*>(ring + k * WORD) = w[k];
        }
    };
    auto head_for = [&](uint64_t bit) -> uint32_t {  // moves `org` to suit a walk down to this bit address; its offset
        const uintptr_t to = uintptr_t(bit >> 9 << 6) - 128;
        const uint32_t down = uint32_t(org - to);
        at += down * 8; fetched += down;
        org = to;
        return uint32_t(bit - uint64_t(to) * 8);
    };
    auto begin = [&](uint64_t bit, uint32_t state, uint64_t down_to) {
        org = uintptr_t(down_to >> 9 << 6) - 128;
        at = uint32_t(bit - uint64_t(org) * 8); entry = 4 * state;
        fetched = (at >> 3 & ~15u) - 32;
        uint4 b[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) b[k] = fetch16(org + fetched + 16 * k, lo16, hi16);
        pending = fetch16(org + fetched - 16, lo16, hi16);
#pragma unroll
        for (int k = 0; k < 3; ++k) park(fetched + 16 * k, b[k]);
    };
    auto refill = [&]() {  // at least 28 bytes below the word in use: two groups and the window
        for (;;) {
            const uint32_t have = (at >> 3 & ~3u) + 4 - fetched;
            if (!__any_sync(__activemask(), have < 32)) break;
            if (have <= 48) { fetched -= 16; park(fetched, pending); pending = fetch16(org + fetched - 16, lo16, hi16); }
        }
    };
    const uint8_t* table = reinterpret_cast<const uint8_t*>(sh.table);
    uint32_t w;  // the next bits, highest first
    auto step = [&]() -> uint32_t {  // one symbol's entry; takes its bits off the window
        const uint32_t e = *reinterpret_cast<const uint32_t*>(table + entry);
        entry = (e >> 16) + 4 * __funnelshift_l(w, 0u, e);  // inside the table whatever the stream holds: the baseline has its low bits clear
        w = __funnelshift_l(0u, w, e);
        return e;
    };
    // The next 96 bits in three words.
    auto window = [&](uint32_t& h0, uint32_t& h1, uint32_t& h2) {
        const uint8_t* r = ring + (((at >> 5) & 15u) + 4) * WORD;
        const uint32_t w3 = *reinterpret_cast<const uint32_t*>(r), w2 = *reinterpret_cast<const uint32_t*>(r - WORD), w1 = *reinterpret_cast<const uint32_t*>(r - 2 * WORD),
                       w0 = *reinterpret_cast<const uint32_t*>(r - 3 * WORD);
        h0 = __funnelshift_r(w2, w3, at); h1 = __funnelshift_r(w1, w2, at); h2 = __funnelshift_r(w0, w1, at);
    };
    // Eight symbols.  Two take at most 22 bits and four 44, so that 32 fresh bits for every two need no check.  `each` gets the
    // number and the bits of every symbol.
    auto group = [&](auto&& each) {
        uint32_t h0, h1, h2;
        window(h0, h1, h2);
        w = h0;
        uint32_t e0 = step(); each(0, e0);
        uint32_t e1 = step(); each(1, e1);
        uint32_t two = (e0 + e1) & 31u;  // the low five bits of the sum: 22 at most
        w = __funnelshift_l(h1, h0, two);
        e0 = step(); each(2, e0);
        e1 = step(); each(3, e1);
        uint32_t used = two + ((e0 + e1) & 31u);
        const bool far = used >= 32;
        const uint32_t g0 = __funnelshift_l(far ? h2 : h1, far ? h1 : h0, used), g1 = __funnelshift_l(far ? 0u : h2, far ? h2 : h1, used);
        w = g0;
        e0 = step(); each(4, e0);
        e1 = step(); each(5, e1);
        two = (e0 + e1) & 31u;
        w = __funnelshift_l(g1, g0, two);
        e0 = step(); each(6, e0);
        e1 = step(); each(7, e1);
        used += two + ((e0 + e1) & 31u);
        return used;
    };
    // ---- walks ----
    uint32_t who = l, node = l * SEGS, stand = 0;  // the walk the lane is on, the node behind it, where it stood there: bits below the node << 11 | state
    uint32_t n = 0, most = it.n;                   // symbols since its start (modulo 2^32), and where it is set aside
    bool alive = l + 1 < runs;
    enum { ALL, OWN_RUN, ALONE } walks = ALL;
    auto take_up = [&]() { begin(top_bit - node * apart - (stand >> 11), stand & 2047u, top_bit - (node + 1) * apart); };
    auto set_aside = [&](uint32_t at_node, uint32_t symbols) { alive = false; sh.link[who] = TANS_ASIDE | at_node << 15 | stand; sh.met[who] = symbols; };
    int64_t base = 0;  // the right path: symbols of the chunk minus symbols of the lane; below zero on a lane that had more before it fell in
    auto segment = [&]() -> uint32_t {  // on to the next node: the symbols met
        const uint32_t n0 = n;
        ++node;
        const uint32_t stop = head_for(top_bit - node * apart);
        while (int32_t(at - stop) >= int32_t(2 * TANS_GROUP_BITS) && most - n >= 16) {
            refill();
            at -= group([](int, uint32_t) {});
            at -= group([](int, uint32_t) {});
            n += 16;
        }
        bool over = false;
        while (int32_t(at - stop) > 0 && !over) {  // up to the first boundary at or below the node
            refill();
            const uint32_t need = at - stop;
            uint32_t bits = 0, taken = 0, there = 0, symbols = 0;
            group([&](int, uint32_t e) {
                const bool above = bits < need;
                bits += e & 31u;
                if (above) { taken = bits; there = entry; ++symbols; }
            });
            over = symbols > most - n;
            at -= taken; entry = there; n += symbols;
        }
        if (over) {
            set_aside(node - 1, n0);
            if (walks == ALONE) sh.link[who] = TANS_DEAD;  // the right path: more symbols than the chunk has
            return n - n0;
        }
        stand = (stop - at) << 11 | entry >> 2;
        if ((who == 0 || walks == ALONE) && node % SEGS == 0) {  // the right path, also where it finds no room
            sh.start[node / SEGS] = stand; sh.at[node / SEGS] = uint32_t(base) + n;
        }
        const uint32_t mine = 1u << 31 | who << 16 | stand;
        for (uint32_t k = 0; k < slots; ++k) {
            const uint32_t slot = node * slots + ((stand + k) & (slots - 1));
            const uint32_t old = atomicCAS(&sh.key[slot], 0u, mine);
            if (old == 0) { sh.count[slot] = n; break; }
            if (((old ^ mine) & 0x7FFFu) == 0) {
                alive = false;
                sh.link[who] = slot; sh.met[who] = n;
                break;
            }
        }
        if (alive && node == last_node) { alive = false; sh.link[who] = TANS_FINISHED; sh.met[who] = n; }
        return n - n0;
    };
    uint32_t start0 = 0;
    if (l == 0) {  // run 0 starts behind the eleven bits of the first state
        const uint64_t bit = total_bits - 11;
        const uint8_t* b = bs + (bit >> 3);
        const uint32_t three = uint32_t(b[0]) | uint32_t(b[1]) << 8 | ((bit & 7) > 5 ? uint32_t(b[2]) << 16 : 0u);
        start0 = stand = 11u << 11 | ((three >> (bit & 7)) & 2047u);
        sh.start[0] = start0; sh.at[0] = 0;
        if (!alive) { sh.link[0] = TANS_FINISHED; sh.met[0] = 0; }
    }
    sh.link[l] = alive ? uint32_t(TANS_WALKING) : uint32_t(TANS_FINISHED);
    if (alive) take_up();
    // A damaged or very uneven stream can hold the whole chunk's symbols, or more, between any two nodes, and paths through a repeated pattern never
    // meet: once a warp has walked a quarter of the chunk's symbols the lanes only finish their runs, and the one with the right path goes on
    // alone.  us with three times the symbols / half / a quarter / an eighth, bf16, 2 % normal weights and then two values in turn, 64 Ki
    // symbols, 256 chunks: 4383 / 3163 / 2569 / 2319; 99.9 % zeros 1594 / 1588 / 1871 / 2205; normal planes the same.
    // (In streams of more than 2^31 bits a run whose right start found no room at its node must not become part of the one before.)
    const uint64_t budget = total_bits >> 31 ? 0 : uint64_t(it.n) / 4 + 2048;
    uint64_t spent = 0;
    // As walks end, the others move together into as few warps as hold them, every TANS_GATHER symbols or so.
    uint32_t warps = LANES / 32, looks = 0;
    const uint32_t every = uint32_t(uint64_t(TANS_GATHER) * runs * SEGS / it.n) + 1;
    // The right path is followed from lane 0's on, once nothing moves any more; walks set aside on it are taken up by lane 0.
    uint32_t lane = 0;
    bool too_many = false;
    // The walk whose path the one of `lane` meets, or itself.
    auto met_by = [&](uint32_t walk) -> uint32_t { const uint32_t link = sh.link[walk]; return link < TANS_ASIDE ? (sh.key[link] >> 16) & 0x3FFu : walk; };
    // Whether the right path is known to the last run, in which case the walks still going are none of it: by jumps of doubling length.
    auto complete = [&]() -> bool {
        sh.from[l] = met_by(l);
        tans_sync<LANES>();
#pragma unroll 1
        for (uint32_t d = 1; d < LANES; d *= 2) {
            const uint32_t to = sh.from[sh.from[l]];
            tans_sync<LANES>();
            sh.from[l] = to;
            tans_sync<LANES>();
        }
        const bool done = sh.link[sh.from[0]] == TANS_FINISHED;
        tans_sync<LANES>();
        return done;
    };
    for (;;) {
        const bool go = alive && (walks == ALL ? spent < budget && looks < every : walks == ALONE || node < (who + 1) * SEGS);
        if (__any_sync(0xFFFFFFFFu, go)) {
            uint32_t met = 0;
            if (go) met = segment();
            spent += __reduce_max_sync(0xFFFFFFFFu, met);
            ++looks;
            continue;
        }
        if (walks == ALL) {
            looks = 0;
            if (LANES == 32) {
                __syncwarp();
                if (!__any_sync(0xFFFFFFFFu, alive) || spent >= budget) { walks = OWN_RUN; continue; }
                if (complete()) alive = false;
                continue;
            }
            const uint32_t votes = __ballot_sync(0xFFFFFFFFu, alive);
            if (l % 32 == 0) sh.tally[l / 32] = __popc(votes);
            if (__syncthreads_or(spent >= budget)) { walks = OWN_RUN; continue; }
            if (complete()) { alive = false; walks = OWN_RUN; continue; }
            uint32_t before = 0, total = 0;
#pragma unroll
            for (uint32_t v = 0; v < LANES / 32; ++v) { if (v < l / 32) before += sh.tally[v]; total += sh.tally[v]; }
            const bool gather = (total + 31) / 32 < warps;
            if (gather && alive) {  // every walk stands at a node
                const uint32_t place = before + __popc(votes & ((1u << (l % 32)) - 1u));
                sh.from[place] = who << 24 | node << 15 | stand; sh.base[place] = n;
            }
            __syncthreads();
            if (gather) {
                warps = (total + 31) / 32;
                alive = l < total;
                if (alive) {
                    who = sh.from[l] >> 24; node = sh.from[l] >> 15 & 0x1FFu; stand = sh.from[l] & 0x7FFFu; n = sh.base[l];
                    take_up();
                }
                __syncthreads();
            }
            if (total == 0) walks = OWN_RUN;
            continue;
        }
        uint32_t link;
        if (walks == OWN_RUN) {
            if (alive) set_aside(node, n);
            walks = ALONE;
            // The right path, the walks on it and the symbols before each, by jumps of doubling length: the jumps of every length are kept (the rings
            // are not in use), sums go to the end of the path, and what lane 0 can reach is marked from the longest jump down.
            constexpr uint32_t LOG = LANES == 32 ? 5 : LANES == 64 ? 6 : LANES == 128 ? 7 : 8;
            uint32_t* jump = sh.ring;                                           // [length][lane]
            int64_t* sum = reinterpret_cast<int64_t*>(sh.ring + LOG * LANES);  // [lane]: symbols from the start of this walk's part to the end
            tans_sync<LANES>();
            const uint32_t own = sh.link[l];
            uint32_t to = met_by(l);
            int64_t rest = own < TANS_ASIDE ? int64_t(sh.met[l]) - int64_t(sh.count[own]) : 0;
#pragma unroll 1
            for (uint32_t d = 0; d < LOG; ++d) {
                jump[d * LANES + l] = to; sum[l] = rest;
                tans_sync<LANES>();
                rest += sum[to]; to = jump[d * LANES + to];
                tans_sync<LANES>();
            }
            sum[l] = rest;
            sh.from[l] = l == 0 ? 0 : TANS_NONE;
            tans_sync<LANES>();
            uint32_t end = 0;
#pragma unroll 1
            for (uint32_t d = LOG; d-- > 0;) {
                if (sh.from[l] != TANS_NONE && jump[d * LANES + l] != l) sh.from[jump[d * LANES + l]] = 0;
                end = jump[d * LANES + end];
                tans_sync<LANES>();
            }
            const bool on = sh.from[l] != TANS_NONE;
            const int64_t before = sum[0] - rest;
            tans_sync<LANES>();
            if (on) {
                sh.base[l] = uint32_t(before);
                too_many = own < TANS_ASIDE && before + int64_t(sh.met[l]) > int64_t(it.n);
                if (own < TANS_ASIDE) sh.from[(sh.key[own] >> 16) & 0x3FFu] = own >> slot_bits;
            }
            too_many = LANES == 32 ? __any_sync(0xFFFFFFFFu, too_many) : __syncthreads_or(too_many);
            lane = end;
            base = sum[0] - sum[end];
            tans_sync<LANES>();
        }
        tans_sync<LANES>();
        while ((link = sh.link[lane]) < TANS_ASIDE && !too_many) {
            base += sh.met[lane];
            if (base < 0) base += int64_t(1) << 32;  // (a walk taken up whose count went past 2^32)
            too_many = base > int64_t(it.n);
            base -= sh.count[link];
            lane = (sh.key[link] >> 16) & 0x3FFu;
            if (l == 0) { sh.from[lane] = link >> slot_bits; sh.base[lane] = uint32_t(base); }
        }
        const int64_t before = base + sh.met[lane];
        too_many = too_many || link == TANS_DEAD || before > int64_t(it.n);
        if (too_many || link == TANS_FINISHED) break;
        tans_sync<LANES>();
        if (l == 0) {
            who = lane; node = link >> 15 & 0x1FFu; stand = link & 0x7FFFu;
            n = sh.met[lane]; most = n + uint32_t(int64_t(it.n) - before);
            alive = true;
            take_up();
        }
    }
    if (too_many) { if (l == 0) report(status, it.id, ST_NOT_CONSUMED); return; }  // more symbols than the chunk has
    tans_sync<LANES>();
    // what walks of the right path entered where it is theirs: the starts of the runs
    for (uint32_t slot = l; slot < (last_node + 1) << slot_bits; slot += LANES) {
        const uint32_t key = sh.key[slot], walk = (key >> 16) & 0x3FFu, at_node = slot >> slot_bits;
        if (key == 0 || at_node % SEGS != 0 || sh.from[walk] == TANS_NONE || at_node < sh.from[walk]) continue;
        const uint32_t link = sh.link[walk];
        if (at_node < (link < TANS_ASIDE ? link >> slot_bits : last_node + 1)) { sh.start[at_node / SEGS] = key & 0x7FFFu; sh.at[at_node / SEGS] = sh.base[walk] + sh.count[slot]; }
    }
    tans_sync<LANES>();
    // ---- last pass: the symbols to their places ----
    // With several warps the symbols of a plane that is merged go to the end of the chunk's own output and the block merges them from there,
    // with coalesced accesses; a lone warp merges them as it decodes.
    const bool staged = LANES > 32 && it.fused;
    uint8_t* dst = wr(bases, it.dst);
    uint8_t* stage = staged ? dst + size_t(it.n) * (uint32_t(kind_elem_bytes(it.kind)) - 1) : dst;
    const uint32_t mine = l < runs ? sh.start[l] : TANS_NONE;
    if (mine != TANS_NONE) {
        uint32_t next = l + 1;
        while (next < runs && sh.start[next] == TANS_NONE) ++next;  // no room for the right start at that cut
        const bool last = next >= runs;
        uint32_t pos = sh.at[l], remaining = (last ? it.n : sh.at[next]) - pos;
        const uint64_t end_bit = last ? floor_bit : top_bit - next * SEGS * apart;
        begin(top_bit - l * SEGS * apart - (mine >> 11), mine & 2047u, end_bit);
        // the last run may not read below the stream's first bit; the others are known to end well above theirs
        const uint32_t floor_at = uint32_t(end_bit - uint64_t(org) * 8) - (last ? 0u : 11 + TANS_GROUP_BITS);
        if (int32_t(at - floor_at) < 0) err = ST_STREAM_UNDERRUN;
        auto one_checked = [&]() -> uint32_t {
            if (err) return 0;
            if (at - floor_at < (*reinterpret_cast<const uint32_t*>(table + entry) & 31u)) { err = ST_STREAM_UNDERRUN; return 0; }
            uint32_t h1, h2;
            window(w, h1, h2);
            const uint32_t e = step();
            at -= e & 31u;
            return (e >> 8) & 0xFFu;
        };
        auto eight = [&](uint32_t& s_lo, uint32_t& s_hi) {
            refill();
            if (at - floor_at >= TANS_GROUP_BITS) {
                uint32_t s[8];
                at -= group([&](int j, uint32_t e) { s[j] = e; });
                s_lo = __byte_perm(__byte_perm(s[0], s[1], 0x0051), __byte_perm(s[2], s[3], 0x0051), 0x5410);
                s_hi = __byte_perm(__byte_perm(s[4], s[5], 0x0051), __byte_perm(s[6], s[7], 0x0051), 0x5410);
            } else {
                uint64_t syms = 0;
#pragma unroll 1
                for (int j = 0; j < 8; ++j) syms |= uint64_t(one_checked()) << (8 * j);
                s_lo = uint32_t(syms); s_hi = uint32_t(syms >> 32);
            }
        };
        auto few = [&](uint32_t count) -> uint64_t {  // less than eight, up to a boundary of the output or the end of the run
            uint64_t syms = 0;
            refill();
            if (at - floor_at >= TANS_GROUP_BITS) {
                uint32_t bits = 0, there = 0;
                group([&](int j, uint32_t e) { if (uint32_t(j) < count) { bits += e & 31u; there = entry; syms |= uint64_t((e >> 8) & 0xFFu) << (8 * j); } });
                at -= bits; entry = there;
                return syms;
            }
#pragma unroll 1
            for (uint32_t j = 0; j < count; ++j) syms |= uint64_t(one_checked()) << (8 * j);
            return syms;
        };
        if (LANES > 32) {
            auto bytes = [&](uint32_t count) {
                const uint64_t syms = few(count);
                for (uint32_t k = 0; k < count; ++k) stage[pos + k] = uint8_t(syms >> (8 * k));
                pos += count; remaining -= count;
            };
            const uint32_t head = uint32_t(0u - reinterpret_cast<uintptr_t>(stage + pos)) & 7u;
            if (head) bytes(head < remaining ? head : remaining);
            while (remaining >= 8 && (reinterpret_cast<uintptr_t>(stage + pos) & 31)) {
                uint2 a;
                eight(a.x, a.y);
                *reinterpret_cast<uint2*>(stage + pos) = a;
                pos += 8; remaining -= 8;
            }
#pragma unroll 1
            for (; remaining >= 32; remaining -= 32, pos += 32) {  // whole sectors: a store by lanes that each walk a run of their own costs a pass per lane
                uint4 a, b;
                eight(a.x, a.y); eight(a.z, a.w); eight(b.x, b.y); eight(b.z, b.w);
                stg256_kept(stage + pos, a, b);
            }
            while (remaining >= 8) {
                uint2 a;
                eight(a.x, a.y);
                *reinterpret_cast<uint2*>(stage + pos) = a;
                pos += 8; remaining -= 8;
            }
            if (remaining) bytes(remaining);
        } else {
            const Epilogue ep = make_epilogue(bases, it);
            uint32_t g = remaining ? first_group(ep, pos, remaining) : 8;
            if (g < 8) { emit(ep, pos, g, few(g)); pos += g; remaining -= g; }
            fast_groups(ep, it.n, pos, remaining, eight);
            while (remaining) {
                g = remaining < 8 ? remaining : 8;
                uint64_t syms;
                if (g == 8) { uint32_t lo, hi; eight(lo, hi); syms = lo | uint64_t(hi) << 32; } else syms = few(g);
                emit(ep, pos, g, syms);
                pos += g; remaining -= g;
            }
        }
        if (!err && last && (at != floor_at || entry != 0)) err = ST_NOT_CONSUMED;  // mod.rs:442-449
    }
    if (err) report(status, it.id, err);
    if (staged) {
        tans_sync<LANES>();
        if (it.kind == K_M32) merge_in_place<LANES, 4>(bases, it, dst, stage);
        else merge_in_place<LANES, 2>(bases, it, dst, stage);
    }
}

// The other kernel: a lane per stream, 32 chunks per block, for launches whose chunks fill the GPU that way (tans_kernel).
// One stream per lane and an entry per state: the spread symbols (u8 per state) and (baseline << 5 | bit count) (u16 per
// state), 6 KiB per chunk, so an SM holds 32 chunks whatever the kernel does.  Both tables are laid out [state][lane]: the
// address of an entry is one multiply-add from the state and a lane only touches its own columns.
//
// With 32 streams an SM's throughput is 32 / (time of one symbol), and a lone
// warp pays for every instruction it issues, so the work is split over two
// warps that run on different schedulers.  Warp 0 walks the state chain and
// nothing else: per symbol one table load, three funnel shifts, the count and
// the next state, and one store of the state it left into an exchange buffer.
// Warp 1 turns those states into symbols (the second table), merges them with
// the other planes' bytes, writes the output and keeps the decoder's window of
// stream bytes filled.  They meet once per round of 32 symbols per lane, over
// two exchange buffers in shared memory, on named barriers.  Groups that do
// not fill a round, plane orders without a placing routine below, and the
// checked path near a stream's end run on warp 0 alone.  52 cycles per symbol: 148 us and 27 ns per symbol of a chunk for any
// number of chunks up to 4736, and the same again for every further 4736.
constexpr int TANS_CTA_CHUNKS = 32;
constexpr int TANS_LANES_THREADS = 64;
constexpr int TANS_SYM_BYTES = 2048 * 32;       // [state][lane] of u8
constexpr int TANS_NB_BYTES = 2048 * 2 * 32;    // [state][lane] of u16
constexpr int TANS_RING_WORDS = 64;             // 256 bytes of stream per lane
constexpr int TANS_RING_BYTES = TANS_RING_WORDS * 32 * 4;
constexpr int TANS_XCH_BYTES = 2 * 32 * 32 * 2; // [buffer][symbol of the round][lane] of u16
constexpr int TANS_PUB_BYTES = 2 * 32 * 4;      // [buffer][lane]: read position at the end of the round
constexpr int TANS_HAND_BYTES = 8 * 32 * 4;     // [word][lane]: rounds, position, lowest stream offset fetched, -, first stream offset, window origin (low, high)
constexpr int TANS_NORM_BYTES = 256 * 32 * 2;   // [symbol][lane] of u16: normalised counts while the tables are built (in local memory every state would
                                                // cost an L2 round trip); afterwards the staging area of the other planes' bytes
constexpr int TANS_LANES_SMEM = TANS_SYM_BYTES + TANS_NB_BYTES + TANS_RING_BYTES + TANS_XCH_BYTES + TANS_PUB_BYTES + TANS_HAND_BYTES + TANS_NORM_BYTES;

struct TansRing {
    uint32_t* base;  // &ring[0][lane]
    __device__ __forceinline__ uint32_t& word(uint32_t off) { return base[((off >> 2) & (TANS_RING_WORDS - 1)) * 32]; }
    __device__ __forceinline__ uint8_t byte(uint32_t off) { return reinterpret_cast<uint8_t*>(&word(off))[off & 3]; }
    __device__ __forceinline__ void put(uint32_t off16, uint4 v) {
        word(off16) = v.x; word(off16 + 4) = v.y; word(off16 + 8) = v.z; word(off16 + 12) = v.w;
    }
};
// How a lane's symbols are placed by the second warp.
enum : uint32_t { TP_NONE = 0, TP_PLAIN = 1, TP_M16 = 2, TP_FP8 = 3, TP_M32 = 4 };
__device__ __forceinline__ uint32_t tans_place_mode(const Epilogue& ep) {
    if (!ep.fused) return TP_PLAIN;
    if (ep.kind == K_M16) return TP_M16;
    if (ep.kind == K_E4M3 || ep.kind == K_E5M2) return TP_FP8;
    if (ep.kind == K_M32 && ep.slot == 3) return TP_M32;
    return TP_NONE;
}
__device__ __forceinline__ uint32_t tans_elem_bytes(uint32_t mode) { return mode == TP_M16 ? 2u : mode == TP_M32 ? 4u : 1u; }
__device__ __forceinline__ uint32_t tans_partners(uint32_t mode) { return mode == TP_PLAIN ? 0u : mode == TP_M32 ? 3u : 1u; }
// Rounds of 32 elements that can be placed from `pos` on: the output must sit on a 32-byte boundary and round r reads
// the aligned 32-byte block r + 2 of every partner plane, which must end inside the partner's chunk.
__device__ __forceinline__ uint32_t tans_rounds(const Epilogue& ep, uint32_t mode, uint32_t chunk_n, uint32_t pos, uint32_t remaining) {
    if (mode == TP_NONE) return 0;
    if ((reinterpret_cast<uintptr_t>(ep.dst) + size_t(pos) * tans_elem_bytes(mode)) & 31) return 0;
    uint32_t rounds = remaining >> 5;
    const uint32_t np = tans_partners(mode);
#pragma unroll
    for (uint32_t p = 0; p < 3; ++p) {
        if (p >= np) break;
        const uintptr_t lo = reinterpret_cast<uintptr_t>(ep.partner[p]), hi = lo + chunk_n;
        const uintptr_t q = (lo + pos) & ~uintptr_t(31);
        const uint32_t fit = q + 96 <= hi ? uint32_t((hi - q - 96) >> 5) + 1 : 0;
        rounds = fit < rounds ? fit : rounds;
    }
    return rounds;
}
// The two warps of a block meet on named barriers of 64 threads: the warp that filled (or emptied) an exchange
// buffer arrives, the other one waits.  Every arrival below has exactly one matching wait (both warps run the same
// number of rounds, taken from the same shared-memory words), and a barrier orders the shared-memory accesses of
// the threads that take part without waiting for their global loads in flight, which a memory fence would do.
__device__ __forceinline__ void tans_bar_arrive(uint32_t id) {
    __syncwarp();
    asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void tans_bar_wait(uint32_t id) {
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}
constexpr uint32_t TANS_BAR_FULL = 1, TANS_BAR_EMPTY = 3;  // + buffer index; barrier 0 is __syncthreads

__global__ void __launch_bounds__(TANS_LANES_THREADS, 1) tans_lanes_decode_kernel(const DecodeItem* __restrict__ items, uint32_t n_items, Bases bases, uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = threadIdx.x & 31;
    const bool placer = threadIdx.x >= 32;  // warp 1
    const uint32_t item_idx = blockIdx.x * TANS_CTA_CHUNKS + lane;
    const bool live = item_idx < n_items;
    const DecodeItem it = items[live ? item_idx : 0];
    const uint8_t* src = rd(bases, it.src);
    uint8_t* sym_tab = smem + lane;
    uint8_t* nb_tab = smem + TANS_SYM_BYTES + lane * 2;
    uint8_t* area = smem + TANS_SYM_BYTES + TANS_NB_BYTES;
    TansRing ring{reinterpret_cast<uint32_t*>(area) + lane};
    uint16_t* xch = reinterpret_cast<uint16_t*>(area + TANS_RING_BYTES) + lane;                       // element (b, j) at xch[(b * 32 + j) * 32]
    uint32_t* pub = reinterpret_cast<uint32_t*>(area + TANS_RING_BYTES + TANS_XCH_BYTES) + lane;      // buffer b at pub[b * 32]
    uint32_t* hand = reinterpret_cast<uint32_t*>(area + TANS_RING_BYTES + TANS_XCH_BYTES + TANS_PUB_BYTES) + lane;  // word k at hand[k * 32]
    uint16_t* norm_tab = reinterpret_cast<uint16_t*>(area + TANS_RING_BYTES + TANS_XCH_BYTES + TANS_PUB_BYTES + TANS_HAND_BYTES) + lane;
    auto norm = [&](uint32_t sy) -> uint16_t& { return norm_tab[sy << 5]; };
    auto sym_at = [&](uint32_t u) -> uint8_t& { return sym_tab[u << 5]; };
    auto nb_at = [&](uint32_t u) -> uint16_t& { return *reinterpret_cast<uint16_t*>(nb_tab + (u << 6)); };
    const Epilogue ep = make_epilogue(bases, it);
    const uint32_t mode = tans_place_mode(ep);
    const uintptr_t lo16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_first) & ~uintptr_t(15);
    const uintptr_t hi16 = (reinterpret_cast<uintptr_t>(bases.blob) + bases.blob_end + 15) & ~uintptr_t(15);

    // ---- the placing warp -------------------------------------------------------
    if (placer) {
        __syncthreads();  // tables built, leading groups placed, the hand-over words written
        const uint32_t my_rounds = hand[0];
        const uint32_t max_rounds = __reduce_max_sync(0xFFFFFFFFu, my_rounds);
        uint32_t pos = hand[32], fetched = hand[2 * 32];
        const uint32_t start = hand[4 * 32];
        const uintptr_t org = uintptr_t(hand[5 * 32]) | uintptr_t(hand[6 * 32]) << 32;
        const uint32_t np = tans_partners(mode);
        uintptr_t q[3] = {0, 0, 0};
        uint32_t off[3] = {0, 0, 0};
        // Nothing this warp asks of global memory is waited for in the round that asked: both the other planes' bytes
        // and the stream bytes travel by asynchronous copies (cp.async) straight into shared memory, one group of
        // copies per round, and a round waits for the group issued two rounds earlier.  Partner planes: round r
        // merges the aligned 32-byte blocks r and r + 1 of each plane and requests block r + 3; block k waits in
        // slot k & 3 of a staging area (the space the normalised counts used while the tables were built), laid
        // out [slot][plane][half][lane] in 16-byte units.  Stream bytes go into the decoder's window directly.
        const uint32_t stage = uint32_t(__cvta_generic_to_shared(area + TANS_RING_BYTES + TANS_XCH_BYTES + TANS_PUB_BYTES + TANS_HAND_BYTES)) + lane * 16;
        auto stage_at = [&](uint32_t slot, uint32_t p, uint32_t half) -> uint32_t { return stage + (((slot & 3) * 3 + p) * 2 + half) * 512; };
        auto stage_block = [&](uint32_t slot, uint32_t p) -> Block32 {
            Block32 v;
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]) : "r"(stage_at(slot, p, 0)) : "memory");
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "r"(stage_at(slot, p, 1)) : "memory");
            return v;
        };
        const uint32_t ring_sh = uint32_t(__cvta_generic_to_shared(ring.base));
        Block32 cur[3];
        uint8_t* out = ep.dst + size_t(pos) * tans_elem_bytes(mode);
        if (my_rounds) {
#pragma unroll
            for (uint32_t p = 0; p < 3; ++p) {
                if (p >= np) break;
                const uintptr_t lo = reinterpret_cast<uintptr_t>(ep.partner[p]);
                q[p] = (lo + pos) & ~uintptr_t(31); off[p] = uint32_t((lo + pos) & 31);
                cur[p] = load_block_guarded(q[p], lo, lo + it.n);  // block 0 may start below the chunk
                // blocks 1 and 2: inside the chunk for every lane with a round (tans_rounds)
#pragma unroll
                for (uint32_t k = 1; k < 3; ++k)
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(stage_at(k, p, h)), "l"(q[p] + 32 * k + 16 * h) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");  // so that the first round waits for the group above like every later one
        for (uint32_t r = 0; r < max_rounds; ++r) {
            tans_bar_wait(TANS_BAR_FULL + (r & 1));
            const uint32_t b = r & 1;
            if (r < my_rounds) {
                // Stream bytes: these blocks are visible to the decoder before its round r + 4, by when it is at most
                // 176 bytes below the position it published, so the window is brought down to 241 - 256 bytes below that.
                const int32_t floor_off = int32_t(pub[b * 32]) - 256;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if (int32_t(fetched) - 16 >= floor_off && fetched > start) {
                        fetched -= 16;
                        const uintptr_t a = org + fetched;
                        const uint32_t n = (a >= lo16 && a < hi16) ? 4u : 0u;  // outside the blob's hull: zeros, nothing read
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ring_sh + ((((fetched >> 2) + i) & (TANS_RING_WORDS - 1)) * 32) * 4), "l"(a + 4 * i), "r"(n) : "memory");
                    }
                }
                if (r + 3 <= my_rounds) {
#pragma unroll
                    for (uint32_t p = 0; p < 3; ++p) {
                        if (p >= np) break;
#pragma unroll
                        for (uint32_t h = 0; h < 2; ++h)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(stage_at(r + 3, p, h)), "l"(q[p] + 96 + 16 * h) : "memory");
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 2;" ::: "memory");  // the groups of rounds r - 2 and earlier have landed
            if (r < my_rounds) {
                uint32_t w[8];
                const uint16_t* xs = xch + b * 32 * 32;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const uint32_t sy = sym_at(xs[j * 32]);
                    if ((j & 3) == 0) w[j >> 2] = sy; else w[j >> 2] |= sy << (8 * (j & 3));
                }
                uint32_t pw[3][8];
#pragma unroll
                for (uint32_t p = 0; p < 3; ++p) {
                    if (p >= np) break;
                    const Block32 nxt = stage_block(r + 1, p);
                    extract32(cur[p], nxt, off[p], pw[p]);
                    cur[p] = nxt;
                    q[p] += 32;
                }
                if (mode == TP_PLAIN) {
                    stg256(out, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
                    out += 32;
                } else if (mode == TP_M16) {
                    uint4 v[4];
                    const bool low_plane = ep.slot == 0;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        if (low_plane) { compose16x4(w[2 * g], pw[0][2 * g], v[g].x, v[g].y); compose16x4(w[2 * g + 1], pw[0][2 * g + 1], v[g].z, v[g].w); }
                        else { compose16x4(pw[0][2 * g], w[2 * g], v[g].x, v[g].y); compose16x4(pw[0][2 * g + 1], w[2 * g + 1], v[g].z, v[g].w); }
                    }
                    stg256(out, v[0], v[1]);
                    stg256(out + 32, v[2], v[3]);
                    out += 64;
                } else if (mode == TP_FP8) {
                    const bool high_plane = ep.slot == 0, e4m3 = ep.kind == K_E4M3;
                    uint32_t v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = high_plane ? compose_fp8x4(w[k], pw[0][k], e4m3) : compose_fp8x4(pw[0][k], w[k], e4m3);
                    stg256(out, make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]));
                    out += 32;
                } else {  // TP_M32: bytes 0..2 from the partner planes, byte 3 from this lane (transforms/fusion.rs:287-292)
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        uint32_t v[8];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t t0 = __byte_perm(pw[0][k + h], pw[1][k + h], 0x5140), t1 = __byte_perm(pw[2][k + h], w[k + h], 0x5140);
                            const uint32_t t2 = __byte_perm(pw[0][k + h], pw[1][k + h], 0x7362), t3 = __byte_perm(pw[2][k + h], w[k + h], 0x7362);
                            v[4 * h + 0] = revert32(__byte_perm(t0, t1, 0x5410));
                            v[4 * h + 1] = revert32(__byte_perm(t0, t1, 0x7632));
                            v[4 * h + 2] = revert32(__byte_perm(t2, t3, 0x5410));
                            v[4 * h + 3] = revert32(__byte_perm(t2, t3, 0x7632));
                        }
                        stg256(out, make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]));
                        out += 32;
                    }
                }
            }
            if (r + 2 < max_rounds) tans_bar_arrive(TANS_BAR_EMPTY + b);  // the decoder waits for it before round r + 2
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // the stream bytes asked for in the last two rounds
        hand[2 * 32] = fetched;
        __syncthreads();  // the rounds are over: the decoding warp takes the window back
        return;
    }

    // ---- the decoding warp ------------------------------------------------------
    uint32_t err = ST_OK;
    // header (mod.rs:388-425)
    uint32_t nsym = 0;
    if (!live) err = ST_BAD_HEADER;  // never reported: the lane has no item
    else if (it.src_len < 3 || src[0] != 11) err = ST_BAD_HEADER;
    else {
        nsym = uint32_t(src[1]) | uint32_t(src[2]) << 8;
        if (nsym < 2 || nsym > 256 || 3 + nsym * 3 + 8 > it.src_len) err = ST_BAD_HEADER;
    }
    // tables: the spread walks a running position and the decode entries count earlier states of the same
    // symbol, so both are sequential (mod.rs:199-211,346-369); every lane builds its own chunk's
    if (!err) {
        for (uint32_t i = 0; i < 256; ++i) norm(i) = 0;
        uint32_t sum = 0;
        bool bad = false;
        for (uint32_t i = 0; i < nsym; ++i) {  // no early exit: the loads of later entries need not wait for the checks of earlier ones
            const uint32_t sy = src[3 + 3 * i], fr = uint32_t(src[4 + 3 * i]) | uint32_t(src[5 + 3 * i]) << 8;
            bad |= fr == 0 || norm(sy) != 0;  // mod.rs:404-411
            bad |= fr > 2048;                 // the sum cannot come out right; keeps the 16-bit counters exact
            if (!bad) norm(sy) = uint16_t(fr);
            sum += fr;
        }
        if (bad || sum != 2048) err = ST_BAD_HEADER;
        if (!err) {
            uint32_t pos = 0;
            for (uint32_t sy = 0; sy < 256; ++sy) {
                const uint32_t f = norm(sy);
                for (uint32_t k = 0; k < f; ++k) { sym_at(pos) = uint8_t(sy); pos = (pos + 1283u) & 2047u; }
            }
            // the symbols of eight states are read ahead of the counter updates, which depend on one another through memory
            for (uint32_t u0 = 0; u0 < 2048; u0 += 8) {
                uint32_t sy[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) sy[i] = sym_at(u0 + i);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t x = norm(sy[i]);
                    norm(sy[i]) = uint16_t(x + 1);
                    const uint32_t nb = 11 - (31 - __clz(x));
                    nb_at(u0 + i) = uint16_t((((x << nb) - 2048) << 5) | nb);  // baseline above the bit count: a shift by the entry takes its low five bits
                }
            }
        }
    }
    uint64_t total_bits = 0, bslen = 0;
    const uint8_t* bs = src;
    if (!err) {
        const uint8_t* hp = src + 3 + nsym * 3;
        total_bits = uint64_t(ld_u32_unaligned(hp)) | uint64_t(ld_u32_unaligned(hp + 4)) << 32;
        bs = hp + 8;
        bslen = it.src_len - (3 + nsym * 3 + 8);
        if (total_bits > bslen * 8) err = ST_BAD_HEADER;
    }
    // LIFO reader (mod.rs:118-147): the stream is read from its last byte down, every byte from its high bit
    // down.  The `cnt` unread bits sit at the top of the 64-bit container c_hi:c_lo, the next to be used highest, so taking n bits is
    // one funnel shift; a word read little-endian from below the read position has its bytes in that order.
    // (the container is two words, so that every shift on the way of a symbol is one funnel shift)
    uint32_t c_hi = 0, c_lo = 0;
    int32_t cnt = 0;
    // Stream bytes pass through a 256-byte ring per lane in shared memory, filled downward in aligned 16-byte
    // blocks.  Positions are 32-bit offsets from `org`, a 16-byte aligned address two blocks below the stream.
    // While this warp decodes alone it requests blocks one step ahead (`pending`); a lane's loads must not be
    // waited for by the other lanes of the warp (the scoreboard is per warp), so blocks are taken by all lanes
    // with room at once, when any lane runs low, every few groups.
    const uintptr_t org = (reinterpret_cast<uintptr_t>(bs) & ~uintptr_t(15)) - 32;
    const uint32_t start = uint32_t(reinterpret_cast<uintptr_t>(bs) - org);
    uint32_t rp = start, fetched = start, state = 0;
    uint4 pending = make_uint4(0, 0, 0, 0);
    uint32_t pos = 0, remaining = err ? 0 : it.n;
    auto ring_top_up = [&]() {
        if (__any_sync(__activemask(), rp - fetched < 32 && fetched > start)) {
            if (rp - fetched <= 240 && fetched > start) { fetched -= 16; ring.put(fetched, pending); pending = fetch16(org + fetched - 16, lo16, hi16); }
        }
    };
    auto refill = [&]() {  // up to more than 32 bits, by bytes until the position is word aligned, then by words
        while (uint32_t(cnt) <= 32u && rp > start) {  // (a negative count only occurs in a group that is about to be decoded again)
            if (rp - start >= 4 && (rp & 3) == 0) {
                const uint32_t word = ring.word(rp - 4);
                const uint32_t s = uint32_t(32 - cnt);  // 0..32: the word goes below the cnt bits held
                c_hi |= __funnelshift_lc(word, 0u, s);
                c_lo |= __funnelshift_lc(0u, word, s);
                cnt += 32; rp -= 4;
            } else {
                --rp;
                const uint64_t t = uint64_t(ring.byte(rp)) << (56 - cnt);
                c_hi |= uint32_t(t >> 32); c_lo |= uint32_t(t);
                cnt += 8;
            }
        }
    };
    auto take = [&](uint32_t e) -> uint32_t {  // the bit count (<= 11) is the low five bits of e, which is all a funnel shift looks at
        const uint32_t v = __funnelshift_l(c_hi, 0u, e);  // the top bits; 0 for a count of 0
        c_hi = __funnelshift_l(c_lo, c_hi, e);
        c_lo = __funnelshift_l(0u, c_lo, e);
        cnt -= int32_t(e & 31u);
        return v;
    };
    // one symbol with the reference's checks
    auto one_symbol = [&]() -> uint32_t {
        refill();
        const uint32_t sy = sym_at(state), e = nb_at(state), nb = e & 31u;
        if (int32_t(nb) > cnt) { err = ST_STREAM_UNDERRUN; return sy; }
        state = (e >> 5) + take(e);
        if (state >= 2048) { err = ST_STREAM_UNDERRUN; state = 0; }
        return sy;
    };
    // a refill by one aligned word, taken when 32 bits or fewer are held
    auto refill_word = [&]() {
        if (cnt <= 32) {
            const uint32_t word = ring.word(rp - 4);
            const uint32_t s = uint32_t(32 - cnt);
            c_hi |= __funnelshift_lc(word, 0u, s);
            c_lo |= __funnelshift_lc(0u, word, s);
            cnt += 32; rp -= 4;
        }
    };
    // Eight symbols in two halves of four: after a refill the container holds more than 32 bits (unless the
    // stream is at its end) and four symbols take at most 44, around ten on an exponent plane, so the
    // halves run unchecked; a group that ran out of bits is decoded again one symbol at a time.
    auto dec8 = [&](uint32_t& s_lo, uint32_t& s_hi) {
        const uint32_t hi0 = c_hi, lo0 = c_lo;
        const int32_t cnt0 = cnt;
        ring_top_up();
        const uint32_t rp0 = rp, state0 = state;
        int32_t lowest = 0;
        s_lo = 0; s_hi = 0;
        // Away from the stream's first bytes the read position is word aligned and stays so: a refill is then
        // one word, taken or not, with no loop and no byte steps.  `lowest` starts negative otherwise, which
        // sends the group down the checked path.
        const bool words = (rp & 3) == 0 && rp - start >= 8;
        if (!words) lowest = -1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if ((j & 3) == 0) refill_word();
            const uint32_t sy = sym_at(state), e = nb_at(state);
            state = (e >> 5) + take(e);  // below 2048 whatever the stream holds: the baseline has its low bits clear and the stream adds fewer than 2^count
            if ((j & 3) == 3) lowest |= cnt;  // the count only falls between two refills
            const uint32_t ins = (0x3210u & ~(0xFu << (4 * (j & 3)))) | (4u << (4 * (j & 3)));
            if (j < 4) s_lo = __byte_perm(s_lo, sy, ins); else s_hi = __byte_perm(s_hi, sy, ins);
        }
        if (lowest < 0) {
            c_hi = hi0; c_lo = lo0; cnt = cnt0; rp = rp0; state = state0;
            s_lo = 0; s_hi = 0;
            for (uint32_t j = 0; j < 8 && !err; ++j) {
                uint32_t sy = one_symbol();
                if (j < 4) s_lo |= sy << (8 * j); else s_hi |= sy << (8 * (j - 4));
            }
        }
    };
    auto short_group = [&](uint32_t g) {
        uint64_t syms = 0;
        ring_top_up();
        for (uint32_t j = 0; j < g && !err; ++j) syms |= uint64_t(one_symbol()) << (8 * j);
        emit(ep, pos, g, syms);
        pos += g; remaining -= g;
    };
    uint32_t rounds = 0;
    if (!err) {
        uint32_t bi = uint32_t((total_bits + 7) >> 3);  // bytes that hold declared bits; the next to load is bs[bi-1]
        const uint32_t top = uint32_t(total_bits & 7);
        if (top) { --bi; c_hi = (bs[bi] & ((1u << top) - 1)) << (32 - top); cnt = int32_t(top); }
        rp = start + bi;  // one past the next byte to read (moves down)
        fetched = (rp + 15) & ~15u;
        for (int k = 0; k < 15; ++k) { if (fetched <= start) break; fetched -= 16; ring.put(fetched, fetch16(org + fetched, lo16, hi16)); }
        pending = fetch16(org + fetched - 16, lo16, hi16);
        refill();
        if (cnt < 11) err = ST_STREAM_UNDERRUN; else state = take(11);
        // leading groups, until the elements that follow start on a 32-byte boundary of the output
        if (!err && remaining) {
            uint32_t g = first_group(ep, pos, remaining);
            if (g < 8 || remaining < 16) short_group(g);
        }
        const uint32_t eb = tans_elem_bytes(mode);
        while (!err && mode != TP_NONE && remaining >= 40 && ((reinterpret_cast<uintptr_t>(ep.dst) + size_t(pos) * eb) & 31) != 0) short_group(8);
        if (!err) rounds = tans_rounds(ep, mode, it.n, pos, remaining);
        if (rounds) {
            // hand the window over full: what the second warp adds becomes visible from the fifth round on
            while (int32_t(fetched) - 16 >= int32_t(rp) - 256 && fetched > start) { fetched -= 16; ring.put(fetched, pending); pending = fetch16(org + fetched - 16, lo16, hi16); }
        }
    }
    hand[0] = rounds; hand[32] = pos; hand[2 * 32] = fetched; hand[4 * 32] = start;
    hand[5 * 32] = uint32_t(org); hand[6 * 32] = uint32_t(uint64_t(org) >> 32);
    __syncthreads();
    {
        const uint32_t max_rounds = __reduce_max_sync(0xFFFFFFFFu, rounds);
        for (uint32_t r = 0; r < max_rounds; ++r) {
            if (r >= 2) tans_bar_wait(TANS_BAR_EMPTY + (r & 1));  // the buffer of round r - 2 has been placed
            if (r < rounds) {
                uint16_t* xs = xch + (r & 1) * 32 * 32;
                const uint32_t hi0 = c_hi, lo0 = c_lo, rp0 = rp, state0 = state;
                const int32_t cnt0 = cnt;
                // eight word refills at most: the read position must be word aligned and 32 bytes above the stream's first
                int32_t lowest = ((rp & 3) == 0 && rp - start >= 32) ? 0 : -1;
                if (lowest == 0) {
                    // The word a refill would take is loaded four symbols before the count says whether it is
                    // taken, so that no shared-memory load sits between a symbol's bits and the next state.
                    uint32_t ahead_word = ring.word(rp - 4);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if ((j & 3) == 0) {
                            const bool need = cnt <= 32;
                            const uint32_t sft = uint32_t(32 - cnt);  // clamped to 32 by the shifts; unused when the word is not taken
                            const uint32_t in_hi = __funnelshift_lc(ahead_word, 0u, sft), in_lo = __funnelshift_lc(0u, ahead_word, sft);
                            c_hi |= need ? in_hi : 0u; c_lo |= need ? in_lo : 0u;
                            cnt += need ? 32 : 0; rp -= need ? 4u : 0u;
                            ahead_word = ring.word(rp - 4);
                        }
                        const uint32_t e = nb_at(state);
                        xs[j * 32] = uint16_t(state);
                        state = (e >> 5) + take(e);
                        if ((j & 3) == 3) lowest |= cnt;
                    }
                }
                if (lowest < 0) {  // near the stream's end, or out of bits: again with the reference's checks
                    c_hi = hi0; c_lo = lo0; cnt = cnt0; rp = rp0; state = state0;
                    for (uint32_t j = 0; j < 32; ++j) {
                        xs[j * 32] = uint16_t(state);
                        if (!err) one_symbol();
                    }
                }
                pub[(r & 1) * 32] = rp;
            }
            tans_bar_arrive(TANS_BAR_FULL + (r & 1));
        }
    }
    __syncthreads();
    if (rounds) {
        pos += rounds * 32; remaining -= rounds * 32;
        fetched = hand[2 * 32];
        pending = fetch16(org + fetched - 16, lo16, hi16);
    }
    if (!err) fast_groups(ep, it.n, pos, remaining, dec8);
    while (remaining && !err) short_group(remaining < 8 ? remaining : 8);
    if (!err && (cnt != 0 || rp != start || state != 0)) err = ST_NOT_CONSUMED;  // mod.rs:442-449
    if (err && live) report(status, it.id, err);
}
template <int LANES>
inline void tans_launch_t(const DecodeItem* items, uint32_t n, const Bases& bases, uint32_t* status, cudaStream_t st) {
    tans_decode_kernel<LANES><<<n, LANES, sizeof(TansShared<LANES>), st>>>(items, bases, status);
}
// Lanes per chunk: many shorten a chunk's latency and cost more walks per symbol, so as many as the GPU has room for.  us with
// 256 / 128 / 64 / 32 lanes, bf16: 64 Ki symbols, 148 chunks 195 / 255 / 351 / 586, 592: 429 / 319 / 412 / 838, 1184: 791 / 543 / 568 / 876,
// 2368: 1440 / 888 / 839 / 962; 16 Ki, 296: 184 / 172 / 228 / 491, 1184: 559 / 311 / 322 / 532, 2368: 1021 / 511 / 482 / 629; 8 Ki, 1776:
// 594 / 347 / 271 / 326.  Runs that are long against the way to a meeting (`apart`, in symbols of 1,400) need fewer walks: fp8, 64 Ki, 2368: 2393 /
// 1446 / 1430 / 1298; fp16, 8 Ki, 2368: 506 / 299 / 290 / 226 (bf16, 128 Ki, 3552: 2892 / 1834 / 1763 / 1687).  In chunks that are mostly
// serial the other lanes only cost: 1024 symbols, 2368 chunks 128: 175, 32: 126.  Below TANS_FEW symbols the rounds of blocks count, 12 per SM
// with 64 lanes and 16 with 32; 64 / 32 lanes: 3500 symbols, 1184 chunks 184 / 180, 1776 223 / 200 (fp16 150 / 155, 183 / 184); 6000: 1776 272 / 299,
// 1900 294 / 307, 2368 380 / 315.  Where 32 lanes take as many rounds as 64 (2369 to 3552 chunks, 4737 to 5328) what counts is how the last round
// ends: a few blocks of 32 lanes begin when the first ones of the round before end, some dozens take a round's latency, and the more of them the less
// that matters.  64 / 32 lanes, fp16 (apart 0.08): 32 Ki, 2369 chunks 467 / 462, 2400 465 / 500, 3552 578 / 596, 4737 732 / 694, 4800 734 / 748, 5328 801 /
// 819; 64 Ki, 2400 775 / 808, 2900 869 / 869, 3100 920 / 895, 3552 992 / 946, 4737 1299 / 1176, 5328 1423 / 1326.  fp8 (0.25): 20 Ki, 3330 976 / 1118, 4737
// 1327 / 1400; 32 Ki, 2369 1015 / 956, 3000 1129 / 1192; 64 Ki, 3000 1657 / 1674, 3552 1854 / 1806, 4737 2403 / 2260; a layer of 3330 1829 / 1883.  Bytes of
// 6.4 bits (0.04): 16 Ki, 3000 315 / 303, 4800 440 / 415; 32 Ki, 2376 387 / 388, 2700 405 / 451, 3552 467 / 481, 4737 603 / 555.  Over 588 launches of 8 Ki to 64 Ki
// the rule is 1.004 times the better of the two (geometric mean; 64 always 1.015, 32 1.017), 1.05 at worst (64 1.23, 32 1.14).
constexpr uint32_t TANS_ROUND_64 = 148 * TansShape<64>::BLOCKS, TANS_ROUND_32 = 148 * TansShape<32>::BLOCKS;
inline uint32_t tans_lanes(uint32_t chunks, uint32_t longest, double apart) {
    if (longest < TANS_SHORT) return chunks <= 4 * 148 ? 128 : 32;
    if (chunks <= (longest <= 4096 ? 148 : 2 * 148)) return 256;
    if (chunks <= 6 * 148) return 128;
    if (longest < 4000 && (apart > 0.5 || chunks > TANS_ROUND_64)) return 32;
    if (longest < TANS_FEW) return chunks > TANS_ROUND_64 && chunks <= TANS_ROUND_32 ? 32 : 64;
    if (chunks <= TANS_ROUND_64 || longest <= 65536 * apart) return 64;
    const uint32_t before = (chunks - 1) / TANS_ROUND_32, over = chunks - before * TANS_ROUND_32;  // whole rounds of 32 lanes, chunks in the one after them
    if (longest > 65536 || before < (chunks - 1) / TANS_ROUND_64) return 32;
    if (apart < 0.06) return before == 1 && over >= 32 && longest >= 24 << 10 ? 64 : 32;
    if (before > 1) return (over >= 64 && longest <= 32 << 10) || (apart > 0.2 && longest <= 24 << 10) ? 64 : 32;
    return over >= 4 && (apart > 0.2 || uint64_t(longest) * over <= 44u << 20) ? 64 : 32;
}
// `lanes` per chunk; 1: the kernel with a lane per stream.
inline void tans_launch(const DecodeItem* items, uint32_t n, const Bases& bases, uint32_t* status, uint32_t lanes, cudaStream_t st) {
    switch (lanes) {
        case 256: tans_launch_t<256>(items, n, bases, status, st); break;
        case 128: tans_launch_t<128>(items, n, bases, status, st); break;
        case 64: tans_launch_t<64>(items, n, bases, status, st); break;
        case 32: tans_launch_t<32>(items, n, bases, status, st); break;
        default: tans_lanes_decode_kernel<<<(n + TANS_CTA_CHUNKS - 1) / TANS_CTA_CHUNKS, TANS_LANES_THREADS, TANS_LANES_SMEM, st>>>(items, n, bases, status);
    }
}
// Shared memory of an SM that the launch's blocks take there at once, if they all find room.
inline uint64_t tans_shared(uint32_t n, uint32_t lanes) {
    const uint64_t bytes = lanes == 256 ? sizeof(TansShared<256>) : lanes == 128 ? sizeof(TansShared<128>) : lanes == 64 ? sizeof(TansShared<64>) : lanes == 32 ? sizeof(TansShared<32>) : TANS_LANES_SMEM;
    const uint64_t per_block = lanes == 1 ? TANS_CTA_CHUNKS : 1;
    return (n + 148 * per_block - 1) / (148 * per_block) * (bytes + 1024);
}
template <int LANES>
inline cudaError_t tans_allow_shared_t() {
    const cudaError_t e = cudaFuncSetAttribute(tans_decode_kernel<LANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TansShared<LANES>)));
    return e != cudaSuccess ? e : cudaFuncSetAttribute(tans_decode_kernel<LANES>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}
inline cudaError_t tans_allow_shared() {
    cudaError_t e = cudaFuncSetAttribute(tans_lanes_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TANS_LANES_SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(tans_lanes_decode_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    if ((e = tans_allow_shared_t<256>()) != cudaSuccess || (e = tans_allow_shared_t<128>()) != cudaSuccess ||
        (e = tans_allow_shared_t<64>()) != cudaSuccess) return e;
    return tans_allow_shared_t<32>();
}

// ---- Order1ScaleAC ---------------------------------------------------------
// One range-coder stream per chunk, one warp per chunk, every lane carrying the
// same coder state.  The stream is serial, so what counts is the way from one
// symbol to the next, and that goes through a search: which symbol's share of
// the range the code falls into.  The 256 shares of a context are mostly dust
// (a symbol the plane never showed after this one still has 1 of 4096), so the
// warp keeps the 32 widest in shared memory, one per lane: cumulative count,
// width, symbol and where the symbol's own row lies.  Every lane goes on as if
// its share were the one: new offset and range, renormalised.  One of them is
// right, and three maxima over the warp hand its state to all.  From row to row
// that is a shared-memory read, a multiply-add, a comparison and a maximum (20
// cycles; a vote, its first set bit and a shuffle are 80).  A code that falls into none of the 32 shares is searched among all
// 256 from the serialized state.  Only the code's distance from the low end of
// the range matters (both lose the same bits to renormalisation), so that is
// what is carried.
// Branches are left out of that way as well.  A code outside the 32 shares leaves a range of zero, which no share of any row
// can win again, so one look per eight symbols finds it and the eight are decoded again one by one; the end of a row is looked
// for once per eight symbols too, and the stream's words for eight symbols are read at once, from a buffer in shared memory
// that the warp fills 256 bytes at a time.  280 chunks of 32 Ki scales: 4.12 ms (247 cycles per symbol) with two maxima over
// packed shares and everything else behind them, 4.00 with the lanes' own next states, 2.14 without the branches, 2.09 (120 cycles) with
// the next row asked for before the other two maxima and 64 bits of stream for four symbols instead of a window moved for each; 2400
// chunks 5.88 -> 5.45.  Leading zeros instead of the two comparisons: 2.23, 5.12.
constexpr uint32_t O1_ROW_BYTES = 32 * 12;  // per lane {minus the cumulative count, width}, then per lane the offset of the symbol's row << 8 | symbol
constexpr uint32_t O1_HALF = 64;            // words in half of the stream buffer
// Context rows of a chunk whose state has `state_len` bytes, the marginal's included (0 when the state is too short to hold any).
inline uint32_t o1sac_tables(uint64_t state_len) { return state_len >= 32 + 512 ? uint32_t((state_len - 32 - 512) / 512) + 1 : 0; }

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) o1sac_decode_kernel(const DecodeItem* __restrict__ items, uint32_t n_items, Bases bases, uint32_t* __restrict__ status, uint32_t smem_rows) {
    extern __shared__ __align__(16) uint8_t all_rows[];
    __shared__ uint32_t all_bitmaps[WARPS][8], all_words[WARPS][2 * O1_HALF];
    __shared__ uint16_t all_row_of[WARPS][256];
    // (the maximum tells the compiler that the warp's number is the same for all lanes: 2213 -> 2012 us for a chunk)
    const uint32_t lane = threadIdx.x % 32, warp = WARPS == 1 ? 0 : __reduce_max_sync(0xFFFFFFFFu, threadIdx.x / 32), chunk = blockIdx.x * WARPS + warp;
    if (WARPS > 1 && chunk >= n_items) return;
    uint8_t* smem = all_rows + warp * smem_rows * O1_ROW_BYTES;
    const DecodeItem it = items[chunk];
    const uint8_t* st = rd(bases, it.state);
    uint32_t* bitmap = all_bitmaps[warp];   // contexts that have a row
    uint32_t* words = all_words[warp];      // the stream
    uint16_t* row_of = all_row_of[warp];    // the row a symbol leads to: 0 = marginal, 1 + rank of the context otherwise
    uint32_t err = it.state_version != 1 || it.state_len < 32 + 512 ? uint32_t(ST_BAD_STATE) : uint32_t(ST_OK);
    uint32_t rows = 1;
    if (!err) {
        if (lane < 8) bitmap[lane] = ld_u32_unaligned(st + 4 * lane);
        __syncwarp();
        for (int i = 0; i < 8; ++i) rows += __popc(bitmap[i]);
        // the host sized the launch from the same lengths
        if (it.state_len != 32 + 512 * rows || rows > smem_rows) err = ST_BAD_STATE;
    }
    if (err) { if (lane == 0) report(status, it.id, err); return; }
    for (uint32_t p = lane; p < 256; p += 32) {  // order1_scale_ac.rs:95-103
        uint32_t r = __popc(bitmap[p >> 5] & ((1u << (p & 31)) - 1));
        for (uint32_t b = 0; b < (p >> 5); ++b) r += __popc(bitmap[b]);
        row_of[p] = uint16_t((bitmap[p >> 5] >> (p & 31)) & 1 ? 1 + r : 0);
    }
    __syncwarp();
    // a lane's eight probabilities of a row and the count below the first of them
    auto load_row = [&](uint32_t row, uint32_t v[8]) -> uint32_t {
        const uint8_t* q = st + 32 + 512 * row + 16 * lane;
        const uint64_t a = ld8_unaligned(q), b = ld8_unaligned(q + 8);
        uint32_t sum = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) { v[k] = uint32_t((k < 4 ? a : b) >> (16 * (k & 3))) & 0xFFFFu; sum += v[k]; }
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d); if (lane >= uint32_t(d)) incl += t; }
        return incl - sum;
    };
    for (uint32_t row = 0; row < rows; ++row) {
        uint32_t v[8], cum = load_row(row, v), sum = 0, zero = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) { sum += v[k]; zero |= v[k] == 0; }
        if (__any_sync(0xFFFFFFFFu, zero) || __shfl_sync(0xFFFFFFFFu, cum + sum, 31) != 4096) err = ST_BAD_STATE;  // quantize.rs:53-71
        if (err) break;
        // the smallest width that at most 32 symbols exceed
        auto wider = [&](uint32_t w) -> uint32_t { uint32_t n = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) n += v[k] > w;
            return __reduce_add_sync(0xFFFFFFFFu, n); };
        uint32_t dust = 1;
        if (wider(dust) > 32) {
            uint32_t hi = 4096;  // more than 32 exceed `dust`, at most 32 exceed `hi`
            while (hi - dust > 1) { const uint32_t mid = (hi + dust) >> 1; if (wider(mid) > 32) dust = mid; else hi = mid; }
            dust = hi;
        }
        uint32_t mine = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) mine += v[k] > dust;
        uint32_t at = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, at, d); if (lane >= uint32_t(d)) at += t; }
        const uint32_t used = __shfl_sync(0xFFFFFFFFu, at, 31);
        at -= mine;
        uint2* out = reinterpret_cast<uint2*>(smem + row * O1_ROW_BYTES);
        uint32_t* leads = reinterpret_cast<uint32_t*>(out + 32);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (v[k] > dust) {
                out[at] = make_uint2(0u - cum, v[k]);
                leads[at] = uint32_t(row_of[lane * 8 + k]) * O1_ROW_BYTES << 8 | (lane * 8 + k);
                ++at;
            }
            cum += v[k];
        }
        if (lane >= used) { out[lane] = make_uint2(0, 0); leads[lane] = 0; }  // width 0: never hit
    }
    if (err) { if (lane == 0) report(status, it.id, err); return; }
    __syncwarp();

    Epilogue ep = make_epilogue(bases, it);
    // Stream words, first byte on top, from the aligned word on that holds the first byte; zero past the end.  Word i lies in
    // words[i mod 128]; the half that holds the current word and the next half are there, the one after that is on its way.
    const uintptr_t src = reinterpret_cast<uintptr_t>(rd(bases, it.src)), src_end = src + it.src_len, src_word = src & ~uintptr_t(3);
    auto fetch = [&](uint64_t i) -> uint32_t {
        const uintptr_t q = src_word + 4 * i;
        if (q >= src && q + 4 <= src_end) return __byte_perm(__ldg(reinterpret_cast<const uint32_t*>(q)), 0, 0x0123);
        uint32_t w = 0;
        for (uint32_t k = 0; k < 4; ++k) if (q + k >= src && q + k < src_end) w |= uint32_t(__ldg(reinterpret_cast<const uint8_t*>(q + k))) << (24 - 8 * k);
        return w;
    };
    for (uint32_t i = lane; i < 2 * O1_HALF; i += 32) words[i] = fetch(i);
    uint32_t coming[2] = {fetch(2 * O1_HALF + lane), fetch(2 * O1_HALF + 32 + lane)};
    __syncwarp();
    uint64_t bit = 8 * (src & 3) + 8;  // range_coder.rs:137-155: five bytes start the code register, of which the last four count
    auto word = [&](uint32_t k) { return words[(uint32_t(bit >> 5) + k) & (2 * O1_HALF - 1)]; };
    auto advance = [&](uint32_t bits) {  // at most 128
        const uint64_t half = bit / (32 * O1_HALF);
        bit += bits;
        if (bit / (32 * O1_HALF) != half) {
            __syncwarp();
            words[(half & 1) * O1_HALF + lane] = coming[0];
            words[(half & 1) * O1_HALF + 32 + lane] = coming[1];
            __syncwarp();
            coming[0] = fetch((half + 3) * O1_HALF + lane);
            coming[1] = fetch((half + 3) * O1_HALF + 32 + lane);
        }
    };
    uint32_t offset = __funnelshift_l(word(1), word(0), uint32_t(bit));  // code - low
    advance(32);
    uint32_t rpt = 0xFFFFFFFFu >> 12, row = 0;  // range / 4096; the context's row, in bytes
    const uint32_t row_len = it.row_len ? it.row_len : (it.n ? it.n : 1);
    uint32_t left_in_row = row_len;
    uint32_t rows_at = uint32_t(__cvta_generic_to_shared(smem));
    asm volatile("" : "+r"(rows_at) : : "memory");  // the rows are complete, and what reads them names no memory (rans_pair_at)
    const uint32_t shares = rows_at + lane * 8, leads_at = rows_at + 256 + lane * 4;
    struct Share { uint32_t below, width, lead; };  // a lane's share of the row
    // One symbol, by the 32 shares; rpt is 0 if none of them has it (and stays 0 if it was).  Returns the next row << 8 | symbol; `took` gets
    // the bits taken in its low byte, which is also what a shift takes of it, and `mine` becomes the share of the next row.
    auto load_share = [&]() -> Share {
        Share v;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.below), "=r"(v.width) : "r"(shares + row));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v.lead) : "r"(leads_at + row));
        return v;
    };
    auto most = [](uint32_t v) -> uint32_t { uint32_t r; asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v)); return r; };
    auto by_share = [&](Share& mine, uint32_t window, uint32_t& took) -> uint32_t {
        // "cumulative count <= offset / rpt < count + width" without the division; the products fit 32 bits
        const uint32_t rest = offset + mine.below * rpt, range = mine.width * rpt;
        const bool won = rest < range;
        const uint32_t got = most(won ? mine.lead : 0u);
        const uint32_t b = range < (1u << 16) ? 16u : range < (1u << 24) ? 8u : 0u;  // rpt >= 2^12: two bytes at most
        const uint32_t next = won ? (range << b >> 4 & ~0xFFu) | b : 0u, low = won ? __funnelshift_l(window, rest, b) : 0u;
        row = got >> 8;
        mine = load_share();
        took = most(next);
        offset = most(low);
        rpt = took >> 8;
        return got;
    };
    auto one_symbol = [&]() -> uint32_t {
        const uint32_t was = offset, per = rpt, from = row, window = __funnelshift_l(word(1), word(0), uint32_t(bit));
        Share mine = load_share();
        uint32_t bits, sy = by_share(mine, window, bits) & 0xFFu;
        bits &= 0xFFu;
        if (rpt == 0) {
            // among all 256: the largest index whose count is <= min(offset / rpt, 4095) (order1_scale_ac.rs:474-486)
            uint32_t v[8], c = load_row(from / O1_ROW_BYTES, v), fit = 0, below = 0, w = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (c * per <= was) { ++fit; below = c; w = v[k]; }
                c += v[k];
            }
            sy = __reduce_add_sync(0xFFFFFFFFu, fit) - 1;  // entry 0 counts 0 and always fits
            const uint32_t range = __shfl_sync(0xFFFFFFFFu, w, sy >> 3) * per;
            bits = range < (1u << 16) ? 16u : range < (1u << 24) ? 8u : 0u;
            offset = __funnelshift_l(window, was - __shfl_sync(0xFFFFFFFFu, below, sy >> 3) * per, bits);
            rpt = (range << bits) >> 12;
            row = uint32_t(row_of[sy]) * O1_ROW_BYTES;
        }
        advance(bits);
        if (--left_in_row == 0) { row = 0; left_in_row = row_len; }  // a row's first symbol has no context
        return sy;
    };
    uint64_t pos = 0;
    uint32_t remaining = it.n, g = remaining ? first_group(ep, pos, remaining) : 0;
    while (remaining) {
        uint32_t s_lo = 0, s_hi = 0;
        bool done = false;
        if (g == 8 && left_in_row > 8) {
            const uint32_t offset0 = offset, rpt0 = rpt, row0 = row;
            // the next 64 bits are enough for four symbols: three before the last one take 48 and it needs 16 to go on
            const uint32_t w0 = word(0), w1 = word(1), w2 = word(2), w3 = word(3), w4 = word(4), at = uint32_t(bit) & 31;
            uint32_t hi = __funnelshift_l(w1, w0, at), lo = __funnelshift_l(w2, w1, at), used = 0;
            Share mine = load_share();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j == 4) {
                    const uint32_t to = at + (used & 0xFFu);
                    const bool one = to >= 32, two = to >= 64;
                    const uint32_t a = two ? w2 : one ? w1 : w0, b = two ? w3 : one ? w2 : w1, c = two ? w4 : one ? w3 : w2;
                    hi = __funnelshift_l(b, a, to); lo = __funnelshift_l(c, b, to);
                }
                uint32_t took;
                const uint32_t got = by_share(mine, hi, took), ins = (0x3210u & ~(0xFu << (4 * (j & 3)))) | (4u << (4 * (j & 3)));
                if (j < 4) s_lo = __byte_perm(s_lo, got, ins); else s_hi = __byte_perm(s_hi, got, ins);
                hi = __funnelshift_l(lo, hi, took); lo = __funnelshift_l(0u, lo, took);
                used += took;  // the low byte is the sum of the low bytes: 128 at most
            }
            used &= 0xFFu;
            done = rpt != 0;
            if (done) { advance(used); left_in_row -= 8; }
            else { offset = offset0; rpt = rpt0; row = row0; s_lo = s_hi = 0; }
        }
        if (!done) {
#pragma unroll 1
            for (uint32_t j = 0; j < g; ++j) {
                const uint32_t sy = one_symbol();
                if (j < 4) s_lo |= sy << (8 * j); else s_hi |= sy << (8 * (j - 4));
            }
        }
        if (lane == 0) emit(ep, pos, g, uint64_t(s_lo) | uint64_t(s_hi) << 32);
        pos += g; remaining -= g;
        g = remaining < 8 ? remaining : 8;
    }
}

constexpr uint32_t O1_MAX_ROWS = 257;
// The chain of a chunk is what a plan with block scales waits for, and it is a third longer with other decoders' warps on its scheduler.  So
// where the plan says so (`alone`) four chunks go to a block, one to a scheduler, that takes an SM's shared memory whole, on half of the
// SMs at most; the other decoders have the rest, and are let go a moment later (head_start_kernel): with a block on every SM
// first they would keep these waiting, which nothing but the time rules out.  The MXFP4 / NVFP4 layer, 280 chunks of 32 Ki scales: 2796 -> 2180 us.
constexpr uint32_t O1_ALONE_CHUNKS = 4 * 74, O1_ALONE_BYTES = 220 * 1024;
// `tables` = the most context rows among the items.
inline bool o1sac_alone(uint32_t n, uint32_t tables) { return n <= O1_ALONE_CHUNKS && 4 * (tables < O1_MAX_ROWS ? tables : O1_MAX_ROWS) * O1_ROW_BYTES <= O1_ALONE_BYTES; }
inline void o1sac_launch(const DecodeItem* items, uint32_t n, const Bases& bases, uint32_t* status, uint32_t tables, bool alone, cudaStream_t st) {
    const uint32_t rows = tables < O1_MAX_ROWS ? tables : O1_MAX_ROWS;
    if (alone && o1sac_alone(n, tables)) o1sac_decode_kernel<4><<<(n + 3) / 4, 128, O1_ALONE_BYTES, st>>>(items, n, bases, status, rows);
    else o1sac_decode_kernel<1><<<n, 32, rows * O1_ROW_BYTES, st>>>(items, n, bases, status, rows);
}
// A few microseconds on the stream whose event the other decoders wait for.
__global__ void head_start_kernel() {
    const long long from = clock64();
    while (clock64() - from < 8000) {}
}
inline cudaError_t o1sac_allow_shared_rows() {
    cudaError_t e = cudaFuncSetAttribute(o1sac_decode_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(O1_ALONE_BYTES));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(o1sac_decode_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(O1_MAX_ROWS * O1_ROW_BYTES));
    return e != cudaSuccess ? e : cudaFuncSetAttribute(o1sac_decode_kernel<1>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

// ---- stand-alone merge / copy ---------------------------------------------
constexpr uint32_t MERGE_TILE = 32768;  // elements per CTA: one chunk of the default size, so the search for the item is paid once per chunk
__global__ void __launch_bounds__(256) merge_kernel(const MergeItem* __restrict__ items, const uint32_t* __restrict__ tile_first, uint32_t n_items, Bases bases) {
    // tile_first[i] = first tile index of item i (n_items + 1 entries); find the item by binary search
    uint32_t tile = blockIdx.x;
    uint32_t lo = 0, hi = n_items;
    while (lo + 1 < hi) { uint32_t mid = (lo + hi) >> 1; if (tile_first[mid] <= tile) lo = mid; else hi = mid; }
    const MergeItem it = items[lo];
    uint64_t base = uint64_t(tile - tile_first[lo]) * MERGE_TILE;
    uint32_t n = it.n - base < MERGE_TILE ? uint32_t(it.n - base) : MERGE_TILE;
    int np = kind_planes(int(it.kind));
    const uint8_t* src[4];
    for (int p = 0; p < 4; ++p) src[p] = p < np ? rd(bases, it.src[p]) + base : nullptr;
    uint8_t* dst = wr(bases, it.dst) + base * uint64_t(kind_elem_bytes(int(it.kind)));
    // Sixteen elements per thread where the destination allows it: 16 bytes of every plane (two aligned 16-byte loads,
    // shifted into place; a block that is not wholly inside the plane is read bytewise) and 16 x element size bytes out,
    // on a boundary of that size.  The elements before the first such boundary and after the last go in groups of eight.
    const uint32_t eb = uint32_t(kind_elem_bytes(int(it.kind)));
    const uintptr_t a = reinterpret_cast<uintptr_t>(dst) / eb;
    uint32_t head = uint32_t((16 - (a & 15)) & 15);
    if (head > n) head = n;
    const uint32_t full = (n - head) >> 4, tail_at = head + full * 16;
    auto slow = [&](uint32_t begin, uint32_t end) {  // fewer than 16 elements: at most two groups
        const uint32_t pos = begin + 8 * threadIdx.x;
        if (pos >= end) return;
        const uint32_t count = end - pos < 8 ? end - pos : 8;
        uint64_t b[4] = {0, 0, 0, 0};
        for (int p = 0; p < np; ++p) b[p] = ld_bytes(src[p] + pos, count);
        compose_store(int(it.kind), dst, pos, count, b);
    };
    slow(0, head);
    slow(tail_at, n);
    uintptr_t p_lo[4] = {0, 0, 0, 0}, p_hi[4] = {0, 0, 0, 0};
    for (int p = 0; p < np; ++p) { p_lo[p] = reinterpret_cast<uintptr_t>(rd(bases, it.src[p])); p_hi[p] = p_lo[p] + it.n; }
    for (uint32_t g = threadIdx.x; g < full; g += blockDim.x) {
        const uint32_t pos = head + g * 16;
        uint32_t pw[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            if (p >= np) break;
            const uintptr_t at = reinterpret_cast<uintptr_t>(src[p]) + pos, q = at & ~uintptr_t(15);
            const uint4 cur = load_block16_guarded(q, p_lo[p], p_hi[p]);
            const uint32_t off = uint32_t(at & 15);
            if (off) { const uint4 nxt = load_block16_guarded(q + 16, p_lo[p], p_hi[p]); extract16(cur, nxt, off, pw[p]); }
            else { pw[p][0] = cur.x; pw[p][1] = cur.y; pw[p][2] = cur.z; pw[p][3] = cur.w; }
        }
        merge_store16(int(it.kind), dst + size_t(pos) * eb, pw);
    }
}

// ---- per-plane ops between the split and a terminal, undone in scratch -------
// A CTA of 256 threads owns one tile of POST_TILE bytes; thread t owns the 64
// bytes from 64 t on.  Tiles of all items are numbered through `tile_first`
// like the merge tiles.  IntDelta (transforms/int_delta.rs:36-44, byte width)
// takes three launches: the byte sum of every tile, an exclusive scan of the
// sums per plane, then the running sum inside every tile started from the
// tile's carry.  All arithmetic is modulo 256 per byte (__vadd4).
struct PostTile { PostItem it; uint64_t base; uint32_t n; uint32_t local; };
__device__ __forceinline__ PostTile post_tile_of(const PostItem* items, const uint32_t* tile_first, uint32_t n_items) {
    uint32_t tile = blockIdx.x, lo = 0, hi = n_items;
    while (lo + 1 < hi) { uint32_t mid = (lo + hi) >> 1; if (tile_first[mid] <= tile) lo = mid; else hi = mid; }
    PostTile t;
    t.it = items[lo];
    t.local = tile - tile_first[lo];
    t.base = uint64_t(t.local) * POST_TILE;
    t.n = t.it.n - t.base < POST_TILE ? uint32_t(t.it.n - t.base) : POST_TILE;
    return t;
}
// The thread's 64 bytes as sixteen words, zero beyond the plane's end.  The plane starts on a 256-byte boundary of the scratch arena.
__device__ __forceinline__ void post_load64(const uint8_t* tile, uint32_t n, uint32_t w[16]) {
    const uint32_t at = threadIdx.x * 64;
    if (at + 64 <= n) {
#pragma unroll
        for (int q = 0; q < 4; ++q) { uint4 v = *reinterpret_cast<const uint4*>(tile + at + 16 * q); w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w; }
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            uint32_t v = 0;
            for (int i = 0; i < 4; ++i) if (at + 4 * k + i < n) v |= uint32_t(tile[at + 4 * k + i]) << (8 * i);
            w[k] = v;
        }
    }
}
__device__ __forceinline__ void post_store64(uint8_t* tile, uint32_t n, const uint32_t w[16]) {
    const uint32_t at = threadIdx.x * 64;
    if (at + 64 <= n) {
#pragma unroll
        for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(tile + at + 16 * q) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    } else {
        for (int k = 0; k < 16; ++k) for (int i = 0; i < 4; ++i) if (at + 4 * k + i < n) tile[at + 4 * k + i] = uint8_t(w[k] >> (8 * i));
    }
}
// Sum over the block of one byte-sized value per thread; with `exclusive`, every thread gets the sum of the threads before it.
__device__ __forceinline__ uint32_t post_block_sum(uint32_t v, uint32_t* exclusive) {
    __shared__ uint32_t warp_total[8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d); if (lane >= d) incl += t; }
    __syncthreads();  // the array may still be read from an earlier call
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) { if (k < int(warp)) before += warp_total[k]; total += warp_total[k]; }
    if (exclusive) *exclusive = (before + incl - v) & 0xFFu;
    return total & 0xFFu;
}
__global__ void __launch_bounds__(256) post_tile_sums_kernel(const PostItem* __restrict__ items, const uint32_t* __restrict__ tile_first, uint32_t n_items, Bases bases) {
    const PostTile t = post_tile_of(items, tile_first, n_items);
    if (t.it.op != POST_INTDELTA) return;
    uint32_t w[16], acc = 0;
    post_load64(wr(bases, t.it.plane) + t.base, t.n, w);
#pragma unroll
    for (int k = 0; k < 16; ++k) acc = __vadd4(acc, w[k]);
    acc = (acc + (acc >> 8) + (acc >> 16) + (acc >> 24)) & 0xFFu;
    const uint32_t total = post_block_sum(acc, nullptr);
    if (threadIdx.x == 0) reinterpret_cast<uint32_t*>(wr(bases, t.it.sums))[t.local] = total;
}
// One CTA per plane: the tile sums become the sum of all tiles before each.
__global__ void __launch_bounds__(256) post_scan_sums_kernel(const PostItem* __restrict__ items, uint32_t n_items, Bases bases) {
    const PostItem it = items[blockIdx.x];
    if (it.op != POST_INTDELTA) return;
    uint32_t* sums = reinterpret_cast<uint32_t*>(wr(bases, it.sums));
    const uint64_t tiles = (it.n + POST_TILE - 1) / POST_TILE;
    uint32_t carry = 0;
    for (uint64_t first = 0; first < tiles; first += 256) {
        const uint64_t i = first + threadIdx.x;
        const uint32_t v = i < tiles ? sums[i] : 0u;
        uint32_t excl;
        const uint32_t total = post_block_sum(v, &excl);
        if (i < tiles) sums[i] = (carry + excl) & 0xFFu;
        carry = (carry + total) & 0xFFu;
    }
}
__global__ void __launch_bounds__(256) post_apply_kernel(const PostItem* __restrict__ items, const uint32_t* __restrict__ tile_first, uint32_t n_items, Bases bases) {
    const PostTile t = post_tile_of(items, tile_first, n_items);
    uint8_t* tile = wr(bases, t.it.plane) + t.base;
    uint32_t w[16];
    post_load64(tile, t.n, w);
    if (t.it.op == POST_MZS) {  // transforms/mantissa_zero.rs: inverse shifts every byte left by k
        const uint32_t keep = 0x01010101u * (0xFFu >> t.it.k);
#pragma unroll
        for (int k = 0; k < 16; ++k) w[k] = (w[k] & keep) << t.it.k;
    } else if (t.it.op == POST_INTDELTA) {
        uint32_t run = 0;  // sum of the thread's earlier words, in every byte
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            uint32_t v = w[k];
            v = __vadd4(v, v << 8);
            v = __vadd4(v, v << 16);  // running sum inside the word
            v = __vadd4(v, run);
            run = (v >> 24) * 0x01010101u;
            w[k] = v;
        }
        uint32_t excl;
        post_block_sum(run & 0xFFu, &excl);
        const uint32_t carry = ((reinterpret_cast<const uint32_t*>(rd(bases, t.it.sums))[t.local] + excl) & 0xFFu) * 0x01010101u;
#pragma unroll
        for (int k = 0; k < 16; ++k) w[k] = __vadd4(w[k], carry);
    }
    post_store64(tile, t.n, w);
}

// ---- integrity -------------------------------------------------------------
// CRC-32/IEEE in the reflected form (poly 0xEDB88320).  Each thread takes the
// remainder of one run of plane bytes from state 0, multiplies it by
// x^(8*bytes_after) mod P and XORs it into the plane's accumulator; the host
// adds the init/final terms, which depend only on the plane length.
__host__ __device__ __forceinline__ uint32_t gf2_mulmod(uint32_t a, uint32_t b) {
    uint32_t p = 0;
    for (uint32_t m = 1u << 31; m; m >>= 1) {
        if (a & m) p ^= b;
        b = (b & 1) ? (b >> 1) ^ 0xEDB88320u : b >> 1;
    }
    return p;
}
struct CrcTables { uint32_t byte_table[256]; uint32_t x2n[64]; };  // x2n[k] = x^(2^k) mod P

__host__ __device__ __forceinline__ uint32_t x_pow_8n(const uint32_t* x2n, uint64_t nbytes) {
    uint32_t p = 1u << 31;  // x^0
    uint32_t k = 3;         // x^(8n) = x^(n * 2^3)
    while (nbytes) { if (nbytes & 1) p = gf2_mulmod(x2n[k & 63], p); nbytes >>= 1; ++k; }
    return p;
}

// Plane bytes of one element (byte p = plane p) as their terminals hold them: the forward direction of the per-plane
// ops, from this element's and the previous element's plane bytes.
__device__ __forceinline__ uint32_t terminal_bytes(uint32_t cur, uint32_t prev, uint32_t post, uint32_t post_k, int planes) {
    uint32_t r = 0;
    for (int p = 0; p < planes; ++p) {
        const uint32_t op = (post >> (8 * p)) & 0xFFu, k = (post_k >> (8 * p)) & 0xFFu;
        uint32_t b = (cur >> (8 * p)) & 0xFFu;
        if (op == POST_INTDELTA) b = (b - ((prev >> (8 * p)) & 0xFFu)) & 0xFFu;
        else if (op == POST_MZS) b >>= k;
        r |= b << (8 * p);
    }
    return r;
}

// The byte table is kept 32 times over in shared memory, entry i of lane l at word 32 i + l: a lookup never leaves
// the lane's own bank, whatever the 32 indices of a warp are (one shared copy took 2.15 passes per lookup).  Tensor
// bytes are read 16 at a time; a thread walks its own run, so every wider load saves that many single-sector requests.
__global__ void __launch_bounds__(128) crc_planes_kernel(const VerifyTensor* __restrict__ tensors, uint32_t n_tensors, uint64_t n_runs, Bases bases,
                                                         const CrcTables* __restrict__ tabs, uint32_t* __restrict__ acc) {
    __shared__ uint32_t T32[256 * 32];
    __shared__ uint32_t X[64];
    for (uint32_t i = threadIdx.x; i < 256 * 32; i += blockDim.x) T32[i] = tabs->byte_table[i >> 5];
    if (threadIdx.x < 64) X[threadIdx.x] = tabs->x2n[threadIdx.x];
    __syncthreads();
    uint64_t run = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (run >= n_runs) return;
    const uint32_t* T = T32 + (threadIdx.x & 31);
    auto step = [&](uint32_t crc, uint32_t byte) { return T[((crc ^ byte) & 0xFFu) << 5] ^ (crc >> 8); };
    uint32_t lo = 0, hi = n_tensors;
    while (lo + 1 < hi) { uint32_t mid = (lo + hi) >> 1; if (tensors[mid].first_run <= run) lo = mid; else hi = mid; }
    const VerifyTensor t = tensors[lo];
    uint64_t first = (run - t.first_run) * VERIFY_RUN;
    uint32_t n = t.n_elems - first < VERIFY_RUN ? uint32_t(t.n_elems - first) : VERIFY_RUN;
    const uint8_t* out = rd(bases, t.out);
    uint32_t c[4] = {0, 0, 0, 0};
    const bool wide = !t.post && (reinterpret_cast<uintptr_t>(out + first * uint64_t(kind_elem_bytes(int(t.kind)))) & 15) == 0;
    switch (t.kind) {
        case K_PASS: {
            uint32_t i = 0;
            if (wide) {
                const uint4* q = reinterpret_cast<const uint4*>(out + first);
                uint4 ahead = i + 16 <= n ? __ldg(q) : make_uint4(0, 0, 0, 0);  // the next block is on its way while this one is folded in
                for (; i + 16 <= n; i += 16) {
                    const uint4 v = ahead;
                    ++q;
                    if (i + 2 * 16 <= n) ahead = __ldg(q);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 16; ++k) c[0] = step(c[0], w[k >> 2] >> (8 * (k & 3)));
                }
            }
            for (; i < n; ++i) c[0] = step(c[0], out[first + i]);
            break;
        }
        case K_M16: {
            auto planes_of = [&](uint64_t e) {
                uint32_t v = uint32_t(out[2 * e]) | uint32_t(out[2 * e + 1]) << 8;
                return ((v << 1) & 0xFF00u) | ((v >> 8) & 0x0080u) | (v & 0x007Fu);
            };
            uint32_t i = 0;
            if (wide) {
                const uint4* q = reinterpret_cast<const uint4*>(out + first * 2);
                uint4 ahead = i + 8 <= n ? __ldg(q) : make_uint4(0, 0, 0, 0);  // the next block is on its way while this one is folded in
                for (; i + 8 <= n; i += 8) {
                    const uint4 v = ahead;
                    ++q;
                    if (i + 2 * 8 <= n) ahead = __ldg(q);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {  // two elements per word: the forward reorder of split/dtype16.rs:11-18 on both halves
                        const uint32_t r = ((w[k] << 1) & 0xFF00FF00u) | ((w[k] >> 8) & 0x00800080u) | (w[k] & 0x007F007Fu);
                        c[0] = step(c[0], r); c[1] = step(c[1], r >> 8);
                        c[0] = step(c[0], r >> 16); c[1] = step(c[1], r >> 24);
                    }
                }
            }
            uint32_t prev = (t.post && first) ? planes_of(first - 1) : 0u;
            for (; i < n; ++i) {
                uint32_t r = planes_of(first + i);
                if (t.post) { uint32_t cur = r; r = terminal_bytes(r, prev, t.post, t.post_k, 2); prev = cur; }
                c[0] = step(c[0], r);
                c[1] = step(c[1], r >> 8);
            }
            break;
        }
        case K_M32: {
            auto reorder = [](uint32_t v) { return ((v << 1) & 0xFF000000u) | ((v >> 8) & 0x00800000u) | (v & 0x007FFFFFu); };
            auto planes_of = [&](uint64_t e) { return reorder(ld_u32_unaligned(out + 4 * e)); };
            uint32_t i = 0;
            if (wide) {
                const uint4* q = reinterpret_cast<const uint4*>(out + first * 4);
                uint4 ahead = i + 4 <= n ? __ldg(q) : make_uint4(0, 0, 0, 0);  // the next block is on its way while this one is folded in
                for (; i + 4 <= n; i += 4) {
                    const uint4 v = ahead;
                    ++q;
                    if (i + 2 * 4 <= n) ahead = __ldg(q);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t r = reorder(w[k]);
#pragma unroll
                        for (int p = 0; p < 4; ++p) c[p] = step(c[p], r >> (8 * p));
                    }
                }
            }
            uint32_t prev = (t.post && first) ? planes_of(first - 1) : 0u;
            for (; i < n; ++i) {
                uint32_t r = planes_of(first + i);
                if (t.post) { uint32_t cur = r; r = terminal_bytes(r, prev, t.post, t.post_k, 4); prev = cur; }
#pragma unroll
                for (int p = 0; p < 4; ++p) c[p] = step(c[p], r >> (8 * p));
            }
            break;
        }
        default: {
            auto nibbles = [&](uint32_t v) { return t.kind == K_E4M3 ? (((v & 0x78) << 1) | ((v & 0x80) >> 4) | (v & 0x07)) : (((v & 0x7C) << 1) | ((v & 0x80) >> 5) | (v & 0x03)); };
            uint32_t i = 0;
            if (wide) {
                const uint4* q = reinterpret_cast<const uint4*>(out + first);
                uint4 ahead = i + 16 <= n ? __ldg(q) : make_uint4(0, 0, 0, 0);  // the next block is on its way while this one is folded in
                for (; i + 16 <= n; i += 16) {
                    const uint4 v = ahead;
                    ++q;
                    if (i + 2 * 16 <= n) ahead = __ldg(q);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const uint32_t r = nibbles((w[k >> 2] >> (8 * (k & 3))) & 0xFFu);
                        c[0] = step(c[0], r >> 4); c[1] = step(c[1], r & 0x0F);
                    }
                }
            }
            for (; i < n; ++i) {
                const uint32_t r = nibbles(out[first + i]);
                c[0] = step(c[0], r >> 4);
                c[1] = step(c[1], r & 0x0F);
            }
            break;
        }
    }
    uint32_t shift = x_pow_8n(X, t.n_elems - first - n);
    int np = kind_planes(int(t.kind));
    for (int p = 0; p < np; ++p) atomicXor(&acc[t.acc_base + p], gf2_mulmod(shift, c[p]));
}

// XXH64 (seed 0) of each tensor.  The hash is sequential by design: four accumulators, each fed one 8-byte word of every
// 32-byte stripe through add, rotate and a 64-bit multiply, so four lanes carry the state and a tensor cannot go faster
// than that dependent chain allows.  Tensors hash concurrently, one per block, and the host lists the largest first: the
// longest tensor is the critical path.  Two warps per block: lanes 0-3 of the first work through the stripes of one block of
// words in shared memory and do nothing else; the second warp meanwhile brings the next block from memory and multiplies its
// words by the second prime.  A step adds the next word's product with the multiply of the low halves: its low word and carry
// first, then the high word on top of the cross products, which it can take late.  20 cycles per stripe; 23 with a widening multiply
// that adds both words at once (its high word takes 16), 24 to 38 with the high word, the carry or the cross products joined by adds of
// their own, 27 with the add in front of the rotation.  59 MB, the largest tensor of a fp32 model: 28.2 ms with one warp that did all of
// it, 22.4 with the widening multiply, 19.5 now.
__device__ __forceinline__ uint64_t rotl64(uint64_t x, int r) { return (x << r) | (x >> (64 - r)); }
__device__ __forceinline__ uint64_t ld_u64_unaligned(const uint8_t* p) { return uint64_t(ld_u32_unaligned(p)) | uint64_t(ld_u32_unaligned(p + 4)) << 32; }
constexpr uint32_t XXH_BLOCK = 8192, XXH_THREADS = 64;
// rotl64(s, 31) * P1 + k
__device__ __forceinline__ uint64_t xxh_step(uint64_t s, uint64_t k) {
    constexpr uint64_t P1 = 11400714785074694791ull;
    const uint32_t a = uint32_t(s), b = uint32_t(s >> 32);
    const uint32_t lo = __funnelshift_l(b, a, 31), hi = __funnelshift_l(a, b, 31);
    uint32_t l, h;
    asm("{\n\t.reg .u32 u;\n\tmad.lo.u32 u, %3, %5, %7;\n\tmad.lo.u32 u, %2, %4, u;\n\tmad.lo.cc.u32 %0, %2, %5, %6;\n\tmadc.hi.u32 %1, %2, %5, u;\n\t}"
        : "=&r"(l), "=&r"(h) : "r"(lo), "r"(hi), "r"(uint32_t(P1 >> 32)), "r"(uint32_t(P1)), "r"(uint32_t(k)), "r"(uint32_t(k >> 32)));
    return uint64_t(h) << 32 | l;
}

__global__ void __launch_bounds__(XXH_THREADS) xxh64_kernel(const HashItem* __restrict__ items, uint32_t n_items, Bases bases, uint64_t* __restrict__ out) {
    const uint64_t P1 = 11400714785074694791ull, P2 = 14029467366897019727ull, P3 = 1609587929392839161ull, P4 = 9650029242287828579ull,
                   P5 = 2870177450012600261ull;
    __shared__ __align__(16) uint64_t stage[2][XXH_BLOCK / 8];
    const uint32_t lane = threadIdx.x & 31, idx = blockIdx.x;
    const bool feeds = threadIdx.x >= 32;
    if (idx >= n_items) return;
    const HashItem it = items[idx];
    const uint8_t* p = rd(bases, it.data);
    const uint64_t len = it.len, stripes = len / 32;
    const uint64_t blocks = (stripes * 32 + XXH_BLOCK - 1) / XXH_BLOCK;
    const bool aligned = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
    constexpr int PAIRS = XXH_BLOCK / 16 / 32;  // pairs of words per lane and block
    uint4 nxt[PAIRS];
    auto fetch = [&](uint64_t b) {  // block b; zero behind the last whole stripe
        const uint64_t first = b * (XXH_BLOCK / 16) + lane, end = stripes * 2;
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
            const uint64_t at = first + 32 * k;
            nxt[k] = make_uint4(0, 0, 0, 0);
            if (at >= end) continue;
            if (aligned) nxt[k] = __ldg(reinterpret_cast<const uint4*>(p) + at);
            else {
                const uint64_t x = ld8_unaligned(p + 16 * at), y = ld8_unaligned(p + 16 * at + 8);
                nxt[k] = make_uint4(uint32_t(x), uint32_t(x >> 32), uint32_t(y), uint32_t(y >> 32));
            }
        }
    };
    auto store = [&](uint64_t b) {
        uint64_t* w = stage[b & 1];
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
            const uint4 v = nxt[k];
            const uint64_t x = (uint64_t(v.y) << 32 | v.x) * P2, y = (uint64_t(v.w) << 32 | v.z) * P2;
            reinterpret_cast<uint4*>(w)[k * 32 + lane] = make_uint4(uint32_t(x), uint32_t(x >> 32), uint32_t(y), uint32_t(y >> 32));
        }
    };
    uint64_t v = lane == 0 ? P1 + P2 : lane == 1 ? P2 : lane == 2 ? 0 : 0 - P1;
    if (feeds && blocks) {
        fetch(0);
        store(0);
        if (blocks > 1) fetch(1);
    }
    for (uint64_t b = 0; b < blocks; ++b) {
        __syncthreads();  // block b is in place, and nobody reads the other buffer any more
        if (feeds) {
            if (b + 1 < blocks) store(b + 1);
            if (b + 2 < blocks) fetch(b + 2);
        } else if (lane < 4) {
            const uint64_t* w = stage[b & 1] + lane;
            const uint64_t left = stripes - b * (XXH_BLOCK / 32);
            v += w[0];
            if (left >= XXH_BLOCK / 32) {
#pragma unroll 16
                for (int st = 1; st < int(XXH_BLOCK / 32); ++st) v = xxh_step(v, w[4 * st]);
            } else {
                for (uint32_t st = 1; st < uint32_t(left); ++st) v = xxh_step(v, w[4 * st]);
            }
            v = xxh_step(v, 0);
        }
    }
    if (feeds) return;
    const uint64_t v1 = __shfl_sync(0xFFFFFFFFu, v, 0), v2 = __shfl_sync(0xFFFFFFFFu, v, 1), v3 = __shfl_sync(0xFFFFFFFFu, v, 2), v4 = __shfl_sync(0xFFFFFFFFu, v, 3);
    if (lane != 0) return;
    auto round = [&](uint64_t acc, uint64_t in) { acc += in * P2; acc = rotl64(acc, 31); return acc * P1; };
    auto merge = [&](uint64_t h, uint64_t x) { x = round(0, x); h ^= x; return h * P1 + P4; };
    uint64_t h;
    if (len >= 32) {
        h = rotl64(v1, 1) + rotl64(v2, 7) + rotl64(v3, 12) + rotl64(v4, 18);
        h = merge(h, v1); h = merge(h, v2); h = merge(h, v3); h = merge(h, v4);
    } else h = P5;
    h += len;
    const uint8_t* q = p + stripes * 32;
    const uint8_t* end = p + len;
    while (q + 8 <= end) { h ^= round(0, ld_u64_unaligned(q)); h = rotl64(h, 27) * P1 + P4; q += 8; }
    if (q + 4 <= end) { h ^= uint64_t(ld_u32_unaligned(q)) * P1; h = rotl64(h, 23) * P2 + P3; q += 4; }
    while (q < end) { h ^= uint64_t(*q) * P5; h = rotl64(h, 11) * P1; ++q; }
    h ^= h >> 33; h *= P2; h ^= h >> 29; h *= P3; h ^= h >> 32;
    out[idx] = h;
}

// Copies 16-byte words; the host side uses it to bring a plan's work lists from pinned host memory to the device
// without queueing behind the copy engine's transfers.
__global__ void __launch_bounds__(256) stage_in_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, size_t n16) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n16; i += size_t(gridDim.x) * blockDim.x) dst[i] = src[i];
}

}  // namespace ptwm
