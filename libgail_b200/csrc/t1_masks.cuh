// Tier-1 on whole columns, shared by the encoder's and the decoder's kernels: a warp holds a
// code-block with a column per lane, every per-sample property of it as a 32-bit mask of the
// column's rows (bit r = row r), and works on all rows at once.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"

namespace gb {

// Per 4-bit group of x, its number of set bits.
__device__ __forceinline__ uint32_t nibbleCounts(uint32_t x) {
    x = x - ((x >> 1) & 0x55555555u);
    return (x & 0x33333333u) + ((x >> 2) & 0x33333333u);
}

// Per stripe s of a row mask, at bit 4s: any of its four rows set.
__device__ __forceinline__ uint32_t nibbleAny(uint32_t m) { return (m | (m >> 1) | (m >> 2) | (m >> 3)) & 0x11111111u; }

// Warp-inclusive prefix sum.
__device__ __forceinline__ uint32_t warpScan(uint32_t v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ __forceinline__ uint32_t shUp(uint32_t v, int lane) {
    const uint32_t t = __shfl_up_sync(kFull, v, 1);
    return lane == 0 ? 0u : t;
}
__device__ __forceinline__ uint32_t shDown(uint32_t v, int lane) {
    const uint32_t t = __shfl_down_sync(kFull, v, 1);
    return lane == 31 ? 0u : t;
}

// Bits j and above of x swapped with the low bits of y, in groups of j (m: the low group):
// the step of a bit-matrix transpose (Warren, Hacker's Delight, 7-3).
__device__ __forceinline__ void swapBits(uint32_t& x, uint32_t& y, int j, uint32_t m) {
    const uint32_t lo = (x & m) | ((y << j) & ~m), hi = ((x >> j) & m) | (y & ~m);
    x = lo;
    y = hi;
}

// 32 words as a bit matrix, transposed: afterwards word p holds bit p of every word, word r's
// at bit r.
__device__ __forceinline__ void transpose32(uint32_t v[32]) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {  // whole halves and bytes move as byte permutations
        const uint32_t x = v[k], y = v[k + 16];
        v[k] = __byte_perm(x, y, 0x5410);
        v[k + 16] = __byte_perm(x, y, 0x7632);
    }
#pragma unroll
    for (int k = 0; k < 32; ++k)
        if (!(k & 8)) {
            const uint32_t x = v[k], y = v[k + 8];
            v[k] = __byte_perm(x, y, 0x6240);
            v[k + 8] = __byte_perm(x, y, 0x7351);
        }
#pragma unroll
    for (int k = 0; k < 32; ++k)
        if (!(k & 4)) swapBits(v[k], v[k + 4], 4, 0x0F0F0F0Fu);
#pragma unroll
    for (int k = 0; k < 32; ++k)
        if (!(k & 2)) swapBits(v[k], v[k + 2], 2, 0x33333333u);
#pragma unroll
    for (int k = 0; k < 32; ++k)
        if (!(k & 1)) swapBits(v[k], v[k + 1], 1, 0x55555555u);
}

// Eight row masks into bytes: afterwards byte i of m[s] holds, for row 4 s + i, mask k's bit
// at bit k. Masks that are the constant 0 cost nothing.
__device__ __forceinline__ void rowBytes(uint32_t m[8]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) swapBits(m[k], m[k + 4], 4, 0x0F0F0F0Fu);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (!(k & 2)) swapBits(m[k], m[k + 2], 2, 0x33333333u);
#pragma unroll
    for (int k = 0; k < 8; k += 2) swapBits(m[k], m[k + 1], 1, 0x55555555u);
    // m[j] byte q is row 8 q + j: the two 4 x 4 byte matrices transposed
    uint32_t t[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t a = m[4 * h], b = m[4 * h + 1], c = m[4 * h + 2], d = m[4 * h + 3];
        const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
        const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
        t[0 + h] = __byte_perm(ab0, cd0, 0x5410);
        t[2 + h] = __byte_perm(ab0, cd0, 0x7632);
        t[4 + h] = __byte_perm(ab1, cd1, 0x5410);
        t[6 + h] = __byte_perm(ab1, cd1, 0x7632);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) m[k] = t[k];
}

// The places of a pass's decisions, stripe by stripe and column by column: from c, a lane's decisions
// per stripe as 4-bit groups (15 at most), the decisions before the lane's in its stripe and the
// stripe's in all columns. Counts are 10-bit fields, three stripes a word.
struct StripePlaces {
    uint32_t x[3], t[3];
    __device__ __forceinline__ StripePlaces(uint32_t c, int lane) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t w = ((c >> (12 * k)) & 0xFu) | (((c >> (12 * k + 4)) & 0xFu) << 10) |
                               (k < 2 ? ((c >> (12 * k + 8)) & 0xFu) << 20 : 0u);
            const uint32_t incl = warpScan(w, lane);
            x[k] = incl - w;
            t[k] = __shfl_sync(kFull, incl, 31);
        }
    }
    __device__ __forceinline__ uint32_t before(int s) const { return (x[s / 3] >> (10 * (s % 3))) & 1023u; }
    __device__ __forceinline__ uint32_t all(int s) const { return (t[s / 3] >> (10 * (s % 3))) & 1023u; }
};

// Bit i of x (x < 16) to bit 0 of byte i, by one multiply: the four shifted copies of x land in
// disjoint bit ranges.
__device__ __forceinline__ uint32_t spread1(uint32_t x) { return (x * 0x00204081u) & 0x01010101u; }

// The significance of every row's eight neighbours as the scan order of one pass sees it.
struct Nbr {
    uint32_t l, lu, ld;  // left column at the row, above and below it
    uint32_t r, ru, rd;  // right column
    uint32_t u, d;       // own column above and below
};

// Zero-coding contexts (Table D.1) of all rows, as the four bits of the context number.
__device__ __forceinline__ void zcMasks(const Nbr& q, int orient, uint32_t& c0, uint32_t& c1, uint32_t& c2, uint32_t& c3) {
    // diagonal neighbours: any, at least two, at least three
    const uint32_t dp = q.lu | q.ld, dq = q.ru | q.rd, dAny = dp | dq;
    const uint32_t d2 = (q.lu & q.ld) | (dp & dq) | (q.ru & q.rd);
    if (orient == 3) {
        const uint32_t d3 = (q.lu & q.ld & dq) | (q.ru & q.rd & dp);
        const uint32_t hp = q.l | q.r, vp = q.u | q.d, hv = hp | vp, hv2 = (q.l & q.r) | (hp & vp) | (q.u & q.d);
        const uint32_t e2 = d2 & ~d3, e1 = dAny & ~d2, e0 = ~dAny;
        c3 = d3;                                                      // 8
        c2 = e2 | (e1 & hv);                                          // 7 6, 5 4
        c1 = e2 | (e1 & ~hv) | (e0 & hv2);                            // 7 6, 3, 2
        c0 = (e2 & hv) | (e1 & (hv2 | ~hv)) | (e0 & hv & ~hv2);       // 7, 5 3, 1
        return;
    }
    // HL swaps the horizontal and the vertical neighbours
    const uint32_t ha = orient == 1 ? q.u : q.l, hb = orient == 1 ? q.d : q.r;
    const uint32_t va = orient == 1 ? q.l : q.u, vb = orient == 1 ? q.r : q.d;
    const uint32_t h0 = ~(ha | hb), h1 = ha ^ hb, v1 = va ^ vb, vAny = va | vb;
    c3 = ha & hb;                                                     // 8
    c2 = h1 | (h0 & va & vb);                                         // 7 6 5, 4
    c1 = (h1 & (vAny | dAny)) | (h0 & (v1 | (~vAny & d2)));           // 7 6, 3, 2
    c0 = (h1 & (vAny | ~dAny)) | (h0 & (v1 | (~vAny & dAny & ~d2)));  // 7 5, 3, 1
}

// Sign-coding contexts (Table D.3) of all rows: the context number is 8 + s2 s1 s0, sb the
// coded bit. sgn, sgnL, sgnR: signs of the own, the left and the right column.
__device__ __forceinline__ void scMasks(const Nbr& q, uint32_t sgn, uint32_t sgnL, uint32_t sgnR, uint32_t& s0,
                                        uint32_t& s1, uint32_t& s2, uint32_t& sb) {
    const uint32_t sU = sgn << 1, sD = sgn >> 1;
    const uint32_t lp = q.l & ~sgnL, ln = q.l & sgnL, rp = q.r & ~sgnR, rn = q.r & sgnR;
    const uint32_t up = q.u & ~sU, un = q.u & sU, dp = q.d & ~sD, dn = q.d & sD;
    const uint32_t hPos = (lp & ~rn) | (rp & ~ln), hNeg = (ln & ~rp) | (rn & ~lp);
    const uint32_t vPos = (up & ~dn) | (dp & ~un), vNeg = (un & ~dp) | (dn & ~up);
    const uint32_t h = hPos | hNeg, v = vPos | vNeg, opp = (hPos & vNeg) | (hNeg & vPos);
    s2 = h & ~opp;       // 13 12
    s1 = opp | (~h & v);  // 11, 10
    s0 = ~(h ^ v);       // 13 11, 9
    sb = sgn ^ (hNeg | (~h & vNeg));
}

}  // namespace gb
