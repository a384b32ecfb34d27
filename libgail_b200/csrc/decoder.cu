// Decoder on sm_100a: Tier-1 decoding with dequantisation, inverse 9/7 wavelet, inverse
// ICT and 12-bit packing.
//
// Tier-1 (decodeKernel): one code-block per warp at a time; up to 24 such warps per SM pull
// blocks from a device queue ordered longest codeword first (orderScatterKernel), the heaviest
// on SMs of their own. All lanes run the MQ decoder in step, each also holding one column of
// the block as row masks (t1_masks.cuh): the decoder's serial chain takes one lane's time, and
// the contexts, the refinement pass's list, the bit-planes and the dequantisation are done for
// all columns at once. Untrusted input: bytes past the codeword read as 0xFF, a block whose
// bytes lie outside the codestream decodes as zero, and nothing outside the block's own
// samples is written.
//
// Inverse wavelet (invLevelKernel): per level, 64 x 64 output tiles with a 4-sample halo
// in the interleaved domain, rows then columns (the reference's order), a thread per line,
// whole-sample symmetric mirror at the edges. The last level carries the inverse ICT, the rounding
// and clamping to 12 bits and the interleaved 16-bit store.
//
// Semantics restated from Josephur/libgail core/t1_dec.cpp:45-179,
// kernels/mq_decoder.h:46-114, core/cpu_decode_backend.cpp:36-99 and
// core/dwt_cpu.cpp:96-133, 213-240; bit-identical to the CPU decoder.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <stdexcept>
#include <string>

#include "common.cuh"
#include "decoder.h"
#include "pool.h"
#include "t1_masks.cuh"
#include "t1_tables.h"
#include "tuning.h"

namespace gb {

namespace {

// One code-block per warp: the decode of a block is a serial chain whose control flow depends
// on every decoded bit, so lanes of one warp decoding different blocks would run one after
// another.
constexpr int DEC_THREADS = 32;
constexpr int DEC_CTAS = 24;  // resident warps per SM the registers must allow
constexpr int ORDER_BUCKETS = 128;

__constant__ uint8_t c_sc[9];
__constant__ uint32_t c_mq[47];

// Heavy blocks: the longest codewords, decoded on SMs of their own (at most four per SM, one
// per scheduler) instead of beside 23 other decoding warps, where a block of a thousand
// bytes or more takes the whole launch's time.
constexpr uint32_t kMaxReserveSms = 32;
constexpr uint32_t kMaxHeavy = 4 * kMaxReserveSms;
// Control words: [0] queue head, [1] status, [2] wanted blocks, [3] blocks above the heavy
// limit, [4] the wanted blocks' codeword bytes; from kCtlArrive a counter per reserved SM, from
// kCtlClaim a claim flag per heavy block, from kCtlHist the order's bucket counts, from
// kCtlCursor the places taken in them.
constexpr uint32_t kCtlWanted = 2, kCtlHeavy = 3;
constexpr uint32_t kCtlArrive = 16, kCtlClaim = kCtlArrive + kMaxReserveSms;
constexpr uint32_t kCtlHist = kCtlClaim + kMaxHeavy, kCtlCursor = kCtlHist + ORDER_BUCKETS;
constexpr uint32_t kCtlWords = kCtlCursor + ORDER_BUCKETS;

struct DecArgs {
    const uint8_t* bytes;
    uint64_t size;
    const GbCblkCode* codes;
    const DecBlock* blocks;
    uint32_t n;
    const float* half;  // per band: step / 2
    uint32_t* planes;   // float planes seen as words while decoding
    uint32_t W;
    uint32_t* perm;
    uint32_t* ctl;      // kCtlWords control words, zeroed before the launch
    uint32_t slots;     // the decode launch's warps that are resident together
    uint32_t heavyPct;  // heavy: codeword bytes above heavyPct % of the mean per such warp (0: none)
};

__device__ __forceinline__ uint32_t lenBucket(uint32_t len) {
    if (len < 4) return ORDER_BUCKETS - 1;
    const uint32_t l = 31 - __clz(len);
    return ORDER_BUCKETS - 1 - min(4 * l + ((len >> (l - 2)) & 3u), (uint32_t)ORDER_BUCKETS - 1);
}

// The order, largest codeword first in log-spaced classes, over the whole GPU (a single CTA took
// 58 us for a 4K frame's 25,986 blocks on a B200): per-CTA histograms and byte sums into the control
// words; then every CTA scans the histogram for itself and places its blocks 256 at a time, one
// atomic per bucket and CTA for their places.
__global__ void __launch_bounds__(256) orderCountKernel(DecArgs a) {
    __shared__ uint32_t hist[ORDER_BUCKETS], total, bytes;
    for (int i = threadIdx.x; i < ORDER_BUCKETS; i += blockDim.x) hist[i] = 0;
    if (threadIdx.x == 0) total = bytes = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x)
        if (a.blocks[i].wanted) {
            const uint32_t len = a.codes[i].len;
            atomicAdd(&hist[lenBucket(len)], 1u);
            atomicAdd(&total, 1u);
            atomicAdd(&bytes, min(len, 1u << 20));
        }
    __syncthreads();
    for (int b = threadIdx.x; b < ORDER_BUCKETS; b += blockDim.x)
        if (hist[b]) atomicAdd(a.ctl + kCtlHist + b, hist[b]);
    if (threadIdx.x == 0) {
        atomicAdd(a.ctl + kCtlWanted, total);
        atomicAdd(a.ctl + 4, bytes);
    }
}

__global__ void __launch_bounds__(256) orderScatterKernel(DecArgs a) {
    __shared__ uint32_t base[ORDER_BUCKETS], count[ORDER_BUCKETS], place[ORDER_BUCKETS];
    const int tid = threadIdx.x;
    if (tid < 32) {
        uint32_t v[4], s = 0;
        for (int k = 0; k < 4; ++k) {
            v[k] = a.ctl[kCtlHist + 4 * tid + k];
            s += v[k];
        }
        uint32_t run = warpScan(s, tid) - s;
        for (int k = 0; k < 4; ++k) {
            base[4 * tid + k] = run;
            run += v[k];
        }
    }
    // heavy blocks: above heavyPct % of the mean codeword bytes per resident warp
    const uint64_t limit = (uint64_t)a.ctl[4] * a.heavyPct / (100ull * max(a.slots, 1u));
    for (uint32_t first = blockIdx.x * 256u; first < a.n; first += gridDim.x * 256u) {
        const uint32_t i = first + tid;
        if (tid < ORDER_BUCKETS) count[tid] = 0;
        __syncthreads();
        const bool wanted = i < a.n && a.blocks[i].wanted;
        uint32_t b = 0, rank = 0;
        if (wanted) {
            const uint32_t len = a.codes[i].len;
            b = lenBucket(len);
            rank = atomicAdd(&count[b], 1u);
            if (a.heavyPct && len > limit) atomicAdd(a.ctl + kCtlHeavy, 1u);
        }
        __syncthreads();
        if (tid < ORDER_BUCKETS && count[tid]) place[tid] = base[tid] + atomicAdd(a.ctl + kCtlCursor + tid, count[tid]);
        __syncthreads();
        if (wanted) a.perm[place[b] + rank] = i;
    }
}

// A block's first kCwCache codeword bytes (and two 0xFF after a shorter codeword) are copied
// into shared memory before it is decoded.
constexpr uint32_t kCwCache = 2048;

// Context state word: Qe << 16 | state index << 1 | MPS. s_next[word & 127] holds the words after
// a renormalising MPS and after an LPS.
__device__ __forceinline__ uint32_t stateWord(uint32_t idx, uint32_t mps) { return (c_mq[idx] << 16) | (idx << 1) | mps; }

// MQ decoder (ISO/IEC 15444-1 C.3) over one codeword; bytes past its end read as 0xFF. Every
// lane of the warp holds the same state and takes the same decisions. A and C are kept with the
// 16-bit interval in the upper half; the next two bytes are held in registers, so that a
// byte-in does not wait for memory.
struct MqDecoder {
    uint32_t A, C, bp, end, cached, b0, b1;
    int CT;
    const uint8_t* in;
    const uint8_t* cache;

    __device__ __forceinline__ uint32_t at(uint32_t i) const {
        return i < cached ? (uint32_t)cache[i] : (i < end ? (uint32_t)in[i] : 0xFFu);
    }
    __device__ __forceinline__ void bytein() {
        const bool stuffed = b0 == 0xFFu;
        if (stuffed && b1 > 0x8Fu) {  // a marker: not consumed, ones from here on
            C += 0xFF00u;
            CT = 8;
            return;
        }
        C += b1 << (stuffed ? 9 : 8);
        CT = stuffed ? 7 : 8;
        ++bp;
        b0 = b1;
        b1 = at(bp + 1);
    }
    __device__ __forceinline__ void init(const uint8_t* data, uint32_t len, const uint8_t* copy, uint32_t copied) {
        in = data;
        end = len;
        cache = copy;
        cached = copied;
        bp = 0;
        b0 = at(0);
        b1 = at(1);
        C = b0 << 16;
        bytein();
        C <<= 7;
        CT -= 7;
        A = 0x80000000u;
    }
    // One decision in context state t: whether it is the LPS. succ: the state's successors;
    // tn: the context's next state.
    __device__ __forceinline__ bool decide(uint32_t t, uint2 succ, uint32_t& tn) {
        const uint32_t qe = t & 0xFFFF0000u;
        const uint32_t a = A - qe;
        const bool lower = C < qe, big = a >= qe;  // conditional exchange: the LPS has the larger part
        const bool lps = lower == big;
        A = lower ? qe : a;
        C -= lower ? 0u : qe;
        tn = (int)A >= 0 ? (lps ? succ.y : succ.x) : t;  // a renormalisation moves the state
        int n = __clz((int)A);
        A <<= n;
        if (n > CT) {  // the bits are not in C yet
            do {
                C <<= CT;
                n -= CT;
                bytein();
            } while (n > CT);
        }
        C <<= n;
        CT -= n;
        return lps;
    }
};

// One code-block by one warp. Bound by the MQ decoder's serial chain: a frame's time is at
// least its longest block's. All lanes run the decoder in step, each lane also holding one
// column of the block as row masks and (lanes 0-18) one context's state, so that everything but
// the chain is done for all columns at once: the contexts of a stripe come from boolean
// operations on whole columns, a sample's from one shuffle, a context's state from another.
// The refinement pass changes no significance, so its contexts are laid out as a list first
// and the chain runs down the list with its three states in registers; the bits are put back
// into the columns afterwards. On a B200, the Tier-1 of a 4K picture at 250 Mbit/s: 1.75 ms,
// where lane 0 alone, a sample at a time with the state in shared memory, took 2.39. (The
// longest block spends 188 cycles per refinement decision, about 400 per other one. Slower:
// code bytes fed ahead of their time to save the byte-in's branch, 2.3 ms; flag words per column
// and stripe in shared memory for the contexts, 2.2 ms.)
struct BlockDecoder {
    uint32_t sig, sgn, vis, refined, plane;  // this lane's column; plane: the bits of the plane in hand
    uint32_t state;                          // lanes 0-18: the context's state word
    uint32_t left, right;                    // the neighbouring columns' significance
    const uint2* next;
    const uint8_t* sk;
    MqDecoder mq;
    int lane, orient;

    // One decision in context cx.
    __device__ __forceinline__ uint32_t decode(uint32_t cx) {
        const uint32_t t = __shfl_sync(kFull, state, (int)cx);
        uint32_t tn;
        const bool lps = mq.decide(t, next[t & 127u], tn);
        if ((uint32_t)lane == cx) state = tn;
        return (t & 1u) ^ (lps ? 1u : 0u);
    }
    // The stripe at row r0 as the scan now stands: zc = the zero-coding contexts of its four
    // rows in this lane's column, a byte each (0: no significant neighbour); returns the rows
    // with a significant neighbour.
    __device__ __forceinline__ uint32_t contexts(int r0, uint32_t& zc) {
        left = shUp(sig, lane);
        right = shDown(sig, lane);
        Nbr q;
        q.l = left;
        q.lu = left << 1;
        q.ld = left >> 1;
        q.r = right;
        q.ru = right << 1;
        q.rd = right >> 1;
        q.u = sig << 1;
        q.d = sig >> 1;
        uint32_t c0, c1, c2, c3;
        zcMasks(q, orient, c0, c1, c2, c3);
        zc = spread1((c0 >> r0) & 0xFu) | (spread1((c1 >> r0) & 0xFu) << 1) | (spread1((c2 >> r0) & 0xFu) << 2) |
             (spread1((c3 >> r0) & 0xFu) << 3);
        return q.l | q.lu | q.ld | q.r | q.ru | q.rd | q.u | q.d;
    }
    // Sample (x, r) has its first 1-bit in this plane: its sign, and its significance.
    __device__ __forceinline__ void becomeSig(int x, int r) {
        const uint32_t gl = shUp(sgn, lane), gr = shDown(sgn, lane);
        uint32_t key = ((left >> r) & 1u) | (((gl >> r) & 1u) << 1) | (((right >> r) & 1u) << 2) | (((gr >> r) & 1u) << 3) |
                       ((((sig << 1) >> r) & 1u) << 4) | ((((sgn << 1) >> r) & 1u) << 5) |
                       ((((sig >> 1) >> r) & 1u) << 6) | ((((sgn >> 1) >> r) & 1u) << 7);
        key = __shfl_sync(kFull, key, x);
        const uint32_t c = sk[key];
        const uint32_t neg = decode(c & 31u) ^ (c >> 5);
        if (lane == x) {
            sig |= 1u << r;
            plane |= 1u << r;
            sgn |= neg << r;
        }
    }
};

__global__ void __launch_bounds__(DEC_THREADS, DEC_CTAS) decodeKernel(DecArgs a) {
    // the block's decoded bit-planes, a column per lane
    __shared__ uint32_t s_plane[30][32];
    __shared__ uint32_t s_list[kCblkArea / 4 + 2];  // a refinement pass's contexts, a byte each
    __shared__ uint32_t s_bits[kCblkArea / 32 + 2];  // and its decoded bits
    __shared__ uint2 s_next[2 * 47];
    __shared__ uint8_t s_cw[kCwCache + 2];  // the block's codeword, its first kCwCache bytes
    // sign coding, context | xor bit << 5, by the sign key: bits 0/1 left neighbour
    // significant/negative, 2/3 right, 4/5 above, 6/7 below
    __shared__ uint8_t s_sk[256];
    const int lane = threadIdx.x;
    for (int i = lane; i < 2 * 47; i += 32) {
        const uint32_t e = c_mq[i >> 1], mps = i & 1u;
        s_next[i] = make_uint2(stateWord((e >> 18) & 63u, mps), stateWord((e >> 24) & 63u, mps ^ ((e >> 17) & 1u)));
    }
    for (int k = lane; k < 256; k += 32) {
        auto chi = [&](int bit) { return ((k >> bit) & 1) ? (((k >> (bit + 1)) & 1) ? -1 : 1) : 0; };
        const int hc = max(-1, min(1, chi(0) + chi(2)));
        const int vc = max(-1, min(1, chi(4) + chi(6)));
        s_sk[k] = c_sc[(hc + 1) * 3 + (vc + 1)];
    }
    __syncwarp();
    BlockDecoder d;
    d.next = s_next;
    d.sk = s_sk;
    d.lane = lane;
    const uint32_t count = a.ctl[kCtlWanted], heavy = min(a.ctl[kCtlHeavy], kMaxHeavy);  // the first ones of the order

    auto decodeBlock = [&](const DecBlock& blk, const GbCblkCode& code) {
        const int w = blk.w, h = blk.h, nbps = code.nbps;
        const uint32_t valid = lane < w ? (h >= 32 ? kFull : (1u << h) - 1u) : 0u;
        d.orient = blk.orient;
        d.sig = d.sgn = d.refined = 0;
        // initial states, Table D.7: ZC context 0 state 4, run-length 3, uniform 46
        d.state = stateWord(lane == 0 ? 4u : lane == 17 ? 3u : lane == 18 ? 46u : 0u, 0u);
        d.mq.init(a.bytes + code.offset, code.len, s_cw, min(code.len, kCwCache) + 2u);
        int passes = code.passes, p = nbps;
        uint32_t coded = 0;  // samples coded in the plane in hand
        while (passes > 0 && p > 0) {
            --p;
            const uint32_t sig0 = d.sig;
            d.vis = d.plane = coded = 0;
            if (p != nbps - 1) {
                // significance propagation
                for (int r0 = 0; r0 < h; r0 += 4) {
                    uint32_t zc;
                    uint32_t e4 = ((d.contexts(r0, zc) & valid & ~d.sig) >> r0) & 0xFu;
                    uint32_t cols = __ballot_sync(kFull, e4 != 0);
                    while (cols) {
                        const int x = __ffs(cols) - 1;
                        cols &= cols - 1;
                        uint32_t e = __shfl_sync(kFull, e4, x), z = __shfl_sync(kFull, zc, x), seen = 0;
                        while (e) {
                            const int i = __ffs(e) - 1;
                            e &= e - 1;
                            seen |= 1u << i;
                            if (!d.decode((z >> (8 * i)) & 0xFFu)) continue;
                            d.becomeSig(x, r0 + i);
                            // what the scan has not passed may now be eligible
                            e4 = ((d.contexts(r0, zc) & valid & ~d.sig) >> r0) & 0xFu;
                            z = __shfl_sync(kFull, zc, x);
                            e = __shfl_sync(kFull, e4, x) & ~((2u << i) - 1u);
                            cols = __ballot_sync(kFull, e4 != 0) & ~((2u << x) - 1u);
                        }
                        if (lane == x) d.vis |= seen << r0;
                    }
                }
                coded = d.vis;
                if (--passes > 0) {
                    // magnitude refinement: the list of the pass's contexts (2: refined before, 1: a
                    // significant neighbour, 0), stripe by stripe, column by column
                    const uint32_t E = sig0;
                    d.left = shUp(d.sig, lane);
                    d.right = shDown(d.sig, lane);
                    const uint32_t nAny = (d.sig << 1) | (d.sig >> 1) | d.left | (d.left << 1) | (d.left >> 1) | d.right |
                                          (d.right << 1) | (d.right >> 1);
                    uint32_t m[8] = {nAny & ~d.refined, d.refined, 0u, 0u, 0u, 0u, 0u, 0u};
                    rowBytes(m);
                    const StripePlaces places(nibbleCounts(E), lane);
                    uint32_t total = 0;
                    uint8_t* list = reinterpret_cast<uint8_t*>(s_list);
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        uint8_t* o = list + total + places.before(s);
                        total += places.all(s);
                        uint32_t z = m[s];
#pragma unroll
                        for (int i = 0; i < 4; ++i, z >>= 8)
                            if (E & (1u << (4 * s + i))) *o++ = (uint8_t)z;
                    }
                    __syncwarp();
                    // the chain, its three states in registers
                    uint32_t s14 = __shfl_sync(kFull, d.state, 14), s15 = __shfl_sync(kFull, d.state, 15),
                             s16 = __shfl_sync(kFull, d.state, 16);
                    auto refine = [&](uint32_t cx) {
                        const uint32_t t = cx == 2u ? s16 : (cx == 1u ? s15 : s14);
                        uint32_t tn;
                        const bool lps = d.mq.decide(t, s_next[t & 127u], tn);
                        s16 = cx == 2u ? tn : s16;
                        s15 = cx == 1u ? tn : s15;
                        s14 = cx == 0u ? tn : s14;
                        return (t & 1u) ^ (lps ? 1u : 0u);
                    };
                    uint32_t acc = 0, codes = s_list[0];
                    const uint32_t whole = total & ~3u;
#pragma unroll 1
                    for (uint32_t k = 0; k < whole; k += 4) {
                        const uint32_t ahead = s_list[(k >> 2) + 1];
                        uint32_t four = 0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) four |= refine((codes >> (8 * i)) & 3u) << i;
                        acc |= four << (k & 31u);
                        if ((k & 31u) == 28u) {
                            if (lane == 0) s_bits[k >> 5] = acc;
                            acc = 0;
                        }
                        codes = ahead;
                    }
#pragma unroll 1
                    for (uint32_t k = whole; k < total; ++k, codes >>= 8) acc |= refine(codes & 3u) << (k & 31u);
                    if (lane == 0) s_bits[total >> 5] = acc;
                    if (lane == 14) d.state = s14;
                    if (lane == 15) d.state = s15;
                    if (lane == 16) d.state = s16;
                    __syncwarp();
                    total = 0;
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        const uint32_t at = total + places.before(s);
                        total += places.all(s);
                        uint32_t bits = __funnelshift_r(s_bits[at >> 5], s_bits[(at >> 5) + 1], at & 31u);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (E & (1u << (4 * s + i))) {
                                d.plane |= (bits & 1u) << (4 * s + i);
                                bits >>= 1;
                            }
                    }
                    __syncwarp();
                    d.refined |= E;
                    coded |= E;
                    --passes;
                }
            }
            if (passes > 0) {
                // cleanup, with run-length coding of quiet columns
                const uint32_t E = valid & ~d.sig & ~d.vis;
                for (int r0 = 0; r0 < h; r0 += 4) {
                    const uint32_t e4 = (E >> r0) & 0xFu;
                    uint32_t cols = __ballot_sync(kFull, e4 != 0);
                    if (!cols) continue;
                    uint32_t zc;
                    d.contexts(r0, zc);
                    // quiet columns: all four rows in cleanup, none with a significant neighbour
                    uint32_t runs = __ballot_sync(kFull, e4 == 0xFu && zc == 0u);
                    while (cols) {
                        const int x = __ffs(cols) - 1;
                        cols &= cols - 1;
                        uint32_t e = __shfl_sync(kFull, e4, x), z = __shfl_sync(kFull, zc, x);
                        int i = -1;  // the row that turned significant
                        if ((runs >> x) & 1u) {
                            if (!d.decode(17u)) continue;
                            i = (int)d.decode(18u) << 1;
                            i |= (int)d.decode(18u);
                        }
                        for (;;) {
                            if (i >= 0) {
                                d.becomeSig(x, r0 + i);
                                d.contexts(r0, zc);
                                z = __shfl_sync(kFull, zc, x);
                                e &= ~((2u << i) - 1u);
                                runs = __ballot_sync(kFull, e4 == 0xFu && zc == 0u);
                            }
                            i = -1;
                            while (e && i < 0) {
                                const int k = __ffs(e) - 1;
                                e &= e - 1;
                                if (d.decode((z >> (8 * k)) & 0xFFu)) i = k;
                            }
                            if (i < 0) break;
                        }
                    }
                }
                coded |= E;
                --passes;
            }
            s_plane[p][lane] = d.plane;  // read by this lane alone
        }
        // The words of the column: the sign, twice the magnitude, and the mid-point of the planes
        // not decoded (below the last plane for the samples coded in it, else one above), then
        // rows: a transpose, and word * step / 2 in floats.
        uint32_t v[32];
#pragma unroll
        for (int k = 0; k < 30; ++k) v[k + 1] = k >= p && k < nbps ? s_plane[k][lane] : 0u;
        v[0] = 0u;
        v[31] = d.sgn;
#pragma unroll
        for (int k = 0; k < 30; ++k)
            if (k == p) {
                v[k] |= d.sig & coded;
                v[k + 1] |= d.sig & ~coded;
            }
        transpose32(v);
        const float half = a.half[blk.band];
        float* out = reinterpret_cast<float*>(a.planes + blk.dst) + lane;
        if (lane < w) {
#pragma unroll
            for (int r = 0; r < 32; ++r)
                if (r < h) {
                    // 0 stays 0 whatever the step (an infinite one included)
                    const float mag = v[r] ? (float)(v[r] & 0x7FFFFFFFu) * half : 0.f;
                    out[(size_t)r * a.W] = (v[r] & 0x80000000u) ? -mag : mag;
                }
        }
    };

    // Lane 0 picks each block. The heavy blocks (the first of the order): on a reserved SM
    // (%smid below the reserved count), the first four warps to arrive take one each and every
    // other warp leaves, so that the SM runs their serial chains alone; the other warps take
    // blocks from the queue, then any heavy block no reserved SM's warp took (a grid that did
    // not reach every reserved SM). At least a sixteenth of the grid does not leave so: beside other
    // launches that hold the rest of the GPU, the reserved SMs can be all that this one gets, and
    // those warps finish the queue there.
    uint32_t smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    const uint32_t reserved = (heavy + 3) / 4;
    const uint32_t mayLeave = (gridDim.x - divUp(gridDim.x, 16u)) / max(reserved, 1u);  // of each reserved SM
    int phase = smid < reserved ? 0 : 1;  // 0 reserved SM, 1 queue, 2 unclaimed heavy blocks, 3 done
    uint32_t fb = 0;
    for (;;) {
        uint32_t j = 0xFFFFFFFFu;
        if (lane == 0) {
            if (phase == 0) {
                const uint32_t k = atomicAdd(a.ctl + kCtlArrive + smid, 1u), hi = 4 * smid + k;
                if (k < 4 && hi < heavy && atomicExch(a.ctl + kCtlClaim + hi, 1u) == 0) j = a.perm[hi];
                phase = k < mayLeave ? 3 : 1;
            }
            if (phase == 1 && j == 0xFFFFFFFFu) {
                const uint32_t q = heavy + atomicAdd(a.ctl, 1u);  // longest codewords first
                if (q < count) j = a.perm[q];
                else phase = 2;
            }
            if (phase == 2) {
                while (fb < heavy && atomicExch(a.ctl + kCtlClaim + fb, 1u) != 0) ++fb;
                if (fb < heavy) j = a.perm[fb++];
                else phase = 3;
            }
        }
        j = __shfl_sync(kFull, j, 0);
        if (j == 0xFFFFFFFFu) break;
        const DecBlock blk = a.blocks[j];
        GbCblkCode code = a.codes[j];
        // a block that cannot be decoded counts as empty: all zero
        if (code.nbps < 1 || code.nbps > 30 || (uint64_t)code.offset + code.len > a.size) code.passes = 0;
        if (code.passes == 0) {
            float* out = reinterpret_cast<float*>(a.planes + blk.dst) + lane;
            if (lane < blk.w)
                for (int r = 0; r < blk.h; ++r) out[(size_t)r * a.W] = 0.f;
            continue;
        }
        const uint8_t* src = a.bytes + code.offset;
        const uint32_t kept = min(code.len, kCwCache);
        for (uint32_t i = lane; i < kept; i += 32) s_cw[i] = src[i];
        if (lane < 2) s_cw[kept + lane] = code.len > kept + lane ? src[kept + lane] : 0xFFu;
        __syncwarp();
        decodeBlock(blk, code);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------- inverse DWT
constexpr int TS = 64, HALO = 4, TW = TS + 2 * HALO, TP = TW + 1;
// -delta, -gamma, -beta, -alpha
__device__ __forceinline__ constexpr float unlift(int s) {
    return s == 0 ? -(float)0.443506852043971
                  : s == 1 ? -(float)0.882911075530934 : s == 2 ? -(float)-0.052980118572961 : -(float)-1.586134342059924;
}
constexpr float kK = (float)1.230174104914001;
constexpr float kInvK = (float)(1.0 / 1.230174104914001);

__device__ __forceinline__ int mirror(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i;
    if (n == 1) return 0;
    const int period = 2 * (n - 1);
    i %= period;
    if (i < 0) i += period;
    return i < n ? i : period - i;
}

struct InvArgs {
    int w, h;            // this level's output (interleaved) size
    int snx, sny;        // low-band sizes
    const float* A;      // Mallat planes (high bands of this level; LL too at the top level)
    uint64_t aComp;
    int aStride;
    const float* ll;     // LL of this level (the previous inverse output), or NULL: take it from A
    uint64_t llComp;
    int llStride;
    float* out;          // LL of the level below (interleaved), or NULL at the last level
    uint64_t outComp;
    int outStride;
    uint16_t* pix;       // last level: interleaved 12-bit X'Y'Z' output
    int shift;
};

// One line of a tile, `step` floats between samples: the scaling, then the lifting steps undone
// in reverse (-delta and -beta on even samples, -gamma and -alpha on odd ones), in streaming
// order as sample j arrives, which gives every sample the same operands as step by step. The
// TS samples the tile outputs are written back in place, five behind the loads.
__device__ __forceinline__ void unliftLine(float* t, int step) {
    float x[TW];
#pragma unroll
    for (int j = 0; j < TW + 5; ++j) {
        if (j < TW) x[j] = t[j * step] * ((j & 1) ? kInvK : kK);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int i = j - 1 - s;
            const bool odd = s & 1;
            if (i >= (odd ? 1 : 2) && i <= (odd ? TW - 3 : TW - 2) && (i & 1) == (odd ? 1 : 0))
                x[i] = x[i] + unlift(s) * (x[i - 1] + x[i + 1]);
        }
        const int k = j - 5;
        if (k >= HALO && k < TW - HALO) t[k * step] = x[k];
    }
}

// Threads of a CTA: a thread per line of every component it holds (LAST: three, else one), in
// whole warps.
template <bool LAST>
__host__ __device__ constexpr int ivThreads() {
    return LAST ? 256 : 96;
}

// One level of one tile. Bound by instruction issue and load latency: a thread lifts a whole
// line in registers, as in the encoder's front end. All levels of a 4K picture on a B200:
// 0.187 ms, where a thread per sample and step, in shared memory throughout, took 0.482.
template <bool LAST>
__global__ void __launch_bounds__(ivThreads<LAST>(), LAST ? 3 : 8) invLevelKernel(InvArgs a) {
    extern __shared__ float smem[];
    constexpr int NC = LAST ? 3 : 1, THREADS = ivThreads<LAST>(), WARPS = THREADS / 32, PLANE = TW * TP;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = blockIdx.x, ty = blockIdx.y;
    const int x0 = tx * TS - HALO, y0 = ty * TS - HALO;
    const int w = a.w, h = a.h;
    // the tile, interleaved: a warp per row, a lane's columns the same in every row
    const int gx[3] = {mirror(x0 + lane, w), mirror(x0 + lane + 32, w), mirror(x0 + min(lane + 64, TW - 1), w)};
#pragma unroll 1
    for (int k = 0; k < NC; ++k) {
        const int comp = LAST ? k : (int)blockIdx.z;
        const float* A = a.A + comp * a.aComp;
        const float* LL = a.ll ? a.ll + comp * a.llComp : A;
        const int llStride = a.ll ? a.llStride : a.aStride;
#pragma unroll 3
        for (int ly = warp; ly < TW; ly += WARPS) {
            const int gy = mirror(y0 + ly, h), hy = gy >> 1;
            const float* low = (gy & 1) ? A + (size_t)(a.sny + hy) * a.aStride : LL + (size_t)hy * llStride;
            const float* high = ((gy & 1) ? low : A + (size_t)hy * a.aStride) + a.snx;
            float* t = smem + k * PLANE + ly * TP;
            const float v0 = (gx[0] & 1 ? high : low)[gx[0] >> 1], v1 = (gx[1] & 1 ? high : low)[gx[1] >> 1];
            const float v2 = lane < TW - 64 ? (gx[2] & 1 ? high : low)[gx[2] >> 1] : 0.f;
            t[lane] = v0;
            t[lane + 32] = v1;
            if (lane < TW - 64) t[lane + 64] = v2;
        }
    }
    __syncthreads();
    // rows, those of the halo too, then columns
    if (w >= 2)
        for (int i = tid; i < NC * TW; i += THREADS) unliftLine(smem + (i / TW) * PLANE + (i % TW) * TP, 1);
    __syncthreads();
    if (h >= 2)
        for (int i = tid; i < NC * TS; i += THREADS) unliftLine(smem + (i / TS) * PLANE + HALO + i % TS, TP);
    __syncthreads();
    if (LAST) {
        // two pixels a thread, as three words where the row starts on a word
        const bool words = ((uintptr_t)a.pix & 3u) == 0 && (w & 1) == 0;
        for (int ly = warp; ly < TS; ly += WARPS) {
            const int gy = y0 + HALO + ly, px = x0 + HALO + 2 * lane;
            if (gy >= h || px >= w) continue;
            uint32_t c[6];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float* t = smem + (HALO + ly) * TP + HALO + 2 * lane + i;
                const float v0 = t[0], v1 = t[PLANE], v2 = t[2 * PLANE];
                const float v[3] = {v0 + (float)1.402 * v2, v0 + (float)(-0.34413) * v1 + (float)(-0.71414) * v2,
                                    v0 + (float)1.772 * v1};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int code = (int)floorf(v[k] + 2048.5f);
                    c[3 * i + k] = (uint32_t)min(max(code, 0), 4095) << a.shift;
                }
            }
            uint16_t* o = a.pix + ((size_t)gy * w + px) * 3;
            if (words) {
                uint32_t* o32 = reinterpret_cast<uint32_t*>(o);
#pragma unroll
                for (int k = 0; k < 3; ++k) o32[k] = c[2 * k] | (c[2 * k + 1] << 16);
            } else {
                const int n = px + 1 < w ? 6 : 3;
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if (k < n) o[k] = (uint16_t)c[k];
            }
        }
    } else {
        float* out = a.out + blockIdx.z * a.outComp;
        for (int ly = warp; ly < TS; ly += WARPS) {
            const int gy = y0 + HALO + ly, px = x0 + HALO + lane;
            if (gy >= h) break;
            const float* t = smem + (HALO + ly) * TP + HALO + lane;
            if (px < w) out[(size_t)gy * a.outStride + px] = t[0];
            if (px + 32 < w) out[(size_t)gy * a.outStride + px + 32] = t[32];
        }
    }
}

// reduce == levels: the picture is the LL band as it is.
__global__ void colorOutKernel(const float* A, uint64_t comp, int stride, int w, int h, uint16_t* pix, int shift) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= w || y >= h) return;
    const size_t i = (size_t)y * stride + x;
    const float y0 = A[i], y1 = A[comp + i], y2 = A[2 * comp + i];
    const float v[3] = {y0 + (float)1.402 * y2, y0 + (float)(-0.34413) * y1 + (float)(-0.71414) * y2, y0 + (float)1.772 * y1};
    uint16_t* o = pix + ((size_t)y * w + x) * 3;
    for (int c = 0; c < 3; ++c) {
        const int code = (int)floorf(v[c] + 2048.5f);
        o[c] = (uint16_t)(min(max(code, 0), 4095) << shift);
    }
}

constexpr size_t kInvSmemLast = (size_t)3 * TW * TP * 4;
constexpr size_t kInvSmem = (size_t)TW * TP * 4;


}  // namespace

void decoderInit() {
    uint8_t sc[9];
    uint32_t mq[47];
    signTable(sc);
    mqTable(mq);
    GB_CHECK(cudaMemcpyToSymbol(c_sc, sc, sizeof sc));
    GB_CHECK(cudaMemcpyToSymbol(c_mq, mq, sizeof mq));
    GB_CHECK(cudaFuncSetAttribute(invLevelKernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInvSmemLast));
}

// Decodes of this process on a device between enqueue() and the end of finish().
static std::atomic<int>& decodesOn(int dev) {
    static std::atomic<int> n[64];
    return n[dev & 63];
}

void DecoderSlot::ended() {
    if (counted_) decodesOn(dev_).fetch_sub(1);
    counted_ = false;
}

uint64_t decoderSlotBytes(const Layout& L, const GailCudaDecodeSettings& s) {
    const uint64_t npix = (uint64_t)L.width * L.height, ll = (uint64_t)L.levelW(1) * L.levelH(1);
    const uint64_t out = (uint64_t)L.levelW(s.reduce) * L.levelH(s.reduce) * 6;
    return npix * 12 + 2 * ll * 12 + out + (uint64_t)L.numCblks() * (12 + 12 + 4) + (4ull << 20);
}

DecoderSlot::DecoderSlot(int device, const Layout& L, const GailCudaDecodeSettings& s, bool heavySms) : dev_(device), L_(L), s_(s) {
    heavySms_ = heavySms;
    if (s.reduce < 0 || s.reduce > L.levels) throw std::runtime_error("more resolution levels left out than the stream has");
    outW_ = L.levelW(s.reduce);
    outH_ = L.levelH(s.reduce);
    try {
        GB_CHECK(cudaSetDevice(dev_));
        GB_CHECK(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
        for (auto& e : ev_) GB_CHECK(cudaEventCreate(&e));
        for (auto& e : bandEv_) GB_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        const uint64_t npix = (uint64_t)L.width * L.height, ll = (uint64_t)L.levelW(1) * L.levelH(1);
        const uint64_t n = (uint64_t)L.numCblks();
        auto alloc = [&](auto*& p, uint64_t bytes) {
            void* q = nullptr;
            check(deviceAlloc(&q, std::max<uint64_t>(bytes, 16)), "device memory for a decoder slot");
            allocs_.push_back(q);
            p = static_cast<std::remove_reference_t<decltype(p)>>(q);
        };
        alloc(dPlanes_, npix * 12);
        alloc(dLL_[0], ll * 12);
        alloc(dLL_[1], ll * 12);
        alloc(dHalf_, L.bands.size() * 4);
        alloc(dCodes_, n * sizeof(GbCblkCode));
        alloc(dBlocks_, n * sizeof(DecBlock));
        alloc(dPerm_, n * 4);
        alloc(dCtl_, kCtlWords * 4);
        alloc(dOut_, (uint64_t)outW_ * outH_ * 6);
        check(cudaHostAlloc((void**)&hOut_, std::max<uint64_t>(16, (uint64_t)outW_ * outH_ * 6), cudaHostAllocDefault),
              "pinned host memory");
        check(cudaHostAlloc((void**)&hCodes_, std::max<uint64_t>(16, n * sizeof(GbCblkCode)), cudaHostAllocDefault),
              "pinned host memory");
        check(cudaHostAlloc((void**)&hHalf_, L.bands.size() * 4 + 16, cudaHostAllocDefault), "pinned host memory");
        check(cudaHostAlloc((void**)&hCtl_, 64, cudaHostAllocDefault), "pinned host memory");
        capBytes_ = 1500000;
        alloc(dBytes_, capBytes_);
        check(cudaHostAlloc((void**)&hBytes_, capBytes_, cudaHostAllocDefault), "pinned host memory");
        std::vector<DecBlock> blocks(n);
        const int maxRes = L.levels - s.reduce;
        for (uint64_t i = 0; i < n; ++i) {
            const CodeBlock& cb = L.cblks[i];
            const GbSubband& b = L.bands[cb.band];
            blocks[i] = {(uint32_t)((uint64_t)b.comp * npix + (uint64_t)(b.py0 + cb.y0) * L.width + b.px0 + cb.x0),
                         (uint16_t)cb.w, (uint16_t)cb.h, (uint8_t)b.orient, (uint8_t)cb.band,
                         (uint8_t)(b.res <= maxRes ? 1 : 0), 0};
        }
        GB_CHECK(cudaMemcpy(dBlocks_, blocks.data(), n * sizeof(DecBlock), cudaMemcpyHostToDevice));
    } catch (...) {
        release();
        throw;
    }
}

DecoderSlot::~DecoderSlot() { release(); }

void DecoderSlot::release() {
    cudaSetDevice(dev_);
    if (st_) cudaStreamSynchronize(st_);
    ended();
    for (void* p : allocs_) cudaFree(p);
    allocs_.clear();
    for (void* p : {(void*)hOut_, (void*)hCodes_, (void*)hHalf_, (void*)hCtl_, (void*)hBytes_})
        if (p) cudaFreeHost(p);
    hOut_ = nullptr;
    hCodes_ = nullptr;
    hHalf_ = nullptr;
    hCtl_ = nullptr;
    hBytes_ = nullptr;
    for (auto& e : ev_)
        if (e) {
            cudaEventDestroy(e);
            e = nullptr;
        }
    for (auto& e : bandEv_)
        if (e) {
            cudaEventDestroy(e);
            e = nullptr;
        }
    if (st_) cudaStreamDestroy(st_);
    st_ = nullptr;
    cudaGetLastError();
}

void DecoderSlot::decode(const Layout& frame, const uint8_t* data, size_t size, const GbCblkCode* blocks, size_t numBlocks,
                         void* dst, ptrdiff_t strideBytes, GailCudaDecodeTimings* tm) {
    const uint64_t rowBytes = (uint64_t)outW_ * 6;
    // page-locked caller rows (a serving layer's pinned buffers): the picture goes there
    // from the device directly
    cudaPointerAttributes at{};
    const bool pinned = cudaPointerGetAttributes(&at, dst) == cudaSuccess && at.type == cudaMemoryTypeHost &&
                        strideBytes >= (ptrdiff_t)rowBytes;
    cudaGetLastError();
    if (pinned) {
        enqueue(frame, data, size, blocks, numBlocks, tm && tm->wantWavelet, dst, strideBytes);
        finish(tm);
        return;
    }
    // pageable rows: the picture comes back in bands, and the host pool copies each band
    // into the caller's rows as soon as it has arrived, while the next bands are in flight
    // (52 MB at 4K: copied after the whole download it added its full time to the decode)
    enqueue(frame, data, size, blocks, numBlocks, tm && tm->wantWavelet, nullptr, 0, kBands);
    parallelFor(kBands, [&](int k) {
        GB_CHECK(cudaSetDevice(dev_));
        GB_CHECK(cudaEventSynchronize(bandEv_[k]));
        const int y0 = (int)((int64_t)outH_ * k / kBands), y1 = (int)((int64_t)outH_ * (k + 1) / kBands);
        const uint8_t* src = (const uint8_t*)hOut_ + (uint64_t)y0 * rowBytes;
        uint8_t* out = (uint8_t*)dst + (ptrdiff_t)y0 * strideBytes;
        if (strideBytes == (ptrdiff_t)rowBytes) {
            std::memcpy(out, src, rowBytes * (uint64_t)(y1 - y0));
        } else {
            for (int y = y0; y < y1; ++y, src += rowBytes, out += strideBytes) std::memcpy(out, src, rowBytes);
        }
    });
    finish(tm);
}

void DecoderSlot::enqueue(const Layout& frame, const uint8_t* data, size_t size, const GbCblkCode* blocks,
                          size_t numBlocks, bool wantWavelet, void* pinnedDst, ptrdiff_t dstStride, int bands) {
    if (bands < 1 || bands > kBands) throw std::logic_error("picture bands out of range");
    t0_ = std::chrono::steady_clock::now();
    if (frame.width != L_.width || frame.height != L_.height || frame.levels != L_.levels ||
        frame.bands.size() != L_.bands.size() || (int)numBlocks != L_.numCblks())
        throw std::logic_error("frame does not match the layout the slot was made for");
    if (size > 0xFFFFFFFFull) throw std::runtime_error("codestream too large");
    GB_CHECK(cudaSetDevice(dev_));
    const cudaStream_t st = st_;
    const uint64_t npix = (uint64_t)L_.width * L_.height, n = numBlocks;
    GB_CHECK(cudaStreamSynchronize(st));  // the slot's pinned buffers are free again
    if (size > capBytes_) {
        cudaFree(dBytes_);
        allocs_.erase(std::find(allocs_.begin(), allocs_.end(), (void*)dBytes_));
        cudaFreeHost(hBytes_);
        dBytes_ = nullptr;
        hBytes_ = nullptr;
        capBytes_ = size + size / 2;
        void* q = nullptr;
        check(deviceAlloc(&q, capBytes_), "device memory for a decoder slot");
        dBytes_ = (uint8_t*)q;
        allocs_.push_back(q);
        check(cudaHostAlloc((void**)&hBytes_, capBytes_, cudaHostAllocDefault), "pinned host memory");
    }
    std::memcpy(hBytes_, data, size);
    std::memcpy(hCodes_, blocks, n * sizeof(GbCblkCode));
    for (size_t i = 0; i < frame.bands.size(); ++i) hHalf_[i] = 0.5f * frame.bands[i].delta;
    wantWavelet_ = wantWavelet;
    // Heavy blocks get SMs of their own while no other decode is in flight: a second one beside it
    // finds little else free than the SMs the first keeps for its heavy blocks, and must not
    // leave them to those. Two threads of 4K decodes on a B200: 350 pictures a second, 223 when
    // both reserve SMs; four threads of 2K ones 704 and 640.
    ended();
    counted_ = true;
    const bool alone = decodesOn(dev_).fetch_add(1) == 0;

    GB_CHECK(cudaEventRecord(ev_[0], st));
    GB_CHECK(cudaMemcpyAsync(dBytes_, hBytes_, size, cudaMemcpyHostToDevice, st));
    GB_CHECK(cudaMemcpyAsync(dCodes_, hCodes_, n * sizeof(GbCblkCode), cudaMemcpyHostToDevice, st));
    GB_CHECK(cudaMemcpyAsync(dHalf_, hHalf_, frame.bands.size() * 4, cudaMemcpyHostToDevice, st));
    GB_CHECK(cudaMemsetAsync(dCtl_, 0, kCtlWords * 4, st));
    // every sample of a wanted block is written; the tap also shows the resolutions left out
    if (wantWavelet) GB_CHECK(cudaMemsetAsync(dPlanes_, 0, npix * 12, st));
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_);
    const Tuning tu = tuningFor(L_.profile);
    const uint32_t grid = std::min<uint32_t>((uint32_t)n, (uint32_t)(sms * tu.decCtasPerSm));
    DecArgs da{dBytes_, size, dCodes_, dBlocks_, (uint32_t)n, dHalf_, (uint32_t*)dPlanes_, (uint32_t)L_.width, dPerm_, dCtl_,
               std::min(grid, (uint32_t)(sms * DEC_CTAS)), heavySms_ && alone ? (uint32_t)tu.decHeavyPct : 0u};
    const uint32_t og = std::max(1u, std::min(divUp((uint32_t)n, 256u), (uint32_t)sms * 2u));
    orderCountKernel<<<og, 256, 0, st>>>(da);
    orderScatterKernel<<<og, 256, 0, st>>>(da);
    decodeKernel<<<grid, DEC_THREADS, 0, st>>>(da);
    GB_CHECK(cudaGetLastError());
    GB_CHECK(cudaEventRecord(ev_[1], st));
    // inverse wavelet, levels top down; the last one writes the picture (the planes are only
    // read, so the wavelet tap can still be copied out after it)
    const int stop = s_.reduce;
    const int llStride = L_.levelW(1);
    const uint64_t llComp = (uint64_t)L_.levelW(1) * L_.levelH(1);
    const int shift = s_.highBits ? 4 : 0;
    if (stop == L_.levels) {
        colorOutKernel<<<dim3(divUp(outW_, 256), outH_), 256, 0, st>>>(dPlanes_, npix, L_.width, outW_, outH_, dOut_, shift);
    }
    for (int l = L_.levels; l > stop; --l) {
        InvArgs a{};
        a.w = L_.levelW(l - 1);
        a.h = L_.levelH(l - 1);
        a.snx = L_.levelW(l);
        a.sny = L_.levelH(l);
        a.A = dPlanes_;
        a.aComp = npix;
        a.aStride = L_.width;
        a.ll = l == L_.levels ? nullptr : dLL_[l & 1];
        a.llComp = llComp;
        a.llStride = llStride;
        const bool last = l - 1 == stop;
        a.out = last ? nullptr : dLL_[(l - 1) & 1];
        a.outComp = llComp;
        a.outStride = llStride;
        a.pix = dOut_;
        a.shift = shift;
        if (last)
            invLevelKernel<true><<<dim3(divUp(a.w, TS), divUp(a.h, TS), 1), ivThreads<true>(), kInvSmemLast, st>>>(a);
        else
            invLevelKernel<false><<<dim3(divUp(a.w, TS), divUp(a.h, TS), 3), ivThreads<false>(), kInvSmem, st>>>(a);
    }
    GB_CHECK(cudaGetLastError());
    GB_CHECK(cudaEventRecord(ev_[2], st));
    const uint64_t rowBytes = (uint64_t)outW_ * 6;
    if (pinnedDst) {
        GB_CHECK(cudaMemcpy2DAsync(pinnedDst, (size_t)dstStride, dOut_, rowBytes, rowBytes, (size_t)outH_,
                                   cudaMemcpyDeviceToHost, st));
    } else {
        for (int k = 0; k < bands; ++k) {
            const uint64_t y0 = (uint64_t)outH_ * k / bands, y1 = (uint64_t)outH_ * (k + 1) / bands;
            GB_CHECK(cudaMemcpyAsync((uint8_t*)hOut_ + y0 * rowBytes, (const uint8_t*)dOut_ + y0 * rowBytes,
                                     (y1 - y0) * rowBytes, cudaMemcpyDeviceToHost, st));
            if (bands > 1) GB_CHECK(cudaEventRecord(bandEv_[k], st));
        }
    }
    GB_CHECK(cudaMemcpyAsync(hCtl_, dCtl_, 64, cudaMemcpyDeviceToHost, st));
    GB_CHECK(cudaEventRecord(ev_[3], st));
}

const uint16_t* DecoderSlot::finish(GailCudaDecodeTimings* tm) {
    GB_CHECK(cudaSetDevice(dev_));
    GB_CHECK(cudaStreamSynchronize(st_));
    ended();
    GB_CHECK(cudaGetLastError());
    // a warp that finds the queue empty has taken a number past its end, then every heavy block
    // nobody claimed
    if (hCtl_[0] <= hCtl_[kCtlWanted] - std::min(hCtl_[kCtlHeavy], kMaxHeavy))
        throw std::runtime_error("the decoder left code-blocks out");
    const uint64_t npix = (uint64_t)L_.width * L_.height;
    if (wantWavelet_)
        for (int c = 0; c < 3; ++c) {
            wavelet_[c].resize(npix);
            GB_CHECK(cudaMemcpy(wavelet_[c].data(), dPlanes_ + c * npix, npix * 4, cudaMemcpyDeviceToHost));
        }
    if (tm) {
        float a = 0, b = 0, c = 0;
        cudaEventElapsedTime(&a, ev_[0], ev_[1]);
        cudaEventElapsedTime(&b, ev_[1], ev_[2]);
        cudaEventElapsedTime(&c, ev_[2], ev_[3]);
        tm->t1 = a;
        tm->dwt = b;
        tm->color = c;
        tm->total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0_).count();
        tm->numWavelet = wantWavelet_ ? npix : 0;
        for (int k = 0; k < 3; ++k) tm->wavelet[k] = wantWavelet_ ? wavelet_[k].data() : nullptr;
    }
    return hOut_;
}

}  // namespace gb
