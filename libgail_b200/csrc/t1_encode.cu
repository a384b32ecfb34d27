// EBCOT Tier-1 encoder for sm_100a.
//
// Stage 1, context modelling (t1CmKernel): one warp per code-block. Lane x owns column x
// of the block and keeps its state as 32-bit row masks (bit r = row r): significance,
// sign, refined-before, coded-in-this-plane, and the bit-planes (one bit transpose per block).
// The only sequential dependency of the scan order (columns left to right, rows top down)
// that matters is significance propagation, where a sample that becomes significant makes
// later samples eligible; it is solved as a least fixpoint over the warp, which is the causal
// result because the dependency graph runs strictly along the scan order. The contexts of
// all rows come from boolean operations on the masks (t1_masks.cuh). Each lane then emits
// its column's decisions in scan order and a warp prefix sum places them; a plane's
// decisions are staged in shared memory and copied out with coalesced stores. Per-pass symbol
// counts and distortion reductions are written.
//
// Stage 2, ordering (t1OrderCountKernel, t1OrderScatterKernel): counting sort of the blocks by decision count, most
// first, so the longest serial MQ chains start first.
//
// Stage 3, MQ coding (t1MqKernel): one lane per code-block; a warp takes the next 32 blocks
// of the order at once. The coder takes 16 decisions at a time in branch-free select form,
// then the bytes they completed; its contexts live in shared memory, and its input is
// loaded 32 decisions ahead. The MQ state at each pass's end is recorded.
//
// Stage 4, truncation lengths (t1TruncKernel): a warp per block, a lane per pass; each
// pass's length is found from its recorded MQ state and the final codeword bytes. Kept
// out of the MQ kernel, whose lanes would otherwise stall on these byte reads one block
// end at a time while their warp-mates code.
//
// Semantics restated from ISO/IEC 15444-1 Annexes C and D as the reference coder applies
// them (Josephur/libgail core/t1_ref.cpp:52-292, kernels/mq_encoder.h:48-169,
// kernels/t1_common.h:20-53); bit-exact with it for every block.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "t1_encode.cuh"
#include "t1_masks.cuh"
#include "capi_util.h"
#include "t1_tables.h"
#include "tuning.h"

namespace gb {

namespace {

constexpr int CM_WARPS = 4;          // warps (code-blocks in flight) per CTA
constexpr int CM_THREADS = CM_WARPS * 32;
constexpr int CM_CTAS = 7;           // resident CTAs per SM of the context-modelling kernel
// Staging bytes per warp: one plane's decisions. A sample takes one refinement decision
// or at most two (zero coding and sign) in a plane, and a run-length stripe column adds at
// most two more (run, two position decisions, sign, in place of one zero-coding decision):
// 2 * 1024 + 2 * 256 = 2560 for a 32x32 block.
constexpr int STAGE = 2560 + 64;
constexpr int MQ_THREADS = 128;
constexpr int ORDER_BUCKETS = 128;

__constant__ uint32_t c_mq[47];      // Qe | switch << 17 | NMPS << 18 | NLPS << 24

// Early termination after plane p of a block (the reference's stopAfterPlane,
// core/t1_ref.cpp:115-162), with every float operation in the CPU's order: the estimates'
// terms a lane each, their sums in order. The plane's `count` decisions are at pb; hist is
// zero before and after. The same on every lane.
__device__ __noinline__ bool stopAfterPlane(const T1Job& J, const uint8_t* pb, uint32_t count, uint32_t* hist, float slope,
                                            int32_t planeDist, int p, int w, int h, int lane) {
    for (uint32_t i = lane; i < count; i += 32) {
        const uint32_t s = pb[i];
        atomicAdd(&hist[s >> 1], (s & 1u) ? 0x10000u : 1u);
    }
    __syncwarp();
    const uint32_t hv = lane < 19 ? hist[lane] : 0u;
    __syncwarp();
    if (lane < 19) hist[lane] = 0;
    if (p == 0) return false;
    const float n0 = (float)(hv & 0xFFFFu), n1 = (float)(hv >> 16), n = __fadd_rn(n0, n1);
    float term = 0.f;
    if (n > 0.f) {
        const float l0 = log2f(__fdiv_rn(fmaxf(n0, 0.5f), n));
        const float l1 = log2f(__fdiv_rn(fmaxf(n1, 0.5f), n));
        const float t = __fadd_rn(__fmul_rn(n0, l0), __fmul_rn(n1, l1));
        term = __fadd_rn(-t, 2.f);
    }
    const uint32_t used = __ballot_sync(kFull, n > 0.f);
    float bits = 0.f;
    for (int cx = 0; cx < 19; ++cx) {
        const float t = __shfl_sync(kFull, term, cx);
        if ((used >> cx) & 1u) bits = __fadd_rn(bits, t);
    }
    const float bytes = __fadd_rn(__fmul_rn(bits, 0.125f), 1.f);
    const float lim = __fmul_rn(slope, bytes);
    const float dabs =
        __fmul_rn(__fmul_rn(__fmul_rn((float)planeDist, exp2f((float)(2 * p))), 1.f / 4096.f), J.dscale);
    if (!(dabs < lim)) return false;
    float e = 0.f;
    const float step = exp2f((float)p);
    for (int y = 0; y < h; ++y) {
        const uint32_t m = J.coeffs[32 * y + lane] & 0x7FFFFFFFu;
        const float v = __fmul_rn((float)m, 1.f / 64.f);
        const uint32_t qq = m >> (p + kFracBits);
        const float rec = qq == 0 ? 0.f : __fmul_rn(__fadd_rn((float)qq, 0.5f), step);
        const float d = __fsub_rn(v, rec);
        const float d2 = __fmul_rn(d, d);
        for (int x = 0; x < w; ++x) e = __fadd_rn(e, __shfl_sync(kFull, d2, x));
    }
    return __fmul_rn(e, J.dscale) < lim;
}

// Context modelling of block `job` by one warp: its decisions to its symbol region, its
// pass table and info words. planes: the warp's 32 x 32 words, buf: its plane staging, hist:
// its 19 context counters. Returns the block's decisions (the same on every lane).
//
// Bound by instruction issue. Every step but the byte stores works on whole columns: a lane
// holds its column's bit-planes as 32-bit row masks (one 32 x 32 bit transpose per block, the
// planes then kept in shared memory), finds the contexts of all 32 rows at once in boolean
// form, turns them into decision bytes by an 8 x 8 bit transpose, and gets the distortions from
// the set bits of the planes below. The significance propagation is one fixpoint over the whole
// block; inside a column the chain of newly significant rows is the carry of an addition.
// On a B200, per 4K frame (25,986 blocks): 0.37 ms, where per stripe and row with table lookups
// it was 0.92 ms; for the 48 blocks of a 64 x 64 frame 43 us, where it was 121.
__device__ __forceinline__ uint32_t cmJob(const T1Launch& P, uint32_t job, uint32_t (*planes)[32], uint8_t* buf,
                                          uint32_t* hist, int lane) {
    uint32_t* status = P.ctl + 1;
    const T1Job J = P.jobs[job];
    const int w = (J.geom & 31u) + 1, h = ((J.geom >> 5) & 31u) + 1, orient = (J.geom >> 10) & 3u;
    const int maxPasses = (J.geom >> 12) & 127u;
    const float slope = P.slope ? P.slope[J.slope] : 0.f;

    // lane x loads column x, words outside w x h as 0, and transposes it: planes[p] holds bit p
    // of the column's words (plane 31: the signs)
    uint32_t sgn;
    int nbps;
    {
        uint32_t v[32];
#pragma unroll
        for (int r = 0; r < 32; ++r) v[r] = J.coeffs[32 * r + lane];
        if (w < 32 || h < 32) {
#pragma unroll
            for (int r = 0; r < 32; ++r)
                if (lane >= w || r >= h) v[r] = 0u;
        }
        uint32_t any = 0;
#pragma unroll
        for (int r = 0; r < 32; ++r) any |= v[r];
        const uint32_t top = (__reduce_or_sync(kFull, any) & 0x7FFFFFFFu) >> kFracBits;
        nbps = top ? 32 - __clz(top) : 0;
        uint32_t* info = P.info + 4 * (size_t)job;
        if (nbps == 0 || 3 * nbps - 2 > kMaxPasses) {
            if (lane == 0) {
                info[0] = nbps > 0 ? (uint32_t)nbps : 0u;
                info[1] = 0;
                info[2] = 0;
                info[3] = 0;
                if (nbps) atomicOr(status, kErrTooManyPlanes);
            }
            __syncwarp();
            return 0u;
        }
        transpose32(v);
        sgn = v[31];
#pragma unroll
        for (int p = 0; p < 31; ++p) planes[p][lane] = v[p];  // read by this lane alone
    }
    if (lane < 19) hist[lane] = 0;
    __syncwarp();

    const uint32_t valid = lane < w ? (h >= 32 ? kFull : ((1u << h) - 1u)) : 0u;
    const uint32_t sgnL = shUp(sgn, lane), sgnR = shDown(sgn, lane);
    uint32_t sig = 0, refined = 0, symTotal = 0;
    int np = 0;
    uint8_t* gsym = J.sym;

    for (int p = nbps - 1; p >= 0 && np < maxPasses; --p) {
        const uint32_t Bp = planes[p + kFracBits][lane];
        const uint32_t sig0 = sig;
        uint32_t vis = 0, count = 0;
        // the plane's decisions are staged at the alignment their region has in global
        // memory, so that they go out as 16-byte vectors
        uint8_t* const pb = buf + (symTotal & 15u);
        int32_t planeDist = 0;
#pragma unroll 1
        for (int type = (p == nbps - 1 ? 2 : 0); type < 3 && np < maxPasses; ++type) {
            // (1) the pass's row masks: E = rows coded, NEW = rows that become significant
            const uint32_t S = sig;
            const uint32_t SL = shUp(S, lane), SR = shDown(S, lane);
            // rows with a significant neighbour before the pass
            const uint32_t nAny = (S << 1) | (S >> 1) | SL | (SL << 1) | (SL >> 1) | SR | (SR << 1) | (SR >> 1);
            uint32_t E = 0, NEW = 0, NL = 0, NR = 0;
            if (type == 0) {
                // significance propagation: eligible = insignificant with a significant
                // neighbour in scan order. The dependencies run along the scan order, so the
                // least fixpoint is the scan's result. New neighbours that the scan has passed:
                // the left column down to the row's stripe end, the right column's row above at
                // a stripe's start, the own column's rows above.
                const uint32_t cand = valid & ~S, grow = cand & Bp;
                uint32_t elig = nAny;
                if (__any_sync(kFull, cand & elig)) {
#pragma unroll 1
                    for (int it = 0; it < 1025; ++it) {  // every turn but the last adds a sample
                        const uint32_t seed = grow & elig;
                        // down each run of rows that turn significant once eligible: the carry
                        // of the addition clears the run's rows from its lowest seed on
                        NEW = seed | (grow & ~(grow + seed));
                        NL = shUp(NEW, lane);
                        NR = shDown(NEW, lane);
                        elig = nAny | NL | (NL << 1) | ((NL >> 1) & 0x77777777u) | ((NR << 1) & 0x11111111u);
                        if (!__any_sync(kFull, grow & elig & ~NEW)) break;
                    }
                    E = cand & (elig | (NEW << 1));
                }
                sig = S | NEW;
                vis = E;
            } else if (type == 1) {
                E = sig0;  // refinement of what was significant before this plane
            } else {
                E = valid & ~S & ~vis;  // cleanup: everything else
                NEW = E & Bp;
                sig = S | NEW;
                NL = shUp(NEW, lane);
                NR = shDown(NEW, lane);
            }
            int32_t total = 0;
            const uint32_t rowsAny = __reduce_or_sync(kFull, E);
            if (rowsAny) {
                // (2) decision bytes of every row, byte i of word s for row 4 s + i; EZ = rows
                //     with a zero-coding (or refinement) decision; runs = cleanup's run-length
                //     stripes, newRun those with a new sample, its index in runHi / runLo (bit 4 s)
                uint32_t m[8];
                uint32_t EZ = E, runs = 0, newRun = 0, runHi = 0, runLo = 0;
                int32_t dist;
                if (type == 1) {
                    // context 16 (refined before), 15 (a significant neighbour) or 14, and the bit
                    m[0] = Bp;
                    m[1] = nAny & ~refined;
                    m[2] = refined;
                    m[3] = m[4] = m[5] = m[6] = m[7] = 0u;
                    rowBytes(m);
#pragma unroll
                    for (int s = 0; s < 8; ++s) m[s] += 0x1C1C1C1Cu;
                    // distRef over E: with X_k the rows whose plane k below agrees with the bit,
                    // 64 sum 2^k |X_k| - 1024 |bit set| - 960 |bit clear|
                    dist = -1024 * __popc(E & Bp) - 960 * __popc(E & ~Bp);
#pragma unroll
                    for (int k = 0; k < kFracBits; ++k) dist += (64 << k) * __popc(E & ~(planes[p + k][lane] ^ Bp));
                } else {
                    Nbr q;
                    q.l = SL | NL;
                    q.lu = q.l << 1;
                    q.ld = (SL >> 1) | ((NL >> 1) & 0x77777777u);
                    q.r = SR;
                    q.ru = (SR << 1) | ((NR << 1) & 0x11111111u);
                    q.rd = SR >> 1;
                    q.u = sig << 1;
                    q.d = S >> 1;
                    if (type == 2) {
                        // run-length mode: all four rows in cleanup, and no significant neighbour
                        // when the scan reaches the stripe's column
                        const uint32_t full = E & (E >> 1) & (E >> 2) & (E >> 3) & 0x11111111u;
                        runs = full & ~nibbleAny(q.l | q.lu | q.ld | q.r | q.ru | q.rd | q.d | (q.u & 0x11111111u));
                        const uint32_t runRows = runs * 0xFu, N = NEW & runRows;
                        // rows of run stripes from the first new sample on; that row's zero-coding
                        // decision is replaced by the run decision and its index
                        const uint32_t fill =
                            N | ((N << 1) & 0xEEEEEEEEu) | ((N << 2) & 0xCCCCCCCCu) | ((N << 3) & 0x88888888u);
                        EZ = (E & ~runRows) | (fill & (fill << 1) & 0xEEEEEEEEu);
                        newRun = nibbleAny(N);
                        runHi = newRun & ~(N | (N >> 1));
                        runLo = newRun & ~N & ((N >> 1) | ~(N >> 2));
                    }
                    // a new row's bit is 1, so bit 0 carries the sign decision's bit instead
                    zcMasks(q, orient, m[1], m[2], m[3], m[4]);
                    scMasks(q, sgn, sgnL, sgnR, m[5], m[6], m[7], m[0]);
                    m[0] &= NEW;
                    rowBytes(m);
                    // distSig over NEW: the bit is set, so 192 * 64 - 9216 and 192 per unit below
                    dist = 3072 * __popc(NEW);
#pragma unroll
                    for (int k = 0; k < kFracBits; ++k) dist += (192 << k) * __popc(NEW & planes[p + k][lane]);
                }
                total = __reduce_add_sync(kFull, dist);
                // (3) decisions per stripe, and each lane's place among them
                const uint32_t c = nibbleCounts(EZ) + nibbleCounts(NEW) + runs + 2u * newRun;
                const StripePlaces places(c, lane);
                // (4) every lane writes its decisions, stripe after stripe
                uint32_t before = count;  // decisions of the pass's stripes so far
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int r0 = 4 * s;
                    uint8_t* o = pb + before + places.before(s);
                    before += places.all(s);
                    if (type == 1) {
                        uint32_t z = m[s];
#pragma unroll
                        for (int i = 0; i < 4; ++i, z >>= 8)
                            if (EZ & (1u << (r0 + i))) *o++ = (uint8_t)z;
                    } else {
                        uint32_t z = (m[s] & 0x1E1E1E1Eu) | spread1((NEW >> r0) & 0xFu);
                        uint32_t g = 0x10101010u | ((m[s] >> 4) & 0x0E0E0E0Eu) | (m[s] & 0x01010101u);
                        if (runs & (1u << r0)) {
                            *o++ = (uint8_t)((17u << 1) | ((newRun >> r0) & 1u));
                            if (newRun & (1u << r0)) {
                                o[0] = (uint8_t)((18u << 1) | ((runHi >> r0) & 1u));
                                o[1] = (uint8_t)((18u << 1) | ((runLo >> r0) & 1u));
                                o += 2;
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i, z >>= 8, g >>= 8) {
                            if (EZ & (1u << (r0 + i))) *o++ = (uint8_t)z;
                            if (NEW & (1u << (r0 + i))) *o++ = (uint8_t)g;
                        }
                    }
                }
                count = before;
            }
            if (type == 1) refined |= sig0;
            if (lane == 0) {
                P.passEnd[(size_t)job * kMaxPasses + np] = symTotal + count;
                P.passDist[(size_t)job * kMaxPasses + np] = total;
            }
            ++np;
            planeDist += total;
        }
        // the plane's decisions to the block's region
        __syncwarp();
        if (symTotal + count <= J.cap) {
            const uint32_t head = min(count, (16u - (symTotal & 15u)) & 15u);
            if ((uint32_t)lane < head) gsym[symTotal + lane] = pb[lane];
            const uint32_t nv = (count - head) >> 4;
            const uint4* s4 = reinterpret_cast<const uint4*>(pb + head);
            uint4* d4 = reinterpret_cast<uint4*>(gsym + symTotal + head);
            for (uint32_t i = lane; i < nv; i += 32) d4[i] = s4[i];
            const uint32_t done = head + 16u * nv;
            if ((uint32_t)lane < count - done) gsym[symTotal + done + lane] = pb[done + lane];
        } else if (lane == 0) {
            atomicOr(status, kErrSymbolSpace);
        }
        bool stop = false;
        if (slope > 0.f) stop = stopAfterPlane(J, pb, count, hist, slope, planeDist, p, w, h, lane);
        symTotal += count;
        __syncwarp();
        if (stop) break;
    }
    if (lane == 0) {
        uint32_t* info = P.info + 4 * (size_t)job;
        info[0] = (uint32_t)nbps;
        info[1] = (uint32_t)np;
        info[2] = symTotal;
        info[3] = 0;
        atomicAdd(P.ctl + 2, symTotal);
    }
    __syncwarp();
    return symTotal;
}

__global__ void __launch_bounds__(CM_THREADS, CM_CTAS) t1CmKernel(T1Launch P) {
    __shared__ uint32_t s_planes[CM_WARPS][32][32];
    __shared__ __align__(16) uint8_t s_stage[CM_WARPS][STAGE];
    __shared__ uint32_t s_hist[CM_WARPS][19];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (uint32_t job = blockIdx.x * CM_WARPS + wid; job < P.n; job += gridDim.x * CM_WARPS)
        cmJob(P, job, s_planes[wid], s_stage[wid], s_hist[wid], lane);
}

// ---------------------------------------------------------------------------- ordering
__device__ __forceinline__ uint32_t orderBucket(uint32_t s) {
    // log-spaced classes, four per octave; the most decisions first
    if (s < 4) return ORDER_BUCKETS - 1;
    const uint32_t l = 31 - __clz(s);
    const uint32_t cls = min(4 * l + ((s >> (l - 2)) & 3u), (uint32_t)ORDER_BUCKETS - 1);
    return ORDER_BUCKETS - 1 - cls;
}

// The first blocks of the order are MQ-coded alone in a warp (its lane 0), one per warp at most: the
// longest serial chains, which would otherwise run beside 31 neighbours. As many as have
// P.soloDecisions decisions or more, up to maxSolo: half the warps of a batched launch, whose
// soloDecisions is a power of two and so the limit of a class; up to every warp of a smaller one,
// whose soloDecisions is 1 (the last class holds blocks without a decision too: a warp that gets
// one goes on at once).
__global__ void __launch_bounds__(1024) t1OrderKernel(T1Launch P, uint32_t maxSolo) {
    __shared__ uint32_t hist[ORDER_BUCKETS];
    __shared__ uint32_t solo;
    for (int i = threadIdx.x; i < ORDER_BUCKETS; i += blockDim.x) hist[i] = 0;
    if (threadIdx.x == 0) solo = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < P.n; i += blockDim.x) {
        const uint32_t d = P.info[4 * (size_t)i + 2];
        atomicAdd(&hist[orderBucket(d)], 1u);
        if (d >= P.soloDecisions) atomicAdd(&solo, 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) P.ctl[3] = min(solo, maxSolo);
    if (threadIdx.x < 32) {
        // exclusive scan of 128 counters by one warp, four per lane
        const int lane = threadIdx.x;
        uint32_t v[4], s = 0;
        for (int k = 0; k < 4; ++k) {
            v[k] = hist[4 * lane + k];
            s += v[k];
        }
        const uint32_t incl = warpScan(s, lane);
        uint32_t run = incl - s;
        for (int k = 0; k < 4; ++k) {
            hist[4 * lane + k] = run;
            run += v[k];
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < P.n; i += blockDim.x)
        P.perm[atomicAdd(&hist[orderBucket(P.info[4 * (size_t)i + 2])], 1u)] = i;
}

// Words of a launch's work area the wide ordering uses (those of the persistent launch's
// solo count, bucket histogram and list: a launch is one or the other).
constexpr uint32_t kWSoloWide = 2, kWHistWide = 16, kWCursorWide = 16 + ORDER_BUCKETS;

// The same ordering over the whole GPU, for launches with a work area (its head zeroed
// before): per-CTA histograms summed into the work area; then every CTA scans that histogram
// for itself and places its blocks 256 at a time, one atomic per bucket and CTA for their
// places. Blocks within a bucket land in any order, as in the one-CTA form (the order only
// decides which lane codes a block when, never its bytes). Bound by launches and latency: a
// 4K frame's 25,986 blocks in 12 us on a B200, 29 with the scan a launch of its own and an
// atomic per block.
__global__ void __launch_bounds__(256) t1OrderCountKernel(T1Launch P) {
    __shared__ uint32_t hist[ORDER_BUCKETS];
    __shared__ uint32_t solo;
    for (int i = threadIdx.x; i < ORDER_BUCKETS; i += blockDim.x) hist[i] = 0;
    if (threadIdx.x == 0) solo = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        const uint32_t d = P.info[4 * (size_t)i + 2];
        atomicAdd(&hist[orderBucket(d)], 1u);
        if (d >= P.soloDecisions) atomicAdd(&solo, 1u);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < ORDER_BUCKETS; b += blockDim.x)
        if (hist[b]) atomicAdd(P.work + kWHistWide + b, hist[b]);
    if (threadIdx.x == 0 && solo) atomicAdd(P.work + kWSoloWide, solo);
}

__global__ void __launch_bounds__(256) t1OrderScatterKernel(T1Launch P, uint32_t maxSolo) {
    __shared__ uint32_t base[ORDER_BUCKETS], count[ORDER_BUCKETS], place[ORDER_BUCKETS];
    const int tid = threadIdx.x;
    if (tid < 32) {
        uint32_t v[4], s = 0;
        for (int k = 0; k < 4; ++k) {
            v[k] = P.work[kWHistWide + 4 * tid + k];
            s += v[k];
        }
        uint32_t run = warpScan(s, tid) - s;
        for (int k = 0; k < 4; ++k) {
            base[4 * tid + k] = run;
            run += v[k];
        }
    }
    if (blockIdx.x == 0 && tid == 0) P.ctl[3] = min(P.work[kWSoloWide], maxSolo);
    for (uint32_t first = blockIdx.x * 256u; first < P.n; first += gridDim.x * 256u) {
        const uint32_t i = first + tid;
        if (tid < ORDER_BUCKETS) count[tid] = 0;
        __syncthreads();
        uint32_t b = 0, rank = 0;
        if (i < P.n) {
            b = orderBucket(P.info[4 * (size_t)i + 2]);
            rank = atomicAdd(&count[b], 1u);
        }
        __syncthreads();
        if (tid < ORDER_BUCKETS && count[tid])
            place[tid] = base[tid] + atomicAdd(P.work + kWCursorWide + tid, count[tid]);
        __syncthreads();
        if (i < P.n) P.perm[place[b] + rank] = i;
    }
}

// ---------------------------------------------------------------------------- MQ coding
// The layout of a lane's MQ memory: 20 context states (19 contexts and the null context, whose
// decisions change nothing) and a round's 16 steps, word i of either CS words after word i - 1. A
// decision byte is context << 1 | bit; CS is such that the context's byte offset is the byte
// shifted left by SHIFT, its bit masked off.
template <int CS>
struct MqLayout {
    static_assert(CS == 32 || CS == 128, "context stride");
    static constexpr int SHIFT = CS == 128 ? 8 : 6;
    static constexpr uint32_t kCtxMask = 0x3Eu << SHIFT;
    // Context state word: Qe << 16 | the byte offset of its successors, in which bit SHIFT is the
    // MPS (where a decision byte shifted left by SHIFT has its bit) and the state index fills
    // the other bits from 3 on.
    __device__ static uint32_t word(uint32_t idx, uint32_t mps) {
        const uint32_t low = idx & ((1u << (SHIFT - 3)) - 1u), high = idx >> (SHIFT - 3);
        const uint32_t qe = c_mq[idx] << 16;
        return qe | ((uint32_t)__clz((int)qe) << 10) | (high << (SHIFT + 1)) | (mps << SHIFT) | (low << 3);
    }
};
constexpr uint32_t kOffMask = 0x3F8u;   // the successors' offset in a state word
constexpr uint32_t kNullByte = 19u << 1;  // a decision in the null context (state word 0)
constexpr int MQ_CTX = 20, MQ_ROUND = 16, MQ_WORDS = MQ_CTX + MQ_ROUND;

// The code register of one block: the interval's base, the bits shifted out of it, the bytes.
struct Coder {
    uint32_t C, B;
    int CT, bp;
    uint8_t* out;
    uint32_t cap;
    bool overflow;

    // Annex C BYTEOUT with its three cases as selects: after 0xFF a stuffed bit (7 bits
    // next); otherwise a carry into the pending byte, which may make it 0xFF.
    __device__ __forceinline__ void byteout() {
        const bool carry = B != 0xFFu && C >= 0x8000000u;
        B += carry ? 1u : 0u;
        C &= carry ? 0x7FFFFFFu : 0xFFFFFFFFu;
        const bool stuff = B == 0xFFu;
        if (bp >= 0) {
            if ((uint32_t)bp < cap) out[bp] = (uint8_t)B;
            else overflow = true;
        }
        ++bp;
        B = (C >> (stuff ? 20 : 19)) & 0xFFu;
        C &= stuff ? 0xFFFFFu : 0x7FFFFu;
        CT = stuff ? 7 : 8;
    }
    // A: the interval, 16 bits
    __device__ __forceinline__ uint32_t flush(uint32_t A) {
        const uint32_t tempc = C + A;
        C |= 0xFFFFu;
        if (C >= tempc) C -= 0x8000u;
        C <<= CT;
        byteout();
        C <<= CT;
        byteout();
        if (B != 0xFFu) {
            if ((uint32_t)bp < cap) out[bp] = (uint8_t)B;
            else overflow = true;
            return (uint32_t)(bp + 1);
        }
        return (uint32_t)bp;
    }
};

// Control words of a persistent launch (T1Launch::work, zeroed before it), then the
// order's bucket counters (offsets once scanned), then the list of blocks whose MQ coding
// is done, in the order they finished (block + 1; 0 = not yet written).
enum : uint32_t {
    kWCmHead = 0,      // next block to model
    kWCmDone = 1,      // blocks modelled
    kWSolo = 2,        // blocks of soloDecisions decisions or more
    kWScanDone = 3,    // the order's bucket offsets are ready
    kWScatHead = 4,    // next chunk of the order's scatter
    kWScatDone = 5,
    kWSoloHead = 6,    // next solo block to claim
    kWTruncTail = 7,   // entries in the list
    kWTruncHead = 8,   // next entry to take for truncation lengths
    kWHist = 16,
    kWList = 16 + 2 * ORDER_BUCKETS,
};
static_assert(kWList == kT1WorkHead, "work layout");
static_assert(kWSoloWide == kWSolo && kWHistWide == kWHist, "the wide ordering's words");

// Loads of what other warps of a persistent launch wrote during the launch, into lines an
// SM may have read before (the info words, MQ states and codewords that truncation reads)
// go around L1, which SMs do not keep coherent with one another; the separate kernels load
// normally.
template <bool PERS, class T>
__device__ __forceinline__ T ldx(const T* p) {
    if constexpr (PERS) return __ldcg(p);
    else return *p;
}

// Shortest prefix >= minLen that a decoder reading 1-bits past the end decodes exactly
// up to the snapshot, never ending on 0xFF. Same arithmetic as the oracle's mq_trunc.
template <bool PERS>
__device__ uint32_t truncLen(uint4 s, const uint8_t* buf, uint32_t len, uint32_t minLen) {
    const int bp = (int)s.x;
    const uint32_t C = s.y, A = s.z & 0xFFFFu, B = s.w;
    const int CT = (int)(s.z >> 16);
    const int base = 43 - CT;
    const unsigned long long low = ((unsigned long long)B << base) + ((unsigned long long)C << 16);
    const unsigned long long high = low + ((unsigned long long)A << 16);
    unsigned long long acc = 0;
    int used = 0;
    for (int i = bp; i < (int)len; ++i) {
        const uint32_t byte = i >= 0 ? ldx<PERS>(buf + i) : 0u;
        const int sh = base - used;
        if (sh < 0) break;
        acc += (unsigned long long)byte << sh;
        const unsigned long long tail = 1ull << sh;
        const uint32_t l = (uint32_t)(i + 1);
        if (l >= minLen && byte != 0xFFu && acc + tail <= high && acc + tail > low) return l;
        used += byte == 0xFFu ? 7 : 8;
    }
    return len;
}

// s_next: by a state word's offset, its successors after an MPS that renormalises and after an
// LPS; s_init: the initial state words of Table D.7 (ZC context 0 state 4, run-length 3,
// uniform 46, every other 0).
template <int CS>
__device__ __forceinline__ void mqTables(uint2* s_next, uint32_t* s_init) {
    using M = MqLayout<CS>;
    for (int i = threadIdx.x; i < 2 * 47; i += blockDim.x) {
        const uint32_t idx = i >> 1, mps = i & 1u, e = c_mq[idx];
        s_next[(M::word(idx, mps) & kOffMask) >> 3] =
            make_uint2(M::word((e >> 18) & 63u, mps), M::word((e >> 24) & 63u, mps ^ ((e >> 17) & 1u)));
    }
    if (threadIdx.x == 0) {
        s_init[0] = M::word(0, 0);
        s_init[1] = M::word(4, 0);
        s_init[2] = M::word(3, 0);
        s_init[3] = M::word(46, 0);
    }
}

// MQ coding, a lane per block, until the queue is empty. s_mq: the CTA's MQ memory (MqLayout),
// lane0: this lane's first word in it. warpId: the warp's place among the solo warps of a
// separate MQ launch. PERS (a persistent launch): the solo blocks go to the first warps to get
// here, and each block, coded or empty, is listed for its truncation lengths when it is done.
//
// Bound by the serial chain of a block's decisions (one-frame launches) or by instruction
// issue (batched ones). 16 decisions are a straight line of code without a branch: decisions
// outside the lane's pass (before its position, after the pass's end) count as decisions in the
// null context, so every lane of the warp takes the same 16 steps. The bytes are taken out
// after them, where a byte completed in the middle of a decision made nearly every decision
// of a warp take the byte's branch as well. A round sets up 32 decisions (16 at a time: 3-5 %
// slower). On a B200, per 4K frame (154 M decisions): 0.95 ms alone (1.11 with a lane for every
// block) where the coder with the branch took 2.21, 0.50 ms of a batch of eight; the 48 blocks of a
// 64 x 64 frame 0.48 ms, where they took 1.35. CHAIN: the form with the shorter chain and a few more instructions,
// for one-frame launches (1.15 against 1.18 ms).
template <int CS, bool PERS, bool CHAIN>
__device__ __forceinline__ void mqRun(const T1Launch& P, uint32_t* s_mq, uint32_t lane0, const uint2* s_next,
                                      const uint32_t* s_init, uint32_t warpId) {
    using M = MqLayout<CS>;
    uint32_t* status = P.ctl + 1;
    const int lane = threadIdx.x & 31;
    uint8_t* const ctxBytes = reinterpret_cast<uint8_t*>(s_mq);
    uint32_t* const steps = s_mq + MQ_CTX * CS + lane0;
    const uint32_t laneByte = 4u * lane0;
    auto ctxAt = [&](uint32_t off) -> uint32_t& { return *reinterpret_cast<uint32_t*>(ctxBytes + off); };

    // Per-lane state of the block in hand: the interval A (in the upper half), the next decision
    // (pos), the 32 decisions around it (cur) and after those (nxt).
    uint32_t job = 0, pos = 0, nsym = 0, np = 0, k = 0, nextEnd = 0, A = 0;
    uint32_t laterEnd = 0;  // the pass end after nextEnd, loaded one pass ahead
    const uint8_t* sym = nullptr;
    uint4 cur[2], nxt[2];
    Coder e;
    e.cap = 0;
    bool have = false;

    auto listed = [&](uint32_t j) {
        if constexpr (PERS) {
            __threadfence();  // the block's results before its list entry
            const uint32_t slot = atomicAdd(P.work + kWTruncTail, 1u);
            atomicExch(P.work + kWList + slot, j + 1);
        }
    };
    auto load = [&](uint32_t at) {
        return at < nsym ? ldx<false>(reinterpret_cast<const uint4*>(sym + at)) : make_uint4(0, 0, 0, 0);
    };
    // the MQ state at every pass end the position has reached; false when the block is done
    auto passEnds = [&] {
        while (k < np && pos == nextEnd) {
            P.snaps[(size_t)job * kMaxPasses + k] =
                make_uint4((uint32_t)e.bp, e.C, (A >> 16) | ((uint32_t)e.CT << 16), e.B);
            ++k;
            nextEnd = laterEnd;  // loaded a pass ago: no wait here
            laterEnd = k + 1 < np ? ldx<false>(P.passEnd + (size_t)job * kMaxPasses + k + 1) : 0xFFFFFFFFu;
        }
        if (k < np) return true;
        // flush, and the codeword's length (the truncation lengths are found afterwards, a
        // warp per block)
        const uint32_t len = e.flush(A >> 16);
        if (e.overflow) atomicOr(status, kErrCodewordSpace);
        P.info[4 * (size_t)job + 3] = e.overflow ? 0u : len;
        listed(job);
        return false;
    };
    // starts block j; false when there is nothing (more) to code
    auto begin = [&](uint32_t j) {
        job = j;
        np = ldx<false>(P.info + 4 * (size_t)job + 1);
        nsym = ldx<false>(P.info + 4 * (size_t)job + 2);
        if (np == 0) {
            P.info[4 * (size_t)job + 3] = 0;
            listed(job);
            return false;
        }
        const T1Job J = P.jobs[job];
        sym = J.sym;
        e.out = J.cw;
        e.cap = J.cap;
        A = 0x80000000u;
        e.C = 0;
        e.CT = 12;
        e.bp = -1;
        e.B = 0;
        e.overflow = false;
#pragma unroll
        for (int c = 0; c < 19; ++c) s_mq[c * CS + lane0] = s_init[c == 0 ? 1 : c == 17 ? 2 : c == 18 ? 3 : 0];
        s_mq[19 * CS + lane0] = 0u;
        pos = 0;
        k = 0;
        nextEnd = ldx<false>(P.passEnd + (size_t)job * kMaxPasses);
        laterEnd = np > 1 ? ldx<false>(P.passEnd + (size_t)job * kMaxPasses + 1) : 0xFFFFFFFFu;
        cur[0] = load(0);
        cur[1] = load(16);
        nxt[0] = load(32);
        nxt[1] = load(48);
        return passEnds();
    };
    // 16 decisions, those outside the pass in the null context
    auto steps16 = [&](const uint4& c) {
        const uint32_t w[4] = {c.x, c.y, c.z, c.w};
        // decision b of the round shifted left by SHIFT (its other bytes beside it)
        auto shifted = [&](int b) {
            const int sh = 8 * (b & 3) - M::SHIFT;
            return sh >= 0 ? w[b >> 2] >> sh : w[b >> 2] << -sh;
        };
        uint32_t v = shifted(0), at = (v & M::kCtxMask) | laneByte, t = ctxAt(at);
        unsigned long long code = e.C;  // the code register with the round's shifts
        uint32_t shift = 0;
#pragma unroll
        for (int b = 0; b < MQ_ROUND; ++b) {
            const uint32_t vNext = b < MQ_ROUND - 1 ? shifted(b + 1) : 0u, atNext = (vNext & M::kCtxMask) | laneByte;
            const uint32_t ahead = b < MQ_ROUND - 1 ? ctxAt(atNext) : 0u;  // unless this decision changes it
            const uint2 succ = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(s_next) + (t & kOffMask));
            const uint32_t qe = t & 0xFFFF0000u, a = A - qe;
            const bool lps = ((v ^ t) & (1u << M::SHIFT)) != 0;
            const bool upper = (a >= qe) != lps;  // which sub-interval the decision takes
            const uint32_t q = upper ? qe : 0u;
            uint32_t n;
            if constexpr (CHAIN) {
                // the shift without a count of leading zeros, whose latency is most of the chain:
                // Qe's is in the state word, and what is left of the interval needs two at most
                const uint32_t nq = (t >> 10) & 15u;
                const uint32_t lowerA = qe << nq;
                const bool p1 = (int)a >= 0, p2 = a < 0x40000000u;
                const uint32_t upperA = p2 ? a << 2 : p1 ? a << 1 : a;
                A = upper ? upperA : lowerA;
                n = upper ? (p2 ? 2u : p1 ? 1u : 0u) : nq;
            } else {
                A = upper ? a : qe;
                n = (uint32_t)__clz((int)A);
                A <<= n;
            }
            const uint32_t renormed = lps ? succ.y : succ.x;
            const uint32_t after = lps || (int)a >= 0 ? renormed : t;  // renormalises: a below 0x8000, or the LPS
            ctxAt(at) = after;
            steps[b * CS] = q | n;
            code = (code + (q >> 16)) << n;
            shift += n;
            t = atNext == at ? after : ahead;
            at = atNext;
            v = vNext;
        }
        // The bytes the round completed, all from the register as it stands after the round. At
        // its own time a byte had not yet the carry of what was added since: the same byte
        // comes out one higher at once instead of at the next byte, except an 0xFF, after which
        // the coder keeps room for the carry instead of passing it on. A byte that may have been
        // one (it and the three bits below read 0 after a carry), and a round of more shifts
        // than the register holds, are done over from the steps, byte by byte.
        const Coder before = e;
        bool redo = shift > 32u;
        int left = redo ? 0 : (int)shift;
        uint32_t keep = 0xFFFFFFFFu;
        while (left >= e.CT) {
            left -= e.CT;
            e.C = (uint32_t)(code >> left) & keep;
            redo = redo || (e.C & 0x7FF0000u) == 0u;
            e.byteout();
            keep = 0x7FFFFFFu;
        }
        e.CT -= left;
        e.C = (uint32_t)code;
        if (keep != 0xFFFFFFFFu) e.C &= (1u << (27 - e.CT)) - 1u;
        if (redo) {
            e = before;
#pragma unroll 1
            for (int b = 0; b < MQ_ROUND; ++b) {
                const uint32_t x = steps[b * CS];
                e.C += x >> 16;
                int n = (int)(x & 31u);
                while (n >= e.CT) {
                    e.C <<= e.CT;
                    n -= e.CT;
                    e.byteout();
                }
                e.C <<= n;
                e.CT -= n;
            }
        }
    };

    // the decisions from pos to the end of its 32 or of its pass
    auto round = [&] {
        const uint32_t first = pos & ~31u, lo = pos & 31u, hi = min(32u, nextEnd - first);
        uint4 c0 = cur[0], c1 = cur[1];
        const uint32_t in = (hi == 32u ? kFull : (1u << hi) - 1u) & ~((1u << lo) - 1u);
        if (in != kFull) {
            uint32_t* const w[8] = {&c0.x, &c0.y, &c0.z, &c0.w, &c1.x, &c1.y, &c1.z, &c1.w};
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t m = spread1((in >> (4 * q)) & 0xFu) * 0xFFu;
                *w[q] = (*w[q] & m) | (kNullByte * 0x01010101u & ~m);
            }
        }
        pos = first + hi;
        if (hi == 32u) {
            cur[0] = nxt[0];
            cur[1] = nxt[1];
            nxt[0] = load(pos + 32u);
            nxt[1] = load(pos + 48u);
        }
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            if ((in >> (16 * half)) & 0xFFFFu) steps16(c0);
            c0 = c1;
        }
    };

    // A solo warp first codes its solo block (perm[0 .. solo)) on its lane 0 while the other
    // lanes wait. Then the warp takes the next 32 blocks of the order at once, a lane each,
    // and codes them until the last of them is done: the order is largest first in narrow
    // size classes, so the 32 are about the same length, and the lanes start, run and end
    // their blocks together instead of each claiming its next block at its own time (which
    // left a third of the lanes of a warp idle at any moment).
    const uint32_t solo = ldx<false>(P.ctl + 3);
    uint32_t mine = warpId;
    if constexpr (PERS) {
        if (lane == 0) mine = atomicAdd(P.work + kWSoloHead, 1u);
        mine = __shfl_sync(kFull, mine, 0);
    }
    bool alone = mine < solo;  // warp-uniform
    for (;;) {
        if (alone) {
            have = lane == 0 && begin(ldx<false>(P.perm + mine));
            alone = false;
        } else {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(P.ctl, 32u);
            base = __shfl_sync(kFull, base, 0);
            if (solo + base >= P.n) break;  // warp-uniform
            const uint32_t qi = solo + base + lane;
            have = qi < P.n && begin(ldx<false>(P.perm + qi));
        }
        while (__any_sync(kFull, have)) {
            if (have) {
                round();
                if (pos == nextEnd) have = passEnds();
            }
        }
    }
}

// MINB: CTAs per SM the registers must allow. A launch of a frame or two has fewer lanes
// than the GPU holds and runs uncapped; wide batched launches run at 6 CTAs per SM (24 frames
// of 4K served on a B200: 30.5 ms, 2 % more at 8 CTAs; 10 would spill).
template <int MINB>
__global__ void __launch_bounds__(MQ_THREADS, MINB) t1MqKernel(T1Launch P) {
    __shared__ uint2 s_next[128];
    __shared__ uint32_t s_init[4];
    __shared__ uint32_t s_mq[MQ_WORDS * MQ_THREADS];
    mqTables<MQ_THREADS>(s_next, s_init);
    __syncthreads();
    mqRun<MQ_THREADS, false, MINB == 1>(P, s_mq, threadIdx.x, s_next, s_init, blockIdx.x * (MQ_THREADS / 32) + (threadIdx.x >> 5));
}

// Truncation lengths of one block by one warp: lane q finds the shortest prefix for pass q
// from the MQ state recorded at its end, as if no earlier pass constrained it; lane 0 then
// walks the passes in order and, where a pass's shortest prefix is shorter than an earlier
// pass's length, searches again from that length (the lengths of a block never decrease).
// The last pass takes the whole codeword.
template <bool PERS>
__device__ __forceinline__ void truncJob(const T1Launch& P, uint32_t job, int lane) {
    const uint32_t np = ldx<PERS>(P.info + 4 * (size_t)job + 1), len = ldx<PERS>(P.info + 4 * (size_t)job + 3);
    if (np == 0 || len == 0) return;  // nothing coded, or an overflow already reported
    const uint8_t* cw = P.jobs[job].cw;
    const size_t base = (size_t)job * kMaxPasses;
    uint32_t c0 = 0, c1 = 0;  // the unconstrained lengths of passes lane and lane + 32
    if ((uint32_t)lane + 1 < np) c0 = truncLen<PERS>(ldx<PERS>(P.snaps + base + lane), cw, len, 1);
    if ((uint32_t)lane + 33 < np) c1 = truncLen<PERS>(ldx<PERS>(P.snaps + base + lane + 32), cw, len, 1);
    uint32_t prev = 1, mine0 = 0, mine1 = 0;
    for (uint32_t q = 0; q < np; ++q) {
        const uint32_t c = __shfl_sync(kFull, q < 32 ? c0 : c1, q & 31);
        uint32_t L = len;
        if (q + 1 < np) {
            L = c;
            if (L < prev && lane == 0) L = truncLen<PERS>(ldx<PERS>(P.snaps + base + q), cw, len, prev);
            L = __shfl_sync(kFull, L, 0);
        }
        if ((q & 31) == (uint32_t)lane) (q < 32 ? mine0 : mine1) = L;
        prev = max(prev, L);
    }
    if ((uint32_t)lane < np) P.passLen[base + lane] = mine0;
    if ((uint32_t)lane + 32 < np) P.passLen[base + lane + 32] = mine1;
}

// Kept out of the MQ kernel, whose lanes would otherwise stall on these byte reads one
// block end at a time while their warp-mates code.
constexpr int TRUNC_THREADS = 256;

__global__ void __launch_bounds__(TRUNC_THREADS) t1TruncKernel(T1Launch P) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (TRUNC_THREADS / 32);
    for (uint32_t job = blockIdx.x * (TRUNC_THREADS / 32) + (threadIdx.x >> 5); job < P.n; job += warps)
        truncJob<false>(P, job, lane);
}

// ---------------------------------------------------------------------------- one launch
__device__ __forceinline__ uint32_t ldAcquire(const uint32_t* p) {
    uint32_t x;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
    return x;
}

__device__ __forceinline__ uint32_t ldRelaxed(const uint32_t* p) {
    uint32_t x;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
    return x;
}

constexpr uint64_t kQueueWaitNs = 2000000000ull;  // a persistent launch's longest wait

// Waits until *p >= v (polling with relaxed loads, backing off from 0.25 to 8 us so that
// thousands of waiting warps leave L2 to the working ones; the caller acquires once it
// holds); gives up after limitNs (2 s in the launches) with kErrQueueWait set, so that a
// launch whose other warps stopped returns.
__device__ bool waitFor(const uint32_t* p, uint32_t v, uint32_t* status, uint64_t limitNs = kQueueWaitNs) {
    uint64_t t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    uint32_t nap = 256;
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        if (ldRelaxed(p) >= v) return true;
        __nanosleep(nap);
        nap = min(nap * 2, 8192u);
        if ((it & 63u) == 63u) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t1 - t0 > limitNs) break;
        }
    }
    atomicOr(status, kErrQueueWait);
    return false;
}

// Lane 0 waits until *p >= v, then every lane makes its own acquire load of *p: the memory
// model orders later loads after the writes that preceded the release only for the thread
// that performs the acquire, not for lanes that hear of the value from lane 0 by shuffle.
// Returns *p as every lane read it, 0 when the wait gave up (warp-uniform).
__device__ __forceinline__ uint32_t warpWaitFor(const uint32_t* p, uint32_t v, uint32_t* status, int lane,
                                                uint64_t limitNs = kQueueWaitNs) {
    const bool ok = lane == 0 ? waitFor(p, v, status, limitNs) : true;
    if (!__shfl_sync(kFull, ok, 0)) return 0u;
    return ldAcquire(p);
}

constexpr uint32_t SCAT_CHUNK = 256;  // blocks per claim of the order's scatter

// The whole Tier-1 stage in one launch, every warp through the same phases, each fed by a
// device queue: (1) context modelling, a block per claim; (2) the order (counting sort by
// decision count, most first: the warp that models the last block scans the bucket
// counters the modelling filled, every warp scatters chunks of blocks); (3) MQ coding, a
// lane per block, the heaviest blocks alone in the first warps to arrive; (4) truncation
// lengths, a warp per block in the order the blocks finished MQ coding, by every warp done
// with MQ coding. A warp waits only for work that a running warp has claimed (it reaches
// the wait after the queue it drew from ran dry), so the launch cannot deadlock whatever
// its grid and whatever runs beside it; every wait is bounded all the same. A lane reads
// what other warps wrote only after its own acquire load of the word that announced it.
// Each warp's context-modelling memory holds its lanes' MQ contexts afterwards.
__global__ void __launch_bounds__(CM_THREADS, 7) t1PersistentKernel(T1Launch P, uint32_t maxSolo) {
    struct WarpCm {
        uint32_t planes[32][32];
        uint8_t stage[STAGE];
    };
    union WarpMem {
        WarpCm cm;
        uint32_t mq[MQ_WORDS * 32];
    };
    __shared__ __align__(16) WarpMem s_w[CM_WARPS];
    __shared__ uint32_t s_hist[CM_WARPS][19];
    __shared__ uint2 s_next[128];
    __shared__ uint32_t s_init[4];
    mqTables<32>(s_next, s_init);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t* work = P.work;
    uint32_t* status = P.ctl + 1;

    // (1) context modelling
    for (;;) {
        uint32_t job = 0;
        if (lane == 0) job = atomicAdd(work + kWCmHead, 1u);
        job = __shfl_sync(kFull, job, 0);
        if (job >= P.n) break;
        const uint32_t nsym = cmJob(P, job, s_w[wid].cm.planes, s_w[wid].cm.stage, s_hist[wid], lane);
        if (lane == 0) {
            atomicAdd(work + kWHist + orderBucket(nsym), 1u);
            if (nsym >= P.soloDecisions) atomicAdd(work + kWSolo, 1u);
        }
        __threadfence();  // the block's decisions and tables before it counts as done
        __syncwarp();
        uint32_t done = 0;
        if (lane == 0) done = atomicAdd(work + kWCmDone, 1u);
        // (2) the order: bucket offsets by the warp that modelled the last block
        if (__shfl_sync(kFull, done, 0) != P.n - 1) continue;
        ldAcquire(work + kWCmDone);
        uint32_t v[4], sum = 0;
        for (int q = 0; q < 4; ++q) {
            v[q] = __ldcg(work + kWHist + 4 * lane + q);
            sum += v[q];
        }
        uint32_t run = warpScan(sum, lane) - sum;
        for (int q = 0; q < 4; ++q) {
            work[kWHist + 4 * lane + q] = run;
            run += v[q];
        }
        if (lane == 0) P.ctl[3] = min(__ldcg(work + kWSolo), maxSolo);
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(work + kWScanDone, 1u);
    }
    if (!warpWaitFor(work + kWScanDone, 1u, status, lane)) return;
    const uint32_t chunks = divUp(P.n, SCAT_CHUNK);
    for (;;) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(work + kWScatHead, 1u);
        c = __shfl_sync(kFull, c, 0);
        if (c >= chunks) break;
        const uint32_t end = min(P.n, (c + 1) * SCAT_CHUNK);
        for (uint32_t i = c * SCAT_CHUNK + lane; i < end; i += 32)
            P.perm[atomicAdd(work + kWHist + orderBucket(__ldcg(P.info + 4 * (size_t)i + 2)), 1u)] = i;
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicAdd(work + kWScatDone, 1u);
    }
    if (!warpWaitFor(work + kWScatDone, chunks, status, lane)) return;
    // (3) MQ coding, the lanes' contexts in the warp's modelling memory
    __syncwarp();
    mqRun<32, true, false>(P, s_w[wid].mq, (uint32_t)lane, s_next, s_init, 0);
    __syncwarp();
    // (4) truncation lengths, the list's entries in turn (an entry not yet written belongs
    // to a block whose MQ coding a running lane holds)
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(work + kWTruncHead, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= P.n) break;
        const uint32_t j = warpWaitFor(work + kWList + i, 1u, status, lane);
        if (j == 0) return;
        truncJob<true>(P, j - 1, lane);
    }
}

// One warp waits, as the persistent launch's warps wait, on a flag nothing sets: the
// failure-detection path of that launch (a partner warp that never announces its work)
// made to run out without a fault.
__global__ void waitSelftestKernel(const uint32_t* flag, uint32_t* status, uint64_t limitNs) {
    warpWaitFor(flag, 1u, status, (int)(threadIdx.x & 31), limitNs);
}

}  // namespace

uint32_t t1WaitSelftest(uint32_t limitMs, float* elapsedMs) {
    uint32_t* d = nullptr;  // [0] the flag, [1] the status word
    cudaEvent_t e[2] = {nullptr, nullptr};
    uint32_t h[2] = {0, 0};
    auto release = [&] {
        for (auto& x : e)
            if (x) cudaEventDestroy(x);
        if (d) cudaFree(d);
    };
    try {
        GB_CHECK(cudaMalloc(&d, 8));
        GB_CHECK(cudaMemset(d, 0, 8));
        for (auto& x : e) GB_CHECK(cudaEventCreate(&x));
        GB_CHECK(cudaEventRecord(e[0], 0));
        waitSelftestKernel<<<1, 32>>>(d, d + 1, (uint64_t)limitMs * 1000000ull);
        GB_CHECK(cudaGetLastError());
        GB_CHECK(cudaEventRecord(e[1], 0));
        GB_CHECK(cudaMemcpy(h, d, 8, cudaMemcpyDeviceToHost));
        if (elapsedMs) GB_CHECK(cudaEventElapsedTime(elapsedMs, e[0], e[1]));
    } catch (...) {
        release();
        throw;
    }
    release();
    return h[1];
}

cudaError_t kernelsLoadable() {
    cudaFuncAttributes attr;
    return cudaFuncGetAttributes(&attr, t1OrderKernel);
}

void t1Init() {
    uint32_t mq[47];
    mqTable(mq);
    GB_CHECK(cudaMemcpyToSymbol(c_mq, mq, sizeof mq));
}

// Resident CTAs per SM of the persistent kernel, queried once per device index (devices
// of different kinds in one process each get their own figure).
static int persistentOccupancy(int dev) {
    constexpr int kMaxDevices = 64;
    static std::mutex mutex;
    static int occ[kMaxDevices] = {};
    if (dev < 0 || dev >= kMaxDevices) dev = 0;
    std::lock_guard<std::mutex> lock(mutex);
    if (!occ[dev]) {
        int o = 0;
        GB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, t1PersistentKernel, CM_THREADS, 0));
        occ[dev] = max(o, 1);
    }
    return occ[dev];
}

void t1Encode(const T1Launch& launch, cudaStream_t st, cudaEvent_t* marks) {
    if (launch.n == 0) return;
    T1Launch L = launch;
    const Tuning def = defaultTuning();
    if (!L.soloDecisions) L.soloDecisions = def.soloDecisions;
    if (!L.cmCtasPerSm) L.cmCtasPerSm = (uint16_t)def.cmCtasPerSm;
    if (!L.mqCtasPerSm) L.mqCtasPerSm = (uint16_t)def.mqCtasPerSm;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (L.persistent && L.work) {
        // one CTA per resident slot (the kernel is correct with any grid; more would only wait)
        const int occ = persistentOccupancy(dev);
        const uint32_t grid = min(divUp(L.n, CM_WARPS), (uint32_t)(sms * occ));
        GB_CHECK(cudaMemsetAsync(L.work, 0, t1WorkWords(L.n) * 4, st));
        t1PersistentKernel<<<grid, CM_THREADS, 0, st>>>(L, grid * CM_WARPS / 2);
        GB_CHECK(cudaGetLastError());
        if (marks) {
            GB_CHECK(cudaEventRecord(marks[0], st));
            GB_CHECK(cudaEventRecord(marks[1], st));
        }
        return;
    }
    const uint32_t cmBlocks = min(divUp(L.n, CM_WARPS), (uint32_t)sms * L.cmCtasPerSm);
    t1CmKernel<<<cmBlocks, CM_THREADS, 0, st>>>(L);
    if (marks) GB_CHECK(cudaEventRecord(marks[0], st));
    const uint32_t warps = (uint32_t)sms * 4u;
    const bool wide = divUp(L.n, MQ_THREADS) > warps;
    uint32_t mqBlocks, maxSolo;
    if (wide) {
        // A wide (batched) launch gives each lane two blocks on average, so that lanes whose
        // blocks end early take more from the queue; blocks of soloDecisions or more are coded
        // alone, up to half the warps.
        mqBlocks = min(divUp(L.n, MQ_THREADS * 2u), (uint32_t)sms * L.mqCtasPerSm);
        maxSolo = mqBlocks * (MQ_THREADS / 32) / 2;
    } else {
        // A launch of a frame or a few is bound by its longest blocks' chains (105 cycles a
        // decision alone in a warp, 150 beside 31 others, a third more with a second warp on the
        // scheduler): one warp per scheduler while that leaves a lane at most one and a half
        // blocks, else two, and the longest blocks alone first, as many as leave a lane for every
        // other block or one for every twelve schedulers. 4K frame (25,986 blocks): 946 us; 1,105
        // with a lane for each block and so a second warp on a third of the schedulers, 1,170 with
        // no block alone, within 1 % of 946 from 16 to 96 of them alone. Two warps per scheduler
        // and one, us: 26,000 blocks of 2K frames 1,006 and 1,019, 52,000 1,196 and 1,562, 71,000
        // 1,501 and 2,067 (with a lane for each block 1,100, 1,658 and 1,838).
        const uint32_t lanes = warps * 32u;
        mqBlocks = min(divUp(L.n, MQ_THREADS / 32), (uint32_t)sms * (L.n > lanes + lanes / 2 ? 2u : 1u));
        maxSolo = max(warps / 12u, L.n < lanes ? (lanes - L.n) / 31u : 0u);
        L.soloDecisions = 1;
    }
    if (L.work) {  // over the whole GPU: a batch of frames has 100,000 blocks and more
        const uint32_t og = min(divUp(L.n, 256u), (uint32_t)sms * 2u);
        GB_CHECK(cudaMemsetAsync(L.work, 0, kT1WorkHead * 4, st));
        t1OrderCountKernel<<<og, 256, 0, st>>>(L);
        t1OrderScatterKernel<<<og, 256, 0, st>>>(L, maxSolo);
    } else {
        t1OrderKernel<<<1, 1024, 0, st>>>(L, maxSolo);
    }
    if (marks) GB_CHECK(cudaEventRecord(marks[1], st));
    if (!wide) t1MqKernel<1><<<mqBlocks, MQ_THREADS, 0, st>>>(L);
    else t1MqKernel<6><<<mqBlocks, MQ_THREADS, 0, st>>>(L);
    t1TruncKernel<<<min(divUp(L.n, (uint32_t)(TRUNC_THREADS / 32)), (uint32_t)sms * 8u), TRUNC_THREADS, 0, st>>>(L);
    GB_CHECK(cudaGetLastError());
}

}  // namespace gb
