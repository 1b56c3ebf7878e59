// Particle -> mesh mass assignment (NGP / CIC / TSC) for sm_100a.
//
// Replaces getDensity_NGP / getDensity_CIC / getDensity_TSC,
// Source/massFunctions.cpp:35-98, :678-790, :1050-1165.
//
// Pipeline (no float atomics, bitwise deterministic):
//   1. bin_count   : each CTA takes a contiguous chunk of particles and
//                    computes, per particle, the reference's FP32 home cell
//                    (bit-exact key) and the mesh bricks its stencil
//                    touches; a shared-memory histogram per CTA is added to
//                    per-brick counters.  Also lost particles, max |w|.
//   2. scan        : exclusive scan of the brick counts: every brick owns a
//                    contiguous payload range, its counter becomes its
//                    append cursor.
//   3. bin_scatter : the particles again; one 16-byte payload per touched
//                    brick (home cell relative to the brick, exact
//                    fractional offset in fixed point, weight) at the next
//                    slot of the brick's cursor (one global atomic each).
//   4. deposit     : one CTA per brick accumulates its payloads into a
//                    shared-memory tile of 64-bit fixed-point cell sums kept
//                    as two 32-bit words (32-bit shared atomics, the carry
//                    detected from the returned old value).  Integer sums do
//                    not depend on arrival order, so the result is
//                    deterministic; the tile is written once, coalesced, as
//                    FP32/FP64 (or uint32 counts for NGP).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cam_assign_device.cuh"
#include "cam_internal.h"

namespace cam {
namespace {

constexpr int kBinThreads = 1024;
constexpr int kDepositThreads = 512;
constexpr int kScatterThreads = 512;  // scatter pass: two CTAs per SM
constexpr int kSmemBricks = 16384;  // per-CTA brick histogram in shared memory (64 KB)
using namespace asg;


// Calls one(i, x, y, z, w) for the particles p0 + i, i in [0, count), the
// threads of the CTA taking consecutive particles, the next one's loads in
// flight meanwhile.  Scalar loads: 128 bytes per warp and array either way,
// and no selects to pick a particle out of a float4.  Unit weights when w is
// null.
template <typename F>
__device__ __forceinline__ void for_particles(const float *__restrict__ x, const float *__restrict__ y,
                                              const float *__restrict__ z, const float *__restrict__ w, int64_t p0,
                                              int64_t count, F &&one)
{
    const bool weighted = w != nullptr;
    int64_t i = threadIdx.x;
    float ax = 0.f, ay = 0.f, az = 0.f, aw = 1.f;
    if (i < count) {
        ax = __ldcs(x + p0 + i);
        ay = __ldcs(y + p0 + i);
        az = __ldcs(z + p0 + i);
        if (weighted) aw = __ldcs(w + p0 + i);
    }
#pragma unroll 1
    while (i < count) {
        const int64_t j = i + blockDim.x;
        float bx = 0.f, by = 0.f, bz = 0.f, bw = 1.f;
        if (j < count) {
            bx = __ldcs(x + p0 + j);
            by = __ldcs(y + p0 + j);
            bz = __ldcs(z + p0 + j);
            if (weighted) bw = __ldcs(w + p0 + j);
        }
        one((int)i, ax, ay, az, aw);
        ax = bx;
        ay = by;
        az = bz;
        aw = bw;
        i = j;
    }
}

// Adds the CTA's lost count and weight statistics, one atomic per warp.
__device__ __forceinline__ void flush_stats(unsigned long long lost_n, unsigned int wmax, unsigned int neg,
                                            unsigned int wminc, unsigned long long *__restrict__ lost,
                                            unsigned int *__restrict__ wstat)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        lost_n += __shfl_down_sync(0xffffffffu, lost_n, off);
        wmax = max(wmax, __shfl_down_sync(0xffffffffu, wmax, off));
        neg |= __shfl_down_sync(0xffffffffu, neg, off);
        wminc = max(wminc, __shfl_down_sync(0xffffffffu, wminc, off));
    }
    if ((threadIdx.x & 31) == 0) {
        if (lost_n) atomicAdd(lost, lost_n);
        if (wmax) atomicMax(wstat, wmax);
        if (neg) atomicOr(wstat + 1, 1u);  // some weight is negative
        if (wminc) atomicMax(wstat + 6, wminc);  // smallest nonzero |w|
    }
}

// Pass 1.  Block b counts the records of particles [b chunk, (b+1) chunk)
// per brick into table[brick * kCursorStride] (through a shared-memory
// histogram when SMEM, nb <= kSmemBricks), plus lost particles and the
// weight statistics.
template <int SCHEME, bool SMEM>
__global__ void __launch_bounds__(kBinThreads)
count_kernel(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
             const float *__restrict__ w, int64_t np, int64_t chunk, const __grid_constant__ AssignGeom g, int nb,
             uint32_t *__restrict__ table, unsigned long long *__restrict__ lost, unsigned int *__restrict__ wstat)
{
    extern __shared__ uint32_t hist[];
    if (SMEM) {
        for (int i = threadIdx.x; i < nb; i += blockDim.x) hist[i] = 0u;
        __syncthreads();
    }
    unsigned long long my_lost = 0;
    unsigned int my_wmax = 0, my_neg = 0, my_wminc = 0;
    const bool weighted = w != nullptr;
    const int64_t p0 = (int64_t)blockIdx.x * chunk;
    for_particles(x, y, z, w, p0, min(chunk, np - p0), [&](int, float px, float py, float pz, float wt) {
        count_one<SCHEME, SMEM>(px, py, pz, wt, weighted, g, hist, table, my_lost, my_wmax, my_neg, my_wminc);
    });
    flush_stats(my_lost, my_wmax, my_neg, my_wminc, lost, wstat);
    if (SMEM) {
        __syncthreads();
        for (int i = threadIdx.x; i < nb; i += blockDim.x)
            if (hist[i]) atomicAdd(table + (int64_t)i * kCursorStride, hist[i]);
    }
}

// Pass 3 for meshes with more bricks than a staged tile sorts (kStageBricks):
// every record takes the next slot of its brick's cursor (table, the
// exclusive scan of the counts or zero for slabs) with one global atomic.  A
// brick's records are appended contiguously by all CTAs, so its few open
// 128-byte lines fill in L2 and are written back whole.  The order of records
// inside a brick varies from run to run; the deposit's integer sums do not
// depend on it.  SLAB: records into per-brick slabs, with the weight
// statistics and lost count gathered here (no count pass).
template <int SCHEME, bool SLAB>
__global__ void __launch_bounds__(kScatterThreads, 2)
append_kernel(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
              const float *__restrict__ w, int64_t np, int64_t chunk, const __grid_constant__ AssignGeom g,
              uint32_t *__restrict__ table, uint4 *__restrict__ payload, unsigned long long *__restrict__ lost,
              unsigned int *__restrict__ wstat, uint64_t cap, unsigned int *__restrict__ ovf, uint32_t slab)
{
    unsigned long long my_lost = 0;
    unsigned int my_wmax = 0, my_neg = 0, my_wminc = 0;
    const bool weighted = w != nullptr;
    const int64_t p0 = (int64_t)blockIdx.x * chunk;
    for_particles(x, y, z, w, p0, min(chunk, np - p0), [&](int, float px, float py, float pz, float wt) {
        const unsigned long long before = my_lost;
        append_one<SCHEME, kCursorStride>(px, py, pz, wt, g, table, payload, cap, ovf, my_lost, SLAB ? slab : 0u);
        if (SLAB && weighted && my_lost == before) weight_stats(wt, my_wmax, my_neg, my_wminc);
    });
    if (SLAB) flush_stats(my_lost, my_wmax, my_neg, my_wminc, lost, wstat);
}

// Pass 3, staged: each CTA sorts a tile of particles' records by brick in
// shared memory and appends every brick's run with one cursor atomic and
// consecutive 16-byte stores.
//   1. each particle's record for its first brick goes to its stage slot; a
//      shared counter per brick gives its rank in the tile.  Particles whose
//      stencil crosses brick faces are queued;
//   2. the queue's further records (next bricks) are staged the same way,
//      by full warps; past the stage's capacity a record is appended on its
//      own, as append_kernel does;
//   3. per brick: the cursor is advanced by the tile's count (one atomic),
//      and an exclusive scan of the counts orders the stage by brick (perm);
//   4. records leave in that order: neighbouring threads write neighbouring
//      slots of a brick's run.
// Shared memory: stage [recs] 16 bytes, key and rank [recs] (18 + 14 bits),
// bricks [nb], perm [recs] 16 bits (the queue lives there before step 3).
// tile <= 8192, recs <= 16384, nb <= kStageBricks.
constexpr int kStageThreads = 1024;
constexpr int kStageBricks = 4096;
constexpr int kStagePer = kStageBricks / kStageThreads;
constexpr int kStageTile = 8192;
constexpr size_t kStageSmem = 226 * 1024;
__host__ __device__ constexpr size_t stage_bytes(int recs, int nb)
{
    return (size_t)recs * 22 + (size_t)nb * 4 + 16;
}

template <int SCHEME, bool SLAB>
__global__ void __launch_bounds__(kStageThreads, 1)
staged_kernel(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
              const float *__restrict__ w, int64_t np, int tile, int recs, const __grid_constant__ AssignGeom g, int nb,
              uint32_t *__restrict__ table, uint4 *__restrict__ payload, unsigned long long *__restrict__ lost,
              unsigned int *__restrict__ wstat, uint64_t cap, unsigned int *__restrict__ ovf, uint32_t slab)
{
    extern __shared__ __align__(16) unsigned char stage_smem[];
    __shared__ uint32_t warp_sums[kStageThreads / 32];
    __shared__ uint32_t s_queued, s_extra, s_total;
    uint4 *const stage = reinterpret_cast<uint4 *>(stage_smem);
    uint32_t *const kr = reinterpret_cast<uint32_t *>(stage + recs);  // key << 14 | rank; ~0: no record
    uint32_t *const bin = kr + recs;                                  // [nb]
    uint16_t *const perm = reinterpret_cast<uint16_t *>(bin + nb);    // [recs]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool weighted = w != nullptr;
    unsigned long long my_lost = 0;
    unsigned int my_wmax = 0, my_neg = 0, my_wminc = 0;
    const uint32_t slab_v = SLAB ? slab : 0u;
    const int per = (nb + kStageThreads - 1) / kStageThreads;  // bricks per thread in step 3
    for (int b = tid; b < nb; b += kStageThreads) bin[b] = 0u;
    if (tid == 0) s_queued = s_extra = 0u;
    __syncthreads();
    for (int64_t p0 = (int64_t)blockIdx.x * tile; p0 < np; p0 += (int64_t)gridDim.x * tile) {
        const int count = (int)min((int64_t)tile, np - p0);
        // 1. first bricks
        for_particles(x, y, z, w, p0, count, [&](int i, float px, float py, float pz, float wt) {
            const float pos[3] = {px, py, pz};
            int c[3], bl[3], cl[3];
            float t[3] = {0.f, 0.f, 0.f};
            if (!locate<SCHEME, true>(pos, g, c, t)) {
                if (SLAB) ++my_lost;
                kr[i] = ~0u;
                return;
            }
            if (SLAB && weighted) weight_stats(wt, my_wmax, my_neg, my_wminc);
            unsigned cross = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) cross |= brick_axis<SCHEME>(g, a, c[a], bl[a], cl[a]) ? 1u << a : 0u;
            const int key = (bl[0] * g.nb[1] + bl[1]) * g.nb[2] + bl[2];
            const uint32_t rank = atomicAdd(bin + key, 1u);
            stage[i] = make_uint4(pack_axis(cl[0], t[0]), pack_axis(cl[1], t[1]), pack_axis(cl[2], t[2]),
                                  __float_as_uint(wt));
            kr[i] = ((uint32_t)key << 14) | rank;
            if (SCHEME != CAM_NGP && cross) perm[atomicAdd(&s_queued, 1u)] = (uint16_t)(i | (cross << 13));
        });
        __syncthreads();
        // 2. the next bricks of the queued particles
        if (SCHEME != CAM_NGP) {
            const int nq = (int)s_queued;
            for (int q = tid; q < nq; q += kStageThreads) {
                const unsigned ent = perm[q];
                const int i = (int)(ent & 8191u);
                const unsigned cross = ent >> 13;
                const uint4 rec = stage[i];
                const int key = (int)(kr[i] >> 14);
                int bl[3], step[3];
                const int r = g.nb[2] == 1 ? key : (int)__umulhi((unsigned)key, g.kmagic[0]);
                bl[2] = key - r * g.nb[2];
                bl[0] = g.nb[1] == 1 ? r : (int)__umulhi((unsigned)r, g.kmagic[1]);
                bl[1] = r - bl[0] * g.nb[1];
                key_steps(g, bl, step);
                for (unsigned m = cross; m; m = (m - 1u) & cross) {
                    const int k = key + (m & 1u ? step[0] : 0) + (m & 2u ? step[1] : 0) + (m & 4u ? step[2] : 0);
                    const uint4 nrec = next_brick_record(g, rec, bl, m);
                    const int at = tile + (int)atomicAdd(&s_extra, 1u);
                    if (at < recs) {
                        const uint32_t rank = atomicAdd(bin + k, 1u);
                        stage[at] = nrec;
                        kr[at] = ((uint32_t)k << 14) | rank;
                    } else {
                        put_record(payload, nrec, k, atomicAdd(table + (int64_t)k * kCursorStride, 1u), slab_v, cap, ovf);
                    }
                }
            }
            __syncthreads();
        }
        // 3. cursors and the order by brick
        const int extra = min((int)s_extra, recs - tile);
        uint32_t base[kStagePer];
        {
            uint32_t cnt[kStagePer], sum = 0;
#pragma unroll
            for (int j = 0; j < kStagePer; ++j) {
                const int b = tid * per + j;
                cnt[j] = j < per && b < nb ? bin[b] : 0u;
                base[j] = cnt[j] ? atomicAdd(table + (int64_t)b * kCursorStride, cnt[j]) : 0u;
                sum += cnt[j];
            }
            uint32_t incl = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += v;
            }
            if (lane == 31) warp_sums[wid] = incl;
            __syncthreads();
            if (wid == 0) {
                const uint32_t ws = warp_sums[lane];
                uint32_t wi = ws;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, wi, off);
                    if (lane >= off) wi += v;
                }
                warp_sums[lane] = wi - ws;
                if (lane == 31) s_total = wi;
            }
            __syncthreads();
            uint32_t run = warp_sums[wid] + incl - sum;
#pragma unroll
            for (int j = 0; j < kStagePer; ++j) {
                const int b = tid * per + j;
                if (j < per && b < nb) bin[b] = run;
                run += cnt[j];
            }
        }
        __syncthreads();
        for (int i = tid; i < count; i += kStageThreads) {
            const uint32_t k = kr[i];
            if (k != ~0u) perm[bin[k >> 14] + (k & 16383u)] = (uint16_t)i;
        }
        for (int i = tile + tid; i < tile + extra; i += kStageThreads) {
            const uint32_t k = kr[i];
            perm[bin[k >> 14] + (k & 16383u)] = (uint16_t)i;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kStagePer; ++j) {
            const int b = tid * per + j;
            if (j < per && b < nb) bin[b] = base[j];
        }
        __syncthreads();
        // 4. out, in brick order
        const int total = (int)s_total;
#pragma unroll 2
        for (int i = tid; i < total; i += kStageThreads) {
            const int at = perm[i];
            const uint32_t k = kr[at];
            put_record(payload, stage[at], (int)(k >> 14), bin[k >> 14] + (k & 16383u), slab_v, cap, ovf);
        }
        __syncthreads();
        for (int b = tid; b < nb; b += kStageThreads) bin[b] = 0u;
        if (tid == 0) s_queued = s_extra = 0u;
        __syncthreads();
    }
    if (SLAB) flush_stats(my_lost, my_wmax, my_neg, my_wminc, lost, wstat);
}

// Brick starts in one CTA (nb <= kOffThreads * kOffItems): thread t scans
// the counts of bricks [t * kOffItems, (t + 1) * kOffItems) in order, the
// per-thread sums are scanned across the CTA, and every brick's start goes
// to start[b] and to its padded cursor (which held its count); start[nb] =
// *total = all records.
constexpr int kOffThreads = 1024;
constexpr int kOffItems = 16;
__global__ void __launch_bounds__(kOffThreads)
brick_offsets_kernel(uint32_t *__restrict__ padded, int nb, uint32_t *__restrict__ start, uint32_t *__restrict__ total)
{
    __shared__ uint32_t warp_sums[kOffThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int base = threadIdx.x * kOffItems;
    uint32_t v[kOffItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kOffItems; ++i) {
        v[i] = base + i < nb ? padded[(int64_t)(base + i) * kCursorStride] : 0u;
        s += v[i];
    }
    uint32_t incl = s;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += o;
    }
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const uint32_t ws = warp_sums[lane];
        uint32_t wi = ws;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, wi, off);
            if (lane >= off) wi += o;
        }
        warp_sums[lane] = wi - ws;
        if (lane == 31) {
            start[nb] = wi;
            *total = wi;
        }
    }
    __syncthreads();
    uint32_t run = warp_sums[wid] + incl - s;
#pragma unroll
    for (int i = 0; i < kOffItems; ++i) {
        if (base + i < nb) {
            start[base + i] = run;
            padded[(int64_t)(base + i) * kCursorStride] = run;
        }
        run += v[i];
    }
}

// The largest brick record count, start[b + 1] - start[b], into *out
// (atomicMax; *out zeroed before).
__global__ void __launch_bounds__(256)
brick_max_kernel(const uint32_t *__restrict__ start, int nb, unsigned int *__restrict__ out)
{
    unsigned m = 0u;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
        m = max(m, start[b + 1] - start[b]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// counts[b] = padded[b * kCursorStride] (contiguous, for the scan).
__global__ void compact_counts_kernel(const uint32_t *__restrict__ padded, int nb, uint32_t *__restrict__ counts)
{
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
        counts[b] = padded[(int64_t)b * kCursorStride];
}

// start[b] = scanned count of brick b (its first payload), start[nb] = total;
// the padded cursors start there.
__global__ void brick_starts_kernel(const uint32_t *__restrict__ scanned, int nb,
                                    const uint32_t *__restrict__ total, uint32_t *__restrict__ start,
                                    uint32_t *__restrict__ cursor)
{
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x) {
        const uint32_t v = b < nb ? scanned[b] : *total;
        start[b] = v;
        if (b < nb) cursor[(int64_t)b * kCursorStride] = v;
    }
}

// Pass 4: one CTA per brick, two CTAs of 512 threads per SM.  Bound by the
// shared-memory atomics (one per stencil cell, 3.7 wavefronts each: 32 random
// cells on 32 banks) and, for NGP and CIC, by the latency of the record
// loads.  256^3, 16.8 M weighted particles: TSC 417 -> 341 us, CIC 200 ->
// 156, NGP 136 -> 122 with the stencil on constant offsets from one address
// (508 warp instructions per 32 TSC records before; 78% issue).
template <int SCHEME, typename OutT>
__global__ void __launch_bounds__(kDepositThreads, 2)
deposit_kernel(const uint4 *__restrict__ payload, const uint32_t *__restrict__ start, uint32_t nrec,
               AssignGeom g, const unsigned int *__restrict__ wstat, int weighted,
               OutT *__restrict__ mesh, double *__restrict__ brick_sum, uint32_t slab,
               const uint32_t *__restrict__ slab_count)
{
    extern __shared__ __align__(16) uint32_t tile32[];
    __shared__ long long red[kDepositThreads / 32];
    const int B = blockIdx.x;
    const int B2 = B % g.nb[2];
    const int B1 = (B / g.nb[2]) % g.nb[1];
    const int B0 = B / (g.nb[2] * g.nb[1]);
    const int o[3] = {B0 * g.b[0], B1 * g.b[1], B2 * g.b[2]};
    const int e[3] = {min(g.b[0], g.n[0] - o[0]), min(g.b[1], g.n[1] - o[1]),
                      min(g.b[2], g.n[2] - o[2])};
    const unsigned fold = (g.nb[0] == 1 ? 1u : 0u) | (g.nb[1] == 1 ? 2u : 0u) | (g.nb[2] == 1 ? 4u : 0u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    zero_tile(tile32, e, threadIdx.x, kDepositThreads);
    __syncthreads();

    // records beyond the payload's capacity nrec were not written (overflow
    // flag); with slabs, the brick's records are the first of its slab (the
    // host keeps every slab index below 2^32)
    const uint32_t beg = slab ? (uint32_t)B * slab : min(start[B], nrec);
    const uint32_t end = slab ? beg + min(slab_count[(int64_t)B * kCursorStride], slab) : min(start[B + 1], nrec);
    const bool nonneg = !weighted || wstat[1] == 0u;
    const int s = fixed_scale(wstat, weighted, end - beg);
    // 2^s as two exact factors (s may exceed the float exponent range)
    const float f1 = scalbnf(1.0f, s / 2), f2 = scalbnf(1.0f, s - s / 2);
    deposit_records<SCHEME>(payload, beg, end, e, f1, f2, nonneg, tile32, warp, kDepositThreads / 32, lane);
    __syncthreads();

    const double sc = ldexp(1.0, -s);
    long long acc = store_tile<OutT>(tile32, o, e, g.n, fold, s, sc, mesh, warp, kDepositThreads / 32, lane);
    // Deterministic block sum of the integer cell sums.
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long tot = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += red[i];
        brick_sum[B] = ldexp((double)tot, -s);
    }
}

// Keys only (cam_cell_keys).
template <int SCHEME>
__global__ void keys_kernel(const float *__restrict__ x, const float *__restrict__ y,
                            const float *__restrict__ z, int64_t np, AssignGeom g,
                            int64_t *__restrict__ keys)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t ncell = (int64_t)g.n[0] * g.n[1] * g.n[2];
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += stride) {
        const float pos[3] = {x[p], y[p], z[p]};
        int c[3];
        keys[p] = home_cell<SCHEME>(pos, g, c)
                      ? (int64_t)c[2] + (int64_t)g.n[2] * ((int64_t)c[1] + (int64_t)g.n[1] * c[0])
                      : ncell;
    }
}

int grid_for(int64_t work, int threads)
{
    const int64_t blocks = (work + threads - 1) / threads;
    const int64_t cap = (int64_t)kNumSMs * 8;
    return (int)std::max<int64_t>(1, std::min(blocks, cap));
}

}  // namespace

AssignGeom make_geom(const cam_grid &gr, int scheme, int64_t np)
{
    AssignGeom g{};
    for (int a = 0; a < 3; ++a) {
        CAM_REQUIRE(gr.n[a] >= 1 && gr.n[a] <= (1 << 20), CAM_E_INVAL, "grid size out of range");
        CAM_REQUIRE(std::isfinite(gr.L[a]) && gr.L[a] > 0.f, CAM_E_INVAL, "box side must be > 0");
        g.n[a] = (int)gr.n[a];
        g.L[a] = gr.L[a];
        g.d[a] = gr.d[a] != 0.f ? gr.d[a] : gr.L[a] / (float)gr.n[a];
        g.mn[a] = gr.min[a];
        CAM_REQUIRE(std::isfinite(g.d[a]) && g.d[a] > 0.f, CAM_E_INVAL, "cell size must be > 0");
        CAM_REQUIRE(std::isfinite(g.mn[a]), CAM_E_INVAL, "box origin must be finite");
    }
    // Brick extents: z 32 (128-byte rows), y and x 16; shrunk (to 4) while
    // the mesh has too few bricks to fill the GPU.  TSC needs >= 3 cells
    // per brick axis unless one brick spans the axis.
    g.b[2] = std::min(g.n[2], 32);
    g.b[1] = std::min(g.n[1], 16);
    g.b[0] = std::min(g.n[0], 16);
    auto nbricks = [&]() {
        int64_t t = 1;
        for (int a = 0; a < 3; ++a) t *= (g.n[a] + g.b[a] - 1) / g.b[a];
        return t;
    };
    const int64_t want = std::min<int64_t>(4 * kNumSMs, std::max<int64_t>(1, np / 4096));
    while (nbricks() < want && (g.b[0] > 4 || g.b[1] > 4)) {
        if (g.b[0] >= g.b[1] && g.b[0] > 4) g.b[0] = (g.b[0] + 1) / 2;
        else g.b[1] = (g.b[1] + 1) / 2;
    }
    // A stencil of width <= 3 must never span three bricks: a partial last
    // brick keeps at least 2 cells (shrink the brick until it does).
    for (int a = 0; a < 3; ++a) {
        while (g.b[a] < g.n[a] && g.n[a] % g.b[a] != 0 && g.n[a] % g.b[a] < 2 && g.b[a] > 3) --g.b[a];
        g.nb[a] = (g.n[a] + g.b[a] - 1) / g.b[a];
        g.bmagic[a] = (unsigned)(((1ull << 32) + (uint64_t)g.b[a] - 1) / (uint64_t)g.b[a]);
        g.inv_d[a] = 1.0f / g.d[a];
        g.e_last[a] = g.n[a] - (g.nb[a] - 1) * g.b[a];
        g.nf[a] = (float)g.n[a];
        // home_cell divides exactly when a quotient u <= n lies within
        // 4e-7 max(u, 1) of an integer; a little more is set aside here
        g.safe[a] = 0.5f - (4.2e-7f * (float)(g.n[a] + 1) + 1e-6f);
        g.origin |= g.mn[a] != 0.0f;
    }
    for (int a = 0; a < 2; ++a)
        g.kmagic[a] = g.nb[2 - a] > 1 ? (unsigned)(((1ull << 32) + (uint64_t)g.nb[2 - a] - 1) / (uint64_t)g.nb[2 - a]) : 0u;
    (void)scheme;
    return g;
}

template <int SCHEME>
static void assign_impl(cam_ctx *ctx, const float *x, const float *y, const float *z,
                        const float *w, int64_t np, const AssignGeom &g, AssignOut &out)
{
    const int64_t nb = (int64_t)g.nb[0] * g.nb[1] * g.nb[2];
    CAM_REQUIRE(nb < (1ll << 31), CAM_E_UNSUPPORTED, "too many mesh bricks");
    // Count pass: one CTA of 1024 threads per SM (its brick histogram in
    // shared memory), contiguous chunks of >= 4096 particles.
    const int G = (int)std::max<int64_t>(1, std::min<int64_t>(kNumSMs, (np + 4095) / 4096));
    const int64_t chunk = std::max<int64_t>(1, (np + G - 1) / G);
    const bool smem_hist = nb <= kSmemBricks;
    // per-brick counters, one per 128-byte line (counts, then cursors)
    auto *table = static_cast<uint32_t *>(scratch(ctx, "asg.cursor", (size_t)nb * kCursorStride * sizeof(uint32_t)));
    auto *start = static_cast<uint32_t *>(scratch(ctx, "asg.start", (nb + 1) * sizeof(uint32_t)));
    auto *stats = static_cast<unsigned long long *>(scratch(ctx, "asg.stats", 64));
    auto *bsum = static_cast<double *>(scratch(ctx, "asg.bsum", nb * sizeof(double)));
    unsigned long long *d_lost = stats;
    unsigned int *d_wmax = reinterpret_cast<unsigned int *>(stats + 1);
    uint32_t *d_total = reinterpret_cast<uint32_t *>(stats + 2);
    unsigned int *d_ovf = reinterpret_cast<unsigned int *>(stats + 3);
    CAM_CUDA_TRY(cudaMemsetAsync(table, 0, (size_t)nb * kCursorStride * sizeof(uint32_t), ctx->stream));
    CAM_CUDA_TRY(cudaMemsetAsync(stats, 0, 64, ctx->stream));

    // Expected records per particle of a uniform catalogue: a stencil
    // crosses a face of a brick of extent b with probability (W-1)/b per
    // axis; at most two bricks per axis.
    double f = 1.0;
    uint64_t per = 1;
    for (int a = 0; a < 3; ++a) {
        if (SCHEME == CAM_NGP || g.nb[a] == 1) continue;
        f *= 1.0 + std::min(1.0, (double)(Stencil<SCHEME>::W - 1) / g.b[a]);
        per *= 2;
    }
    // Slabs (deferred jobs): every brick gets a fixed slab of the payload,
    // sized from the clumping the last exact job run of this mesh shape
    // measured (a slab that overflows makes the job rerun exactly, which
    // measures again); no count pass and no scan then, and the scatter
    // gathers the statistics.  Only while the slabs stay within twice the
    // expected records (or 2^20 records): the scatter slows as the slabs
    // spread its appends over more memory (256^3: 0.37 ms per job densely
    // packed, 0.48 in slabs of twice, 0.55 of four times the mean brick).
    // A context with an HBM budget keeps the exact path, whose payload the
    // budget was sized for.
    const double est_brick = (double)np * f / (double)nb;
    const int64_t shape = ((int64_t)g.n[0] << 32) | ((int64_t)g.n[1] << 16) | (int64_t)g.n[2];
    uint32_t slab = 0;
    if (out.defer && !ctx->sync_free && !ctx->slabs_off && !ctx->budget && np > 0) {
        const auto it = ctx->slab_clump.find(shape);
        if (it != ctx->slab_clump.end()) {
            const uint64_t cap = slab_capacity(it->second * est_brick);
            const double room = std::max(2.0 * (double)np * f, (double)(1u << 20));
            if ((double)nb * (double)cap <= room && (uint64_t)nb * cap < (1ull << 32)) slab = (uint32_t)cap;
        }
    }

    const size_t hsmem = smem_hist ? (size_t)nb * sizeof(uint32_t) : 0;
    auto count_k = smem_hist ? count_kernel<SCHEME, true> : count_kernel<SCHEME, false>;
    if (!slab) {
        smem_at_least(count_k, hsmem);
        CAM_LAUNCH_NAMED(ctx, "assign_bin_count", count_k, G, kBinThreads, hsmem, x, y, z, w, np, chunk, g, (int)nb,
                         table, d_lost, d_wmax);
        if (nb <= (int64_t)kOffThreads * kOffItems) {
            CAM_LAUNCH_NAMED(ctx, "assign_starts", brick_offsets_kernel, 1, kOffThreads, 0, table, (int)nb, start,
                             d_total);
        } else {
            auto *counts = static_cast<uint32_t *>(scratch(ctx, "asg.counts", (size_t)nb * sizeof(uint32_t)));
            const unsigned sg = (unsigned)std::min<int64_t>((nb + 256) / 256, 1024);
            CAM_LAUNCH_NAMED(ctx, "assign_starts", compact_counts_kernel, sg, 256, 0, table, (int)nb, counts);
            exclusive_scan_u32(ctx, counts, nb, d_total);
            CAM_LAUNCH_NAMED(ctx, "assign_starts", brick_starts_kernel, sg, 256, 0, counts, (int)nb, d_total, start,
                             table);
        }
        // the fullest brick, for the slabs of later deferred jobs
        if (!ctx->sync_free) {
            CAM_LAUNCH_NAMED(ctx, "assign_starts", brick_max_kernel, 64, 256, 0, start, (int)nb,
                             reinterpret_cast<unsigned int *>(stats + 5));
            out.brick_est = est_brick;
            out.brick_shape = shape;
        }
    }

    uint64_t total = 0;
    if (slab) {
        total = (uint64_t)nb * slab;
        out.n_lost = -1;
        out.n_in = -1;
    } else if (ctx->sync_free) {
        // No host round trip (stream capture): size the payload for the
        // provable bound, one record per touched brick and at most two
        // bricks per axis.  Lost count and max |w| stay on the device
        // (asg.stats) for the caller to read back with the results.
        total = (uint64_t)np * per;
        CAM_REQUIRE(total < (1ull << 32), CAM_E_UNSUPPORTED, "payload bound exceeds 2^32 records");
        out.n_lost = -1;
        out.n_in = -1;
    } else if (out.defer) {
        // No host round trip: the expected record count of a uniform
        // catalogue (a stencil crosses a face of a brick of extent b with
        // probability (W-1)/b per axis) with a 25% margin, never below what
        // this context used before nor above the provable bound.  The
        // scatter flags records past it; the caller then reruns.
        const uint64_t bound = (uint64_t)np * per;
        uint64_t est = (uint64_t)((double)np * f * 1.25) + 65536;
        est = std::min(bound, std::max(est, ctx->asg_cap));
        total = std::min<uint64_t>(est, 0xffffffffull);
        ctx->asg_cap = std::max(ctx->asg_cap, total);
        out.n_lost = -1;
        out.n_in = -1;
    } else {
        // Payload size and diagnostics back to the host (one synchronisation),
        // with the fullest brick's record count for later slabs.
        unsigned long long hstats[6] = {0, 0, 0, 0, 0, 0};
        CAM_CUDA_TRY(cudaMemcpyAsync(hstats, stats, sizeof(hstats), cudaMemcpyDeviceToHost, ctx->stream));
        CAM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        total = (uint32_t)(hstats[2] & 0xffffffffu);
        ctx->asg_cap = std::max<uint64_t>(ctx->asg_cap, total);  // deferred runs size from it
        out.brick_max = hstats[5] & 0xffffffffu;
        const unsigned int wmax_bits = (unsigned int)(hstats[1] & 0xffffffffu);
        CAM_REQUIRE(!w || wmax_bits < 0x7f800000u, CAM_E_NONFINITE, "a particle weight is NaN or infinite");
        out.n_lost = (int64_t)hstats[0];
        out.n_in = np - out.n_lost;
    }

    uint4 *payload = static_cast<uint4 *>(scratch(ctx, "asg.payload", std::max<size_t>(total, 1) * sizeof(uint4)));
    if (nb <= kStageBricks) {
        // Tiles as large as the stage holds with the expected records (15%
        // margin on the extra ones), split evenly over the SMs.
        const int recs = (int)std::min<size_t>(16384, (kStageSmem - 16 - (size_t)nb * 4) / 22);
        const double room = (double)recs / (1.0 + 1.15 * (f - 1.0));
        const int64_t most = std::max<int64_t>(1024, std::min<int64_t>(kStageTile, (int64_t)room));
        const int64_t rounds = std::max<int64_t>(1, (np + kNumSMs * most - 1) / (kNumSMs * most));
        const int64_t even = (np + kNumSMs * rounds - 1) / (kNumSMs * rounds);
        const int tile = (int)std::min<int64_t>(most, std::max<int64_t>(1024, (even + 31) & ~(int64_t)31));
        const int64_t tiles = (np + tile - 1) / tile;
        const unsigned grid_s = (unsigned)std::max<int64_t>(1, std::min<int64_t>(kNumSMs, tiles));
        const size_t ssmem = stage_bytes(recs, (int)nb);
        auto k = slab ? staged_kernel<SCHEME, true> : staged_kernel<SCHEME, false>;
        smem_at_least(k, ssmem);
        CAM_LAUNCH_NAMED(ctx, "assign_bin_scatter", k, grid_s, kStageThreads, ssmem, x, y, z, w, np, tile, recs, g,
                         (int)nb, table, payload, d_lost, d_wmax, total, d_ovf, slab);
    } else {
        const int G2 = (int)std::max<int64_t>(1, std::min<int64_t>(2 * kNumSMs, (np + 4095) / 4096));
        const int64_t chunk2 = std::max<int64_t>(1, (np + G2 - 1) / G2);
        auto k = slab ? append_kernel<SCHEME, true> : append_kernel<SCHEME, false>;
        CAM_LAUNCH_NAMED(ctx, "assign_bin_scatter", k, G2, kScatterThreads, 0, x, y, z, w, np, chunk2, g, table, payload,
                         d_lost, d_wmax, total, d_ovf, slab);
    }

    const size_t smem = (size_t)tile_words(g.b[0]) * sizeof(uint32_t);
    const int weighted = w != nullptr;
    auto launch_dep = [&](auto kern, auto *mesh) {
        smem_at_least(kern, smem);
        CAM_LAUNCH_NAMED(ctx, "assign_deposit", kern, (unsigned)nb, kDepositThreads, smem, payload, start,
                         (uint32_t)std::min<uint64_t>(total, 0xffffffffull), g, d_wmax, weighted, mesh, bsum, slab,
                         table);
    };
    if (out.precision == CAM_F32)
        launch_dep(deposit_kernel<SCHEME, float>, static_cast<float *>(out.mesh));
    else if (out.precision == CAM_F64)
        launch_dep(deposit_kernel<SCHEME, double>, static_cast<double *>(out.mesh));
    else
        launch_dep(deposit_kernel<SCHEME, uint32_t>, static_cast<uint32_t *>(out.mesh));
    // out.d_sum[0] = sum of the mesh, out.d_sum[1] = mean per cell
    if (out.d_sum) reduce_sum_f64(ctx, bsum, nb, out.d_sum, (double)g.n[0] * g.n[1] * g.n[2]);
}

unsigned long long *assign_stats(cam_ctx *ctx)
{
    return static_cast<unsigned long long *>(scratch(ctx, "asg.stats", 64));
}

void assign_device(cam_ctx *ctx, const float *x, const float *y, const float *z,
                   const float *w, int64_t np, const cam_grid &grid, int scheme, AssignOut &out)
{
    CAM_REQUIRE(np >= 0, CAM_E_INVAL, "negative particle count");
    CAM_REQUIRE(np == 0 || (x && y && z), CAM_E_INVAL, "null particle coordinates");
    CAM_REQUIRE(np < (1ll << 31), CAM_E_UNSUPPORTED, "more than 2^31 particles per call");
    const AssignGeom g = make_geom(grid, scheme, np);
    if (out.precision == -1)
        CAM_REQUIRE(scheme == CAM_NGP && w == nullptr, CAM_E_INVAL, "integer counts need unweighted NGP");
    switch (scheme) {
    case CAM_NGP: assign_impl<CAM_NGP>(ctx, x, y, z, w, np, g, out); break;
    case CAM_CIC: assign_impl<CAM_CIC>(ctx, x, y, z, w, np, g, out); break;
    case CAM_TSC: assign_impl<CAM_TSC>(ctx, x, y, z, w, np, g, out); break;
    default: throw Error{CAM_E_INVAL, "unknown mass assignment scheme"};
    }
}

void cell_keys_device(cam_ctx *ctx, const float *x, const float *y, const float *z, int64_t np,
                      const cam_grid &grid, int scheme, int64_t *keys)
{
    const AssignGeom g = make_geom(grid, scheme, np);
    if (np == 0) return;
    const int gb = grid_for(np, 256);
    switch (scheme) {
    case CAM_NGP: CAM_LAUNCH(ctx, keys_kernel<CAM_NGP>, gb, 256, 0, x, y, z, np, g, keys); break;
    case CAM_CIC: CAM_LAUNCH(ctx, keys_kernel<CAM_CIC>, gb, 256, 0, x, y, z, np, g, keys); break;
    case CAM_TSC: CAM_LAUNCH(ctx, keys_kernel<CAM_TSC>, gb, 256, 0, x, y, z, np, g, keys); break;
    default: throw Error{CAM_E_INVAL, "unknown mass assignment scheme"};
    }
}

}  // namespace cam
