// Particle -> mesh mass assignment (NGP / CIC / TSC) for sm_100a.
//
// Replaces getDensity_NGP / getDensity_CIC / getDensity_TSC,
// Source/massFunctions.cpp:35-98, :678-790, :1050-1165.
//
// Pipeline (no float atomics, bitwise deterministic):
//   1. count   : per particle, the reference's FP32 home cell (bit-exact key)
//                and the mesh bricks its stencil touches, counted per brick;
//                lost particles, weight statistics.  An exclusive scan gives
//                every brick its range of the payload.  Deferred runs skip
//                this and give every brick a slab (see assign_impl).
//   2. scatter : the particles again; one 16-byte record per touched brick
//                (home cell relative to the brick, exact fractional offset
//                in fixed point, weight), sorted by brick within a tile in
//                shared memory and appended in runs; meshes with more bricks
//                than a tile counts sort by super-brick first (sort_kernel).
//   3. deposit : one CTA per brick accumulates its records into a
//                shared-memory tile of 64-bit fixed-point cell sums kept
//                as two 32-bit words (32-bit shared atomics, the carry
//                detected from the returned old value).  Integer sums do
//                not depend on arrival order, so the result is
//                deterministic; the tile is written once, coalesced, as
//                FP32/FP64 (or uint32 counts for NGP).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cam_assign_device.cuh"
#include "cam_internal.h"

namespace cam {
namespace {

constexpr int kBinThreads = 1024;
constexpr int kDepositThreads = 640;  // two CTAs per SM in 48 registers (512: TSC 333 -> 342 us at 256^3, NGP 101 -> 105)
constexpr int kScatterThreads = 512;  // scatter pass: two CTAs per SM
constexpr int kSmemBricks = 16384;  // per-CTA brick histogram in shared memory (64 KB)
using namespace asg;


// Calls one(i, x, y, z, w) for the particles p0 + i, i in [0, count), the
// NT threads of the CTA taking consecutive particles, two per iteration with
// all their loads ahead of the work.  Scalar loads: 128 bytes per warp and
// array either way, and no selects to pick a particle out of a float4.  Unit
// weights when w is null.
template <int NT, typename F>
__device__ __forceinline__ void for_particles(const float *__restrict__ x, const float *__restrict__ y,
                                              const float *__restrict__ z, const float *__restrict__ w, int64_t p0,
                                              int count, F &&one)
{
    x += p0;
    y += p0;
    z += p0;
    if (w) w += p0;
    int i = threadIdx.x;
#pragma unroll 1
    for (; i + NT < count; i += 2 * NT) {
        const float ax = __ldcs(x + i), ay = __ldcs(y + i), az = __ldcs(z + i);
        const float bx = __ldcs(x + i + NT), by = __ldcs(y + i + NT), bz = __ldcs(z + i + NT);
        float aw = 1.0f, bw = 1.0f;
        if (w) {
            aw = __ldcs(w + i);
            bw = __ldcs(w + i + NT);
        }
        one(i, ax, ay, az, aw);
        one(i + NT, bx, by, bz, bw);
    }
    if (i < count) one(i, __ldcs(x + i), __ldcs(y + i), __ldcs(z + i), w ? __ldcs(w + i) : 1.0f);
}

// Adds the CTA's lost count and weight statistics, one atomic per warp.
__device__ __forceinline__ void flush_stats(unsigned int lost_n, const WeightStats &ws,
                                            unsigned long long *__restrict__ lost, unsigned int *__restrict__ wstat)
{
    lost_n = __reduce_add_sync(0xffffffffu, lost_n);
    const unsigned wmax = __reduce_max_sync(0xffffffffu, ws.wmax);
    const unsigned neg = __reduce_or_sync(0xffffffffu, ws.neg());
    const unsigned wminc = __reduce_max_sync(0xffffffffu, ws.wminc());
    if ((threadIdx.x & 31) == 0) {
        if (lost_n) atomicAdd(lost, (unsigned long long)lost_n);
        if (wmax) atomicMax(wstat, wmax);
        if (neg) atomicOr(wstat + 1, 1u);  // some weight is negative
        if (wminc) atomicMax(wstat + 6, wminc);  // smallest nonzero |w|
    }
}

// Pass 1.  Block b counts the records of particles [b chunk, (b+1) chunk)
// per brick into table[brick * g.cstride] (through a shared-memory
// histogram when SMEM, nb <= kSmemBricks), plus lost particles and the
// weight statistics.
template <int SCHEME, bool SMEM>
__global__ void __launch_bounds__(kBinThreads)
count_kernel(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
             const float *__restrict__ w, int64_t np, unsigned chunk, const __grid_constant__ AssignGeom g, int nb,
             uint32_t *__restrict__ table, unsigned long long *__restrict__ lost, unsigned int *__restrict__ wstat)
{
    chain_begin();
    extern __shared__ uint32_t hist[];
    if (SMEM) {
        for (int i = threadIdx.x; i < nb; i += kBinThreads) hist[i] = 0u;
        __syncthreads();
    }
    unsigned int my_lost = 0;
    WeightStats ws;
    const bool weighted = w != nullptr;
    const int64_t p0 = (int64_t)blockIdx.x * chunk;
    const int count = (int)max((int64_t)0, min((int64_t)chunk, np - p0));
    for_particles<kBinThreads>(x, y, z, w, p0, count, [&](int, float px, float py, float pz, float wt) {
        count_one<SCHEME, SMEM>(px, py, pz, wt, weighted, g, hist, table, my_lost, ws);
    });
    flush_stats(my_lost, ws, lost, wstat);
    if (SMEM) {
        __syncthreads();
        for (int i = threadIdx.x; i < nb; i += kBinThreads)
            if (hist[i]) atomicAdd(table + (int64_t)i * g.cstride, hist[i]);
    }
}

// Pass 3 for meshes with more bricks than a staged tile counts (kStageBins):
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
              const float *__restrict__ w, int64_t np, unsigned chunk, const __grid_constant__ AssignGeom g,
              uint32_t *__restrict__ table, uint4 *__restrict__ payload, unsigned long long *__restrict__ lost,
              unsigned int *__restrict__ wstat, uint64_t cap, unsigned int *__restrict__ ovf, uint32_t slab)
{
    chain_begin();
    unsigned int my_lost = 0;
    WeightStats ws;
    const bool weighted = w != nullptr;
    const int64_t p0 = (int64_t)blockIdx.x * chunk;
    const int count = (int)max((int64_t)0, min((int64_t)chunk, np - p0));
    for_particles<kScatterThreads>(x, y, z, w, p0, count, [&](int, float px, float py, float pz, float wt) {
        const bool in = append_one<SCHEME>(px, py, pz, wt, g, table, payload, cap, ovf, SLAB ? slab : 0u);
        if (SLAB && !in) ++my_lost;
        if (SLAB && in && weighted) ws.add(wt);
    });
    if (SLAB) flush_stats(my_lost, ws, lost, wstat);
}

// ---- staged scatter ---------------------------------------------------------
// A CTA sorts a tile of particles by bin in shared memory and appends every
// bin's run with one cursor atomic and consecutive 16-byte stores.
//   LEVEL 0: particles straight into bricks (bins: all bricks);
//   LEVEL 1: particles (x, y, z, w) into super-bricks, boxes of s.gs bricks,
//            by an approximate home cell; anything outside the box or not
//            finite goes to a last bin (bins: s.count + 1);
//   LEVEL 2: the particles of one super-brick into bricks (bins: its bricks
//            and one more on every side); a brick outside them and the last
//            bin's particles are appended one by one.
// One level costs a cursor atomic and a run of a few records per brick and
// tile (4.6 records at 256^3 with tiles of 8192); two levels write the
// particles once more but both in long runs.  16.8 M particles onto 256^3
// (2048 bricks), NGP, CIC, TSC: one level 216, 284, 325 us, two levels 316,
// 410, 443, record by record 345, 441, 530 (one level 190, 271, 306 with the
// next tile's particles prefetched).  134 M CIC particles onto 512^3 (16384
// bricks, more than a tile counts): two levels 3.09 ms, record by record 4.64.
// Steps of a tile:
//   1. each particle's record for its first brick (LEVEL 1: the particle)
//      goes to its stage slot, and a shared counter per bin gives its rank
//      among the tile's.  Particles whose stencil crosses brick faces are
//      queued;
//   2. the queue's further records (next bricks) are staged the same way,
//      by full warps; past the stage's capacity a record is appended on its
//      own, as append_kernel does;
//   3. per bin the cursor is advanced by the tile's count (one atomic, its
//      latency behind the next steps), and an exclusive scan of the counts
//      gives the bin's place in the order;
//   4. slot and bin of every record are written to its place in the order
//      (over its bin and rank, which every thread has read by then);
//   5. records leave in that order: neighbouring threads write neighbouring
//      slots of a bin's run.
// What bounds it is the shared-memory pipe (two passes of 16 bytes per record
// and a random 4-byte access per count, rank and place) and the instructions
// of step 1.  Shared memory: stage [recs] 16 bytes, bins, order [recs] 4 bytes
// (bin << 14 | rank, then bin << 14 | slot), the queue, LEVEL 2 the tile starts.
constexpr int kStageBins = 4096;   // bins of a tile sort, LEVEL 0
constexpr int kMaxSupers = 1023;
constexpr int kMaxLocal = 1024;    // bricks around one super-brick, LEVEL 2 (10 bits in the queue)
constexpr int kStageTile = 8192;   // particles per tile (13 bits in the queue)

// One CTA of 1024 threads per SM for LEVEL 0, whose runs are the longer the
// larger its tile (two of 512: 216 -> 221, 284 -> 296, 325 -> 335 us for NGP,
// CIC, TSC as above); four of 256 for the others, whose runs are long anyway
// (two of 512 at 512^3: LEVEL 1 0.98 -> 0.95 ms, LEVEL 2 2.16 -> 2.14).
constexpr int stage_threads(int level) { return level == 0 ? 1024 : 256; }
constexpr int stage_ctas(int level) { return 1024 / stage_threads(level); }
constexpr size_t stage_budget(int level) { return (226 / stage_ctas(level) - 1) * 1024; }
// Two levels where one level's tiles cannot count the bricks, from a million
// particles on.  Uniform particles in slabs, two levels against record by
// record: 384^3 CIC 260 and 236 us at 1 M, 325 and 308 at 4 M; 512^3 TSC 505
// and 495 at 1 M, 605 and 591 at 4 M.  Both sides cross between 4 M and 30 M
// (512^3, 67 M, counted exactly: CIC 2.94 and 3.32 ms, TSC 3.75 and 4.34), so
// the line lies low: up to a tenth of a call is lost below the crossing.
constexpr int64_t kTwoLevelParticles = 1000000;
// bytes besides the 20 per record
inline size_t stage_fixed(int level, int nbins)
{
    return (size_t)nbins * 4 + (level == 2 ? (size_t)nbins * 8 + (kMaxSupers + 2) * 4 : 0);
}

// Super-bricks: gs bricks per axis (the last may have fewer), ns per axis.
struct SuperGeom {
    int gs[3], ns[3];
    int count;       // ns[0] ns[1] ns[2]
    int D[3];        // LEVEL 2 bins per axis: gs + 2, or all bricks when ns = 1
    float inv[3];    // 1 / (cells per super-brick)
    unsigned dmagic[2];  // ceil(2^32 / D[2]), ceil(2^32 / D[1])
    uint32_t cap;    // slots per super-brick (slabs), 0: dense ranges from beg
};

struct SortArgs {
    const float *x, *y, *z, *w;  // LEVEL 0 and 1
    int64_t np;
    int tile, recs, nbins;
    uint32_t *cursor;            // of the bricks (LEVEL 0, 2)
    uint32_t *scursor;           // of the super-bricks (LEVEL 1, 2)
    const uint32_t *sbeg;        // dense super-brick ranges [count + 2]
    float4 *part;                // particles by super-brick
    uint64_t part_cap;
    uint4 *payload;
    uint64_t cap;
    uint32_t slab;
    unsigned long long *lost;
    unsigned int *wstat, *ovf;
    int weighted;
};

__device__ __forceinline__ int super_of(const AssignGeom &g, const SuperGeom &s, float px, float py, float pz)
{
    const float p[3] = {px, py, pz};
    int c[3];
    bool in = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float u = (p[a] - g.mn[a]) * g.inv_d[a];
        in = in && u >= 0.0f && u < g.nf[a];
        c[a] = min((int)(u * s.inv[a]), s.ns[a] - 1);
    }
    return in ? (c[0] * s.ns[1] + c[1]) * s.ns[2] + c[2] : s.count;
}

// First slot of super-brick k and the particles it holds.
__device__ __forceinline__ void super_range(const SortArgs &A, const SuperGeom &s, int k, uint32_t &beg, uint32_t &cnt)
{
    if (s.cap) {
        beg = (uint32_t)k * s.cap;
        cnt = min(A.scursor[k], k == s.count ? (uint32_t)(A.part_cap - beg) : s.cap);
    } else {
        beg = A.sbeg[k];
        cnt = A.sbeg[k + 1] - beg;
    }
}

// Tiles of LEVEL 2: tstart[k] = tiles of the super-bricks before k, for k in
// [0, count + 1]; returns all tiles.  Called by every thread.
template <int NT>
__device__ __forceinline__ int tile_starts(const SortArgs &A, const SuperGeom &s, uint32_t *tstart, uint32_t *warp_sums)
{
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int PER = (kMaxSupers + 1 + NT - 1) / NT;
    uint32_t n[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int k = tid * PER + j;
        n[j] = 0;
        if (k <= s.count) {
            uint32_t beg, cnt;
            super_range(A, s, k, beg, cnt);
            n[j] = (cnt + (uint32_t)A.tile - 1u) / (uint32_t)A.tile;
        }
        sum += n[j];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
    }
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (int k = 0; k < wid; ++k) before += warp_sums[k];
    uint32_t run = before + incl - sum;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int k = tid * PER + j;
        if (k <= s.count) tstart[k] = run;
        run += n[j];
        if (k == s.count) tstart[k + 1] = run;
    }
    __syncthreads();
    return (int)tstart[s.count + 1];
}

// The super-brick of tile t: the last k with tstart[k] <= t (and a tile).
__device__ __forceinline__ int super_of_tile(const uint32_t *tstart, int count, int t)
{
    int lo = 0, hi = count;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tstart[mid] <= (uint32_t)t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// First brick of super-brick k's bins along each axis.
__device__ __forceinline__ void local_origin(const SuperGeom &s, int k, int o[3])
{
    const int c2 = k % s.ns[2], r = k / s.ns[2];
    const int c1 = r % s.ns[1], c0 = r / s.ns[1];
    o[0] = s.ns[0] == 1 ? 0 : c0 * s.gs[0] - 1;
    o[1] = s.ns[1] == 1 ? 0 : c1 * s.gs[1] - 1;
    o[2] = s.ns[2] == 1 ? 0 : c2 * s.gs[2] - 1;
}
// Brick coordinate bl as a coordinate of those bins (>= D: not among them),
// and back.
__device__ __forceinline__ int to_local(const AssignGeom &g, int a, int o, int bl)
{
    const int l = bl - o;
    return l < 0 ? l + g.nb[a] : (l >= g.nb[a] ? l - g.nb[a] : l);
}
__device__ __forceinline__ int to_brick(const AssignGeom &g, int a, int o, int l)
{
    int b = o + l;
    if (b < 0) b += g.nb[a];
    if (b >= g.nb[a]) b -= g.nb[a];
    return b;
}

__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// As for_particles, for particles stored as (x, y, z, w).
template <int NT, typename F>
__device__ __forceinline__ void for_packed(const float4 *__restrict__ in, int count, F &&one)
{
    int i = threadIdx.x;
#pragma unroll 1
    for (; i + NT < count; i += 2 * NT) {
        const float4 a = __ldcs(in + i), b = __ldcs(in + i + NT);
        one(i, a.x, a.y, a.z, a.w);
        one(i + NT, b.x, b.y, b.z, b.w);
    }
    if (i < count) {
        const float4 a = __ldcs(in + i);
        one(i, a.x, a.y, a.z, a.w);
    }
}

template <int SCHEME, bool SLAB, int LEVEL>
__global__ void __launch_bounds__(stage_threads(LEVEL), stage_ctas(LEVEL))
sort_kernel(const __grid_constant__ SortArgs A, const __grid_constant__ AssignGeom g, const __grid_constant__ SuperGeom s)
{
    chain_begin();
    constexpr int NT = stage_threads(LEVEL);
    constexpr int MAXBINS = LEVEL == 0 ? kStageBins : (LEVEL == 1 ? kMaxSupers + 1 : kMaxLocal);
    constexpr int PER = (MAXBINS + NT - 1) / NT;
    constexpr uint32_t kNone = ~0u;
    constexpr int MAXREC = ((int)stage_budget(LEVEL) / 20 + NT - 1) / NT;  // records per thread
    extern __shared__ __align__(16) unsigned char stage_smem[];
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t s_queued, s_extra, s_total;
    const int nbins = A.nbins, tile = A.tile, recs = A.recs;
    uint4 *const stage = reinterpret_cast<uint4 *>(stage_smem);
    uint32_t *const bin = reinterpret_cast<uint32_t *>(stage + recs);  // [nbins]
    uint32_t *const brick = bin + nbins;                               // LEVEL 2 [nbins]: the bin's brick
    uint32_t *const limit = brick + nbins;                             // LEVEL 2 [nbins]: end of its slots
    uint32_t *const tstart = limit + nbins;                            // LEVEL 2 [kMaxSupers + 2]
    uint32_t *const order = LEVEL == 2 ? tstart + kMaxSupers + 2 : bin + nbins;  // [recs]
    uint16_t *const queue = reinterpret_cast<uint16_t *>(order + recs);          // [tile], LEVEL 0 and 2
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t slab = SLAB ? A.slab : 0u;
    unsigned int my_lost = 0;
    WeightStats ws;
    const int per = (nbins + NT - 1) / NT;  // bins per thread in step 3
    for (int b = tid; b < nbins; b += NT) bin[b] = 0u;
    if (tid == 0) s_queued = s_extra = 0u;
    __syncthreads();
    int64_t tiles;
    int64_t t0, t1, tstep;
    if (LEVEL == 2) {  // consecutive tiles: the super-brick changes rarely
        tiles = tile_starts<NT>(A, s, tstart, warp_sums);
        const int64_t each = (tiles + gridDim.x - 1) / gridDim.x;
        t0 = blockIdx.x * each;
        t1 = min(tiles, t0 + each);
        tstep = 1;
    } else {
        tiles = (A.np + tile - 1) / tile;
        t0 = blockIdx.x;
        t1 = tiles;
        tstep = gridDim.x;
    }
    int sup = -1, org[3] = {0, 0, 0};
    for (int64_t t = t0; t < t1; t += tstep) {
        int count;
        int64_t p0 = 0;
        if (LEVEL == 2) {
            int k = sup < 0 ? super_of_tile(tstart, s.count, (int)t) : sup;
            while (tstart[k + 1] <= (uint32_t)t) ++k;
            uint32_t beg, cnt;
            super_range(A, s, k, beg, cnt);
            const uint32_t off = ((uint32_t)t - tstart[k]) * (uint32_t)tile;
            p0 = (int64_t)beg + off;
            count = (int)min((uint32_t)tile, cnt - off);
            if (k == s.count) {  // outside the box, wrapped or lost: one by one
                for_packed<NT>(A.part + p0, count, [&](int, float px, float py, float pz, float wt) {
                    const bool in = append_one<SCHEME>(px, py, pz, wt, g, A.cursor, A.payload, A.cap,
                                                                      A.ovf, slab);
                    if (SLAB && !in) ++my_lost;
                    if (SLAB && in && A.weighted) ws.add(wt);
                });
                sup = k;
                continue;
            }
            if (k != sup) {
                sup = k;
                local_origin(s, k, org);
                for (int b = tid; b < nbins; b += NT) {
                    const int l2 = b % s.D[2], r = b / s.D[2];
                    const int gk = (to_brick(g, 0, org[0], r / s.D[1]) * g.nb[1] + to_brick(g, 1, org[1], r % s.D[1])) *
                                       g.nb[2] + to_brick(g, 2, org[2], l2);
                    brick[b] = (uint32_t)gk;
                    limit[b] = slab ? (uint32_t)(gk + 1) * slab : (uint32_t)min(A.cap, (uint64_t)0xffffffffu);
                }
                __syncthreads();
            }
        } else {
            p0 = t * tile;
            count = (int)min((int64_t)tile, A.np - p0);
        }
        // 1. first bins
        auto first = [&](int i, float px, float py, float pz, float wt) {
            if (LEVEL == 1) {
                const int key = super_of(g, s, px, py, pz);
                const uint32_t rank = atomicAdd(bin + key, 1u);
                stage[i] = make_uint4(__float_as_uint(px), __float_as_uint(py), __float_as_uint(pz), __float_as_uint(wt));
                order[i] = ((uint32_t)key << 14) | rank;
                return;
            }
            int c[3], bl[3], cl[3];
            uint32_t off[3];
            if (!locate<SCHEME, true>(px, py, pz, g, c, off)) {
                if (SLAB) ++my_lost;
                order[i] = kNone;
                return;
            }
            if (SLAB && A.weighted) ws.add(wt);
            unsigned cross = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) cross |= brick_axis<SCHEME>(g, a, c[a], bl[a], cl[a]) ? 1u << a : 0u;
            int key;
            if (LEVEL == 0) {
                key = (bl[0] * g.nb[1] + bl[1]) * g.nb[2] + bl[2];
            } else {
                const int l0 = to_local(g, 0, org[0], bl[0]), l1 = to_local(g, 1, org[1], bl[1]),
                          l2 = to_local(g, 2, org[2], bl[2]);
                if (l0 >= s.D[0] || l1 >= s.D[1] || l2 >= s.D[2]) {
                    order[i] = kNone;
                    append_one<SCHEME>(px, py, pz, wt, g, A.cursor, A.payload, A.cap, A.ovf, slab);
                    return;
                }
                key = (l0 * s.D[1] + l1) * s.D[2] + l2;
            }
            const uint32_t rank = atomicAdd(bin + key, 1u);
            stage[i] = make_uint4(pack_axis(cl[0], off[0]), pack_axis(cl[1], off[1]), pack_axis(cl[2], off[2]),
                                  __float_as_uint(wt));
            order[i] = ((uint32_t)key << 14) | rank;
            if (SCHEME != CAM_NGP && cross) queue[atomicAdd(&s_queued, 1u)] = (uint16_t)(i | (cross << 13));
        };
        if (LEVEL == 2) for_packed<NT>(A.part + p0, count, first);
        else for_particles<NT>(A.x, A.y, A.z, A.w, p0, count, first);
        __syncthreads();
        // 2. the next bricks of the queued particles
        if (LEVEL != 1 && SCHEME != CAM_NGP) {
            const int nq = (int)s_queued;
            const int d1 = LEVEL == 0 ? g.nb[1] : s.D[1], d2 = LEVEL == 0 ? g.nb[2] : s.D[2];
            for (int q = tid; q < nq; q += NT) {
                const unsigned ent = queue[q];
                const int i = (int)(ent & 8191u);
                const unsigned cross = ent >> 13;
                const uint4 rec = stage[i];
                const int key = (int)(order[i] >> 14);
                const int r = d2 == 1 ? key : (int)__umulhi((unsigned)key, LEVEL == 0 ? g.kmagic[0] : s.dmagic[0]);
                int l[3], bl[3], step[3];
                l[2] = key - r * d2;
                l[0] = d1 == 1 ? r : (int)__umulhi((unsigned)r, LEVEL == 0 ? g.kmagic[1] : s.dmagic[1]);
                l[1] = r - l[0] * d1;
                unsigned outside = 0u;  // LEVEL 2: axes along which the next brick is not among the bins
                if (LEVEL == 0) {
                    bl[0] = l[0];
                    bl[1] = l[1];
                    bl[2] = l[2];
                    key_steps(g, bl, step);
                } else {
                    const int stride[3] = {d1 * d2, d2, 1};
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        bl[a] = to_brick(g, a, org[a], l[a]);
                        step[a] = stride[a];
                        if (l[a] + 1 == s.D[a]) {
                            step[a] = -l[a] * stride[a];  // every brick of the axis is a bin: periodic
                            if (s.ns[a] > 1) outside |= 1u << a;
                        }
                    }
                }
#pragma unroll 1
                for (unsigned m = cross; m; m = (m - 1u) & cross) {
                    const uint4 nrec = next_brick_record(g, rec, bl, m);
                    int k = key + (m & 1u ? step[0] : 0) + (m & 2u ? step[1] : 0) + (m & 4u ? step[2] : 0);
                    int at = recs;
                    if (!(m & outside)) at = tile + (int)atomicAdd(&s_extra, 1u);
                    if (at < recs) {
                        const uint32_t rank = atomicAdd(bin + k, 1u);
                        stage[at] = nrec;
                        order[at] = ((uint32_t)k << 14) | rank;
                    } else {
                        if (LEVEL == 2) {
                            int gs[3];
                            key_steps(g, bl, gs);
                            k = (bl[0] * g.nb[1] + bl[1]) * g.nb[2] + bl[2] + (m & 1u ? gs[0] : 0) +
                                (m & 2u ? gs[1] : 0) + (m & 4u ? gs[2] : 0);
                        }
                        put_record(A.payload, nrec, k, atomicAdd(A.cursor + k, 1u), slab, A.cap,
                                   A.ovf);
                    }
                }
            }
            __syncthreads();
        }
        // the next tile's particles start on their way to L2: step 1 then
        // waits for L2 and not for memory
        if (LEVEL == 2) {
            if (t + 1 < t1) {
                const float4 *next = A.part + p0 + count;  // mostly the same super-brick's
                for (int i = tid * 8; i < tile && p0 + count + i < (int64_t)A.part_cap; i += NT * 8) prefetch_l2(next + i);
            }
        } else {
            const int64_t q0 = p0 + (int64_t)gridDim.x * tile;
            for (int i = tid * 32; i < tile && q0 + i < A.np; i += NT * 32) {
                prefetch_l2(A.x + q0 + i);
                prefetch_l2(A.y + q0 + i);
                prefetch_l2(A.z + q0 + i);
                if (A.w) prefetch_l2(A.w + q0 + i);
            }
        }
        // 3. cursors and the bins' places
        const int extra = LEVEL == 1 ? 0 : min((int)s_extra, recs - tile);
        uint32_t slot0[PER], place[PER];  // of the run's first record
        {
            uint32_t cnt[PER], sum = 0;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int b = tid * per + j;
                cnt[j] = j < per && b < nbins ? bin[b] : 0u;
                slot0[j] = 0u;
                if (cnt[j]) {
                    const int at = LEVEL == 2 ? (int)brick[b] : b;
                    slot0[j] = atomicAdd((LEVEL == 1 ? A.scursor : A.cursor) + at, cnt[j]);
                }
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
            uint32_t run = __reduce_add_sync(0xffffffffu, lane < wid ? warp_sums[lane] : 0u) + incl - sum;
            if (tid == NT - 1) s_total = run + sum;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int b = tid * per + j;
                if (j < per && b < nbins) bin[b] = run;
                place[j] = run;
                run += cnt[j];
            }
        }
        __syncthreads();
        // 4. the order
        {
            const int end = tile + extra;
            uint32_t to[MAXREC], what[MAXREC];
#pragma unroll
            for (int j = 0; j < MAXREC; ++j) {
                const int i = tid + j * NT;
                const uint32_t o = i < count || (i >= tile && i < end) ? order[i] : kNone;
                to[j] = kNone;
                if (o != kNone) to[j] = bin[o >> 14] + (o & 16383u);
                what[j] = (o & ~16383u) | (uint32_t)i;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < MAXREC; ++j)
                if (to[j] != kNone) order[to[j]] = what[j];
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int b = tid * per + j;
            if (j < per && b < nbins) {
                uint32_t first_slot = slot0[j] - place[j];
                if (LEVEL == 2 && SLAB) first_slot += brick[b] * slab;
                if (LEVEL == 1) first_slot += (uint32_t)b * s.cap;
                bin[b] = first_slot;
            }
        }
        __syncthreads();
        // 5. out, in that order
        const int total = (int)s_total;
        bool over = false;
#pragma unroll 4
        for (int i = tid; i < total; i += NT) {
            const uint32_t o = order[i];
            const unsigned k = o >> 14;
            const uint4 rec = stage[o & 16383u];
            const uint32_t slot = bin[k] + (uint32_t)i;
            uint64_t at = slot;
            bool fits;
            if (LEVEL == 0) {
                fits = SLAB ? slot < slab : slot < A.cap;
                if (SLAB) at = (uint64_t)k * slab + slot;
            } else if (LEVEL == 1) {
                // the last bin takes what is left of the buffer
                fits = s.cap && (int)k < s.count ? slot < (k + 1u) * s.cap : slot < A.part_cap;
            } else {
                fits = slot < limit[k];
            }
            if (fits) (LEVEL == 1 ? reinterpret_cast<uint4 *>(A.part) : A.payload)[at] = rec;
            over = over || !fits;
        }
        if (over) atomicOr(A.ovf, 1u);
        __syncthreads();
        for (int b = tid; b < nbins; b += NT) bin[b] = 0u;
        if (tid == 0) s_queued = s_extra = 0u;
        __syncthreads();
    }
    if (SLAB && LEVEL != 1) flush_stats(my_lost, ws, A.lost, A.wstat);
}

// Particles per super-brick (two levels, exact ranges).
__global__ void __launch_bounds__(kBinThreads)
super_count_kernel(const __grid_constant__ SortArgs A, const __grid_constant__ AssignGeom g,
                   const __grid_constant__ SuperGeom s, unsigned chunk)
{
    chain_begin();
    __shared__ uint32_t hist[kMaxSupers + 1];
    for (int i = threadIdx.x; i <= s.count; i += kBinThreads) hist[i] = 0u;
    __syncthreads();
    const int64_t p0 = (int64_t)blockIdx.x * chunk;
    const int count = (int)max((int64_t)0, min((int64_t)chunk, A.np - p0));
    for_particles<kBinThreads>(A.x, A.y, A.z, (const float *)nullptr, p0, count,
                               [&](int, float px, float py, float pz, float) {
                                   atomicAdd(hist + super_of(g, s, px, py, pz), 1u);
                               });
    __syncthreads();
    for (int i = threadIdx.x; i <= s.count; i += kBinThreads)
        if (hist[i]) atomicAdd(A.scursor + i, hist[i]);
}

// Super-brick ranges from their counts (one CTA): beg[k], beg[count + 1] =
// all particles, cursors at their starts, *fullest = the largest count of a
// super-brick (the last bin left out).
__global__ void __launch_bounds__(1024)
super_offsets_kernel(uint32_t *__restrict__ scursor, int count, uint32_t *__restrict__ beg, unsigned int *__restrict__ fullest)
{
    chain_begin();
    __shared__ uint32_t sums[32];
    const int k = threadIdx.x, lane = k & 31, wid = k >> 5;
    const uint32_t n = k <= count ? scursor[k] : 0u;
    uint32_t incl = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
    }
    if (lane == 31) sums[wid] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < wid; ++w) before += sums[w];
    if (k <= count) {
        beg[k] = before + incl - n;
        scursor[k] = before + incl - n;
        if (k == count) beg[k + 1] = before + incl;
    }
    const unsigned m = __reduce_max_sync(0xffffffffu, k < count ? n : 0u);
    if (lane == 0 && m) atomicMax(fullest, m);
}

// Records per brick from particles sorted by super-brick (the count pass of
// two levels): a shared histogram over the super-brick's bins, flushed when
// the super-brick changes, with the lost count and weight statistics.
template <int SCHEME>
__global__ void __launch_bounds__(512, 2)
super_tally_kernel(const __grid_constant__ SortArgs A, const __grid_constant__ AssignGeom g,
                   const __grid_constant__ SuperGeom s)
{
    chain_begin();
    constexpr int NT = 512;
    extern __shared__ __align__(16) unsigned char tally_smem[];
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t s_queued;
    uint32_t *const bin = reinterpret_cast<uint32_t *>(tally_smem);  // [nbins]
    uint32_t *const tstart = bin + A.nbins;                          // [kMaxSupers + 2]
    uint16_t *const queue = reinterpret_cast<uint16_t *>(tstart + kMaxSupers + 2);  // [tile]: key | cross << 10
    const int tid = threadIdx.x;
    unsigned int my_lost = 0;
    WeightStats ws;
    for (int b = tid; b < A.nbins; b += NT) bin[b] = 0u;
    if (tid == 0) s_queued = 0u;
    __syncthreads();
    const int64_t tiles = tile_starts<NT>(A, s, tstart, warp_sums);
    const int64_t each = (tiles + gridDim.x - 1) / gridDim.x;
    const int64_t t0 = blockIdx.x * each, t1 = min(tiles, t0 + each);
    int sup = -1, org[3] = {0, 0, 0};
    auto flush = [&]() {
        for (int b = tid; b < A.nbins; b += NT) {
            const uint32_t n = bin[b];
            if (!n) continue;
            const int l2 = b % s.D[2], r = b / s.D[2];
            const int gk = (to_brick(g, 0, org[0], r / s.D[1]) * g.nb[1] + to_brick(g, 1, org[1], r % s.D[1])) * g.nb[2] +
                           to_brick(g, 2, org[2], l2);
            atomicAdd(A.cursor + gk, n);
            bin[b] = 0u;
        }
    };
    for (int64_t t = t0; t < t1; ++t) {
        int k = sup < 0 ? super_of_tile(tstart, s.count, (int)t) : sup;
        while (tstart[k + 1] <= (uint32_t)t) ++k;
        uint32_t beg, cnt;
        super_range(A, s, k, beg, cnt);
        const uint32_t off = ((uint32_t)t - tstart[k]) * (uint32_t)A.tile;
        const float4 *in = A.part + beg + off;
        const int count = (int)min((uint32_t)A.tile, cnt - off);
        if (k != sup) {
            if (sup >= 0 && sup < s.count) flush();
            sup = k;
            if (k < s.count) local_origin(s, k, org);
            __syncthreads();
        }
        if (k == s.count) {
            for_packed<NT>(in, count, [&](int, float px, float py, float pz, float wt) {
                count_one<SCHEME, false>(px, py, pz, wt, A.weighted != 0, g, nullptr, A.cursor, my_lost, ws);
            });
            continue;
        }
        for_packed<NT>(in, count, [&](int, float px, float py, float pz, float wt) {
            int c[3], bl[3], cl;
            uint32_t o[3];
            if (!locate<SCHEME, false>(px, py, pz, g, c, o)) {
                ++my_lost;
                return;
            }
            unsigned cross = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) cross |= brick_axis<SCHEME>(g, a, c[a], bl[a], cl) ? 1u << a : 0u;
            const int l0 = to_local(g, 0, org[0], bl[0]), l1 = to_local(g, 1, org[1], bl[1]),
                      l2 = to_local(g, 2, org[2], bl[2]);
            // a stencil that leaves the bins (never, but for a particle the
            // approximate home cell put on the wrong side)
            bool in_bins = l0 < s.D[0] && l1 < s.D[1] && l2 < s.D[2];
            if (SCHEME != CAM_NGP)
                in_bins = in_bins && !((cross & 1u) && s.ns[0] > 1 && l0 + 1 == s.D[0]) &&
                          !((cross & 2u) && s.ns[1] > 1 && l1 + 1 == s.D[1]) &&
                          !((cross & 4u) && s.ns[2] > 1 && l2 + 1 == s.D[2]);
            if (!in_bins) {
                count_one<SCHEME, false>(px, py, pz, wt, A.weighted != 0, g, nullptr, A.cursor, my_lost, ws);
                return;
            }
            if (A.weighted) ws.add(wt);
            const int key = (l0 * s.D[1] + l1) * s.D[2] + l2;
            atomicAdd(bin + key, 1u);
            if (SCHEME != CAM_NGP && cross) queue[atomicAdd(&s_queued, 1u)] = (uint16_t)(key | (cross << 10));
        });
        __syncthreads();
        if (SCHEME != CAM_NGP) {
            const int nq = (int)s_queued;
            for (int q = tid; q < nq; q += NT) {
                const unsigned ent = queue[q];
                const int key = (int)(ent & 1023u);
                const unsigned cross = ent >> 10;
                const int r = s.D[2] == 1 ? key : (int)__umulhi((unsigned)key, s.dmagic[0]);
                int l[3], step[3];
                l[2] = key - r * s.D[2];
                l[0] = s.D[1] == 1 ? r : (int)__umulhi((unsigned)r, s.dmagic[1]);
                l[1] = r - l[0] * s.D[1];
                const int stride[3] = {s.D[1] * s.D[2], s.D[2], 1};
#pragma unroll
                for (int a = 0; a < 3; ++a) step[a] = l[a] + 1 == s.D[a] ? -l[a] * stride[a] : stride[a];
#pragma unroll 1
                for (unsigned m = cross; m; m = (m - 1u) & cross)
                    atomicAdd(bin + key + (m & 1u ? step[0] : 0) + (m & 2u ? step[1] : 0) + (m & 4u ? step[2] : 0), 1u);
            }
            __syncthreads();
            if (tid == 0) s_queued = 0u;
            __syncthreads();
        }
    }
    __syncthreads();
    if (sup >= 0 && sup < s.count) flush();
    flush_stats(my_lost, ws, A.lost, A.wstat);
}

// Brick starts in one CTA (nb <= kOffThreads * kOffItems): thread t scans
// the counts of bricks [t * kOffItems, (t + 1) * kOffItems) in order, the
// per-thread sums are scanned across the CTA, and every brick's start goes
// to start[b] and to its cursor (which held its count); start[nb] =
// *total = all records.
constexpr int kOffThreads = 1024;
constexpr int kOffItems = 16;
__global__ void __launch_bounds__(kOffThreads)
brick_offsets_kernel(uint32_t *__restrict__ table, int stride, int nb, uint32_t *__restrict__ start, uint32_t *__restrict__ total)
{
    chain_begin();
    __shared__ uint32_t warp_sums[kOffThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int base = threadIdx.x * kOffItems;
    uint32_t v[kOffItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kOffItems; ++i) {
        v[i] = base + i < nb ? table[(int64_t)(base + i) * stride] : 0u;
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
            table[(int64_t)(base + i) * stride] = run;
        }
        run += v[i];
    }
}

// The largest brick record count, start[b + 1] - start[b], into *out
// (atomicMax; *out zeroed before).
__global__ void __launch_bounds__(256)
brick_max_kernel(const uint32_t *__restrict__ start, int nb, unsigned int *__restrict__ out)
{
    chain_begin();
    unsigned m = 0u;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
        m = max(m, start[b + 1] - start[b]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// counts[b] = table[b * stride] (contiguous, for the scan).
__global__ void compact_counts_kernel(const uint32_t *__restrict__ table, int stride, int nb, uint32_t *__restrict__ counts)
{
    chain_begin();
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
        counts[b] = table[(int64_t)b * stride];
}

// start[b] = scanned count of brick b (its first payload), start[nb] = total;
// the cursors start there.
__global__ void brick_starts_kernel(const uint32_t *__restrict__ scanned, int nb,
                                    const uint32_t *__restrict__ total, uint32_t *__restrict__ start,
                                    uint32_t *__restrict__ cursor, int stride)
{
    chain_begin();
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x) {
        const uint32_t v = b < nb ? scanned[b] : *total;
        start[b] = v;
        if (b < nb) cursor[(int64_t)b * stride] = v;
    }
}

// Pass 4: one CTA per brick, two CTAs per SM.  Bound by the
// shared-memory atomics (one per stencil cell, 3.7 wavefronts each: 32 random
// cells on 32 banks) and, for NGP and CIC, by the latency of the record
// loads.  256^3, 16.8 M weighted particles: TSC 417 -> 333 us, CIC 200 ->
// 148, NGP 136 -> 101 with the stencil on constant offsets from one address
// (508 warp instructions per 32 TSC records before; 78% issue) and the record
// loads two groups ahead.
template <int SCHEME, typename OutT>
__global__ void __launch_bounds__(kDepositThreads, 2)
deposit_kernel(const uint4 *__restrict__ payload, const uint32_t *__restrict__ start, uint32_t nrec,
               AssignGeom g, const unsigned int *__restrict__ wstat, int weighted,
               OutT *__restrict__ mesh, double *__restrict__ brick_sum, uint32_t slab,
               const uint32_t *__restrict__ slab_count, unsigned int *__restrict__ host_ovf)
{
    chain_begin();
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
    // records beyond the payload's capacity nrec were not written (overflow
    // flag); with slabs, the brick's records are the first of its slab (the
    // host keeps every slab index below 2^32)
    const uint32_t beg = slab ? (uint32_t)B * slab : min(start[B], nrec);
    const uint32_t end = slab ? beg + min(slab_count[(int64_t)B * g.cstride], slab) : min(start[B + 1], nrec);
    RecordStream rec;
    rec.open(payload, beg, end, warp, kDepositThreads / 32, lane);
    const unsigned heaviest = weighted ? wstat[0] : 0u, overflow = wstat[4];
    const bool nonneg = !weighted || wstat[1] == 0u;
    const int s = fixed_scale(wstat, weighted, end - beg);
    // 2^s as two exact factors (s may exceed the float exponent range)
    const float f1 = scalbnf(1.0f, s / 2), f2 = scalbnf(1.0f, s - s / 2);
    // a weight that is not finite, or records that found no room (the call
    // fails, or runs again exactly): the mesh, which may be the caller's, is
    // left as it is
    if (heaviest >= 0x7f800000u || overflow != 0u) {
        if (host_ovf && blockIdx.x == 0 && threadIdx.x == 0 && overflow != 0u) *host_ovf = 1u;
        return;
    }
    zero_tile(tile32, e, threadIdx.x, kDepositThreads);
    __syncthreads();
    deposit_records<SCHEME>(rec, e, f1, f2, nonneg, tile32);
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
    chain_begin();
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
        g.origin |= g.mn[a] != 0.0f;
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
    // A stencil of three cells must never span three bricks (its particle has
    // records in two at most along an axis): a partial last brick keeps at
    // least 2 cells.  The extent shrinks until it does, or grows where no
    // smaller one leaves 0 or 2 (N = 13, 25, 37, 49, 61, ..., when many
    // particles had made the bricks 4 or 3 cells).
    constexpr int largest[3] = {16, 16, 32};
    for (int a = 0; a < 3; ++a) {
        auto one_left = [&](int b) { return b < g.n[a] && g.n[a] % b == 1; };
        int b = g.b[a];
        while (one_left(b) && b > 3) --b;
        if (one_left(b))
            for (b = g.b[a]; one_left(b) && b < largest[a];) ++b;
        CAM_REQUIRE(scheme != CAM_TSC || !one_left(b), CAM_E_UNSUPPORTED,
                    "no brick extent leaves a TSC stencil within two bricks");  // N = 720721 alone
        g.b[a] = b;
        g.nb[a] = (g.n[a] + g.b[a] - 1) / g.b[a];
        g.inv_d[a] = 1.0f / g.d[a];
        g.e_last[a] = g.n[a] - (g.nb[a] - 1) * g.b[a];
        g.nf[a] = (float)g.n[a];
        g.half_d[a] = 0.5f * g.d[a];
        g.off_scale[a] = g.inv_d[a] * 16777216.0f;
        // an axis that one brick spans: brick 0 always, nothing crosses
        const bool whole = g.nb[a] == 1;
        const int reach = scheme == CAM_TSC ? 2 : 1;  // from the stencil's first to its last cell
        g.bmagic[a] = whole ? 0u : (unsigned)(((1ull << 32) + (uint64_t)g.b[a] - 1) / (uint64_t)g.b[a]);
        g.lo0[a] = whole ? -1 : g.n[a] - 1;
        g.cross_b[a] = whole ? INT32_MAX : g.b[a] - reach;
        g.cross_n[a] = whole ? INT32_MAX : g.n[a] - reach;
        // home_cell divides exactly when a quotient u <= n lies within
        // 4e-7 max(u, 1) of an integer; a little more is set aside here.
        // A quotient u < n - thr means x - min <= (n - thr) d (1 + 3e-7)
        // before rounding, which is inside the box if that is below its
        // rounded end less min.
        const float thr = 4.2e-7f * (float)(g.n[a] + 1) + 1e-6f;
        const double end = (double)(g.mn[a] + g.L[a]) - (double)g.mn[a];
        const double nd = (double)g.n[a] * (double)g.d[a];
        // How far n * d may be off L.  Without an origin locate() puts a CIC
        // position v in [-d, 0) into cell n - 1, the reference into the cell
        // of v + L: the same one if n - L / d is below thr less the roundings
        // of v + L and of its quotient (1.2e-7 n cells); d = L / n rounded is
        // off by 6e-8 n cells.  Nothing else here depends on n * d being L.
        const double off = scheme == CAM_CIC && !g.origin ? 0.5 * thr : 1e-3 * std::max(1.0, 1e-3 * g.n[a]);
        const bool regular = g.n[a] >= 4 && std::isfinite(g.off_scale[a]) && std::isnormal(g.inv_d[a]) && ((double)g.n[a] - thr) * g.d[a] * (1.0 + 3e-7) < end &&
                             std::fabs(nd - (double)g.L[a]) <= off * g.d[a];
        g.safe[a] = regular ? 0.5f - thr : -1.0f;
    }
    for (int a = 0; a < 2; ++a)
        g.kmagic[a] = g.nb[2 - a] > 1 ? (unsigned)(((1ull << 32) + (uint64_t)g.nb[2 - a] - 1) / (uint64_t)g.nb[2 - a]) : 0u;
    g.cstride = 1;
    return g;
}

// The super-bricks of a mesh: brick groups doubled along the axis where they
// are shortest until at most `most` remain.
static SuperGeom super_geom(const AssignGeom &g, int most)
{
    SuperGeom s{};
    for (int a = 0; a < 3; ++a) s.gs[a] = 1;
    for (;;) {
        int64_t count = 1;
        int grow = -1;
        for (int a = 0; a < 3; ++a) {
            s.ns[a] = (g.nb[a] + s.gs[a] - 1) / s.gs[a];
            count *= s.ns[a];
            if (s.ns[a] > 1 && (grow < 0 || s.gs[a] * g.b[a] < s.gs[grow] * g.b[grow])) grow = a;
        }
        if (count <= most) {
            s.count = (int)count;
            break;
        }
        s.gs[grow] *= 2;
    }
    for (int a = 0; a < 3; ++a) {
        s.D[a] = s.ns[a] == 1 ? g.nb[a] : s.gs[a] + 2;
        s.inv[a] = 1.0f / (float)(s.gs[a] * g.b[a]);
    }
    for (int a = 0; a < 2; ++a)
        s.dmagic[a] = (unsigned)(((1ull << 32) + (uint64_t)s.D[2 - a] - 1) / (uint64_t)std::max(s.D[2 - a], 2));
    return s;
}
static int local_bins_of(const SuperGeom &s) { return s.D[0] * s.D[1] * s.D[2]; }

template <int SCHEME>
static void assign_impl(cam_ctx *ctx, const float *x, const float *y, const float *z,
                        const float *w, int64_t np, const AssignGeom &geom, AssignOut &out)
{
    const int64_t nb = (int64_t)geom.nb[0] * geom.nb[1] * geom.nb[2];
    CAM_REQUIRE(nb < (1ll << 31), CAM_E_UNSUPPORTED, "too many mesh bricks");
    // Count pass: one CTA of 1024 threads per SM (its brick histogram in
    // shared memory), contiguous chunks of >= 4096 particles.
    const int G = (int)std::max<int64_t>(1, std::min<int64_t>(kNumSMs, (np + 4095) / 4096));
    const unsigned chunk = (unsigned)std::max<int64_t>(1, (np + G - 1) / G);
    const bool smem_hist = nb <= kSmemBricks;
    // Two levels of sorting when the records would otherwise leave a tile in
    // runs of a few per brick.
    const bool plain_ctx = !ctx->sync_free && !ctx->slabs_off && !ctx->budget && !ctx->lean;
    SuperGeom sg{};
    if (plain_ctx && nb > kStageBins && np >= kTwoLevelParticles &&
        (uint64_t)np * sizeof(float4) <= ctx->device_bytes / 16 && geom.safe[0] > 0.f && geom.safe[1] > 0.f &&
        geom.safe[2] > 0.f)
        // as few super-bricks as LEVEL 2 has bins for: LEVEL 1's runs are the
        // longer (512^3: 128 of them 0.95 ms, 512 of them 1.87, LEVEL 2 alike)
        for (int most = 128; most <= 1024 && sg.count == 0; most *= 2) {
            const SuperGeom s = super_geom(geom, std::min(most, kMaxSupers));
            if (local_bins_of(s) <= kMaxLocal) sg = s;
        }
    AssignGeom g = geom;
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
    // sized from the clumping the exact runs of this mesh shape measured (a
    // slab that overflows makes the call rerun exactly, which measures
    // again); no count pass and no scan then, and the scatter
    // gathers the statistics.  With two levels the super-bricks get slabs of
    // their own the same way.  Only while the slabs stay within twice the
    // expected records (or 2^20 records), three times with two levels, which
    // limits memory: slabs are the faster at any size (a layer of 1 to 6
    // times the mean density: 16.8 M TSC particles onto 256^3 640-650 us with
    // slabs of 1.1 to 6.8 times the records, 735-747 counted exactly; 67 M
    // onto 512^3 2.99-3.00 and 3.75 ms).
    // A context with an HBM budget keeps the exact path, whose payload the
    // budget was sized for, and so does one whose device is short of memory
    // (run_as_fits); nor do slabs take more than a quarter of the device's
    // memory, or sorted particles a sixteenth, an eighth in slabs.
    const double est_brick = (double)np * f / (double)nb;
    const AssignShape shape{g.n[0], g.n[1], g.n[2], g.b[0], g.b[1], g.b[2], SCHEME};
    double est_super = (double)np;
    for (int a = 0; a < 3 && sg.count > 0; ++a)
        est_super *= (double)std::min(sg.gs[a] * g.b[a], g.n[a]) / (double)g.n[a];
    const uint64_t beyond = std::max<uint64_t>(65536, (uint64_t)np / 256);  // room of the last bin, with slabs
    uint32_t slab = 0;
    if (out.defer && plain_ctx && np > 0) {
        const auto it = ctx->slab_clump.find(shape);
        if (it != ctx->slab_clump.end()) {
            SlabClump &clump = it->second;
            const bool two = sg.count > 0;
            const double room = std::min({std::max((two ? 3.0 : 2.0) * (double)np * f, (double)(1u << 20)), 4294967295.0,
                                          (double)(ctx->device_bytes / 4 / sizeof(uint4))});
            const uint64_t cap = slab_within(clump.brick.value * est_brick, (uint64_t)(room / (double)nb) & ~(uint64_t)3);
            const bool bricks_fit = cap > 0;
            // With more than 128 super-bricks a shape too clumped for slabs
            // runs exactly in one level, which does not measure its
            // super-bricks.  Particles in lattice order, whose records append
            // to a few bricks at a time, gain by it (768^3, 453 M TSC
            // particles: counts 4.45 ms and records 8.8, in two levels 5.0 +
            // 3.4 + 8.0), particles in random order lose (226 M CIC onto
            // 768^3 11.9 and 10.0 ms, 131 M onto 640^3 6.8 and 5.7).
            // If the bricks have come to fit since, they are measured anew.
            if (sg.count > 128 && bricks_fit && clump.since_super >= 4) clump.super = Clump{};
            bool fits = bricks_fit;
            if (two) {
                const double sroom = std::min(2.0 * (double)np + (double)(1u << 20), 4294967295.0 - (double)beyond);
                sg.cap = fits && clump.super.value > 0.0
                             ? (uint32_t)slab_within(clump.super.value * est_super, (uint64_t)(sroom / sg.count) & ~(uint64_t)3)
                             : 0u;
                fits = sg.cap > 0;
            }
            if (fits) slab = (uint32_t)cap;
            else if (sg.count > 128 && clump.super.value > 0.0) sg = SuperGeom{};
        }
    }
    const bool two = sg.count > 0;
    const bool staged = two || nb <= kStageBins;
    g.cstride = staged ? 1 : kPaddedStride;
    // statistics and per-brick counters (counts, then cursors): one buffer,
    // zeroed at once
    const size_t head_bytes = kAssignHead + (size_t)nb * g.cstride * sizeof(uint32_t);
    auto *stats = static_cast<unsigned long long *>(scratch(ctx, "asg.head", head_bytes));
    auto *table = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(stats) + kAssignHead);
    auto *start = static_cast<uint32_t *>(scratch(ctx, "asg.start", (nb + 1) * sizeof(uint32_t)));
    auto *bsum = static_cast<double *>(scratch(ctx, "asg.bsum", nb * sizeof(double)));
    unsigned long long *d_lost = stats;
    unsigned int *d_wmax = reinterpret_cast<unsigned int *>(stats + 1);
    uint32_t *d_total = reinterpret_cast<uint32_t *>(stats + 2);
    unsigned int *d_ovf = reinterpret_cast<unsigned int *>(stats + 3);
    CAM_CUDA_TRY(cudaMemsetAsync(stats, 0, head_bytes, ctx->stream));

    // What the sort kernels share; tile and recs are set per level.
    SortArgs A{};
    A.x = x;
    A.y = y;
    A.z = z;
    A.w = w;
    A.np = np;
    A.cursor = table;
    A.lost = d_lost;
    A.wstat = d_wmax;
    A.ovf = d_ovf;
    A.slab = slab;
    A.weighted = w != nullptr;
    // Tiles as large as the stage holds with the expected records (15% margin
    // on the extra ones); LEVEL 0 and 1: split evenly over the resident CTAs.
    auto tile_for = [&](int level, int nbins, double records) {
        A.nbins = nbins;
        const size_t bytes = stage_budget(level) - stage_fixed(level, nbins);
        const double fr = 1.0 + 1.15 * (records - 1.0);
        const double each = 20.0 * fr + (level == 1 ? 0.0 : 2.0);
        const int64_t most = std::max<int64_t>(512, std::min<int64_t>(kStageTile, (int64_t)((double)bytes / each)));
        // a batch's jobs run beside each other: fewer, larger tiles cost less
        // in all (32 jobs, CIC, split over 16, 32, 64, 148 CTAs: 32^3 with
        // 300,000 particles 1.09, 1.10, 1.10, 1.16 ms; 64^3 with 262,144 1.02,
        // 1.02, 1.05, 1.14; 128^3 with 600,000 1.93, 1.94, 1.98, 1.98)
        const int64_t ctas = ctx->sync_free ? 32 : stage_ctas(level) * kNumSMs;
        const int64_t rounds = std::max<int64_t>(1, (np + ctas * most - 1) / (ctas * most));
        const int64_t even = (np + ctas * rounds - 1) / (ctas * rounds);
        A.tile = (int)(level == 2 ? most & ~(int64_t)31
                                  : std::min<int64_t>(most, std::max<int64_t>(1024, (even + 31) & ~(int64_t)31)));
        // small jobs leave the rest of the shared memory to other streams'
        // kernels: no more than twice the expected further records
        const size_t want = (size_t)((double)A.tile * (1.0 + 2.0 * (records - 1.0))) + (level == 1 ? 0 : 512);
        A.recs = (int)std::min<size_t>(std::min<size_t>(16383, want), (bytes - (level == 1 ? 0 : (size_t)A.tile * 2)) / 20);
        const int64_t tiles = (np + A.tile - 1) / A.tile;
        return (unsigned)std::max<int64_t>(1, std::min<int64_t>(stage_ctas(level) * kNumSMs, tiles));
    };
    auto sort_bytes = [&](int level) {
        return (size_t)A.recs * 20 + (level == 1 ? 0 : (size_t)A.tile * 2) + stage_fixed(level, A.nbins);
    };
    const int local_bins = two ? local_bins_of(sg) : 0;

    if (two) {
        A.part_cap = slab ? (uint64_t)sg.count * sg.cap + beyond : (uint64_t)np;
        A.part = static_cast<float4 *>(scratch(ctx, "asg.part", A.part_cap * sizeof(float4)));
        A.scursor = static_cast<uint32_t *>(
            scratch(ctx, "asg.scursor", (size_t)(kMaxSupers + 1) * sizeof(uint32_t)));
        auto *sbeg = static_cast<uint32_t *>(scratch(ctx, "asg.sbeg", (kMaxSupers + 3) * sizeof(uint32_t)));
        A.sbeg = sbeg;
        CAM_CUDA_TRY(cudaMemsetAsync(A.scursor, 0, (size_t)(sg.count + 1) * sizeof(uint32_t), ctx->stream));
        if (!slab) {
            CAM_LAUNCH_NAMED(ctx, "assign_super_count", super_count_kernel, G, kBinThreads, 0, A, g, sg, chunk);
            CAM_LAUNCH_NAMED(ctx, "assign_starts", super_offsets_kernel, 1, 1024, 0, A.scursor, sg.count, sbeg,
                             reinterpret_cast<unsigned int *>(stats + 6));
            out.super_est = est_super;
        }
        const unsigned grid = tile_for(1, sg.count + 1, 1.0);
        const size_t smem1 = sort_bytes(1);
        auto k = sort_kernel<CAM_NGP, false, 1>;
        smem_at_least(k, smem1);
        CAM_LAUNCH_NAMED(ctx, "assign_super_sort", k, grid, stage_threads(1), smem1, A, g, sg);
    }

    const size_t hsmem = smem_hist ? (size_t)nb * sizeof(uint32_t) : 0;
    auto count_k = smem_hist ? count_kernel<SCHEME, true> : count_kernel<SCHEME, false>;
    if (!slab) {
        if (two) {
            A.nbins = local_bins;
            A.tile = kStageTile;
            const size_t tsmem = (size_t)local_bins * 4 + (kMaxSupers + 2) * 4 + (size_t)A.tile * 2;
            CAM_LAUNCH_NAMED(ctx, "assign_bin_count", super_tally_kernel<SCHEME>, 2 * kNumSMs, 512, tsmem, A, g, sg);
        } else {
            smem_at_least(count_k, hsmem);
            CAM_LAUNCH_NAMED(ctx, "assign_bin_count", count_k, G, kBinThreads, hsmem, x, y, z, w, np, chunk, g, (int)nb,
                             table, d_lost, d_wmax);
        }
        if (nb <= (int64_t)kOffThreads * kOffItems) {
            CAM_LAUNCH_NAMED(ctx, "assign_starts", brick_offsets_kernel, 1, kOffThreads, 0, table, g.cstride, (int)nb, start,
                             d_total);
        } else {
            auto *counts = static_cast<uint32_t *>(scratch(ctx, "asg.counts", (size_t)nb * sizeof(uint32_t)));
            const unsigned blocks = (unsigned)std::min<int64_t>((nb + 256) / 256, 1024);
            CAM_LAUNCH_NAMED(ctx, "assign_starts", compact_counts_kernel, blocks, 256, 0, table, g.cstride, (int)nb, counts);
            exclusive_scan_u32(ctx, counts, nb, d_total);
            CAM_LAUNCH_NAMED(ctx, "assign_starts", brick_starts_kernel, blocks, 256, 0, counts, (int)nb, d_total, start,
                             table, g.cstride);
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
        // for the caller to read back with the results.
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
        unsigned long long hstats[8] = {};
        CAM_CUDA_TRY(cudaMemcpyAsync(hstats, stats, sizeof(hstats), cudaMemcpyDeviceToHost, ctx->stream));
        CAM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        total = (uint32_t)(hstats[2] & 0xffffffffu);
        ctx->asg_cap = std::max<uint64_t>(ctx->asg_cap, total);  // deferred runs size from it
        out.brick_max = hstats[5] & 0xffffffffu;
        out.super_max = hstats[6] & 0xffffffffu;
        const unsigned int wmax_bits = (unsigned int)(hstats[1] & 0xffffffffu);
        CAM_REQUIRE(!w || wmax_bits < 0x7f800000u, CAM_E_NONFINITE, "a particle weight is NaN or infinite");
        out.n_lost = (int64_t)hstats[0];
        out.n_in = np - out.n_lost;
    }

    uint4 *payload = static_cast<uint4 *>(scratch(ctx, "asg.payload", std::max<size_t>(total, 1) * sizeof(uint4)));
    A.payload = payload;
    A.cap = total;
    if (staged) {
        const int level = two ? 2 : 0;
        const unsigned grid = tile_for(level, two ? local_bins : (int)nb, f);
        const size_t ssmem = sort_bytes(level);
        auto k = two ? (slab ? sort_kernel<SCHEME, true, 2> : sort_kernel<SCHEME, false, 2>)
                     : (slab ? sort_kernel<SCHEME, true, 0> : sort_kernel<SCHEME, false, 0>);
        smem_at_least(k, ssmem);
        CAM_LAUNCH_NAMED(ctx, "assign_bin_scatter", k, grid, stage_threads(level), ssmem, A, g, sg);
    } else {
        const int G2 = (int)std::max<int64_t>(1, std::min<int64_t>(2 * kNumSMs, (np + 4095) / 4096));
        const unsigned chunk2 = (unsigned)std::max<int64_t>(1, (np + G2 - 1) / G2);
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
                         table, out.host_ovf);
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
    return static_cast<unsigned long long *>(scratch(ctx, "asg.head", kAssignHead));
}

void assign_device(cam_ctx *ctx, const float *x, const float *y, const float *z,
                   const float *w, int64_t np, const cam_grid &grid, int scheme, AssignOut &out)
{
    CAM_REQUIRE(np >= 0, CAM_E_INVAL, "negative particle count");
    CAM_REQUIRE(np == 0 || (x && y && z), CAM_E_INVAL, "null particle coordinates");
    CAM_REQUIRE(np < (1ll << 31), CAM_E_UNSUPPORTED, "more than 2^31 particles per call");
    const AssignGeom g = make_geom(grid, scheme, np);
    struct Assigning {
        cam_ctx *c;
        explicit Assigning(cam_ctx *ctx) : c(ctx) { c->assigning = true; }
        ~Assigning() { c->assigning = false; }
    } assigning(ctx);
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
