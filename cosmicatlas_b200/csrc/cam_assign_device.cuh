// Device functions of the mass assignment shared by the multi-CTA passes
// (cam_assign.cu) and the one-CTA-per-job pipeline of the device request
// loop (cam_devloop.cu): the reference's FP32 home cell, the exact
// fractional offsets, the payload record format, the stencil deposit into a
// haloed 64-bit fixed-point tile and its conversion.  Both paths use these
// same functions, so a job's mesh is bit-identical whichever runs it.
// Replaces getDensity_NGP / getDensity_CIC / getDensity_TSC,
// Source/massFunctions.cpp:35-98, :678-790, :1050-1165.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cam_internal.h"

namespace cam {
namespace asg {

// Global per-brick counters and append cursors sit one per 128-byte line:
// atomics on one line are serialised in its L2 slice, so packed counters
// would funnel all bricks through a few slices.
constexpr int kCursorStride = 32;

// Reference FP32 home cell (see orc_keys / ref_home in the oracle).
// NGP: x on [min, min+L); CIC: x - d/2 wrapped once by +-L then [min, min+L);
// TSC: x on [min, min+L].  i = floor((x-min)/d) in IEEE float, then mod N.
template <int SCHEME>
__device__ __forceinline__ bool home_cell(const float p[3], const AssignGeom &g, int c[3])
{
    float q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float v = p[a];
        if (SCHEME == CAM_CIC) {
            v = __fsub_rn(v, __fmul_rn(0.5f, g.d[a]));
            if (v < 0.0f) v = __fadd_rn(v, g.L[a]);
            if (v >= g.L[a]) v = __fsub_rn(v, g.L[a]);
        }
        q[a] = v;
    }
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float hi = __fadd_rn(g.mn[a], g.L[a]);
        ok = ok && (SCHEME == CAM_TSC ? (q[a] >= g.mn[a] && q[a] <= hi)
                                      : (q[a] >= g.mn[a] && q[a] < hi));
    }
    if (!ok) return false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // floor of the IEEE quotient fl(t / d).  The product with 1/d is
        // within 2^-22 u of it; unless that product is this close to an
        // integer both have the same floor, otherwise divide exactly.
        const float t = __fsub_rn(q[a], g.mn[a]);
        float u = __fmul_rn(t, g.inv_d[a]);
        if (fabsf(u - rintf(u)) <= fmaxf(u, 1.0f) * 4.0e-7f) u = __fdiv_rn(t, g.d[a]);
        const int i = (int)floorf(u);
        // fmod(float(i), float(N)): i <= N whenever d = L/N; any i >= 0 otherwise
        c[a] = i < g.n[a] ? i : (i == g.n[a] ? 0 : i % g.n[a]);
    }
    return true;
}

// cell / b for the brick extent b (exact for cell < 2^21, b <= 2^11).
__device__ __forceinline__ int brick_of(int cell, int b, unsigned magic)
{
    return b == 1 ? cell : (int)__umulhi((unsigned)cell, magic);
}

// Exact offset t = (x - min)/d - 1/2 - c in cells, nearest periodic image,
// in FP32 with error-free transformations: TwoSum for x - min and a fused
// multiply-add for the subtraction of (c + 1/2) d (the product is exact
// inside the FMA); the residual (|r| <= 1.5 d) is scaled by 1/d.
// |error| <= ~2e-7 cells.
__device__ __forceinline__ float exact_offset(float x, float mn, float d, float inv_d, int c, int n)
{
    const float hi = __fsub_rn(x, mn);
    const float bb = __fsub_rn(hi, x);
    const float lo = __fadd_rn(__fsub_rn(x, __fsub_rn(hi, bb)), __fsub_rn(-mn, bb));
    const float u = hi * inv_d;
    float ci = (float)c + 0.5f;
    const float diff = u - ci;
    if (diff > 0.5f * (float)n) ci += (float)n;
    else if (diff < -0.5f * (float)n) ci -= (float)n;
    const float r = __fadd_rn(__fmaf_rn(-ci, d, hi), lo);
    return r * inv_d;
}

template <int SCHEME>
struct Stencil {
    static constexpr int W = SCHEME == CAM_NGP ? 1 : (SCHEME == CAM_CIC ? 2 : 3);
    static constexpr int FIRST = SCHEME == CAM_TSC ? -1 : 0;
};

// First and last stencil cells of a home cell c in [0, n), wrapped
// periodically: the stencil reaches at most one cell below 0 (TSC) and at
// most one cell at or above n, so one conditional add or subtract each.
template <int SCHEME>
__device__ __forceinline__ void stencil_ends(int c, int n, int &lo, int &hi)
{
    using St = Stencil<SCHEME>;
    lo = c + St::FIRST;
    hi = c + St::FIRST + St::W - 1;
    if constexpr (St::FIRST < 0) lo = lo < 0 ? lo + n : lo;
    if constexpr (St::FIRST + St::W - 1 > 0) hi = hi >= n ? hi - n : hi;
}

// Payload word per axis: bits 26..31 = home cell relative to the brick + 8,
// bits 0..25 = round(t * 2^24) + 2^24 (t in [-1, 3)).
__device__ __forceinline__ uint32_t pack_axis(int cl, float t)
{
    int tq = __float2int_rn(t * 16777216.0f) + 16777216;
    tq = min(max(tq, 0), (1 << 26) - 1);
    return ((uint32_t)(cl + 8) << 26) | (uint32_t)tq;
}
__device__ __forceinline__ void unpack_axis(uint32_t v, int &cl, float &t)
{
    cl = (int)(v >> 26) - 8;
    t = (float)((int)(v & 0x3FFFFFFu) - 16777216) * (1.0f / 16777216.0f);
}

__device__ __forceinline__ int brick_linear(const AssignGeom &g, int b0, int b1, int b2)
{
    return (b0 * g.nb[1] + b1) * g.nb[2] + b2;
}

// One particle of pass 1: the bricks its stencil touches (the brick of its
// first stencil cell and, along each axis whose stencil crosses a brick
// face, the next brick, periodically) each get one count.
template <int SCHEME, bool SMEM>
__device__ __forceinline__ void count_one(float px, float py, float pz, float wt, bool weighted, const AssignGeom &g,
                                          uint32_t *hist, uint32_t *__restrict__ table, unsigned long long &my_lost,
                                          unsigned int &my_wmax, unsigned int &my_neg, unsigned int &my_wminc)
{
    using St = Stencil<SCHEME>;
    const float pos[3] = {px, py, pz};
    int c[3] = {0, 0, 0};
    if (!home_cell<SCHEME>(pos, g, c)) {
        ++my_lost;
        return;
    }
    if (weighted) {
        my_wmax = max(my_wmax, __float_as_uint(fabsf(wt)));
        my_neg |= wt < 0.0f;
        if (wt != 0.0f) my_wminc = max(my_wminc, 0x7fffffffu - __float_as_uint(fabsf(wt)));
    }
    int bl[3];
    bool two[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int lo, hi;
        stencil_ends<SCHEME>(c[a], g.n[a], lo, hi);
        bl[a] = brick_of(lo, g.b[a], g.bmagic[a]);
        two[a] = St::W > 1 && brick_of(hi, g.b[a], g.bmagic[a]) != bl[a];
    }
    const int s1 = g.nb[2], s0 = g.nb[1] * g.nb[2];
    const int k0 = bl[0] * s0 + bl[1] * s1 + bl[2];
    // key step to the next brick along each axis (periodic)
    const int d2 = bl[2] + 1 == g.nb[2] ? -bl[2] : 1;
    const int d1 = (bl[1] + 1 == g.nb[1] ? -bl[1] : 1) * s1;
    const int d0 = (bl[0] + 1 == g.nb[0] ? -bl[0] : 1) * s0;
    auto add = [&](int key) {
        if (SMEM) atomicAdd(hist + key, 1u);
        else atomicAdd(table + (int64_t)key * kCursorStride, 1u);
    };
    add(k0);
    if (two[2]) add(k0 + d2);
    if (two[1]) {
        add(k0 + d1);
        if (two[2]) add(k0 + d1 + d2);
    }
    if (two[0]) {
        add(k0 + d0);
        if (two[2]) add(k0 + d0 + d2);
        if (two[1]) {
            add(k0 + d0 + d1);
            if (two[2]) add(k0 + d0 + d1 + d2);
        }
    }
}

// One particle of pass 3 (see bin_kernel).  slab > 0: the brick's records
// go to its own slab of `slab` records (payload[key * slab + slot], the
// counter starting at 0), and the weight statistics are gathered here
// (there is no count pass); my_wminc then receives the smallest nonzero
// |w| as count_one keeps it.
template <int SCHEME, bool SCATTER, bool SMEM, int CSTRIDE = kCursorStride>
__device__ __forceinline__ void bin_one(float px, float py, float pz, float wt, bool weighted,
                                        const AssignGeom &g, int G, int blk, uint32_t *hist,
                                        uint32_t *__restrict__ table, uint4 *__restrict__ payload, uint64_t cap,
                                        unsigned int *ovf, unsigned long long &my_lost, unsigned int &my_wmax,
                                        unsigned int &my_neg, unsigned int *my_wminc = nullptr, uint32_t slab = 0)
{
    using St = Stencil<SCHEME>;
    const float pos[3] = {px, py, pz};
    int c[3] = {0, 0, 0};
    if (!home_cell<SCHEME>(pos, g, c)) {
        ++my_lost;
        return;
    }
    if (weighted && (!SCATTER || my_wminc)) {
        my_wmax = max(my_wmax, __float_as_uint(fabsf(wt)));
        my_neg |= wt < 0.0f;
        if (SCATTER && wt != 0.0f) *my_wminc = max(*my_wminc, 0x7fffffffu - __float_as_uint(fabsf(wt)));
    }
    // Bricks touched along each axis: 1 or 2.
    int bl[3], nbx[3];
    float t[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int lo, hi;
        stencil_ends<SCHEME>(c[a], g.n[a], lo, hi);
        bl[a] = brick_of(lo, g.b[a], g.bmagic[a]);
        nbx[a] = (brick_of(hi, g.b[a], g.bmagic[a]) == bl[a]) ? 1 : 2;
        if (SCHEME != CAM_NGP && SCATTER) t[a] = exact_offset(pos[a], g.mn[a], g.d[a], g.inv_d[a], c[a], g.n[a]);
    }
#pragma unroll
    for (int i0 = 0; i0 < 2; ++i0) {
        if (i0 >= nbx[0]) break;
        const int b0 = (bl[0] + i0 == g.nb[0]) ? 0 : bl[0] + i0;
#pragma unroll
        for (int i1 = 0; i1 < 2; ++i1) {
            if (i1 >= nbx[1]) break;
            const int b1 = (bl[1] + i1 == g.nb[1]) ? 0 : bl[1] + i1;
#pragma unroll
            for (int i2 = 0; i2 < 2; ++i2) {
                if (i2 >= nbx[2]) break;
                const int b2 = (bl[2] + i2 == g.nb[2]) ? 0 : bl[2] + i2;
                const int key = brick_linear(g, b0, b1, b2);
                // SMEM: the CTA's shared counters (count: its histogram;
                // scatter: its own cursors into each brick's range);
                // otherwise the global counts / the brick's append cursor
                const uint32_t slot = SMEM ? atomicAdd(hist + key, 1u)
                                           : atomicAdd(table + (int64_t)key * CSTRIDE, 1u);
                if (SCATTER) {
                    const int o[3] = {b0 * g.b[0], b1 * g.b[1], b2 * g.b[2]};
                    uint32_t word[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        // Home cell relative to the brick origin: the periodic
                        // image in [-1, e], e = brick extent, which holds
                        // whenever the stencil touches the brick.
                        const int e = min(g.b[a], g.n[a] - o[a]);
                        int cl = c[a] - o[a];
                        if (cl < -1) cl += g.n[a];
                        else if (cl > e) cl -= g.n[a];
                        word[a] = pack_axis(cl, t[a]);
                    }
                    // records past the payload's capacity (a deferred
                    // estimate that fell short) or past a full slab are
                    // flagged, not written
                    const bool fits = slab ? slot < slab : slot < cap;
                    const uint64_t at = slab ? (uint64_t)key * slab + slot : (uint64_t)slot;
                    if (fits) payload[at] = make_uint4(word[0], word[1], word[2], __float_as_uint(wt));
                    else atomicOr(ovf, 1u);
                }
            }
        }
    }
}

// Cell sum q (units of 2^-s) as the output type; sc = 2^-s, so q * sc is
// exact in double (|q| < 2^63, -97 <= s <= 180) and the float output is one
// rounding of the exact value.
template <typename OutT>
__device__ __forceinline__ OutT convert_out(long long q, int s, double sc);
template <>
__device__ __forceinline__ float convert_out<float>(long long q, int, double sc)
{
    return __double2float_rn((double)q * sc);
}
template <>
__device__ __forceinline__ double convert_out<double>(long long q, int, double sc)
{
    return (double)q * sc;
}
template <>
__device__ __forceinline__ uint32_t convert_out<uint32_t>(long long q, int s, double)
{
    return (uint32_t)(q >> s);
}

// floor(i / d) for i, d < 2^16: multiply-high by m = ceil(2^32 / d) (d > 1).
__device__ __forceinline__ unsigned div_small(unsigned i, unsigned d, unsigned m)
{
    return d == 1u ? i : __umulhi(i, m);
}

// ---- the deposit tile ------------------------------------------------------
// Brick cell (li, lj, lk), each in [-1, e], has its 64-bit fixed-point sum in
// two 32-bit words of shared memory: the low word at slot
// (li + 1) kTileS0 + (lj + 1) kTileS1 + lk + 1 and the high word kTileHi
// slots further.  The strides are those of the largest brick whatever the
// brick's extent, so a record's whole stencil is one address plus constant
// offsets.  The cells at -1 and e are a halo: a record deposits its stencil
// with no per-cell test, and what lands in the halo belongs to neighbouring
// bricks (which hold the particle's own record) and is dropped -- or, along
// an axis that one brick spans, is the periodic image of the opposite edge
// and is folded back when the tile is stored.
constexpr int kTileS1 = 34;
constexpr int kTileS0 = 18 * kTileS1;
constexpr int kTileHi = 18 * kTileS0;
// Shared-memory words of the tile of a brick of extent b0 along x.
__host__ __device__ constexpr int tile_words(int b0) { return kTileHi + (b0 + 2) * kTileS0; }

// Zeroes the slots of a brick of extents e; tid of nthr threads.
__device__ __forceinline__ void zero_tile(uint32_t *tile, const int e[3], int tid, int nthr)
{
    const unsigned pw = (unsigned)((e[1] + 2) * kTileS1 + 3) / 4u;  // 16-byte words per plane
    const unsigned m = (unsigned)((0x100000000ull + pw - 1) / pw);
    const unsigned tot = (unsigned)(e[0] + 2) * pw;
    uint4 *lo = reinterpret_cast<uint4 *>(tile), *hi = reinterpret_cast<uint4 *>(tile + kTileHi);
    for (unsigned i = tid; i < tot; i += nthr) {
        const unsigned pl = div_small(i, pw, m);
        const unsigned at = pl * (kTileS0 / 4) + (i - pl * pw);
        lo[at] = make_uint4(0u, 0u, 0u, 0u);
        hi[at] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// One axis of a record: the stencil weights and the tile coordinate of the
// first of its W consecutive cells.  A TSC stencil centred on a halo cell
// (home cell -1 or e) would reach one cell past the halo: its weights are
// moved by one so that the three cells lie inside, the one that left the
// tile being replaced by a zero on the other side.
template <int SCHEME>
__device__ __forceinline__ int axis_base(uint32_t word, int e, float wa[3])
{
    int cl;
    float t;
    unpack_axis(word, cl, t);
    if (SCHEME == CAM_NGP) return min(cl, e - 1) + 1;
    if (SCHEME == CAM_CIC) {
        wa[0] = 1.0f - t;
        wa[1] = t;
        return min(cl, e - 1) + 1;
    }
    const float hm = 0.5f - t, hp = 0.5f + t;
    const float w0 = 0.5f * hm * hm, w1 = 0.75f - t * t, w2 = 0.5f * hp * hp;
    const bool below = cl < 0, above = cl >= e;
    wa[0] = below ? w1 : (above ? 0.0f : w0);
    wa[1] = below ? w2 : (above ? w0 : w1);
    wa[2] = below ? 0.0f : (above ? w1 : w2);
    return below ? 0 : (above ? e - 1 : cl);
}

// Adds W consecutive non-negative contributions (units of the quantum) to
// the cells at byte address a + OFF: one 32-bit shared atomic each, whose
// old value tells whether the low word wrapped; a wrap adds one to the high
// word.  Written as predicated instructions on immediate offsets: as C++
// (pointer arithmetic per cell, a branch around the carry) a TSC cell cost
// 18.8 warp instructions; see deposit_kernel.
template <int W, int OFF>
__device__ __forceinline__ void add_run(uint32_t a, uint32_t m0, uint32_t m1, uint32_t m2)
{
    constexpr int HI = OFF + 4 * kTileHi;
    if constexpr (W == 1) {
        asm volatile(
            "{\n\t.reg .u32 o0;\n\t.reg .pred p0;\n\t"
            "atom.shared.add.u32 o0, [%0+%2], %1;\n\t"
            "add.u32 o0, o0, %1;\n\t"
            "setp.lt.u32 p0, o0, %1;\n\t"
            "@p0 red.shared.add.u32 [%0+%3], 1;\n\t}"
            ::"r"(a), "r"(m0), "n"(OFF), "n"(HI) : "memory");
    } else if constexpr (W == 2) {
        asm volatile(
            "{\n\t.reg .u32 o0, o1;\n\t.reg .pred p0, p1;\n\t"
            "atom.shared.add.u32 o0, [%0+%3], %1;\n\t"
            "atom.shared.add.u32 o1, [%0+%4], %2;\n\t"
            "add.u32 o0, o0, %1;\n\t"
            "add.u32 o1, o1, %2;\n\t"
            "setp.lt.u32 p0, o0, %1;\n\t"
            "setp.lt.u32 p1, o1, %2;\n\t"
            "@p0 red.shared.add.u32 [%0+%5], 1;\n\t"
            "@p1 red.shared.add.u32 [%0+%6], 1;\n\t}"
            ::"r"(a), "r"(m0), "r"(m1), "n"(OFF), "n"(OFF + 4), "n"(HI), "n"(HI + 4) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .u32 o0, o1, o2;\n\t.reg .pred p0, p1, p2;\n\t"
            "atom.shared.add.u32 o0, [%0+%4], %1;\n\t"
            "atom.shared.add.u32 o1, [%0+%5], %2;\n\t"
            "atom.shared.add.u32 o2, [%0+%6], %3;\n\t"
            "add.u32 o0, o0, %1;\n\t"
            "add.u32 o1, o1, %2;\n\t"
            "add.u32 o2, o2, %3;\n\t"
            "setp.lt.u32 p0, o0, %1;\n\t"
            "setp.lt.u32 p1, o1, %2;\n\t"
            "setp.lt.u32 p2, o2, %3;\n\t"
            "@p0 red.shared.add.u32 [%0+%7], 1;\n\t"
            "@p1 red.shared.add.u32 [%0+%8], 1;\n\t"
            "@p2 red.shared.add.u32 [%0+%9], 1;\n\t}"
            ::"r"(a), "r"(m0), "r"(m1), "r"(m2), "n"(OFF), "n"(OFF + 4), "n"(OFF + 8), "n"(HI), "n"(HI + 4),
            "n"(HI + 8) : "memory");
    }
}

// The rows (i, j) of a non-negative stencil, unrolled at compile time.
template <int SCHEME, int I, int J>
__device__ __forceinline__ void add_rows(uint32_t a, float ws, float wi, const float w0[3], const float w1[3],
                                         const float w2[3])
{
    constexpr int W = Stencil<SCHEME>::W;
    const float ni = J == 0 ? ws * w0[I] : wi;
    const float wij = ni * w1[J];
    const uint32_t m0 = __float2uint_rn(wij * w2[0]);
    const uint32_t m1 = W > 1 ? __float2uint_rn(wij * w2[1]) : 0u;
    const uint32_t m2 = W > 2 ? __float2uint_rn(wij * w2[2]) : 0u;
    add_run<W, 4 * (I * kTileS0 + J * kTileS1)>(a, m0, m1, m2);
    if constexpr (J + 1 < W) add_rows<SCHEME, I, J + 1>(a, ws, ni, w0, w1, w2);
    else if constexpr (I + 1 < W) add_rows<SCHEME, I + 1, 0>(a, ws, ni, w0, w1, w2);
}

// Any contribution: signed, or of 2^32 quanta and more (a particle much
// heavier than the lightest, which sets the quantum).  |v| < 2^31 converts
// in 32 bits, the rest in 64.  The high word takes the upper 32 bits of the
// two's complement plus the carry of the low word.
__device__ __forceinline__ void add_fixed(uint32_t *lo, float v)
{
    uint32_t ql, qh;
    if (fabsf(v) < 2147483648.0f) {
        const int q = __float2int_rn(v);
        ql = (uint32_t)q;
        qh = q < 0 ? 0xffffffffu : 0u;
    } else {
        const long long q = __float2ll_rn(v);
        ql = (uint32_t)(unsigned long long)q;
        qh = (uint32_t)((unsigned long long)q >> 32);
    }
    const uint32_t old = atomicAdd(lo, ql);
    const uint32_t carry = (uint32_t)(old + ql) < old ? 1u : 0u;
    const uint32_t hadd = qh + carry;
    if (hadd) atomicAdd(lo + kTileHi, hadd);
}

// The record's stencil by add_fixed.  Not inlined: few records need it, and
// its 27 general conversions would crowd the common path out of the
// instruction cache.
struct RecordWeights {
    float w[3][3];
};
template <int SCHEME>
__device__ __noinline__ void deposit_general(RecordWeights r, float ws, uint32_t *at)
{
    constexpr int W = Stencil<SCHEME>::W;
#pragma unroll 1
    for (int i = 0; i < W; ++i)
#pragma unroll 1
        for (int j = 0; j < W; ++j) {
            const float wij = SCHEME == CAM_NGP ? ws : ws * r.w[0][i] * r.w[1][j];
#pragma unroll 1
            for (int k = 0; k < W; ++k)
                add_fixed(at + i * kTileS0 + j * kTileS1 + k, SCHEME == CAM_NGP ? wij : wij * r.w[2][k]);
        }
}

// The payload records [beg, end) of one brick into its tile; whole warps
// take 32 consecutive records (warp `warp` of nwarp), the next 32 already
// on their way.  Lanes past the end deposit zeros.  ws = weight * 2^s; the
// stencil weights are <= 1 and, up to a rounding next to a cell face (CIC),
// non-negative, so |ws| < 2^32 bounds every contribution; a warp with any
// record that this does not hold for takes the general form (the same
// integers).
template <int SCHEME>
__device__ __forceinline__ void deposit_records(const uint4 *__restrict__ payload, uint32_t beg, uint32_t end,
                                                const int e[3], float f1, float f2, bool nonneg, uint32_t *tile,
                                                int warp, int nwarp, int lane)
{
    const uint32_t tile_addr = (uint32_t)__cvta_generic_to_shared(tile);
    const uint32_t zero_word = (8u << 26) | (1u << 24);  // home cell 0, offset 0
    const uint4 none = make_uint4(zero_word, zero_word, zero_word, 0u);
    const uint32_t step = 32u * (uint32_t)nwarp;
    uint32_t p = beg + 32u * (uint32_t)warp + (uint32_t)lane;
    uint4 v = p < end ? payload[p] : none;
    for (uint32_t left = beg + 32u * (uint32_t)warp; left < end; left += step) {
        p += step;
        const uint4 vn = p < end ? payload[p] : none;
        float w0[3] = {1.f, 1.f, 1.f}, w1[3] = {1.f, 1.f, 1.f}, w2[3] = {1.f, 1.f, 1.f};
        const int i0 = axis_base<SCHEME>(v.x, e[0], w0);
        const int i1 = axis_base<SCHEME>(v.y, e[1], w1);
        const int i2 = axis_base<SCHEME>(v.z, e[2], w2);
        const float ws = (__uint_as_float(v.w) * f1) * f2;
        const int slot = i0 * kTileS0 + i1 * kTileS1 + i2;
        bool fast = nonneg && ws < 4294967296.0f;
        if (SCHEME == CAM_CIC)
            fast = fast && w0[0] >= 0.f && w0[1] >= 0.f && w1[0] >= 0.f && w1[1] >= 0.f && w2[0] >= 0.f && w2[1] >= 0.f;
        if (__all_sync(0xffffffffu, fast)) {
            add_rows<SCHEME, 0, 0>(tile_addr + 4u * (uint32_t)slot, ws, ws, w0, w1, w2);
        } else {
            const RecordWeights r = {{{w0[0], w0[1], w0[2]}, {w1[0], w1[1], w1[2]}, {w2[0], w2[1], w2[2]}}};
            deposit_general<SCHEME>(r, ws, tile + slot);
        }
        v = vn;
    }
}

// Sum of the tile's images of interior coordinates (li, lj, lk): itself and,
// along axes that one brick spans, the halo cells that are its periodic
// images (fold: bit a set for such an axis).
__device__ __forceinline__ long long folded_cell(const uint32_t *tile, int li, int lj, int lk, const int e[3],
                                                 unsigned fold)
{
    const int l[3] = {li, lj, lk};
    int img[3][3], cnt[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        cnt[a] = 1;
        img[a][0] = l[a] + 1;
        img[a][1] = img[a][2] = 0;
        if ((fold >> a) & 1u) {
            if (l[a] == 0) img[a][cnt[a]++] = e[a] + 1;
            if (l[a] == e[a] - 1) {
                if (cnt[a] == 1) img[a][1] = 0;
                else img[a][2] = 0;
                ++cnt[a];
            }
        }
    }
    unsigned long long q = 0;
    for (int i = 0; i < cnt[0]; ++i)
        for (int j = 0; j < cnt[1]; ++j)
            for (int k = 0; k < cnt[2]; ++k) {
                const int c = img[0][i] * kTileS0 + img[1][j] * kTileS1 + img[2][k];
                q += ((unsigned long long)tile[c + kTileHi] << 32) | tile[c];
            }
    return (long long)q;
}

// The tile's interior cells as OutT into the mesh (o: the brick's first
// cell, n: mesh sides), one row along z per warp; returns this thread's sum
// of the integer cell sums.
template <typename OutT>
__device__ __forceinline__ long long store_tile(const uint32_t *tile, const int o[3], const int e[3], const int n[3],
                                                unsigned fold, int s, double sc, OutT *__restrict__ mesh, int warp,
                                                int nwarp, int lane)
{
    long long acc = 0;
    const unsigned e1 = (unsigned)e[1];
    const unsigned m1 = e1 > 1u ? (unsigned)((0x100000000ull + e1 - 1) / e1) : 0u;
    if (lane < e[2]) {
        for (int r = warp; r < e[0] * e[1]; r += nwarp) {
            const int li = (int)div_small((unsigned)r, e1, m1), lj = r - li * e[1];
            const int c = (li + 1) * kTileS0 + (lj + 1) * kTileS1 + lane + 1;
            long long q;
            if (fold == 0u) q = (long long)(((unsigned long long)tile[c + kTileHi] << 32) | tile[c]);
            else q = folded_cell(tile, li, lj, lane, e, fold);
            acc += q;
            mesh[((int64_t)(o[0] + li) * n[1] + (o[1] + lj)) * n[2] + o[2] + lane] = convert_out<OutT>(q, s, sc);
        }
    }
    return acc;
}

// Pass 4: one CTA per brick, cell sums in 64-bit fixed point of quantum
// 2^-s.  The scale puts the heaviest weight just below 2^31 (one 32-bit
// atomic per contribution) unless that leaves the lightest nonzero weight
// fewer than 2^21 quanta; then the lightest sets it (2^-s <= min|w| 2^-21)
// and heavy contributions take the 64-bit path.  Either way every
// contribution of the lightest particle is rounded to within 2.4e-7 of its
// own weight, whatever the heaviest weighs.  The scale is capped so that no
// cell of the brick can overflow: a cell takes at most one contribution
// (stencil weight <= 1) per record of its brick, so max|w| 2^s * nrec <
// 2^62.  Unit weights use s = 30; NGP counts convert by a shift.
// wstat[0] = bits of max |w|, wstat[1] != 0 if some weight is negative,
// wstat[6] = 0x7fffffff - bits of min nonzero |w| (0: no nonzero weight).
__device__ __forceinline__ int fixed_scale(const unsigned int *wstat, int weighted, uint32_t nrec)
{
    float wmax = 1.0f, wmin = 1.0f;
    if (weighted) {
        if (wstat[6] == 0u) return 0;  // every weight is zero
        wmax = __uint_as_float(wstat[0]);
        wmin = __uint_as_float(0x7fffffffu - wstat[6]);
    }
    int emax = 0, emin = 0;
    frexpf(wmax, &emax);
    frexpf(wmin, &emin);
    const int bits = 32 - __clz(nrec | 1u);  // nrec < 2^bits
    return min(max(31 - emax, 22 - emin), 62 - emax - bits);
}

}  // namespace asg
}  // namespace cam
