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

// Global per-brick counters and append cursors: packed where a tile's bricks
// are advanced together (the lanes of a warp then share a request; 32 words
// apart the staged scatter of 16.8 M CIC particles onto 256^3 takes 330 us
// instead of 285), one per 128-byte line where every record takes its own
// atomic (append_kernel): those on one line are serialised in its L2 slice.
constexpr int kPaddedStride = 32;

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

// Cell centre (in cells) nearest to the position u = (x - min) / d: c + 1/2 of
// the home cell c or its periodic image.
__device__ __forceinline__ float nearest_centre(float u, float ci, float nf)
{
    const float diff = u - ci;
    if (diff > 0.5f * nf) ci += nf;
    else if (diff < -0.5f * nf) ci -= nf;
    return ci;
}

// Exact residual (x - min) - ci d, in FP32 with error-free transformations:
// TwoSum for x - min (nothing to do for min = 0) and a fused multiply-add
// for the subtraction of ci d (the product is exact inside the FMA).  The
// offset is the residual (|r| <= 1.5 d) times 1/d: |error| <= ~2e-7 cells.
__device__ __forceinline__ float exact_residual(float x, float mn, float d, float ci, bool origin)
{
    if (!origin) return __fmaf_rn(-ci, d, x);
    const float hi = __fsub_rn(x, mn);
    const float bb = __fsub_rn(hi, x);
    const float lo = __fadd_rn(__fsub_rn(x, __fsub_rn(hi, bb)), __fsub_rn(-mn, bb));
    return __fadd_rn(__fmaf_rn(-ci, d, hi), lo);
}

template <int SCHEME>
struct Stencil {
    static constexpr int W = SCHEME == CAM_NGP ? 1 : (SCHEME == CAM_CIC ? 2 : 3);
    static constexpr int FIRST = SCHEME == CAM_TSC ? -1 : 0;
};

// Payload word per axis: bits 26..31 = home cell relative to the brick + 8,
// bits 0..25 = round(t * 2^24) + 2^24 (t in [-1, 3)), the fixed-point offset.
__device__ __forceinline__ uint32_t fixed_offset(float t)
{
    const int tq = __float2int_rn(t * 16777216.0f) + 16777216;
    return (uint32_t)min(max(tq, 0), (1 << 26) - 1);
}
__device__ __forceinline__ uint32_t pack_axis(int cl, uint32_t off) { return ((uint32_t)(cl + 8) << 26) + off; }
__device__ __forceinline__ void unpack_axis(uint32_t v, int &cl, float &t)
{
    cl = (int)(v >> 26) - 8;
    t = (float)((int)(v & 0x3FFFFFFu) - 16777216) * (1.0f / 16777216.0f);
}

// Home cell c[] and fixed-point offsets off[] of any particle (false: lost).
// Out of line: few particles take it (see locate).
struct Located {
    int c[3];
    uint32_t off[3];
    bool ok;
};
template <int SCHEME>
__device__ __noinline__ Located locate_general(const AssignGeom &g, float px, float py, float pz)
{
    const float p[3] = {px, py, pz};
    Located r;
    r.ok = home_cell<SCHEME>(p, g, r.c);
    for (int a = 0; a < 3; ++a) {
        float t = 0.0f;
        if (SCHEME != CAM_NGP && r.ok) {
            const float ci = nearest_centre(__fsub_rn(p[a], g.mn[a]) * g.inv_d[a], (float)r.c[a] + 0.5f, g.nf[a]);
            t = exact_residual(p[a], g.mn[a], g.d[a], ci, true) * g.inv_d[a];
        }
        r.off[a] = fixed_offset(t);
    }
    return r;
}

// Home cell c[] of a particle as home_cell gives it (false: lost) and, with
// OFFSETS, its fixed-point offsets off[] from the cell centre.  The common
// case (see AssignGeom::safe) takes the floor by one addition of 3 2^22
// rounded down -- the float then holds the integer in its low bits -- and
// needs no test against the box: a particle outside it has a quotient outside
// [0, n).  A CIC particle in the first half cell has its home cell at -1, the
// periodic image of n - 1; with an origin the reference wraps positions below
// zero instead, whatever the origin, and so does this.  |offset| < 1.1, so it
// needs no clamp.
template <int SCHEME, bool OFFSETS>
__device__ __forceinline__ bool locate(float px, float py, float pz, const AssignGeom &g, int c[3], uint32_t off[3])
{
    constexpr int LOW = SCHEME == CAM_CIC ? 1 : 0;
    const float p[3] = {px, py, pz};
    float ci[3], image[3];
    bool rare = false;
    const bool origin = g.origin != 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float v = SCHEME == CAM_CIC ? __fsub_rn(p[a], g.half_d[a]) : p[a];
        image[a] = 0.0f;
        if (SCHEME == CAM_CIC && origin) {
            if (v < 0.0f) {
                v = __fadd_rn(v, g.L[a]);
                image[a] = -g.nf[a];
            }
            if (v >= g.L[a]) {
                v = __fsub_rn(v, g.L[a]);
                image[a] += g.nf[a];
            }
        }
        const float u = __fmul_rn(__fsub_rn(v, g.mn[a]), g.inv_d[a]);
        const float f = __fadd_rd(u, 12582912.0f);
        const int k = __float_as_int(f) - (0x4b400000 - LOW);  // home cell, + 1 for CIC
        ci[a] = (f - 12582912.0f) + 0.5f;
        rare = rare || !(fabsf(u - ci[a]) < g.safe[a]) || (unsigned)k >= (unsigned)(g.n[a] + LOW);
        if (SCHEME == CAM_CIC && origin) rare = rare || k == 0;
        c[a] = SCHEME == CAM_CIC ? (k == 0 ? g.n[a] - 1 : k - 1) : k;
    }
    if (rare) {
        const Located r = locate_general<SCHEME>(g, px, py, pz);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            c[a] = r.c[a];
            off[a] = r.off[a];
        }
        return r.ok;
    }
    if (OFFSETS) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (SCHEME == CAM_NGP) {
                off[a] = 1u << 24;
                continue;
            }
            const float r = exact_residual(p[a], g.mn[a], g.d[a], ci[a] + image[a], origin);
            off[a] = (uint32_t)(__float2int_rn(r * g.off_scale[a]) + 16777216);
        }
    }
    return true;
}

// The brick of a particle's first stencil cell along axis a: its coordinate
// bl, the home cell relative to it (cl in [0, e], e its extent), and whether
// the stencil reaches into the next brick (periodic).
template <int SCHEME>
__device__ __forceinline__ bool brick_axis(const AssignGeom &g, int a, int c, int &bl, int &cl)
{
    const int lo = SCHEME == CAM_TSC ? (c == 0 ? g.lo0[a] : c - 1) : c;
    bl = (int)__umulhi((unsigned)lo, g.bmagic[a]);
    const int in = lo - bl * g.b[a];
    cl = SCHEME == CAM_TSC ? in + 1 : in;
    if (SCHEME == CAM_NGP) return false;
    return in >= g.cross_b[a] || lo >= g.cross_n[a];
}

// Step of the brick number to the next brick along each axis (periodic).
__device__ __forceinline__ void key_steps(const AssignGeom &g, const int bl[3], int step[3])
{
    const int s1 = g.nb[2], s0 = g.nb[1] * g.nb[2];
    step[0] = (bl[0] + 1 == g.nb[0] ? -bl[0] : 1) * s0;
    step[1] = (bl[1] + 1 == g.nb[1] ? -bl[1] : 1) * s1;
    step[2] = bl[2] + 1 == g.nb[2] ? -bl[2] : 1;
}

// A record as the next brick along the axes of mask m sees it: the home
// cell relative to a brick falls by the extent of the brick before it.
__device__ __forceinline__ uint4 next_brick_record(const AssignGeom &g, uint4 r, const int bl[3], unsigned m)
{
    auto ext = [&](int a) { return (uint32_t)(bl[a] == g.nb[a] - 1 ? g.e_last[a] : g.b[a]) << 26; };
    if (m & 1u) r.x -= ext(0);
    if (m & 2u) r.y -= ext(1);
    if (m & 4u) r.z -= ext(2);
    return r;
}

// Weight statistics of a thread's particles: largest |w| (bits), smallest
// w, and smallest nonzero |w| as bits - 1 (a zero weight wraps to the
// largest value).
struct WeightStats {
    unsigned wmax = 0u, wmin1 = 0xffffffffu;
    float low = 0.0f;
    __device__ __forceinline__ void add(float w)
    {
        const unsigned b = __float_as_uint(w) & 0x7fffffffu;
        wmax = max(wmax, b);
        wmin1 = min(wmin1, b - 1u);
        low = fminf(low, w);
    }
    // the words of wstat (fixed_scale): some weight is negative; 0x7fffffff
    // minus the bits of the smallest nonzero |w| (0: every weight is zero)
    __device__ __forceinline__ unsigned neg() const { return low < 0.0f ? 1u : 0u; }
    __device__ __forceinline__ unsigned wminc() const { return wmin1 == 0xffffffffu ? 0u : 0x7fffffffu - (wmin1 + 1u); }
};

// One particle of the count pass: the bricks its stencil touches (the brick
// of its first stencil cell and, along each axis whose stencil crosses a
// brick face, the next brick, periodically) each get one count.
template <int SCHEME, bool SMEM>
__device__ __forceinline__ void count_one(float px, float py, float pz, float wt, bool weighted, const AssignGeom &g,
                                          uint32_t *hist, uint32_t *__restrict__ table, unsigned int &my_lost,
                                          WeightStats &ws)
{
    int c[3], bl[3], cl, step[3];
    uint32_t off[3];
    if (!locate<SCHEME, false>(px, py, pz, g, c, off)) {
        ++my_lost;
        return;
    }
    if (weighted) ws.add(wt);
    unsigned cross = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) cross |= brick_axis<SCHEME>(g, a, c[a], bl[a], cl) ? 1u << a : 0u;
    const int key = (bl[0] * g.nb[1] + bl[1]) * g.nb[2] + bl[2];
    auto add = [&](int k) {
        if (SMEM) atomicAdd(hist + k, 1u);
        else atomicAdd(table + (int64_t)k * g.cstride, 1u);
    };
    add(key);
    if (SCHEME == CAM_NGP || cross == 0u) return;
    key_steps(g, bl, step);
    // unrolled: some lane of nearly every warp takes most of the seven
#pragma unroll
    for (unsigned m = 1; m < 8; ++m)
        if ((cross & m) == m) add(key + (m & 1u ? step[0] : 0) + (m & 2u ? step[1] : 0) + (m & 4u ? step[2] : 0));
}

// Writes one record at `slot` of brick `key`: slab > 0, its own slab of
// `slab` records (payload[key * slab + slot]); otherwise payload[slot].
// Records past a full slab or past the payload's capacity (a deferred
// estimate that fell short) are flagged, not written.
__device__ __forceinline__ void put_record(uint4 *__restrict__ payload, uint4 rec, int key, uint32_t slot,
                                           uint32_t slab, uint64_t cap, unsigned int *ovf)
{
    const bool fits = slab ? slot < slab : slot < cap;
    const uint64_t at = slab ? (uint64_t)key * slab + slot : (uint64_t)slot;
    if (fits) payload[at] = rec;
    else atomicOr(ovf, 1u);
}

// One particle appended record by record: every touched brick's cursor
// (cursor[key * g.cstride]) gives the next slot.  Returns false if it is lost.
template <int SCHEME>
__device__ __forceinline__ bool append_one(float px, float py, float pz, float wt, const AssignGeom &g,
                                           uint32_t *__restrict__ cursor, uint4 *__restrict__ payload, uint64_t cap,
                                           unsigned int *ovf, uint32_t slab)
{
    int c[3], bl[3], cl[3], step[3];
    uint32_t off[3];
    if (!locate<SCHEME, true>(px, py, pz, g, c, off)) return false;
    unsigned cross = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) cross |= brick_axis<SCHEME>(g, a, c[a], bl[a], cl[a]) ? 1u << a : 0u;
    const int key = (bl[0] * g.nb[1] + bl[1]) * g.nb[2] + bl[2];
    const uint32_t slot = atomicAdd(cursor + (int64_t)key * g.cstride, 1u);
    const uint4 rec = make_uint4(pack_axis(cl[0], off[0]), pack_axis(cl[1], off[1]), pack_axis(cl[2], off[2]),
                                 __float_as_uint(wt));
    put_record(payload, rec, key, slot, slab, cap, ovf);
    if (SCHEME == CAM_NGP || cross == 0u) return true;
    key_steps(g, bl, step);
#pragma unroll
    for (unsigned m = 1; m < 8; ++m) {
        if ((cross & m) != m) continue;
        const int k = key + (m & 1u ? step[0] : 0) + (m & 2u ? step[1] : 0) + (m & 4u ? step[2] : 0);
        const uint32_t sl = atomicAdd(cursor + (int64_t)k * g.cstride, 1u);
        put_record(payload, next_brick_record(g, rec, bl, m), k, sl, slab, cap, ovf);
    }
    return true;
}

// Cell sum q (units of 2^-s) as the output type; sc = 2^-s (-97 <= s <= 180).
// Up to |q| = 2^53 q * sc is exact in double and the float output one rounding
// of the exact value; a larger sum is rounded to double first.
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

// A thread's share of the payload records [beg, end) of one brick: whole
// warps take 32 consecutive records (warp `warp` of nwarp), two such groups
// ahead of the one in work; open() starts the first loads, so that they run
// while the tile is zeroed.  Lanes past the end get a record of weight zero.
struct RecordStream {
    const uint4 *payload;
    uint32_t p, first, end, step;
    uint4 a, b;
    __device__ __forceinline__ uint4 load(uint32_t i) const
    {
        const uint32_t zero_word = (8u << 26) | (1u << 24);  // home cell 0, offset 0
        return i < end ? __ldcs(payload + i) : make_uint4(zero_word, zero_word, zero_word, 0u);
    }
    __device__ __forceinline__ void open(const uint4 *__restrict__ pay, uint32_t beg, uint32_t end_, int warp, int nwarp,
                                         int lane)
    {
        payload = pay;
        end = end_;
        step = 32u * (uint32_t)nwarp;
        first = beg + 32u * (uint32_t)warp;
        p = first + (uint32_t)lane;
        a = load(p);
        b = load(p + step);
    }
};

// Deposits a brick's records into its tile.  ws = weight * 2^s; the stencil
// weights are <= 1 and, up to a rounding next to a cell face (CIC),
// non-negative, so |ws| < 2^32 bounds every contribution; a warp with any
// record that this does not hold for takes the general form (the same
// integers).
template <int SCHEME>
__device__ __forceinline__ void deposit_records(RecordStream &r, const int e[3], float f1, float f2, bool nonneg,
                                                uint32_t *tile)
{
    const uint32_t tile_addr = (uint32_t)__cvta_generic_to_shared(tile);
#pragma unroll 1
    for (uint32_t left = r.first; left < r.end; left += r.step) {
        const uint4 v = r.a;
        r.a = r.b;
        r.b = r.load(r.p + 2u * r.step);
        r.p += r.step;
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
            const RecordWeights rw = {{{w0[0], w0[1], w0[2]}, {w1[0], w1[1], w1[2]}, {w2[0], w2[1], w2[2]}}};
            deposit_general<SCHEME>(rw, ws, tile + slot);
        }
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
// wstat[4] != 0 (deposit_kernel only): some records were not written.
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
