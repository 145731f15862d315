// Device kernels of the PBF solver step (sm_103a).
//
// One thread per particle; blocks walk a device-resident tile list in a
// grid-stride loop, each tile belonging to one scene, so the same kernels run
// a single scene (the plain step) or hundreds of scenes (the batched engine)
// with a fixed launch shape that a CUDA graph can capture once.
//
// Data layout (flat arrays over every scene's particle slots):
//   x, v                          : float4, the particles' state (xyz)
//   xs                            : float4, sorted positions; later (x, |omega|)
//   xa, xb                        : float4, working positions; (position, lambda)
//   xold                          : float4, old position, sorted slot in w
//   pa, pb                        : float4 + float2, (x, v) for the post passes
//   w, vs                         : float4, vorticity; velocities in sorted order
//   key, slot, tmp, perm          : uint32 per particle
//   nbr                           : rows of 16 bytes per particle (4 u32 or 8 u16
//                                   list slots), row after row
//   count / offsets               : uint32 per cell (+1 deleted bucket per scene)
//
// Integer work (predict, cell hash, stable counting sort, neighbour
// acceptance) uses explicitly rounded intrinsics so that it is bit-exact
// against the CPU oracle.  Floating-point solver math follows the reference's
// operation order but uses rsqrtf (as the reference does).
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "pbf_internal.h"
#include "pbf_scan.cuh"
#include "pbf_sort.cuh"
#include "pbf103.h"

namespace pbf103 {
namespace {

// ---------------------------------------------------------------- helpers --

// static_cast<int>(floor(p / cell_width)), src/pbf/interaction/cuda/pbf_grid.h:20-33,
// with IEEE division (the reference build used -prec-div=false).
__device__ __forceinline__ int32_t cell_coord(float p, float cw)
{
    return __float2int_rd(__fdiv_rn(p, cw));
}

// calcGridHash with power-of-two wrap, pbf_grid.h:53-61.
__device__ __forceinline__ uint32_t hash3(uint32_t x, uint32_t y, uint32_t z, const SceneDesc &d)
{
    x &= d.gx - 1u;
    y &= d.gy - 1u;
    z &= d.gz - 1u;
    return z * d.gx * d.gy + y * d.gx + x;
}

// Alias class of a cell: which of the 2 x 2 x 2 periodic copies of the
// power-of-two table the (unwrapped) cell lies in.  With the table sized for
// cells of 2h (calcGridSize, pbf_type.cpp:141-162) but cells h wide, a
// bucket holds particles of cells G apart; only one class of a bucket can
// hold neighbours of a given cell.  Cells 2G apart share a class; they are
// far apart, so the distance test still rejects them.
__device__ __forceinline__ uint32_t alias_class(int32_t cx, int32_t cy, int32_t cz, const SceneDesc &d)
{
    const int sx = __ffs(d.gx) - 1, sy = __ffs(d.gy) - 1, sz = __ffs(d.gz) - 1;
    return (uint32_t)(((cz >> sz) & 1) << 2 | ((cy >> sy) & 1) << 1 | ((cx >> sx) & 1));
}

// Packed FP32 (two lanes of one 64-bit register pair per instruction):
// each lane is rounded exactly as the scalar operation (flush-to-zero like
// the rest of the build), so a pair of x and y terms costs one instruction
// and gives the scalar bits.
__device__ __forceinline__ void sub2(float &d0, float &d1, float a0, float a1, float b0, float b1)
{
    asm("{\n\t.reg .b64 pa, pb, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\t"
        "mov.b64 pb, {%4, %5};\n\t"
        "sub.rn.ftz.f32x2 pd, pa, pb;\n\t"
        "mov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// c0 = fma(a0, b0, c0), c1 = fma(a1, b1, c1)
__device__ __forceinline__ void fma2(float &c0, float &c1, float a0, float a1, float b0, float b1)
{
    asm("{\n\t.reg .b64 pa, pb, pc;\n\t"
        "mov.b64 pa, {%2, %3};\n\t"
        "mov.b64 pb, {%4, %5};\n\t"
        "mov.b64 pc, {%0, %1};\n\t"
        "fma.rn.ftz.f32x2 pc, pa, pb, pc;\n\t"
        "mov.b64 {%0, %1}, pc;\n\t}"
        : "+f"(c0), "+f"(c1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// r^2 exactly as findPair computes it (pbf_neighbor_search_util.cu:398):
// fmaf(dz, dz, fmaf(dy, dy, dx * dx)), no further contraction.
__device__ __forceinline__ float dist2_exact(float4 a, float4 b)
{
    float d0, d1;
    sub2(d0, d1, a.x, a.y, b.x, b.y);
    const float d2 = __fsub_rn(a.z, b.z);
    return __fmaf_rn(d2, d2, __fmaf_rn(d1, d1, __fmul_rn(d0, d0)));
}

// A listed pair at current positions (memorizeKernelPair,
// src/pbf/solver/cuda/pbf_kernel_memorization.cu:14-56, restated): the
// difference d = x_i - x_j, r^2, the poly6 value W = alpha w and the spiky
// gradient grad W = beta s d, with the scene factors alpha and beta left
// out of the per-pair terms (the sums apply them once per particle):
//   w = (1 - r^2 / h^2)^3                for r <= h, else 0
//   s = (1 - r / h)^2 / r                for 0 < r <= h, else 0
//   sr = s r = |grad W| / |beta|
// The clamps replace the reference's branches: 1 - r^2/h^2 and 1 - r/h are
// clamped at 0 (r > h), and r^2 enters the reciprocal square root no smaller
// than kMinR2, so a pair at distance 0 (d = 0, r = 0) gets a finite s (up
// to 1e15), a gradient s d of exactly 0 and sr = 0, as the reference's
// r^2 > 0 test gives.  |grad W|^2 is taken as sr^2, not s^2 r^2: the
// latter overflows at r = 0.
// Products and sums are rounded one by one or fused where written
// (__fmaf_rn), never contracted by the compiler, so every pass that calls
// these, in one lane or split over lanes, gets the same bits.
constexpr float kMinR2 = 1e-30f;

struct PairGeo {
    float d0, d1, d2, r2;
};

// PK: d0 and d1 by one packed subtraction (the same bits; faster in the
// delta-p pass of large steps, slower in the small steps' passes: measured)
template <bool PK = false>
__device__ __forceinline__ PairGeo pair_geo(float4 xi, float4 xj)
{
    PairGeo g;
    if (PK) {
        sub2(g.d0, g.d1, xi.x, xi.y, xj.x, xj.y);
    } else {
        g.d0 = __fsub_rn(xi.x, xj.x);
        g.d1 = __fsub_rn(xi.y, xj.y);
    }
    g.d2 = __fsub_rn(xi.z, xj.z);
    g.r2 = __fmaf_rn(g.d2, g.d2, __fmaf_rn(g.d1, g.d1, __fmul_rn(g.d0, g.d0)));
    return g;
}

struct PairWS {
    float W, s, sr;
};

// per-scene constants of the pair math, in registers for a particle's loop
struct PairConst {
    float ih2, inv_h;
};

__device__ __forceinline__ PairConst pair_const(const SceneDesc &d) { return PairConst{d.ih2, d.inv_h}; }

__device__ __forceinline__ PairWS pair_ws(float r2, const PairConst &c)
{
    const float inv_r = rsqrtf(fmaxf(r2, kMinR2));
    const float t = fmaxf(__fmaf_rn(-r2, c.ih2, 1.f), 0.f);
    const float W = __fmul_rn(__fmul_rn(t, t), t);
    const float r = __fmul_rn(r2, inv_r);
    const float u = fmaxf(__fmaf_rn(-r, c.inv_h, 1.f), 0.f);
    const float s = __fmul_rn(inv_r, __fmul_rn(u, u));
    return PairWS{W, s, __fmul_rn(s, r)};
}

// The sums of calcScalingFactorCUDA (pbf_constraint.cu:168-209) over a
// particle's list, added in list order, without the factors alpha and
// beta: sum w (W = alpha w), sum s d (grad W = beta s d) and sum (s r)^2.
// A particle's own pair (w = 1, no gradient) is not stored in its list; the
// passes start ks at 1 for it.
struct LamSum {
    float ks = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f, kg2 = 0.f;
    __device__ __forceinline__ void add(float W, float s, float d0, float d1, float d2, float sr)
    {
        ks = __fadd_rn(ks, W);
        g0 = __fmaf_rn(s, d0, g0);
        g1 = __fmaf_rn(s, d1, g1);
        g2 = __fmaf_rn(s, d2, g2);
        kg2 = __fmaf_rn(sr, sr, kg2);
    }
    __device__ __forceinline__ void add(const PairGeo &g, const PairWS &k) { add(k.W, k.s, g.d0, g.d1, g.d2, k.sr); }
    // lambda = C / (m^2 / rho0^2 |grad C|^2 + eps), with C = alpha m / rho0
    // sum w - 1 and m^2 / rho0^2 |grad C|^2 = m^2 beta^2 / rho0^2 K
    __device__ __forceinline__ float lambda(const SceneDesc &d) const
    {
        const float C = __fmaf_rn(ks, d.lam_c, -1.f);
        const float K = __fmaf_rn(g0, g0, __fmaf_rn(g2, g2, __fmaf_rn(g1, g1, kg2)));
        return __fdiv_rn(C, __fmaf_rn(d.lam_k, K, d.relax));
    }
};

// A pair past the list's end adds exactly nothing: its W, s and s r are 0
// (its difference is finite: small steps pad with the particle itself, whose
// difference is 0 or, for a non-finite position, NaN, as all its sums are).
__device__ __forceinline__ PairWS masked(const PairWS &k, bool on)
{
    return PairWS{on ? k.W : 0.f, on ? k.s : 0.f, on ? k.sr : 0.f};
}

// one listed pair's terms of the lambda sums
__device__ __forceinline__ void lam_add(LamSum &ls, float4 xi, float4 xj, const PairConst &c)
{
    const PairGeo g = pair_geo(xi, xj);
    ls.add(g, pair_ws(g.r2, c));
}

// WspikyDerivative, src/pbf/kernel/cuda/detail/pbf_kernel.inl:48-63.
__device__ __forceinline__ float wspiky_d(float r, float kinv_h)
{
    const float q = r * kinv_h;
    if (q <= 1.f) {
        const float ih2 = kinv_h * kinv_h;
        const float t = 1.f - q;
        return -14.3239448745f * (ih2 * ih2) * t * t;
    }
    return 0.f;
}

// responseInnerSphereBoundary, src/pbf/solver/cuda/boundary/pbf_sphere_boundary.cu:8-34
__device__ __forceinline__ void inner_sphere(bool &hit, float3 &dp, float3 p, float4 s)
{
    const float c0 = s.x - p.x, c1 = s.y - p.y, c2 = s.z - p.z;
    const float d2 = fmaf(c2, c2, fmaf(c1, c1, c0 * c0));
    if (d2 > s.w * s.w) {
        const float rinv = rsqrtf(d2);
        hit = true;
        dp.x = fmaf(c0, 1.0001f, dp.x);
        dp.y = fmaf(c1, 1.0001f, dp.y);
        dp.z = fmaf(c2, 1.0001f, dp.z);
        dp.x = fmaf(-s.w, c0 * rinv, dp.x);
        dp.y = fmaf(-s.w, c1 * rinv, dp.y);
        dp.z = fmaf(-s.w, c2 * rinv, dp.z);
    }
}

// responsePlaneBoundary, src/pbf/solver/cuda/boundary/pbf_plane_boundary.cu:6-45.
// Both of its hit cases need the projected point p behind the plane
// ((p - on) . n < 0); that is tested first, so a particle clear of the plane
// (the common case) skips the rest, with the same result.
__device__ __forceinline__ void plane(bool &hit, float3 &dp, float3 o, float3 p, float4 on, float4 n)
{
    const float pb0 = p.x - on.x, pb1 = p.y - on.y, pb2 = p.z - on.z;
    const float pb_n = fmaf(pb2, n.z, fmaf(pb1, n.y, pb0 * n.x));
    if (!(pb_n < 0.f)) return;
    const float pa0 = o.x - on.x, pa1 = o.y - on.y, pa2 = o.z - on.z;
    const float pa_n = fmaf(pa2, n.z, fmaf(pa1, n.y, pa0 * n.x));
    float3 is;
    if (pa_n == 0.f && pb_n == 0.f) {
        return;
    } else if (pa_n >= 0.f && pb_n < 0.f) {
        hit = true;
        const float f = fabsf(pa_n) / (fabsf(pa_n) + fabsf(pb_n));
        is.x = o.x + (p.x - o.x) * f;
        is.y = o.y + (p.y - o.y) * f;
        is.z = o.z + (p.z - o.z) * f;
    } else if (pa_n < 0.f && pb_n < 0.f) {
        hit = true;
        const float dd = -fmaf(on.z, n.z, fmaf(on.y, n.y, on.x * n.x));
        const float t = -(fmaf(p.z, n.z, fmaf(p.y, n.y, p.x * n.x)) + dd) / fmaf(n.z, n.z, fmaf(n.y, n.y, n.x * n.x));
        is.x = p.x + t * n.x;
        is.y = p.y + t * n.y;
        is.z = p.z + t * n.z;
    } else {
        return;
    }
    const float di0 = p.x - is.x, di1 = p.y - is.y, di2 = p.z - is.z;
    const float c = fmaf(di2, n.z, fmaf(di1, n.y, di0 * n.x));
    dp.x += -c * n.x;
    dp.y += -c * n.y;
    dp.z += -c * n.z;
}

// responseCollisionCUDA, src/pbf/solver/cuda/pbf_response_collision.cu:12-66 (and the
// fixed-sphere variant, pbf_constraint.cu:262-315).  old_x is the current
// position, as in the reference (pbf_response_collision.cu:31).  The
// reference repeats until no primitive reports a hit; here at most max_coll
// passes.  Returns false when the bound was reached.  A pass is a function
// of dp alone, so a pass that hits but leaves dp bit-for-bit unchanged (a
// projection too small to move the position, which the reference would
// repeat forever) would repeat identically up to the bound: the loop stops
// there with the same dp and the same result.
__device__ bool collide(const SceneDesc &d, const float4 *__restrict__ bnd, float3 x, float3 &dp)
{
    if (d.clear_box) {  // a box's walls: a position inside the clear box hits none, so pass 1 is the last
        const float px = x.x + dp.x, py = x.y + dp.y, pz = x.z + dp.z;
        if (d.box_lo[0] <= px && px <= d.box_hi[0] && d.box_lo[1] <= py && py <= d.box_hi[1] &&
            d.box_lo[2] <= pz && pz <= d.box_hi[2])
            return true;
    }
    for (uint32_t pass = 0; pass < d.max_coll; ++pass) {
        const float3 before = dp;
        float3 p = make_float3(x.x + dp.x, x.y + dp.y, x.z + dp.z);
        bool hit = false;
        if (d.builtin_sphere) {
            inner_sphere(hit, dp, p, make_float4(3.f, 3.f, 3.f, 3.f));
        } else {
            const float4 *b = bnd + d.b_off;
            const uint32_t ns = d.n_inner + d.n_outer;  // outer spheres use the inner routine
            for (uint32_t k = 0; k < ns; ++k) {
                inner_sphere(hit, dp, p, __ldg(b + k));
                p = make_float3(x.x + dp.x, x.y + dp.y, x.z + dp.z);
            }
            b += ns;
            for (uint32_t k = 0; k < d.n_planes; ++k) {
                plane(hit, dp, x, p, __ldg(b + 2 * k), __ldg(b + 2 * k + 1));
                p = make_float3(x.x + dp.x, x.y + dp.y, x.z + dp.z);
            }
        }
        if (!hit) return true;
        if (__float_as_uint(dp.x) == __float_as_uint(before.x) && __float_as_uint(dp.y) == __float_as_uint(before.y) &&
            __float_as_uint(dp.z) == __float_as_uint(before.z))
            return false;  // fixed point: every later pass repeats this one
    }
    return false;
}

// Visit the particles of the 27 cells around xp in the reference's order
// (z, y, x from -1 to 1; ascending sorted index inside a cell,
// pbf_neighbor_search_util.cu:428-452), as contiguous sorted-index ranges:
// r(st, en) gets [st, en) and returns false to stop the walk.  When the
// three x-cells of a row are consecutive hashes their particles form one
// range.  Every cell is visited (the reference-form XSPH and vorticity
// walks); with fewer than 3 cells on an axis a wrapped cell is visited more
// than once, as in the reference.
template <class R>
__device__ __forceinline__ void walk27_ranges(const SceneDesc &d, const uint32_t *__restrict__ offsets,
                                              uint32_t shift, float4 xp, R &&r)
{
    const uint32_t gx = (uint32_t)cell_coord(xp.x, d.cw), gy = (uint32_t)cell_coord(xp.y, d.cw),
                   gz = (uint32_t)cell_coord(xp.z, d.cw);
    const uint32_t *off = offsets + d.c_off;
    const uint32_t mx = d.gx - 1u;
    const uint32_t x0c = (gx - 1u) & mx, x2c = (gx + 1u) & mx;
    const bool contiguous = (x2c == x0c + 2u);
#pragma unroll 1
    for (int rr = 0; rr < 9; ++rr) {
        const int dz = rr / 3 - 1, dy = rr % 3 - 1;
        const uint32_t row = ((gz + (uint32_t)dz) & (d.gz - 1u)) * d.gx * d.gy +
                             ((gy + (uint32_t)dy) & (d.gy - 1u)) * d.gx;
        const uint32_t nseg = contiguous ? 1u : 3u;
#pragma unroll 1
        for (uint32_t sg = 0; sg < nseg; ++sg) {
            const uint32_t lo = contiguous ? x0c : (gx + sg - 1u) & mx;
            const uint32_t hi = contiguous ? x2c : lo;
            if (!r(__ldg(off + row + lo) + shift, __ldg(off + row + hi + 1u) + shift)) return;
        }
    }
}

// The neighbour-search walk: the same 27 cells in the same order as
// walk27_ranges, one range per cell, and inside a cell's bucket only the
// particles of the cell's alias class (chist holds the bucket's class
// ends): a bucket of one class is its range, a bucket
// without the class is skipped, and a mixed bucket gives the class's
// sub-range (working slots hold a mixed bucket grouped by class).
// Candidates of the other classes lie at least G - 1 cells away and can
// never be accepted, and each class keeps its sorted order, so the
// accepted sequence is the reference's.  Buckets marked kClassWhole (and
// every bucket of a scene with an axis of fewer than 4 cells, where the
// reference visits wrapped cells twice) are visited whole, in sorted order.
// r(st, en) gets the range of working slots.
//
// The walk is restricted to cells that can hold a particle within h of xp
// (the binned position): a cell whose nearest point is farther than h holds
// no accepted candidate, so skipping it leaves the visited sequence of
// accepted candidates unchanged.  A 1e-3 relative margin covers the rounding
// of the cell assignment.  It applies only when every axis has at least 4
// cells (with fewer, the reference visits wrapped cells more than once).
template <class R>
__device__ __forceinline__ void walk27_cells(const SceneDesc &d, const uint32_t *__restrict__ offsets,
                                             const uint64_t *__restrict__ chist, uint32_t shift, float4 xp, R &&r)
{
    const int32_t icx = cell_coord(xp.x, d.cw), icy = cell_coord(xp.y, d.cw), icz = cell_coord(xp.z, d.cw);
    const bool prune = d.gx >= 4 && d.gy >= 4 && d.gz >= 4;
    float lx = 0.f, ly = 0.f, lz = 0.f, rx = 0.f, ry = 0.f, rz = 0.f;
    if (prune) {
        lx = xp.x - (float)icx * d.cw;
        ly = xp.y - (float)icy * d.cw;
        lz = xp.z - (float)icz * d.cw;
        rx = d.cw - lx;
        ry = d.cw - ly;
        rz = d.cw - lz;
    }
    const float lim = d.h2 * 1.001f;
    const int sx = __ffs(d.gx) - 1, sy = __ffs(d.gy) - 1, sz = __ffs(d.gz) - 1;
    const uint32_t *off = offsets + d.c_off;
    const uint64_t *ch = chist + d.c_off;
    // The walk is bound by issued instructions (75% issue-active).  The loops
    // leave by their conditions alone (no continue, no return), so every
    // branch meets again at its own loop's end and a warp's lanes walk the
    // same cell together: at 5.95 M particles in 256 scenes the list walk
    // took 1,376 us with early exits, 1,333 without; a class's range by two
    // byte selections instead of counts and a byte sum, 1,405 -> 1,376.
    bool go = true;
#pragma unroll 1
    for (int rr = 0; rr < 9 && go; ++rr) {  // rows (dz, dy), z outermost: the reference's walk order
        const int dz = rr / 3 - 1, dy = rr % 3 - 1;
        bool mid = true, left = true, right = true;
        if (prune) {
            const float ez = dz < 0 ? lz : (dz > 0 ? rz : 0.f);
            const float ey = dy < 0 ? ly : (dy > 0 ? ry : 0.f);
            const float eyz2 = ey * ey + ez * ez;
            mid = eyz2 <= lim;
            left = eyz2 + lx * lx <= lim;
            right = eyz2 + rx * rx <= lim;
        }
        if (mid) {
            const int32_t ty = icy + dy, tz = icz + dz;
            const uint32_t row = ((uint32_t)tz & (d.gz - 1u)) * d.gx * d.gy + ((uint32_t)ty & (d.gy - 1u)) * d.gx;
            const uint32_t cyz = (uint32_t)(((tz >> sz) & 1) << 2 | ((ty >> sy) & 1) << 1);
#pragma unroll 1
            for (int dx = -1; dx <= 1 && go; ++dx) {
                if (dx == 0 || (dx < 0 ? left : right)) {
                    const int32_t tx = icx + dx;
                    const uint32_t b = row + ((uint32_t)tx & (d.gx - 1u));
                    uint32_t st = __ldg(off + b);
                    uint32_t en = __ldg(off + b + 1);
                    const uint64_t h = __ldg(reinterpret_cast<const unsigned long long *>(ch + b));
                    // an empty bucket's class ends are stale: leave its range empty
                    if (h != kClassWhole && st != en) {  // the class's sub-range
                        const uint32_t c = cyz | (uint32_t)((tx >> sx) & 1);
                        const uint32_t h0 = (uint32_t)h, h1 = (uint32_t)(h >> 32);
                        en = st + (__byte_perm(h0, h1, c) & 0xFFu);
                        st += __byte_perm(h0 << 8, __funnelshift_l(h0, h1, 8), c) & 0xFFu;
                    }
                    if (st < en) go = r(st + shift, en + shift);
                }
            }
        }
    }
}

// walk27 with the per-neighbour work taken out of the walk: candidates that
// pass accept(j) are queued in a small per-thread buffer and handed to use(j)
// in batches, so the neighbour math is not executed masked for every
// candidate of the walk.  use() sees the accepted candidates in walk order.
template <class A, class U>
__device__ __forceinline__ void walk27_batched(const SceneDesc &d, const uint32_t *__restrict__ offsets,
                                               uint32_t shift, float4 xp, A &&accept, U &&use)
{
    constexpr int kBuf = 32;
    uint32_t buf[kBuf];
    int nb = 0;
    walk27_ranges(d, offsets, shift, xp, [&](uint32_t st, uint32_t en) -> bool {
        for (uint32_t j = st; j < en; ++j) {
            if (accept(j)) {
                buf[nb++] = j;
                if (nb == kBuf) {
                    for (int k = 0; k < kBuf; ++k) use(buf[k]);
                    nb = 0;
                }
            }
        }
        return true;
    });
    for (int k = 0; k < nb; ++k) use(buf[k]);
}

// The neighbour list is stored in quads of slots: slot k of particle slot i
// at nbr[(k / 4 * stride + i) * 4 + k % 4] (stride = particle slots), so a
// thread's four consecutive slots are one aligned 16-byte load and the
// quads of a warp's particles lie side by side (coalesced).  list_of is a
// particle's base, list_slot the offset of its slot k.
__device__ __forceinline__ uint32_t *list_of(uint32_t *nbr, uint32_t i) { return nbr + 4ull * i; }
__device__ __forceinline__ uint64_t list_slot(uint32_t k, uint64_t stride)
{
    return (uint64_t)(k >> 2) * stride * 4u + (k & 3u);
}

// One 16-byte row of a particle's list (a quad of u32 or an oct of u16
// slots), loaded and stored as streaming data (evict-first): the lists of a
// batch (hundreds of MB) pass through L2 once per pass, and the hint keeps
// them from evicting the positions the same passes gather (batched step
// +1%, the list-form vorticity pass -4%, interleaved A/B).
__device__ __forceinline__ uint4 list_ld(const uint4 *p) { return __ldcs(p); }
__device__ __forceinline__ void list_st(uint4 *p, uint4 v) { __stcs(p, v); }

__device__ __forceinline__ uint32_t quad_at(const uint4 &v, int j)
{
    return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w));
}

// Scenes of at most kList16Max particle slots (every batched scene) keep
// their lists as u16 scene-local indices in octs of 8 slots: slot k of
// particle slot i at nbr16[((k / 8) * stride + i) * 8 + k % 8], the same
// 16-byte rows as the quads of u32 lists, half as many of them, so a pass
// reads half the list bytes.  list16_slot is the u16 offset of slot k from
// the particle's base (list_of, as for quads).
__device__ __forceinline__ uint64_t list16_slot(uint32_t k, uint64_t stride)
{
    return (uint64_t)(k >> 3) * stride * 8u + (k & 7u);
}

__device__ __forceinline__ uint32_t oct_at(const uint4 &v, int j)
{
    const uint32_t w = j < 2 ? v.x : (j < 4 ? v.y : (j < 6 ? v.z : v.w));
    return (j & 1) ? (w >> 16) : (w & 0xFFFFu);
}

// Visit slots [k0, k0 + n) of a particle's list: ld(q) loads the record of
// index q, use(record, on) adds it.  All n records are requested before the
// first is used; with PART only the first `left` slots are the list's, the
// others load the particle's own record (self) and are used with on = false,
// so a list's last slots cost one round trip together, not one each.  A list
// of 30 neighbours ends in a partial chunk of 8 in most warps; with its slots
// taken one by one (and the whole chunk's loads left to the compiler's order)
// the passes at 256 scenes, 5.95 M particles, u16 lists, were: lambda 3 x 285,
// delta-p 4 x 301, omega 448, and are 3 x 261, 4 x 291, 381 us.
template <int N, bool PART, class IDX, class LD, class USE>
__device__ __forceinline__ void list_group(uint32_t left, uint32_t self, IDX &&idx, LD &&ld, USE &&use)
{
    decltype(ld(0u)) rec[N];
#pragma unroll
    for (int c = 0; c < N; ++c) rec[c] = ld(!PART || (uint32_t)c < left ? idx(c) : self);
#pragma unroll
    for (int c = 0; c < N; ++c) use(rec[c], !PART || (uint32_t)c < left);
}

// Visit list slots [0, nn) of one particle in list order.  Indices are
// requested CH at a time (CH / 4 quads), one chunk ahead of their use; the
// chunk (loads in flight against registers) is each pass's choice.  The
// last, partial chunk is taken in groups of four.
template <int CH, class LD, class USE>
__device__ __forceinline__ void list_walk(const uint32_t *__restrict__ nl, uint64_t stride, uint32_t nn, uint32_t self,
                                          LD &&ld, USE &&use)
{
    constexpr int NQ = (CH + 3) / 4;  // (a u16 list's group of 2 compiles, unused, as one quad)
    const uint4 *p = reinterpret_cast<const uint4 *>(nl);  // quad kq of the particle at p[kq * stride]
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    uint4 qn[NQ];
#pragma unroll
    for (int c = 0; c < NQ; ++c) qn[c] = ((uint32_t)(4 * c) < nn) ? list_ld(p + c * stride) : z;
    uint32_t k0 = 0;
    for (; k0 + CH <= nn; k0 += CH) {
        uint4 q[NQ];
#pragma unroll
        for (int c = 0; c < NQ; ++c) q[c] = qn[c];
        p += NQ * stride;
#pragma unroll
        for (int c = 0; c < NQ; ++c) qn[c] = (k0 + CH + 4 * c < nn) ? list_ld(p + c * stride) : z;
        list_group<CH, false>(CH, self, [&](int c) { return quad_at(q[c >> 2], c & 3); }, ld, use);
    }
#pragma unroll
    for (int c = 0; c < NQ; ++c)
        if (k0 + 4 * c < nn)
            list_group<4, true>(nn - k0 - 4 * c, self, [&](int e) { return quad_at(qn[c], e); }, ld, use);
}

// list_walk over a u16 list: octs requested one chunk (8 slots) ahead, the
// records of G slots at a time; ld gets base + the scene-local index: the
// working slot for base = the scene's first slot, the scene-local index itself
// for base = 0 (for arrays offset by the scene's first slot, which saves the
// add per slot; measured faster in the vorticity-apply pass only).
template <int G, class LD, class USE>
__device__ __forceinline__ void list_walk16(const uint32_t *__restrict__ nl, uint64_t stride, uint32_t nn,
                                            uint32_t base, uint32_t self, LD &&ld, USE &&use)
{
    const uint4 *p = reinterpret_cast<const uint4 *>(nl);  // oct ko of the particle at p[ko * stride]
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    uint4 qn = (0u < nn) ? list_ld(p) : z;
    uint32_t k0 = 0;
    for (; k0 + 8 <= nn; k0 += 8) {
        const uint4 q = qn;
        p += stride;
        qn = (k0 + 8 < nn) ? list_ld(p) : z;
#pragma unroll
        for (int h = 0; h < 8; h += G)
            list_group<G, false>(G, self, [&](int c) { return base + oct_at(q, h + c); }, ld, use);
    }
#pragma unroll
    for (int h = 0; h < 8; h += 4)
        if (k0 + h < nn)
            list_group<4, true>(nn - k0 - h, self, [&](int c) { return base + oct_at(qn, h + c); }, ld, use);
}

// The list of one particle in either form: u32 quads (indices are working
// slots) or u16 octs (scene-local indices, base = the scene's first slot).
template <int CH, class LD, class USE>
__device__ __forceinline__ void list_walk_any(bool l16, const uint32_t *__restrict__ nl, uint64_t stride, uint32_t nn,
                                              uint32_t base, uint32_t self, LD &&ld, USE &&use)
{
    if (l16)
        list_walk16<CH>(nl, stride, nn, base, self, ld, use);
    else
        list_walk<CH>(nl, stride, nn, self, ld, use);
}

// Small, latency-bound steps: a pass's time is one thread's chain of dependent
// loads, so the list is read 32 slots at a time (all their rows at once) and
// the neighbours' records 16 at a time, instead of one row and 8 (and the
// last, partial row's one by one): at 4,096 particles (each kernel alone, cold
// caches) delta-p 10.4 -> 7.8 us, omega 12.0 -> 8.7, its second pass 12.1 ->
// 9.1.  ld(q) loads the record of slot base + q, use(record, on)
// adds it in list order; slots past the count load the particle's own record
// (self, as q) and are used with on = false.  rows: 16-byte rows a list has.
template <class LD, class USE>
__device__ __forceinline__ void list_walk_wide(bool l16, const uint32_t *__restrict__ nl, uint64_t stride, uint32_t rows,
                                               uint32_t nn, uint32_t base, uint32_t self, LD &&ld, USE &&use)
{
    const uint4 *p = reinterpret_cast<const uint4 *>(nl);
    uint32_t k0 = 0;
    do {  // the first rows are requested whatever the count, beside it
        uint32_t q[32];
        if (l16) {
            uint4 r[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) r[j] = k0 / 8 + j < rows ? list_ld(p + (uint64_t)(k0 / 8 + j) * stride) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (uint32_t c = 0; c < 32; ++c) q[c] = base + oct_at(r[c / 8], c % 8);
        } else {
            uint4 r[8];
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) r[j] = k0 / 4 + j < rows ? list_ld(p + (uint64_t)(k0 / 4 + j) * stride) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (uint32_t c = 0; c < 32; ++c) q[c] = quad_at(r[c / 4], c % 4);
        }
#pragma unroll
        for (uint32_t h = 0; h < 32; h += 16) {
            if (k0 + h < nn) {
                decltype(ld(0u)) rec[16];
#pragma unroll
                for (uint32_t c = 0; c < 16; ++c) rec[c] = ld(k0 + h + c < nn ? q[h + c] : self);
#pragma unroll
                for (uint32_t c = 0; c < 16; ++c) use(rec[c], k0 + h + c < nn);
            }
        }
        k0 += 32;
    } while (k0 < nn);
}

// The smallest steps: a particle's list over LANES lanes, 32 / LANES slots of
// every 32 a lane (whole rows).  Every lane loads its records and makes their
// terms; the sums then go from lane to lane, each adding its own terms to what
// the lane before it had, so the additions are the one-lane walk's, in its
// order.  All the lanes end with the whole sums.  Few particles leave a
// scheduler with one warp or none, and a pass's time is that warp's: 32 slots
// in two groups of 16 took 3,700 to 6,200 cycles of its 5,000 to 7,200.
template <uint32_t LANES, class SUM, class IDX, class LD>
__device__ __forceinline__ void lanes_sum(uint32_t k0, uint32_t nn, uint32_t self, SUM &sum, IDX &&idx, LD &&ld)
{
    constexpr uint32_t N = 32 / LANES;  // slots a lane
    const uint32_t sub = threadIdx.x % LANES, gmask = ((1u << LANES) - 1u) << (threadIdx.x & (32u - LANES));
    const uint32_t m = k0 + N * sub;
    decltype(ld(0u)) rec[N];
#pragma unroll
    for (uint32_t c = 0; c < N; ++c) rec[c] = ld(m + c < nn ? idx(c) : self);
    typename SUM::Term t[N];
#pragma unroll
    for (uint32_t c = 0; c < N; ++c) t[c] = sum.term(rec[c], m + c < nn);
#pragma unroll
    for (uint32_t l = 0; l < LANES; ++l) {
        if (k0 + N * l < nn) {
#pragma unroll
            for (uint32_t c = 0; c < N; ++c) sum.add(t[c]);
        }
        sum.template pass<LANES>(gmask, l);
    }
}

template <uint32_t LANES, class SUM, class LD>
__device__ __forceinline__ void list_walk_lanes(bool l16, const uint32_t *__restrict__ nl, uint64_t stride,
                                                uint32_t rows, uint32_t nn, uint32_t base, uint32_t self, SUM &sum,
                                                LD &&ld)
{
    const uint4 *p = reinterpret_cast<const uint4 *>(nl);
    constexpr uint32_t N = 32 / LANES;  // slots a lane
    const uint32_t sub = threadIdx.x % LANES;
    uint32_t k0 = 0;
    do {
        const uint32_t m = k0 + N * sub;
        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
        uint32_t q[N];
        if (l16) {
            uint4 r[N / 8];
#pragma unroll
            for (uint32_t j = 0; j < N / 8; ++j) r[j] = m / 8 + j < rows ? list_ld(p + (uint64_t)(m / 8 + j) * stride) : z;
#pragma unroll
            for (uint32_t c = 0; c < N; ++c) q[c] = base + oct_at(r[c / 8], c % 8);
        } else {
            uint4 r[N / 4];
#pragma unroll
            for (uint32_t j = 0; j < N / 4; ++j) r[j] = m / 4 + j < rows ? list_ld(p + (uint64_t)(m / 4 + j) * stride) : z;
#pragma unroll
            for (uint32_t c = 0; c < N; ++c) q[c] = quad_at(r[c / 4], c % 4);
        }
        lanes_sum<LANES>(k0, nn, self, sum, [&](uint32_t c) { return q[c]; }, ld);
        k0 += 32;
    } while (k0 < nn);
}

// Small steps' blocks: kSmallBlock threads, tile / kSmallBlock of them a tile,
// so that few particles spread over many SMs, one block for every part of
// every tile the launch shape allows for.  A tile's header (scene << 10 |
// live particles, first working slot, scene's first slot, scene's slots minus
// its sorted offsets; written beside the dense sort, 0 particles past the
// last tile) is one load in place of a chain of four: tile count, tile, scene
// record, scene's live count (lambda 7.9 -> 6.1 us, delta-p 7.8 -> 6.3, the
// whole step of 4,096 particles 80 -> 69).
#define SMALL_LOOP_BEGIN                                                      \
    {                                                                         \
        const uint32_t parts_ = tile / kSmallBlock;                           \
        const uint4 hd_ = __ldg(a.tile_hdr + blockIdx.x / parts_);            \
        const uint32_t k_ = (blockIdx.x % parts_) * kSmallBlock + threadIdx.x / LANES; \
        if (k_ >= (hd_.x & 1023u)) return;                                    \
        const uint32_t s = hd_.x >> 10, i = hd_.y + k_, p_off = hd_.z;
#define SMALL_LOOP_END }

// The list passes of small steps: LANES = 1, or kLanes lanes a particle (and
// kLanes times the threads a block), of which the first finishes.
template <uint32_t LANES, class SUM, class LD>
__device__ __forceinline__ bool small_sum(const StepArgs &a, bool l16, uint32_t i, uint32_t p_off, SUM &sum, LD &&ld)
{
    if (LANES == 1) {
        list_walk_wide(l16, list_of(a.nbr, i), a.nbr_stride, a.nbr_rows, a.nnb[i], p_off, i, ld,
                       [&](const decltype(ld(0u)) &r, bool on) { sum.add(sum.term(r, on)); });
        return true;
    }
    list_walk_lanes<LANES>(l16, list_of(a.nbr, i), a.nbr_stride, a.nbr_rows, a.nnb[i], p_off, i, sum, ld);
    return threadIdx.x % LANES == 0;
}

// Per-tile prologue shared by the particle kernels.
#define TILE_LOOP_BEGIN                                                   \
    const uint32_t n_tiles_ = a.ctrl->n_tiles;                            \
    for (uint32_t t_ = blockIdx.x; t_ < n_tiles_; t_ += gridDim.x) {      \
        const uint32_t s = __ldg(a.tile_scene + t_);                      \
        const uint32_t local = __ldg(a.tile_start + t_) + threadIdx.x;
#define TILE_LOOP_END }

// --------------------------------------------------------------- kernels --

// predict (pbf_solve.cpp:16-25 -> multiplyAddCUDA x2, pbf_predict.cu:15-45),
// calcHash (pbf_neighbor_search_util.cu:20-37), checkDeleteParticle
// (pbf_delete.cu:9-28; deleted key = ncell, one past the last cell) and the
// histogram of countingSort (insertAndCountCUDA, pbf_counting_sort.cu:21-32).
// PACKED: the input phase is read from the packed AoS float3 buffers of a
// packed-input step (what k_unpack would have written), and the particles
// are numbered afresh.
struct PhaseIn {
    float4 x, v;
    uint32_t id;
};
template <bool PACKED>
__device__ __forceinline__ PhaseIn load_phase(const StepArgs &a, const SceneDesc &d, uint32_t s, uint32_t local)
{
    if (PACKED) {
        const PackedIn pin = *a.pin;
        const uint64_t q = 3ull * ((uint64_t)a.pack_off[s] + local);
        return PhaseIn{make_float4(pin.x[q], pin.x[q + 1], pin.x[q + 2], 0.f),
                       pin.v ? make_float4(pin.v[q], pin.v[q + 1], pin.v[q + 2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f),
                       local};
    }
    const uint32_t i = d.p_off + local;
    return PhaseIn{a.x[i], a.v[i], a.id[i]};
}

struct Predicted {
    float4 ps;  // .w: the id
    uint32_t key, cls;
};
template <bool PACKED>
__device__ __forceinline__ Predicted predict_particle(const StepArgs &a, const SceneDesc &d, uint32_t s,
                                                      uint32_t local, uint32_t n, const PhaseIn &in)
{
    if (PACKED && local == 0) a.next_id[s] = n;
    const float4 xv = in.x, vv = in.v;
    const uint32_t id = in.id;
    const float dt = d.dt;
    float4 ps;
    ps.x = __fmaf_rn(__fmaf_rn(d.g[0], dt, vv.x), dt, xv.x);
    ps.y = __fmaf_rn(__fmaf_rn(d.g[1], dt, vv.y), dt, xv.y);
    ps.z = __fmaf_rn(__fmaf_rn(d.g[2], dt, vv.z), dt, xv.z);
    ps.w = __uint_as_float(id);  // the id travels with the prediction to the gather
    const int32_t cx = cell_coord(ps.x, d.cw), cy = cell_coord(ps.y, d.cw), cz = cell_coord(ps.z, d.cw);
    uint32_t key = hash3((uint32_t)cx, (uint32_t)cy, (uint32_t)cz, d);
    uint32_t cls = alias_class(cx, cy, cz, d);
    if (ps.x < d.amin[0] || d.amax[0] < ps.x || ps.y < d.amin[1] || d.amax[1] < ps.y || ps.z < d.amin[2] ||
        d.amax[2] < ps.z) {
        key = d.ncell;
        cls = 0;
    }
    if (!(isfinite(ps.x) && isfinite(ps.y) && isfinite(ps.z))) atomicOr(a.flags + s, PBF_FLAG_NONFINITE);
    return Predicted{ps, key, cls};
}

template <bool PACKED>
__global__ void __launch_bounds__(512) k_predict_hash(StepArgs a)
{
    TILE_LOOP_BEGIN
    const uint32_t n = a.scene_num[s];
    if (local >= n) continue;
    const SceneDesc d = a.scenes[s];
    const Predicted p = predict_particle<PACKED>(a, d, s, local, n, load_phase<PACKED>(a, d, s, local));
    const uint32_t i = d.p_off + local;
    a.cls[i] = (uint8_t)p.cls;
    a.xs[i] = p.ps;
    a.key[i] = p.key;
    a.slot[i] = atomicAdd(a.count + d.c_off + p.key, 1u);
    TILE_LOOP_END
}

// ---- exclusive scan of the cell counts (reduce, spine, down-sweep) ----
__global__ void __launch_bounds__(256) k_scan_reduce(StepArgs a)
{
    __shared__ uint32_t ws[kScanWarps];
    const uint32_t n = a.ctrl->n_cells;
    const uint32_t ntile = (n + kScanTile - 1) / kScanTile;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t t = blockIdx.x; t < ntile; t += gridDim.x) {
        const uint32_t base = t * kScanTile + warp * kScanItemsPerWarp;
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) {
            const uint32_t idx = base + j * 32 + lane;
            if (idx < n) sum += a.count[idx];
        }
#pragma unroll
        for (uint32_t o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) ws[warp] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t tot = 0;
            for (uint32_t k = 0; k < kScanWarps; ++k) tot += ws[k];
            a.bsum[t] = tot;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(1024) k_scan_spine(StepArgs a)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    const uint32_t n = a.ctrl->n_cells;
    const uint32_t ntile = (n + kScanTile - 1) / kScanTile;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        carry = 0;
        *a.dense = 0;  // the bucket queues of this step's rank kernel
        *a.mid = 0;
    }
    __syncthreads();
    for (uint32_t base = 0; base < ntile; base += 1024) {
        const uint32_t idx = base + threadIdx.x;
        const uint32_t v = idx < ntile ? a.bsum[idx] : 0u;
        const uint32_t inc = warp_incl_scan(v);
        if (lane == 31) ws[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const uint32_t wv = ws[lane];
            ws[lane] = warp_incl_scan(wv) - wv;
        }
        __syncthreads();
        const uint32_t c = carry;
        if (idx < ntile) a.bsum[idx] = c + ws[warp] + inc - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry = c + ws[warp] + inc;
        __syncthreads();
    }
    if (threadIdx.x == 0) a.offsets[n] = carry;
}

// The whole scan in one block for tables of at most 1024 * R cells, R
// rounds of 1024 held in registers: every round's counts are requested at
// once (coalesced), the rounds' warp scans run side by side, one warp turns
// the rounds' warp totals into offsets (carrying across rounds in order),
// and the offsets are written coalesced.  Two barriers in all.
template <uint32_t R>
__global__ void __launch_bounds__(1024) k_scan_single_reg(StepArgs a)
{
    __shared__ uint32_t ws[R][32];
    const uint32_t n = a.ctrl->n_cells;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    if (t == 0) {
        *a.dense = 0;  // the bucket queues of this step's rank kernel
        *a.mid = 0;
    }
    uint32_t v[R], inc[R];
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) {
        const uint32_t idx = k * 1024u + t;
        v[k] = idx < n ? a.count[idx] : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) {
        inc[k] = warp_incl_scan(v[k]);
        if (lane == 31) ws[k][warp] = inc[k];
    }
    __syncthreads();
    if (warp == 0) {  // exclusive prefix of every (round, warp) total, rounds in order
        uint32_t carry = 0;
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            const uint32_t wv = ws[k][lane];
            const uint32_t wi = warp_incl_scan(wv);
            ws[k][lane] = carry + wi - wv;
            carry += __shfl_sync(0xffffffffu, wi, 31);
        }
        if (lane == 0) a.offsets[n] = carry;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) {
        const uint32_t idx = k * 1024u + t;
        if (idx < n) {
            a.offsets[idx] = ws[k][warp] + inc[k] - v[k];
            a.count[idx] = 0u;  // ready for the next step's histogram
        }
    }
}

// The whole scan in one thread-block cluster (cluster_scan), for the tables
// between the one-block scan and the three-kernel one.  Bound by the latency
// of the one launch: 32,769 cells (event-timed, launch included) took 27.7 us
// in one block looping over rounds of 1024 cells and take 8.4 here (9.3 in a
// cluster of 8), 65,537 cells 20.2 us in three kernels and 9.3 here.
template <uint32_t R>
__global__ void __launch_bounds__(1024) k_scan_cluster(StepArgs a)
{
    const uint32_t n = a.ctrl->n_cells;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.dense = 0;  // the bucket queues of this step's rank kernel
        *a.mid = 0;
    }
    const uint32_t all = cluster_scan<R>([&](uint32_t c) { return a.count[c]; }, n, [&](uint32_t c, uint32_t offset, uint32_t) {
        a.offsets[c] = offset;
        a.count[c] = 0u;  // ready for the next step's histogram
    });
    if (blockIdx.x == 0 && threadIdx.x == 0) a.offsets[n] = all;
}

__global__ void __launch_bounds__(256) k_scan_down(StepArgs a)
{
    __shared__ uint32_t ws[kScanWarps];
    const uint32_t n = a.ctrl->n_cells;
    const uint32_t ntile = (n + kScanTile - 1) / kScanTile;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t t = blockIdx.x; t < ntile; t += gridDim.x) {
        const uint32_t base = t * kScanTile + warp * kScanItemsPerWarp;
        uint32_t vals[16];
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) {
            const uint32_t idx = base + j * 32 + lane;
            vals[j] = idx < n ? a.count[idx] : 0u;
            sum += vals[j];
        }
        uint32_t wsum = sum;
#pragma unroll
        for (uint32_t o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
        if (lane == 0) ws[warp] = wsum;
        __syncthreads();
        uint32_t run = a.bsum[t];
        for (uint32_t k = 0; k < warp; ++k) run += ws[k];
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) {
            const uint32_t idx = base + j * 32 + lane;
            const uint32_t inc = warp_incl_scan(vals[j]);
            if (idx < n) {
                a.offsets[idx] = run + inc - vals[j];
                a.count[idx] = 0u;  // ready for the next step's histogram
            }
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        __syncthreads();
    }
}

// tmp entries of scenes up to kClsLimit particles carry the member's alias
// class above its input index.
constexpr uint32_t kClsShift = 29;
constexpr uint32_t kClsLimit = 1u << kClsShift;

// Scatter into the cell buckets in atomic-slot order (sortByCountingCUDA,
// pbf_counting_sort.cu:120-134).
__global__ void __launch_bounds__(512) k_scatter(StepArgs a)
{
    TILE_LOOP_BEGIN
    const uint32_t n = a.scene_num[s];
    if (local >= n) continue;
    const SceneDesc d = a.scenes[s];
    const uint32_t i = d.p_off + local;
    const uint32_t pos = a.offsets[d.c_off + a.key[i]] + a.slot[i];
    // the alias class rides in the top bits (scenes below 2^29 particles)
    a.tmp[pos] = d.capacity <= kClsLimit ? local | ((uint32_t)a.cls[i] << kClsShift) : local;
    TILE_LOOP_END
}

// A bucket's class ends from its class counts (8 bytes, byte c of class c):
// byte c = members of classes 0..c, so class c is [byte c - 1, byte c) of the
// bucket.  Buckets of up to kClassMax members (their bytes never are
// kClassWhole).
__device__ __forceinline__ uint64_t class_ends(uint64_t counts) { return counts * 0x0101010101010101ull; }
constexpr uint32_t kClassMax = 254;

// Stable rank inside each bucket (count of smaller input indices): the
// permutation of a stable sort by cell (cub::DeviceRadixSort::SortPairs
// order), which reorderDataCUDA (pbf_neighbor_search_util.cu:143-154) then
// applies.  One thread per cell, cells in order, so the cell ranges, the
// bucket entries and the bucket's part of the permutation are read and
// written contiguously whatever the particles' input order.  Buckets of up
// to kMidMin members are ranked here; larger ones are queued for
// k_dense_sort (a warp per bucket up to kDenseMin members, a block beyond:
// a shared-memory sort up to kStableLimit members, a radix sort in global
// memory above, which degenerate inputs and mass deletion can reach).
constexpr uint32_t kStableLimit = 4096;
constexpr uint32_t kDenseMin = 64;
static_assert(kStableLimit * sizeof(uint32_t) == sizeof(RadixSmem), "the radix sort reuses the bitonic buffer");
__global__ void __launch_bounds__(kCellTileMax) k_rank_cells(StepArgs a)
{
    const uint32_t n0 = a.ctrl->n_tiles, nct = a.ctrl->n_cell_tiles;
    for (uint32_t t_ = blockIdx.x; t_ < nct; t_ += gridDim.x) {
        // the tile's scene: its fields once per tile, in registers
        const uint32_t s = __ldg(a.tile_scene + n0 + t_);
        const SceneDesc *sd = a.scenes + s;
        const uint32_t ncell = __ldg(&sd->ncell), c_off = __ldg(&sd->c_off), p_off = __ldg(&sd->p_off);
        const bool packed = __ldg(&sd->capacity) <= kClsLimit;
        const bool grouped = packed && __ldg(&sd->gx) >= 4 && __ldg(&sd->gy) >= 4 && __ldg(&sd->gz) >= 4;
        const uint32_t lc = __ldg(a.tile_start + n0 + t_) + threadIdx.x;
        if (lc > ncell) continue;  // local cells 0..ncell (ncell: the deleted bucket)
        const uint32_t gk = c_off + lc;
        const uint32_t st = __ldg(a.offsets + gk), en = __ldg(a.offsets + gk + 1);
        if (st == en) continue;
        const uint32_t b = en - st;
        if (b > kMidMin) {
            uint32_t *q = b > kDenseMin ? a.dense : a.mid;
            const uint32_t k = atomicAdd(q, 1u);
            q[1 + 2 * k] = gk;
            q[2 + 2 * k] = s;
            continue;
        }
        const uint32_t g0 = p_off + (st - __ldg(a.offsets + c_off));
        const uint32_t imask = packed ? kClsLimit - 1u : 0xFFFFFFFFu;
        // the alias class rides in the entries' top bits (scenes below 2^29
        // particles); the walk copy groups a bucket by class when the grid
        // is at least 4 cells on every axis
        uint32_t e[kMidMin];
        uint64_t hist = 0;
        for (uint32_t t = 0; t < b; ++t) {
            e[t] = __ldg(a.tmp + st + t);
            hist += 1ull << (8u * (packed ? e[t] >> kClsShift : 0u));
        }
        const uint32_t c0 = packed ? e[0] >> kClsShift : 0u;
        const bool mixed = grouped && hist != ((uint64_t)b << (8u * c0));
        for (uint32_t t = 0; t < b; ++t) {
            const uint32_t it = e[t] & imask, ct = packed ? e[t] >> kClsShift : 0u;
            uint32_t rank = 0, below = 0, frank = 0;
            for (uint32_t u = 0; u < b; ++u) {
                const uint32_t iu = e[u] & imask, cu = packed ? e[u] >> kClsShift : 0u;
                rank += iu < it ? 1u : 0u;
                below += cu < ct ? 1u : 0u;
                frank += (cu == ct && iu < it) ? 1u : 0u;
            }
            a.perm[g0 + rank] = it;
            a.wpos[g0 + rank] = g0 + (mixed ? below + frank : rank);
        }
        a.chist[gk] = grouped ? class_ends(hist) : kClassWhole;
    }
}

// A particle's place in its bucket of at most kDenseMin members [st, en), by
// counting: the members with a smaller input index (stable sorted order), and
// for a bucket of several alias classes (grouped) also the members of a
// smaller class and those of its class with a smaller input index (its place
// in working order), and the bucket's class histogram.
struct Place {
    uint32_t rank, work;
    uint64_t hist;
};
template <class LD>
__device__ __forceinline__ Place bucket_place(LD &&ld, uint32_t st, uint32_t en, uint32_t local, uint32_t my_cls,
                                              uint32_t imask, bool grouped)
{
    Place p;
    p.rank = 0;
    p.hist = (uint64_t)(en - st) << (8u * my_cls);  // every member of my class
    uint32_t diff = 0;
    for (uint32_t t = st; t < en; t += 8) {  // 8 members requested together
        uint32_t e[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) e[k] = t + k < en ? ld(t + k) : 0u;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (t + k < en) {
                p.rank += ((e[k] & imask) < local) ? 1u : 0u;
                diff |= (e[k] >> kClsShift) ^ my_cls;
            }
        }
    }
    p.work = p.rank;
    if (grouped && diff) {
        uint32_t below = 0, frank = 0;
        p.hist = 0;
        for (uint32_t t = st; t < en; ++t) {
            const uint32_t e = ld(t);
            const uint32_t mc = e >> kClsShift;
            below += (mc < my_cls) ? 1u : 0u;
            frank += (mc == my_cls && (e & imask) < local) ? 1u : 0u;
            p.hist += 1ull << (8u * mc);
        }
        p.work = below + frank;
    }
    return p;
}

// A dense bucket: queued by its first member by atomic slot.
__device__ __forceinline__ void queue_dense(const StepArgs &a, uint32_t slot, uint32_t gk, uint32_t s)
{
    if (slot != 0) return;
    const uint32_t k = atomicAdd(a.dense, 1u);
    a.dense[1 + 2 * k] = gk;
    a.dense[2 + 2 * k] = s;
}

// The same ranks from the particle side, for small steps (latency bound:
// the per-cell kernel's b^2 loop in one thread lengthens the critical
// path): each particle counts the smaller input indices of its bucket.
// Buckets above kDenseMin members (of any size) are queued for
// k_dense_sort; nothing is queued for the warp tier.
__global__ void __launch_bounds__(512) k_rank_reorder(StepArgs a)
{
    TILE_LOOP_BEGIN
    const uint32_t n = a.scene_num[s];
    if (local >= n) continue;
    const SceneDesc d = a.scenes[s];
    const uint32_t i = d.p_off + local;
    const uint32_t gk = d.c_off + a.key[i];
    const uint32_t st = a.offsets[gk], en = a.offsets[gk + 1];
    const bool packed = d.capacity <= kClsLimit;
    const bool grouped = packed && d.gx >= 4 && d.gy >= 4 && d.gz >= 4;
    if (en - st > kDenseMin) {
        queue_dense(a, a.slot[i], gk, s);
        continue;
    }
    const Place p = bucket_place([&](uint32_t t) { return __ldg(a.tmp + t); }, st, en, local, a.cls[i],
                                 packed ? kClsLimit - 1u : 0xFFFFFFFFu, grouped);
    const uint32_t g0 = d.p_off + (st - a.offsets[d.c_off]);
    // only 4-byte entries are scattered here; k_gather moves the 16-byte
    // particle data in sorted order (coalesced writes, as the reference's
    // reorderDataCUDA gathers).  Buckets holding more than one alias class
    // also place the particle in working order.
    a.wpos[g0 + p.rank] = g0 + p.work;
    if (p.rank == 0) a.chist[gk] = grouped ? class_ends(p.hist) : kClassWhole;
    a.perm[g0 + p.rank] = local;
    TILE_LOOP_END
}

// Buckets queued by the rank kernels (k_rank_cells queues medium and dense
// ones, k_rank_reorder dense ones).  Medium ones (kMidMin+1 .. kDenseMin
// members) first, a warp each: members in lanes, each ranked by counting
// over the others (broadcast by shuffle).  Dense ones (kDenseMin+1 ..
// kStableLimit) then, a block each: the bucket entries (input index, alias
// class in the top bits) are sorted in shared memory by input index (the
// stable sorted order) and, when the bucket mixes classes, by (class, index)
// (the walk copy's order).  Both give the permutation, class counts and
// walk-copy places of k_rank_cells' per-bucket count.  Buckets above
// kStableLimit get a block each too: a radix sort by input index in global
// memory (block_radix_stable), walked whole.
__device__ __forceinline__ uint32_t dense_key(uint32_t e, uint32_t imask)
{
    return e == 0xFFFFFFFFu ? 0xFFFFFFFFu : (e & imask);  // padding sorts last
}

template <bool FULL, class SYNC>
__device__ void bitonic_sort(uint32_t *v, uint32_t n, uint32_t imask, SYNC &&sync)
{
    for (uint32_t size = 2; size <= n; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t t = threadIdx.x; t < (n >> 1); t += kRadixThreads) {
                const uint32_t i = 2 * stride * (t / stride) + (t % stride), j = i + stride;
                const uint32_t vi = v[i], vj = v[j];
                const uint32_t ki = FULL ? vi : dense_key(vi, imask), kj = FULL ? vj : dense_key(vj, imask);
                const bool asc = (i & size) == 0;
                if ((ki > kj) == asc) {
                    v[i] = vj;
                    v[j] = vi;
                }
            }
            sync();
        }
    }
}

// Small steps: the header of tile t (SMALL_LOOP_BEGIN), and the scene's live
// count with its first tile's.
__device__ __forceinline__ void put_tile_header(const StepArgs &a, uint32_t t, uint32_t tile)
{
    uint4 h = make_uint4(0u, 0u, 0u, 0u);
    if (t < a.ctrl->n_tiles) {
        const uint32_t s = __ldg(a.tile_scene + t), start = __ldg(a.tile_start + t);
        const SceneDesc &d = a.scenes[s];
        const uint32_t live = a.offsets[d.c_off + d.ncell] - a.offsets[d.c_off];
        if (start == 0) a.scene_num[s] = live;  // deleted particles leave the scene
        const uint32_t n = start < live ? min(tile, live - start) : 0u;
        h = make_uint4(s << 10 | n, d.p_off + start, d.p_off, d.p_off - a.offsets[d.c_off]);
    }
    a.tile_hdr[t] = h;
}

// The queued dense buckets, a block each (by its first kRadixThreads threads).
template <class SYNC>
__device__ __forceinline__ void sort_dense_buckets(const StepArgs &a, uint32_t nd, uint32_t (&S)[kStableLimit],
                                                   uint32_t (&W)[kStableLimit], SYNC &&sync)
{
    __shared__ uint32_t chist_cnt[8], rbase[16], rtot[16];
    for (uint32_t k = blockIdx.x; k < nd; k += gridDim.x) {
        const uint32_t gk = a.dense[1 + 2 * k], s = a.dense[2 + 2 * k];
        const SceneDesc &d = a.scenes[s];
        const uint32_t st = a.offsets[gk], en = a.offsets[gk + 1], b = en - st;
        const uint32_t base = a.offsets[d.c_off];
        const uint32_t g0 = d.p_off + (st - base);
        const bool packed = d.capacity <= kClsLimit;
        const uint32_t imask = packed ? kClsLimit - 1u : 0xFFFFFFFFu;
        if (b > kStableLimit) {  // the bucket's scatter entries are scratch once sorted into perm
            block_radix_stable(a.tmp + st, a.perm + g0, b, imask, radix_bits(d.capacity),
                               *reinterpret_cast<RadixSmem *>(S), rbase, rtot, sync);
            for (uint32_t t = threadIdx.x; t < b; t += kRadixThreads) a.wpos[g0 + t] = g0 + t;
            if (threadIdx.x == 0) a.chist[gk] = kClassWhole;
            sync();
            continue;
        }
        const bool grouped = packed && b <= kClassMax && d.gx >= 4 && d.gy >= 4 && d.gz >= 4;
        uint32_t P = 1;
        while (P < b) P <<= 1;
        if (threadIdx.x < 8) chist_cnt[threadIdx.x] = 0;
        sync();
        for (uint32_t t = threadIdx.x; t < P; t += kRadixThreads) {
            const uint32_t e = t < b ? a.tmp[st + t] : 0xFFFFFFFFu;
            S[t] = e;
            W[t] = e;
            if (t < b && grouped) atomicAdd(&chist_cnt[e >> kClsShift], 1u);
        }
        sync();
        bitonic_sort<false>(S, P, imask, sync);
        uint64_t hist = 0;
        uint32_t classes = 0;
        for (uint32_t c = 0; c < 8; ++c) {
            hist |= (uint64_t)chist_cnt[c] << (8u * c);
            classes += chist_cnt[c] ? 1u : 0u;
        }
        const bool mixed = grouped && classes > 1;
        if (mixed) bitonic_sort<true>(W, P, imask, sync);  // (class, index) order
        for (uint32_t t = threadIdx.x; t < b; t += kRadixThreads) {
            a.perm[g0 + t] = S[t] & imask;
            if (!mixed) a.wpos[g0 + t] = g0 + t;
        }
        if (mixed) {
            for (uint32_t w = threadIdx.x; w < b; w += kRadixThreads) {
                const uint32_t key = W[w] & imask;  // its place in S (sorted by index)
                uint32_t lo = 0, hi = b;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if ((S[mid] & imask) < key) lo = mid + 1;
                    else hi = mid;
                }
                a.wpos[g0 + lo] = g0 + w;
            }
        }
        if (threadIdx.x == 0) a.chist[gk] = grouped ? class_ends(hist) : kClassWhole;
        sync();
    }
}

// small_tiles: small steps, the tile headers of their list passes too (a
// thread a tile, while the queues are read).
__global__ void __launch_bounds__(kRadixThreads) k_dense_sort(StepArgs a, uint32_t tile, uint32_t small_tiles)
{
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < small_tiles; t += gridDim.x * blockDim.x)
        put_tile_header(a, t, tile);
    {
        const uint32_t nm = *(volatile const uint32_t *)a.mid;
        const uint32_t lane = threadIdx.x & 31u, wpb = blockDim.x >> 5;
        for (uint32_t k = blockIdx.x * wpb + (threadIdx.x >> 5); k < nm; k += gridDim.x * wpb) {
            const uint32_t gk = a.mid[1 + 2 * k], s = a.mid[2 + 2 * k];
            const SceneDesc &d = a.scenes[s];
            const uint32_t st = a.offsets[gk], b = a.offsets[gk + 1] - st;
            const uint32_t g0 = d.p_off + (st - a.offsets[d.c_off]);
            const bool packed = d.capacity <= kClsLimit;
            const uint32_t imask = packed ? kClsLimit - 1u : 0xFFFFFFFFu;
            const bool grouped = packed && d.gx >= 4 && d.gy >= 4 && d.gz >= 4;
            const bool h0 = lane < b, h1 = 32u + lane < b;
            const uint32_t e0 = h0 ? a.tmp[st + lane] : 0u, e1 = h1 ? a.tmp[st + 32u + lane] : 0u;
            const uint32_t i0 = e0 & imask, i1 = e1 & imask;
            const uint32_t c0 = packed ? e0 >> kClsShift : 0u, c1 = packed ? e1 >> kClsShift : 0u;
            uint64_t hist = (h0 ? 1ull << (8u * c0) : 0ull) + (h1 ? 1ull << (8u * c1) : 0ull);
#pragma unroll
            for (uint32_t o = 16; o > 0; o >>= 1) hist += __shfl_xor_sync(0xffffffffu, hist, o);
            const uint32_t cf = __shfl_sync(0xffffffffu, c0, 0);
            const bool mixed = grouped && hist != ((uint64_t)b << (8u * cf));
            uint32_t r0 = 0, b0 = 0, f0 = 0, r1 = 0, b1 = 0, f1 = 0;
            for (uint32_t u = 0; u < b; ++u) {
                const uint32_t eu = __shfl_sync(0xffffffffu, u < 32u ? e0 : e1, u & 31u);
                const uint32_t iu = eu & imask, cu = packed ? eu >> kClsShift : 0u;
                r0 += iu < i0 ? 1u : 0u;
                b0 += cu < c0 ? 1u : 0u;
                f0 += (cu == c0 && iu < i0) ? 1u : 0u;
                r1 += iu < i1 ? 1u : 0u;
                b1 += cu < c1 ? 1u : 0u;
                f1 += (cu == c1 && iu < i1) ? 1u : 0u;
            }
            if (h0) {
                a.perm[g0 + r0] = i0;
                a.wpos[g0 + r0] = g0 + (mixed ? b0 + f0 : r0);
            }
            if (h1) {
                a.perm[g0 + r1] = i1;
                a.wpos[g0 + r1] = g0 + (mixed ? b1 + f1 : r1);
            }
            if (lane == 0) a.chist[gk] = grouped ? class_ends(hist) : kClassWhole;
        }
    }
    __shared__ __align__(16) uint32_t S[kStableLimit];
    __shared__ uint32_t W[kStableLimit];
    sort_dense_buckets(a, *(volatile const uint32_t *)a.dense, S, W, BlockSync());
}

// Reorder (reorderDataCUDA x2, pbf_neighbor_search_util.cu:143-154): predicted
// and old positions and ids of the sorted slots, each into its working slot.
// Working slots are the sorted slots, except that a bucket of several alias
// classes is grouped by class, so the neighbour walk reads one range per
// cell.  The solver works in working slots throughout; the old position's .w
// holds the sorted slot, where the step's results go.  PACKED: old positions
// from the packed input.
//
// Bound by the random 16-byte reads in input order.  One working array, not
// the sorted positions and a grouped copy of the mixed buckets beside them:
// 98 -> 86 us at 5.95 M particles in 256 scenes, and the neighbour walk, whose
// candidates' slots are then their indices, 1,428 -> 1,405 us.
template <bool PACKED>
__device__ __forceinline__ void gather_slot(const StepArgs &a, uint32_t s, uint32_t p_off, uint32_t g)
{
    const uint32_t li = a.perm[g];
    const uint32_t w = a.wpos[g];
    const uint32_t i = p_off + li;
    const float4 ps = a.xs[i];
    a.xa[w] = make_float4(ps.x, ps.y, ps.z, 0.f);
    const float gs = __uint_as_float(g);
    if (PACKED) {
        const float *px = a.pin->x + 3ull * ((uint64_t)a.pack_off[s] + li);
        a.xold[w] = make_float4(px[0], px[1], px[2], gs);
    } else {
        const float4 xo = a.x[i];
        a.xold[w] = make_float4(xo.x, xo.y, xo.z, gs);
    }
    a.id_tmp[w] = __float_as_uint(ps.w);  // the id, stored beside the prediction
}

template <bool PACKED>
__global__ void __launch_bounds__(512) k_gather(StepArgs a)
{
    TILE_LOOP_BEGIN
    const uint32_t n = a.scene_num[s];
    if (local >= n) continue;
    const uint32_t p_off = a.scenes[s].p_off;
    gather_slot<PACKED>(a, s, p_off, p_off + local);
    TILE_LOOP_END
}

// Small steps: the live slots, by tile headers.
template <bool PACKED>
__global__ void __launch_bounds__(kSmallBlock) k_gather_small(StepArgs a, uint32_t tile)
{
    constexpr uint32_t LANES = 1;
    SMALL_LOOP_BEGIN
    gather_slot<PACKED>(a, s, p_off, i);
    SMALL_LOOP_END
}

// The smallest steps: everything before the neighbour walk (prediction, cell
// hash and counts; scan; scatter; ranks and tile headers; reorder) in one
// cluster of 1024-thread blocks, a particle a thread, R rounds of 1024 cells a
// block.  Sorted and working orders are the separate kernels'.
//
// Bound by latency: five cluster barriers (counts cleared, counted, block
// totals, offsets, scattered; 850 cycles each with nothing to drain, 1,500 with
// stores; a sixth where buckets are dense) and the loads between them, 12,000
// cycles in all, against six launches and the reload in each of what the phase
// before knew: set, step and get of 4,096 particles 79 -> 74 us, of 10,000 at
// h = 1.4 spacings 68 -> 63.  A particle keeps its prediction, bucket and slot in
// registers through the phases and writes its records into its working slot
// itself; counts and offsets are the blocks' shared memory.  Two particles a
// thread took 32,768 particles' step from 88.2 to 90.1 us, so such steps keep
// a kernel per phase.
template <uint32_t R, bool PACKED>
__global__ void __launch_bounds__(1024) k_front(StepArgs a, uint32_t tile_shift, uint32_t small_tiles)
{
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), blocks = cluster.num_blocks(), threads = blocks * 1024u;
    // a cluster's warps take the particles in turn, block after block, so few
    // particles spread over all its SMs
    const uint32_t gid = ((threadIdx.x >> 5) * blocks + rank) * 32u + (threadIdx.x & 31u);
    const uint32_t t = gid >> tile_shift;
    // the tile is requested beside the count of tiles (the lists have room)
    const uint32_t n_tiles = a.ctrl->n_tiles, n_cells = a.ctrl->n_cells;
    const uint32_t s = t < small_tiles ? __ldg(a.tile_scene + t) : 0u;
    const uint32_t local = (t < small_tiles ? __ldg(a.tile_start + t) : 0u) + (gid & ((1u << tile_shift) - 1u));
    // the cells' counts, then offsets, block after block in shared memory
    static_assert(kFrontRounds * 1024u <= kStableLimit, "the dense buckets' sort reuses them");
    __shared__ __align__(16) uint32_t cells[kStableLimit], counts[kStableLimit];
    constexpr uint32_t kShift = R == 1 ? 10 : (R == 2 ? 11 : 12), kMask = (1u << kShift) - 1u;
    static_assert(R * 1024u == 1u << kShift, "a power of two of cells a block");
    for (uint32_t k = 0; k < R; ++k) counts[k * 1024u + threadIdx.x] = 0u;
    auto zeroed = cluster.barrier_arrive();
    if (gid == 0) *a.dense = 0;
    const SceneDesc *sd = a.scenes + s;
    bool live = false;  // (with a particle)
    uint32_t gk = 0, slot = 0, cls = 0;
    PhaseIn in;
    float4 ps;
    if (t < n_tiles) {
        const uint32_t n = a.scene_num[s];
        // (its particle is requested beside the scene's count: slots up to the capacity exist)
        if (!PACKED) in = load_phase<PACKED>(a, *sd, s, min(local, sd->capacity - 1u));
        live = local < n;
        if (live) {
            if (PACKED) in = load_phase<PACKED>(a, *sd, s, local);
            const Predicted p = predict_particle<PACKED>(a, *sd, s, local, n, in);
            ps = p.ps;
            gk = sd->c_off + p.key;
            cls = p.cls;
        }
    }
    cluster.barrier_wait(std::move(zeroed));
    if (live) slot = atomicAdd(cluster.map_shared_rank(counts + (gk & kMask), gk >> kShift), 1u);
    cluster.sync();
    const uint32_t all = cluster_scan<R, true>([&](uint32_t c) { return counts[c & kMask]; }, n_cells,
                                         [&](uint32_t c, uint32_t offset, uint32_t) {
                                             cells[c & kMask] = offset;
                                             a.offsets[c] = offset;
                                         });
    if (gid == 0) a.offsets[n_cells] = all;
    cluster.sync();
    uint32_t st = 0, en = 0, base = 0;
    if (live) {
        st = *cluster.map_shared_rank(cells + (gk & kMask), gk >> kShift);
        en = st + *cluster.map_shared_rank(counts + (gk & kMask), gk >> kShift);
        base = *cluster.map_shared_rank(cells + (sd->c_off & kMask), sd->c_off >> kShift);
        a.tmp[st + slot] = local | cls << kClsShift;
        if (en - st > kDenseMin) queue_dense(a, slot, gk, s);
    }
    cluster.sync();
    if (live) {
        a.xs[sd->p_off + local] = ps;
        a.key[sd->p_off + local] = gk - sd->c_off;
    }
    if (live && en - st <= kDenseMin) {
        const bool grouped = sd->gx >= 4 && sd->gy >= 4 && sd->gz >= 4;
        const Place p = bucket_place([&](uint32_t u) { return a.tmp[u]; }, st, en, local, cls, kClsLimit - 1u, grouped);
        const uint32_t g0 = sd->p_off + (st - base), g = g0 + p.rank, w = g0 + p.work;
        a.wpos[g] = w;
        a.perm[g] = local;
        if (p.rank == 0) a.chist[gk] = grouped ? class_ends(p.hist) : kClassWhole;
        if (gk != sd->c_off + sd->ncell) {  // not deleted
            a.xa[w] = make_float4(ps.x, ps.y, ps.z, 0.f);
            a.xold[w] = make_float4(in.x.x, in.x.y, in.x.z, __uint_as_float(g));
            a.id_tmp[w] = __float_as_uint(ps.w);
        }
    }
    // (from the last thread down: the first ones hold the particles of a step with few)
    for (uint32_t h = threads - 1u - gid; h < small_tiles; h += threads) put_tile_header(a, h, 1u << tile_shift);
    const uint32_t nd = *(volatile const uint32_t *)a.dense;  // (complete since the last barrier)
    if (nd == 0) return;
    if (threadIdx.x < kRadixThreads) sort_dense_buckets(a, nd, cells, counts, RadixSync());
    cluster.sync();
    // the dense buckets' particles, through the permutation
    if (t < n_tiles && local < a.offsets[sd->c_off + sd->ncell] - a.offsets[sd->c_off])
        gather_slot<PACKED>(a, s, sd->p_off, sd->p_off + local);
}

// Neighbour list (detectNeighborsCUDA<uint32_t>, pbf_neighbor_search_util.cu:454-482,
// cap max_pair-1, self included) fused with the iteration-0 lambda
// (calcScalingFactorCUDA cached, pbf_constraint.cu:168-209): at iteration 0
// the working positions are the sorted predicted positions, so the pair
// terms can be summed while the list is built.
// SMEM: the accepted indices are collected in shared memory ([slot][thread]
// per block, conflict-free), then written to the list in whole rows (a
// warp's 16-byte stores contiguous) instead of one scattered store per
// accepted candidate, and summed as they are read.  Otherwise (lists beyond
// kNbSmemMax a block) they are stored directly and read back.
template <bool SMEM>
__global__ void __launch_bounds__(512, 2) k_neighbors_lambda(StepArgs a)
{
    extern __shared__ uint32_t s_list[];  // SMEM: [slot][threadIdx.x]
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const uint32_t shift = d.p_off - base;
    const float4 xp = a.xa[i];
    const float h2 = d.h2;
    const PairConst pc = pair_const(d);
    const uint32_t cap = d.cap;
    const uint64_t stride = a.nbr_stride;
    uint32_t *nl = list_of(a.nbr, i);
    uint16_t *nl16 = reinterpret_cast<uint16_t *>(nl);  // u16 lists: scene-local indices
    const bool l16 = d.list16 != 0;
    const float4 *__restrict__ xa = a.xa;
    // phase 1: the walk only tests and records (lanes of a warp accept
    // different candidates, so pair math inside the walk would run masked
    // for almost every candidate)
    // Candidates are fetched kNbFetch at a time (more loads in flight; a
    // group past the range's end reads up to kNbFetch - 1 records beyond it,
    // never accepted: xa carries that many spare records), all of the
    // group is tested first (independent chains), then the accepted ones are
    // appended in order up to the cap, so the first `cap` accepted ones are
    // the reference's.
    // The particle itself is accepted (r^2 = 0) and counts toward the cap at
    // its walk position, but the list does not store it: its pair terms are
    // w(0) = 1 in the density sum and exactly 0 everywhere else.  selfat
    // records the position (the debug getter's reference-layout list puts it
    // back), and the lambda sums start from 1.  SMEM: the walk collects
    // every accepted candidate, the particle's own slot is found in shared
    // memory afterwards and left out of the write-out, so the candidate loop
    // carries no extra state; otherwise the walk skips it as it stores.
    constexpr uint32_t kNbFetch = 4;
    uint32_t cnt = 0, selfat = kNotListed;
    walk27_cells(d, a.offsets, a.chist, shift, xp, [&](uint32_t st, uint32_t en) -> bool {
        for (uint32_t q0 = st; q0 < en; q0 += kNbFetch) {
            float4 c[kNbFetch];
            const float4 *pq = xa + q0;
#pragma unroll
            for (uint32_t k = 0; k < kNbFetch; ++k) c[k] = __ldg(pq + k);
            bool acc[kNbFetch];
#pragma unroll
            for (uint32_t k = 0; k < kNbFetch; ++k) acc[k] = (q0 + k < en) && dist2_exact(xp, c[k]) < h2;
#pragma unroll
            for (uint32_t k = 0; k < kNbFetch; ++k) {
                if (acc[k] && cnt < cap) {
                    const uint32_t q = q0 + k;
                    if (SMEM) {
                        s_list[cnt * blockDim.x + threadIdx.x] = q;
                    } else {
                        const uint32_t ks = cnt - (selfat < cnt ? 1u : 0u);  // stored entries before this one
                        if (q == i) {
                            // met again (an axis of one cell is visited three times): the last
                            // place is the one left out, so the earlier one is stored after all
                            if (selfat != kNotListed) {
                                for (uint32_t e = ks; e > selfat; --e) {
                                    if (l16)
                                        nl16[list16_slot(e, stride)] = nl16[list16_slot(e - 1u, stride)];
                                    else
                                        nl[list_slot(e, stride)] = nl[list_slot(e - 1u, stride)];
                                }
                                if (l16)
                                    nl16[list16_slot(selfat, stride)] = (uint16_t)(i - d.p_off);
                                else
                                    nl[list_slot(selfat, stride)] = i;
                            }
                            selfat = cnt;
                        } else if (l16)
                            nl16[list16_slot(ks, stride)] = (uint16_t)(q - d.p_off);
                        else
                            nl[list_slot(ks, stride)] = q;
                    }
                    ++cnt;
                }
            }
            if (cnt == cap) return false;
        }
        return true;
    });
    const uint32_t *rd = s_list + threadIdx.x;
    if (SMEM) {
        for (uint32_t k = 0; k < cnt; ++k)
            if (rd[k * blockDim.x] == i) selfat = k;
    }
    cnt -= selfat < cnt ? 1u : 0u;  // entries stored
    a.nnb[i] = (uint8_t)cnt;
    a.selfat[i] = (uint8_t)selfat;
    // phase 2: lambda over the list (direct stores: read back by plain loads,
    // the read-only path may not see this kernel's own stores)
    LamSum ls;
    if (selfat != kNotListed) ls.ks = 1.f;
    if (SMEM) {  // the list from shared memory, written out as it is summed
        // stored entry k is shared-memory entry k, or k + 1 from the
        // particle's own slot on
        auto src = [&](uint32_t k) { return rd[(k + (k >= selfat ? 1u : 0u)) * blockDim.x]; };
        // the list out in whole quads (u32) or octs (u16): one 16-byte store
        // per four or eight slots (slots past the count in the last one are
        // padding, never read), and the same eight slots' pairs, four at a
        // time (past the end: the particle itself, masked).  Written out
        // first and read again for the pairs: 1,335 us at 5.95 M particles in
        // 256 scenes, 1,300 so
        uint4 *wq = reinterpret_cast<uint4 *>(nl);
        for (uint32_t k0 = 0; k0 < cnt; k0 += 8) {
            uint32_t q[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) q[k] = k0 + k < cnt ? src(k0 + k) : i;
            if (l16) {
                uint32_t w[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) w[k] = __byte_perm(q[2 * k] - d.p_off, q[2 * k + 1] - d.p_off, 0x5410);
                list_st(wq + (uint64_t)(k0 >> 3) * stride, make_uint4(w[0], w[1], w[2], w[3]));
            } else {
                list_st(wq + (uint64_t)(k0 >> 2) * stride, make_uint4(q[0], q[1], q[2], q[3]));
                if (k0 + 4 < cnt) list_st(wq + (uint64_t)((k0 >> 2) + 1) * stride, make_uint4(q[4], q[5], q[6], q[7]));
            }
#pragma unroll
            for (uint32_t h = 0; h < 8; h += 4) {
                if (h == 0 || k0 + h < cnt) {
                    float4 x[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) x[k] = __ldg(xa + q[h + k]);
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) {
                        const PairGeo g = pair_geo(xp, x[k]);
                        ls.add(g, masked(pair_ws(g.r2, pc), k0 + h + k < cnt));
                    }
                }
            }
        }
    } else {
#pragma unroll 4
        for (uint32_t k = 0; k < cnt; ++k) {
            const uint32_t q = l16 ? d.p_off + nl16[list16_slot(k, stride)] : nl[list_slot(k, stride)];
            lam_add(ls, xp, __ldg(xa + q), pc);
        }
    }
    a.xb[i] = make_float4(xp.x, xp.y, xp.z, ls.lambda(d));  // the first delta-p pass gathers both
    TILE_LOOP_END
}

// The lambda sums of a particle over records of positions.
struct LamWalk {
    float4 xp;
    PairConst pc;
    LamSum ls;
    struct Term {
        PairGeo g;
        PairWS k;
    };
    __device__ __forceinline__ Term term(const float4 &xj, bool on) const
    {
        const PairGeo g = pair_geo(xp, xj);
        return Term{g, masked(pair_ws(g.r2, pc), on)};
    }
    __device__ __forceinline__ void add(const Term &t) { ls.add(t.g, t.k); }
    template <uint32_t LANES>
    __device__ __forceinline__ void pass(uint32_t gmask, uint32_t lane)
    {
        for (float *f : {&ls.ks, &ls.g0, &ls.g1, &ls.g2, &ls.kg2}) *f = __shfl_sync(gmask, *f, lane, LANES);
    }
};

// Small (latency-bound) steps' walk, one particle a lane.  The one-lane walk of
// large steps is a chain of dependent loads a cell at a time: the cell's
// range, then its candidates four at a time.  Here the 27 ranges of each of
// the warp's distinct cells are looked up first, all at once, by the warp's
// lanes together (lanes hold consecutive working slots, so a cell's particles
// are neighbouring lanes), and each lane then goes through the ranges near
// it with the next 8 candidates requested before it tests the current 8.
// Lists, counts and lambda as k_neighbors_lambda's.  The whole step of 32,768
// particles 95 -> 88 us, of 65,000 132 -> 114 us, against four lanes a
// particle that each looked up and walked a run of the nine rows.
//
// Shared memory: the block's accepted slots [slot][thread], then per warp the
// ranges and the cells' coordinates.
__device__ __forceinline__ uint32_t near_cells(const SceneDesc &d, float4 xp, int32_t icx, int32_t icy, int32_t icz)
{
    // bit 9 (dz + 1) + 3 (dy + 1) + dx + 1: cells that can hold a particle
    // within h of xp (see walk27_cells)
    if (d.gx < 4 || d.gy < 4 || d.gz < 4) return 0x7FFFFFFu;
    const float lx = xp.x - (float)icx * d.cw, ly = xp.y - (float)icy * d.cw, lz = xp.z - (float)icz * d.cw;
    const float rx = d.cw - lx, ry = d.cw - ly, rz = d.cw - lz;
    const float lim = d.h2 * 1.001f;
    uint32_t m = 0;
#pragma unroll
    for (int rr = 0; rr < 9; ++rr) {
        const int dz = rr / 3 - 1, dy = rr % 3 - 1;
        const float ez = dz < 0 ? lz : (dz > 0 ? rz : 0.f);
        const float ey = dy < 0 ? ly : (dy > 0 ? ry : 0.f);
        const float eyz2 = ey * ey + ez * ez;
        if (eyz2 <= lim) m |= 2u << (3 * rr);
        if (eyz2 <= lim && eyz2 + lx * lx <= lim) m |= 1u << (3 * rr);
        if (eyz2 <= lim && eyz2 + rx * rx <= lim) m |= 4u << (3 * rr);
    }
    return m;
}

// The candidate ranges of a warp's distinct cells (n of them, coordinates in
// cells), 27 a cell, by the warp's lanes: lane k takes cell k of the 27 around
// each.  A range is the slots that hold the cell's particles, as walk27_cells
// visits them; none when x >= y.
__device__ __forceinline__ void warp_ranges(const SceneDesc &d, const StepArgs &a, uint32_t shift, uint32_t n,
                                            const int32_t *cells, uint2 *rng)
{
    const uint32_t lane = threadIdx.x & 31u;
    const int32_t dz = (int32_t)(lane / 9u) - 1, dy = (int32_t)(lane / 3u % 3u) - 1, dx = (int32_t)(lane % 3u) - 1;
    const uint32_t *off = a.offsets + d.c_off;
    const uint64_t *ch = a.chist + d.c_off;
    if (lane < 27) {
#pragma unroll 4
        for (uint32_t c = 0; c < n; ++c) {
            const int32_t tx = cells[3 * c] + dx, ty = cells[3 * c + 1] + dy, tz = cells[3 * c + 2] + dz;
            const uint32_t b = hash3((uint32_t)tx, (uint32_t)ty, (uint32_t)tz, d);
            uint32_t st = __ldg(off + b), en = __ldg(off + b + 1);
            const uint64_t h = __ldg(reinterpret_cast<const unsigned long long *>(ch + b));
            if (h != kClassWhole && st != en) {  // an empty bucket's class ends are stale
                const uint32_t k = alias_class(tx, ty, tz, d);
                const uint32_t h0 = (uint32_t)h, h1 = (uint32_t)(h >> 32);
                en = st + (__byte_perm(h0, h1, k) & 0xFFu);
                st += __byte_perm(h0 << 8, __funnelshift_l(h0, h1, 8), k) & 0xFFu;
            }
            rng[27 * c + lane] = make_uint2(st + shift, en + shift);
        }
    }
    __syncwarp();
}

// A lane's walk over the ranges todo of its cell's 27: puts the slots accepted
// in order, at most cap, and returns their number; self: the particle's own
// place among them.
template <class PUT>
__device__ __forceinline__ uint32_t walk_ranges(const uint2 *mine, uint32_t todo, const float4 *__restrict__ xa,
                                                float4 xp, float h2, uint32_t cap, uint32_t i, uint32_t &self, PUT &&put)
{
    // the next 8 candidates: [q, min(q + 8, en)); q == en when none are left
    uint32_t q = 0, en = 0;
    auto next = [&]() {
        q += 8;
        while (q >= en && todo) {
            const uint2 r = mine[__ffs((int)todo) - 1];
            todo &= todo - 1u;
            q = r.x;
            en = r.y;
        }
        if (q >= en) q = en = 0;
    };
    float4 c[8];
    auto load = [&]() {
        if (q < en) {
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) c[k] = __ldg(xa + q + k);  // up to 7 spare records past the range
        }
    };
    next();
    load();
    uint32_t cnt = 0;
    while (q < en && cnt < cap) {
        float4 t[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) t[k] = c[k];
        const uint32_t q0 = q, left = en - q;
        next();
        load();
        bool acc[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) acc[k] = k < left && dist2_exact(xp, t[k]) < h2;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (acc[k] && cnt < cap) {
                if (q0 + k == i) self = cnt;
                put(cnt, q0 + k);
                ++cnt;
            }
        }
    }
    return cnt;
}

__global__ void __launch_bounds__(kSmallBlock, 8) k_neighbors_small(StepArgs a, uint32_t tile)
{
    extern __shared__ __align__(8) uint32_t s_small[];
    const uint32_t parts = tile / kSmallBlock;
    const uint4 hd = __ldg(a.tile_hdr + blockIdx.x / parts);
    const uint32_t kk = (blockIdx.x % parts) * kSmallBlock + threadIdx.x, lane = threadIdx.x & 31u;
    const uint32_t n = hd.x & 1023u;
    if (kk - lane >= n) return;  // whole warps
    const bool on = kk < n;
    const uint32_t i = hd.y + kk, p_off = hd.z, shift = hd.w;
    const float4 xp = on ? a.xa[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const SceneDesc d = a.scenes[hd.x >> 10];
    const uint32_t cap = d.cap;
    uint32_t *list = s_small + threadIdx.x;
    uint32_t *const warps = s_small + cap * kSmallBlock;
    uint2 *rng = reinterpret_cast<uint2 *>(warps) + (threadIdx.x >> 5) * (32u * 27u);
    int32_t *cells = reinterpret_cast<int32_t *>(warps + (kSmallBlock >> 5) * (32u * 27u * 2u)) + (threadIdx.x >> 5) * 96u;
    const int32_t icx = cell_coord(xp.x, d.cw), icy = cell_coord(xp.y, d.cw), icz = cell_coord(xp.z, d.cw);
    const int32_t ux = __shfl_up_sync(0xffffffffu, icx, 1), uy = __shfl_up_sync(0xffffffffu, icy, 1),
                  uz = __shfl_up_sync(0xffffffffu, icz, 1);
    const bool same = ux == icx && uy == icy && uz == icz;
    const uint32_t heads = __ballot_sync(0xffffffffu, on && (lane == 0 || !same));
    const uint32_t seg = __popc(heads & (0xFFFFFFFFu >> (31u - lane))) - 1u;  // the lane's cell of the warp's
    if (heads >> lane & 1u) {
        cells[3 * seg] = icx;
        cells[3 * seg + 1] = icy;
        cells[3 * seg + 2] = icz;
    }
    __syncwarp();
    warp_ranges(d, a, shift, __popc(heads), cells, rng);
    if (!on) return;  // no warp-wide operation follows
    uint32_t todo = near_cells(d, xp, icx, icy, icz);
    const uint2 *mine = rng + 27u * seg;
    const float4 *__restrict__ xa = a.xa;
    // the particle itself is accepted and counts toward the cap, but is not
    // stored (see k_neighbors_lambda)
    uint32_t selfat = kNotListed;
    uint32_t cnt = walk_ranges(mine, todo, xa, xp, d.h2, cap, i, selfat,
                               [&](uint32_t k, uint32_t q) { list[k * kSmallBlock] = q; });
    cnt -= selfat < cnt ? 1u : 0u;
    a.nnb[i] = (uint8_t)cnt;
    a.selfat[i] = (uint8_t)selfat;
    LamSum ls;
    if (selfat != kNotListed) ls.ks = 1.f;
    const PairConst pc = pair_const(d);
    const uint64_t stride = a.nbr_stride;
    uint4 *row = reinterpret_cast<uint4 *>(list_of(a.nbr, i));
    for (uint32_t k0 = 0; k0 < cnt; k0 += 16) {
        uint32_t s[16];  // slots past the count load the particle itself and add nothing
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k)
            s[k] = k0 + k < cnt ? list[(k0 + k + (k0 + k >= selfat ? 1u : 0u)) * kSmallBlock] : i;
        float4 x[16];
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k) x[k] = __ldg(xa + s[k]);
        if (d.list16) {
#pragma unroll
            for (uint32_t j = 0; j < 16; j += 8) {
                uint32_t w[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) w[k] = (s[j + 2 * k] - p_off) | (s[j + 2 * k + 1] - p_off) << 16;
                if (k0 + j < cnt) list_st(row + (uint64_t)((k0 + j) >> 3) * stride, make_uint4(w[0], w[1], w[2], w[3]));
            }
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 16; j += 4)
                if (k0 + j < cnt)
                    list_st(row + (uint64_t)((k0 + j) >> 2) * stride, make_uint4(s[j], s[j + 1], s[j + 2], s[j + 3]));
        }
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k) {
            const PairGeo g = pair_geo(xp, x[k]);
            ls.add(g, masked(pair_ws(g.r2, pc), k0 + k < cnt));
        }
    }
    a.xb[i] = make_float4(xp.x, xp.y, xp.z, ls.lambda(d));  // the first delta-p pass gathers both
}

// The smallest steps: the same walk over kSplit lanes a particle, so that few
// particles still fill the SMs and each lane's chain is a quarter: every lane
// takes a run of the near cells into its own part of shared memory, a prefix
// over the group's counts lays the runs end to end up to the cap (the
// reference's first cap accepted candidates in walk order), lane k writes
// every fourth row of the list, and the lambda sums go from lane to lane over
// 8 slots each (lanes_sum; the one-lane sums, bit for bit).  The step of 4,096 particles 73 -> 68 us
// against the split without shared ranges; a fourth block a SM (64 registers)
// spills and takes 72.
__global__ void __launch_bounds__(kSplitBlock, 3) k_neighbors_split(StepArgs a, uint32_t tile)
{
    extern __shared__ __align__(8) uint32_t s_small[];
    const uint32_t parts = tile / kSmallBlock, p = threadIdx.x / kSplit;
    const uint4 hd = __ldg(a.tile_hdr + blockIdx.x / parts);
    const uint32_t k0 = (blockIdx.x % parts) * kSmallBlock, kk = k0 + p, lane = threadIdx.x & 31u;
    const uint32_t sub = lane % kSplit, gmask = ((1u << kSplit) - 1u) << (lane & ~(kSplit - 1u));
    const uint32_t n = hd.x & 1023u;
    if (k0 + (threadIdx.x & ~31u) / kSplit >= n) return;  // whole warps
    const bool on = kk < n;
    const uint32_t i = hd.y + kk, p_off = hd.z, shift = hd.w;
    const float4 xp = on ? a.xa[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const SceneDesc d = a.scenes[hd.x >> 10];
    const uint32_t cap = d.cap;
    // shared memory: every lane's accepted slots [slot][thread], the merged
    // lists [slot][particle], then per warp the ranges and the cells
    uint32_t *run = s_small + threadIdx.x, *list = s_small + cap * kSplitBlock + p;
    uint32_t *const warps = s_small + cap * (kSplitBlock + kSmallBlock);
    constexpr uint32_t kParts = 32 / kSplit;  // particles, and so cells, of a warp
    uint2 *rng = reinterpret_cast<uint2 *>(warps) + (threadIdx.x >> 5) * (kParts * 27u);
    int32_t *cells = reinterpret_cast<int32_t *>(warps + (kSplitBlock >> 5) * (kParts * 27u * 2u)) +
                     (threadIdx.x >> 5) * (3u * kParts);
    const int32_t icx = cell_coord(xp.x, d.cw), icy = cell_coord(xp.y, d.cw), icz = cell_coord(xp.z, d.cw);
    const int32_t ux = __shfl_up_sync(0xffffffffu, icx, 1), uy = __shfl_up_sync(0xffffffffu, icy, 1),
                  uz = __shfl_up_sync(0xffffffffu, icz, 1);
    const bool same = ux == icx && uy == icy && uz == icz;
    const uint32_t heads = __ballot_sync(0xffffffffu, on && (lane == 0 || !same));
    const uint32_t seg = __popc(heads & (0xFFFFFFFFu >> (31u - lane))) - 1u;
    if (heads >> lane & 1u) {
        cells[3 * seg] = icx;
        cells[3 * seg + 1] = icy;
        cells[3 * seg + 2] = icz;
    }
    __syncwarp();
    warp_ranges(d, a, shift, __popc(heads), cells, rng);
    if (!on) return;  // whole groups; only the groups' own lanes meet from here on
    uint32_t todo = near_cells(d, xp, icx, icy, icz);
    {  // this lane's run of the near cells
        const uint32_t m = __popc(todo), lo = m * sub / kSplit, hi = m * (sub + 1) / kSplit;
        for (uint32_t k = 0; k < lo; ++k) todo &= todo - 1u;
        uint32_t rest = todo;
        for (uint32_t k = lo; k < hi; ++k) rest &= rest - 1u;
        todo ^= rest;
    }
    const float4 *__restrict__ xa = a.xa;
    uint32_t tself = kNotListed;
    const uint32_t cnt = walk_ranges(rng + 27u * seg, todo, xa, xp, d.h2, cap, i, tself,
                                     [&](uint32_t k, uint32_t q) { run[k * kSplitBlock] = q; });
    uint32_t incl = cnt;
#pragma unroll
    for (uint32_t o = 1; o < kSplit; o <<= 1) {
        const uint32_t v = __shfl_up_sync(gmask, incl, o, kSplit);
        if (sub >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(gmask, incl, kSplit - 1, kSplit), pre = incl - cnt;
    // the particle's own place in the group's list (one lane holds it)
    uint32_t gself = tself != kNotListed ? pre + tself : 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t o = 1; o < kSplit; o <<= 1) gself = min(gself, __shfl_xor_sync(gmask, gself, o, kSplit));
    const bool listed = gself < cap;
    for (uint32_t t = 0; t < cnt && pre + t < cap; ++t) {
        const uint32_t g = pre + t;
        if (g != gself) list[(g - (g > gself ? 1u : 0u)) * kSmallBlock] = run[t * kSplitBlock];
    }
    const uint32_t nn = min(total, cap) - (listed ? 1u : 0u);
    __syncwarp(gmask);
    {  // the list's rows, one lane each in turn
        const uint64_t stride = a.nbr_stride;
        uint4 *row = reinterpret_cast<uint4 *>(list_of(a.nbr, i));
        const uint32_t per = d.list16 ? 8u : 4u;
        for (uint32_t r = sub; r * per < nn; r += kSplit) {
            uint32_t s[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) s[k] = k < per && r * per + k < nn ? list[(r * per + k) * kSmallBlock] - p_off : 0u;
            if (d.list16)
                list_st(row + r * stride, make_uint4(s[0] | s[1] << 16, s[2] | s[3] << 16, s[4] | s[5] << 16, s[6] | s[7] << 16));
            else
                list_st(row + r * stride, make_uint4(s[0] + p_off, s[1] + p_off, s[2] + p_off, s[3] + p_off));
        }
    }
    LamWalk o{xp, pair_const(d), LamSum()};
    if (listed) o.ls.ks = 1.f;
    for (uint32_t k0 = 0; k0 < nn; k0 += 32)
        lanes_sum<kSplit>(
            k0, nn, i, o, [&](uint32_t c) { return list[(k0 + 8 * sub + c) * kSmallBlock]; },
            [&](uint32_t q) -> float4 { return __ldg(xa + q); });
    if (sub == 0) {
        a.nnb[i] = (uint8_t)nn;
        a.selfat[i] = listed ? (uint8_t)gself : kNotListed;
        a.xb[i] = make_float4(xp.x, xp.y, xp.z, o.ls.lambda(d));  // the first delta-p pass gathers both
    }
}

// lambda for iterations >= 1 (memorizeKernelCalc + calcScalingFactor,
// pbf_kernel_memorization.cu:93-134 and pbf_constraint.cu:168-209, without the
// per-pair cache: W and grad W are recomputed from positions).  One thread
// per particle; the neighbour sums run in list order.  (position, lambda) goes
// into the other buffer, which the delta-p pass gathers.
template <int kChunk>
__global__ void __launch_bounds__(512, 2) k_lambda(StepArgs a, const float4 *__restrict__ xc, float4 *__restrict__ xo)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const PairConst pc = pair_const(d);
    const float4 xp = xc[i];
    LamSum ls;
    if (a.selfat[i] != kNotListed) ls.ks = 1.f;  // the particle's own w(0), not stored in the list
    list_walk_any<kChunk>(
        d.list16 != 0, list_of(a.nbr, i), a.nbr_stride, a.nnb[i], d.p_off, i,
        [&](uint32_t q) -> float4 { return __ldg(xc + q); },
        [&](const float4 &xj, bool on) {
            const PairGeo g = pair_geo(xp, xj);
            ls.add(g, masked(pair_ws(g.r2, pc), on));
        });
    xo[i] = make_float4(xp.x, xp.y, xp.z, ls.lambda(d));
    TILE_LOOP_END
}

// (two lanes: 3 blocks a SM, 136-168 registers; 4 at 128 spill nothing but take
// 72.1 us a step of 16,384 particles against 70.3, 5 at 96 spill and take 76.2)
template <uint32_t LANES>
__global__ void __launch_bounds__(kSmallBlock *LANES, LANES == 1 ? 8 : 3) k_lambda_small(StepArgs a, uint32_t tile,
                                                                 const float4 *__restrict__ xc,
                                                                 float4 *__restrict__ xo)
{
    SMALL_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    LamWalk o{xc[i], pair_const(d), LamSum()};
    if (a.selfat[i] != kNotListed) o.ls.ks = 1.f;
    if (small_sum<LANES>(a, d.list16 != 0, i, p_off, o, [&](uint32_t q) -> float4 { return __ldg(xc + q); }))
        xo[i] = make_float4(o.xp.x, o.xp.y, o.xp.z, o.ls.lambda(d));
    SMALL_LOOP_END
}

// s_corr forms, selected once per tile (a tile belongs to one scene).
enum ScorrForm { kScorrReference, kScorrTextbook, kScorrOff, kScorrTextbook4 };

struct ScorrConst {
    float sci;  // max(-lambda_i, 0), the reference form's own share
    float c;    // the factor of w^n: 10 alpha^4 / W(0.4h)^4 (reference), k alpha^n / W(dq h)^n (textbook)
    int sn;
};

// -(lambda_i + lambda_j + s_corr) for a pair (the coefficient of grad W in
// calcPositionUpdateCUDA, pbf_position_update.cu:131-188).  s_corr as a
// constant times a power of w = W / alpha: reference 10 W^4 / W(0.4h)^4
// (max(-lambda_i, 0) + max(-lambda_j, 0)) (pbf_position_update.cu:136-146),
// textbook k (W / W(dq h))^n (Macklin and Mueller 2013, eq. 13); its last
// product is fused into the sum.
template <int FORM>
__device__ __forceinline__ float dp_coef(float li, float lj, float W, const ScorrConst &c)
{
    const float ll = __fadd_rn(li, lj);
    if (FORM == kScorrReference) {
        const float w2 = __fmul_rn(W, W);
        const float tc = __fmul_rn(c.c, __fmul_rn(w2, w2));
        return -__fmaf_rn(__fadd_rn(c.sci, fmaxf(-lj, 0.f)), tc, ll);
    } else if (FORM == kScorrTextbook4) {
        const float w2 = __fmul_rn(W, W);
        return -__fmaf_rn(c.c, __fmul_rn(w2, w2), ll);
    } else if (FORM == kScorrTextbook) {
        float pw = 1.f;
        for (int e = 0; e < c.sn; ++e) pw = __fmul_rn(pw, W);
        return -__fmaf_rn(c.c, pw, ll);
    }
    return -ll;
}

__device__ __forceinline__ ScorrConst scorr_const(const SceneDesc &d, float li)
{
    ScorrConst c;
    c.sci = fmaxf(-li, 0.f);
    c.c = d.tensile_mode == PBF_TENSILE_REFERENCE ? d.tens_c : d.scorr_c;
    c.sn = d.scorr_n;
    return c;
}

// Where a step's velocity goes after a stage, by the scene's next stage: the
// list forms of vorticity and XSPH read it in working order beside the
// position (pa = x, y, z, vx; pb = vy, vz), the walk forms in sorted order
// (vs), and without a further stage it is the result.  slot() gives the
// sorted slot; i is the working slot.
template <class G>
__device__ __forceinline__ void put_velocity(const StepArgs &a, bool list_next, bool walk_next, uint32_t i, G &&slot,
                                             float4 x, float4 v)
{
    if (list_next) {
        a.pa[i] = make_float4(x.x, x.y, x.z, v.x);
        a.pb[i] = make_float2(v.y, v.z);
    } else {
        (walk_next ? a.vs : a.v)[slot()] = v;
    }
}

// The final position, velocity ((x_new - x_old) / dt: updateVelocityCUDA,
// pbf_update.cu:25-39) and id of working slot i.
__device__ __forceinline__ void put_final(const StepArgs &a, const SceneDesc &d, uint32_t i, float4 xn)
{
    const float4 xo = a.xold[i];
    const uint32_t g = __float_as_uint(xo.w);
    const float4 vn = make_float4(d.inv_dt * (xn.x - xo.x), d.inv_dt * (xn.y - xo.y), d.inv_dt * (xn.z - xo.z), 0.f);
    a.x[g] = xn;
    a.id[g] = a.id_tmp[i];  // ids follow the particles into sorted order
    const bool no_vort = d.vort_mode == PBF_VORTICITY_OFF;
    put_velocity(a, d.vort_mode == PBF_VORTICITY_TEXTBOOK || (no_vort && d.xsph_mode == PBF_XSPH_LIST),
                 d.vort_mode == PBF_VORTICITY_REFERENCE || (no_vort && d.xsph_mode == PBF_XSPH_WALK), i,
                 [&] { return g; }, xn, vn);
}

// A particle's delta-p from the list sum: scale, boundary response
// (pbf_response_collision.cu:12-66), x += dp (updateInterimPositionCUDA,
// pbf_constraint.cu:335-345) into the second buffer, so neighbours still read
// the old positions; on the last iteration the step's results.
__device__ __forceinline__ void dp_finish(const StepArgs &a, const SceneDesc &d, uint32_t s, uint32_t i, float4 xp,
                                          float3 sum, float4 *__restrict__ xo, int last)
{
    float3 dp = make_float3(sum.x * d.dp_k, sum.y * d.dp_k, sum.z * d.dp_k);  // m beta / rho0
    const bool ok = collide(d, a.bnd, make_float3(xp.x, xp.y, xp.z), dp);
    if (!ok) atomicOr(a.flags + s, PBF_FLAG_COLLISION_LIMIT);
    const float4 xn = make_float4(xp.x + dp.x, xp.y + dp.y, xp.z + dp.z, 0.f);
    if (last)
        put_final(a, d, i, xn);
    else
        xo[i] = xn;
}

// The s_corr form once per tile (a tile belongs to one scene): f<FORM>().
template <class F>
__device__ __forceinline__ float3 by_scorr(const SceneDesc &d, F &&f)
{
    if (d.tensile_mode == PBF_TENSILE_REFERENCE) return f(std::integral_constant<int, kScorrReference>());
    if (d.tensile_mode == PBF_TENSILE_TEXTBOOK && d.scorr_n == 4) return f(std::integral_constant<int, kScorrTextbook4>());
    if (d.tensile_mode == PBF_TENSILE_TEXTBOOK) return f(std::integral_constant<int, kScorrTextbook>());
    return f(std::integral_constant<int, kScorrOff>());
}

// One pair's share of the sum of -(lambda_i + lambda_j + s_corr) grad W (the
// body of calcPositionUpdateCUDA, pbf_position_update.cu:131-188): adds
// (coefficient * s) d.  Lambdas in .w.  PK: the x and y differences and sums by
// one packed operation each (the same bits; measured faster in large steps only).
template <int FORM, bool PK>
struct DpSum {
    float4 xp;
    PairConst pc;
    ScorrConst sc;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
    __device__ __forceinline__ DpSum(const SceneDesc &d, float4 x) : xp(x), pc(pair_const(d)), sc(scorr_const(d, x.w)) {}
    struct Term {
        float f, d0, d1, d2;
    };
    __device__ __forceinline__ Term term(const float4 &xq, bool on) const
    {
        const PairGeo g = pair_geo<PK>(xp, xq);
        const PairWS k = pair_ws(g.r2, pc);
        const float f = __fmul_rn(dp_coef<FORM>(xp.w, xq.w, k.W, sc), k.s);
        return Term{on ? f : 0.f, g.d0, g.d1, g.d2};
    }
    __device__ __forceinline__ void add(const Term &t)
    {
        if (PK) {
            fma2(s0, s1, t.f, t.f, t.d0, t.d1);
        } else {
            s0 = __fmaf_rn(t.f, t.d0, s0);
            s1 = __fmaf_rn(t.f, t.d1, s1);
        }
        s2 = __fmaf_rn(t.f, t.d2, s2);
    }
    template <uint32_t LANES>
    __device__ __forceinline__ void pass(uint32_t gmask, uint32_t lane)
    {
        for (float *f : {&s0, &s1, &s2}) *f = __shfl_sync(gmask, *f, lane, LANES);
    }
};

// delta-p with s_corr (calcPositionUpdateCUDA cached, pbf_position_update.cu:131-188),
// in list order.  Chunks of 4: 4 x 277 us at 5.95 M particles in 256 scenes
// (290 in chunks of 8), 4 x 34 at 1 M of h = 1.4 spacings (38), the same at 1 M of
// h = 2 spacings; the pair's longer arithmetic leaves fewer registers than lambda's.
__global__ void __launch_bounds__(512, 2) k_dp(StepArgs a, const float4 *__restrict__ xc, float4 *__restrict__ xo,
                                               int last)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (last && local == 0) a.scene_num[s] = live;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 xp = xc[i];
    const float3 sum = by_scorr(d, [&](auto form) {
        DpSum<decltype(form)::value, true> o(d, xp);
        list_walk_any<4>(
            d.list16 != 0, list_of(a.nbr, i), a.nbr_stride, a.nnb[i], d.p_off, i,
            [&](uint32_t q) -> float4 { return __ldg(xc + q); }, [&](const float4 &xq, bool on) { o.add(o.term(xq, on)); });
        return make_float3(o.s0, o.s1, o.s2);
    });
    dp_finish(a, d, s, i, xp, sum, xo, last);
    TILE_LOOP_END
}

template <uint32_t LANES>
__global__ void __launch_bounds__(kSmallBlock *LANES, LANES == 1 ? 8 : 3) k_dp_small(StepArgs a, uint32_t tile, const float4 *__restrict__ xc,
                                                             float4 *__restrict__ xo, int last)
{
    SMALL_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    const float4 xp = xc[i];
    bool first = true;
    const float3 sum = by_scorr(d, [&](auto form) {
        DpSum<decltype(form)::value, false> o(d, xp);
        first = small_sum<LANES>(a, d.list16 != 0, i, p_off, o, [&](uint32_t q) -> float4 { return __ldg(xc + q); });
        return make_float3(o.s0, o.s1, o.s2);
    });
    if (first) dp_finish(a, d, s, i, xp, sum, xo, last);
    SMALL_LOOP_END
}

// iters == 0: positions stay at the prediction; v from the velocity update.
__global__ void __launch_bounds__(512) k_finalize(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local == 0) a.scene_num[s] = live;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 xn = a.xa[i];
    put_final(a, d, i, make_float4(xn.x, xn.y, xn.z, 0.f));
    TILE_LOOP_END
}

// A neighbour's (x, v) as the list passes load it.
struct PhaseRec {
    float4 A;
    float2 B;
};

// Vorticity, pass 1 (calcVorticityCUDA, pbf_vorticity_confinement.cu:87-115):
// omega_i = m/rho0 * sum_j (v_j - v_i) x r_hat * W'(r).
struct OmegaSum {
    float4 xi, vi;
    float kh, w0 = 0.f, w1 = 0.f, w2 = 0.f;
    __device__ __forceinline__ OmegaSum(float4 x, float4 v, float k) : xi(x), vi(v), kh(k) {}
    struct Term {
        float c0, c1, c2, wd;
        bool on;
    };
    __device__ __forceinline__ Term term(float4 xj, float vx, float vy, float vz, bool on) const
    {
        const float p0 = xj.x - xi.x, p1 = xj.y - xi.y, p2 = xj.z - xi.z;
        const float r2 = p0 * p0 + p1 * p1 + p2 * p2;
        const float inv_r = rsqrtf(r2);
        const float v0 = vx - vi.x, v1 = vy - vi.y, v2 = vz - vi.z;
        return Term{v1 * p2 - v2 * p1, v2 * p0 - v0 * p2, v0 * p1 - v1 * p0, wspiky_d(r2 * inv_r, kh) * inv_r,
                    on && r2 > 0.f};
    }
    __device__ __forceinline__ Term term(const PhaseRec &r, bool on) const { return term(r.A, r.A.w, r.B.x, r.B.y, on); }
    __device__ __forceinline__ void add(const Term &t)
    {
        if (t.on) {
            w0 += t.c0 * t.wd;
            w1 += t.c1 * t.wd;
            w2 += t.c2 * t.wd;
        }
    }
    __device__ __forceinline__ void add(float4 xj, float vx, float vy, float vz, bool on = true)
    {
        add(term(xj, vx, vy, vz, on));
    }
    template <uint32_t LANES>
    __device__ __forceinline__ void pass(uint32_t gmask, uint32_t lane)
    {
        for (float *f : {&w0, &w1, &w2}) *f = __shfl_sync(gmask, *f, lane, LANES);
    }
};

// omega, and |omega| once per particle beside the position (xs is free after
// the reorder): pass 2 gathers both with one load per neighbour
__device__ __forceinline__ void put_omega(const StepArgs &a, const SceneDesc &d, uint32_t i, const OmegaSum &o)
{
    const float mr = d.m * d.inv_rho0;
    const float4 wi = make_float4(mr * o.w0, mr * o.w1, mr * o.w2, 0.f);
    a.w[i] = wi;
    a.xs[i] = make_float4(o.xi.x, o.xi.y, o.xi.z, sqrtf(wi.x * wi.x + wi.y * wi.y + wi.z * wi.z));
}

// The list form: the textbook kernel over the step's neighbour list, working
// slots, neighbours' (x, v) in pa and pb.  One instance per list format (each
// skips the other format's scenes) keeps its registers, and so its
// occupancy, to that format's loop.
template <bool L16>
__global__ void __launch_bounds__(512, 2) k_vort_omega(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.vort_mode != PBF_VORTICITY_TEXTBOOK || (d.list16 != 0) != L16) continue;
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 A = a.pa[i];
    const float2 B = a.pb[i];
    OmegaSum o(A, make_float4(A.w, B.x, B.y, 0.f), d.inv_h);
    const float4 *__restrict__ pa = a.pa;
    const float2 *__restrict__ pb = a.pb;
    // groups of 4 in 64 registers: 381 us (u16, 5.95 M particles) and 80 us
    // (u32, 1 M); groups of 8 hold 48 record registers and take 550 us
    list_walk_any<4>(
        L16, list_of(a.nbr, i), a.nbr_stride, a.nnb[i], d.p_off, i,
        [&](uint32_t q) -> PhaseRec { return PhaseRec{__ldg(pa + q), __ldg(pb + q)}; },
        [&](const PhaseRec &r, bool on) { o.add(r.A, r.A.w, r.B.x, r.B.y, on); });
    put_omega(a, d, i, o);
    TILE_LOOP_END
}

template <uint32_t LANES>
__global__ void __launch_bounds__(kSmallBlock *LANES, LANES == 1 ? 8 : 3) k_vort_omega_small(StepArgs a, uint32_t tile)
{
    SMALL_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.vort_mode != PBF_VORTICITY_TEXTBOOK) return;
    const float4 *__restrict__ pa = a.pa;
    const float2 *__restrict__ pb = a.pb;
    const float4 A = pa[i];
    const float2 B = pb[i];
    OmegaSum o(A, make_float4(A.w, B.x, B.y, 0.f), d.inv_h);
    if (small_sum<LANES>(a, d.list16 != 0, i, p_off, o,
                         [&](uint32_t q) -> PhaseRec { return PhaseRec{__ldg(pa + q), __ldg(pb + q)}; }))
        put_omega(a, d, i, o);
    SMALL_LOOP_END
}

// The reference's uncapped 27-cell walk over final positions in sorted order,
// with h passed where 1/h is expected (pbf_vorticity_confinement.cu:28).
__global__ void __launch_bounds__(512) k_vort_omega_walk(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.vort_mode != PBF_VORTICITY_REFERENCE) continue;
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 *__restrict__ x = a.x;
    const float4 *__restrict__ vs = a.vs;
    const float4 xi = x[i];
    OmegaSum o(xi, vs[i], d.h);
    // the kernel scaled by h reaches the whole 27-cell block
    walk27_batched(
        d, a.offsets, d.p_off - base, xi,
        [&](uint32_t j) -> bool {
            const float4 xj = __ldg(x + j);
            const float p0 = xj.x - xi.x, p1 = xj.y - xi.y, p2 = xj.z - xi.z;
            return p0 * p0 + p1 * p1 + p2 * p2 > 0.f;
        },
        [&](uint32_t j) {
            const float4 vj = __ldg(vs + j);
            o.add(__ldg(x + j), vj.x, vj.y, vj.z);
        });
    put_omega(a, d, i, o);
    TILE_LOOP_END
}

// Vorticity, pass 2 (addVorticityConfinementCUDA, pbf_vorticity_confinement.cu:192-222):
// the sum of |omega_j| grad W.
struct EtaSum {
    float4 xi;
    float kh, sgn, n0 = 0.f, n1 = 0.f, n2 = 0.f;
    __device__ __forceinline__ EtaSum(float4 x, float k, float sg) : xi(x), kh(k), sgn(sg) {}
    struct Term {
        float f, p0, p1, p2;
        bool on;
    };
    __device__ __forceinline__ Term term(float4 xj, bool on) const  // (x_j, |omega_j|)
    {
        const float p0 = xj.x - xi.x, p1 = xj.y - xi.y, p2 = xj.z - xi.z;
        const float r2 = p0 * p0 + p1 * p1 + p2 * p2;
        const float inv_r = rsqrtf(r2);
        return Term{sgn * xj.w * wspiky_d(r2 * inv_r, kh) * inv_r, p0, p1, p2, on && r2 > 0.f};
    }
    __device__ __forceinline__ void add(const Term &t)
    {
        if (t.on) {
            n0 += t.f * t.p0;
            n1 += t.f * t.p1;
            n2 += t.f * t.p2;
        }
    }
    __device__ __forceinline__ void add(float4 xj, bool on = true) { add(term(xj, on)); }
    template <uint32_t LANES>
    __device__ __forceinline__ void pass(uint32_t gmask, uint32_t lane)
    {
        for (float *f : {&n0, &n1, &n2}) *f = __shfl_sync(gmask, *f, lane, LANES);
    }
};

// The list form's velocity change, and where the velocity goes next.
__device__ __forceinline__ void put_confinement(const StepArgs &a, const SceneDesc &d, uint32_t i, const EtaSum &e)
{
    const float4 wi = a.w[i];
    const float mr = d.m * d.inv_rho0;
    const float4 A = a.pa[i];
    const float2 B = a.pb[i];
    float4 v = make_float4(A.w, B.x, B.y, 0.f);
    float n0 = e.n0 * mr, n1 = e.n1 * mr, n2 = e.n2 * mr;
    const float ln = sqrtf(n0 * n0 + n1 * n1 + n2 * n2);
    if (ln > 0.f) {
        n0 /= ln; n1 /= ln; n2 /= ln;
        const float c0 = n1 * wi.z - n2 * wi.y, c1 = n2 * wi.x - n0 * wi.z, c2 = n0 * wi.y - n1 * wi.x;
        v.x = v.x + d.dt * d.vort_eps * c0;
        v.y = v.y + d.dt * d.vort_eps * c1;
        v.z = v.z + d.dt * d.vort_eps * c2;
    }
    put_velocity(a, d.xsph_mode == PBF_XSPH_LIST, d.xsph_mode == PBF_XSPH_WALK, i,
                 [&] { return __float_as_uint(a.xold[i].w); }, A, v);
}

template <bool L16>
__global__ void __launch_bounds__(512, 2) k_vort_apply(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.vort_mode != PBF_VORTICITY_TEXTBOOK || (d.list16 != 0) != L16) continue;
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    // u16 lists index the array offset by the scene's first slot (no add per slot)
    const float4 *__restrict__ xw = a.xs + (L16 ? d.p_off : 0u);
    EtaSum e(a.xs[i], d.inv_h, -1.f);
    // u16 in groups of 2: 282 us at 5.95 M particles (286 by 4, 294 by 8, 274
    // slot by slot); u32 by 4: 59 us at 1 M (62 slot by slot); 128 against
    // 150 us for a batch with both formats
    list_walk_any<(L16 ? 2 : 4)>(
        L16, list_of(a.nbr, i), a.nbr_stride, a.nnb[i], 0u, L16 ? i - d.p_off : i,
        [&](uint32_t q) -> float4 { return __ldg(xw + q); }, [&](const float4 &xj, bool on) { e.add(xj, on); });
    put_confinement(a, d, i, e);
    TILE_LOOP_END
}

template <uint32_t LANES>
__global__ void __launch_bounds__(kSmallBlock *LANES, LANES == 1 ? 8 : 3) k_vort_apply_small(StepArgs a, uint32_t tile)
{
    SMALL_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.vort_mode != PBF_VORTICITY_TEXTBOOK) return;
    const float4 *__restrict__ xw = a.xs;
    EtaSum e(xw[i], d.inv_h, -1.f);
    if (small_sum<LANES>(a, d.list16 != 0, i, p_off, e, [&](uint32_t q) -> float4 { return __ldg(xw + q); }))
        put_confinement(a, d, i, e);
    SMALL_LOOP_END
}

// The reference's form (sorted order throughout; the XSPH list form that may
// follow reads working order).
__global__ void __launch_bounds__(512) k_vort_apply_walk(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.vort_mode != PBF_VORTICITY_REFERENCE) continue;
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 *__restrict__ x = a.x;
    const float4 *__restrict__ xw = a.xs;
    const float4 xi = x[i];
    EtaSum e(xi, d.h, 1.f);
    walk27_batched(
        d, a.offsets, d.p_off - base, xi,
        [&](uint32_t j) -> bool {
            const float4 xj = __ldg(x + j);
            const float p0 = xj.x - xi.x, p1 = xj.y - xi.y, p2 = xj.z - xi.z;
            return p0 * p0 + p1 * p1 + p2 * p2 > 0.f;
        },
        [&](uint32_t j) { e.add(__ldg(xw + j)); });
    const float4 wi = a.w[i];
    float4 v = a.vs[i];
    float n0 = e.n0, n1 = e.n1, n2 = e.n2;
    if (sqrtf(n0 * n0 + n1 * n1 + n2 * n2) > 0.f) {
        n0 = n0 * d.m * d.inv_rho0;
        n1 = n1 * d.m * d.inv_rho0;
        n2 = n2 * d.m * d.inv_rho0;
        const float ln = sqrtf(n0 * n0 + n1 * n1 + n2 * n2);
        n0 /= ln; n1 /= ln; n2 /= ln;
        const float c0 = n1 * wi.z - n2 * wi.y, c1 = n2 * wi.x - n0 * wi.z, c2 = n0 * wi.y - n1 * wi.x;
        v.x = v.x + d.vort_eps * c0 / d.inv_rho0 * d.dt;
        v.y = v.y + d.vort_eps * c1 / d.inv_rho0 * d.dt;
        v.z = v.z + d.vort_eps * c2 / d.inv_rho0 * d.dt;
    }
    put_velocity(a, d.xsph_mode == PBF_XSPH_LIST, d.xsph_mode == PBF_XSPH_WALK, a.wpos[i], [&] { return i; }, xi, v);
    TILE_LOOP_END
}

// XSPH (calcXSPHCUDA, pbf_xsph.cu:84-113): v_i += c m/rho0 sum_j (v_j - v_i) W(r_ij),
// NaN guard.  Bound by the L1 wavefronts of its gathers: a neighbour's
// position and velocity as 16 + 8 bytes instead of two float4 took the list
// form from 446 to 358 us at 5.95 M particles (u16 lists), 96 to 75 us at
// 1,048,576 (u32 lists).
struct XsphSum {
    float4 xi, vi;
    float ih2, alpha6, s0 = 0.f, s1 = 0.f, s2 = 0.f;
    __device__ __forceinline__ XsphSum(float4 x, float4 v, const SceneDesc &d)
        : xi(x), vi(v), ih2(d.inv_h * d.inv_h), alpha6(d.alpha6)
    {
    }
    struct Term {
        float W, v0, v1, v2;
        bool on;
    };
    __device__ __forceinline__ Term term(float4 xj, float vx, float vy, float vz, bool on) const
    {
        const float p0 = xj.x - xi.x, p1 = xj.y - xi.y, p2 = xj.z - xi.z;
        // Wpoly6 from r^2 (q^2 = r^2 / h^2 instead of (|r| / h)^2: no square
        // root per pair; the two differ by rounding only)
        const float q2 = (p0 * p0 + p1 * p1 + p2 * p2) * ih2;
        const float t = 1.f - q2;
        return Term{q2 <= 1.f ? alpha6 * t * t * t : 0.f, vx - vi.x, vy - vi.y, vz - vi.z, on};
    }
    __device__ __forceinline__ Term term(const PhaseRec &r, bool on) const { return term(r.A, r.A.w, r.B.x, r.B.y, on); }
    __device__ __forceinline__ void add(const Term &t)
    {
        if (t.on) {  // (not W = 0: an infinite velocity's difference from itself is NaN)
            s0 += t.v0 * t.W;
            s1 += t.v1 * t.W;
            s2 += t.v2 * t.W;
        }
    }
    __device__ __forceinline__ void add(float4 xj, float vx, float vy, float vz, bool on = true)
    {
        add(term(xj, vx, vy, vz, on));
    }
    template <uint32_t LANES>
    __device__ __forceinline__ void pass(uint32_t gmask, uint32_t lane)
    {
        for (float *f : {&s0, &s1, &s2}) *f = __shfl_sync(gmask, *f, lane, LANES);
    }
    __device__ __forceinline__ float4 result(const SceneDesc &d) const
    {
        float4 out = vi;
        if (!(isnan(s0) || isnan(s1) || isnan(s2))) {
            const float c = d.xsph_c * d.m * d.inv_rho0;
            out.x = vi.x + c * s0;
            out.y = vi.y + c * s1;
            out.z = vi.z + c * s2;
        }
        return out;
    }
};

template <bool L16>
__global__ void __launch_bounds__(512) k_xsph(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.xsph_mode != PBF_XSPH_LIST || (d.list16 != 0) != L16) continue;
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 *__restrict__ pa = a.pa;
    const float2 *__restrict__ pb = a.pb;
    const float4 A = a.pa[i];
    const float2 B = a.pb[i];
    XsphSum o(A, make_float4(A.w, B.x, B.y, 0.f), d);
    // groups of 8: 358 us (u16, 5.95 M particles) and 75 us (u32, 1 M), 372 and 77 in groups of 4
    list_walk_any<8>(
        L16, list_of(a.nbr, i), a.nbr_stride, a.nnb[i], d.p_off, i,
        [&](uint32_t q) -> PhaseRec { return PhaseRec{__ldg(pa + q), __ldg(pb + q)}; },
        [&](const PhaseRec &r, bool on) { o.add(r.A, r.A.w, r.B.x, r.B.y, on); });
    a.v[__float_as_uint(a.xold[i].w)] = o.result(d);
    TILE_LOOP_END
}

template <uint32_t LANES>
__global__ void __launch_bounds__(kSmallBlock *LANES, LANES == 1 ? 8 : 3) k_xsph_small(StepArgs a, uint32_t tile)
{
    SMALL_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.xsph_mode != PBF_XSPH_LIST) return;
    const float4 *__restrict__ pa = a.pa;
    const float2 *__restrict__ pb = a.pb;
    const float4 A = pa[i];
    const float2 B = pb[i];
    XsphSum o(A, make_float4(A.w, B.x, B.y, 0.f), d);
    if (small_sum<LANES>(a, d.list16 != 0, i, p_off, o,
                         [&](uint32_t q) -> PhaseRec { return PhaseRec{__ldg(pa + q), __ldg(pb + q)}; }))
        a.v[__float_as_uint(a.xold[i].w)] = o.result(d);
    SMALL_LOOP_END
}

// The reference's uncapped 27-cell walk (scenes with PBF_XSPH_WALK), sorted
// order.
__global__ void __launch_bounds__(512) k_xsph_walk(StepArgs a)
{
    TILE_LOOP_BEGIN
    const SceneDesc d = a.scenes[s];
    if (d.xsph_mode != PBF_XSPH_WALK) continue;
    const uint32_t base = a.offsets[d.c_off];
    const uint32_t live = a.offsets[d.c_off + d.ncell] - base;
    if (local >= live) continue;
    const uint32_t i = d.p_off + local;
    const float4 *__restrict__ x = a.x;
    const float4 *__restrict__ vs = a.vs;
    const float4 xi = x[i];
    XsphSum o(xi, vs[i], d);
    // W = 0 beyond h: those candidates add nothing (a non-finite velocity
    // of a non-neighbour is no longer folded into the sum; such particles
    // raise PBF_FLAG_NONFINITE in the next step's prediction)
    const float rcut2 = d.h2 * 1.0001f;
    walk27_batched(
        d, a.offsets, d.p_off - base, xi,
        [&](uint32_t j) -> bool {
            const float4 xj = __ldg(x + j);
            const float p0 = xj.x - xi.x, p1 = xj.y - xi.y, p2 = xj.z - xi.z;
            return p0 * p0 + p1 * p1 + p2 * p2 <= rcut2;
        },
        [&](uint32_t j) {
            const float4 vj = __ldg(vs + j);
            o.add(__ldg(x + j), vj.x, vj.y, vj.z);
        });
    a.v[i] = o.result(d);
    TILE_LOOP_END
}

__global__ void __launch_bounds__(512) k_unpack(StepArgs a, const uint32_t *__restrict__ pack_off,
                                                const float *__restrict__ sx, const float *__restrict__ sv)
{
    TILE_LOOP_BEGIN
    const uint32_t n = a.scene_num[s];
    if (local >= n) continue;
    const uint64_t q = (uint64_t)pack_off[s] + local;
    const uint32_t i = a.scenes[s].p_off + local;
    a.x[i] = make_float4(sx[3 * q], sx[3 * q + 1], sx[3 * q + 2], 0.f);
    a.v[i] = sv ? make_float4(sv[3 * q], sv[3 * q + 1], sv[3 * q + 2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    a.id[i] = local;  // a whole-scene upload numbers the particles afresh
    if (local == 0) a.next_id[s] = n;
    TILE_LOOP_END
}

__global__ void __launch_bounds__(512) k_pack(StepArgs a, const uint32_t *__restrict__ pack_off,
                                              float *__restrict__ dx, float *__restrict__ dv)
{
    TILE_LOOP_BEGIN
    const uint32_t n = a.scene_num[s];
    if (local >= n) continue;
    const uint64_t q = (uint64_t)pack_off[s] + local;
    const uint32_t i = a.scenes[s].p_off + local;
    if (dx) {
        const float4 t = a.x[i];
        dx[3 * q] = t.x;
        dx[3 * q + 1] = t.y;
        dx[3 * q + 2] = t.z;
    }
    if (dv) {
        const float4 t = a.v[i];
        dv[3 * q] = t.x;
        dv[3 * q + 1] = t.y;
        dv[3 * q + 2] = t.z;
    }
    TILE_LOOP_END
}

__global__ void k_set_u32(uint32_t *dst, uint32_t value) { *dst = value; }

// Packed offsets of the active scenes from their live counts, on the device:
// pack_off[active[k]] = the counts of active[0..k) summed, counts[k] = the
// count of active[k] (k-th active scene in slot order).  One block.
__global__ void __launch_bounds__(1024) k_pack_offsets(const uint32_t *__restrict__ active, uint32_t n_active,
                                                       const uint32_t *__restrict__ scene_num,
                                                       uint32_t *__restrict__ pack_off, uint32_t *__restrict__ counts)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    if (t == 0) carry = 0;
    __syncthreads();
    for (uint32_t k0 = 0; k0 < n_active; k0 += blockDim.x) {
        const uint32_t k = k0 + t;
        const uint32_t id = k < n_active ? active[k] : 0u;
        const uint32_t c = k < n_active ? scene_num[id] : 0u;
        const uint32_t incl = warp_incl_scan(c);
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        if (warp == 0) ws[lane] = warp_incl_scan(lane < (blockDim.x >> 5) ? ws[lane] : 0u);
        __syncthreads();
        const uint32_t before = carry + (warp ? ws[warp - 1] : 0u) + incl - c;
        if (k < n_active) {
            pack_off[id] = before;
            counts[k] = c;
        }
        __syncthreads();
        if (t == blockDim.x - 1) carry = before + c;
        __syncthreads();
    }
}

__global__ void k_aos3_to_f4(const float *__restrict__ src, float4 *__restrict__ dst, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = make_float4(src[3 * i], src[3 * i + 1], src[3 * i + 2], 0.f);
}

// A scene's n uploaded particles widened into the phase and numbered, and the
// scene's counters, in one launch: five small launches (x, v, ids, two
// counters) took 15.4 us for 4,096 particles, this one 3.8.  next_id:
// null for an append, whose ids continue from *id0 (bumped by a launch of its
// own: other blocks may not have read it yet).
__global__ void k_load_phase(const float *__restrict__ sx, const float *__restrict__ sv, float4 *__restrict__ x,
                             float4 *__restrict__ v, uint32_t *__restrict__ id, const uint32_t *id0, uint32_t *next_id,
                             uint32_t *scene_num, uint32_t n, uint32_t total)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *scene_num = total;
        if (next_id) *next_id = n;
    }
    if (i >= n) return;
    const uint32_t first = next_id ? 0u : *id0;
    x[i] = make_float4(sx[3 * i], sx[3 * i + 1], sx[3 * i + 2], 0.f);
    v[i] = sv ? make_float4(sv[3 * i], sv[3 * i + 1], sv[3 * i + 2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    id[i] = first + i;
}

// Either or both of x, v narrowed for the caller.  num: the particle count on
// the device (n is then its bound), written to num_out, pinned host memory, as
// a release: whoever sees it sees what the stream's earlier work wrote.  (The
// fence goes out before the count is requested: 0.4 us less than after it.)
__global__ void k_store_phase(const float4 *__restrict__ x, const float4 *__restrict__ v, float *__restrict__ dx,
                              float *__restrict__ dv, uint32_t n, const uint32_t *__restrict__ num,
                              uint32_t *num_out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (num) {
        if (i == 0) asm volatile("fence.acq_rel.sys;" ::: "memory");
        n = min(n, __ldg(num));
        if (i == 0) asm volatile("st.relaxed.sys.u32 [%0], %1;" ::"l"(num_out), "r"(n) : "memory");
    }
    if (i >= n) return;
    if (dx) {
        const float4 t = x[i];
        dx[3 * i] = t.x;
        dx[3 * i + 1] = t.y;
        dx[3 * i + 2] = t.z;
    }
    if (dv) {
        const float4 t = v[i];
        dv[3 * i] = t.x;
        dv[3 * i + 1] = t.y;
        dv[3 * i + 2] = t.z;
    }
}

}  // namespace

// The large steps' lambda pass by neighbour chunk, selected at run time.
using LambdaFn = void (*)(StepArgs, const float4 *, float4 *);
static LambdaFn lambda_fn(uint32_t chunk) { return chunk == 4 ? k_lambda<4> : k_lambda<8>; }

// Resident blocks per SM of each kernel at a tile size (cached per device,
// tile and chunk: the step asks for its launch shape every time it runs).
Occupancy occupancy(uint32_t tile, uint32_t chunk)
{
    static std::mutex mu;
    static std::map<std::tuple<int, uint32_t, uint32_t>, Occupancy> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, tile, chunk);
    {
        std::lock_guard<std::mutex> lk(mu);
        const auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    auto occ_b = [](const void *fn, uint32_t block) -> uint32_t {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, (int)block, 0);
        return b > 0 ? (uint32_t)b : 1u;
    };
    auto occ = [&](const void *fn) { return occ_b(fn, tile); };
    auto mn = [](uint32_t a, uint32_t b) { return a < b ? a : b; };
    Occupancy o;
    o.light = mn(mn(mn(occ((const void *)k_predict_hash<false>), occ((const void *)k_predict_hash<true>)),
                    occ((const void *)k_scatter)),
                 mn(mn(occ((const void *)k_rank_reorder), mn(occ((const void *)k_gather<false>),
                                                             occ((const void *)k_gather<true>))),
                    occ((const void *)k_finalize)));
    o.cells = occ_b((const void *)k_rank_cells, kCellTileMax);
    o.nb = occ((const void *)k_neighbors_lambda<false>);
    cudaFuncSetAttribute((const void *)k_neighbors_lambda<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kNbSmemMax);
    cudaFuncSetAttribute((const void *)k_neighbors_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNbSmemMax);
    cudaFuncSetAttribute((const void *)k_neighbors_split, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNbSmemMax);
    o.lambda = occ((const void *)lambda_fn(chunk));
    o.dp = occ((const void *)k_dp);
    o.omega[0] = occ((const void *)k_vort_omega<false>);
    o.omega[1] = occ((const void *)k_vort_omega<true>);
    o.apply[0] = occ((const void *)k_vort_apply<false>);
    o.apply[1] = occ((const void *)k_vort_apply<true>);
    o.xsph[0] = occ((const void *)k_xsph<false>);
    o.xsph[1] = occ((const void *)k_xsph<true>);
    std::lock_guard<std::mutex> lk(mu);
    cache[key] = o;
    return o;
}

void launch_aos3_to_f4(const float *src, float4 *dst, uint32_t n, cudaStream_t st)
{
    if (n) k_aos3_to_f4<<<(n + 255) / 256, 256, 0, st>>>(src, dst, n);
}

void launch_load_phase(const float *sx, const float *sv, float4 *x, float4 *v, uint32_t *id, uint32_t *next_id,
                       uint32_t *scene_num, uint32_t n, uint32_t total, bool append, cudaStream_t st)
{
    k_load_phase<<<n ? (n + 255) / 256 : 1, 256, 0, st>>>(sx, sv, x, v, id, next_id, append ? nullptr : next_id,
                                                          scene_num, n, total);
}

void launch_store_phase(const float4 *x, const float4 *v, float *dx, float *dv, uint32_t n, cudaStream_t st,
                        const uint32_t *num, uint32_t *num_out)
{
    if (n) k_store_phase<<<(n + 255) / 256, 256, 0, st>>>(x, v, dx, dv, n, num, num_out);
}

void launch_set_u32(uint32_t *dst, uint32_t value, cudaStream_t st) { k_set_u32<<<1, 1, 0, st>>>(dst, value); }

void launch_pack_offsets(const uint32_t *active, uint32_t n_active, const uint32_t *scene_num, uint32_t *pack_off,
                         uint32_t *counts, cudaStream_t st)
{
    if (n_active) k_pack_offsets<<<1, 1024, 0, st>>>(active, n_active, scene_num, pack_off, counts);
}

void launch_unpack(const StepArgs &a, const LaunchShape &sh, const uint32_t *pack_off, const float *src_x,
                   const float *src_v, cudaStream_t st)
{
    k_unpack<<<sh.grid, sh.tile, 0, st>>>(a, pack_off, src_x, src_v);
}

void launch_pack(const StepArgs &a, const LaunchShape &sh, const uint32_t *pack_off, float *dst_x, float *dst_v,
                 cudaStream_t st)
{
    k_pack<<<sh.grid, sh.tile, 0, st>>>(a, pack_off, dst_x, dst_v);
}

__global__ void k_set_packed_in(PackedIn *dst, const float *x, const float *v) { *dst = PackedIn{x, v}; }

void launch_set_packed_in(PackedIn *dst, const float *x, const float *v, cudaStream_t st)
{
    k_set_packed_in<<<1, 1, 0, st>>>(dst, x, v);
}

using ScanFn = void (*)(StepArgs);
static ScanFn scan_cluster_fn(uint32_t rounds)
{
    switch (rounds) {
    case 1: return k_scan_cluster<1>;
    case 2: return k_scan_cluster<2>;
    case 4: return k_scan_cluster<4>;
    case 8: return k_scan_cluster<8>;
    case 16: return k_scan_cluster<16>;
    default: return k_scan_cluster<kScanRoundsMax>;
    }
}

using FrontFn = void (*)(StepArgs, uint32_t, uint32_t);
static FrontFn front_fn(uint32_t rounds, bool packed)
{
    switch (rounds) {
    case 1: return packed ? k_front<1, true> : k_front<1, false>;
    case 2: return packed ? k_front<2, true> : k_front<2, false>;
    default: return packed ? k_front<4, true> : k_front<4, false>;
    }
}

// The largest cluster the scan may use on the current device (16 blocks of
// 1024 threads are beyond the portable size; a device without room for one
// such cluster takes 8), asked once per device.
uint32_t scan_cluster_limit()
{
    static std::mutex mu;
    static std::map<int, uint32_t> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto it = cache.find(dev);
    if (it != cache.end()) return it->second;
    bool ok = true;
    for (uint32_t r : {1u, 2u, 4u, 8u, 16u, kScanRoundsMax}) ok = allows_cluster(scan_cluster_fn(r)) && ok;
    for (uint32_t r = 1; r <= kFrontRounds; r *= 2)
        ok = allows_cluster(front_fn(r, false)) && allows_cluster(front_fn(r, true)) && ok;
    cache[dev] = ok ? kScanClusterMax : 8u;
    return cache[dev];
}

uint32_t enqueue_step(const StepArgs &a, const LaunchShape &sh, int iters, uint32_t post,
                      cudaStream_t st, StepHook *hook, bool packed)
{
    uint32_t nl = 0;
    const dim3 g(sh.grid), b(sh.tile);
#define PBF_LAUNCHED(name)                \
    do {                                  \
        ++nl;                             \
        if (hook) hook->launched(name);   \
    } while (0)
    const uint32_t gs = sh.small_tiles * (sh.tile / kSmallBlock);  // small steps: a block per part of a tile
    const uint32_t ls = kSmallBlock * (sh.small_lanes ? kLanes : 1u);  // threads of their list passes' blocks
    const bool front = sh.front && !hook;  // (a profile gets the phases one by one)
    if (front) {
        launch_cluster(front_fn(sh.front, packed), sh.front_cluster, st, a, sh.tile_shift, sh.small_tiles);
        PBF_LAUNCHED("k_front");
    } else {
        if (packed)
            k_predict_hash<true><<<g, b, 0, st>>>(a);
        else
            k_predict_hash<false><<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_predict_hash");
        if (sh.scan_grid == 0 && sh.scan_cluster) {
            launch_cluster(scan_cluster_fn(sh.scan_rounds), sh.scan_cluster, st, a);
            PBF_LAUNCHED("k_scan_single");  // the profile's name for the scan in one launch
        } else if (sh.scan_grid == 0) {  // small table: one block
            switch (sh.scan_rounds) {  // rounds of 1024 cells held in registers
#define PBF_SCAN_ROUNDS(r) \
        case r: k_scan_single_reg<r><<<1, 1024, 0, st>>>(a); break;
            PBF_SCAN_ROUNDS(1) PBF_SCAN_ROUNDS(2) PBF_SCAN_ROUNDS(3) PBF_SCAN_ROUNDS(4)
            PBF_SCAN_ROUNDS(5) PBF_SCAN_ROUNDS(6) PBF_SCAN_ROUNDS(7)
#undef PBF_SCAN_ROUNDS
            default: k_scan_single_reg<8><<<1, 1024, 0, st>>>(a); break;
            }
            PBF_LAUNCHED("k_scan_single");
        } else {
            k_scan_reduce<<<sh.scan_grid, 256, 0, st>>>(a);
            PBF_LAUNCHED("k_scan_reduce");
            k_scan_spine<<<1, 1024, 0, st>>>(a);
            PBF_LAUNCHED("k_scan_spine");
            k_scan_down<<<sh.scan_grid, 256, 0, st>>>(a);
            PBF_LAUNCHED("k_scan_down");
        }
        k_scatter<<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_scatter");
        if (sh.rank_each) {
            k_rank_reorder<<<g, b, 0, st>>>(a);
            PBF_LAUNCHED("k_rank_reorder");
        } else {
            k_rank_cells<<<sh.grid_cells, sh.cell_tile, 0, st>>>(a);
            PBF_LAUNCHED("k_rank_cells");
        }
        k_dense_sort<<<sh.grid, kRadixThreads, 0, st>>>(a, sh.tile, sh.small ? sh.small_tiles : 0u);
        PBF_LAUNCHED("k_dense_sort");
        if (sh.small && packed)
            k_gather_small<true><<<gs, kSmallBlock, 0, st>>>(a, sh.tile);
        else if (sh.small)
            k_gather_small<false><<<gs, kSmallBlock, 0, st>>>(a, sh.tile);
        else if (packed)
            k_gather<true><<<g, b, 0, st>>>(a);
        else
            k_gather<false><<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_gather");
    }
    if (sh.small) {
        if (sh.small_split)
            k_neighbors_split<<<gs, kSplitBlock, sh.nb_smem, st>>>(a, sh.tile);
        else
            k_neighbors_small<<<gs, kSmallBlock, sh.nb_smem, st>>>(a, sh.tile);
        PBF_LAUNCHED("k_neighbors_split");  // the profile's name for a small step's walk
    } else {
        if (sh.nb_smem)
            k_neighbors_lambda<true><<<sh.grid_nb, b, sh.nb_smem, st>>>(a);
        else
            k_neighbors_lambda<false><<<sh.grid_nb, b, 0, st>>>(a);
        PBF_LAUNCHED("k_neighbors_lambda");
    }
    for (int it = 0; it < iters; ++it) {  // positions in xa, (position, lambda) in xb
        const int last = it == iters - 1 ? 1 : 0;
        if (it > 0) {
            if (sh.small) {
                (sh.small_lanes ? k_lambda_small<kLanes> : k_lambda_small<1>)<<<gs, ls, 0, st>>>(a, sh.tile, a.xa, a.xb);
            } else {
                lambda_fn(sh.chunk)<<<sh.grid_lambda, b, 0, st>>>(a, a.xa, a.xb);
            }
            PBF_LAUNCHED("k_lambda");
        }
        if (sh.small) {
            (sh.small_lanes ? k_dp_small<kLanes> : k_dp_small<1>)<<<gs, ls, 0, st>>>(a, sh.tile, a.xb, a.xa, last);
        } else {
            k_dp<<<sh.grid_dp, b, 0, st>>>(a, a.xb, a.xa, last);
        }
        PBF_LAUNCHED("k_dp");
    }
    if (iters <= 0) {
        k_finalize<<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_finalize");
    }
    // the list forms: one instance per list format present, or the small steps'
    const bool l16 = (post & kPostList16) != 0, l32 = (post & kPostList32) != 0;
#define PBF_POST(kernel, grid)                                               \
    if (sh.small) {                                                          \
        (sh.small_lanes ? kernel##_small<kLanes> : kernel##_small<1>)<<<gs, ls, 0, st>>>(a, sh.tile); \
        PBF_LAUNCHED(#kernel);                                               \
    } else {                                                                 \
        if (l32) {                                                           \
            kernel<false><<<grid[0], b, 0, st>>>(a);                         \
            PBF_LAUNCHED(#kernel);                                           \
        }                                                                    \
        if (l16) {                                                           \
            kernel<true><<<grid[1], b, 0, st>>>(a);                          \
            PBF_LAUNCHED(#kernel);                                           \
        }                                                                    \
    }
    if (post & kPostVortTextbook) {
        PBF_POST(k_vort_omega, sh.grid_omega)
        PBF_POST(k_vort_apply, sh.grid_apply)
    }
    if (post & kPostVortReference) {
        k_vort_omega_walk<<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_vort_omega_walk");
        k_vort_apply_walk<<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_vort_apply_walk");
    }
    if (post & kPostXsphList) {
        PBF_POST(k_xsph, sh.grid_xsph)
    }
#undef PBF_POST
    if (post & kPostXsphWalk) {
        k_xsph_walk<<<g, b, 0, st>>>(a);
        PBF_LAUNCHED("k_xsph_walk");
    }
#undef PBF_LAUNCHED
    return nl;
}

}  // namespace pbf103
