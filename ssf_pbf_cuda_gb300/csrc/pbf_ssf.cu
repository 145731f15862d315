// Headless screen-space fluid (SSF) rendering: the reference's per-frame GL
// passes (src/main.cpp:372-564; shaders in asset/shader/) written as CUDA
// kernels that fill device image buffers.  Nothing here touches a graphics
// API: the rasteriser's coverage and attribute interpolation, the depth
// test, bilinear texture filtering and blending are spelled out.
//
// Images are row-major, row 0 at the bottom (GL window coordinates); pixel
// (i, j) has its centre at (i + 0.5, j + 0.5).
//
// This file is compiled with -fmad=false: every product and sum is rounded
// on its own, in the order written, like the CPU restatement built with
// -ffp-contract=off.  The depth splat and the normal pass therefore agree
// with it bit for bit; blur and shading differ only where expf / powf do.
#include <type_traits>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>

#include "pbf_after.cuh"
#include "pbf_engine.h"

#define CK(call)                                              \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess) {                              \
            pbf103::set_last_error(#call, e_);                \
            return PBF_ERROR_CUDA;                            \
        }                                                     \
    } while (0)

namespace pbf103 {
void set_last_error(const char *what, cudaError_t e);

namespace {

constexpr uint32_t kMaxSide = 8192;    // pixel-centre texel fetches stay exact up to here
constexpr uint32_t kEmptyDepth = 0x3f800000u;  // 1.0f, the depth clear (main.cpp:71-72)

// Per-frame constants, passed by value to every kernel.
struct Frame {
    uint32_t w, h, mode, clear8;  // clear8: the clear colour as RGBA8
    float proj[16], view[16], inv_proj[16];  // column-major m[c * 4 + r]
    float radius, point_scale, znear, zfar;
    float blur_radius, blur_scale, thickness, pad1;
    float clear[4];
    float incident[3];
    float inv_w, inv_h;  // 1 / width, 1 / height: tex_coord = (i + 0.5) * inv_w
};

// GLSL mat4 * vec4 (column-major), summed in column order.
__host__ __device__ inline float4 mat_vec(const float *m, float x, float y, float z, float w)
{
    return make_float4(m[0] * x + m[4] * y + m[8] * z + m[12] * w, m[1] * x + m[5] * y + m[9] * z + m[13] * w,
                       m[2] * x + m[6] * y + m[10] * z + m[14] * w, m[3] * x + m[7] * y + m[11] * z + m[15] * w);
}

__host__ __device__ inline float dot3(float ax, float ay, float az, float bx, float by, float bz)
{
    return ax * bx + ay * by + az * bz;
}

// ------------------------------------------------------------ depth splat --

// What the fragments of one particle share.
struct Splat {
    float x0, y0;       // quad: window corner a; sprite: window centre
    float rx, ry;       // quad: 1 / window width, height of the quad; sprite: 1 / size
    float ez;           // view-space depth of the centre (pos_from_eye.z)
    int i0, j0;         // first covered pixel column / row
    uint32_t bw, bh;    // covered pixel box
};

__device__ inline int clamp_pix(float v, uint32_t n)
{
    v = fminf(fmaxf(v, -1.f), (float)n);
    return (int)v;
}

// Pixels whose centre c satisfies lo <= c < hi: [first, last], clipped to
// the image; false when none.
__device__ inline bool centre_range(float lo, float hi, uint32_t n, int &first, int &last)
{
    int a = max(clamp_pix(floorf(lo - 0.5f), n), 0);
    for (int k = 0; k < 3 && a < (int)n && !((float)a + 0.5f >= lo); ++k) ++a;
    int b = min(clamp_pix(floorf(hi - 0.5f) + 1.f, n), (int)n - 1);
    for (int k = 0; k < 3 && b >= a && !((float)b + 0.5f < hi); ++k) --b;
    first = a;
    last = b;
    return a <= b && a < (int)n && (float)a + 0.5f >= lo && (float)b + 0.5f < hi;
}

// Per-particle set-up.  false: nothing of the particle reaches the image.
__device__ inline bool splat_setup(const Frame &f, float px, float py, float pz, Splat &s)
{
    const float4 e = mat_vec(f.view, px, py, pz, 1.f);  // vw * vec4(Position, 1), World = identity
    const float hw = (float)f.w * 0.5f, hh = (float)f.h * 0.5f;
    s.ez = e.z;
    float x0, x1, y0, y1;
    if (f.mode == PBF_SSF_SPLAT_QUAD) {
        // ssf_object.geom:21-50: corners P.xy +- 0.5 point_radius at P.zw
        const float hr = 0.5f * f.radius;
        const float ax = e.x - hr, ay = e.y - hr, dx = e.x + hr, by = e.y + hr;
        const float4 ca = mat_vec(f.proj, ax, ay, e.z, e.w);
        const float4 cd = mat_vec(f.proj, dx, ay, e.z, e.w);
        const float4 cb = mat_vec(f.proj, ax, by, e.z, e.w);
        // clip z and w depend on (z, w) alone, so the four corners clip alike
        if (!(-ca.w <= ca.z && ca.z <= ca.w)) return false;
        x0 = ca.x / ca.w * hw + hw;
        x1 = cd.x / cd.w * hw + hw;
        y0 = ca.y / ca.w * hh + hh;
        y1 = cb.y / cb.w * hh + hh;
        // counter-clockwise strip a, d, b, c is front-facing; a mirrored
        // quad is culled (GL_CULL_FACE, main.cpp:73)
        if (!(x1 > x0 && y1 > y0)) return false;
        s.x0 = x0;
        s.y0 = y0;
        s.rx = 1.f / (x1 - x0);
        s.ry = 1.f / (y1 - y0);
    } else {
        // ssf_point_sprite.vert:19-27: size = pointRadius * (pointScale / dist)
        const float dist = sqrtf(dot3(e.x, e.y, e.z, e.x, e.y, e.z));
        const float size = f.radius * (f.point_scale / dist);
        const float4 c = mat_vec(f.proj, e.x, e.y, e.z, 1.f);
        // a point is kept whole or dropped by its vertex's clip test
        if (!(-c.w <= c.x && c.x <= c.w && -c.w <= c.y && c.y <= c.w && -c.w <= c.z && c.z <= c.w)) return false;
        if (!(size > 0.f)) return false;
        const float xw = c.x / c.w * hw + hw, yw = c.y / c.w * hh + hh, half = size * 0.5f;
        x0 = xw - half;
        x1 = xw + half;
        y0 = yw - half;
        y1 = yw + half;
        s.x0 = xw;
        s.y0 = yw;
        s.rx = s.ry = 1.f / size;
    }
    int i1, j1;
    if (!centre_range(x0, x1, f.w, s.i0, i1) || !centre_range(y0, y1, f.h, s.j0, j1)) return false;
    s.bw = (uint32_t)(i1 - s.i0 + 1);
    s.bh = (uint32_t)(j1 - s.j0 + 1);
    return true;
}

// One fragment: ssf_object.frag:18-35 / ssf_point_sprite.frag:17-31.
// Returns the window depth, or a negative value when nothing is written.
// With the projection's z and w rows free of x and y, the depth needs only
// the z of pixelPos: clip.z / clip.w = (P22 z + P32) / (P23 z + P33).
__device__ inline float splat_fragment(const Frame &f, const Splat &s, int i, int j)
{
    const float cx = (float)i + 0.5f, cy = (float)j + 0.5f;
    float nx, ny;
    if (f.mode == PBF_SSF_SPLAT_QUAD) {
        // vertex_uv * 2 - 1; w is constant over the quad, so the perspective-
        // correct interpolation is the screen-space one
        nx = ((cx - s.x0) * s.rx) * 2.f - 1.f;
        ny = ((cy - s.y0) * s.ry) * 2.f - 1.f;
    } else {
        // gl_PointCoord (origin upper left) * (2, -2) + (-1, 1)
        nx = (0.5f + (cx - s.x0) * s.rx) * 2.f + -1.f;
        ny = (0.5f - (cy - s.y0) * s.ry) * -2.f + 1.f;
    }
    const float mag = nx * nx + ny * ny;
    if (mag > 1.f) return -1.f;  // discard: outside the circle
    const float pz = s.ez + sqrtf(1.f - mag) * f.radius;
    const float d = (f.proj[10] * pz + f.proj[14]) / (f.proj[11] * pz + f.proj[15]);
    if (d != d) return -1.f;
    return fminf(fmaxf(d, 0.f), 1.f) + 0.f;  // clamped to the depth range; + 0 turns -0 into +0
}

// Early depth rejection, exact: a fragment's view z lies between the centre's
// and the front point's (nz = 0 .. 1), and the depth formula is monotone there
// unless its denominator changes sign, so no fragment is nearer than the nearer
// of the two by more than the formula's rounding: a pixel already holding a
// depth at or below the bound keeps it.  A sphere that reaches past the eye
// plane has fragments at any depth: bound 0.
__device__ inline float depth_bound(const Frame &f, float pz)
{
    const float num = f.proj[10] * pz + f.proj[14], den = f.proj[11] * pz + f.proj[15];
    if (!(den > 0.f)) return 0.f;
    // |float - exact| <= 2^-22 (|P22 pz| + |P32|) / den + ulp / 2; four times that
    return num / den - 4.f * (2.3841858e-7f * (fabsf(f.proj[10] * pz) + fabsf(f.proj[14])) / den + 6e-8f);
}

__device__ inline uint32_t front_bound(const Frame &f, float ez)
{
    const float b0 = depth_bound(f, ez), b1 = depth_bound(f, ez + f.radius);
    if (!(b0 > 0.f && b1 > 0.f)) return 0u;  // also NaN
    return __float_as_uint(fminf(fminf(b0, b1), 1.f));
}

// A particle's splat as the raster kernel reads it (32 B): (x0, y0, rx, ry)
// and (ez bits, depth bound bits, i0 | j0 << 16, bw | bh << 16); bw = 0 when
// nothing of the particle reaches the image.
struct SplatRec {
    float4 a;
    uint4 b;
};

// One thread per particle: the per-particle set-up, once.
template <int STRIDE>
__global__ void __launch_bounds__(256) k_ssf_setup(const float *__restrict__ x, const uint32_t *__restrict__ n_dev,
                                                   uint32_t n_arg, Frame f, SplatRec *__restrict__ rec)
{
    after_previous();
    release_next();
    const uint32_t n = n_dev ? *n_dev : n_arg;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float *xp = x + (size_t)p * STRIDE;
        Splat s;
        SplatRec r;
        if (splat_setup(f, __ldg(xp), __ldg(xp + 1), __ldg(xp + 2), s)) {
            r.a = make_float4(s.x0, s.y0, s.rx, s.ry);
            r.b = make_uint4(__float_as_uint(s.ez), front_bound(f, s.ez), (uint32_t)s.i0 | ((uint32_t)s.j0 << 16),
                             s.bw | (s.bh << 16));
        } else {
            r.a = make_float4(0.f, 0.f, 0.f, 0.f);
            r.b = make_uint4(0u, 0u, 0u, 0u);
        }
        rec[p] = r;
    }
}

// Particle bound up to which a frame is drawn by pixel boxes: the device has
// most of such a set in flight at once, so tile bounds reject little.  Frames
// by boxes and by tiles: 12,000 particles at 640 x 360 49.5 and 51.6 us, 20,000 at
// 1280 x 720 75.1 and 75.4, 32,768 82.2 and 80.1, 100,000 at 1001 x 563 96 and 83.
constexpr uint32_t kBoxRaster = 20000;
// Small images are drawn by boxes too: their depths stay in L1, which the box
// raster reads through, where tiles go to L2 for theirs (96 KB at the larger
// bound, which very many particles, less often near the front, do not gain
// from).  Frames by tiles and by boxes, 60,000 and 200,000 particles near the
// eye: 64 x 36 80 -> 35 and 177 -> 61 us, 128 x 72 60 -> 39 and 148 -> 66, 192 x 108
// 71 -> 46 and 128 -> 80, 320 x 180 78 -> 72 and 123 -> 133; 1,000,000 before the
// camera: 128 x 72 260 -> 209, 192 x 108 178 -> 210.
constexpr uint32_t kBoxPixels = 16384, kBoxPixelsFew = 24576, kBoxFew = 262144;

// One warp per particle, lanes over its pixel box (stepped without
// division): every pixel tests its own depth alone.
__global__ void __launch_bounds__(256) k_ssf_raster_box(const SplatRec *rec,
                                                    const uint32_t *__restrict__ n_dev, uint32_t n_arg, Frame f,
                                                    uint32_t *__restrict__ depth)
{
    after_previous();  // (no release: its cached depth reads end before the next launch's blocks start)
    const uint32_t n = n_dev ? *n_dev : n_arg;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    // Draw near particles first, so the early rejection finds nearer depths
    // already in place: particle sets are often ordered along one axis
    // (lattices, cell-sorted phases), so walk them in reverse when the last
    // particle sits nearer the camera than the first.  Order changes no
    // result: the depth test keeps the minimum.
    bool reverse = false;
    if (n > 1) {
        const float z0 = __uint_as_float(rec[0].b.x), z1 = __uint_as_float(rec[n - 1].b.x);
        reverse = z1 > z0;  // view space looks down -z: larger z is nearer
    }
    for (uint32_t p0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); p0 < n; p0 += warps) {
        const uint32_t p = reverse ? n - 1 - p0 : p0;
        const uint4 rb = rec[p].b;
        const uint32_t bw = rb.w & 0xffffu;
        if (bw == 0u) continue;
        const float4 ra = rec[p].a;
        Splat q;
        q.x0 = ra.x;
        q.y0 = ra.y;
        q.rx = ra.z;
        q.ry = ra.w;
        q.ez = __uint_as_float(rb.x);
        q.i0 = (int)(rb.z & 0xffffu);
        q.j0 = (int)(rb.z >> 16);
        q.bw = bw;
        q.bh = rb.w >> 16;
        const uint32_t bound = rb.y;
        const uint32_t dj = 32u / q.bw, di = 32u % q.bw;
        // two cursors, 32 fragments apart, so two depth loads are in flight
        uint32_t ci = lane % q.bw, cj = lane / q.bw;
        uint32_t ci2 = ci + di, cj2 = cj + dj;
        if (ci2 >= q.bw) {
            ci2 -= q.bw;
            ++cj2;
        }
        while (cj < q.bh) {
            const bool two = cj2 < q.bh;
            const int i1 = q.i0 + (int)ci, j1 = q.j0 + (int)cj, i2 = q.i0 + (int)ci2, j2 = q.j0 + (int)cj2;
            uint32_t *d1 = depth + (size_t)j1 * f.w + (uint32_t)i1;
            uint32_t *d2 = two ? depth + (size_t)j2 * f.w + (uint32_t)i2 : d1;
            const uint32_t c1 = *d1, c2 = *d2;
            if (c1 > bound) {
                const float d = splat_fragment(f, q, i1, j1);
                if (d >= 0.f && __float_as_uint(d) < c1) atomicMin(d1, __float_as_uint(d));
            }
            if (two && c2 > bound) {
                const float d = splat_fragment(f, q, i2, j2);
                if (d >= 0.f && __float_as_uint(d) < c2) atomicMin(d2, __float_as_uint(d));
            }
            // both cursors advance 64 fragments
            ci = ci2 + di;
            cj = cj2 + dj;
            if (ci >= q.bw) {
                ci -= q.bw;
                ++cj;
            }
            ci2 = ci + di;
            cj2 = cj + dj;
            if (ci2 >= q.bw) {
                ci2 -= q.bw;
                ++cj2;
            }
        }
    }
}

// One warp per particle, over the 8 x 4 pixel tiles its pixel box touches.
// The depth test (GL_LESS against the cleared 1.0) is an atomic minimum on
// the float bits, which order like the values in [0, 1]; the result does not
// depend on the order of fragments.
//
// Bound by fragments that cannot win: hundreds of particles overlap a pixel.
// zmax holds an upper bound of every tile's depths (the largest depth a warp
// saw there, which depths only fall below), so a particle whose front is not
// nearer skips a tile by one read, 32 tiles at once over the lanes; a pixel's
// own depth rejects the rest.  By pixel boxes with the per-pixel test alone
// 32,768 particles at 1280 x 720 take 21 us and 524,288 at 1920 x 1080 330 us,
// by tiles 19 and 96, 91 with each particle's record requested a particle
// ahead (a frame 199 -> 194 us).
constexpr int kAhead = 4;  // two tiles at a time: 524,288 particles 209 us a frame against 202
__global__ void __launch_bounds__(256) k_ssf_raster(const SplatRec *rec,
                                                    const uint32_t *__restrict__ n_dev, uint32_t n_arg, Frame f,
                                                    uint32_t *__restrict__ depth, uint32_t *__restrict__ zmax)
{
    after_previous();
    release_next();
    const uint32_t n = n_dev ? *n_dev : n_arg;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t tw = (f.w + 7u) >> 3;  // tiles of a row
    // Draw near particles first, so the early rejection finds nearer depths
    // already in place: particle sets are often ordered along one axis
    // (lattices, cell-sorted phases), so walk them in reverse when the last
    // particle sits nearer the camera than the first.  Order changes no
    // result: the depth test keeps the minimum.
    bool reverse = false;
    if (n > 1) {
        const float z0 = __uint_as_float(rec[0].b.x), z1 = __uint_as_float(rec[n - 1].b.x);
        reverse = z1 > z0;  // view space looks down -z: larger z is nearer
    }
    uint32_t p0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    uint4 nb = make_uint4(0u, 0u, 0u, 0u);
    float4 na = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p0 < n) {
        const uint32_t p = reverse ? n - 1 - p0 : p0;
        nb = rec[p].b;
        na = rec[p].a;
    }
    for (; p0 < n; p0 += warps) {
        const uint4 rb = nb;
        const float4 ra = na;
        if (p0 + warps < n) {  // the next particle's record is requested a particle ahead
            const uint32_t p = reverse ? n - 1 - (p0 + warps) : p0 + warps;
            nb = rec[p].b;
            na = rec[p].a;
        }
        Splat q;
        q.bw = rb.w & 0xffffu;
        if (q.bw == 0u) continue;
        q.x0 = ra.x;
        q.y0 = ra.y;
        q.rx = ra.z;
        q.ry = ra.w;
        q.ez = __uint_as_float(rb.x);
        q.i0 = (int)(rb.z & 0xffffu);
        q.j0 = (int)(rb.z >> 16);
        q.bh = rb.w >> 16;
        const uint32_t bound = rb.y;
        const uint32_t tx0 = (uint32_t)q.i0 >> 3, ty0 = (uint32_t)q.j0 >> 2;
        const uint32_t ntx = (((uint32_t)q.i0 + q.bw - 1u) >> 3) - tx0 + 1u;
        const uint32_t nt = ntx * ((((uint32_t)q.j0 + q.bh - 1u) >> 2) - ty0 + 1u);
        for (uint32_t t0 = 0; t0 < nt; t0 += 32) {
            const uint32_t t = t0 + lane, row = t / ntx;
            const uint32_t tx = tx0 + t - row * ntx, ty = ty0 + row;
            const uint32_t zt = t < nt ? __ldcg(zmax + (size_t)ty * tw + tx) : 0u;
            uint32_t open = __ballot_sync(0xffffffffu, zt > bound);
            while (open) {  // the same in every lane; kAhead tiles at a time, their depths requested together
                uint32_t l[kAhead], i[kAhead], j[kAhead], c[kAhead];
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    l[k] = open ? (uint32_t)__ffs((int)open) - 1u : 32u;  // 32: no further tile
                    open &= open - 1u;
                    i[k] = __shfl_sync(0xffffffffu, tx, l[k] & 31u) * 8u + (lane & 7u);
                    j[k] = __shfl_sync(0xffffffffu, ty, l[k] & 31u) * 4u + (lane >> 3);
                    c[k] = l[k] < 32u && i[k] < f.w && j[k] < f.h ? __ldcg(depth + (size_t)j[k] * f.w + i[k]) : 0u;
                }
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    if (l[k] < 32u) {
                        if (i[k] - (uint32_t)q.i0 < q.bw && j[k] - (uint32_t)q.j0 < q.bh && c[k] > bound) {
                            const float z = splat_fragment(f, q, (int)i[k], (int)j[k]);
                            if (z >= 0.f && __float_as_uint(z) < c[k]) {
                                c[k] = __float_as_uint(z);
                                atomicMin(depth + (size_t)j[k] * f.w + i[k], c[k]);
                            }
                        }
                        const uint32_t most = __reduce_max_sync(0xffffffffu, c[k]);
                        if (lane == l[k] && most < zt) atomicMin(zmax + (size_t)ty * tw + tx, most);
                    }
                }
            }
        }
    }
}

__global__ void k_ssf_fill(uint32_t *__restrict__ dst, uint32_t value, uint32_t n)
{
    release_next();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = value;
}

// --------------------------------------------------------- screen passes --

// ssf_blur.frag:27-34
__device__ inline float linearize(float d, const Frame &f) { return (2.f * f.znear) / (f.zfar + f.znear - d * (f.zfar - f.znear)); }
__device__ inline float exponentialize(float l, const Frame &f)
{
    return (f.zfar + f.znear - (2.f * f.znear) / l) / (f.zfar - f.znear);
}

// uvToEye: ssf_blur.frag:36-42 and ssf_shading.frag flip y (t * -2 + 1);
// ssf_normal.frag:17-23 does not (t * 2 - 1).
__device__ inline float3 uv_to_eye(const Frame &f, float s, float t, float d, bool flip)
{
    const float x = s * 2.f - 1.f;
    const float y = flip ? t * -2.f + 1.f : t * 2.f - 1.f;
    const float4 c = mat_vec(f.inv_proj, x, y, d, 1.f);
    return make_float3(c.x / c.w, c.y / c.w, c.z / c.w);
}

// gl_FragDepth written into a depth target cleared to 1.0 with GL_LESS
__device__ inline float depth_store(float v)
{
    if (v != v) return 1.f;
    return fminf(fmaxf(v, 0.f), 1.f);
}

// ssf_blur.frag:44-139: 8 taps along s and 8 along t (the centre twice), each
// texture(tex, (s, t)) of a one-channel float texture with GL_LINEAR and
// GL_CLAMP_TO_EDGE (filter weights of 8 fractional bits, as in the texture
// unit, so a fetch at a texel centre returns the texel itself),
// spatial weight exp(-x^2 r) and the range term as written.  exp(-x^2 r)
// depends on |x| only, so its five values are computed once; the range
// weight is exp(-0) = 1 where the shader's r2 is 0.
__global__ void __launch_bounds__(256) k_ssf_blur(const float *in, float *out, Frame f)
{
    after_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= f.w || j >= f.h) return;
    // the centre tap: at a texel centre the 8-bit filter weights round to 0
    // and 1 (sides up to 8192), so the filtered value is the texel itself
    // (__ldca: loads as plain ones, see after_previous, in the order written;
    // as plain ones they are grouped by the compiler, and a frame of 12,000
    // particles at 1920 x 1080 takes 130 us, not 126)
    const float ed = __ldca(in + (size_t)j * f.w + i);
    if (ed == 1.f) {
        out[(size_t)j * f.w + i] = 1.f;
        return;
    }
    const float s = ((float)i + 0.5f) * f.inv_w, t = ((float)j + 0.5f) * f.inv_h;
    const float lin = linearize(ed, f);
    const float3 p = uv_to_eye(f, s, t, ed, true);
    const float dist = sqrtf(dot3(p.x, p.y, p.z, p.x, p.y, p.z));
    const float br = f.blur_radius * f.blur_scale / dist;
    float wk[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) wk[k] = expf(-((float)(k * k) * br));
    float sum = 0.f, wsum = 0.f;
#pragma unroll
    for (int axis = 0; axis < 2; ++axis) {
        // The axis's 8 taps move along it alone: across it the filter weight
        // is 0 or 1 (as for the centre tap), so each is a blend of two texels
        // of one line, and the axis's texels are requested before the first
        // is used: one tap at a time, each waiting for its texels, a pass
        // over a 1280 x 720 frame took 15.8 us, so 12.1; 11.5 with the centre tap,
        // which is the texel itself, taken as such.  Issue-bound from there (66%
        // issue-active; all 32 texels at once are no faster).
        const uint32_t N = axis == 0 ? f.w : f.h, M = axis == 0 ? f.h : f.w;
        const float at = axis == 0 ? s : t, v = (axis == 0 ? t : s) * (float)M - 0.5f, fv = floorf(v);
        const int line = min(max(clamp_pix(fv, M) + (rintf((v - fv) * 256.f) != 0.f ? 1 : 0), 0), (int)M - 1);
        const float *base = axis == 0 ? in + (size_t)line * f.w : in + line;
        const size_t step = axis == 0 ? 1 : f.w;
        float a[8], t0[8], t1[8];
        auto texels = [&](auto inside) {
#pragma unroll
            for (int k = -4; k < 4; ++k) {
                if (k == 0) continue;
                const float u = (at + (float)k * br) * (float)N - 0.5f, fu = floorf(u);
                a[k + 4] = rintf((u - fu) * 256.f) * (1.f / 256.f);
                if (decltype(inside)::value) {
                    const float *t = base + (uint32_t)fu * step;
                    t0[k + 4] = __ldca(t);
                    t1[k + 4] = __ldca(t + step);
                } else {
                    const int iu = clamp_pix(fu, N);
                    const int i0 = min(max(iu, 0), (int)N - 1), i1 = min(max(iu + 1, 0), (int)N - 1);
                    t0[k + 4] = __ldca(base + i0 * step);
                    t1[k + 4] = __ldca(base + i1 * step);  // weight 0: adds +0
                }
            }
        };
        // with a spacing br of at least 0 a tap's coordinate grows with k (each
        // rounding keeps the order), so the first and the last one tell whether
        // all texels are inside; most pixels' are, and need no clamps and one
        // address a tap: a frame at 1600 x 900 110 -> 105 us, at 1920 x 1080 193 ->
        // 188, no change at 1280 x 720.  A negative spacing (its sign is the
        // product's of two parameters) or NaN takes the clamps.
        if (br >= 0.f && (at + -4.f * br) * (float)N - 0.5f >= 0.f &&
            (at + 3.f * br) * (float)N - 0.5f < (float)(N - 1u))
            texels(std::true_type());
        else
            texels(std::false_type());
#pragma unroll
        for (int k = -4; k < 4; ++k) {
            if (k == 0) {  // the pixel itself: weights exp(-0) = 1
                sum = sum + lin;
                wsum = wsum + 1.f;
                continue;
            }
            const float a1 = 1.f - a[k + 4];
            const float sd = a1 * t0[k + 4] + a[k + 4] * t1[k + 4];
            if (sd != 1.f) {
                const float sl = linearize(sd, f);
                const float w = wk[k < 0 ? -k : k];
                const float diff = sl - lin;
                const float r2 = fabsf(diff) < 0.01f ? diff * 100.f : 0.f;
                const float g = r2 != 0.f ? expf(-r2 * r2) : 1.f;
                sum = sum + sl * w * g;
                wsum = wsum + w * g;
            }
        }
    }
    if (wsum > 0.f) sum = sum / wsum;
    out[(size_t)j * f.w + i] = depth_store(exponentialize(sum, f));
}

__device__ inline float3 eye_at(const Frame &f, const float *D, int i, int j)
{
    const int ic = min(max(i, 0), (int)f.w - 1), jc = min(max(j, 0), (int)f.h - 1);
    const float s = ((float)i + 0.5f) * f.inv_w, t = ((float)j + 0.5f) * f.inv_h;
    return uv_to_eye(f, s, t, D[(size_t)jc * f.w + ic], false);
}

// ssf_normal.frag:25-36: normalize(cross(dFdx(p), dFdy(p))) with fine
// derivatives of the 2x2 pixel quad; a quad partner on the empty side (or
// past an odd edge) still supplies its position, as a helper invocation does.
__global__ void __launch_bounds__(256) k_ssf_normal(const float *D, float4 *N, Frame f)
{
    after_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= f.w || j >= f.h) return;
    const size_t o = (size_t)j * f.w + i;
    if (D[o] == 1.f) {  // discard: the target keeps its clear colour
        N[o] = make_float4(f.clear[0], f.clear[1], f.clear[2], f.clear[3]);
        return;
    }
    const int ie = (int)(i & ~1u), je = (int)(j & ~1u);
    const float3 px0 = eye_at(f, D, ie, (int)j), px1 = eye_at(f, D, ie + 1, (int)j);
    const float3 py0 = eye_at(f, D, (int)i, je), py1 = eye_at(f, D, (int)i, je + 1);
    const float dxx = px1.x - px0.x, dxy = px1.y - px0.y, dxz = px1.z - px0.z;
    const float dyx = py1.x - py0.x, dyy = py1.y - py0.y, dyz = py1.z - py0.z;
    const float cx = dxy * dyz - dyy * dxz, cy = dxz * dyx - dyz * dxx, cz = dxx * dyy - dyx * dxy;
    const float inv = 1.f / sqrtf(dot3(cx, cy, cz, cx, cy, cz));
    N[o] = make_float4(cx * inv, cy * inv, cz * inv, 1.f);
}

__device__ inline float clamp01(float v) { return fminf(fmaxf(v, 0.f), 1.f); }

// ssf_shading.frag:36-83, blended (SRC_ALPHA, ONE_MINUS_SRC_ALPHA) onto the
// cleared 8-bit framebuffer (main.cpp:541-564): source and factors clamp to
// [0, 1] first, as for a fixed-point colour buffer.
__global__ void __launch_bounds__(256) k_ssf_shade(const float *D, const float4 *N, float4 *C, uchar4 *C8, Frame f)
{
    after_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= f.w || j >= f.h) return;
    const size_t o = (size_t)j * f.w + i;
    const float ed = D[o];
    if (ed == 1.f) {  // most pixels: the clear colour, its 8-bit form from the host
        C[o] = make_float4(f.clear[0], f.clear[1], f.clear[2], f.clear[3]);
        C8[o] = make_uchar4(f.clear8 & 255u, f.clear8 >> 8 & 255u, f.clear8 >> 16 & 255u, f.clear8 >> 24);
        return;
    }
    float4 out;
    {
        const float4 n = N[o];
        const float th = clamp01(f.thickness);
        const float s = ((float)i + 0.5f) * f.inv_w, t = ((float)j + 0.5f) * f.inv_h;
        const float3 p = uv_to_eye(f, s, t, ed, true);
        const float il = f.incident[0], jl = f.incident[1], kl = f.incident[2];
        const float vr = 1.f / sqrtf(dot3(-p.x, -p.y, -p.z, -p.x, -p.y, -p.z));
        const float vx = -p.x * vr, vy = -p.y * vr, vz = -p.z * vr;
        const float hx = il + vx, hy = jl + vy, hz = kl + vz;
        const float hr = 1.f / sqrtf(dot3(hx, hy, hz, hx, hy, hz));
        const float specular = powf(fmaxf(0.f, dot3(hx * hr, hy * hr, hz * hr, n.x, n.y, n.z)), 50.f);
        const float diffuse = fmaxf(0.f, dot3(il, jl, kl, n.x, n.y, n.z));
        const float r0 = 0.3f;
        const float fres = r0 + (1.f - r0) * powf(1.f - dot3(n.x, n.y, n.z, vx, vy, vz), 5.f);
        const float ar = expf(-5.f * th), ag = expf(-1.f * th), ab = expf(-0.1f * th);
        const float a = th;
        const float ia = 1.f - a;
        out.x = clamp01(clamp01(ar * diffuse + specular * 1.f + 1.f * fres) * a + f.clear[0] * ia);
        out.y = clamp01(clamp01(ag * diffuse + specular * 1.f + 1.f * fres) * a + f.clear[1] * ia);
        out.z = clamp01(clamp01(ab * diffuse + specular * 1.f + 1.f * fres) * a + f.clear[2] * ia);
        out.w = clamp01(a * a + f.clear[3] * ia);
    }
    C[o] = out;
    C8[o] = make_uchar4((unsigned char)rintf(clamp01(out.x) * 255.f), (unsigned char)rintf(clamp01(out.y) * 255.f),
                        (unsigned char)rintf(clamp01(out.z) * 255.f), (unsigned char)rintf(clamp01(out.w) * 255.f));
}

// ------------------------------------------------------------------ host --

bool inverse4(const float *m, float *out)
{
    // Gauss-Jordan with partial pivoting in double, rounded once to float
    double a[4][8];
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) {
            a[r][c] = m[c * 4 + r];
            a[r][c + 4] = r == c ? 1.0 : 0.0;
        }
    for (int c = 0; c < 4; ++c) {
        int piv = c;
        for (int r = c + 1; r < 4; ++r)
            if (std::fabs(a[r][c]) > std::fabs(a[piv][c])) piv = r;
        if (a[piv][c] == 0.0 || !std::isfinite(a[piv][c])) return false;
        if (piv != c)
            for (int k = 0; k < 8; ++k) std::swap(a[c][k], a[piv][k]);
        const double d = a[c][c];
        for (int k = 0; k < 8; ++k) a[c][k] /= d;
        for (int r = 0; r < 4; ++r) {
            if (r == c) continue;
            const double g = a[r][c];
            for (int k = 0; k < 8; ++k) a[r][k] -= g * a[c][k];
        }
    }
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) out[c * 4 + r] = (float)a[r][c + 4];
    return true;
}

}  // namespace
}  // namespace pbf103

using namespace pbf103;

struct pbf_ssf_renderer {
    int device = 0;
    int sms = 0;
    pbf_ssf_params p{};
    Frame f{};
    uint32_t *depth = nullptr;
    float *blur[2] = {nullptr, nullptr};
    float4 *normal = nullptr, *color = nullptr;
    uchar4 *rgba8 = nullptr;
    const float *blurred = nullptr, *blur_input = nullptr;
    SplatRec *rec = nullptr;   // per-particle splat records, grown to the largest particle bound seen
    uint32_t rec_cap = 0;
    uint32_t launches = 0;
};

namespace {

inline cudaStream_t S(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// glm::normalize: x * inversesqrt(dot(x, x)), inversesqrt = 1 / sqrt
void normalize3(float v[3])
{
    const float inv = 1.f / std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    v[0] = v[0] * inv;
    v[1] = v[1] * inv;
    v[2] = v[2] * inv;
}

void cross3(const float a[3], const float b[3], float out[3])
{
    out[0] = a[1] * b[2] - b[1] * a[2];
    out[1] = a[2] * b[0] - b[2] * a[0];
    out[2] = a[0] * b[1] - b[0] * a[1];
}

// Pixels between which the screen passes' blocks take 32 x 8 pixels, not
// 32 x 4: mostly empty frames are bound by their blocks' start, covered ones by
// the pixels' arithmetic.  A frame of one particle and of 32,768 in us, by 4
// rows and by 8: 1280 x 720 35 and 64, 33 and 64; 1600 x 900 45 and 81, 39 and
// 81; 1920 x 1080 58 and 105, 48 and 104; 3840 x 2160 197 and 341, 170 and 332;
// 4096 x 2400 229 and 399, 202 and 393; 5120 x 2880 353 and 604, 350 and 615.
constexpr uint32_t kTallFrom = 1500000, kTallTo = 10000000;

// 8 x 4 pixel tiles of the image (their depth bounds follow the depth image)
inline uint32_t tiles(const Frame &f) { return ((f.w + 7u) / 8u) * ((f.h + 3u) / 4u); }

pbf_status launch_frame(pbf_ssf_renderer *r, const float *x, int stride, const uint32_t *n_dev, uint32_t n,
                        uint32_t n_upper, cudaStream_t st)
{
    CK(cudaSetDevice(r->device));
    const Frame &f = r->f;
    const uint32_t px = f.w * f.h;
    uint32_t launches = 0;
    // Every launch but the first is set up while the one before runs
    // (launch_after): 20,000 particles at 640 x 360 45 -> 31 us, 32,768 at 1280 x 720
    // 79 -> 63, 524,288 at 1920 x 1080 188 -> 175.
    // the depth image and the tile bounds after it
    k_ssf_fill<<<std::min<uint32_t>((px + 255) / 256, (uint32_t)r->sms * 8), 256, 0, st>>>(r->depth, kEmptyDepth,
                                                                                           px + tiles(f));
    ++launches;
    if (n_upper) {
        if (n_upper > r->rec_cap) {
            // the only allocation on the frame path: the first frame of a
            // larger particle bound (cudaFree waits for frames in flight)
            CK(cudaFree(r->rec));
            r->rec = nullptr;
            r->rec_cap = 0;
            CK(cudaMalloc(&r->rec, sizeof(SplatRec) * (size_t)n_upper));
            r->rec_cap = n_upper;
        }
        const uint32_t sblocks = std::min<uint32_t>((n_upper + 255) / 256, (uint32_t)r->sms * 8);
        if (stride == 4)
            launch_after(k_ssf_setup<4>, sblocks, 256, st, x, n_dev, n, f, r->rec);
        else
            launch_after(k_ssf_setup<3>, sblocks, 256, st, x, n_dev, n, f, r->rec);
        // a warp per particle while they fit the device at once; larger sets
        // by tiles take half the warps, so that fewer far particles start
        // before the near ones' depths are in place
        const uint32_t want = (n_upper + 7) / 8, most = (uint32_t)r->sms * 8;
        if (n_upper <= kBoxRaster || px <= kBoxPixels || (px <= kBoxPixelsFew && n_upper <= kBoxFew))
            launch_after(k_ssf_raster_box, std::min(want, most), 256, st, r->rec, n_dev, n, f, r->depth);
        else
            launch_after(k_ssf_raster, want <= most ? want : most / 2, 256, st, r->rec, n_dev, n, f, r->depth,
                         r->depth + px);
        launches += 2;
    }
    const uint32_t rows = px >= kTallFrom && px <= kTallTo ? 8u : 4u;
    const dim3 blk(32, rows), grd((f.w + 31) / 32, (f.h + rows - 1) / rows);
    const float *src = reinterpret_cast<const float *>(r->depth), *prev = src;
    for (uint32_t k = 0; k < r->p.blur_passes; ++k) {
        float *dst = r->blur[k & 1];  // even, odd, even ... (main.cpp:430-509)
        launch_after(k_ssf_blur, grd, blk, st, src, dst, f);
        ++launches;
        prev = src;
        src = dst;
    }
    launch_after(k_ssf_normal, grd, blk, st, src, r->normal, f);
    launch_after(k_ssf_shade, grd, blk, st, reinterpret_cast<const float *>(r->depth), r->normal, r->color, r->rgba8, f);
    launches += 2;
    CK(cudaGetLastError());
    r->blurred = src;
    r->blur_input = prev;
    r->launches = launches;
    return PBF_SUCCESS;
}

pbf_status image(pbf_ssf_renderer *r, int which, void **ptr, uint64_t *bytes)
{
    const uint64_t px = (uint64_t)r->f.w * r->f.h;
    switch (which) {
    case PBF_SSF_DEPTH: *ptr = r->depth; *bytes = 4 * px; break;
    case PBF_SSF_BLURRED: *ptr = const_cast<float *>(r->blurred); *bytes = 4 * px; break;
    case PBF_SSF_BLUR_INPUT: *ptr = const_cast<float *>(r->blur_input); *bytes = 4 * px; break;
    case PBF_SSF_NORMAL: *ptr = r->normal; *bytes = 16 * px; break;
    case PBF_SSF_COLOR: *ptr = r->color; *bytes = 16 * px; break;
    case PBF_SSF_RGBA8: *ptr = r->rgba8; *bytes = 4 * px; break;
    default: return PBF_ERROR_INVALID_ARGUMENT;
    }
    return PBF_SUCCESS;
}

void free_renderer(pbf_ssf_renderer *r)
{
    cudaSetDevice(r->device);
    cudaFree(r->depth);
    cudaFree(r->blur[0]);
    cudaFree(r->blur[1]);
    cudaFree(r->normal);
    cudaFree(r->color);
    cudaFree(r->rgba8);
    cudaFree(r->rec);
    delete r;
}

}  // namespace

extern "C" {

pbf_status pbf_ssf_params_init(pbf_ssf_params *p)
{
    if (!p) return PBF_ERROR_INVALID_ARGUMENT;
    std::memset(p, 0, sizeof(*p));
    p->width = 1280;
    p->height = 720;
    // src/common/controls.cpp:12-26 (initial state) and :66-110 (matrices)
    const float pi = 3.14159265358979323846f;
    const float h_ang = pi, v_ang = pi * -0.1f;
    const float znear = 0.1f, zfar = 50.f;
    const float dir[3] = {std::cos(v_ang) * std::sin(h_ang), std::sin(v_ang), std::cos(v_ang) * std::cos(h_ang)};
    const float right[3] = {std::sin(h_ang - 3.14f / 2.0f), 0.f, std::cos(h_ang - 3.14f / 2.0f)};
    float up[3];
    cross3(right, dir, up);
    // glm::perspective(45.0f, 4/3, near, far), fovy in radians
    const float fovy = 45.0f, aspect = 4.0f / 3.0f;
    const float tan_half = std::tan(fovy / 2.0f);
    float *P = p->projection;
    P[0] = 1.0f / (aspect * tan_half);
    P[5] = 1.0f / tan_half;
    P[10] = -(zfar + znear) / (zfar - znear);
    P[11] = -1.0f;
    P[14] = -(2.0f * zfar * znear) / (zfar - znear);
    // glm::lookAt(eye, eye + direction, up)
    const float eye[3] = {2.0f, 4.0f, 10.0f};
    const float center[3] = {eye[0] + dir[0], eye[1] + dir[1], eye[2] + dir[2]};
    float fw[3] = {center[0] - eye[0], center[1] - eye[1], center[2] - eye[2]};
    normalize3(fw);
    float sd[3];
    cross3(fw, up, sd);
    normalize3(sd);
    float u[3];
    cross3(sd, fw, u);
    float *V = p->view;
    V[0] = sd[0];
    V[4] = sd[1];
    V[8] = sd[2];
    V[1] = u[0];
    V[5] = u[1];
    V[9] = u[2];
    V[2] = -fw[0];
    V[6] = -fw[1];
    V[10] = -fw[2];
    V[12] = -(sd[0] * eye[0] + sd[1] * eye[1] + sd[2] * eye[2]);
    V[13] = -(u[0] * eye[0] + u[1] * eye[1] + u[2] * eye[2]);
    V[14] = fw[0] * eye[0] + fw[1] * eye[1] + fw[2] * eye[2];
    V[15] = 1.0f;
    p->point_radius = 0.18f;
    p->point_scale = P[5] * ((float)p->height * 0.5f);
    p->near_plane = znear;
    p->far_plane = zfar;
    p->blur_radius = 0.0000055f;
    p->blur_scale = (float)p->height / std::tan(45.f * 0.5f * 3.1415f / 180.f);
    p->blur_passes = 3;
    p->splat_mode = PBF_SSF_SPLAT_QUAD;
    p->thickness = 0.6f;
    p->clear_color[0] = p->clear_color[1] = p->clear_color[2] = 0.6f;
    p->clear_color[3] = 1.f;
    return PBF_SUCCESS;
}

pbf_status pbf_ssf_create(int device, const pbf_ssf_params *p, pbf_ssf_renderer **out)
{
    if (!p || !out) return PBF_ERROR_INVALID_ARGUMENT;
    *out = nullptr;
    if (p->width < 1 || p->height < 1 || p->width > kMaxSide || p->height > kMaxSide) return PBF_ERROR_BAD_PARAMETER;
    if (p->splat_mode > PBF_SSF_SPLAT_SPRITE || p->blur_passes > 64) return PBF_ERROR_BAD_PARAMETER;
    for (int k = 0; k < 16; ++k)
        if (!std::isfinite(p->projection[k]) || !std::isfinite(p->view[k])) return PBF_ERROR_BAD_PARAMETER;
    const float *P = p->projection;
    // x_clip on (x, z, w), y_clip on (y, z, w), z_clip and w_clip on (z, w)
    if (P[4] != 0.f || P[1] != 0.f || P[2] != 0.f || P[6] != 0.f || P[3] != 0.f || P[7] != 0.f)
        return PBF_ERROR_BAD_PARAMETER;
    if (!(p->point_radius > 0.f) || !(p->near_plane > 0.f) || !(p->far_plane > p->near_plane) ||
        !std::isfinite(p->far_plane) || !std::isfinite(p->blur_radius) || !std::isfinite(p->blur_scale) ||
        !std::isfinite(p->point_scale) || !std::isfinite(p->thickness))
        return PBF_ERROR_BAD_PARAMETER;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return PBF_ERROR_NO_DEVICE;
    if (device < 0 || device >= ndev) return PBF_ERROR_INVALID_ARGUMENT;
    pbf_ssf_renderer *r = new (std::nothrow) pbf_ssf_renderer;
    if (!r) return PBF_ERROR_OUT_OF_MEMORY;
    r->device = device;
    r->p = *p;
    Frame &f = r->f;
    f.w = p->width;
    f.h = p->height;
    f.mode = p->splat_mode;
    std::memcpy(f.proj, p->projection, sizeof f.proj);
    std::memcpy(f.view, p->view, sizeof f.view);
    if (!inverse4(f.proj, f.inv_proj)) {
        delete r;
        return PBF_ERROR_BAD_PARAMETER;
    }
    f.radius = p->point_radius;
    f.point_scale = p->point_scale;
    f.znear = p->near_plane;
    f.zfar = p->far_plane;
    f.blur_radius = p->blur_radius;
    f.blur_scale = p->blur_scale;
    f.thickness = p->thickness;
    std::memcpy(f.clear, p->clear_color, sizeof f.clear);
    for (int k = 0; k < 4; ++k)
        f.clear8 |= (uint32_t)std::nearbyint(std::fmin(std::fmax(f.clear[k], 0.f), 1.f) * 255.f) << (8 * k);
    f.inv_w = 1.f / (float)f.w;
    f.inv_h = 1.f / (float)f.h;
    // lightDir = View * World * vec4(1, 4, 1, 0) (ssf_shading.frag:39), normalised once
    const float4 l = mat_vec(f.view, 1.f, 4.f, 1.f, 0.f);
    float inc[3] = {l.x, l.y, l.z};
    normalize3(inc);
    std::memcpy(f.incident, inc, sizeof inc);
    const size_t px = (size_t)f.w * f.h;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaMalloc(&r->depth, 4 * (px + tiles(f)));
    if (e == cudaSuccess) e = cudaMalloc(&r->blur[0], 4 * px);
    if (e == cudaSuccess) e = cudaMalloc(&r->blur[1], 4 * px);
    if (e == cudaSuccess) e = cudaMalloc(&r->normal, 16 * px);
    if (e == cudaSuccess) e = cudaMalloc(&r->color, 16 * px);
    if (e == cudaSuccess) e = cudaMalloc(&r->rgba8, 4 * px);
    if (e != cudaSuccess) {
        set_last_error("pbf_ssf_create", e);
        free_renderer(r);
        return e == cudaErrorMemoryAllocation ? PBF_ERROR_OUT_OF_MEMORY : PBF_ERROR_CUDA;
    }
    r->blurred = r->blur_input = reinterpret_cast<const float *>(r->depth);
    *out = r;
    return PBF_SUCCESS;
}

pbf_status pbf_ssf_destroy(pbf_ssf_renderer *r)
{
    if (!r) return PBF_ERROR_INVALID_ARGUMENT;
    free_renderer(r);
    return PBF_SUCCESS;
}

pbf_status pbf_ssf_render(pbf_ssf_renderer *r, const float *x_dev, uint32_t n, void *st)
{
    if (!r || (n && !x_dev)) return PBF_ERROR_INVALID_ARGUMENT;
    return launch_frame(r, x_dev, 3, nullptr, n, n, S(st));
}

pbf_status pbf_ssf_render_scene(pbf_ssf_renderer *r, pbf_batch *b, uint32_t scene_id, void *st)
{
    if (!r || !b) return PBF_ERROR_INVALID_ARGUMENT;
    Batch::SceneArrays A;
    pbf_status rc = b->b.scene_arrays(scene_id, &A);
    if (rc != PBF_SUCCESS) return rc;
    if (b->b.device() != r->device) return PBF_ERROR_INVALID_ARGUMENT;
    return launch_frame(r, reinterpret_cast<const float *>(A.x), 4, A.scene_num, 0, A.capacity, S(st));
}

pbf_status pbf_ssf_render_particles(pbf_ssf_renderer *r, pbf_handle *h, void *st)
{
    if (!r || !h) return PBF_ERROR_INVALID_ARGUMENT;
    Batch::SceneArrays A;
    pbf_status rc = h->b.scene_arrays(h->scene, &A);
    if (rc != PBF_SUCCESS) return rc;
    if (h->b.device() != r->device) return PBF_ERROR_INVALID_ARGUMENT;
    return launch_frame(r, reinterpret_cast<const float *>(A.x), 4, A.scene_num, 0, A.capacity, S(st));
}

pbf_status pbf_ssf_image_device(pbf_ssf_renderer *r, int which, void **ptr, uint64_t *bytes)
{
    if (!r || !ptr || !bytes) return PBF_ERROR_INVALID_ARGUMENT;
    return image(r, which, ptr, bytes);
}

pbf_status pbf_ssf_get_image(pbf_ssf_renderer *r, int which, void *dst, int dst_dev, void *st)
{
    if (!r || !dst) return PBF_ERROR_INVALID_ARGUMENT;
    void *src = nullptr;
    uint64_t bytes = 0;
    pbf_status rc = image(r, which, &src, &bytes);
    if (rc != PBF_SUCCESS) return rc;
    CK(cudaSetDevice(r->device));
    CK(cudaMemcpyAsync(dst, src, bytes, dst_dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, S(st)));
    if (!dst_dev) CK(cudaStreamSynchronize(S(st)));
    return PBF_SUCCESS;
}

pbf_status pbf_ssf_frame_constants(const pbf_ssf_renderer *r, float inv_projection[16], float incident[3])
{
    if (!r) return PBF_ERROR_INVALID_ARGUMENT;
    if (inv_projection) std::memcpy(inv_projection, r->f.inv_proj, sizeof r->f.inv_proj);
    if (incident) std::memcpy(incident, r->f.incident, sizeof r->f.incident);
    return PBF_SUCCESS;
}

pbf_status pbf_ssf_last_launches(const pbf_ssf_renderer *r, uint32_t *n)
{
    if (!r || !n) return PBF_ERROR_INVALID_ARGUMENT;
    *n = r->launches;
    return PBF_SUCCESS;
}

}  // extern "C"
