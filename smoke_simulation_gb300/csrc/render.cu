// Headless half-angle slice renderer (smk_render): the reference's two-pass volume drawing
// restated as two CUDA kernels.
//
// The reference (project/main.cpp:369-419, 474-476) draws proxy plane i into the eye buffer
// using the light buffer as it stands after planes 0..i-1, then draws the same plane into the
// light buffer.  The light buffer after plane k therefore only depends on the light's own rays,
// so it is computed for every plane first, in parallel over light texels (k_render_light: each
// texel marches the planes and stores its colour after each one; its alpha is read by nothing), and the eye buffer is then
// computed in parallel over pixels (k_render_eye: each pixel marches the planes in drawing
// order, reading the light buffer of the previous plane).  Two launches per frame, no
// dependence between pixels.
//
// Instruction issue bounds both marches (80 and 68 % of the issue slots; a sample takes some 130
// instructions of the light's march, 300 of the eye's), so a ray visits only the planes it can meet in the
// box (plane_range), divides by remainder steps, clamps an index with one instruction, reads a texel's
// colour with one load and packs its arithmetic in pairs; a warp covers 8 x 4 pixels and 40 registers
// keep six blocks an SM.  80^3, 1280 x 720, 100 planes, 512 x 512 light texels: 541 us a frame with every
// plane visited and scalar loads and divisions, 347 with the plane range, wide texels and the plane table,
// 203 now (light 55, of which the 210 MB of slices take 31 at the copy rate; eye 145).
//
// Per fragment (texVolume.frag:27-52, light.frag:16-23): the plane point is where the pixel's
// ray meets the plane (what rasterising the plane-box polygon and interpolating its world
// position yields), kept when it lies in the box and between the near and far planes; density
// from the 3D texture (linear filtering, clamp to edge, texel centres at (i + 0.5) / n, the
// shader's coordinate ((p - box) / (n / 2) + 1) / 2 with integer n / 2); the light colour from
// the light buffer at the point's light-projected position (linear filtering, repeat: the
// framebuffer texture's default wrap).  Eye colour = light colour, alpha = density; front-to-back
// premultiplies and blends (ONE_MINUS_DST_ALPHA, ONE), back-to-front blends (SRC_ALPHA,
// ONE_MINUS_SRC_ALPHA) with alpha (ONE, ONE_MINUS_SRC_ALPHA); the light buffer blends (0,0,0,d)
// with (SRC_ALPHA, ONE_MINUS_SRC_ALPHA) / (ONE, ONE_MINUS_SRC_ALPHA).  Every stored value is
// rounded to half precision (RGBA16F framebuffers, labhelper/fbo.cpp:46).  Weights are float
// (the GL texture unit's fixed-point weights are not reproduced).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <string>

#include "../../include/smoke_gb300.h"
#include "common.cuh"
#include "sim_internal.h"

namespace smk {

namespace {

struct V3 {
    float x, y, z;
};
__host__ __device__ inline V3 mk(float x, float y, float z) { return V3{x, y, z}; }
__host__ __device__ inline V3 operator+(V3 a, V3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__host__ __device__ inline V3 operator-(V3 a, V3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__host__ __device__ inline V3 operator*(V3 a, float s) { return mk(a.x * s, a.y * s, a.z * s); }
__host__ __device__ inline float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__host__ __device__ inline V3 cross3(V3 a, V3 b) {
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
inline V3 norm3(V3 a) { return a * (1.0f / sqrtf(dot3(a, a))); }

// A perspective view (the camera or the light): origin, orthonormal basis as lookAt builds it,
// and the NDC scales (aspect * tan(fovy / 2), tan(fovy / 2)).
struct ViewSetup {
    V3 eye, s, u, f;
    float sx, sy, znear, zfar;
    int w, h;
};

struct Setup {
    ViewSetup cam, light;
    V3 start, end, n;  // planes: start + (end - start) * (i + 0.5) / planes, normal n
    int planes;
    int back_to_front;
    V3 box_min, box_max, box_pos, tex_half, tex_inv;  // tex_inv = 1 / tex_half
    V3 half_n;                                        // half the cells of each axis
    float one;  // 1
    float clear[3];  // the light buffer's clear colour (half-rounded)
    float bg[3];
};

ViewSetup make_view(V3 eye, V3 dir, V3 up, float fovy_deg, float aspect, float zn, float zf, int w, int h) {
    ViewSetup v;
    v.eye = eye;
    v.f = norm3(dir);
    v.s = norm3(cross3(v.f, up));
    v.u = cross3(v.s, v.f);
    const float th = (float)tan(0.5 * (double)fovy_deg * 3.14159265358979323846 / 180.0);
    v.sx = aspect * th;
    v.sy = th;
    v.znear = zn;
    v.zfar = zf;
    v.w = w;
    v.h = h;
    return v;
}

// Round-to-nearest-even to half precision and back (the value an RGBA16F texel holds), two at a time.
__device__ __forceinline__ void h16(float x, float y, float* a, float* b) {
    const float2 r = __half22float2(__floats2half2_rn(x, y));
    *a = r.x;
    *b = r.y;
}

// moderate: every length in the setup lies where quot() is exact (the kernels' EXACT form).
Setup make_setup(const smk_render_params& rp, int nx, int ny, int nz, bool* moderate) {
    Setup S;
    const V3 cam = mk(rp.camera_pos[0], rp.camera_pos[1], rp.camera_pos[2]);
    const V3 up = mk(rp.up[0], rp.up[1], rp.up[2]);
    const V3 lp = mk(rp.light_pos[0], rp.light_pos[1], rp.light_pos[2]);
    const V3 box = mk(rp.box_pos[0], rp.box_pos[1], rp.box_pos[2]);
    S.cam = make_view(cam, mk(rp.camera_dir[0], rp.camera_dir[1], rp.camera_dir[2]), up, rp.fovy_deg,
                      (float)rp.width / (float)rp.height, rp.znear, rp.zfar, rp.width, rp.height);
    S.light = make_view(lp, box - lp, up, rp.light_fovy_deg, 1.0f, rp.light_znear, rp.light_zfar, rp.light_res,
                        rp.light_res);
    // half vector and drawing order (main.cpp:660-661, 676-687)
    const V3 cam_view = box - cam, light_view = box - lp;
    const V3 cn = norm3(cam_view), ln = norm3(light_view);
    V3 half = cn + ln;
    if (dot3(cn, ln) < 0.0f) half = mk(-cn.x, -cn.y, -cn.z) + ln;
    S.back_to_front = dot3(cam_view, light_view) < 0.0f ? 1 : 0;
    // planes between the box corners' extreme projections on the half vector, measured from the
    // world origin with the corners at +-dimensions / 2 (boundingBox.cpp:135-181)
    const V3 dims = mk(rp.cell_size * nx, rp.cell_size * ny, rp.cell_size * nz);
    const V3 hd = dims * 0.5f;
    S.n = norm3(half);
    float mn = 0.0f, mx = 0.0f;
    for (int c = 0; c < 8; ++c) {
        const V3 corner = mk((c & 1) ? hd.x : -hd.x, (c & 2) ? hd.y : -hd.y, (c & 4) ? hd.z : -hd.z);
        const float d = dot3(corner, S.n);
        if (c == 0 || d < mn) mn = d;
        if (c == 0 || d > mx) mx = d;
    }
    S.start = S.n * mn;
    S.end = S.n * mx;
    S.planes = rp.planes;
    S.box_pos = box;
    S.box_min = box - hd;
    S.box_max = box + hd;
    S.tex_half = mk((float)(nx / 2), (float)(ny / 2), (float)(nz / 2));
    S.tex_inv = mk(1.0f / S.tex_half.x, 1.0f / S.tex_half.y, 1.0f / S.tex_half.z);
    S.one = 1.0f;
    S.half_n = mk(0.5f * (float)nx, 0.5f * (float)ny, 0.5f * (float)nz);
    const float far = 1e9f;
    auto near_by = [&](V3 a) { return fabsf(a.x) < far && fabsf(a.y) < far && fabsf(a.z) < far; };
    *moderate = near_by(cam) && near_by(lp) && near_by(box) && near_by(dims) && S.cam.znear >= 1e-6f &&
                S.light.znear >= 1e-6f && S.cam.zfar <= 1e12f && S.light.zfar <= 1e12f;
    for (int k = 0; k < 3; ++k) {
        S.clear[k] = __half2float(__float2half_rn(rp.light_color[k]));
        S.bg[k] = rp.bg_color[k];
    }
    return S;
}

// a / b correctly rounded from y = 1 / b correctly rounded (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990): the first remainder step brings the quotient
// within one ulp, the second then rounds it correctly.  b stays away from the ends of the exponent range,
// and quotients so small that the remainder underflows do not count where this is used.  A march divides
// by the same number at every plane, and six divisions a sample were a third of its instructions.
__device__ __forceinline__ float quot(float a, float b, float y) {
    float q = a * y;
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
// The same for two quotients at once; nb = -b.
__device__ __forceinline__ float2 quot2(float2 a, float2 nb, float2 y) {
    float2 q = __fmul2_rn(a, y);
    q = __ffma2_rn(__ffma2_rn(nb, q, a), y, q);
    return __ffma2_rn(__ffma2_rn(nb, q, a), y, q);
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
// a (1 - w) + b w, each product rounded by itself: the sum is a product with S.one, which the compiler does
// not know, as it would contract a packed addition (or a product with a literal 1) with one of them.
__device__ __forceinline__ float2 mix2(const Setup& S, float2 a, float2 b, float ow, float w) {
    return __ffma2_rn(__fmul2_rn(a, both(ow)), both(S.one), __fmul2_rn(b, both(w)));
}
__device__ __forceinline__ bool quot_range(float b) { return fabsf(b) > 1e-12f && fabsf(b) < 1e12f; }

__device__ __forceinline__ bool inside(const Setup& S, V3 p) {
    return p.x >= S.box_min.x && p.x <= S.box_max.x && p.y >= S.box_min.y && p.y <= S.box_max.y &&
           p.z >= S.box_min.z && p.z <= S.box_max.z;
}

// The distance of plane i from view V along the planes' normal: the same for every ray, so a block
// computes it once for up to MAX_TABLE planes (a division and 15 other operations per ray and plane less);
// planes past the table compute it at each ray.
constexpr int MAX_TABLE = 2048;
__device__ __forceinline__ float plane_distance(const Setup& S, const ViewSetup& V, int i) {
    const float ti = ((float)i + 0.5f) / (float)S.planes;
    const V3 pp = S.start + (S.end - S.start) * ti;
    return dot3(pp - V.eye, S.n);
}
__device__ __forceinline__ void plane_table(const Setup& S, const ViewSetup& V, float* table) {
    for (int i = (int)threadIdx.x; i < S.planes && i < MAX_TABLE; i += (int)blockDim.x) table[i] = plane_distance(S, V, i);
    __syncthreads();
}

// A range [i0, i1] of planes outside of which the ray meets no plane inside the box: the ray's segment
// in the box grown by m, more than the rounding of a hit point (a few 1e-7 of the distances involved),
// and 1.5 planes more on each side for the rounding of a plane's index, which the guard on b bounds by
// half a plane.  Every plane where an estimate is not usable (planes too close together for FP32, NaN).
__device__ __forceinline__ void plane_range(const Setup& S, const ViewSetup& V, V3 d, float denom, int& i0, int& i1) {
    i0 = 0;
    i1 = S.planes - 1;
    const float ext = fmaxf(fmaxf(S.box_max.x - S.box_min.x, S.box_max.y - S.box_min.y), S.box_max.z - S.box_min.z);
    const float far = fmaxf(fmaxf(fabsf(V.eye.x), fabsf(V.eye.y)), fabsf(V.eye.z));
    const float at = fmaxf(fmaxf(fabsf(S.box_pos.x), fabsf(S.box_pos.y)), fabsf(S.box_pos.z));
    const float m = 1e-3f * ext + 1e-4f * (far + at);
    float lo = -3e38f, hi = 3e38f;
    const float dd[3] = {d.x, d.y, d.z}, ee[3] = {V.eye.x, V.eye.y, V.eye.z};
    const float mn[3] = {S.box_min.x, S.box_min.y, S.box_min.z}, mx[3] = {S.box_max.x, S.box_max.y, S.box_max.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (fabsf(dd[k]) < 1e-6f) continue;  // nearly parallel to the sides: no bound from this axis
        const float a = __fdividef(mn[k] - m - ee[k], dd[k]), b = __fdividef(mx[k] + m - ee[k], dd[k]);
        lo = fmaxf(lo, fminf(a, b));
        hi = fminf(hi, fmaxf(a, b));
    }
    // plane i is met at t = (a + b (i + 0.5) / planes) / denom
    const float a = dot3(S.start - V.eye, S.n), b = dot3(S.end - S.start, S.n);
    if (!(b > 4e-6f * (float)S.planes * (far + at + ext)) || !(fabsf(lo) < 1e30f) || !(fabsf(hi) < 1e30f)) return;
    if (lo > hi) {
        // the ray misses the grown box; what the estimate's own rounding could hide is far smaller than m
        i1 = -1;
        return;
    }
    const float scale = (float)S.planes / b;
    const float f = (lo * denom - a) * scale, g = (hi * denom - a) * scale;
    const float first = fminf(f, g) - 2.0f, last = fmaxf(f, g) + 1.0f;  // index = f - 0.5
    if (!(first > -1e9f && last < 1e9f)) return;
    i0 = max(i0, (int)floorf(first));
    i1 = min(i1, (int)ceilf(last));
}

// The point where the ray of pixel (px, py) of view V meets plane i (at distance dist), if it is drawn there.
// inv: 1 / denom, or 0 where quot() must not be used.
__device__ __forceinline__ bool plane_hit(const Setup& S, const ViewSetup& V, V3 d, float denom, float inv, float dist,
                                          V3* p) {
    if (denom == 0.0f) return false;
    const float t = inv != 0.0f ? quot(dist, denom, inv) : dist / denom;
    if (!(t >= V.znear && t <= V.zfar)) return false;
    *p = V.eye + d * t;
    return inside(S, *p);
}

__device__ __forceinline__ V3 ray_dir(const ViewSetup& V, int px, int py) {
    const float nx = (2.0f * ((float)px + 0.5f)) / (float)V.w - 1.0f;
    const float ny = (2.0f * ((float)py + 0.5f)) / (float)V.h - 1.0f;
    return (V.f + V.s * (nx * V.sx)) + V.u * (ny * V.sy);
}

// texture(gridTex, ((p - box) / (n / 2) + 1) / 2).r with linear filtering and clamp to edge
template <bool EXACT, typename T>
__device__ float sample_density(const Setup& S, const T* rho, const Grid& g, V3 p) {
    const V3 r = p - S.box_pos;
    V3 t;
    if (EXACT) {
        const float2 xy = quot2(make_float2(r.x, r.y), make_float2(-S.tex_half.x, -S.tex_half.y),
                                make_float2(S.tex_inv.x, S.tex_inv.y));
        t = mk(xy.x, xy.y, quot(r.z, S.tex_half.z, S.tex_inv.z));
    } else {
        t = mk(r.x / S.tex_half.x, r.y / S.tex_half.y, r.z / S.tex_half.z);
    }
    // ((t + 1) / 2) n: the halving is exact, so it goes into the factor
    const float ux = (t.x + 1.0f) * S.half_n.x - 0.5f, uy = (t.y + 1.0f) * S.half_n.y - 0.5f,
                uz = (t.z + 1.0f) * S.half_n.z - 0.5f;
    const float fx = floorf(ux), fy = floorf(uy), fz = floorf(uz);
    const float ax = ux - fx, ay = uy - fy, az = uz - fz;
    const int ix = (int)fx, iy = (int)fy, iz = (int)fz;  // clamped from both sides by one instruction each
    const int x0 = __vimin_s32_relu(ix, g.nx - 1), x1 = __viaddmin_s32_relu(ix, 1, g.nx - 1);
    const int y0 = __vimin_s32_relu(iy, g.ny - 1), y1 = __viaddmin_s32_relu(iy, 1, g.ny - 1);
    const int z0 = __vimin_s32_relu(iz, g.nz - 1), z1 = __viaddmin_s32_relu(iz, 1, g.nz - 1);
    const T* c = rho + g.idx(x0, y0, z0);
    const int dx = x1 - x0, dy = g.X * (y1 - y0), dz = g.XY * (z1 - z0);
    // lower and upper plane side by side in packed arithmetic
    const float2 v00 = make_float2(ldv(c, 0), ldv(c, dz)), v10 = make_float2(ldv(c, dx), ldv(c, dz + dx));
    const float2 v01 = make_float2(ldv(c, dy), ldv(c, dz + dy)), v11 = make_float2(ldv(c, dy + dx), ldv(c, dz + dy + dx));
    const float ox = 1.0f - ax;
    const float2 cz = mix2(S, mix2(S, v00, v10, ox, ax), mix2(S, v01, v11, ox, ax), 1.0f - ay, ay);
    return cz.x * (1.0f - az) + cz.y * az;
}

__device__ __forceinline__ int wrapi(int v, int n) {
    const int r = v % n;
    return r < 0 ? r + n : r;
}

// A texel's colour (its alpha is not read): one 8-byte load.
struct Colour {
    float2 rg;
    float b;
};
__device__ __forceinline__ Colour texel(const __half* t) {
    const uint2 r = *reinterpret_cast<const uint2*>(t);
    return Colour{__half22float2(*reinterpret_cast<const __half2*>(&r.x)),
                  __low2float(*reinterpret_cast<const __half2*>(&r.y))};
}

// texture(lightMap, uv).rgb of one plane's light buffer: linear filtering, repeat
__device__ Colour sample_light(const Setup& S, const __half* L, int R, float u, float v) {
    const float sx = fminf(fmaxf(u * (float)R - 0.5f, -1.0e6f), 1.0e6f);
    const float sy = fminf(fmaxf(v * (float)R - 0.5f, -1.0e6f), 1.0e6f);
    const float fx = floorf(sx), fy = floorf(sy);
    const float ax = sx - fx, ay = sy - fy;
    const int ix = (int)fx, iy = (int)fy;
    const __half *r0, *r1;  // texel x0 of both rows
    int dx = 4;             // from there to texel x1
    if ((unsigned)ix < (unsigned)(R - 1) && (unsigned)iy < (unsigned)(R - 1)) {
        r0 = L + 4 * (size_t)(ix + R * iy);
        r1 = r0 + 4 * R;
    } else {
        const int x0 = wrapi(ix, R), x1 = wrapi(ix + 1, R);
        r0 = L + 4 * (size_t)(x0 + R * wrapi(iy, R));
        r1 = L + 4 * (size_t)(x0 + R * wrapi(iy + 1, R));
        dx = 4 * (x1 - x0);
    }
    const Colour t00 = texel(r0), t10 = texel(r0 + dx), t01 = texel(r1), t11 = texel(r1 + dx);
    const float ox = 1.0f - ax, oy = 1.0f - ay;
    const float2 b = mix2(S, make_float2(t00.b, t01.b), make_float2(t10.b, t11.b), ox, ax);
    return Colour{mix2(S, mix2(S, t00.rg, t10.rg, ox, ax), mix2(S, t01.rg, t11.rg, ox, ax), oy, ay), b.x * oy + b.y * ay};
}

// The pixel of this thread: a block draws 16 x 16 pixels, a warp 8 x 4 of them, so that the texels and
// cells its rays gather at one plane lie close together.
__device__ __forceinline__ bool tile_pixel(int w, int h, int* px, int* py) {
    const int across = (w + 15) / 16, t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
    *px = ((int)blockIdx.x % across) * 16 + (warp & 1) * 8 + (lane & 7);
    *py = ((int)blockIdx.x / across) * 16 + (warp >> 1) * 4 + (lane >> 3);
    return *px < w && *py < h;
}
inline int tile_blocks(int w, int h) { return ((w + 15) / 16) * ((h + 15) / 16); }

// The light buffer after every plane: slices[i] = RGBA16F light buffer after drawing plane i.
template <typename T, bool EXACT>
__global__ void __launch_bounds__(256, 6) k_render_light(const Setup S, const T* __restrict__ rho, const Grid g, __half* __restrict__ slices,
                               int* __restrict__ any_odd) {
    __shared__ float table[MAX_TABLE];
    plane_table(S, S.light, table);
    const int R = S.light.w;
    int lx, ly;
    const bool mine = tile_pixel(R, R, &lx, &ly);
    const int id = lx + R * ly;
    const V3 d = ray_dir(S.light, lx, ly);
    const float denom = dot3(d, S.n);
    const float inv = EXACT && quot_range(denom) ? __frcp_rn(denom) : 0.0f;
    float c[3] = {S.clear[0], S.clear[1], S.clear[2]};
    const size_t plane_stride = (size_t)R * R * 4;
    int i0, i1;
    plane_range(S, S.light, d, denom, i0, i1);
    __half2 rg = __floats2half2_rn(c[0], c[1]), b1 = __floats2half2_rn(c[2], 1.0f);
    bool odd = false;  // a stored value with a sign, an infinity or a NaN
#pragma unroll
    for (int k = 0; k < 3; ++k) odd |= __float_as_uint(c[k]) >= 0x7f800000u;
    for (int i = 0; i < (mine ? S.planes : 0); ++i) {
        V3 p;
        if (i >= i0 && i <= i1 &&
            plane_hit(S, S.light, d, denom, inv, i < MAX_TABLE ? table[i] : plane_distance(S, S.light, i), &p)) {
            const float a = sample_density<EXACT>(S, rho, g, p);
            const float om = 1.0f - a;
            rg = __floats2half2_rn(c[0] * om, c[1] * om);
            b1 = __floats2half2_rn(c[2] * om, 1.0f);
            c[0] = __low2float(rg);
            c[1] = __high2float(rg);
            c[2] = __low2float(b1);
#pragma unroll
            for (int k = 0; k < 3; ++k) odd |= __float_as_uint(c[k]) >= 0x7f800000u;
        }
        *reinterpret_cast<uint2*>(slices + plane_stride * i + 4 * (size_t)id) =
            make_uint2(*reinterpret_cast<const unsigned*>(&rg), *reinterpret_cast<const unsigned*>(&b1));
    }
    odd = __syncthreads_or(odd);
    if (odd && threadIdx.x == 0) atomicOr(any_odd, 1);
}

template <typename T, bool EXACT>
__global__ void __launch_bounds__(256, 6) k_render_eye(const Setup S, const T* __restrict__ rho, const Grid g,
                             const __half* __restrict__ slices, const int* __restrict__ any_odd,
                             float* __restrict__ eye, float* __restrict__ comp) {
    __shared__ float table[MAX_TABLE];
    plane_table(S, S.cam, table);
    const int W = S.cam.w, H = S.cam.h, R = S.light.w;
    const bool all_plain = *any_odd == 0;
    int px, py;
    if (!tile_pixel(W, H, &px, &py)) return;
    const int id = px + W * py;
    const V3 d = ray_dir(S.cam, px, py);
    const float denom = dot3(d, S.n);
    const float inv = EXACT && quot_range(denom) ? __frcp_rn(denom) : 0.0f;
    float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const size_t plane_stride = (size_t)R * R * 4;
    int i0, i1;
    plane_range(S, S.cam, d, denom, i0, i1);
    for (int i = i0; i <= i1; ++i) {
        V3 p;
        if (!plane_hit(S, S.cam, d, denom, inv, i < MAX_TABLE ? table[i] : plane_distance(S, S.cam, i), &p)) continue;
        const float a = sample_density<EXACT>(S, rho, g, p);
        if (__float_as_uint(a) == 0u && all_plain && 1.0f - e[3] >= 0.0f && 1.0f - e[3] < 3e38f) {
            // empty space adds (+0, +0, +0, +0) to the pixel: no look at the light buffer, whose values are
            // all finite and without a sign here.  The sum still turns a -0 into +0.
#pragma unroll
            for (int k = 0; k < 4; ++k) e[k] += 0.0f;
            continue;
        }
        Colour lc{make_float2(S.clear[0], S.clear[1]), S.clear[2]};
        if (i > 0) {
            // light-projected position: NDC of the light view, mapped to [0, 1]
            const V3 q = p - S.light.eye;
            const float depth = dot3(q, S.light.f);
            const float bu = S.light.sx * depth, bv = S.light.sy * depth;
            float u = dot3(q, S.light.s), v = dot3(q, S.light.u);
            if (EXACT && bu == bv && quot_range(bu)) {  // the light's view is square
                const float2 uv = quot2(make_float2(u, v), both(-bu), both(__frcp_rn(bu)));
                u = uv.x;
                v = uv.y;
            } else {
                u = u / bu;
                v = v / bv;
            }
            u = u * 0.5f + 0.5f;
            v = v * 0.5f + 0.5f;
            lc = sample_light(S, slices + plane_stride * (i - 1), R, u, v);
        }
        if (S.back_to_front) {
            const float om = 1.0f - a;
            h16(lc.rg.x * a + e[0] * om, lc.rg.y * a + e[1] * om, &e[0], &e[1]);
            h16(lc.b * a + e[2] * om, a + e[3] * om, &e[2], &e[3]);
        } else {
            const float om = 1.0f - e[3];
            h16((lc.rg.x * a) * om + e[0], (lc.rg.y * a) * om + e[1], &e[0], &e[1]);
            h16((lc.b * a) * om + e[2], a * om + e[3], &e[2], &e[3]);
        }
    }
    float* o = eye + 4 * (size_t)id;
    o[0] = e[0];
    o[1] = e[1];
    o[2] = e[2];
    o[3] = e[3];
    if (comp) {
        float* c = comp + 3 * (size_t)id;
        const float om = 1.0f - e[3];
        c[0] = e[0] * e[3] + S.bg[0] * om;
        c[1] = e[1] * e[3] + S.bg[1] * om;
        c[2] = e[2] * e[3] + S.bg[2] * om;
    }
}

template <bool EXACT, typename T>
void draw(const Setup& S, const T* rho, const Grid& g, __half* slices, int* any_odd, float* eye, float* comp, cudaStream_t st) {
    k_render_light<T, EXACT><<<tile_blocks(S.light.w, S.light.w), 256, 0, st>>>(S, rho, g, slices, any_odd);
    k_render_eye<T, EXACT><<<tile_blocks(S.cam.w, S.cam.h), 256, 0, st>>>(S, rho, g, slices, any_odd, eye, comp);
}

}  // namespace
}  // namespace smk

using namespace smk;

extern "C" {

void smk_default_render_params(smk_render_params* rp) {
    if (!rp) return;
    *rp = smk_render_params{};
    rp->width = 1280;
    rp->height = 720;
    rp->light_res = 512;
    rp->planes = 100;
    const float cam[3] = {1.0f, 20.0f, 100.0f};
    const float len = sqrtf(cam[0] * cam[0] + cam[1] * cam[1] + cam[2] * cam[2]);
    for (int k = 0; k < 3; ++k) {
        rp->camera_pos[k] = cam[k];
        rp->camera_dir[k] = -cam[k] * (1.0f / len);
    }
    rp->up[1] = 1.0f;
    rp->fovy_deg = 45.0f;
    rp->znear = 5.0f;
    rp->zfar = 2000.0f;
    rp->light_pos[0] = 120.0f;
    rp->light_pos[1] = 80.0f;
    rp->light_fovy_deg = 45.0f;
    rp->light_znear = 5.0f;
    rp->light_zfar = 2000.0f;
    rp->light_color[0] = 0.9882f;
    rp->light_color[1] = 0.9333f;
    rp->light_color[2] = 0.7549f;
    rp->cell_size = 1.0f;
    for (int k = 0; k < 3; ++k) rp->bg_color[k] = 20.0f / 255.0f;
}

int smk_render(smk_sim* sim, const smk_render_params* rp, float* eye_rgba, float* composite_rgb, void* stream) {
    if (!sim || !rp || !eye_rgba) return smk_fail(SMK_ERR_INVALID, "null argument");
    if (rp->width < 1 || rp->height < 1 || rp->light_res < 1 || rp->planes < 1 || rp->planes > 100000 ||
        (long long)rp->width * rp->height > (1LL << 28) || rp->light_res > 16384 || !(rp->cell_size > 0.0f))
        return smk_fail(SMK_ERR_INVALID, "invalid render parameters");
    if (sim->g.nx < 2 || sim->g.ny < 2 || sim->g.nz < 2)
        return smk_fail(SMK_ERR_INVALID, "the renderer needs at least 2 cells per axis");
    DeviceGuard dg(sim->device);
    cudaStream_t st = (cudaStream_t)stream;
    const size_t slice_bytes = (size_t)rp->planes * rp->light_res * rp->light_res * 4 * sizeof(__half);
    const size_t need = slice_bytes + sizeof(int);
    if (sim->render_scratch_bytes < need) {
        if (sim->render_scratch) cudaFree(sim->render_scratch);
        sim->render_scratch = nullptr;
        sim->render_scratch_bytes = 0;
        SMK_CUDA(cudaMalloc(&sim->render_scratch, need));
        sim->render_scratch_bytes = need;
    }
    bool moderate;
    const Setup S = make_setup(*rp, sim->g.nx, sim->g.ny, sim->g.nz, &moderate);
    __half* slices = static_cast<__half*>(sim->render_scratch);
    int* any_odd = reinterpret_cast<int*>(static_cast<char*>(sim->render_scratch) + slice_bytes);
    const float* rho = sim->rho[sim->index_now ^ 1];
    SMK_CUDA(cudaMemsetAsync(any_odd, 0, sizeof(int), st));
    if (sim->rho_bf16) {
        const __nv_bfloat16* r = reinterpret_cast<const __nv_bfloat16*>(rho);
        moderate ? draw<true>(S, r, sim->g, slices, any_odd, eye_rgba, composite_rgb, st)
                 : draw<false>(S, r, sim->g, slices, any_odd, eye_rgba, composite_rgb, st);
    } else {
        moderate ? draw<true>(S, rho, sim->g, slices, any_odd, eye_rgba, composite_rgb, st)
                 : draw<false>(S, rho, sim->g, slices, any_odd, eye_rgba, composite_rgb, st);
    }
    SMK_CUDA(cudaGetLastError());
    return SMK_OK;
}

}  // extern "C"
