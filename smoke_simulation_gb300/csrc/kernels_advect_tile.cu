// Velocity advection (velocityAdvectionU/V/W, smokeSimulation.cu:527-615) with the velocity
// planes staged in shared memory by TMA.
//
// A CTA of 32 x 8 threads owns a 32 x 16 tile of cells in x-y and a run of consecutive planes, and
// walks them in ascending z, a thread computing the cells of two rows y and y + 1.  Each plane of u, v
// and w arrives as a 40 x 18 box (the tile plus one cell on every side, the x origin rounded
// down to a 16-byte boundary) in a four-slot ring: while plane z is computed, planes z - 1,
// z and z + 1 are resident and plane z + 2 is in flight.  The three 8-point averages of a cell
// read planes z - 1 and z at fixed offsets from one shared-memory address.  Where every backtrace of
// the two cells is shorter than REACH, the eight corners of each sample lie in the window and both
// cells go through packed arithmetic (sample_pair; without the clamps in tiles that cannot need them);
// otherwise each cell by itself reads the window or, past it, global memory (sample_win).  The
// arithmetic is the reference's, term for term (avgU/V/W and sampleSmoke, common.cuh).  The grouped
// form runs the same tiles over every grid of a batch.
//
// Instruction issue bounds it (75 % of the slots, 46 % of the warps at 64 registers): 256^3 FP32 took
// 200 us with one cell a thread and scalar arithmetic (388 instructions a cell, 203 M in all), 162 us now
// (143 M); its 510 MB would take 75 us at the copy rate.  85 registers and three CTAs an SM: 165 us.
//
// Each iteration has one barrier: after it every thread has finished plane z - 1, so thread 0
// refills the slot of plane z - 2 with plane z + 2.  Waits on the ring's mbarriers are bounded;
// on a timeout the CTA records the error, waits (bounded) for its own copies still in flight
// and returns.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "tb_common.cuh"

namespace smk {

namespace {

using namespace tb;

constexpr int AT_TX = 32, AT_TY = 8;          // threads
constexpr int AT_ROWS = 2 * AT_TY;             // cell rows of the tile: two per thread
constexpr int AT_W = 40;                  // window columns: x in [x_tile - 4, x_tile + 36)
constexpr int AT_H = AT_ROWS + 2;         // window rows: y in [y_tile - 1, y_tile + 17)
constexpr int AT_PSTR = 736;              // floats per field plane: 40 x 18, padded to 128 bytes
constexpr int AT_SLOTS = 4;
constexpr int AT_BOX_BYTES = AT_W * AT_H * 4;
constexpr int AT_OX = 4;                  // a cell's column in the window = tx + AT_OX

static_assert(AT_PSTR * 4 % 128 == 0 && AT_PSTR >= AT_W * AT_H, "plane stride");

struct AdvMaps {
    CUtensorMap u, v, w;
};

// A trilinear sample of one field (sampleSmoke's arithmetic) whose corners are read from the
// window planes pm, pc, pp (planes z - 1, z, z + 1; the window's origin is (wx0, wy0)) when
// they lie there, else from global memory.
template <int HX, int HY, int HZ>
__device__ __forceinline__ float sample_win(const float* __restrict__ f, const Grid& g, const float* pm,
                                            const float* pc, const float* pp, int wx0, int wy0, int z, float px,
                                            float py, float pz) {
    const int lx = g.nx - 1, ly = g.ny - 1, lz = g.nz - 1;
    const float mx = (float)(unsigned)lx, my = (float)(unsigned)ly, mz = (float)(unsigned)lz;
    const float xs = fmaxf(fminf(px, mx), 1.0f) - (HX ? 0.5f : 0.0f);
    const float ys = fmaxf(fminf(py, my), 1.0f) - (HY ? 0.5f : 0.0f);
    const float zs = fmaxf(fminf(pz, mz), 1.0f) - (HZ ? 0.5f : 0.0f);
    const int x0 = __float2int_rz(xs);
    const float xw1 = xs - (float)x0;
    const float xw0 = 1.0f - xw1;
    const int y0 = __float2int_rz(ys);
    const float yw1 = ys - (float)y0;
    const float yw0 = 1.0f - yw1;
    const int z0 = __float2int_rz(zs);
    const float zw1 = zs - (float)z0;
    const float zw0 = 1.0f - zw1;
    // the upper corner repeats the lower one only on a delta-0 axis clamped to the last cell
    const bool sy = HY || y0 < ly;
    const bool sz = HZ || z0 < lz;
    const bool sx = HX || x0 < lx;
    const unsigned ux = (unsigned)(x0 - wx0), uy = (unsigned)(y0 - wy0), uz = (unsigned)(z0 - (z - 1));
    float a000, a010, a001, a011, b100, b110, b101, b111;
    if (ux <= (unsigned)(AT_W - 2) && uy <= (unsigned)(AT_H - 2) && uz <= 1u) {
        const int o = (int)(uy * AT_W + ux);
        const float* q0 = (uz ? pc : pm) + o;
        const float* q1 = sz ? (uz ? pp : pc) + o : q0;
        const int oy = sy ? AT_W : 0;
        a000 = q0[0];
        b100 = q0[1];
        a010 = q0[oy];
        b110 = q0[oy + 1];
        a001 = q1[0];
        b101 = q1[1];
        a011 = q1[oy];
        b111 = q1[oy + 1];
    } else {
        const float* r00 = f + (x0 + y0 * g.X + z0 * g.XY);
        const float* r10 = r00 + (sy ? g.X : 0);
        const float* r01 = r00 + (sz ? g.XY : 0);
        const float* r11 = r01 + (sy ? g.X : 0);
        a000 = r00[0];
        a010 = r10[0];
        a001 = r01[0];
        a011 = r11[0];
        b100 = r00[1];
        b110 = r10[1];
        b101 = r01[1];
        b111 = r11[1];
    }
    const float a100 = sx ? b100 : a000, a110 = sx ? b110 : a010, a101 = sx ? b101 : a001,
                a111 = sx ? b111 : a011;
    // the eight terms' products as packed pairs (each lane one IEEE product, the same bits).  The
    // products feed products and scalar sums only: ptxas contracts a packed product followed by a
    // packed add into a fused multiply-add, even with -fmad=false and explicit .rn forms
    const float2 xw = make_float2(xw0, xw1);
    const float2 xy0 = __fmul2_rn(xw, make_float2(yw0, yw0)), xy1 = __fmul2_rn(xw, make_float2(yw1, yw1));
    const float2 z0v = make_float2(zw0, zw0), z1v = make_float2(zw1, zw1);
    const float2 p0 = __fmul2_rn(__fmul2_rn(xy0, z0v), make_float2(a000, a100));
    const float2 p1 = __fmul2_rn(__fmul2_rn(xy1, z0v), make_float2(a010, a110));
    const float2 p2 = __fmul2_rn(__fmul2_rn(xy0, z1v), make_float2(a001, a101));
    const float2 p3 = __fmul2_rn(__fmul2_rn(xy1, z1v), make_float2(a011, a111));
    return p0.x + p0.y + p1.x + p1.y + p2.x + p2.y + p3.x + p3.y;
}

__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// Multipliers of packed sums: a x 1 and a x -1 with a factor the compiler does not know.  It would
// contract a packed addition (or a product with a literal 1) with the product before it.
struct Ones {
    float2 one, mone;
};

// The clamp's upper ends n - 1 of the three axes, and the bits of 2^23 + them.
struct Tops {
    float x, y, z;
    int bx, by, bz;
};

// The same sample for the cells of rows y and y + 1 at once (lane x: row y), for positions at most
// REACH cells from the cells' own: their corners lie in the window, so there is no fallback.  win: the
// field's window; fm, fc, fp: where the planes z - 1, z, z + 1 would have the column and row whose floats
// have no bits set, so that the bits of 2^23 + a column and a row index them; kz: the bits of 2^23 + z.
// Floors are packed sums with 2^23 rounded down.
// EDGE: the positions may need the clamp to [1, n - 1].
template <int HX, int HY, int HZ, bool EDGE>
__device__ __forceinline__ float2 sample_pair(const float* win, const Tops& top, unsigned fm, unsigned fc, unsigned fp, int kz,
                                              float2 px, float2 py, float2 pz, const Ones& k) {
    if (EDGE) {
        const float mx = top.x, my = top.y, mz = top.z;
        px = make_float2(fmaxf(fminf(px.x, mx), 1.0f), fmaxf(fminf(px.y, mx), 1.0f));
        py = make_float2(fmaxf(fminf(py.x, my), 1.0f), fmaxf(fminf(py.y, my), 1.0f));
        pz = make_float2(fmaxf(fminf(pz.x, mz), 1.0f), fmaxf(fminf(pz.y, mz), 1.0f));
    }
    if (HX) px = __fadd2_rn(px, both(-0.5f));
    if (HY) py = __fadd2_rn(py, both(-0.5f));
    if (HZ) pz = __fadd2_rn(pz, both(-0.5f));
    const float2 bx = __fadd2_rd(px, both(8388608.0f)), by = __fadd2_rd(py, both(8388608.0f)),
                 bz = __fadd2_rd(pz, both(8388608.0f));
    const float2 x1 = __ffma2_rn(__fadd2_rn(bx, both(-8388608.0f)), k.mone, px);
    const float2 y1 = __ffma2_rn(__fadd2_rn(by, both(-8388608.0f)), k.mone, py);
    const float2 z1 = __ffma2_rn(__fadd2_rn(bz, both(-8388608.0f)), k.mone, pz);
    const float2 x0 = __ffma2_rn(x1, k.mone, both(1.0f)), y0 = __ffma2_rn(y1, k.mone, both(1.0f)),
                 z0 = __ffma2_rn(z1, k.mone, both(1.0f));
    float2 a[8];  // corners 000, 100, 010, 110, 001, 101, 011, 111
    auto corners = [&](float cbx, float cby, float cbz, auto put) {
        const int jx = __float_as_int(cbx), jy = __float_as_int(cby), jz = __float_as_int(cbz);
        const unsigned o = (unsigned)jx + AT_W * (unsigned)jy;
        const bool at = jz == kz;
        const int l = (int)((at ? fc : fm) + o);
        int h = (int)((at ? fp : fc) + o), oy = AT_W;
        bool sx = true;
        if (EDGE) {  // the upper corner repeats the lower one on a delta-0 axis clamped to the last cell
            if (!HZ && jz == top.bz) h = l;
            if (!HY && jy == top.by) oy = 0;
            if (!HX) sx = jx != top.bx;
        }
        const float q0 = win[l], q2 = win[l + oy], q4 = win[h], q6 = win[h + oy];
        put(0, q0);
        put(1, sx ? win[l + 1] : q0);
        put(2, q2);
        put(3, sx ? win[l + oy + 1] : q2);
        put(4, q4);
        put(5, sx ? win[h + 1] : q4);
        put(6, q6);
        put(7, sx ? win[h + oy + 1] : q6);
    };
    corners(bx.x, by.x, bz.x, [&](int i, float v) { a[i].x = v; });
    corners(bx.y, by.y, bz.y, [&](int i, float v) { a[i].y = v; });
    // the eight terms in the reference's order
    const float2 w00 = __fmul2_rn(x0, y0), w10 = __fmul2_rn(x1, y0), w01 = __fmul2_rn(x0, y1), w11 = __fmul2_rn(x1, y1);
    float2 s = __fmul2_rn(__fmul2_rn(w00, z0), a[0]);
    s = __ffma2_rn(__fmul2_rn(__fmul2_rn(w10, z0), a[1]), k.one, s);
    s = __ffma2_rn(__fmul2_rn(__fmul2_rn(w01, z0), a[2]), k.one, s);
    s = __ffma2_rn(__fmul2_rn(__fmul2_rn(w11, z0), a[3]), k.one, s);
    s = __ffma2_rn(__fmul2_rn(__fmul2_rn(w00, z1), a[4]), k.one, s);
    s = __ffma2_rn(__fmul2_rn(__fmul2_rn(w10, z1), a[5]), k.one, s);
    s = __ffma2_rn(__fmul2_rn(__fmul2_rn(w01, z1), a[6]), k.one, s);
    return __ffma2_rn(__fmul2_rn(__fmul2_rn(w11, z1), a[7]), k.one, s);
}

// max(m, |x|); NaN if either is, so that a NaN never counts as near.
__device__ __forceinline__ float reach(float m, float x) {
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(fabsf(x)));
    return m;
}
constexpr float REACH = 0.9f;  // a backtrace of one cell at most, with room for the positions' rounding

struct AdvWindow {
    alignas(128) float win[AT_SLOTS][3][AT_PSTR];
    alignas(8) uint64_t mbar[AT_SLOTS];
};

// The tile (bx, by) for planes zs .. zs + zc - 1.
template <typename To>
__device__ __forceinline__ void advect_tile(AdvWindow& sh, const AdvMaps& maps, const Grid& g,
                                            const float* __restrict__ u0, const float* __restrict__ v0,
                                            const float* __restrict__ w0, To* __restrict__ u1, To* __restrict__ v1,
                                            To* __restrict__ w1, const uint8_t* __restrict__ flags, float dt, int* kerr,
                                            int bx, int by, int zs, int zc, float one, const Tops& top) {
    auto& win = sh.win;
    auto& mbar = sh.mbar;
    const int tx = (int)threadIdx.x, ty = (int)threadIdx.y;
    const bool leader = tx == 0 && ty == 0;
    const int xt = bx * AT_TX, yt = 1 + by * AT_ROWS;
    const int ze = min(zs + zc, g.nz);  // planes [zs, ze) are advected; [zs - 1, ze] are read
    const int wx0 = xt - AT_OX, wy0 = yt - 1;

    // plane p goes to slot p & 3; its barrier phase counts the slot's earlier uses in this CTA
    auto issue = [&](int p) {
        const int s = p & (AT_SLOTS - 1);
        const uint32_t bar = smem_u32(&mbar[s]);
        mbar_expect_tx(bar, 3u * AT_BOX_BYTES);
        tma_load_3d(smem_u32(&win[s][0][0]), &maps.u, wx0, wy0, p, bar);
        tma_load_3d(smem_u32(&win[s][1][0]), &maps.v, wx0, wy0, p, bar);
        tma_load_3d(smem_u32(&win[s][2][0]), &maps.w, wx0, wy0, p, bar);
    };
    auto parity = [&](int p) { return (uint32_t)(((p - (zs - 1)) >> 2) & 1); };
    if (leader) {
        for (int s = 0; s < AT_SLOTS; ++s) mbar_init(smem_u32(&mbar[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int p = zs - 1; p <= min(zs + 1, ze); ++p) issue(p);
    }
    __syncthreads();

    const int x = xt + tx, y = yt + 2 * ty;
    // the faces of row y + r that this thread may advect below the last plane, as flag bits
    auto may = [&](int r) {
        const bool live = x >= 1 && x < g.nx && y + r < g.ny, inx = x <= g.nx - 2, iny = y + r <= g.ny - 2;
        return !live ? 0u : (iny ? F_XM : 0u) | (inx ? F_YM : 0u) | (inx && iny ? F_ZM : 0u);
    };
    const unsigned may0 = may(0), may1 = may(1);
    const uint8_t* fl = flags + g.idx(x, y, zs);  // loaded one plane ahead
    unsigned f0 = may0 ? fl[0] : 0u, f1 = may1 ? fl[g.X] : 0u;
    const int oc = (2 * ty + 1) * AT_W + tx + AT_OX;  // row y's offset in a window plane
    const float xf = (float)x, yf = (float)y;
    const Ones k{both(one), both(-one)};
    const float2 dt2 = both(dt);
    const unsigned kxy = 0x4b000000u + (unsigned)wx0 + AT_W * (0x4b000000u + (unsigned)wy0);
    // no position of this tile's columns and rows leaves [1, n - 1]
    const bool inner = xt >= 2 && xt + AT_TX <= g.nx - 2 && yt >= 2 && yt + AT_ROWS <= g.ny - 2;
    const float* wf = &win[0][0][0];
    int issued = min(zs + 1, ze);  // last plane issued (leader)
    int waited = zs - 2;           // last plane this thread has seen complete
    if (mbar_wait(smem_u32(&mbar[(zs - 1) & 3]), parity(zs - 1))) {
        waited = zs - 1;
        if (mbar_wait(smem_u32(&mbar[zs & 3]), parity(zs))) waited = zs;
    }
    bool ok = waited == zs;

    for (int z = zs; z < ze; ++z) {
        if (z > zs) {
            // every thread is done with plane z - 2's slot; refill it with plane z + 2
            if (__syncthreads_or(!ok)) break;
            if (leader && z + 2 <= ze) issue(issued = z + 2);
        } else if (leader && z + 2 <= ze) {
            issue(issued = z + 2);
        }
        const unsigned in = z <= g.nz - 2 ? F_XM | F_YM | F_ZM : F_ZM;
        const unsigned m0 = f0 & F_SELF ? f0 & may0 & in : 0u, m1 = f1 & F_SELF ? f1 & may1 & in : 0u;
        fl += g.XY;
        if (z + 1 < ze) {
            if (may0) f0 = fl[0];
            if (may1) f1 = fl[g.X];
        }
        if (ok) ok = mbar_wait(smem_u32(&mbar[(z + 1) & 3]), parity(z + 1));
        if (!ok) continue;
        waited = z + 1;
        if (!(m0 | m1)) continue;
        const int i = g.idx(x, y, z);
        // planes z - 1, z, z + 1 of u; v and w follow at AT_PSTR and 2 AT_PSTR
        const int um = ((z - 1) & 3) * 3 * AT_PSTR, uc = (z & 3) * 3 * AT_PSTR, up = ((z + 1) & 3) * 3 * AT_PSTR;
        auto pair = [&](int o) { return make_float2(wf[o], wf[o + AT_W]); };
        // avgU/avgV/avgW of both cells, in the reference's order (common.cuh)
        auto average = [&](int a, int b, int dx, int dy) {
            float2 s = __fadd2_rn(pair(a), pair(a + dx));
            s = __fadd2_rn(s, pair(a + dy));
            s = __fadd2_rn(s, pair(a + dx + dy));
            s = __fadd2_rn(s, pair(b));
            s = __fadd2_rn(s, pair(b + dx));
            s = __fadd2_rn(s, pair(b + dy));
            s = __fadd2_rn(s, pair(b + dx + dy));
            return __fmul2_rn(s, both(0.125f));
        };
        const int vo = AT_PSTR + oc, wo = 2 * AT_PSTR + oc;
        const float2 au = average(um + oc, uc + oc, 1, -AT_W);
        const float2 av = average(um + vo, uc + vo, -1, AT_W);
        const float2 aw = average(uc + wo, um + wo, -1, -AT_W);
        const float2 cu = pair(uc + oc), cv = pair(uc + vo), cw = pair(uc + wo);
        const float2 tu = __fmul2_rn(dt2, au), tv = __fmul2_rn(dt2, av), tw = __fmul2_rn(dt2, aw);
        const float2 su = __fmul2_rn(dt2, cu), sv = __fmul2_rn(dt2, cv), sw = __fmul2_rn(dt2, cw);
        float far = fabsf(tu.x);
        for (float t : {tu.y, tv.x, tv.y, tw.x, tw.y, su.x, su.y, sv.x, sv.y, sw.x, sw.y}) far = reach(far, t);
        const float zf = (float)z;
        if (far <= REACH) {
            auto near_by = [&](auto edge) {
                constexpr bool EDGE = decltype(edge)::value;
                const float2 x2 = both(xf), xh = both(xf + 0.5f), z2 = both(zf), zh = both(zf + 0.5f);
                const float2 y2 = make_float2(yf, yf + 1.0f), yh = make_float2(yf + 0.5f, yf + 1.5f);
                const int kz = 0x4b000000 + z;
                if ((m0 | m1) & F_XM) {
                    const float2 r = sample_pair<0, 1, 1, EDGE>(wf, top, um - kxy, uc - kxy, up - kxy, kz, __ffma2_rn(su, k.mone, x2),
                                                                __ffma2_rn(tv, k.mone, yh), __ffma2_rn(tw, k.mone, zh), k);
                    if (m0 & F_XM) stv(u1, i, r.x);
                    if (m1 & F_XM) stv(u1, i + g.X, r.y);
                }
                if ((m0 | m1) & F_YM) {
                    const float2 r = sample_pair<1, 0, 1, EDGE>(wf + AT_PSTR, top, um - kxy, uc - kxy, up - kxy, kz,
                                                                __ffma2_rn(tu, k.mone, xh), __ffma2_rn(sv, k.mone, y2),
                                                                __ffma2_rn(tw, k.mone, zh), k);
                    if (m0 & F_YM) stv(v1, i, r.x);
                    if (m1 & F_YM) stv(v1, i + g.X, r.y);
                }
                if ((m0 | m1) & F_ZM) {
                    const float2 r = sample_pair<1, 1, 0, EDGE>(wf + 2 * AT_PSTR, top, um - kxy, uc - kxy, up - kxy, kz,
                                                                __ffma2_rn(tu, k.mone, xh), __ffma2_rn(tv, k.mone, yh),
                                                                __ffma2_rn(sw, k.mone, z2), k);
                    if (m0 & F_ZM) stv(w1, i, r.x);
                    if (m1 & F_ZM) stv(w1, i + g.X, r.y);
                }
            };
            if (inner && z >= 2 && z <= g.nz - 3)
                near_by(std::false_type{});
            else
                near_by(std::true_type{});
            continue;
        }
        // a longer backtrace in one of the two cells: each by itself, window or global memory
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            const unsigned m = c ? m1 : m0;
            const int ic = i + (c ? g.X : 0);
            const float yc = yf + (float)c;
            const float du = c ? su.y : su.x, dv = c ? sv.y : sv.x, dw = c ? sw.y : sw.x;
            const float eu = c ? tu.y : tu.x, ev = c ? tv.y : tv.x, ew = c ? tw.y : tw.x;
            const float *pm = wf + um, *pc = wf + uc, *pp = wf + up;
            if (m & F_XM)
                stv(u1, ic, sample_win<0, 1, 1>(u0, g, pm, pc, pp, wx0, wy0, z, xf - du, yc + 0.5f - ev, zf + 0.5f - ew));
            if (m & F_YM)
                stv(v1, ic, sample_win<1, 0, 1>(v0, g, pm + AT_PSTR, pc + AT_PSTR, pp + AT_PSTR, wx0, wy0, z,
                                                xf + 0.5f - eu, yc - dv, zf + 0.5f - ew));
            if (m & F_ZM)
                stv(w1, ic, sample_win<1, 1, 0>(w0, g, pm + 2 * AT_PSTR, pc + 2 * AT_PSTR, pp + 2 * AT_PSTR, wx0, wy0, z,
                                                xf + 0.5f - eu, yc + 0.5f - ev, zf - dw));
        }
    }
    if (__syncthreads_or(!ok)) {
        // a plane never arrived: record it and wait (bounded) for this CTA's copies in flight
        if (leader) {
            atomicExch(kerr, 1);
            for (int p = waited + 1; p <= issued; ++p) mbar_wait(smem_u32(&mbar[p & 3]), parity(p));
        }
        __syncthreads();
    }
}

template <typename To>
__global__ void __launch_bounds__(AT_TX * AT_TY, 4)
k_advect_velocity_tile(const __grid_constant__ AdvMaps maps, Grid g, const float* __restrict__ u0,
                       const float* __restrict__ v0, const float* __restrict__ w0, To* __restrict__ u1,
                       To* __restrict__ v1, To* __restrict__ w1, const uint8_t* __restrict__ flags, float dt,
                       int* kerr, int cz0, int zc, float one, Tops top) {
    __shared__ AdvWindow sh;
    advect_tile(sh, maps, g, u0, v0, w0, u1, v1, w1, flags, dt, kerr, (int)blockIdx.x, (int)blockIdx.y,
                1 + (cz0 + (int)blockIdx.z) * zc, zc, one, top);
}

// One grid of a grouped velocity advection.
struct GroupAdvGrid {
    AdvMaps maps;
    Grid g;
    Tops top;
    const float *u0, *v0, *w0;
    void *u1, *v1, *w1;
    const uint8_t* flags;
    int* kerr;
    float dt;
    int tiles_x, tiles_y, zc;
};

// Every tile of the grids whose advected faces are To, one CTA a tile (starts: prefix sums of the tiles).
template <typename To>
__global__ void __launch_bounds__(AT_TX * AT_TY, 4)
k_group_advect_velocity(const GroupAdvGrid* __restrict__ grids, const int* __restrict__ starts, int n, float one) {
    __shared__ AdvWindow sh;
    const int j = find_grid(starts, n, (int)blockIdx.x);
    const GroupAdvGrid& d = grids[j];
    const int local = (int)blockIdx.x - starts[j], tx = d.tiles_x, ty = d.tiles_y, zc = d.zc;
    const Grid g = d.g;
    const Tops top = d.top;
    if (threadIdx.x == 0 && threadIdx.y == 0) {  // the maps were written by a copy into the table
        tensormap_acquire(&d.maps.u);
        tensormap_acquire(&d.maps.v);
        tensormap_acquire(&d.maps.w);
    }
    advect_tile(sh, d.maps, g, d.u0, d.v0, d.w0, (To*)d.u1, (To*)d.v1, (To*)d.w1, d.flags, d.dt, d.kerr, local % tx,
                (local / tx) % ty, 1 + (local / (tx * ty)) * zc, zc, one, top);
}

Tops tops_of(const Grid& g) {
    return Tops{(float)(g.nx - 1),     (float)(g.ny - 1),     (float)(g.nz - 1),
                0x4b000000 + g.nx - 1, 0x4b000000 + g.ny - 1, 0x4b000000 + g.nz - 1};
}

}  // namespace

static int tiles_x(const Grid& g) { return (g.nx + AT_TX - 1) / AT_TX; }
static int tiles_y(const Grid& g) { return (g.ny - 1 + AT_ROWS - 1) / AT_ROWS; }

struct AdvectMaps {
    AdvMaps set[2];
    int n;
};

AdvectMaps* create_advect_maps(const Grid& g, const float* const* u, const float* const* v, const float* const* w,
                               int n) {
    if (n < 1 || n > 2) return nullptr;
    AdvectMaps* m = new AdvectMaps();
    m->n = n;
    bool ok = true;
    for (int k = 0; k < n && ok; ++k)
        ok = tb::encode_3d_box(&m->set[k].u, u[k], false, g, AT_W, AT_H) &&
             tb::encode_3d_box(&m->set[k].v, v[k], false, g, AT_W, AT_H) &&
             tb::encode_3d_box(&m->set[k].w, w[k], false, g, AT_W, AT_H);
    if (!ok) {
        delete m;
        return nullptr;
    }
    return m;
}

void destroy_advect_maps(AdvectMaps* m) { delete m; }

template <typename To>
int launch_advect_velocity_tile(const AdvectMaps* m, int set, const Grid& g, const float* u0, const float* v0,
                                const float* w0, To* u1, To* v1, To* w1, const uint8_t* flags, float dt, int* kerr,
                                cudaStream_t st, int c0, int c1) {
    if (m == nullptr || set < 0 || set >= m->n) return -1;
    if (g.nx < 2 || g.ny < 2 || g.nz < 2) return 0;
    const int chunks = advect_velocity_chunks(g);
    if (c1 < 0 || c1 > chunks) c1 = chunks;
    if (c0 < 0) c0 = 0;
    if (c1 <= c0) return 0;
    const dim3 grid((unsigned)tiles_x(g), (unsigned)tiles_y(g), (unsigned)(c1 - c0));
    k_advect_velocity_tile<To><<<grid, dim3(AT_TX, AT_TY), 0, st>>>(m->set[set], g, u0, v0, w0, u1, v1, w1, flags, dt,
                                                                     kerr, c0, advect_velocity_chunk_planes(g), 1.0f, tops_of(g));
    return 0;
}

// Sixteen planes a chunk read each plane 1.1 times; small grids halve the chunks until two CTAs an SM have
// work, as a CTA's planes follow one another (32^3, two tiles: both advections take 28 us with two chunks,
// 12 with thirty-one; 80^3: 11 us less).
int advect_velocity_chunk_planes(const Grid& g) {
    int zc = 16;
    while (zc > 1 && tiles_x(g) * tiles_y(g) * ((g.nz - 1 + zc - 1) / zc) < 304) zc /= 2;
    return zc;
}

int advect_velocity_chunks(const Grid& g) {
    const int zc = advect_velocity_chunk_planes(g);
    return g.nz < 2 ? 0 : (g.nz - 1 + zc - 1) / zc;
}

size_t group_advect_record_bytes() { return sizeof(GroupAdvGrid); }

int group_advect_fill(void* rec, const AdvectMaps* m, int set, const Grid& g, const float* const* in, void* const* out,
                      const uint8_t* flags, int* kerr, float dt, int zc) {
    if (m == nullptr || set < 0 || set >= m->n || g.nx < 2 || g.ny < 2 || g.nz < 2) return 0;
    GroupAdvGrid d;
    memset(&d, 0, sizeof(d));
    d.maps = m->set[set];
    d.g = g;
    d.top = tops_of(g);
    d.u0 = in[0];
    d.v0 = in[1];
    d.w0 = in[2];
    d.u1 = out[0];
    d.v1 = out[1];
    d.w1 = out[2];
    d.flags = flags;
    d.kerr = kerr;
    d.dt = dt;
    d.tiles_x = tiles_x(g);
    d.tiles_y = tiles_y(g);
    d.zc = zc;
    memcpy(rec, &d, sizeof(d));
    return d.tiles_x * d.tiles_y * ((g.nz - 1 + zc - 1) / zc);
}

int launch_group_advect_velocity(const void* recs, const int* starts, int n, int total, bool bf16, cudaStream_t st) {
    if (total <= 0) return 0;
    const GroupAdvGrid* d = static_cast<const GroupAdvGrid*>(recs);
    if (bf16)
        k_group_advect_velocity<__nv_bfloat16><<<(unsigned)total, dim3(AT_TX, AT_TY), 0, st>>>(d, starts, n, 1.0f);
    else
        k_group_advect_velocity<float><<<(unsigned)total, dim3(AT_TX, AT_TY), 0, st>>>(d, starts, n, 1.0f);
    return (int)cudaGetLastError();
}

template int launch_advect_velocity_tile<float>(const AdvectMaps*, int, const Grid&, const float*, const float*,
                                                const float*, float*, float*, float*, const uint8_t*, float, int*,
                                                cudaStream_t, int, int);
template int launch_advect_velocity_tile<__nv_bfloat16>(const AdvectMaps*, int, const Grid&, const float*,
                                                        const float*, const float*, __nv_bfloat16*,
                                                        __nv_bfloat16*, __nv_bfloat16*, const uint8_t*, float, int*,
                                                        cudaStream_t, int, int);

}  // namespace smk
