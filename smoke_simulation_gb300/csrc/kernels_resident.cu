// Whole solves of small and middle grids in one launch, the iterate resident in shared memory.
//
// Below about 130^3 cells a colour pass is too short to launch by itself (32^3: 1.9 us a launch, 80^3:
// 4.3 us) and a blocked march too short to fill the chip (64^3: about 20 us per three sweeps, most of it
// halo planes).  Here the grid's interior is cut into boxes of rows along y and z, one per CTA, all
// resident at once (a cooperative launch of at most one CTA per SM); a CTA keeps its box in shared
// memory through all passes, and after each pass sends the cells (or faces) on the box's four sides to
// the neighbours.
//
// Exchange.  A value travels with the number of its pass in one 64-bit store; the receiver polls its own
// element until the number is there.  That is one trip through L2 per pass (about 0.7 us) instead of
// a barrier's three (fence, flag, data), and CTAs only wait for their neighbours.  The two colours have
// elements of their own: a box may send its next pass before the neighbour has read this one, but
// the pass after that needs the neighbour's next values, which are sent after it has read these.  The
// elements start at zero (a memset ahead of every launch), pass numbers at 1.  The tolerance check gathers
// one maximum per CTA in the first one, which hands out the largest, the same way (the largest form: all
// to all).  Waits are bounded: a thread that gives up, or sees *kerr set, makes its CTA record the error and leave,
// and the others follow.
//
// Layout.  The two colours of a row are separate: cell x of parity c = (x + y + z) & 1 is element x / 2
// of colour row c, so the cells of a pass are consecutive, and so are all their neighbours, which lie in
// the other colour (element x / 2 of the four rows around; x / 2 and x / 2 - 1 or + 1 in its own).  A
// thread has the same cells in every pass: their constants stay in registers, the sides' cells come
// first so that their values are under way while the others are computed.
//
// Arithmetic as in the other kernels of each scheme, so the results are theirs, bit for bit.
//
// What bounds it: up to about 64^3 the exchange (0.95 us a pass at 32^3, of which a pass's arithmetic is
// 0.1), above it instruction issue (about 60 warp instructions a cell in the pressure form, 120 in the
// velocity form).  us per 30 sweeps (a check every 6) and per 30 iterations, before (the faster of one pass per
// launch and blocked) and now: 32^3 155 -> 68 and 113 -> 66; 64^3 205 -> 78 and 155 -> 82; 80^3 218 -> 95
// and 261 -> 129; 100^3 238 -> 150 and 369 -> 234; 127^3 286 -> 265 and 552 -> 369.  Not kept: all loads of four
// cells ahead of their updates in the pressure form (80^3 83 -> 100 us without checks), 1024 threads on small
// grids (64^3 65 -> 73), 512 with 14 cells each on large ones (127^3 228 -> 324).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "exact_scale.cuh"
#include "kernels.h"
#include "stage_bodies.cuh"

namespace smk {

namespace {

constexpr unsigned RES_POLLS = 1u << 21;      // about a second
constexpr size_t RES_SMEM = 224 * 1024;  // dynamic; the tables and the reduction take up to 2 KB more

struct ResidentArgs {
    Grid g;
    int by, bz, cy, cz;   // rows of a box, boxes along y and z
    int hx;               // cells of one colour in a row
    int hp;               // elements of a colour row
    int sy, sz;           // elements of a y side and of a z side in the exchange buffer
    int half;             // elements of all sides of all boxes
    unsigned long long* ex;  // [colour][cta][y sides, z sides], then [group parity][cta] check maxima and
                             // [group parity] their maximum
    int* kerr;
};

__device__ __forceinline__ void ex_put(unsigned long long* p, float v, unsigned pass) {
    const unsigned long long x = ((unsigned long long)pass << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(x) : "memory");
}

__device__ __forceinline__ unsigned long long ex_load(const unsigned long long* p) {
    unsigned long long x;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(__cvta_generic_to_global(p)) : "memory");
    return x;
}

// Row number r of a box of by x bz rows, the rows on its sides first.
__device__ __forceinline__ void box_row(int r, int by, int bz, int& yy, int& zz) {
    const int ends = bz > 1 ? 2 * by : by;  // z sides
    if (r < ends) {
        zz = r < by ? 0 : bz - 1;
        yy = r < by ? r : r - by;
        return;
    }
    r -= ends;
    const int mid = bz - 2, cols = by > 1 ? 2 : 1;  // y sides of the planes between
    if (r < mid * cols) {
        zz = 1 + r % mid;
        yy = r < mid ? 0 : by - 1;
        return;
    }
    r -= mid * cols;
    zz = 1 + r / (by - 2);
    yy = 1 + r % (by - 2);
}

enum : unsigned { SIDE_YM = 0, SIDE_YP = 1, SIDE_ZM = 2, SIDE_ZP = 3 };

// A CTA's box: interior rows y0 .. y0 + by - 1, z0 .. z0 + bz - 1.
struct Box {
    int iy, iz, cta, y0, z0, by, bz;
    __device__ __forceinline__ Box(const ResidentArgs& a) {
        cta = (int)blockIdx.x;
        iy = cta % a.cy;
        iz = cta / a.cy;
        y0 = 1 + iy * a.by;
        z0 = 1 + iz * a.bz;
        by = min(a.by, a.g.ny - 1 - y0);
        bz = min(a.bz, a.g.nz - 1 - z0);
    }
    __device__ __forceinline__ bool has(unsigned side, const ResidentArgs& a) const {
        return side == SIDE_YM ? iy > 0 : side == SIDE_YP ? iy + 1 < a.cy : side == SIDE_ZM ? iz > 0 : iz + 1 < a.cz;
    }
    // The neighbour across `side`; what it sends towards this box is on its opposite side.
    __device__ __forceinline__ int across(unsigned side, const ResidentArgs& a) const {
        return side == SIDE_YM ? cta - 1 : side == SIDE_YP ? cta + 1 : side == SIDE_ZM ? cta - a.cy : cta + a.cy;
    }
    __device__ __forceinline__ int rows(unsigned side) const { return side < SIDE_ZM ? bz : by; }
};

// Where a side begins among a box's elements.
__device__ __forceinline__ int side_base(const ResidentArgs& a, unsigned side) {
    return side < SIDE_ZM ? (int)side * a.sy : 2 * a.sy + (int)(side - SIDE_ZM) * a.sz;
}
__device__ __forceinline__ size_t box_base(const ResidentArgs& a, int cta) { return (size_t)cta * 2 * (size_t)(a.sy + a.sz); }

// What a thread keeps of its cells: slot s is element i = tid + s * RT of the box's (row, h) pairs, both
// colours of it.  word: the element of colour 0 in shared memory (16 bits), acc of colour 0 and 1 (three
// bits each from 16, 0 where a pass does not update the cell), the parity of y + z (bit 22), the sides it
// lies on that have a neighbour (bits 24..27); send: its element on the y sides (16 bits) and z sides.
struct Slot {
    unsigned word, send;
};
constexpr unsigned SLOT_NONE = 0xffffffffu;

__device__ __forceinline__ Slot make_slot(const ResidentArgs& a, const Box& box, int i, int ry, int off,
                                          const uint8_t* flags) {
    // a slot beyond the box: an element of its first row that no pass updates or sends
    Slot t{(unsigned)((off * ry + off) * 2 * a.hp), 0u};
    const int r = i / a.hx, h = i - r * a.hx;
    if (r >= box.by * box.bz) return t;
    int yy, zz;
    box_row(r, box.by, box.bz, yy, zz);
    const int y = box.y0 + yy, z = box.z0 + zz;
    t.word = (unsigned)(((zz + off) * ry + yy + off) * 2 * a.hp + h) | ((unsigned)((y + z) & 1) << 22);
    for (int c = 0; c < 2; ++c) {
        const int x = 2 * h + ((y + z + c) & 1);
        if (x < 1 || x > a.g.nx - 2) continue;
        const unsigned f = flags[a.g.idx(x, y, z)];
        if (f & F_PROJ) t.word |= (unsigned)__popc(f & F_NBRS) << (16 + 3 * c);
    }
    if (yy == 0 && box.has(SIDE_YM, a)) t.word |= 1u << 24;
    if (yy == box.by - 1 && box.has(SIDE_YP, a)) t.word |= 1u << 25;
    if (zz == 0 && box.has(SIDE_ZM, a)) t.word |= 1u << 26;
    if (zz == box.bz - 1 && box.has(SIDE_ZP, a)) t.word |= 1u << 27;
    t.send = (unsigned)(zz * a.hx + h) | ((unsigned)(yy * a.hx + h) << 16);
    return t;
}

// Receive: element k of this thread's share of the neighbours' sides: where it is in the exchange
// buffer, and the element of shared memory (colour row 0) it goes to; `to` gives the latter for
// (side, row of the side, h).
template <int RT, int NR, typename To>
__device__ __forceinline__ void make_receives(const ResidentArgs& a, const Box& box, unsigned (&from)[NR], unsigned (&dst)[NR],
                                              To to) {
#pragma unroll
    for (int k = 0; k < NR; ++k) from[k] = SLOT_NONE, dst[k] = 0u;
    int first = 0;
    for (unsigned side = 0; side < 4; ++side) {
        if (!box.has(side, a)) continue;
        const int n = box.rows(side) * a.hx;
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            const int i = (int)threadIdx.x + k * RT - first;
            if (i < 0 || i >= n) continue;
            const int row = i / a.hx, h = i - row * a.hx;
            from[k] = (unsigned)(box_base(a, box.across(side, a)) + (size_t)(side_base(a, side ^ 1u) + i));
            dst[k] = to(side, row, h);
        }
        first += n;
    }
}

// Poll this thread's elements of pass `pass` and hand each to `put(k, value)`.
template <int NR, typename Put>
__device__ __forceinline__ bool receive(const ResidentArgs& a, const unsigned long long* ex, const unsigned (&from)[NR],
                                        unsigned pass, Put put) {
    unsigned left = 0u;
#pragma unroll
    for (int k = 0; k < NR; ++k)
        if (from[k] != SLOT_NONE) left |= 1u << k;
    for (unsigned n = 0; left != 0u; ++n) {
        unsigned long long x[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k)
            if (left & (1u << k)) x[k] = ex_load(ex + from[k]);
#pragma unroll
        for (int k = 0; k < NR; ++k)
            if ((left & (1u << k)) && (unsigned)(x[k] >> 32) == pass) {
                put(k, __uint_as_float((unsigned)x[k]));
                left &= ~(1u << k);
            }
        if (n >= RES_POLLS || ((n & 1023u) == 1023u && *(volatile const int*)a.kerr != 0)) return left == 0u;
    }
    return true;
}

__device__ __forceinline__ void send_sides(const ResidentArgs& a, unsigned long long* mine, const Slot& t, unsigned pass,
                                           float ym, float yp, float zm, float zp) {
    const unsigned ey = t.send & 0xffffu, ez = t.send >> 16;
    if (t.word & (1u << 24)) ex_put(mine + side_base(a, SIDE_YM) + ey, ym, pass);
    if (t.word & (1u << 25)) ex_put(mine + side_base(a, SIDE_YP) + ey, yp, pass);
    if (t.word & (1u << 26)) ex_put(mine + side_base(a, SIDE_ZM) + ez, zm, pass);
    if (t.word & (1u << 27)) ex_put(mine + side_base(a, SIDE_ZP) + ez, zp, pass);
}

// ---- pressure form ----------------------------------------------------------------------------

// The red-black SOR of one grid, all sweeps, with the tolerance rule: P in place, the residual maxima and
// the decision in `status` as the other kernels leave them.  Shared memory: the box's rows with a ring
// of neighbour rows.
template <int RT, int NS, int NR>
__global__ void __launch_bounds__(RT, 1)
k_resident_sor(const __grid_constant__ ResidentArgs a, float* __restrict__ P, const float* __restrict__ b,
               const uint8_t* __restrict__ flags, const __grid_constant__ WAcc wa, int max_sweeps, int check_every,
               float tol, StepStatus* __restrict__ status) {
    extern __shared__ float sm[];
    __shared__ float wtab[8 * 32];  // omega/acc, one copy per lane
    constexpr bool GATHER = RT * NS <= 4096;
    __shared__ unsigned red[RT / 32];
    __shared__ unsigned red2[GATHER ? RT / 32 : 1], all;  // GATHER: every box's maxima, the result
    const Grid g = a.g;
    const Box box(a);
    const int tid = (int)threadIdx.x, lane = tid & 31;
    const int ry = box.by + 2, HP = a.hp, rowstep = 2 * HP, planestep = ry * rowstep;

    for (int i = tid; i < 8 * 32; i += RT) wtab[i] = wa.w[i >> 5];
    for (int i = tid, n = ry * (box.bz + 2) * g.nx; i < n; i += RT) {
        const int r = i / g.nx, x = i - r * g.nx, zz = r / ry, y = box.y0 - 1 + r - zz * ry, z = box.z0 - 1 + zz;
        sm[(2 * r + ((x + y + z) & 1)) * HP + (x >> 1)] = P[g.idx(x, y, z)];
    }
    Slot slot[NS];
    float bv[NS][2];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        slot[s] = make_slot(a, box, tid + s * RT, ry, 1, flags);
        bv[s][0] = bv[s][1] = 0.0f;
        const unsigned w = slot[s].word;
        const int e = (int)(w & 0xffffu), r = e / rowstep, h = e - r * rowstep, zz = r / ry;
        const int i0 = g.idx(0, box.y0 - 1 + r - zz * ry, box.z0 - 1 + zz), p = (int)(w >> 22) & 1;
        if (w & (7u << 16)) bv[s][0] = b[i0 + 2 * h + p];
        if (w & (7u << 19)) bv[s][1] = b[i0 + 2 * h + (p ^ 1)];
    }
    unsigned from[NR], dst[NR];
    make_receives<RT, NR>(a, box, from, dst, [&](unsigned side, int row, int h) {
        const int r = side == SIDE_YM ? (row + 1) * ry : side == SIDE_YP ? (row + 1) * ry + box.by + 1
                    : side == SIDE_ZM ? row + 1 : (box.bz + 1) * ry + row + 1;
        return (unsigned)(r * rowstep + h);
    });
    unsigned long long* const mine = a.ex + box_base(a, box.cta);
    const int ctas = a.cy * a.cz;
    unsigned long long* const maxima = a.ex + 2 * (size_t)a.half;

    // fma(-acc, P, b + sum) of a cell of colour c: the kernels' residual
    auto residual = [&](unsigned w, int c, unsigned acc, float bc, float& pc) {
        const float* own = sm + (w & 0xffffu) + c * HP;
        const float* row = own + (c == 0 ? HP : -HP) + (int)(((w >> 22) ^ (unsigned)c) & 1u);  // x + 1 = 2 h + s + 1
        const float sx = row[-1] + row[0], sy = own[(c == 0 ? HP : -HP) - rowstep] + own[(c == 0 ? HP : -HP) + rowstep],
                    sz = own[(c == 0 ? HP : -HP) - planestep] + own[(c == 0 ? HP : -HP) + planestep];
        pc = own[0];
        // -acc: acc in bits 20..22 of the mantissa of 8.0f counts ones
        return fmaf(8.0f - __uint_as_float((acc << 20) | 0x41000000u), pc, bc + ((sx + sy) + sz));
    };

    __syncthreads();
    unsigned pass = 0;
    int group = 0;
    bool bad = false;
    for (int sweep = 0; sweep < max_sweeps && !bad; ++sweep) {
        if (tol != 0.0f && sweep % check_every == 0) {  // below 0: residuals are recorded and end nothing
            unsigned m = 0u;
#pragma unroll
            for (int s = 0; s < NS; ++s)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const unsigned w = slot[s].word, acc = (w >> (16 + 3 * c)) & 7u;
                    float pc;
                    if (acc) m = max(m, __float_as_uint(fabsf(residual(w, c, acc, bv[s][c], pc))));
                }
            const unsigned tag = (unsigned)group + 1u;
            unsigned long long* at = maxima + (size_t)(group & 1) * ctas;
            if constexpr (GATHER) {
                // Box 0 gathers every box's maximum and hands the result out in one word: with every box polling
                // every other's, the polls of 144 boxes met at the same lines (5.5 us a check at 32^3, 1.8 now).  The
                // sweeps' barriers lie between the uses of `red` and `all` by two checks.
                auto warps = [&](const unsigned* r) {
                    return __reduce_max_sync(0xffffffffu, lane < RT / 32 ? r[lane] : 0u);
                };
                unsigned long long* const verdict = maxima + 2 * (size_t)ctas + (group & 1);
                m = __reduce_max_sync(0xffffffffu, m);
                if (lane == 0) red[tid >> 5] = m;
                __syncthreads();
                if (tid < 32) {
                    m = warps(red);
                    if (tid == 0) ex_put(at + box.cta, __uint_as_float(m), tag);
                }
                if (box.cta == 0) {
                    const unsigned one[1] = {tid < ctas ? (unsigned)tid : SLOT_NONE};
                    m = 0u;
                    bad = !receive<1>(a, at, one, tag, [&](int, float v) { m = __float_as_uint(v); });
                    m = __reduce_max_sync(0xffffffffu, m);
                    if (lane == 0) red2[tid >> 5] = m;
                    bad = __syncthreads_or(bad);
                    if (tid < 32 && !bad) {
                        m = warps(red2);
                        if (tid == 0) {
                            ex_put(verdict, __uint_as_float(m), tag);
                            all = m;
                        }
                    }
                } else if (tid == 0) {
                    const unsigned one[1] = {0u};
                    bad = !receive<1>(a, verdict, one, tag, [&](int, float v) { all = __float_as_uint(v); });
                }
                bad = __syncthreads_or(bad);
                if (bad) break;
                m = all;
            } else {
                // every box polls every other's: the gather's code costs the sweeps of this form its registers
                // (127^3 without checks 232 -> 236 us, a check 6.5 -> 5.2)
                for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (lane == 0) red[tid >> 5] = m;
                __syncthreads();
                if (tid == 0) {
                    for (int k = 1; k < RT / 32; ++k) m = max(m, red[k]);
                    ex_put(at + box.cta, __uint_as_float(m), tag);
                }
                unsigned one[1] = {tid < ctas ? (unsigned)tid : SLOT_NONE};
                m = 0u;
                bad = !receive<1>(a, at, one, tag, [&](int, float v) { m = __float_as_uint(v); });
                for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
                __syncthreads();  // red has been read
                if (lane == 0) red[tid >> 5] = m;
                bad = __syncthreads_or(bad);
                if (bad) break;
                for (int k = 0; k < RT / 32; ++k) m = max(m, red[k]);
            }
            const bool done = __uint_as_float(m) <= tol;
            if (box.cta == 0 && tid == 0) {
                status->rmax_bits[group] = m;
                if (done) {
                    status->done = 1;
                    status->done_group = group;
                }
            }
            if (done) break;
            ++group;
            if constexpr (!GATHER) __syncthreads();
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (bad) break;
            ++pass;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const unsigned w = slot[s].word, acc = (w >> (16 + 3 * c)) & 7u;
                float pc;
                const float r = residual(w, c, acc, bv[s][c], pc);
                const float v = acc ? fmaf(wtab[acc * 32 + lane], r, pc) : pc;
                if (acc) sm[(w & 0xffffu) + c * HP] = v;
                if (w >> 24) send_sides(a, mine + (size_t)c * a.half, slot[s], pass, v, v, v, v);
            }
            bad = !receive<NR>(a, a.ex + (size_t)c * a.half, from, pass, [&](int k, float v) { sm[dst[k] + c * HP] = v; });
            bad = __syncthreads_or(bad);
        }
    }
    if (bad && tid == 0) atomicExch(a.kerr, 1);
    __syncthreads();
    for (int i = tid, n = box.by * box.bz * g.nx; i < n; i += RT) {
        const int r = i / g.nx, x = i - r * g.nx, zz = r / box.by, yy = r - zz * box.by, y = box.y0 + yy, z = box.z0 + zz;
        P[g.idx(x, y, z)] = sm[(2 * ((zz + 1) * ry + yy + 1) + ((x + y + z) & 1)) * HP + (x >> 1)];
    }
}

// ---- velocity form ------------------------------------------------------------------------------

// The reference scheme's red-black passes (k_project_velocity) on u, v, w in place.  Shared memory: the
// three lower faces of every position of the box, the v faces of the rows above it and the w faces of
// the plane above; a side's faces are held by both boxes that touch them, and whichever updated one
// in a pass sends it.
template <int RT, int NS, int NR>
__global__ void __launch_bounds__(RT, 1)
k_resident_vel(const __grid_constant__ ResidentArgs a, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
               const uint8_t* __restrict__ flags, int iterations, const __grid_constant__ OmegaSplit os, double omega) {
    extern __shared__ float sm[];
    __shared__ float2 ztab[8 * 32];  // zh, zl by acc, one copy per lane
    const Grid g = a.g;
    const Box box(a);
    const int tid = (int)threadIdx.x, lane = tid & 31;
    constexpr int GB = NS < 4 ? NS : 4;
    const int HP = a.hp, rowstep = 2 * HP;
    const int yrows = box.by + 1;  // rows of v per plane
    float* const su = sm;
    float* const sv = su + box.by * box.bz * rowstep;
    float* const sw = sv + yrows * box.bz * rowstep;

    for (int i = tid; i < 8 * 32; i += RT) {
        const int acc = i >> 5;
        const DivSplit z = div_split(acc < 1 ? 1 : acc > 6 ? 6 : acc);
        ztab[i] = make_float2(z.zh, z.zl);
    }
    const int px = g.nx + 1;
    auto load = [&](float* to, const float* fr, int rows, int planes) {
        for (int i = tid, n = rows * planes * px; i < n; i += RT) {
            const int r = i / px, x = i - r * px, zz = r / rows, y = box.y0 + r - zz * rows, z = box.z0 + zz;
            to[(2 * r + ((x + y + z) & 1)) * HP + (x >> 1)] = fr[g.idx(x, y, z)];
        }
    };
    load(su, u, box.by, box.bz);
    load(sv, v, yrows, box.bz);
    load(sw, w, box.by, box.bz + 1);
    Slot slot[NS];
    unsigned open[NS];  // neighbour bits (six each) of the two colours, 0 where not projectable
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        slot[s] = make_slot(a, box, tid + s * RT, box.by, 0, flags);
        open[s] = 0u;
        const unsigned wd = slot[s].word;
        const int e = (int)(wd & 0xffffu), r = e / rowstep, h = e - r * rowstep, zz = r / box.by;
        const int i0 = g.idx(0, box.y0 + r - zz * box.by, box.z0 + zz), p = (int)(wd >> 22) & 1;
        if (wd & (7u << 16)) open[s] |= (flags[i0 + 2 * h + p] >> 1) & 63u;
        if (wd & (7u << 19)) open[s] |= ((flags[i0 + 2 * h + (p ^ 1)] >> 1) & 63u) << 6;
        open[s] |= (unsigned)zz << 12;  // v has one row more per plane: its element is zz rows further
    }
    // what a neighbour sends: the faces between the boxes, as elements of v (y sides) or w (z sides); the
    // one below updates them through its upper faces (positions of the other colour), the one above
    // through its own
    unsigned from[NR], dst[NR];
    make_receives<RT, NR>(a, box, from, dst, [&](unsigned side, int row, int h) {
        const int base = side == SIDE_YM ? row * yrows * rowstep : side == SIDE_YP ? (row * yrows + box.by) * rowstep
                       : side == SIDE_ZM ? row * rowstep : (box.bz * box.by + row) * rowstep;
        const int at = (int)((side < SIDE_ZM ? sv : sw) - sm) + base + h;
        return (unsigned)at | ((side == SIDE_YM || side == SIDE_ZM) ? 0x80000000u : 0u);
    });
    unsigned long long* const mine = a.ex + box_base(a, box.cta);
    __syncthreads();

    bool bad = false;
    const int H = 2 * iterations;
    for (int p2 = 0; p2 < H && !bad; p2 += 2) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (bad) break;
            const unsigned pass = (unsigned)(p2 + c + 1);
#pragma unroll
            for (int s0 = 0; s0 < NS; s0 += GB) {
                // the cells of a pass do not read each other's faces: the loads of a group of slots are
                // issued together
                float f[GB][6];
#pragma unroll
                for (int k = 0; k < GB; ++k)
                    if (s0 + k < NS) {
                        const unsigned wd = slot[s0 + k].word;
                        const int o = c == 0 ? HP : -HP;
                        const float* pu = su + (wd & 0xffffu) + c * HP;
                        const float* pv = pu + (sv - su) + (int)(open[s0 + k] >> 12) * rowstep;
                        const float* pw = pu + (sw - su);
                        f[k][0] = pu[0];
                        f[k][1] = pu[o + (int)(((wd >> 22) ^ (unsigned)c) & 1u)];
                        f[k][2] = pv[0];
                        f[k][3] = pv[o + rowstep];
                        f[k][4] = pw[0];
                        f[k][5] = pw[o + box.by * rowstep];
                    }
#pragma unroll
                for (int k = 0; k < GB; ++k)
                    if (s0 + k < NS) {
                        const unsigned wd = slot[s0 + k].word, acc = (wd >> (16 + 3 * c)) & 7u;
                        const unsigned nb = open[s0 + k] >> (6 * c);
                        float uc = f[k][0], ux = f[k][1], vc = f[k][2], vy = f[k][3], wc = f[k][4], wz = f[k][5];
                        const float x = -(-uc + ux + -vc + vy + -wc + wz);
                        const float2 z = ztab[acc * 32 + lane];
                        const float q = div_fast(x, z.x, z.y);
                        const float rest = scale_rest(q, os);
                        float pt = fmaf(q, os.wh, rest);
                        const bool rare = acc && (es_rare(x) || (!os.rational && !scale_sure(q, rest, os)));
                        if (__any_sync(0xffffffffu, rare))
                            pt = cell_pt_rare(pt, rare, x, ((nb & 63u) << 8) | (acc ? ES_ENTRY_PROJ : 0u), z.x, z.y, os,
                                              omega);
                        if (acc) {
                            // u -= p_t * s(x - 1) and so on: the product with 0 keeps its sign
                            const float z0 = pt * 0.0f;
                            uc = uc - ((nb & 1u) ? pt : z0);
                            ux = ux + ((nb & 2u) ? pt : z0);
                            vc = vc - ((nb & 4u) ? pt : z0);
                            vy = vy + ((nb & 8u) ? pt : z0);
                            wc = wc - ((nb & 16u) ? pt : z0);
                            wz = wz + ((nb & 32u) ? pt : z0);
                            const int o = c == 0 ? HP : -HP;
                            float* pu = su + (wd & 0xffffu) + c * HP;
                            float* pv = pu + (sv - su) + (int)(open[s0 + k] >> 12) * rowstep;
                            float* pw = pu + (sw - su);
                            pu[0] = uc;
                            pu[o + (int)(((wd >> 22) ^ (unsigned)c) & 1u)] = ux;
                            pv[0] = vc;
                            pv[o + rowstep] = vy;
                            pw[0] = wc;
                            pw[o + box.by * rowstep] = wz;
                        }
                        if (wd >> 24) send_sides(a, mine + (size_t)c * a.half, slot[s0 + k], pass, vc, vy, wc, wz);
                    }
            }
            bad = !receive<NR>(a, a.ex + (size_t)c * a.half, from, pass, [&](int k, float val) {
                sm[(dst[k] & 0x7fffffffu) + ((dst[k] >> 31) ^ (unsigned)c) * HP] = val;
            });
            bad = __syncthreads_or(bad);
        }
    }
    if (bad && tid == 0) atomicExch(a.kerr, 1);
    __syncthreads();
    // positions of the box, and where it ends the interior the faces beyond it
    auto store = [&](const float* fr, float* to, int rows, int planes, int own_rows, int own_planes) {
        for (int i = tid, n = rows * planes * px; i < n; i += RT) {
            const int r = i / px, x = i - r * px, zz = r / rows, yy = r - zz * rows, y = box.y0 + yy, z = box.z0 + zz;
            if (yy < own_rows && zz < own_planes) to[g.idx(x, y, z)] = fr[(2 * r + ((x + y + z) & 1)) * HP + (x >> 1)];
        }
    };
    store(su, u, box.by, box.bz, box.by, box.bz);
    store(sv, v, yrows, box.bz, box.iy + 1 < a.cy ? box.by : yrows, box.bz);
    store(sw, w, box.by, box.bz + 1, box.by, box.iz + 1 < a.cz ? box.bz : box.bz + 1);
}

// ---- host side ------------------------------------------------------------------------------------

// Threads and cells of one colour per thread: 512 threads (128 registers) up to 4 cells, then 1024 (64
// registers; twice the warps to hide a pass's latencies: 127^3, 14 cells of 512 threads 5.4 us a
// pass, 7 of 1024 3.8; 64^3 the other way round, 1.1 and 1.2).
struct ResShape {
    int rt, ns;
};
constexpr ResShape RES_SHAPES[] = {{512, 1}, {512, 2}, {512, 4}, {1024, 4}, {1024, 7}};
constexpr int RES_NR = 3;  // received elements per thread

size_t res_smem(const ResidentPlan& p, bool velocity) {
    const size_t row = 2 * sizeof(float) * (size_t)p.hp;
    return velocity ? row * ((size_t)3 * p.by * p.bz + p.bz + p.by) : row * (size_t)(p.by + 2) * (size_t)(p.bz + 2);
}

ResidentArgs res_args(const Grid& g, const ResidentPlan& p, void* ex, int* kerr) {
    ResidentArgs a;
    a.g = g;
    a.by = p.by;
    a.bz = p.bz;
    a.cy = p.cy;
    a.cz = p.cz;
    a.hx = p.hx;
    a.hp = p.hp;
    a.sy = p.bz * p.hx;
    a.sz = p.by * p.hx;
    a.half = p.cy * p.cz * 2 * (a.sy + a.sz);
    a.ex = static_cast<unsigned long long*>(ex);
    a.kerr = kerr;
    return a;
}

template <int RT, int NS>
int res_launch_sor(const ResidentArgs& a, const ResidentPlan& p, float* P, const float* b, const uint8_t* flags,
                   const WAcc& wa, int max_sweeps, int check_every, float tol, StepStatus* status, cudaStream_t st) {
    void* args[] = {(void*)&a, (void*)&P, (void*)&b, (void*)&flags, (void*)&wa, (void*)&max_sweeps, (void*)&check_every,
                    (void*)&tol, (void*)&status};
    return (int)cudaLaunchCooperativeKernel((const void*)k_resident_sor<RT, NS, RES_NR>, dim3((unsigned)(p.cy * p.cz)),
                                            dim3(RT), args, res_smem(p, false), st);
}

template <int RT, int NS>
int res_launch_vel(const ResidentArgs& a, const ResidentPlan& p, float* u, float* v, float* w, const uint8_t* flags,
                   int iterations, const OmegaSplit& os, double omega, cudaStream_t st) {
    void* args[] = {(void*)&a, (void*)&u, (void*)&v, (void*)&w, (void*)&flags, (void*)&iterations, (void*)&os, (void*)&omega};
    return (int)cudaLaunchCooperativeKernel((const void*)k_resident_vel<RT, NS, RES_NR>, dim3((unsigned)(p.cy * p.cz)),
                                            dim3(RT), args, res_smem(p, true), st);
}

}  // namespace

bool resident_plan(const Grid& g, bool velocity, int sms, ResidentPlan* out) {
    const int iy = g.ny - 2, iz = g.nz - 2;
    if (g.nx < 3 || iy < 1 || iz < 1 || sms < 1) return false;
    if (sms > 512) sms = 512;  // a CTA's threads poll one maximum each
    float best = 0.0f;
    bool found = false;
    for (int c = 1; c <= std::min(iy, sms); ++c) {
        ResidentPlan p;
        p.by = (iy + c - 1) / c;
        p.cy = (iy + p.by - 1) / p.by;
        const int cz = std::min(iz, sms / p.cy);
        if (cz < 1) continue;
        p.bz = (iz + cz - 1) / cz;
        p.cz = (iz + p.bz - 1) / p.bz;
        p.hx = g.nx / 2;
        p.hp = g.nx / 2 + 1;
        const long long cells = (long long)p.by * p.bz * p.hx, halo = 2LL * (p.by + p.bz) * p.hx;
        p.ns = 0;
        for (const ResShape& r : RES_SHAPES)
            if (p.ns == 0 && cells <= (long long)r.rt * r.ns && halo <= (long long)r.rt * RES_NR) {
                p.rt = r.rt;
                p.ns = r.ns;
            }
        if (p.ns == 0 || std::max(p.by, p.bz) * (long long)p.hx > 65535) continue;
        if (res_smem(p, velocity) > RES_SMEM || res_smem(p, velocity) / sizeof(float) > 65535) continue;
        // a pass costs its slots, and its sides' elements once more to send and receive
        const float cost = (float)((cells + p.rt - 1) / p.rt * p.rt) + (float)halo;
        if (!found || cost < best) {
            found = true;
            best = cost;
            *out = p;
        }
    }
    return found;
}

size_t resident_exchange_bytes(const ResidentPlan& p) {
    const size_t ctas = (size_t)p.cy * (size_t)p.cz;
    return (2 * ctas * 2 * (size_t)(p.by + p.bz) * (size_t)p.hx + 2 * ctas + 2) * sizeof(unsigned long long);
}

int prepare_resident_kernels() {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    bool ok = true;
    if (smem_attribute_set((const void*)k_resident_vel<1024, 7, RES_NR>, (int)RES_SMEM)) return 0;
#define SMK_RES_ATTR(RT, NS)                                                                                          \
    ok = ok && cudaFuncSetAttribute(k_resident_sor<RT, NS, RES_NR>, at, (int)RES_SMEM) == cudaSuccess &&                \
         cudaFuncSetAttribute(k_resident_vel<RT, NS, RES_NR>, at, (int)RES_SMEM) == cudaSuccess
    SMK_RES_ATTR(512, 1);
    SMK_RES_ATTR(512, 2);
    SMK_RES_ATTR(512, 4);
    SMK_RES_ATTR(1024, 4);
    SMK_RES_ATTR(1024, 7);
#undef SMK_RES_ATTR
    return ok ? 0 : -1;
}

int launch_resident_sor(const Grid& g, const ResidentPlan& p, void* ex, int* kerr, float* P, const float* b,
                        const uint8_t* flags, const float* wacc7, int max_sweeps, int check_every, float tol,
                        StepStatus* status, cudaStream_t st) {
    const ResidentArgs a = res_args(g, p, ex, kerr);
    WAcc wa;
    for (int k = 0; k < 7; ++k) wa.w[k] = wacc7[k];
    wa.w[7] = 0.0f;
    if (p.rt == 1024)
        return p.ns == 4 ? res_launch_sor<1024, 4>(a, p, P, b, flags, wa, max_sweeps, check_every, tol, status, st)
                         : res_launch_sor<1024, 7>(a, p, P, b, flags, wa, max_sweeps, check_every, tol, status, st);
    switch (p.ns) {
        case 1: return res_launch_sor<512, 1>(a, p, P, b, flags, wa, max_sweeps, check_every, tol, status, st);
        case 2: return res_launch_sor<512, 2>(a, p, P, b, flags, wa, max_sweeps, check_every, tol, status, st);
        default: return res_launch_sor<512, 4>(a, p, P, b, flags, wa, max_sweeps, check_every, tol, status, st);
    }
}

int launch_resident_vel(const Grid& g, const ResidentPlan& p, void* ex, int* kerr, float* u, float* v, float* w,
                        const uint8_t* flags, int iterations, double omega, cudaStream_t st) {
    const ResidentArgs a = res_args(g, p, ex, kerr);
    const OmegaSplit os = omega_split(omega);
    if (p.rt == 1024)
        return p.ns == 4 ? res_launch_vel<1024, 4>(a, p, u, v, w, flags, iterations, os, omega, st)
                         : res_launch_vel<1024, 7>(a, p, u, v, w, flags, iterations, os, omega, st);
    switch (p.ns) {
        case 1: return res_launch_vel<512, 1>(a, p, u, v, w, flags, iterations, os, omega, st);
        case 2: return res_launch_vel<512, 2>(a, p, u, v, w, flags, iterations, os, omega, st);
        default: return res_launch_vel<512, 4>(a, p, u, v, w, flags, iterations, os, omega, st);
    }
}

}  // namespace smk
