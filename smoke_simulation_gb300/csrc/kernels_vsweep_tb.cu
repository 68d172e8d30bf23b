// Temporally blocked red-black SOR of the reference scheme: the reference's in-place velocity
// projection (project/smokeSimulation.cu:356-394, 30 iterations per step at :795-801) with T
// colour passes per pass over HBM, bit-exact with one pass per launch (k_project_velocity).
//
// The reference's pass over colour c updates every interior fluid cell with (x + y + z + c) even
// and at least one fluid neighbour: from its six faces, div = -u_x + u_x+1 + -v_y + v_y+1 + -w_z
// + w_z+1 (left to right), p_t = float(double(-div / acc) * omega), and then
// u_x -= p_t*s(x-1), u_x+1 += p_t*s(x+1), v_y -= p_t*s(y-1), v_y+1 += p_t*s(y+1), w_z -= p_t*s(z-1),
// w_z+1 += p_t*s(z+1).  Within a pass no two updated cells share a face, so every face changes at
// most once per pass, and a face between cells a (below/left) and b is changed either by b
// ("own" lower face) or by a (b's face as a's upper face): the value sequence of each face is
// fixed by the pass order alone.
//
// Decomposition (as the pressure-form kernel, kernels_sweep_tb.cu): a CTA of 32 x TY threads
// owns an x-y tile of 64 x 2TY face-grid positions (position i holds the three lower faces u_i,
// v_i, w_i of cell i, the library's shared index) and a z-range, and marches z: at iteration q it
// takes plane q and applies pass t (t = 1..T) to plane q - t.  Each thread owns a 2 x 2 patch
// (columns A = x0, B = x0+1 with x0 even; rows y0, y0+1 with y0 even), so the cells a pass
// updates are A of one row and B of the other, uniformly over the CTA and the same for every
// stage of an iteration.  Pass t on plane p reads faces of planes p and p+1 and writes faces of
// planes p and p+1 (w_z+1), which the same thread holds: the z-ring lives in registers (T + 2
// planes: the plane being loaded, T planes in passes, and the finished plane waiting for its last
// update from above).  In-plane:
//   - x: a B cell's u_x+1 is the next lane's A value (shuffle down); the A cell right of an updated
//     B receives p_t * s through a shuffle up within the same pass;
//   - y: an updated last-row cell reads the v of the thread below's row 0 at the previous pass's
//     end, published in shared memory at the previous iteration; the row-0 cell below an updated
//     last-row cell receives p_t * s one iteration later (the thread above publishes p_t, the
//     receiver applies it before its next pass on that plane: nothing reads that face in between).
// So one barrier per iteration (double-buffered published planes) suffices.  Predicates: a face
// changes only when its updating cell is projectable (the flag byte's bit 7); the receiver of a
// cross-thread update reads the sender's projectable bit from the flag boxes when it loads the
// plane (left neighbour: a shuffle of the flag word; row above: the shared-memory flag box).
//
// Halo, windows and the TMA ring with bounded mbarrier waits are those of the pressure form
// (tb_common.cuh); positions that no pass changes (the boundary ring and everything outside the grid)
// make windows that reach the grid's edge need no halo there.  A launch reads u, v, w and the flags and
// writes u, v, w to a second set of face arrays (the simulation's pressure and rhs buffers, unused by
// this scheme): 25 bytes per position for T/2 iterations.
//
// Arithmetic.  p_t = float(double(-div / acc) * omega) costs five FP32 multiplies and FMAs
// (exact_scale.cuh); a face update is one predicated add; the divergence and the product of a
// thread's two cells are packed FP32 pairs.  Operands that need more go through cell_pt_rare, out of
// line so that its code stays out of the unrolled march (inlined, instruction fetches made a launch
// 15 % slower).
//
// What bounds it: instruction issue (256^3, T = 4, z-chunk 52: 171 us a launch, 61 % of the issue
// slots busy over two uneven waves, 70 % while active; ~120 warp instructions per two cells and pass, halo included;
// HBM at 32 %).  256^3, 30 iterations: one pass per launch 5.20 ms (86.7 us a pass, 0.73 of the
// measured HBM bandwidth and 48 % of the FP64 pipe), T = 4 2.60 ms, T = 2 3.1 ms.  The former form
// (integer 24 x 53-bit product, both corrections and the FP64 path evaluated for every cell) took
// 9.8 ms with T = 4.  Not kept: multipliers 0 / 1 per face from a shared table instead of predicated
// adds (L1 at 72 %, 3.5 ms); passes left out for warps outside a pass's cone (3.8 ms: the branches
// stop the compiler from interleaving the passes).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstring>

#include "common.cuh"
#include "exact_scale.cuh"
#include "kernels.h"
#include "tb_common.cuh"

namespace smk {

namespace {

using namespace tb;

// Tile geometry: TY warps (tile rows of threads) of 2-row patches, ROWS = 2 TY face-grid rows, one CTA
// per SM.  T = 4 holds six planes of three fields in registers (128 a thread: 16 warps); T = 2 holds four
// (80: 24 warps, whose 48-row tile keeps 0.86 of its cells as owned instead of 0.78 with 24 rows).
template <int TY>
struct VTGeom {
    static constexpr int ROWS = 2 * TY;
    static constexpr int BOX_F_BYTES = ROWS * BOX_F * 4;          // one float box
    static constexpr int BOX_B_BYTES = ROWS * BOX_U8;             // the flag box
    static constexpr int STAGE = 3 * BOX_F_BYTES + BOX_B_BYTES;   // u, v, w, flags of one plane
    static constexpr int PROW = (TY + 2) * TX;                    // floats per published plane
    static constexpr int THREADS = TX * TY;
    static constexpr int MAPS = TY == 16 ? 0 : 1;                 // tensor-map set (box height)
    static_assert(STAGE % 128 == 0, "TMA destinations stay 128-byte aligned");
};

struct VMaps {
    CUtensorMap u, v, w, f;
};

// ---- one pass on one cell ----------------------------------------------------------------------

// A cell's ring entry is 16 bits, the byte offset of its quotient's zh, zl (exact_scale.cuh) in a
// shared table with one copy per lane: (f >> 1 & 127) * 256 + lane * 8 for the flag byte f, so that
// a warp's 8-byte reads never meet in a bank whatever its flag bytes are.  The neighbour bits and the
// projectable bit are tested in place:
enum : unsigned {
    C_XM = 1u << 8, C_XP = 1u << 9, C_YM = 1u << 10, C_YP = 1u << 11, C_ZM = 1u << 12, C_ZP = 1u << 13,
    C_PROJ = 1u << 14,
};
constexpr int COEF_BYTES = 128 * 256;

__device__ __forceinline__ unsigned cell_entry(unsigned f, unsigned lane8) { return ((f & 0xfeu) << 7) | lane8; }

// Faces of an updated cell.  The reference adds p_t * s with s = 0 or 1; a face with s = 1 (open)
// takes one predicated add.  With s = 0 the product is a zero, which changes nothing but a face
// that holds -0 (-0 + +0 = +0): closed faces are visited only by warps that hold a -0 somewhere
// (`neg0`; no update makes one from other values).  pl is p_t, or +0 on a cell that is not
// projectable, pu the same with -0: u - +0 and u + -0 leave every u as it is.
__device__ __forceinline__ void face_lower(unsigned c, unsigned bit, float pl, float& u) {
    if (c & bit) u = u - pl;
}
__device__ __forceinline__ void face_upper(unsigned c, unsigned bit, float pu, float& u) {
    if (c & bit) u = u + pu;
}
__device__ __forceinline__ void closed_lower(unsigned c, unsigned bit, float p, float& u) {
    if ((c & (bit | C_PROJ)) == C_PROJ) u = u - p * 0.0f;
}
__device__ __forceinline__ void closed_upper(unsigned c, unsigned bit, float p, float& u) {
    if ((c & (bit | C_PROJ)) == C_PROJ) u = u + p * 0.0f;
}
// What an upper face held by another thread receives: p_t * s, or -0 from a cell that is not projectable.
__device__ __forceinline__ float face_sent(unsigned c, unsigned bit, float pu) { return (c & bit) ? pu : pu * 0.0f; }

// One tile of a launch: T colour passes (nhalf of them when not FULL) starting at colour0.
//
// A thread's 2 x 2 patch is held as two pairs per field, E = (A0, B1) and O = (B0, A1): one
// pattern updates the cells of E, the other those of O, and the divergence and the product of both
// cells are packed FP32 pairs (one issue slot for two cells).
template <int T, int TY, bool FULL>
__device__ __forceinline__ void vsweep_tile(const VMaps& maps, const Grid& g, float* __restrict__ uo,
                                            float* __restrict__ vo, float* __restrict__ wo, int nhalf,
                                            int colour0, int zchunk, const OmegaSplit& os, double omega,
                                            int* __restrict__ kerr) {
    using G = VTGeom<TY>;
    constexpr int VT_STAGE = G::STAGE, VT_BOX_F = G::BOX_F_BYTES, VT_PROW = G::PROW, VT_THREADS = G::THREADS,
                  VT_ROWS = G::ROWS;
    constexpr int R = T + 2;   // register ring: planes q-1-T .. q
    constexpr int S = R / 2;   // TMA stages (stage and phase fixed per unrolled iteration)
    constexpr int NPUB = 2 * (T + 1);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* stages = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    float* pub = reinterpret_cast<float*>(stages + S * VT_STAGE);
    unsigned char* ctab = reinterpret_cast<unsigned char*>(pub + 2 * NPUB * VT_PROW);
    __shared__ __align__(8) uint64_t mbar[S];

    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = ty * TX + tx;
    const bool leader = tid == 0;
    for (int i = tid; i < 128 * TX; i += VT_THREADS) {
        const int acc = __popc((unsigned)((i / TX) & 63));
        const DivSplit z = div_split(acc < 1 ? 1 : acc);
        reinterpret_cast<float2*>(ctab)[i] = make_float2(z.zh, z.zl);
    }
    // the padding rows of every published plane (never written afterwards): nothing received from
    // above the tile (adding -0 leaves a face as it is), and any value below it
    for (int i = tid; i < 2 * NPUB * 2 * TX; i += VT_THREADS) {
        const int lane = i % TX, edge = (i / TX) % 2, set = i / (2 * TX);
        pub[set * VT_PROW + (edge ? (TY + 1) * TX : 0) + lane] = -0.0f;
    }

    // windows over the face grid: (nx+1) x (ny+1) positions, planes 0..nz
    int X0, xlo, xhi, Y0, ylo, yhi;
    sweep_window(g.nx + 1, 2 * TX, T, (int)blockIdx.x, X0, xlo, xhi);
    sweep_window(g.ny + 1, VT_ROWS, T, (int)blockIdx.y, Y0, ylo, yhi);
    const int xf = X0 - (X0 & 3);    // 16-byte aligned float box start
    const int xb = X0 - (X0 & 15);   // 16-byte aligned flag box start
    const int of = X0 - xf + 2 * tx;
    const int ob = X0 - xb + 2 * tx;
    const int x0 = X0 + 2 * tx;
    const int y0 = Y0 + 2 * ty;
    const int za = (int)blockIdx.z * zchunk;
    const int zb = min(za + zchunk, g.nz + 1);
    const bool inx = x0 >= xlo && x0 < xhi;
    bool in[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) in[r] = inx && y0 + r >= ylo && y0 + r < yhi && y0 + r >= 0 && y0 + r <= g.ny;
    const int off0 = x0 + g.X * y0;

    // a plane q is finished at iteration q + 1 + T; planes below 0 are never changed and the
    // zero-initialised ring stands for them, so a chunk near z = 0 starts at plane 0
    const int qend = zb + T;
    int qbeg = za - T < 0 ? 0 : za - T;
    // start one plane lower where needed so that iteration k of every unrolled pass has the
    // update pattern of k's parity (fixed at compile time: one pattern's code per iteration); the
    // extra plane is one more halo plane (zero-filled below plane 0)
    qbeg -= (qbeg + colour0 - 1) & 1;
    const int qfinal = qend;  // last iteration executed

    auto issue = [&](int s, int z) {
        unsigned char* st = stages + s * VT_STAGE;
        const uint32_t bar = smem_u32(&mbar[s]);
        mbar_expect_tx(bar, (uint32_t)VT_STAGE);
        tma_load_3d(smem_u32(st), &maps.u, xf, Y0, z, bar);
        tma_load_3d(smem_u32(st + VT_BOX_F), &maps.v, xf, Y0, z, bar);
        tma_load_3d(smem_u32(st + 2 * VT_BOX_F), &maps.w, xf, Y0, z, bar);
        tma_load_3d(smem_u32(st + 3 * VT_BOX_F), &maps.f, xb, Y0, z, bar);
    };
    if (leader) {
        for (int s = 0; s < S; ++s) mbar_init(smem_u32(&mbar[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int s = 0; s < S && qbeg + s <= qfinal; ++s) issue(s, qbeg + s);
    }

    // slot = plane mod R; [0] = E = (A0, B1), [1] = O = (B0, A1)
    float2 U[2][R], V[2][R], W[2][R];
    unsigned ff[2][R];  // the pair's entries (cell_entry), the first cell's in the low half
    const unsigned lane8 = (unsigned)tx * 8u;
#pragma unroll
    for (int j = 0; j < R; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            U[e][j] = V[e][j] = W[e][j] = make_float2(0.f, 0.f);
            ff[e][j] = lane8 | (lane8 << 16);
        }
    }
    const int me0 = (ty + 1) * TX + tx;
    const float2 wh = make_float2(os.wh, os.wh), wl1 = make_float2(os.wl1, os.wl1), wl2 = make_float2(os.wl2, os.wl2);
    int par = 0;
    int neg0 = 0;  // iterations until the last plane with a -0 in this warp has left the ring
    __syncthreads();  // barriers initialised, table and padding visible

    for (int base = qbeg; base <= qend; base += R) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int q = base + k;
            if (q > qend) break;
            const int st = k % S;
            const uint32_t phase = (uint32_t)((k / S) & 1);
            // the pair every stage of this iteration updates: E on even k, O on odd k (qbeg)
            const int e = k & 1;
            float* cur = pub + par * NPUB * VT_PROW;              // written this iteration
            const float* prv = pub + (par ^ 1) * NPUB * VT_PROW;  // written by the last one

            // ---- plane q into slot k
            const bool ok = mbar_wait(smem_u32(&mbar[st]), phase);
            {
                const unsigned char* S_ = stages + st * VT_STAGE;
                const float* sf32 = reinterpret_cast<const float*>(S_) + 2 * ty * BOX_F + of;
                const unsigned char* sf = S_ + 3 * VT_BOX_F + 2 * ty * BOX_U8 + ob;
                const float2 u0 = *reinterpret_cast<const float2*>(sf32),
                             u1 = *reinterpret_cast<const float2*>(sf32 + BOX_F);
                const float2 v0 = *reinterpret_cast<const float2*>(sf32 + VT_BOX_F / 4),
                             v1 = *reinterpret_cast<const float2*>(sf32 + VT_BOX_F / 4 + BOX_F);
                const float2 w0 = *reinterpret_cast<const float2*>(sf32 + 2 * (VT_BOX_F / 4)),
                             w1 = *reinterpret_cast<const float2*>(sf32 + 2 * (VT_BOX_F / 4) + BOX_F);
                U[0][k] = make_float2(u0.x, u1.y);
                U[1][k] = make_float2(u0.y, u1.x);
                V[0][k] = make_float2(v0.x, v1.y);
                V[1][k] = make_float2(v0.y, v1.x);
                W[0][k] = make_float2(w0.x, w1.y);
                W[1][k] = make_float2(w0.y, w1.x);
                // a -0 is the least 32-bit integer
                auto least = [](float2 a, float2 b) {
                    return min(min(__float_as_int(a.x), __float_as_int(a.y)),
                               min(__float_as_int(b.x), __float_as_int(b.y)));
                };
                const int least_bits = min(min(least(u0, u1), least(v0, v1)), least(w0, w1));
                if (__any_sync(0xffffffffu, least_bits == (int)0x80000000)) neg0 = T + 2;
                const unsigned f0 = *reinterpret_cast<const unsigned short*>(sf);           // A0, B0
                const unsigned f1 = *reinterpret_cast<const unsigned short*>(sf + BOX_U8);  // A1, B1
                ff[0][k] = cell_entry(f0, lane8) | (cell_entry(f1 >> 8, lane8) << 16);
                ff[1][k] = cell_entry(f0 >> 8, lane8) | (cell_entry(f1, lane8) << 16);
            }
            if (__syncthreads_or(!ok)) {
                // a TMA stage never completed: record it, drain what is in flight, stop
                if (leader) {
                    atomicExch(kerr, 1);
                    const int last = min(q + S - 1, qfinal);
                    for (int pq = q; pq <= last; ++pq) {
                        const int d = pq - qbeg;
                        mbar_wait(smem_u32(&mbar[d % S]), (uint32_t)((d / S) & 1));
                    }
                }
                __syncthreads();
                return;
            }
            // every thread has read stage st: refill it with plane q + S
            if (leader && q + S <= qfinal) issue(st, q + S);
            // "pass 0": the v of this plane's row-0 cell that this iteration's pattern updates, read
            // by the thread above at its first pass on this plane (next iteration).  Written after
            // the barrier: the previous iteration's reads of this buffer are all done.
            cur[me0] = V[e][k].x;

            // ---- passes t = 1..T on plane q - t (slot j), reaching into plane q - t + 1 (slot jn)
#pragma unroll
            for (int t = 1; t <= T; ++t) {
                const int j = (k - t + 2 * R) % R;
                const int jn = (k - t + 1 + 2 * R) % R;
                // what the thread above's last-row cell added to this plane's row-0 v face in the
                // pass before (t - 1, at the previous iteration; p_t * s already)
                if (t >= 2 && (FULL || t - 1 <= nhalf)) V[e][j].x += prv[(2 * (t - 1) + 1) * VT_PROW + me0 - TX];
                if (!(FULL || t <= nhalf)) continue;
                // v of the thread below's row-0 cell at the end of the previous pass
                const float vb = prv[(2 * (t - 1)) * VT_PROW + me0 + TX];
                const unsigned o0 = ff[e][j] & 0xffffu, o1 = ff[e][j] >> 16;
                const float2 z0 = *reinterpret_cast<const float2*>(ctab + o0);
                const float2 z1 = *reinterpret_cast<const float2*>(ctab + o1);
                // the upper faces of the two cells.  E: A0's are B0's u, A1's v; B1's the next
                // lane's A1 u, the thread below's v.  O: B0's are the next lane's A0 u, B1's v; A1's
                // B1's u, the thread below's v
                float2 ux, vy;
                if (e == 0) {
                    ux = make_float2(U[1][j].x, __shfl_down_sync(0xffffffffu, U[1][j].y, 1));
                    vy = make_float2(V[1][j].y, vb);
                } else {
                    ux = make_float2(__shfl_down_sync(0xffffffffu, U[0][j].x, 1), U[0][j].y);
                    vy = make_float2(V[0][j].y, vb);
                }
                // div = -u + ux + -v + vy + -w + wz in the reference's order (a zero's sign
                // included); a negated term is an exact product with -1 inside an FMA
                const float2 neg = make_float2(-1.0f, -1.0f);
                float2 dv = __ffma2_rn(U[e][j], neg, ux);
                dv = __fadd2_rn(__ffma2_rn(V[e][j], neg, dv), vy);
                dv = __fadd2_rn(__ffma2_rn(W[e][j], neg, dv), W[e][jn]);
                const float2 qq = make_float2(div_fast(-dv.x, z0.x, z0.y), div_fast(-dv.y, z1.x, z1.y));
                const float2 c2 = __ffma2_rn(qq, wl1, __fmul2_rn(qq, wl2));
                const float2 pp = __ffma2_rn(qq, wh, c2);
                float p0 = pp.x, p1 = pp.y;
                bool r0 = es_rare(dv.x), r1 = es_rare(dv.y);
                if (!os.rational) {
                    r0 = r0 || !scale_sure(qq.x, c2.x, os);
                    r1 = r1 || !scale_sure(qq.y, c2.y, os);
                }
                if (__any_sync(0xffffffffu, r0 || r1)) {
                    p0 = cell_pt_rare(p0, r0, -dv.x, o0, z0.x, z0.y, os, omega);
                    p1 = cell_pt_rare(p1, r1, -dv.y, o1, z1.x, z1.y, os, omega);
                }
                const unsigned w = ff[e][j], w1 = w >> 16;
                const float pl0 = (w & C_PROJ) ? p0 : 0.0f, pl1 = (w1 & C_PROJ) ? p1 : 0.0f;
                const float pu0 = (w & C_PROJ) ? p0 : -0.0f, pu1 = (w1 & C_PROJ) ? p1 : -0.0f;
                // own (lower) faces, and the upper w faces (the next plane's)
                face_lower(w, C_XM, pl0, U[e][j].x);
                face_lower(w1, C_XM, pl1, U[e][j].y);
                face_lower(w, C_YM, pl0, V[e][j].x);
                face_lower(w1, C_YM, pl1, V[e][j].y);
                face_lower(w, C_ZM, pl0, W[e][j].x);
                face_lower(w1, C_ZM, pl1, W[e][j].y);
                face_upper(w, C_ZP, pu0, W[e][jn].x);
                face_upper(w1, C_ZP, pu1, W[e][jn].y);
                // upper u and v faces; the ones another thread holds receive their p_t * s from it
                float m;
                if (e == 0) {
                    m = __shfl_up_sync(0xffffffffu, face_sent(w1, C_XP, pu1), 1);  // lane - 1's B1, for A1
                    face_upper(w, C_XP, pu0, U[1][j].x);
                    U[1][j].y += tx > 0 ? m : -0.0f;
                    face_upper(w, C_YP, pu0, V[1][j].y);
                } else {
                    m = __shfl_up_sync(0xffffffffu, face_sent(w, C_XP, pu0), 1);  // lane - 1's B0, for A0
                    U[0][j].x += tx > 0 ? m : -0.0f;
                    face_upper(w1, C_XP, pu1, U[0][j].y);
                    face_upper(w, C_YP, pu0, V[0][j].y);
                }
                if (neg0 > 0) {
                    closed_lower(w, C_XM, p0, U[e][j].x);
                    closed_lower(w1, C_XM, p1, U[e][j].y);
                    closed_lower(w, C_YM, p0, V[e][j].x);
                    closed_lower(w1, C_YM, p1, V[e][j].y);
                    closed_lower(w, C_ZM, p0, W[e][j].x);
                    closed_lower(w1, C_ZM, p1, W[e][j].y);
                    closed_upper(w, C_ZP, p0, W[e][jn].x);
                    closed_upper(w1, C_ZP, p1, W[e][jn].y);
                    if (e == 0) closed_upper(w, C_XP, p0, U[1][j].x);
                    else closed_upper(w1, C_XP, p1, U[0][j].y);
                    closed_upper(w, C_YP, p0, V[e ^ 1][j].y);
                }
                cur[(2 * t) * VT_PROW + me0] = V[e][j].x;
                cur[(2 * t + 1) * VT_PROW + me0] = face_sent(w1, C_YP, pu1);
            }

            // ---- plane q - 1 - T: its last update (from the thread above's pass T) and the store
            {
                const int js = (k - 1 - T + 2 * R) % R;
                if (FULL) V[e][js].x += prv[(2 * T + 1) * VT_PROW + me0 - TX];
                const int zo = q - 1 - T;
                if (zo >= za && zo < zb) {
                    const size_t at = (size_t)off0 + (size_t)g.XY * zo;
                    if (in[0]) {
                        *reinterpret_cast<float2*>(uo + at) = make_float2(U[0][js].x, U[1][js].x);
                        *reinterpret_cast<float2*>(vo + at) = make_float2(V[0][js].x, V[1][js].x);
                        *reinterpret_cast<float2*>(wo + at) = make_float2(W[0][js].x, W[1][js].x);
                    }
                    if (in[1]) {
                        *reinterpret_cast<float2*>(uo + at + g.X) = make_float2(U[1][js].y, U[0][js].y);
                        *reinterpret_cast<float2*>(vo + at + g.X) = make_float2(V[1][js].y, V[0][js].y);
                        *reinterpret_cast<float2*>(wo + at + g.X) = make_float2(W[1][js].y, W[0][js].y);
                    }
                }
            }
            par ^= 1;
            --neg0;
        }
    }
}

template <int T, int TY, bool FULL>
__global__ void __launch_bounds__(VTGeom<TY>::THREADS, 1)
k_vsweep_tb(const __grid_constant__ VMaps maps, Grid g, float* __restrict__ uo, float* __restrict__ vo,
            float* __restrict__ wo, int nhalf, int colour0, int zchunk, OmegaSplit os, double omega,
            int* __restrict__ kerr) {
    vsweep_tile<T, TY, FULL>(maps, g, uo, vo, wo, nhalf, colour0, zchunk, os, omega, kerr);
}

template <int T, int TY>
constexpr size_t vt_smem_bytes() {
    using G = VTGeom<TY>;
    return 128 + (size_t)((T + 2) / 2) * G::STAGE + sizeof(float) * 2 * 2 * (T + 1) * G::PROW + COEF_BYTES;
}

// The tile height used with depth T.
constexpr int vt_ty(int T) { return T == 2 ? 24 : 16; }

}  // namespace

OmegaSplit omega_split(double w) {
    OmegaSplit s;
    memset(&s, 0, sizeof(s));
    const double a = std::fabs(w);
    if (!(a >= 0x1p-20 && a <= 0x1p20)) {  // zero, extreme or not finite: no cell passes the rounding test
        s.wh = s.wl1 = s.wl2 = NAN;
        return s;
    }
    s.wh = (float)w;
    if (std::fabs((double)s.wh) > a) s.wh = std::nextafterf(s.wh, 0.0f);
    const double wl = w - (double)s.wh;  // exact, at most 29 bits, with the sign of w
    s.wl1 = (float)wl;  // toward zero: wl2 keeps the sign, so that a zero q keeps its own
    if (std::fabs((double)s.wl1) > std::fabs(wl)) s.wl1 = std::nextafterf(s.wl1, 0.0f);
    s.wl2 = (float)(wl - (double)s.wl1);  // exact
    // the least D with |w - n / D| < m 2^(e - 54): fma(w, D, -n) is D times that error, exactly
    const double lim = std::ldexp(a, -54);
    for (int D = 1; D <= 1000 && !s.rational; ++D)
        if (std::fabs(std::fma(w, (double)D, -std::nearbyint(w * D))) < lim * D) s.rational = 1;
    return s;
}

struct VSweepMaps {
    // per box height (0: 32 rows, 1: 48 rows)
    CUtensorMap su[2][2], sv[2][2], sw[2][2];  // [height][state buffer 0/1]
    CUtensorMap xu[2], xv[2], xw[2];           // the scratch face arrays
    CUtensorMap f[2];                          // neighbour flags
};

int vsweep_depth_supported(int T) { return T == 2 || T == 4; }
int vsweep_tile_rows(int T) { return 2 * vt_ty(T); }

int prepare_vsweep_kernels() {
    if (smem_attribute_set((const void*)k_vsweep_tb<4, 16, true>, (int)vt_smem_bytes<4, 16>())) return 0;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const bool ok =
        cudaFuncSetAttribute(k_vsweep_tb<2, 24, true>, a, (int)vt_smem_bytes<2, 24>()) == cudaSuccess &&
        cudaFuncSetAttribute(k_vsweep_tb<2, 24, false>, a, (int)vt_smem_bytes<2, 24>()) == cudaSuccess &&
        cudaFuncSetAttribute(k_vsweep_tb<4, 16, true>, a, (int)vt_smem_bytes<4, 16>()) == cudaSuccess;
    return ok ? 0 : -1;
}

VSweepMaps* create_vsweep_maps(const Grid& g, float* const* u, float* const* v, float* const* w, const float* xu,
                               const float* xv, const float* xw, const uint8_t* flags) {
    VSweepMaps* m = new VSweepMaps();
    const int rows[2] = {VTGeom<16>::ROWS, VTGeom<24>::ROWS};
    bool ok = true;
    for (int h = 0; h < 2 && ok; ++h) {
        ok = tb::encode_3d(&m->f[h], flags, true, g, rows[h]) && tb::encode_3d(&m->xu[h], xu, false, g, rows[h]) &&
             tb::encode_3d(&m->xv[h], xv, false, g, rows[h]) && tb::encode_3d(&m->xw[h], xw, false, g, rows[h]);
        for (int b = 0; b < 2 && ok; ++b)
            ok = tb::encode_3d(&m->su[h][b], u[b], false, g, rows[h]) &&
                 tb::encode_3d(&m->sv[h][b], v[b], false, g, rows[h]) &&
                 tb::encode_3d(&m->sw[h][b], w[b], false, g, rows[h]);
    }
    if (!ok) {
        delete m;
        return nullptr;
    }
    return m;
}

void destroy_vsweep_maps(VSweepMaps* m) { delete m; }

template <int T>
static int launch_vt(const VSweepMaps* m, const Grid& g, int buf, bool from_state, float* uo, float* vo, float* wo,
                     int nhalf, int colour0, int zchunk, double omega, const OmegaSplit& os, int* kerr,
                     cudaStream_t st) {
    constexpr int TY = vt_ty(T);
    using G = VTGeom<TY>;
    constexpr int h = G::MAPS;
    VMaps maps;
    maps.u = from_state ? m->su[h][buf] : m->xu[h];
    maps.v = from_state ? m->sv[h][buf] : m->xv[h];
    maps.w = from_state ? m->sw[h][buf] : m->xw[h];
    maps.f = m->f[h];
    const dim3 grid((unsigned)sweep_windows(g.nx + 1, 2 * TX, T), (unsigned)sweep_windows(g.ny + 1, G::ROWS, T),
                    (unsigned)((g.nz + 1 + zchunk - 1) / zchunk));
    const dim3 block(TX, TY);
    const size_t smem = vt_smem_bytes<T, TY>();
    if constexpr (T == 4)
        k_vsweep_tb<T, TY, true><<<grid, block, smem, st>>>(maps, g, uo, vo, wo, nhalf, colour0, zchunk, os, omega,
                                                            kerr);
    else if (nhalf == T)
        k_vsweep_tb<T, TY, true><<<grid, block, smem, st>>>(maps, g, uo, vo, wo, nhalf, colour0, zchunk, os, omega,
                                                            kerr);
    else
        k_vsweep_tb<T, TY, false><<<grid, block, smem, st>>>(maps, g, uo, vo, wo, nhalf, colour0, zchunk, os, omega,
                                                             kerr);
    return (int)cudaGetLastError();
}

int launch_vsweep_tb(const VSweepMaps* m, const Grid& g, int buf, bool from_state, float* uo, float* vo, float* wo,
                     int T, int nhalf, int colour0, int zchunk, double omega, const OmegaSplit& os, int* kerr,
                     cudaStream_t st) {
    if (!vsweep_depth_supported(T) || nhalf < 1 || nhalf > T || (T == 4 && nhalf != 4) || zchunk < 1) return -1;
    if (T == 2) return launch_vt<2>(m, g, buf, from_state, uo, vo, wo, nhalf, colour0, zchunk, omega, os, kerr, st);
    return launch_vt<4>(m, g, buf, from_state, uo, vo, wo, nhalf, colour0, zchunk, omega, os, kerr, st);
}

}  // namespace smk

// ---- testing: the exact arithmetic's host instances, compared with the double product and the
// IEEE quotient by the CPU tests ----------------------------------------------------------------

namespace {
float host_scale(float q, const smk::OmegaSplit& os, double omega) {
    const float c = smk::scale_rest(q, os);
    if (smk::es_rare(q) || (!os.rational && !smk::scale_sure(q, c, os))) return smk::scale_exact(q, omega);
    return fmaf(q, os.wh, c);
}

// A cell's p_t as the kernel's common and rare paths give it.
float host_pt(float x, int d, const smk::OmegaSplit& os, double omega) {
    const smk::DivSplit z = smk::div_split(d);
    bool ok = false;
    if (!smk::es_rare(x)) {
        const float q = smk::div_fast(x, z.zh, z.zl);
        const float c = smk::scale_rest(q, os);
        if (os.rational || smk::scale_sure(q, c, os)) return fmaf(q, os.wh, c);
    } else if (fabsf(x) < smk::ES_TINY) {
        float p = smk::pt_scaled(x, z.zh, z.zl, os, ok);
        if (ok) return p;
        p = smk::pt_grid(x, d, z.zh, z.zl, os, ok);
        if (ok) return p;
    }
    return smk::scale_exact(smk::div_exact(x, (double)d, 1.0 / d), omega);
}
}  // namespace

extern "C" int smk_test_exact_arith(const float* x, const int* d, int n, double omega, float* scaled,
                                    float* quotient) {
    if (!x || n < 0) return 1;
    const smk::OmegaSplit os = smk::omega_split(omega);
    for (int i = 0; i < n; ++i) {
        if (scaled) scaled[i] = d ? host_scale(x[i], os, omega) : host_pt(x[i], 1, os, omega);
        if (quotient && d) {
            const int k = d[i] < 1 ? 1 : (d[i] > 6 ? 6 : d[i]);
            const smk::DivSplit z = smk::div_split(k);
            quotient[i] = smk::es_rare(x[i]) ? smk::div_exact(x[i], (double)k, 1.0 / k) : smk::div_fast(x[i], z.zh, z.zl);
        }
    }
    return 0;
}

extern "C" int smk_test_exact_cell(const float* x, const int* d, int n, double omega, float* pt) {
    if (!x || !d || !pt || n < 0) return 1;
    const smk::OmegaSplit os = smk::omega_split(omega);
    for (int i = 0; i < n; ++i) pt[i] = host_pt(x[i], d[i] < 1 ? 1 : (d[i] > 6 ? 6 : d[i]), os, omega);
    return 0;
}
