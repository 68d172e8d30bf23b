// Shared device definitions for libsmoke_gb300.
//
// HBM layout.  Every field of one simulation -- density (cells), u, v, w (faces), pressure and
// right-hand side (cells), the solid mask and the neighbour-flag byte (cells) -- uses ONE
// index function  i = x + X*y + XY*z  with X = round_up(nx+1, 16) (64-byte float rows and
// 16-byte flag rows, as TMA tensor maps require) and
// XY = X*(ny+1).  Faces use x <= nx, y <= ny, z <= nz; cells use x < nx, y < ny, z < nz and
// leave the last row/plane unused.  One index therefore addresses a cell and its three
// "lower" faces (u at x, v at y, w at z), exactly like the reference's shared staggered index
// (project/smokeSimulation.cu:146-147, :337), while rows stay aligned for vector access.
//
// The whole library is compiled with -fmad=false so that every float expression rounds
// exactly as written (no contraction); fused multiply-adds appear only as explicit fmaf().
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace smk {

struct Grid {
    int nx, ny, nz;
    int X;   // row pitch in elements
    int XY;  // plane pitch in elements
    __host__ __device__ __forceinline__ int idx(int x, int y, int z) const { return x + X * y + XY * z; }
};

// Neighbour-flag byte per cell, derived from the mask whenever it changes.
enum : uint8_t {
    F_SELF = 1u << 0,  // s(x,y,z)
    F_XM = 1u << 1,    // s(x-1,y,z)
    F_XP = 1u << 2,    // s(x+1,y,z)
    F_YM = 1u << 3,    // s(x,y-1,z)
    F_YP = 1u << 4,    // s(x,y+1,z)
    F_ZM = 1u << 5,    // s(x,y,z-1)
    F_ZP = 1u << 6,    // s(x,y,z+1)
    F_PROJ = 1u << 7,  // updated by the projection: interior, fluid, >= 1 fluid neighbour
    F_NBRS = 0x7E,
};

// Device-side per-step status written by the solver kernels.
struct StepStatus {
    unsigned div_bits;   // max |div u| after projection, as float bits (non-negative)
    int done;            // tolerance reached: later sweep groups are skipped
    int done_group;      // the solve ended at the start of this check group (its residual <= tol)
    unsigned arrivals;   // blocks of the running check launch that have added their residual;
                         // the last one decides and resets it (check_decide)
    unsigned rmax_bits[1];  // max |residual| per check group (flexible; sized at allocation)
};

// The tolerance rule, decided at the end of the launch that records the residual of check
// group `group`: every block calls it once after its block_max_to into rmax_bits[group] (thread
// 0 of the block, which made that atomic); the last of `nblocks` to arrive reads the group's
// residual and, when it is <= tol, ends the solve there (done, done_group) and, for a launch
// that swept from one pressure buffer into the other, points *pcur back at the launch's input
// (in_idx >= 0), so that the passes it applied are dropped.  Returns whether it ended the solve.
__device__ __forceinline__ bool check_decide(StepStatus* status, int group, float tol, unsigned nblocks,
                                             int* pcur, int in_idx) {
    __threadfence();
    const unsigned prev = atomicAdd(&status->arrivals, 1u);
    if (prev + 1u != nblocks) return false;
    __threadfence();
    const float r = __uint_as_float(*(volatile unsigned*)&status->rmax_bits[group]);
    status->arrivals = 0u;
    if (!(r <= tol)) return false;
    status->done = 1;
    status->done_group = group;
    if (pcur != nullptr && in_idx >= 0) *pcur = in_idx;
    return true;
}

// Device-side state of the projection's FP64-checked refinement rounds.
struct RefineStatus {
    unsigned long long div_bits;  // max |div u| of the last measurement (FP64, as IEEE bits)
    int need;                     // the last measurement found a cell above tolerance
    int rounds;                   // correction rounds applied in this step
    int stop;                     // a measurement was within tolerance: later rounds do nothing
    int pad;
};

// Whole solves with the iterate resident in shared memory (kernels_resident.cu): boxes of by x bz rows of
// the interior, cy x cz of them, one CTA each, all resident.
struct ResidentPlan {
    int by, bz, cy, cz;
    int hx, hp;  // cells of one colour in a row; elements of a colour row
    int rt, ns;  // threads, and cells of one colour per thread
};

// Object records (the reference's packing, smokeSimulation.cu:719-725, :750-758).
struct SphereObj { float x, y, z, r; };
struct ObstacleObj { float x, y, z, vx, vy, vz, r; };
struct BoxObj { int x0, y0, z0, x1, y1, z1; float density, vy; int set_vy; };

__device__ __forceinline__ void atomic_max_bits(unsigned* p, float nonneg) {
    atomicMax(p, __float_as_uint(nonneg));
}

// Max-reduce `v` (bit patterns of non-negative floats: the IEEE order, NaN largest) over the
// block, then one atomicMax per block, skipped when the stored value is already larger.  One
// atomic per warp on a single address serialises at L2 and costs ~1 ms on a 256^3 grid.
// Every thread of the block must call it; it ends with a block barrier, so a persistent loop
// may call it again without racing on the shared scratch.
__device__ __forceinline__ void block_max_to(unsigned v, unsigned* dst) {
    __shared__ unsigned red[32];
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int nthreads = blockDim.x * blockDim.y * blockDim.z;
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int lane = tid & 31, warp = tid >> 5, nwarps = (nthreads + 31) >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        unsigned w = lane < nwarps ? red[lane] : 0u;
        for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
        if (lane == 0 && w > *(volatile unsigned*)dst) atomicMax(dst, w);
    }
    __syncthreads();
}

// Whether `kernel` already has `bytes` of dynamic shared memory on this device (the attribute belongs to
// the context: a reset takes it away): the last of a family of kernels that are set together.
inline bool smem_attribute_set(const void* kernel, int bytes) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.maxDynamicSharedSizeBytes >= bytes;
}

// ---- storage types ----------------------------------------------------------------------------
// Fields are stored as float (FP32 form) or bf16 (BF16 storage form); arithmetic is FP32 in
// both.  ldv/stv are the only places a stored value is converted.
__device__ __forceinline__ float ldv(const float* __restrict__ p, int i) { return p[i]; }
__device__ __forceinline__ float ldv(const __nv_bfloat16* __restrict__ p, int i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void stv(float* __restrict__ p, int i, float v) { p[i] = v; }
__device__ __forceinline__ void stv(__nv_bfloat16* __restrict__ p, int i, float v) { p[i] = __float2bfloat16_rn(v); }

// Four consecutive stored values (index a multiple of 4 in a row with 16-byte aligned float or
// 8-byte aligned bf16 rows): one vector load, the raw bits kept so that a store can leave the
// lanes that did not change bit for bit as they were.  A bf16 value widens to float exactly by
// its bits (the conversion ldv makes).
struct Raw4f { float4 v; };
struct Raw4h { uint2 r; };
__device__ __forceinline__ Raw4f ld4raw(const float* p) { return Raw4f{*reinterpret_cast<const float4*>(p)}; }
__device__ __forceinline__ Raw4h ld4raw(const __nv_bfloat16* p) { return Raw4h{*reinterpret_cast<const uint2*>(p)}; }
__device__ __forceinline__ float4 to4(const Raw4f& a) { return a.v; }
__device__ __forceinline__ float4 to4(const Raw4h& a) {
    return make_float4(__uint_as_float(a.r.x << 16), __uint_as_float(a.r.x & 0xffff0000u),
                       __uint_as_float(a.r.y << 16), __uint_as_float(a.r.y & 0xffff0000u));
}
// Store the four values; lane c keeps its raw bits unless bit c of `changed` is set (a float lane
// that did not change holds its loaded value, so storing it is the same).
__device__ __forceinline__ void st4(float* p, const Raw4f&, float4 v, unsigned) {
    *reinterpret_cast<float4*>(p) = v;
}
__device__ __forceinline__ unsigned bf16_bits(float v) {
    return (unsigned)__bfloat16_as_ushort(__float2bfloat16_rn(v));
}
__device__ __forceinline__ void st4(__nv_bfloat16* p, const Raw4h& a, float4 v, unsigned changed) {
    const unsigned h0 = (changed & 1u) ? bf16_bits(v.x) : (a.r.x & 0xffffu);
    const unsigned h1 = (changed & 2u) ? bf16_bits(v.y) : (a.r.x >> 16);
    const unsigned h2 = (changed & 4u) ? bf16_bits(v.z) : (a.r.y & 0xffffu);
    const unsigned h3 = (changed & 8u) ? bf16_bits(v.w) : (a.r.y >> 16);
    *reinterpret_cast<uint2*>(p) = make_uint2(h0 | (h1 << 16), h2 | (h3 << 16));
}
template <typename T> struct Raw4;
template <> struct Raw4<float> { typedef Raw4f type; };
template <> struct Raw4<__nv_bfloat16> { typedef Raw4h type; };

// ---- reference-exact helpers ---------------------------------------------------------------

// The advections (kernels_advect_tile.cu, density_rows) keep the reference's arithmetic, term for term:
//   - avgU/avgV/avgW (smokeSimulation.cu:409-447): 8-point sums in the reference's order, / 8;
//   - sampleSmoke (smokeSimulation.cu:451-484): clamp the position to [1, n-1] with the CELL dims,
//     trilinear weights from (c - delta) - i0, delta 0.5 on an axis or 0, and the eight terms
//     xw * yw * zw * a summed in the order 000, 100, 010, 110, 001, 101, 011, 111 (digits: x, y, z).
// Every call has n >= 2 on every axis (it samples only from cells with an interior neighbour).  After the
// clamp c lies in [1, n-1], so c - delta >= 0.5 and floorf equals truncation, and the reference's
// fminf(i0, n-1) never changes i0.  Its upper corner fminf(i0 + 1, n - 1): with delta = 0.5,
// c - delta <= n - 1.5, so i0 <= n - 2 and the corner is always i0 + 1; with delta = 0 it is i0 + 1 unless
// i0 = n - 1 (a position clamped to the last cell), where it repeats i0.  Integer index arithmetic with
// these facts gives every result of the reference's float index arithmetic.  Every +1 neighbour lies inside
// the arrays (rows hold >= nx+1 elements, planes >= ny+1 rows, the field >= nz+1 planes), so the x+1
// values are loaded at a fixed offset and replaced by the x0 values where the corner repeats.

// Loads issued where they stand (volatile inline PTX): the compiler can neither sink them into
// the conditional block that consumes them nor merge them away, so a warp has a cell's loads in
// flight before it waits on the flag byte that decides whether the cell is updated.
__device__ __forceinline__ float ld_eager(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float ld_eager(const __nv_bfloat16* p) {
    unsigned short h;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(h) : "l"(__cvta_generic_to_global(p)));
    return __bfloat162float(__ushort_as_bfloat16(h));
}

// Tiles of the density advection: 256 (x, row pair) units of the interior by a run of planes.  The units go
// through strips of DENSITY_STRIP columns row pair by row pair, without gaps.
constexpr int DENSITY_THREADS = 256, DENSITY_STRIP = 64;
__host__ __device__ inline int density_units(const Grid& g) {
    return g.nx < 3 || g.ny < 3 ? 0 : (g.nx - 2) * ((g.ny - 1) / 2);
}
__host__ __device__ inline int density_blocks(const Grid& g) {
    return (density_units(g) + DENSITY_THREADS - 1) / DENSITY_THREADS;
}
__device__ __forceinline__ void density_unit(const Grid& g, int unit, int& x, int& y) {
    const int pairs = (g.ny - 1) / 2, strip = unit / (DENSITY_STRIP * pairs), left = strip * DENSITY_STRIP;
    const int wide = min(DENSITY_STRIP, g.nx - 2 - left), r = unit - left * pairs;
    x = 1 + left + r % wide;
    y = 1 + 2 * (r / wide);
}

// The grid j that tile t of a grouped launch belongs to: the last one with starts[j] <= t (starts[0] = 0,
// n grids, t below starts[n]).  Every lane of a warp calls it: one load a lane narrows 32-fold.
__device__ __forceinline__ int find_grid(const int* __restrict__ starts, int n, int t) {
    const int lane = (int)((threadIdx.x + blockDim.x * threadIdx.y) & 31u);
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32, k = lo + lane * step;
        const unsigned at = __ballot_sync(0xffffffffu, k < hi && starts[k] <= t);
        lo += (__popc(at) - 1) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

}  // namespace smk
