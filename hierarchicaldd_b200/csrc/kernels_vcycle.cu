// Subdomain-resident multigrid V-cycle for sm_100a.
//
// One CTA of 512 threads (128 for 8^3) owns one subdomain box for the whole
// V-cycle: the level-0 box (sub+1)^3 cells including its two halo planes per
// axis, and every coarse level, live on its SM.  HBM is touched once to load
// u, b and the flags and once to store u, instead of once per smoothing sweep
// as in the reference (CPU/SPGrid_Library/SPGrid_V_Cycle_Helper.h:156-195, GPU
// CUDA_Kernels/SPGrid_V_Cycle_Helper_CUDA.h:272-301).
//
// Arithmetic follows the reference's float operation order with explicit
// round-to-nearest intrinsics, so no multiply-add is contracted:
//   residual   r = b - sum_faces (u_n - u_c)      (SPGrid_Residual_Legacy.h:52-61)
//   correction u += (omega/face_count) * r        (SPGrid_Correction_Legacy.h:47-80)
//   restriction, prolongation weights and order  (SPGrid_Restriction_Legacy.h:47-186,
//                                                 SPGrid_Prolongation_Legacy.h:46-128)
// Smoothing is Jacobi: every residual of a sweep is computed from the old u.
//
// A level of NX^3 interior cells (NX = sub/2^l - 1: 31, 15, 7, 3, 1) runs as:
// * 31: shared memory holds one u; b and the flags stay in registers (b would
//   not fit beside u and the coarse levels).  A thread owns two x-lines and
//   sweeps them in chunks of four planes: new values of a chunk wait in
//   registers for a CTA barrier, after which nobody reads the chunk's old
//   values any more (a line's own old x neighbour is carried in a register),
//   so the sweep is in place with one barrier per chunk.
// * 15 and 7: two copies of u in shared memory, one barrier per sweep; a
//   thread owns a piece of an x-line and keeps its u, b and flags in
//   registers.  The residual for the restriction goes to the idle copy.
// * 3 and 1: one warp, a cell per lane, neighbours by shuffle, no barrier.
//
// What bounds it: issue slots on level 0 (about 25 instructions a cell and
// sweep, 31^3 cells, a box per SM), then the serial 200 bottom sweeps.  A 4-CTA
// cluster per 32^3 box (slabs of level 0 in distributed shared memory, the
// coarse levels on one of the four) took four SMs per box and a cluster
// barrier per sweep.  Measured per launch, that form and this one: 216 boxes of
// 32^3 (192^3 cells) 2252 and 709 us, 64 boxes (128^3) 669 and 390 us; 64 boxes
// of 16^3 113 and 55 us; 8 boxes of 8^3 124 and 23 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "hdd_common.h"
#include "kernels.h"

namespace hdd {

namespace {

__host__ __device__ constexpr int cells_of(int nx) { return (nx + 2) * (nx + 2) * (nx + 2); }
__host__ __device__ constexpr int pad4(int n) { return (n + 3) & ~3; }

// One level with two copies of u (NX <= 15): a, t (floats), b, flags.
struct Level {
    float *a, *t, *b;
    uint8_t* f;
};
// Shared-memory bytes of a level and of all levels from NX down to `levels`.
__host__ __device__ constexpr int level_bytes(int nx) { return 13 * pad4(cells_of(nx)); }

template <int NX>
__device__ __forceinline__ Level level_at(unsigned char* p) {
    constexpr int n4 = pad4(cells_of(NX));
    Level L;
    L.a = reinterpret_cast<float*>(p);
    L.t = L.a + n4;
    L.b = L.t + n4;
    L.f = reinterpret_cast<uint8_t*>(L.b + n4);
    return L;
}

struct Weights {
    float inv[8], sc64[64], sc8[8];
};

__device__ __forceinline__ float face_res(float res, float n, float c, bool on) {
    const float d = __fsub_rn(res, __fsub_rn(n, c));
    return on ? d : res;
}

// b - sum_faces (u_n - u_c), reference face order -x,+x,-y,+y,-z,+z.
__device__ __forceinline__ float residual6(uint32_t fl, float c, float xm, float xp, float ym, float yp, float zm,
                                           float zp, float b) {
    float res = 0.0f;
    res = face_res(res, xm, c, fl & 0x01u);
    res = face_res(res, xp, c, fl & 0x02u);
    res = face_res(res, ym, c, fl & 0x04u);
    res = face_res(res, yp, c, fl & 0x08u);
    res = face_res(res, zm, c, fl & 0x10u);
    res = face_res(res, zp, c, fl & 0x20u);
    return __fsub_rn(b, res);
}

// A sweep takes cell flags fl when (fl & mask) == value: boundary cells
// (Active and Boundary), interior cells (Active, not Boundary) or all Active.
struct Take {
    uint32_t mask, value;
    __device__ __forceinline__ bool operator()(uint32_t fl) const { return (fl & mask) == value; }
};
__device__ __forceinline__ Take take_boundary() { return {C_ACTIVE | C_BOUNDARY8, C_ACTIVE | C_BOUNDARY8}; }
__device__ __forceinline__ Take take_interior() { return {C_ACTIVE | C_BOUNDARY8, C_ACTIVE}; }
__device__ __forceinline__ Take take_active() { return {C_ACTIVE, C_ACTIVE}; }

// The sweeps of one visit of a level: boundary, interior, boundary smoothing,
// or the bottom's sweeps over all Active cells.
struct Sweeps {
    int nb, ni, bottom;
    __device__ __forceinline__ int count() const { return bottom ? bottom : 2 * nb + ni; }
    __device__ __forceinline__ Take at(int s) const {
        if (bottom) return take_active();
        return (s < nb || s >= nb + ni) ? take_boundary() : take_interior();
    }
};

// ---------------------------------------------------------------------------
// Levels of 15 and 7 cells per axis
// ---------------------------------------------------------------------------

// Pieces an x-line is cut into so that NT threads cover the level.
template <int NX, int NT>
struct Pieces {
    static constexpr int LINES = NX * NX;
    static constexpr int N = NT / LINES >= NX ? NX : (NT / LINES >= 1 ? NT / LINES : 1);
    static constexpr int C = (NX + N - 1) / N;  // cells per piece
    static_assert(LINES * N <= NT, "a thread per piece");
};

// Runs the sweeps from L.a, leaving u in L.a (the copies change places), and
// with `residual` the residual (zero at cells that are not Active) in L.t.
template <int NX, int NT>
__device__ __forceinline__ void sweeps_lines(Level& L, const Sweeps& S, bool residual, const float* inv) {
    using P = Pieces<NX, NT>;
    constexpr int E = NX + 2, PS = E * E, C = P::C;
    const int t = threadIdx.x;
    const bool own = t < P::LINES * P::N;
    const int line = own ? t % P::LINES : 0, k0 = own ? (t / P::LINES) * C : 0;
    const int nk = own ? min(C, NX - k0) : 0;
    const int base = (k0 + 1) * PS + (line / NX + 1) * E + line % NX + 1;
    float u[C], b[C], w[C];
    uint32_t fl[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const bool in = c < nk;
        const int i = base + c * PS;
        u[c] = in ? L.a[i] : 0.0f;
        b[c] = in ? L.b[i] : 0.0f;
        fl[c] = in ? (uint32_t)L.f[i] : 0u;
        w[c] = inv[__popc(fl[c] & C_FACES)];
    }
    const int n = S.count();
    for (int s = 0; s < n + (residual ? 1 : 0); ++s) {
        const bool res = s == n;
        const Take take = res ? take_active() : S.at(s);
        float nu[C];
        if (own) {
            const float xlo = L.a[base - PS], xhi = L.a[base + nk * PS];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (c >= nk) continue;
                const int i = base + c * PS;
                const float xp = c + 1 < nk ? u[c + 1 < C ? c + 1 : c] : xhi;
                const float r = residual6(fl[c], u[c], c > 0 ? u[c > 0 ? c - 1 : 0] : xlo, xp, L.a[i - E], L.a[i + E],
                                          L.a[i - 1], L.a[i + 1], b[c]);
                const bool on = take(fl[c]);
                if (res) nu[c] = on ? r : 0.0f;
                else nu[c] = on ? __fadd_rn(u[c], __fmul_rn(w[c], r)) : u[c];
                L.t[i] = nu[c];
            }
        }
        __syncthreads();
        if (!res) {
#pragma unroll
            for (int c = 0; c < C; ++c) u[c] = nu[c];
            float* q = L.a;
            L.a = L.t;
            L.t = q;
        }
    }
}

// Coarse b = restriction of the residual F.t (zero at halo cells, or HALO: the
// fine level's lower faces from rh, indexed as a tile of SUB cells per axis;
// null rh: zero there).  The coarse u starts at zero.
template <int NX, int NT, bool HALO>
__device__ __forceinline__ void restrict_lines(const Level& F, const Level& Cc, const float* sc64, const float* rh) {
    constexpr int E = NX + 2, PS = E * E, M = (NX - 1) / 2, CE = M + 2, SUB = NX + 1;
    for (int i = threadIdx.x; i < cells_of(M); i += NT) Cc.a[i] = 0.0f;
    for (int q = threadIdx.x; q < M * M * M; q += NT) {
        const int z = q % M, t = q / M, y = t % M, x = t / M;
        const int ci = ((x + 1) * CE + y + 1) * CE + z + 1;
        if (!(Cc.f[ci] & C_ACTIVE)) continue;
        // Fine cells 2C-2 .. 2C+1 per axis (box coordinates, C = x+1).
        float acc = 0.0f;
#pragma unroll
        for (int i2 = 0; i2 < 4; ++i2)
#pragma unroll
            for (int j2 = 0; j2 < 4; ++j2)
#pragma unroll
                for (int k2 = 0; k2 < 4; ++k2) {
                    const int fx = 2 * x + i2, fy = 2 * y + j2, fz = 2 * z + k2;
                    float v;
                    if (HALO && (fx == 0 || fy == 0 || fz == 0)) v = rh ? rh[(fx * SUB + fy) * SUB + fz] : 0.0f;
                    else v = F.t[fx * PS + fy * E + fz];
                    acc = __fadd_rn(acc, __fmul_rn(sc64[(i2 * 4 + j2) * 4 + k2], v));
                }
        Cc.b[ci] = acc;
    }
}

// Prolongation of coarse u (cells per axis CE with halos) added to v at fine
// box cell (x, y, z).  Box origins are even, so box-local parents follow the
// global rule: c = (f+1)/2, parity p = 1 - (f - (2c-1)).
template <int CE>
__device__ __forceinline__ float prolongate_cell(float v, const float* cu, int x, int y, int z, const float* sc8) {
    const int cx = (x + 1) >> 1, cy = (y + 1) >> 1, cz = (z + 1) >> 1;
    const int px = 1 - (x - (2 * cx - 1)), py = 1 - (y - (2 * cy - 1)), pz = 1 - (z - (2 * cz - 1));
    const float* c = cu + (cx * CE + cy) * CE + cz;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int bq = 0; bq < 2; ++bq)
#pragma unroll
            for (int cq = 0; cq < 2; ++cq) {
                const float w = sc8[((a ^ px) * 2 + (bq ^ py)) * 2 + (cq ^ pz)];
                v = __fadd_rn(v, __fmul_rn(w, c[(a - px) * CE * CE + (bq - py) * CE + (cq - pz)]));
            }
    return v;
}

template <int NX, int NT>
__device__ __forceinline__ void prolongate_lines(const Level& F, const Level& Cc, const float* sc8) {
    constexpr int E = NX + 2, CE = (NX - 1) / 2 + 2;
    for (int q = threadIdx.x; q < NX * NX * NX; q += NT) {
        const int z = q % NX + 1, t = q / NX, y = t % NX + 1, x = t / NX + 1;
        const int i = (x * E + y) * E + z;
        if (F.f[i] & C_ACTIVE) F.a[i] = prolongate_cell<CE>(F.a[i], Cc.a, x, y, z, sc8);
    }
}

// ---------------------------------------------------------------------------
// Levels of 3 and 1 cells per axis, by one warp
// ---------------------------------------------------------------------------

// One cell: lane 0 alone.  Once a sweep leaves the value as it is, so do all
// that follow (each depends on nothing else).
__device__ __forceinline__ void sweeps_one(const Level& L, int n, const float* inv) {
    constexpr int i = 13;  // cell (1,1,1) of 3^3
    const uint32_t fl = L.f[i];
    if (!(fl & C_ACTIVE)) return;
    const float b = L.b[i], w = inv[__popc(fl & C_FACES)];
    const float xm = L.a[i - 9], xp = L.a[i + 9], ym = L.a[i - 3], yp = L.a[i + 3], zm = L.a[i - 1], zp = L.a[i + 1];
    float u = L.a[i];
    for (int s = 0; s < n; ++s) {
        const float nu = __fadd_rn(u, __fmul_rn(w, residual6(fl, u, xm, xp, ym, yp, zm, zp, b)));
        if (nu == u) break;
        u = nu;
    }
    L.a[i] = u;
}

// 3^3 cells: lane q < 27 holds cell q and takes interior neighbours by
// shuffle; halo neighbours never change, so they are read once.  With
// `residual`, r (zero at cells that are not Active) in L.t.
__device__ __forceinline__ void sweeps_27(const Level& L, const Sweeps& S, bool residual, const float* inv) {
    const int lane = threadIdx.x & 31;
    const bool own = lane < 27;
    const int q = own ? lane : 0;
    const int x = q / 9 + 1, y = (q / 3) % 3 + 1, z = q % 3 + 1;
    const int i = (x * 5 + y) * 5 + z;
    const uint32_t fl = own ? (uint32_t)L.f[i] : 0u;
    const float b = own ? L.b[i] : 0.0f;
    const float w = inv[__popc(fl & C_FACES)];
    float u = own ? L.a[i] : 0.0f;
    const float hxm = x == 1 ? L.a[i - 25] : 0.0f, hxp = x == 3 ? L.a[i + 25] : 0.0f;
    const float hym = y == 1 ? L.a[i - 5] : 0.0f, hyp = y == 3 ? L.a[i + 5] : 0.0f;
    const float hzm = z == 1 ? L.a[i - 1] : 0.0f, hzp = z == 3 ? L.a[i + 1] : 0.0f;
    auto res = [&]() {
        const float sxm = __shfl_sync(0xffffffffu, u, lane - 9), sxp = __shfl_sync(0xffffffffu, u, lane + 9);
        const float sym = __shfl_sync(0xffffffffu, u, lane - 3), syp = __shfl_sync(0xffffffffu, u, lane + 3);
        const float szm = __shfl_sync(0xffffffffu, u, lane - 1), szp = __shfl_sync(0xffffffffu, u, lane + 1);
        return residual6(fl, u, x == 1 ? hxm : sxm, x == 3 ? hxp : sxp, y == 1 ? hym : sym, y == 3 ? hyp : syp,
                         z == 1 ? hzm : szm, z == 3 ? hzp : szp, b);
    };
    const int n = S.count();
    for (int s = 0; s < n; ++s) {
        const bool on = S.at(s)(fl);
        const float r = res();
        if (on) u = __fadd_rn(u, __fmul_rn(w, r));
    }
    if (residual) {
        const float r = res();
        if (own) L.t[i] = (fl & C_ACTIVE) ? r : 0.0f;
    }
    if (own) L.a[i] = u;
    __syncwarp();
}

// ---------------------------------------------------------------------------
// The V-cycle from a level of NX cells per axis down (u = 0 in L.a, b set)
// ---------------------------------------------------------------------------
// The level's data begin at p, the next level's right behind it; `left` levels
// remain, this one included.  Ends with the CTA synchronised.
template <int NX, int NT>
__device__ __forceinline__ void vcycle_from(unsigned char* p, int left, const VcycleArgs& a, const Weights& W) {
    const Sweeps smooth{a.boundary_itr, a.interior_itr, 0}, bottom{0, 0, a.bottom_itr};
    if constexpr (NX == 3) {
        if (threadIdx.x < 32) {
            const Level L = level_at<3>(p);
            if (left == 1) {
                if (a.bottom_itr > 0) sweeps_27(L, bottom, false, W.inv);
            } else {
                const Level Cc = level_at<1>(p + level_bytes(3));
                sweeps_27(L, smooth, true, W.inv);
                restrict_lines<3, 32, false>(L, Cc, W.sc64, nullptr);
                __syncwarp();
                if (threadIdx.x == 0) sweeps_one(Cc, a.bottom_itr, W.inv);
                __syncwarp();
                prolongate_lines<3, 32>(L, Cc, W.sc8);
                __syncwarp();
                sweeps_27(L, smooth, false, W.inv);
            }
        }
        __syncthreads();
    } else {
        Level L = level_at<NX>(p);
        if (left == 1) {
            if (a.bottom_itr > 0) sweeps_lines<NX, NT>(L, bottom, false, W.inv);
        } else {
            unsigned char* pc = p + level_bytes(NX);
            sweeps_lines<NX, NT>(L, smooth, true, W.inv);
            restrict_lines<NX, NT, false>(L, level_at<(NX - 1) / 2>(pc), W.sc64, nullptr);
            __syncthreads();
            vcycle_from<(NX - 1) / 2, NT>(pc, left - 1, a, W);
            prolongate_lines<NX, NT>(L, level_at<(NX - 1) / 2>(pc), W.sc8);
            __syncthreads();
            sweeps_lines<NX, NT>(L, smooth, false, W.inv);
        }
        // Callers read u from the first copy.
        const Level L0 = level_at<NX>(p);
        if (L.a != L0.a) {
            for (int i = threadIdx.x; i < cells_of(NX); i += NT) L0.a[i] = L.a[i];
            __syncthreads();
        }
    }
}

__device__ __forceinline__ void load_weights(Weights& W, const VcycleArgs& a) {
    if (threadIdx.x < 8) W.inv[threadIdx.x] = a.inv_diag[threadIdx.x];
    if (threadIdx.x < 64) W.sc64[threadIdx.x] = a.restrict_w[threadIdx.x];
    if (threadIdx.x < 8) W.sc8[threadIdx.x] = a.prolong_w[threadIdx.x];
}

// Coarse levels 1 .. levels-1 of the box: u, residual and b zero, flags loaded.
template <int NX, int NT>
__device__ __forceinline__ void clear_levels(unsigned char* p, int level, const VcycleArgs& a, const uint8_t* rec) {
    const Level L = level_at<NX>(p);
    for (int i = threadIdx.x; i < cells_of(NX); i += NT) {
        L.a[i] = 0.0f;
        L.t[i] = 0.0f;
        L.b[i] = 0.0f;
        L.f[i] = rec[a.level_off[level] + i];
    }
    if constexpr (NX > 1) {
        if (level + 1 < a.levels) clear_levels<(NX - 1) / 2, NT>(p + level_bytes(NX), level + 1, a, rec);
    }
}

template <int NX>
int levels_bytes(int levels) {
    int n = level_bytes(NX);
    if constexpr (NX > 1) {
        if (levels > 1) n += levels_bytes<(NX - 1) / 2>(levels - 1);
    }
    return n;
}

// Level-0 u at box cell (x, y, z) in 0 .. SUB: the box's own tile, or a
// neighbour tile's plane 0 on the upper faces (edge cells are never read).
template <int SUB>
__device__ __forceinline__ float load_u0(const VcycleArgs& a, const float* au, int box, int tile, int x, int y, int z) {
    constexpr int TC = SUB * SUB * SUB;
    const bool halo = x == 0 || y == 0 || z == 0 || x == SUB || y == SUB || z == SUB;
    if (halo ? !a.halo_from_u : a.zero_init) return 0.0f;
    const int hi = (x == SUB) + (y == SUB) + (z == SUB);
    if (hi == 0) return au[(size_t)tile * TC + (x * SUB + y) * SUB + z];
    if (hi > 1) return 0.0f;
    const int axis = x == SUB ? 0 : (y == SUB ? 1 : 2);
    const int nt = a.box_nb[3 * box + axis];
    if (nt < 0) return 0.0f;
    return au[(size_t)nt * TC + ((axis == 0 ? 0 : x) * SUB + (axis == 1 ? 0 : y)) * SUB + (axis == 2 ? 0 : z)];
}

// 8^3 and 16^3 boxes: every level with two copies of u in shared memory.
template <int SUB, int NT>
__global__ void __launch_bounds__(NT) vcycle_kernel(VcycleArgs a) {
    constexpr int NX = SUB - 1, E = SUB + 1, TC = SUB * SUB * SUB;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Weights W;
    const int box = blockIdx.x;
    if (a.active && !a.active[blockIdx.y]) return;
    // System blockIdx.y of a batch: its u and b.
    float* const au = a.u + (size_t)blockIdx.y * a.slot_stride;
    const float* const ab = a.b + (size_t)blockIdx.y * a.slot_stride;
    load_weights(W, a);
    const uint8_t* rec = a.box_flags + (size_t)box * a.box_stride;
    const int tile = a.box_tile[box];
    const float* gb = ab + (size_t)tile * TC;
    Level L = level_at<NX>(smem);
    for (int i = threadIdx.x; i < cells_of(NX); i += NT) {
        const int z = i % E, t = i / E, y = t % E, x = t / E;
        const bool in = x > 0 && y > 0 && z > 0 && x < SUB && y < SUB && z < SUB;
        const float u = load_u0<SUB>(a, au, box, tile, x, y, z);
        L.a[i] = u;
        L.t[i] = u;
        L.b[i] = in ? gb[(x * SUB + y) * SUB + z] : 0.0f;
        L.f[i] = rec[a.level_off[0] + i];
    }
    unsigned char* p1 = smem + level_bytes(NX);
    if (a.levels > 1) clear_levels<(NX - 1) / 2, NT>(p1, 1, a, rec);
    __syncthreads();
    const Sweeps smooth{a.boundary_itr, a.interior_itr, 0}, bottom{0, 0, a.bottom_itr};
    // The residual at the lower-face cells, when given (else it is zero there).
    const float* rh = a.r_halo ? a.r_halo + (size_t)blockIdx.y * a.slot_stride + (size_t)tile * TC : nullptr;
    for (int cycle = 0; cycle < a.n_vcycles; ++cycle) {
        if (a.levels == 1) {
            if (a.bottom_itr > 0) sweeps_lines<NX, NT>(L, bottom, false, W.inv);
            continue;
        }
        sweeps_lines<NX, NT>(L, smooth, true, W.inv);
        restrict_lines<NX, NT, true>(L, level_at<(NX - 1) / 2>(p1), W.sc64, rh);
        __syncthreads();
        vcycle_from<(NX - 1) / 2, NT>(p1, a.levels - 1, a, W);
        prolongate_lines<NX, NT>(L, level_at<(NX - 1) / 2>(p1), W.sc8);
        __syncthreads();
        sweeps_lines<NX, NT>(L, smooth, false, W.inv);
    }
    // Store the interior cells (1..SUB-1 per axis) of level 0.
    float* gw = au + (size_t)tile * TC;
    for (int q = threadIdx.x; q < TC; q += NT) {
        const int z = q % SUB, t = q / SUB, y = t % SUB, x = t / SUB;
        if (x == 0 || y == 0 || z == 0) continue;
        gw[q] = L.a[(x * E + y) * E + z];
    }
}

// ---------------------------------------------------------------------------
// 32^3 boxes
// ---------------------------------------------------------------------------
constexpr int kNT32 = 512;

// The x-lines of thread t: (y, z), both 1..31.  Lines whose cells all lie
// within the Boundary band (3 cells) of the box's y/z faces take
// boundary-sweep work on every cell, the others on six; line 0 of the first
// 336 threads is such a line and every other line is not, so that no thread
// has two of them.  Any assignment gives the same results.
__device__ __forceinline__ bool owned_line(int t, int l, int& y, int& z) {
    constexpr int SUB = 32, M1 = SUB - 1, D = 3, W = M1 - 2 * D;
    constexpr int H = 2 * D * M1 + W * 2 * D;  // lines inside the band
    static_assert(H <= kNT32 && kNT32 <= H + W * W && W * W <= 2 * kNT32 - H, "two lines per thread");
    auto band = [](int i) { return i < D ? i + 1 : SUB - 2 * D + i; };  // 1..D, SUB-D..SUB-1
    auto light = [&](int k) { y = D + 1 + k / W; z = D + 1 + k % W; };
    if (t < H) {
        if (l == 1) light(t);
        else if (t < 2 * D * M1) { y = band(t / M1); z = t % M1 + 1; }
        else { const int r = t - 2 * D * M1; y = D + 1 + r / (2 * D); z = band(r % (2 * D)); }
        return true;
    }
    const int k = l == 0 ? t : kNT32 + (t - H);
    if (k >= W * W) return false;
    light(k);
    return true;
}

constexpr int kU32Bytes = 31 * 33 * 33 * 4;  // planes x = 1..31

size_t smem_bytes_32(int levels) { return kU32Bytes + (levels > 1 ? levels_bytes<15>(levels - 1) : 0); }

// Coarse plane cx of level 1's b from the ring's fine planes 2cx-2 .. 2cx+1.
__device__ __noinline__ void restrict_plane_32(const float* ring, const Level& L1, int cx, const float* sc64) {
    constexpr int E = 33, PS = E * E;
    if (threadIdx.x >= 225) return;
    const int cy = threadIdx.x / 15 + 1, cz = threadIdx.x % 15 + 1, ci = (cx * 17 + cy) * 17 + cz;
    if (!(L1.f[ci] & C_ACTIVE)) return;
    float acc = 0.0f;
#pragma unroll
    for (int i2 = 0; i2 < 4; ++i2) {
        const float* R = ring + ((2 * cx - 2 + i2) % 6) * PS + (2 * cy - 2) * E + 2 * cz - 2;
#pragma unroll
        for (int j2 = 0; j2 < 4; ++j2)
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2)
                acc = __fadd_rn(acc, __fmul_rn(sc64[(i2 * 4 + j2) * 4 + k2], R[j2 * E + k2]));
    }
    L1.b[ci] = acc;
}

__global__ void __launch_bounds__(kNT32, 1) vcycle_kernel_32(VcycleArgs a) {
    constexpr int SUB = 32, NX = 31, E = 33, PS = E * E, TC = SUB * SUB * SUB, NT = kNT32;
    constexpr int CH = 4, NCH = (NX + CH - 1) / CH;  // planes per chunk, chunks
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Weights W;
    const int box = blockIdx.x;
    if (a.active && !a.active[blockIdx.y]) return;
    float* const au = a.u + (size_t)blockIdx.y * a.slot_stride;
    const float* const ab = a.b + (size_t)blockIdx.y * a.slot_stride;
    load_weights(W, a);
    const uint8_t* rec = a.box_flags + (size_t)box * a.box_stride;
    const int tile = a.box_tile[box];
    const float* gb = ab + (size_t)tile * TC;
    float* const U = reinterpret_cast<float*>(smem);  // plane k is x = k + 1
    unsigned char* p1 = smem + kU32Bytes;
    for (int i = threadIdx.x; i < NX * PS; i += NT) {
        const int k = i / PS, rem = i - k * PS, y = rem / E, z = rem - y * E;
        U[i] = load_u0<SUB>(a, au, box, tile, k + 1, y, z);
    }
    if (a.levels > 1) clear_levels<15, NT>(p1, 1, a, rec);
    // Two x-lines per thread: b, flags (a byte per cell) and the x halos in registers.
    int off[2];
    float b[2][NX], hlo[2], hhi[2];
    uint32_t fw[2][(NX + 3) / 4];
    // Planes where every lane's line is fully open (all six faces) or not Active.
    uint32_t open[2];
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        int y = 1, z = 1;
        const bool own = owned_line(threadIdx.x, l, y, z);
        off[l] = y * E + z;
        hlo[l] = own ? load_u0<SUB>(a, au, box, tile, 0, y, z) : 0.0f;
        hhi[l] = own ? load_u0<SUB>(a, au, box, tile, SUB, y, z) : 0.0f;
        uint32_t op = 0;
#pragma unroll
        for (int q = 0; q < (NX + 3) / 4; ++q) fw[l][q] = 0u;
#pragma unroll
        for (int k = 0; k < NX; ++k) {
            b[l][k] = own ? gb[((k + 1) * SUB + y) * SUB + z] : 0.0f;
            const uint32_t fl = own ? (uint32_t)rec[a.level_off[0] + ((k + 1) * E + y) * E + z] : 0u;
            fw[l][k >> 2] |= fl << (8 * (k & 3));
            if ((fl & C_FACES) == C_FACES || !(fl & C_ACTIVE)) op |= 1u << k;
        }
        open[l] = __reduce_and_sync(0xffffffffu, op);
    }
    __syncthreads();
    const float w6 = W.inv[6];
    const float* rh = a.r_halo ? a.r_halo + (size_t)blockIdx.y * a.slot_stride + (size_t)tile * TC : nullptr;
    auto flag = [&](int l, int k) -> uint32_t { return (fw[l][k >> 2] >> (8 * (k & 3))) & 0xffu; };
    // b - A u at cell k of line l (xm, cc, xp: u on the line).
    auto residual = [&](int l, int k, float xm, float cc, float xp) -> float {
        const float* p = U + k * PS + off[l];
        const float ym = p[-E], yp = p[E], zm = p[-1], zp = p[1];
        if (open[l] >> k & 1u) {  // the same branch for the whole warp
            float res = __fsub_rn(0.0f, __fsub_rn(xm, cc));
            res = __fsub_rn(res, __fsub_rn(xp, cc));
            res = __fsub_rn(res, __fsub_rn(ym, cc));
            res = __fsub_rn(res, __fsub_rn(yp, cc));
            res = __fsub_rn(res, __fsub_rn(zm, cc));
            res = __fsub_rn(res, __fsub_rn(zp, cc));
            return __fsub_rn(b[l][k], res);
        }
        return residual6(flag(l, k), cc, xm, xp, ym, yp, zm, zp, b[l][k]);
    };
    const Sweeps smooth{a.boundary_itr, a.interior_itr, 0}, bottom{0, 0, a.bottom_itr};
    const bool coarse = a.levels > 1;
    const int legs = coarse ? 2 : 1;
    for (int pass = 0; pass < legs * a.n_vcycles; ++pass) {
        const bool down = coarse && pass % 2 == 0;
        const Sweeps S = coarse ? smooth : bottom;
        const int n = S.count();
        for (int s = 0; s < n; ++s) {
            const Take take = S.at(s);
            const uint32_t m4 = take.mask * 0x01010101u, v4 = take.value * 0x01010101u;
            float um[2];  // old u of the plane before the chunk
            um[0] = hlo[0];
            um[1] = hlo[1];
#pragma unroll
            for (int ch = 0; ch < NCH; ++ch) {
                float nu[2][CH];
                uint32_t tk[2];
#pragma unroll
                for (int l = 0; l < 2; ++l) {
                    // Keeps the compiler from holding every cell's face tests
                    // and weights, which do not change over the sweeps, in
                    // (spilled) registers.
                    asm volatile("" : "+r"(fw[l][ch]), "+r"(open[l]));
                    // Cells of the chunk that the sweep takes: bytes equal to v4 under m4.
                    const uint32_t x = (fw[l][ch] & m4) ^ v4;
                    tk[l] = (~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x)) & 0x80808080u;
                    const int k0 = ch * CH;
                    if (__any_sync(0xffffffffu, tk[l] != 0)) {
                        float cc = U[k0 * PS + off[l]];
                        float xm = um[l];
#pragma unroll
                        for (int c = 0; c < CH; ++c) {
                            const int k = k0 + c;
                            if (k >= NX) continue;
                            const float xp = k + 1 < NX ? U[(k + 1) * PS + off[l]] : hhi[l];
                            const float r = residual(l, k, xm, cc, xp);
                            const float w = (open[l] >> k & 1u) ? w6 : W.inv[__popc(flag(l, k) & C_FACES)];
                            nu[l][c] = __fadd_rn(cc, __fmul_rn(w, r));
                            xm = cc;
                            cc = xp;
                        }
                        um[l] = xm;
                    } else {
                        um[l] = U[min(k0 + CH - 1, NX - 1) * PS + off[l]];
                    }
                }
                __syncthreads();
#pragma unroll
                for (int l = 0; l < 2; ++l)
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        const int k = ch * CH + c;
                        if (k < NX && (tk[l] >> (8 * c + 7) & 1u)) U[k * PS + off[l]] = nu[l][c];
                    }
            }
        }
        __syncthreads();
        if (!down) continue;
        // Residual planes go through a ring of six 33 x 33 planes (in level 1's
        // two copies of u, idle until the restriction is done): coarse plane cx
        // needs fine planes 2cx-2 .. 2cx+1, and the next two are computed while
        // it is restricted.  Halo cells of the ring stay zero unless the lower
        // faces' residual is given.
        const Level L1 = level_at<15>(p1);
        float* const ring = L1.a;
        static_assert(6 * PS <= 2 * pad4(cells_of(15)), "the ring fits level 1's copies of u");
        for (int i = threadIdx.x; i < 6 * PS; i += NT) ring[i] = 0.0f;
        __syncthreads();
        if (rh) {
            for (int i = threadIdx.x; i < SUB * SUB; i += NT) ring[(i / SUB) * E + i % SUB] = rh[i];
        }
#pragma unroll
        for (int k = 0; k < NX; ++k) {
            constexpr int SL = 6;
            const int x = k + 1;  // fine plane
            float* const R = ring + (x % SL) * PS;
            if (rh && threadIdx.x < 2 * SUB) {  // lower y and z faces
                const int y = threadIdx.x < SUB ? 0 : threadIdx.x - SUB, z = threadIdx.x < SUB ? threadIdx.x : 0;
                R[y * E + z] = rh[(x * SUB + y) * SUB + z];
            }
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const float* p = U + k * PS + off[l];
                const float xm = k > 0 ? p[k > 0 ? -PS : 0] : hlo[l], xp = k + 1 < NX ? p[PS] : hhi[l];
                const float r = residual(l, k, xm, p[0], xp);
                if (l == 0 || threadIdx.x < NX * NX - NT) R[off[l]] = (flag(l, k) & C_ACTIVE) ? r : 0.0f;
            }
            if (x % 2 == 1 && x >= 3) {
                __syncthreads();
                restrict_plane_32(ring, L1, (x - 1) / 2, W.sc64);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 2 * pad4(cells_of(15)); i += NT) ring[i] = 0.0f;
        __syncthreads();
        vcycle_from<15, NT>(p1, a.levels - 1, a, W);
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            if (l == 1 && threadIdx.x >= NX * NX - NT) continue;
            const int y = off[l] / E, z = off[l] % E;
#pragma unroll 2
            for (int k = 0; k < NX; ++k) {
                float* p = U + k * PS + off[l];
                if (rec[a.level_off[0] + (k + 1) * PS + off[l]] & C_ACTIVE)
                    *p = prolongate_cell<17>(*p, L1.a, k + 1, y, z, W.sc8);
            }
        }
        __syncthreads();
    }
    float* gw = au + (size_t)tile * TC;
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        if (l == 1 && threadIdx.x >= NX * NX - NT) continue;
        const int y = off[l] / E, z = off[l] % E;
        for (int k = 0; k < NX; ++k) gw[((k + 1) * SUB + y) * SUB + z] = U[k * PS + off[l]];
    }
}

// A kernel's dynamic shared-memory limit is process-wide state.  Solvers on
// other host threads launch the same kernels with other level counts, so the
// limit is only ever raised, under a lock: a concurrent launch can never find
// it lowered between its own check and its launch.
std::mutex g_smem_mu;
std::map<std::pair<const void*, int>, size_t> g_smem_limit;

cudaError_t ensure_smem_limit(const void* kern, size_t smem) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_smem_mu);
    size_t& have = g_smem_limit[{kern, dev}];
    if (have >= smem) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) have = smem;
    return e;
}

template <int SUB, int NT>
cudaError_t launch_box(const VcycleArgs& a, dim3 grid, cudaStream_t stream) {
    const size_t smem = (size_t)levels_bytes<SUB - 1>(a.levels);
    const cudaError_t e = ensure_smem_limit((const void*)vcycle_kernel<SUB, NT>, smem);
    if (e != cudaSuccess) return e;
    vcycle_kernel<SUB, NT><<<grid, NT, smem, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_vcycle(const VcycleArgs& a, cudaStream_t stream) {
    if (a.nbox == 0) return cudaSuccess;
    if (a.levels < 1 || a.levels > kMaxLevels || (a.sub >> (a.levels - 1)) < 2) return cudaErrorInvalidValue;
    const dim3 grid(a.nbox, std::max(1, a.nslots));
    switch (a.sub) {
        case 8: return launch_box<8, 128>(a, grid, stream);
        case 16: return launch_box<16, 512>(a, grid, stream);
        case 32: {
            const size_t smem = smem_bytes_32(a.levels);
            const cudaError_t e = ensure_smem_limit((const void*)vcycle_kernel_32, smem);
            if (e != cudaSuccess) return e;
            vcycle_kernel_32<<<grid, kNT32, smem, stream>>>(a);
            return cudaGetLastError();
        }
        default: return cudaErrorNotSupported;
    }
}

}  // namespace hdd
