// Whole-grid V-cycle, for domains whose coarse levels couple neighbouring
// subdomain boxes (an exterior region touching Active cells, as the
// reference generator's Neumann bubble: a coarse cell whose children are
// exterior and Active is Active, so it joins the boxes on either side of an
// interface plane).  The reference's CPU V-cycle runs on the whole grid
// (CPU/SPGrid_Library/SPGrid_V_Cycle_Helper.h:70-195), and so does this one:
// one launch per Jacobi sweep (from one copy of u to the other), restriction and
// prolongation per level, on dense x-slowest arrays; the bottom level's sweeps
// are one launch where it fits one CTA.  Float operations
// are those of the per-box kernels (and the reference), in the same order, so
// the result is the same bit for bit.
//
//   smoothing   SPGrid_Residual_Legacy.h:40-61, SPGrid_Correction_Legacy.h:35-76
//   restriction SPGrid_Restriction_Legacy.h:47-186 (the fine stencil 2c-2..2c+1)
//   prolongation SPGrid_Prolongation_Legacy.h:48-118 (parents (f+1)/2, 3/4-1/4 weights)
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <utility>

#include "hdd_common.h"
#include "kernels.h"

namespace hdd {

namespace {

constexpr int kGT = 256;

__device__ __forceinline__ size_t gidx(const int* n, int i, int j, int k) {
    return ((size_t)i * n[1] + j) * n[2] + k;
}

struct Dims3 {
    int n[3];
};

__device__ __forceinline__ float val_or_zero(const Dims3& d, const float* v, int i, int j, int k) {
    if (i < 0 || j < 0 || k < 0 || i >= d.n[0] || j >= d.n[1] || k >= d.n[2]) return 0.0f;
    return v[gidx(d.n, i, j, k)];
}

// b - A u at an Active cell (face order -x,+x,-y,+y,-z,+z).
__device__ __forceinline__ float g_cell_residual(const Dims3& d, const float* u, uint32_t fl, int i, int j, int k, float c,
                                                 float b) {
    float res = 0.0f;
    if (fl & 0x01u) res = __fsub_rn(res, __fsub_rn(val_or_zero(d, u, i - 1, j, k), c));
    if (fl & 0x02u) res = __fsub_rn(res, __fsub_rn(val_or_zero(d, u, i + 1, j, k), c));
    if (fl & 0x04u) res = __fsub_rn(res, __fsub_rn(val_or_zero(d, u, i, j - 1, k), c));
    if (fl & 0x08u) res = __fsub_rn(res, __fsub_rn(val_or_zero(d, u, i, j + 1, k), c));
    if (fl & 0x10u) res = __fsub_rn(res, __fsub_rn(val_or_zero(d, u, i, j, k - 1), c));
    if (fl & 0x20u) res = __fsub_rn(res, __fsub_rn(val_or_zero(d, u, i, j, k + 1), c));
    return __fsub_rn(b, res);
}

// r = b - A u at Active cells.
__global__ void __launch_bounds__(kGT) g_residual(Dims3 d, const uint8_t* __restrict__ f, const float* __restrict__ u,
                                                  float* __restrict__ r, const float* __restrict__ b, size_t n) {
    const size_t x = (size_t)blockIdx.x * kGT + threadIdx.x;
    if (x >= n) return;
    const uint32_t fl = f[x];
    if (!(fl & C_ACTIVE)) return;
    const int k = (int)(x % d.n[2]);
    const size_t t = x / d.n[2];
    const int j = (int)(t % d.n[1]), i = (int)(t / d.n[1]);
    r[x] = g_cell_residual(d, u, fl, i, j, k, u[x], b[x]);
}

// Sweep modes: 1 Boundary cells, 2 interior (Active, not Boundary), 3 all Active.
__device__ __forceinline__ bool g_takes(uint32_t fl, int mode) {
    const bool bnd = fl & C_BOUNDARY8;
    return (fl & C_ACTIVE) && ((mode == 3) || (mode == 1 && bnd) || (mode == 2 && !bnd));
}

// One Jacobi sweep from u to v: v = u + omega/face_count * r on the sweep's
// cells, v = u elsewhere.
__global__ void __launch_bounds__(kGT) g_sweep(Dims3 d, const uint8_t* __restrict__ f, const float* __restrict__ u,
                                               float* __restrict__ v, const float* __restrict__ b, size_t n, int mode,
                                               VcycleWeights w) {
    const size_t x = (size_t)blockIdx.x * kGT + threadIdx.x;
    if (x >= n) return;
    const uint32_t fl = f[x];
    float c = u[x];
    if (g_takes(fl, mode)) {
        const int k = (int)(x % d.n[2]);
        const size_t t = x / d.n[2];
        const int j = (int)(t % d.n[1]), i = (int)(t / d.n[1]);
        const float r = g_cell_residual(d, u, fl, i, j, k, c, b[x]);
        c = __fadd_rn(c, __fmul_rn(w.inv_diag[__popc(fl & C_FACES)], r));
    }
    v[x] = c;
}

// The bottom level's sweeps (mode 3) in one CTA, the grid with a halo of zeros
// in shared memory: two copies of u, b and the flags.  A sweep costs one CTA
// barrier instead of two launches (the whole V-cycle of a 48^3 domain, three
// levels, 1845 us before, 396 us now).
constexpr int kBottomT = 1024;
__global__ void __launch_bounds__(kBottomT) g_bottom(Dims3 d, const uint8_t* __restrict__ f, float* __restrict__ u,
                                                     const float* __restrict__ b, int sweeps, VcycleWeights w) {
    extern __shared__ float sm[];
    __shared__ float inv[8];
    const int sy = d.n[2] + 2, sx = (d.n[1] + 2) * sy, np = (d.n[0] + 2) * sx;
    float *cur = sm, *nxt = sm + np, *bs = sm + 2 * np;
    uint8_t* fs = reinterpret_cast<uint8_t*>(sm + 3 * np);
    if (threadIdx.x < 8) inv[threadIdx.x] = w.inv_diag[threadIdx.x];
    for (int q = threadIdx.x; q < np; q += kBottomT) {
        const int i = q / sx - 1, j = q % sx / sy - 1, k = q % sy - 1;
        const bool in = i >= 0 && j >= 0 && k >= 0 && i < d.n[0] && j < d.n[1] && k < d.n[2];
        const size_t x = in ? gidx(d.n, i, j, k) : 0;
        const float c = in ? u[x] : 0.0f;
        cur[q] = c;
        nxt[q] = c;
        bs[q] = in ? b[x] : 0.0f;
        fs[q] = in ? f[x] : 0;
    }
    __syncthreads();
    for (int s = 0; s < sweeps; ++s) {
        for (int q = threadIdx.x; q < np; q += kBottomT) {
            const uint32_t fl = fs[q];
            if (!(fl & C_ACTIVE)) continue;
            const float c = cur[q];
            float res = 0.0f;
            if (fl & 0x01u) res = __fsub_rn(res, __fsub_rn(cur[q - sx], c));
            if (fl & 0x02u) res = __fsub_rn(res, __fsub_rn(cur[q + sx], c));
            if (fl & 0x04u) res = __fsub_rn(res, __fsub_rn(cur[q - sy], c));
            if (fl & 0x08u) res = __fsub_rn(res, __fsub_rn(cur[q + sy], c));
            if (fl & 0x10u) res = __fsub_rn(res, __fsub_rn(cur[q - 1], c));
            if (fl & 0x20u) res = __fsub_rn(res, __fsub_rn(cur[q + 1], c));
            nxt[q] = __fadd_rn(c, __fmul_rn(inv[__popc(fl & C_FACES)], __fsub_rn(bs[q], res)));
        }
        __syncthreads();
        float* t = cur;
        cur = nxt;
        nxt = t;
    }
    for (int q = threadIdx.x; q < np; q += kBottomT)
        if (fs[q] & C_ACTIVE) u[gidx(d.n, q / sx - 1, q % sx / sy - 1, q % sy - 1)] = cur[q];
}

// Coarse b at Active coarse cells from the fine residual (every fine cell of
// the stencil, whatever its flag; outside the grid counts zero).
__global__ void __launch_bounds__(kGT) g_restrict(Dims3 cd, const uint8_t* __restrict__ cf, float* __restrict__ cb,
                                                  Dims3 fd, const float* __restrict__ fr, size_t n, VcycleWeights w) {
    const size_t x = (size_t)blockIdx.x * kGT + threadIdx.x;
    if (x >= n) return;
    if (!(cf[x] & C_ACTIVE)) return;
    const int k = (int)(x % cd.n[2]);
    const size_t t = x / cd.n[2];
    const int j = (int)(t % cd.n[1]), i = (int)(t / cd.n[1]);
    float acc = 0.0f;
#pragma unroll
    for (int i2 = 0; i2 < 4; ++i2)
#pragma unroll
        for (int j2 = 0; j2 < 4; ++j2)
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2)
                acc = __fadd_rn(acc, __fmul_rn(w.restrict_w[(i2 * 4 + j2) * 4 + k2],
                                               val_or_zero(fd, fr, 2 * i - 2 + i2, 2 * j - 2 + j2, 2 * k - 2 + k2)));
    cb[x] = acc;
}

// Fine u += prolongated coarse u at Active fine cells.
__global__ void __launch_bounds__(kGT) g_prolong(Dims3 fd, const uint8_t* __restrict__ ff, float* __restrict__ fu,
                                                 Dims3 cd, const float* __restrict__ cu, size_t n, VcycleWeights w) {
    const size_t x = (size_t)blockIdx.x * kGT + threadIdx.x;
    if (x >= n) return;
    if (!(ff[x] & C_ACTIVE)) return;
    const int k = (int)(x % fd.n[2]);
    const size_t t = x / fd.n[2];
    const int j = (int)(t % fd.n[1]), i = (int)(t / fd.n[1]);
    const int ci = (i + 1) >> 1, cj = (j + 1) >> 1, ck = (k + 1) >> 1;
    const int pi = 1 - (i - (2 * ci - 1)), pj = 1 - (j - (2 * cj - 1)), pk = 1 - (k - (2 * ck - 1));
    float acc = fu[x];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                acc = __fadd_rn(acc, __fmul_rn(w.prolong_w[((a ^ pi) * 2 + (b ^ pj)) * 2 + (e ^ pk)],
                                               val_or_zero(cd, cu, ci + a - pi, cj + b - pj, ck + e - pk)));
    fu[x] = acc;
}

// Level-0 staging between the tiled vectors and the dense arrays.
// to_dense: dense[c] = tiled value (0 outside stored tiles) where keep[c],
// else 0; keep = Active when active_only, else every cell.
__global__ void __launch_bounds__(kGT) g_from_tiles(TileGeom g, const int* __restrict__ txyz, Dims3 d,
                                                    const float* __restrict__ tiled, float* __restrict__ dense,
                                                    const uint8_t* __restrict__ f0, int drop_active,
                                                    int drop_other) {
    const int t = blockIdx.x, S = g.sub, TC = S * S * S;
    const int ox = txyz[3 * t] * S, oy = txyz[3 * t + 1] * S, oz = txyz[3 * t + 2] * S;
    for (int c = threadIdx.x; c < TC; c += kGT) {
        const int z = c % S, tt = c / S, y = tt % S, xx = tt / S;
        const int gx = ox + xx, gy = oy + y, gz = oz + z;
        if (gx >= d.n[0] || gy >= d.n[1] || gz >= d.n[2]) continue;
        const size_t di = gidx(d.n, gx, gy, gz);
        const bool act = f0[di] & C_ACTIVE;
        float v = tiled[(size_t)t * TC + c];
        if ((act && drop_active) || (!act && drop_other)) v = 0.0f;
        dense[di] = v;
    }
}

// tiled[c] = dense at every stored cell that is not Interface (the V-cycle's
// cells; the interface values stay as they are).
__global__ void __launch_bounds__(kGT) g_to_tiles(TileGeom g, const int* __restrict__ txyz, Dims3 d,
                                                  const float* __restrict__ dense, float* __restrict__ tiled) {
    const int t = blockIdx.x, S = g.sub, TC = S * S * S;
    const int ox = txyz[3 * t] * S, oy = txyz[3 * t + 1] * S, oz = txyz[3 * t + 2] * S;
    for (int c = threadIdx.x; c < TC; c += kGT) {
        const int z = c % S, tt = c / S, y = tt % S, xx = tt / S;
        const int gx = ox + xx, gy = oy + y, gz = oz + z;
        if (gx >= d.n[0] || gy >= d.n[1] || gz >= d.n[2]) continue;
        const size_t q = (size_t)t * TC + c;
        if (g.flags[q] & C_INTERFACE) continue;
        tiled[q] = dense[gidx(d.n, gx, gy, gz)];
    }
}

// Shared memory of the one-CTA bottom: a level of up to 23^3 cells.
constexpr size_t kBottomSmem = 200 * 1024;
void allow_bottom_smem() {
    const cudaError_t e = cudaFuncSetAttribute(g_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBottomSmem);
    if (e != cudaSuccess) throw Error(HDD_ERR_CUDA, std::string("smem attr: ") + cudaGetErrorString(e));
}

unsigned blocks_for(size_t n) { return (unsigned)((n + kGT - 1) / kGT); }

}  // namespace

long long launch_vcycle_global(const GlobalVcycleArgs& a, const TileGeom& g, const int* tile_xyz, float* u,
                               const float* b, const float* r_halo, cudaStream_t st) {
    long long launches = 0;
    auto ok = [&](cudaError_t e) {
        if (e != cudaSuccess) throw Error(HDD_ERR_CUDA, std::string("whole-grid V-cycle: ") + cudaGetErrorString(e));
    };
    auto dims = [&](int l) {
        Dims3 d;
        for (int q = 0; q < 3; ++q) d.n[q] = a.dims[l][q];
        return d;
    };
    auto count = [&](int l) { return (size_t)a.dims[l][0] * a.dims[l][1] * a.dims[l][2]; };
    const Dims3 d0 = dims(0);
    const size_t n0 = count(0);
    // Level-0 state: b from the tiles; u's interface (halo) values and/or
    // initial interior from the tiles; r zero, or the given face residual.
    ok(cudaMemsetAsync(a.b[0], 0, n0 * sizeof(float), st));
    g_from_tiles<<<g.ntiles, kGT, 0, st>>>(g, tile_xyz, d0, b, a.b[0], a.f[0], 0, 0);
    ok(cudaMemsetAsync(a.u[0], 0, n0 * sizeof(float), st));
    if (a.halo_from_u || !a.zero_init)
        g_from_tiles<<<g.ntiles, kGT, 0, st>>>(g, tile_xyz, d0, u, a.u[0], a.f[0], a.zero_init, !a.halo_from_u);
    ok(cudaMemsetAsync(a.r[0], 0, n0 * sizeof(float), st));
    if (r_halo) g_from_tiles<<<g.ntiles, kGT, 0, st>>>(g, tile_xyz, d0, r_halo, a.r[0], a.f[0], 1, 0);
    launches += 3;
    const int L = a.levels;
    // u of each level and the copy a sweep writes.
    float *cur[kMaxLevels], *alt[kMaxLevels];
    for (int l = 0; l < L; ++l) { cur[l] = a.u[l]; alt[l] = a.t[l]; }
    auto sweep = [&](int l, int mode) {
        g_sweep<<<blocks_for(count(l)), kGT, 0, st>>>(dims(l), a.f[l], cur[l], alt[l], a.b[l], count(l), mode, a.w);
        std::swap(cur[l], alt[l]);
        ++launches;
    };
    auto smooth = [&](int l) {
        for (int i = 0; i < a.boundary_itr; ++i) sweep(l, 1);
        for (int i = 0; i < a.interior_itr; ++i) sweep(l, 2);
        for (int i = 0; i < a.boundary_itr; ++i) sweep(l, 1);
    };
    const int lb = L - 1;
    const size_t bottom_smem = 13 * (size_t)(a.dims[lb][0] + 2) * (a.dims[lb][1] + 2) * (a.dims[lb][2] + 2);
    for (int cycle = 0; cycle < a.n_vcycles; ++cycle) {
        for (int l = 0; l < lb; ++l) {
            smooth(l);
            g_residual<<<blocks_for(count(l)), kGT, 0, st>>>(dims(l), a.f[l], cur[l], a.r[l], a.b[l], count(l));
            ok(cudaMemsetAsync(cur[l + 1], 0, count(l + 1) * sizeof(float), st));
            g_restrict<<<blocks_for(count(l + 1)), kGT, 0, st>>>(dims(l + 1), a.f[l + 1], a.b[l + 1], dims(l), a.r[l],
                                                                  count(l + 1), a.w);
            launches += 2;
        }
        if (bottom_smem <= kBottomSmem) {
            allow_bottom_smem();
            g_bottom<<<1, kBottomT, bottom_smem, st>>>(dims(lb), a.f[lb], cur[lb], a.b[lb], a.bottom_itr, a.w);
            ++launches;
        } else {
            for (int i = 0; i < a.bottom_itr; ++i) sweep(lb, 3);
        }
        for (int l = lb - 1; l >= 0; --l) {
            g_prolong<<<blocks_for(count(l)), kGT, 0, st>>>(dims(l), a.f[l], cur[l], dims(l + 1), cur[l + 1], count(l),
                                                             a.w);
            ++launches;
            smooth(l);
        }
    }
    g_to_tiles<<<g.ntiles, kGT, 0, st>>>(g, tile_xyz, d0, cur[0], u);
    ++launches;
    ok(cudaGetLastError());
    return launches;
}

}  // namespace hdd
