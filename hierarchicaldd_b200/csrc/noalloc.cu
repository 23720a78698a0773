// Allocation-free Laplacian + dot product on caller-owned device arrays.
//
// Some callers cannot call cudaMalloc at the point where they need the
// operator: a host framework whose caching allocator already owns the device
// memory budget, or a time-critical loop that must not take the implicit
// device synchronisation of an allocation.  This entry point lets them apply
// y = Project(A x) and read sum(x*y) with nothing allocated per call: the
// per-tile partial sums live in one fixed, file-scope device array.
//
// The kernel applies the tiled path's per-cell arithmetic on dense addresses:
// the same FP64 face sums in the same face order, so y is bit-identical to
// the tiled Laplacian on the same data; the dot sums the same FP32 products
// in FP64, per part of a tile and then over the parts, in an order of its own.  Cells
// outside the stored tiles read as zero (as they do in the tiled vectors) and
// are not written.
//
// The scratch array is shared by every call in the process: two calls whose
// kernels overlap on the GPU race on it.  Every slot a call reads is written
// earlier by that same call, so nothing needs clearing between calls.
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "dev_util.h"
#include "kernels.h"
#include "noalloc.h"

namespace hdd {
namespace {

constexpr int kNT = 256;
constexpr int kMaxDevices = 64;

// FP64 partial sums of x*y, at least one per tile, at most kNoAllocMaxTiles.
static __device__ __align__(256) double g_noalloc_partial[kNoAllocMaxTiles];

std::mutex g_addr_mu;
double* g_addr[kMaxDevices] = {nullptr};

// Work unit: kRowsPerUnit<S> y-rows of an S^3 tile over kPlanes x-planes, one
// thread per (y, z) column.  A thread marches its column along x with the
// previous, current and next value in registers; the z neighbours come from
// the adjacent lanes (a row of S lanes never crosses a warp), the y
// neighbours and the tile-face halos from L1/L2.  The planes are unrolled, so
// all of a unit's loads are in flight together and no index is divided.
// Rows of the caller's dense array start at any 4-byte offset, so loads are
// one float per lane, whole rows at a time.
//
// Bound: at 128^3 the 21 MB of x, flags and y are L2-resident between calls
// and the launch is latency; one CTA per 32^3 tile (64 CTAs looping over 128
// strided cells per thread, two divisions and six branches per cell) took
// 181 us a call with the reduction, these units (1024 CTAs) 18.5 us; on a
// ragged 75 x 93 x 61 box 34 and 12.3 us (10 of them the host's).
constexpr int kPlanes = 8;
template <int S>
struct DenseShape {
    static constexpr int RY = S == 32 ? 8 : S;      // rows per unit
    static constexpr int GT = S * RY;               // threads per unit
    static constexpr int G = kNT / GT;              // units per CTA
    static constexpr int NU = (S / RY) * (S / kPlanes);  // units per tile
};

// Slot = (tile, part) with `parts` parts per tile; a slot walks units part,
// part + parts, ... of its tile and writes one partial sum of x*y.
template <int S>
__global__ void __launch_bounds__(kNT) laplace_dot_dense_kernel(TileGeom g, const int* __restrict__ tile_xyz, int sx,
                                                                int sy, int sz, const float* __restrict__ xv,
                                                                float* __restrict__ yv, double* partial, int parts) {
    using D = DenseShape<S>;
    constexpr int RY = D::RY, GT = D::GT, S2 = S * S, NP = kPlanes;
    __shared__ double red[kNT / 32];
    const int i = threadIdx.x % GT, grp = threadIdx.x / GT;
    const int slot = blockIdx.x * D::G + grp;
    const bool valid = slot < g.ntiles * parts;
    const int t = valid ? slot / parts : 0, part = valid ? slot % parts : 0;
    const int ox = tile_xyz[3 * t] * S, oy = tile_xyz[3 * t + 1] * S, oz = tile_xyz[3 * t + 2] * S;
    bool nb[6];  // a neighbour across the tile face counts only if its tile is stored
#pragma unroll
    for (int f = 0; f < 6; ++f) nb[f] = g.nbr[6 * t + f] >= 0;
    const int z = i % S, gz = oz + z;
    const size_t px = (size_t)sy * sz;  // x-plane stride
    double acc = 0.0;
    for (int u = part; u < D::NU; u += parts) {
        const int y = (u % (S / RY)) * RY + i / S, gy = oy + y;
        const int x0 = (u / (S / RY)) * NP, gx0 = ox + x0;
        const bool col = valid && gy < sy && gz < sz;
        const size_t at = ((size_t)gx0 * sy + gy) * sz + gz;
        const uint16_t* fp = g.flags + (size_t)t * S2 * S + (size_t)x0 * S2 + y * S + z;
        const bool has_ym = y > 0 || nb[2], has_yp = gy + 1 < sy && (y < S - 1 || nb[3]);
        const bool has_zm = nb[4], has_zp = gz + 1 < sz && nb[5];  // read at the row's ends only
        float c[NP + 2];
        uint32_t fl[NP];
#pragma unroll
        for (int k = 0; k < NP + 2; ++k) {
            const int x = x0 + k - 1;
            const bool in = col && gx0 + k - 1 < sx && (x >= 0 || nb[0]) && (x < S || nb[1]);
            c[k] = in ? __ldg(xv + at + (size_t)(k - 1) * px) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) fl[k] = valid ? fp[k * S2] : 0u;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const bool in = col && gx0 + k < sx;
            const float* p = xv + at + (size_t)k * px;
            const float cv = c[k + 1];
            const float ym = in && has_ym ? __ldg(p - sz) : 0.0f, yp = in && has_yp ? __ldg(p + sz) : 0.0f;
            float zm = __shfl_up_sync(0xffffffffu, cv, 1, S), zp = __shfl_down_sync(0xffffffffu, cv, 1, S);
            if (z == 0) zm = in && has_zm ? __ldg(p - 1) : 0.0f;
            if (z == S - 1) zp = in && has_zp ? __ldg(p + 1) : 0.0f;
            float out = 0.0f;
            if (fl[k] & (C_ACTIVE | C_INTERFACE)) {
                const double cd = (double)cv;
                double r = 0.0;
                if (fl[k] & 1u) r -= ((double)c[k] - cd);
                if (fl[k] & 2u) r -= ((double)c[k + 2] - cd);
                if (fl[k] & 4u) r -= ((double)ym - cd);
                if (fl[k] & 8u) r -= ((double)yp - cd);
                if (fl[k] & 16u) r -= ((double)zm - cd);
                if (fl[k] & 32u) r -= ((double)zp - cd);
                out = (float)r;
            }
            if (in) yv[at + (size_t)k * px] = out;
            acc += (double)(cv * out);
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    constexpr int W = GT / 32;  // warps per slot
    if (i == 0 && valid) {
        double v = 0.0;
        for (int w = 0; w < W; ++w) v += red[grp * W + w];
        partial[slot] = v;
    }
}

// Parts per tile: as many as a tile has units while the partial sums fit the
// fixed array (from 32768 / parts tiles on there are CTAs enough without).
template <int S>
int parts_of(int ntiles) {
    int p = DenseShape<S>::NU;
    while (p > 1 && (long long)p * ntiles > kNoAllocMaxTiles) p /= 2;
    return p;
}

template <int S>
int launch_dense(const TileGeom& g, const int* tile_xyz, const int size[3], const float* x, float* y, double* partial,
                 cudaStream_t stream) {
    const int parts = parts_of<S>(g.ntiles), slots = g.ntiles * parts;
    laplace_dot_dense_kernel<S><<<(slots + DenseShape<S>::G - 1) / DenseShape<S>::G, kNT, 0, stream>>>(
        g, tile_xyz, size[0], size[1], size[2], x, y, partial, parts);
    dev::ck(cudaGetLastError(), "laplace_dot_dense_kernel");
    return slots;
}

// Device address of the scratch array on the current device (looked up once
// per device; the host symbol itself is not a device address).
double* scratch_address(int device) {
    if (device < 0 || device >= kMaxDevices) throw Error(HDD_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_addr_mu);
    if (!g_addr[device]) {
        void* p = nullptr;
        dev::ck(cudaGetSymbolAddress(&p, g_noalloc_partial), "cudaGetSymbolAddress(no-alloc scratch)");
        g_addr[device] = static_cast<double*>(p);
    }
    return g_addr[device];
}

}  // namespace

void multiply_dot_dense_device_noalloc(const TileGeom& g, const int* tile_xyz, const int size[3], int device,
                                       const float* x, float* y, double* dot, cudaStream_t stream) {
    if (g.ntiles > kNoAllocMaxTiles)
        throw Error(HDD_ERR_INVALID_ARGUMENT, "domain has " + std::to_string(g.ntiles) +
                                                  " stored tiles; the allocation-free path holds at most " +
                                                  std::to_string(kNoAllocMaxTiles));
    double* partial = scratch_address(device);
    int n = 0;
    if (g.ntiles > 0) {
        if (g.sub == 32) n = launch_dense<32>(g, tile_xyz, size, x, y, partial, stream);
        else if (g.sub == 16) n = launch_dense<16>(g, tile_xyz, size, x, y, partial, stream);
        else if (g.sub == 8) n = launch_dense<8>(g, tile_xyz, size, x, y, partial, stream);
        else throw Error(HDD_ERR_UNSUPPORTED, "tile edge must be 8, 16 or 32");
    }
    dev::ck(launch_reduce_sum(partial, n, dot, stream), "reduce_sum");
}

}  // namespace hdd
