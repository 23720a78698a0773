// Supernodal solves with one CTA per elimination tree (or per group of trees
// with the same factor), forward and backward in one launch; or the two halves
// of the lower trees of a larger plan (sn_solve.cu).
//
// Used for plans whose trees are small enough that a tree's unknowns fit one
// CTA's shared memory: the subdomain interiors of every interface level, the
// interface systems of small domains, and the lower trees of the others.
//
// * The vector of a tree stays in shared memory (FP64) for both directions:
//   the assembled f, then y, then x, each overwriting the last.
// * Fronts of one height (forward) or depth (backward) run together, one warp
//   per front; a front too large for one warp is cut into row chunks and
//   column slices whose partial sums are added in slice order after a barrier.
//   Which warp does what, in which order, is fixed when the plan is built.
// * A warp's whole work, coefficients and indices alike, is one linear stream
//   of 512-byte lines (16 bytes a lane) in the order it is used, read through a
//   ring of kDepth lines in shared memory by cp.async: loads are always whole
//   lines, run ahead across fronts, levels and barriers, and no address depends
//   on a loaded value.  With the same schedule but the records, gather lists
//   and coefficients read where they are used, a tree level cost 5 to 7 us of
//   dependent loads (102 us for the 64 16^3 interiors, n = 1423, of a 64^3
//   domain); it now takes 38 us, against 92 us as separate forward and
//   backward launches of one CTA per block of a front.  32^3 interiors: 169 us
//   for the 64 of a 128^3 domain (345 before), 186 us for 216 (590 before).
//   The price is memory: with headers, indices, rows and columns padded to the
//   lanes and both directions stored, streams are three to four times the
//   coefficients of both directions, 15 times for the tiny fronts of sparse domains.
//   What is left is latency on four warps a scheduler: about 560 cycles of
//   set-up per product and 450 per barrier.  The 32^3 interiors issue in 41 % of
//   the cycles; the conversions of coefficients to FP64 (16 per 2 KB and warp)
//   keep their pipe 40 % busy.
// * Members of a class (trees whose factors are equal: most subdomains of a
//   domain have the same interior matrix) share one stream, and up to K of
//   them are solved by one CTA, which then feeds K products from every
//   coefficient it loads.
// * Backward, x_J = Fw^T [y_J; x_R], streams the transposed blocks: both
//   directions then are products with lanes on rows, without the five shuffle
//   rounds per column that a reduction over rows takes.
//
// The arithmetic is that of sn_solve.cu: FP32 coefficients, exact FP32 x FP32
// products accumulated in FP64, FP64 vectors between fronts, sums in an order
// that depends neither on K nor on scheduling.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "dev_util.h"
#include "sn_streams.h"

namespace hdd {

namespace {

struct RView {
    const RGroup* groups;
    const RWarp* warps;
    const int* off;                    // member -> first unknown
    const int* perm;
    const int* ext;                    // cut trees: unknowns of the plan above, from the member's first
    const char* stream;
    double *upd, *y;
    double* top_upd;                   // cut trees: the plan above's update vectors and solution
    const double* top_x;
    long long ld_upd, ld_y, ld_top_upd, ld_top_x, ld_b, ld_x;
    int ngroups, nrhs;
    int* ctr;                          // forward: counters to clear
    long long n_ctr;
    const int* gate;                   // test seam: nonzero = wait for it to clear
    int* err;
    long long spin_limit;
};

template <int K>
__device__ __forceinline__ void load_k(double (&d)[K], const double* p) {
    if constexpr (K == 1) {
        d[0] = p[0];
    } else {
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const double2 t = *reinterpret_cast<const double2*>(p + k);
            d[k] = t.x;
            d[k + 1] = t.y;
        }
    }
}
template <int K>
__device__ __forceinline__ void store_k(double* p, const double (&d)[K]) {
    if constexpr (K == 1) {
        p[0] = d[0];
    } else {
#pragma unroll
        for (int k = 0; k < K; k += 2) *reinterpret_cast<double2*>(p + k) = make_double2(d[k], d[k + 1]);
    }
}

// One warp's stream through a ring of D batches.  Every lane copies and reads
// its own 16 bytes of a line, so a batch needs no more than the lane's own wait.
// Copies run past the stream's end (the buffer is padded), so nothing counts
// lines.
template <int D>
struct Stream {
    const char* g;    // this lane's next bytes to copy
    char* ring;       // this lane's bytes of the ring's first line
    int pos;          // byte offset of the batch to read next

    __device__ __forceinline__ void fill(int at) {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(ring) + at;
        asm volatile(
            "cp.async.cg.shared.global [%0], [%1], 16;\n\t"
            "cp.async.cg.shared.global [%0+512], [%1+512], 16;\n\t"
            "cp.async.cg.shared.global [%0+1024], [%1+1024], 16;\n\t"
            "cp.async.cg.shared.global [%0+1536], [%1+1536], 16;\n\t"
            "cp.async.commit_group;"
            :
            : "r"(a), "l"(g)
            : "memory");
        g += kBatchBytes;
    }
    __device__ __forceinline__ void start(const char* p, char* r) {
        const int lane = threadIdx.x & 31;
        g = p + lane * 16;
        ring = r + lane * 16;
        pos = 0;
#pragma unroll
        for (int i = 0; i < D; ++i) fill(i * kBatchBytes);
    }
    __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" : : "n"(D - 1) : "memory"); }
    template <class T>
    __device__ __forceinline__ T line(int i) const {
        return *reinterpret_cast<const T*>(ring + pos + i * kLine);
    }
    // The batch is used up: its space is filled again.
    __device__ __forceinline__ void pop() {
        fill(pos);
        pos = pos + kBatchBytes == D * kBatchBytes ? 0 : pos + kBatchBytes;
    }
};

template <int K>
struct Vec {
    double *m, *upd, *top;  // M; update slots in global memory (GS); the plan above's update vectors
};

template <int K>
__device__ __forceinline__ void add_k(double (&s)[K], const double (&w)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) s[k] += w[k];
}

// The sum of two children's entries.
template <int K, bool GS>
__device__ __forceinline__ void pair_sum(const Vec<K>& V, int e0, int e1, double (&s)[K]) {
    const double* p = GS ? V.upd : V.m;
    double w[K];
    load_k<K>(s, p + (size_t)e0 * K);
    load_k<K>(w, p + (size_t)e1 * K);
    add_k<K>(s, w);
}

template <int K, bool GS>
__device__ __forceinline__ void put(const Vec<K>& V, int dst, bool top, const double (&s)[K]) {
    if (GS && dst < 0) {
        store_k<K>(V.upd + (size_t)(-1 - dst) * K, s);
    } else if (!GS && K == 1 && top && dst < 0) {
        V.top[-1 - dst] = s[0];
    } else {
        store_k<K>(V.m + (size_t)dst * K, s);
    }
}

template <int K, bool GS>
__device__ __forceinline__ void assemble_item(const Vec<K>& V, const int4 it) {
    double* p = (GS && it.w ? V.upd : V.m) + (size_t)it.x * K;
    double s[K], w[K];
    load_k<K>(s, p);
    pair_sum<K, GS>(V, it.y, it.z, w);
    add_k<K>(s, w);
    store_k<K>(p, s);
}

// Four steps: the batch's coefficients times the inputs at indices j.
template <int K, int D>
__device__ __forceinline__ void four_steps(Stream<D>& S, const double* m, const int (&j)[4], double (&acc)[K][4]) {
    S.wait();
    float4 w[4];
    double in[4][K];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        w[u] = S.template line<float4>(u);
        load_k<K>(in[u], m + (size_t)j[u] * K);
    }
    S.pop();
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            acc[k][0] = fma((double)w[u].x, in[u][k], acc[k][0]);
            acc[k][1] = fma((double)w[u].y, in[u][k], acc[k][1]);
            acc[k][2] = fma((double)w[u].z, in[u][k], acc[k][2]);
            acc[k][3] = fma((double)w[u].w, in[u][k], acc[k][3]);
        }
}

template <int K, int D, bool GS>
__device__ __forceinline__ void op_product(Stream<D>& S, const Vec<K>& V, const int4 h, const int4 dst, const int4 p2,
                                           const int4 p3) {
    const int lmq = (h.x >> 4) & 15, flags = (h.x >> 8) & 255, groups = h.x >> 16;
    double acc[K][4];
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[k][e] = 0.0;
    if (flags & kTransposed) {
        int4 ix[4] = {p2, p3, p2, p3};
        int n = 2;  // index lines in ix, eight steps each
        for (int g = 0; g < groups;) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q < n && g < groups) {
                    const int j[4] = {ix[q].x & 0xffff, (int)((uint32_t)ix[q].x >> 16), ix[q].y & 0xffff,
                                      (int)((uint32_t)ix[q].y >> 16)};
                    four_steps<K, D>(S, V.m, j, acc);
                    ++g;
                }
                if (q < n && g < groups) {
                    const int j[4] = {ix[q].z & 0xffff, (int)((uint32_t)ix[q].z >> 16), ix[q].w & 0xffff,
                                      (int)((uint32_t)ix[q].w >> 16)};
                    four_steps<K, D>(S, V.m, j, acc);
                    ++g;
                }
            }
            if (g < groups) {
                S.wait();
#pragma unroll
                for (int q = 0; q < 4; ++q) ix[q] = S.template line<int4>(q);
                S.pop();
                n = 4;
            }
        }
    } else {
        if (flags & kItem) {
            if (p3.x >= 0) assemble_item<K, GS>(V, p3);
            __syncwarp();
        }
        int c = h.y & 0xffff;
        const int d = (h.y >> 16) & 15;
        for (int g = 1; g < groups; ++g) {
            const int j[4] = {c, c + d, c + 2 * d, c + 3 * d};
            four_steps<K, D>(S, V.m, j, acc);
            c += 4 * d;
        }
        const int j[4] = {h.z & 0xffff, (int)((uint32_t)h.z >> 16), h.w & 0xffff, (int)((uint32_t)h.w >> 16)};
        four_steps<K, D>(S, V.m, j, acc);
    }
    // The column slices, summed by a fixed shuffle tree.
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
        if ((1 << lmq) <= o) {
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[k][e] += __shfl_xor_sync(0xffffffffu, acc[k][e], o);
        }
    __syncwarp();  // every lane has read the front's inputs: its unknowns may be overwritten
    if ((threadIdx.x & 31) >> lmq == 0) {
        const int d[4] = {dst.x, dst.y, dst.z, dst.w};
        if (flags & kPairs) {
            const int a[4] = {p2.x, p2.y, p2.z, p2.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                double s[K];
                pair_sum<K, GS>(V, a[e] & 0xffff, (int)((uint32_t)a[e] >> 16), s);
#pragma unroll
                for (int k = 0; k < K; ++k) acc[k][e] = s[k] + acc[k][e];
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            double s[K];
#pragma unroll
            for (int k = 0; k < K; ++k) s[k] = acc[k][e];
            put<K, GS>(V, d[e], flags & kTopRoot, s);
        }
    }
}

template <int K, bool GS>
__device__ __forceinline__ void finish_item(const Vec<K>& V, const int4 it, int nsl, int stride, bool top) {
    double t[K], s[K];
    pair_sum<K, GS>(V, it.z, it.w, s);
    const double* p = V.m + (size_t)it.x * K;
    load_k<K>(t, p);
#pragma unroll 4
    for (int q = 1; q < nsl; ++q) {
        double w[K];
        load_k<K>(w, p + (size_t)(q * stride) * K);
        add_k<K>(t, w);
    }
    add_k<K>(s, t);
    put<K, GS>(V, it.y, top, s);
}

// Runs a stream to its end.
template <int K, int D, bool GS>
__device__ __forceinline__ void run_stream(Stream<D>& S, const Vec<K>& V) {
    for (;;) {
        S.wait();
        const int4 h = S.template line<int4>(0), l1 = S.template line<int4>(1), l2 = S.template line<int4>(2),
                   l3 = S.template line<int4>(3);
        S.pop();
        const int type = h.x & 15, count = h.x >> 16;
        if (type == kProduct) {
            op_product<K, D, GS>(S, V, h, l1, l2, l3);
        } else if (type == kAssemble) {
            if (l1.x >= 0) assemble_item<K, GS>(V, l1);
            if (count > 1 && l2.x >= 0) assemble_item<K, GS>(V, l2);
            if (count > 2 && l3.x >= 0) assemble_item<K, GS>(V, l3);
        } else if (type == kFinish) {
            const bool top = (h.x >> 8) & kTopRoot;
            if (l1.x >= 0) finish_item<K, GS>(V, l1, h.y & 0xffff, h.z, top);
            if (count > 1 && l2.x >= 0) finish_item<K, GS>(V, l2, h.y & 0xffff, h.z, top);
            if (count > 2 && l3.x >= 0) finish_item<K, GS>(V, l3, h.y & 0xffff, h.z, top);
        } else if (type == kEnd) {
            return;
        }
        int bars = (int)((uint32_t)h.y >> 20);
        if (bars == 0) __syncwarp();
        for (; bars > 0; --bars) __syncthreads();
    }
}

// MODE: whole trees, both directions; or the forward / backward half of cut
// trees, with y kept in global memory between the halves.
constexpr int kWhole = 0, kForward = 1, kBackward = 2;

// What a launch does once besides its groups.
template <int NT, int MODE>
__device__ __forceinline__ void once(const RView& P) {
    if (MODE != kBackward && blockIdx.x == 0 && threadIdx.x == 0) {
        // Test seam: a set gate is a dependency that nothing satisfies.
        bool ok = false;
        for (long long i = 0; i < P.spin_limit && !ok; ++i) {
            ok = *reinterpret_cast<const volatile int*>(P.gate) == 0;
            if (!ok) __nanosleep(128);
        }
        if (!ok) atomicExch(P.err, 1);
    }
    if (MODE == kForward)
        for (long long i = (long long)blockIdx.x * NT + threadIdx.x; i < P.n_ctr; i += (long long)gridDim.x * NT) P.ctr[i] = 0;
}

template <int K, int KM, int NT, int MODE, bool GS>
__device__ __forceinline__ void solve_group(const RView& P, const RGroup& G, int rhs, const float* b_old,
                                            float* x_old, char* smem, bool first) {
    constexpr int D = depth_of(KM);
    const int warp = threadIdx.x >> 5;
    const RWarp W = P.warps[G.warps + warp];
    // Shared memory: the warps' rings, then M.
    Vec<K> V;
    V.m = reinterpret_cast<double*>(smem + (size_t)(NT / 32) * D * kBatchBytes);
    V.upd = P.upd + rhs * P.ld_upd + G.upd;
    V.top = P.top_upd + rhs * P.ld_top_upd + G.top;
    double* y = P.y + rhs * P.ld_y + G.y;
    Stream<D> S;
    S.start(P.stream + G.stream + (long long)(W.first + (MODE == kBackward ? W.nf : 0)) * kLine,
            smem + (size_t)warp * D * kBatchBytes);
    int off[K];
#pragma unroll
    for (int k = 0; k < K; ++k) off[k] = P.off[G.member0 + min(k, G.count - 1)];
    const int* perm = P.perm + G.perm;
    if (first) once<NT, MODE>(P);
    if (threadIdx.x < K) V.m[(size_t)(G.n + G.next) * K + threadIdx.x] = 0.0;  // the zero
    if (MODE != kBackward) {
        const float* b = b_old + rhs * P.ld_b;
        for (int i = threadIdx.x; i < G.n; i += NT) {
            const int p = perm[i];
            double d[K];
#pragma unroll
            for (int k = 0; k < K; ++k) d[k] = (double)b[off[k] + p];
            store_k<K>(V.m + (size_t)i * K, d);
        }
        __syncthreads();
        run_stream<K, D, GS>(S, V);
    }
    if (MODE == kForward) {
        __syncthreads();
        for (int i = threadIdx.x; i < G.n; i += NT) y[i] = V.m[i];
    }
    if (MODE == kBackward) {
        const double* tx = P.top_x + rhs * P.ld_top_x;
        for (int i = threadIdx.x; i < G.n; i += NT) V.m[i] = y[i];
        for (int i = threadIdx.x; i < G.next; i += NT) V.m[G.n + i] = tx[off[0] + P.ext[G.ext + i]];
        __syncthreads();
    }
    if (MODE != kForward) {
        run_stream<K, D, GS>(S, V);
        __syncthreads();
        float* x = x_old + rhs * P.ld_x;
        for (int i = threadIdx.x; i < G.n; i += NT) {
            const int p = perm[i];
            double d[K];
            load_k<K>(d, V.m + (size_t)i * K);
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < G.count) x[off[k] + p] = (float)d[k];
        }
    }
    asm volatile("cp.async.wait_group 0;" : : : "memory");
    __syncthreads();  // the next group reuses shared memory
}

constexpr int resident_min_blocks(int nt) { return 512 / nt; }

template <int KM, int NT, int MODE, bool GS>
__global__ void __launch_bounds__(NT, resident_min_blocks(NT))
    sn_resident_kernel(RView P, const float* __restrict__ b_old, float* __restrict__ x_old) {
    extern __shared__ __align__(16) char smem[];
    for (int w = blockIdx.x; w < P.ngroups * P.nrhs; w += gridDim.x) {
        const RGroup G = P.groups[w / P.nrhs];
        const int rhs = w % P.nrhs;
        if (KM > 1 && G.count > 1) solve_group<KM, KM, NT, MODE, GS>(P, G, rhs, b_old, x_old, smem, w == (int)blockIdx.x);
        else solve_group<1, KM, NT, MODE, GS>(P, G, rhs, b_old, x_old, smem, w == (int)blockIdx.x);
    }
}

// Shared-memory limits only ever grow, so a later, smaller plan cannot
// invalidate an earlier plan's launches.
std::mutex g_smem_mu;
std::map<std::pair<const void*, int>, size_t> g_smem_limit;

template <int KM, int NT, int MODE, bool GS>
void prepare_kernel(int device, size_t smem, int& per_sm) {
    auto kern = sn_resident_kernel<KM, NT, MODE, GS>;
    std::lock_guard<std::mutex> lock(g_smem_mu);
    size_t& have = g_smem_limit[{(const void*)kern, device}];
    if (smem > have) {
        dev::ck(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attr");
        have = smem;
    }
    dev::ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem), "occupancy");
}

// The kernel instances.
template <int K, int N, bool G>
struct Instance {
    static constexpr int KM = K, NT = N;
    static constexpr bool GS = G;
};
template <class F>
void dispatch_cut(int nt, F f) {
    if (nt == 256) f(std::integral_constant<int, 256>());
    else f(std::integral_constant<int, 512>());
}
template <class F>
void dispatch_whole(int km, int nt, bool gs, F f) {
    if (nt == 128) {  // small trees: slots in shared memory (ResidentSchedule::plan)
        if (gs) throw Error(HDD_ERR_INTERNAL, "no kernel of four warps with slots in global memory");
        if (km == 1) f(Instance<1, 128, false>());
        else if (km == 2) f(Instance<2, 128, false>());
        else f(Instance<4, 128, false>());
    } else if (km == 1) {
        if (gs) f(Instance<1, 512, true>());
        else f(Instance<1, 512, false>());
    } else if (km == 2) {
        if (gs) f(Instance<2, 512, true>());
        else f(Instance<2, 512, false>());
    } else {
        if (gs) f(Instance<4, 512, true>());
        else f(Instance<4, 512, false>());
    }
}

}  // namespace

bool ResidentPlan::build(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets, dev::Staging& stage,
                         cudaStream_t s) {
    release();
    std::vector<Shape> shapes;
    std::vector<std::vector<Member>> members;
    whole_shapes(factors, offsets, shapes, members);
    for (size_t f = 0; f < factors.size(); ++f) n = std::max(n, offsets[f] + factors[f]->n);
    cut = false;
    return build_shapes(shapes, members, stage, s);
}

bool ResidentPlan::build_cut(const std::vector<Shape>& shapes, const std::vector<std::vector<Member>>& members,
                             dev::Staging& stage, cudaStream_t s) {
    release();
    cut = true;
    return build_shapes(shapes, members, stage, s);
}

bool ResidentPlan::build_shapes(const std::vector<Shape>& shapes, const std::vector<std::vector<Member>>& members,
                                dev::Staging& stage, cudaStream_t s) {
    int dev_id = 0, nsm = 0;
    dev::ck(cudaGetDevice(&dev_id), "cudaGetDevice");
    dev::ck(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev_id), "SM count");
    ResidentSchedule S;
    if (!S.plan(shapes, members, cut, nsm)) {
        release();
        return false;
    }
    max_n = S.max_n;
    km = S.km;
    nt = S.nt;
    smem = S.smem;
    global_slots = S.global_slots;
    ngroups = (int)S.groups.size();
    upd_len = S.upd_len;
    y_len = S.y_len;
    bytes = 0;
    float* d = nullptr;
    dev::upload_packed(S.streams(), S.total(), [&](size_t i) { return S.at(i); },
                       [&](size_t i, float* dst) { S.write(i, dst); }, stage, s, d, bytes);
    d_stream = reinterpret_cast<char*>(d);
    auto nonempty = [](std::vector<int>& v) -> const std::vector<int>& {
        if (v.empty()) v.push_back(0);
        return v;
    };
    d_groups = dev::upload(S.groups, s, bytes);
    d_warps = dev::upload(S.warps, s, bytes);
    d_off = dev::upload(nonempty(S.off), s, bytes);
    d_perm = dev::upload(nonempty(S.perm), s, bytes);
    d_ext = dev::upload(nonempty(S.ext), s, bytes);
    d_gate = dev::alloc_zero<int>(1, bytes, s);
    // Algorithmic bytes of one solve: each class's coefficients once per
    // direction, b read and x written.
    solve_bytes = 2 * 4.0 * S.coef + 8.0 * n;
    int per_sm = 0;
    if (cut) {
        dispatch_cut(nt, [&](auto t) {
            prepare_kernel<1, decltype(t)::value, kForward, false>(dev_id, smem, per_sm);
            prepare_kernel<1, decltype(t)::value, kBackward, false>(dev_id, smem, per_sm);
        });
    } else {
        dispatch_whole(km, nt, global_slots, [&](auto t) {
            using T = decltype(t);
            prepare_kernel<T::KM, T::NT, kWhole, T::GS>(dev_id, smem, per_sm);
        });
    }
    resident = std::max(1, per_sm) * nsm;
    dev::ck(cudaStreamSynchronize(s), "plan upload");
    return true;
}

void ResidentPlan::release() {
    dev::release(d_groups); dev::release(d_warps);
    dev::release(d_off); dev::release(d_perm); dev::release(d_ext); dev::release(d_stream); dev::release(d_gate);
    n = max_n = ngroups = 0;
    upd_len = y_len = 0;
    bytes = 0;
}

void ResidentPlan::launch(int mode, const ResidentScratch& sc, const TopVectors& top, int* err, int grid_div,
                          long long spin_limit, const float* b_old, float* x_old, cudaStream_t s, int nrhs,
                          long long ld_b, long long ld_x) const {
    const RView P{d_groups, d_warps, d_off, d_perm, d_ext, d_stream, sc.upd, sc.y, top.upd, top.x,
                  upd_len, y_len, top.ld_upd, top.ld_x, ld_b, ld_x, ngroups, nrhs, top.ctr, top.n_ctr, d_gate, err,
                  spin_limit};
    const int all = ngroups * nrhs;
    const int grid = grid_div > 1 ? std::min(all, std::max(1, (resident + grid_div - 1) / grid_div)) : all;
    if (mode == kWhole)
        dispatch_whole(km, nt, global_slots, [&](auto t) {
            using T = decltype(t);
            sn_resident_kernel<T::KM, T::NT, kWhole, T::GS><<<grid, T::NT, smem, s>>>(P, b_old, x_old);
        });
    else
        dispatch_cut(nt, [&](auto t) {
            constexpr int NT = decltype(t)::value;
            if (mode == kForward) sn_resident_kernel<1, NT, kForward, false><<<grid, NT, smem, s>>>(P, b_old, x_old);
            else sn_resident_kernel<1, NT, kBackward, false><<<grid, NT, smem, s>>>(P, b_old, x_old);
        });
    dev::ck(cudaGetLastError(), "sn resident");
}

void ResidentPlan::set_gate(int v, cudaStream_t s) {
    dev::ck(cudaMemcpyAsync(d_gate, &v, sizeof(int), cudaMemcpyHostToDevice, s), "gate");
    dev::ck(cudaStreamSynchronize(s), "gate");
}

}  // namespace hdd
