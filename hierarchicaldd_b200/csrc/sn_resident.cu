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
//   domain); it now takes 40 us, against 92 us as separate forward and
//   backward launches of one CTA per block of a front.  32^3 interiors: 170 us
//   for the 64 of a 128^3 domain (345 before), 191 us for 216 (590 before).
//   What is left is instruction issue: 16 conversions (4 cycles each on a
//   scheduler) and 16 FP64 multiply-adds per 2 KB of coefficients and warp,
//   about 560 cycles of set-up per product and 450 per barrier.
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
#include <array>
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "dev_util.h"
#include "sigma.h"

namespace hdd {

// Lines of one warp's stream from the class's first: forward, then backward.
struct RWarp {
    int first, nf, nb, pad;
};
// One CTA's work: `count` members of a class.
struct RGroup {
    long long stream;         // byte offset of the class's streams
    long long upd, y;         // offsets of the group's scratch, in doubles
    int n, perm;              // unknowns; offset of perm
    int next, ext;            // unknowns of the plan above that cut trees read; offset of their indices
    int warps;                // offset of the class's warps
    int member0, count, pad;
};

namespace {

constexpr int kLine = 512;              // bytes of a line: 16 a lane
constexpr int kBatch = 4;               // lines copied, waited for and released together
constexpr int kBatchBytes = kBatch * kLine;
// Batches in flight per warp (K trees per CTA; the vectors of more leave less room).
__host__ __device__ constexpr int depth_of(int k) { return k == 1 ? 4 : 2; }

// Operations of a stream.  Each starts with a batch whose first line is the
// header, an int4 for every lane: {type | log2 of the lanes on row quads << 4 |
// flags << 8, count, index, distance}.
enum : int {
    kEnd = 0,
    kNothing = 1,   // (a barrier)
    // Items on 1 to 3 lines (count), one per lane: {index, first, second entry,
    // 1 when the index is a slot (GS)}: M[index] += the two entries.
    kAssemble = 2,
    // A block of a front times its inputs: count groups of four steps (a batch
    // each), index: the lane's first column (forward), distance: from a lane's
    // column to its next.  Lines: destinations of four rows a lane; forward the
    // rows' pairs of children's entries (16 bits each) and one item of an
    // assembly before; backward the columns' indices for the first sixteen
    // steps (eight 16-bit indices a lane and line), a batch of four more such
    // lines following every further 32 steps.
    kProduct = 3,
    // Items on 1 to 3 lines: {first partial sum, destination, first, second
    // entry}; index: slices, distance: between their partial sums.
    kFinish = 4
};
constexpr int kBar = 1;        // CTA barrier after it
constexpr int kPairs = 2;      // the rows have children's entries
constexpr int kItem = 4;       // the product starts with an assembly
constexpr int kTransposed = 8;
constexpr int kTopRoot = 16;   // destinations -1 - entry are the plan above's update vectors
// Indices are into the CTA's array M: the vector, rows outside cut trees, a
// zero (a pair's missing entries), an unused entry (results of no row), partial
// sums and, where they fit, update slots.  GS: slots are in global memory
// instead (destination -1 - slot; a pair's entries are slots, slot 0 the zero).

struct RView {
    const RGroup* groups;
    const RWarp* warps;
    const int* off;                    // member -> first unknown
    const int* perm;
    const int* ext;                    // cut trees: unknowns of the plan above
    const char* stream;
    double *upd, *y;
    double* top_upd;                   // cut trees: the plan above's update vectors and solution
    const double* top_x;
    long long ld_upd, ld_y, ld_top_upd, ld_top_x, ld_b, ld_x;
    int ngroups, nrhs;
    int entries;                       // doubles of all of a CTA's Ms
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
    const int lmq = (h.x >> 4) & 15, flags = h.x >> 8, groups = h.y;
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
            assemble_item<K, GS>(V, p3);
            __syncwarp();
        }
        int c = h.z;
        for (int g = 0; g < groups; ++g) {
            const int j[4] = {c, c + h.w, c + 2 * h.w, c + 3 * h.w};
            four_steps<K, D>(S, V.m, j, acc);
            c += 4 * h.w;
        }
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
        const int type = h.x & 15;
        if (type == kProduct) {
            op_product<K, D, GS>(S, V, h, l1, l2, l3);
        } else if (type == kAssemble) {
            if (l1.x >= 0) assemble_item<K, GS>(V, l1);
            if (h.y > 1 && l2.x >= 0) assemble_item<K, GS>(V, l2);
            if (h.y > 2 && l3.x >= 0) assemble_item<K, GS>(V, l3);
        } else if (type == kFinish) {
            const bool top = (h.x >> 8) & kTopRoot;
            if (l1.x >= 0) finish_item<K, GS>(V, l1, h.z, h.w, top);
            if (h.y > 1 && l2.x >= 0) finish_item<K, GS>(V, l2, h.z, h.w, top);
            if (h.y > 2 && l3.x >= 0) finish_item<K, GS>(V, l3, h.z, h.w, top);
        } else if (type == kEnd) {
            return;
        }
        if ((h.x >> 8) & kBar) __syncthreads();
        else __syncwarp();
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
    V.top = P.top_upd + rhs * P.ld_top_upd;
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
        for (int i = threadIdx.x; i < G.next; i += NT) V.m[G.n + i] = tx[P.ext[G.ext + i]];
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
    // Products read past a front's columns (times zero): no NaN may be there.
    double* m = reinterpret_cast<double*>(smem + (size_t)(NT / 32) * depth_of(KM) * kBatchBytes);
    for (int i = threadIdx.x; i < P.entries; i += NT) m[i] = 0.0;
    __syncthreads();
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
    if (nt == 128) {  // trees of a few hundred unknowns at most: no slots
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

// ---------------------------------------------------------------------------
// Host side: the schedule of one class
// ---------------------------------------------------------------------------
struct Op {
    int type, flags;
    int front, r0, rows, c0, c1, po;  // product; po: first of its partial sums (-1: not split)
    int i0, i1;                       // assembly, finish: items
    int nsl, stride;                  // finish
    int batches() const;
};

struct ClassPlan {
    int n = 0, slots = 0, part_len = 0;  // unknowns; update slots and partial sums at a time
    int zero = 0, none = 0, part0 = 0;   // indices in M: the zero, the unused entry, the first partial sum
    std::vector<int> perm, ext;
    std::vector<int> fronts;             // the factor's fronts
    std::vector<int> c0;                 // index of each front's first unknown
    std::vector<std::vector<int>> idx;   // index of every row of each front
    std::vector<std::vector<int>> dst;   // destination of every row of each front, forward (kSlot + slot: a slot)
    // Children's entries of every row of each front: first slot (a row's are consecutive) and count.
    std::vector<std::vector<int>> slot, cnt;
    std::vector<char> root;              // whether the front's update vector belongs to the plan above
    std::vector<std::array<int, 4>> items;
    std::vector<std::vector<Op>> fwd, bwd;  // per warp
    double coef = 0;                     // coefficients of one direction
    int slot0 = 0;                       // index in M of slot 0 (negative: slots are in global memory)
    // Entries of M without slots, and the reach of products past their columns.
    int entries() const { return part0 + part_len; }
    static constexpr int kReach = 128;
};
// While M is not laid out, slots are numbered from kSlot on and kZero is the zero.
constexpr int kSlot = 0x20000000, kZero = 0x10000000;

int log2_lanes(int rows) {
    const int nq = (rows + 3) / 4;
    return nq <= 4 ? 2 : (nq <= 8 ? 3 : (nq <= 16 ? 4 : 5));
}
int groups_of(int rows, int cols) {
    const int ns = 32 >> log2_lanes(rows);
    return ((cols + ns - 1) / ns + 3) / 4;
}
// Index batches of a backward product after the header's two lines.
int index_batches(int groups) { return groups <= 4 ? 0 : (groups - 4 + 7) / 8; }
constexpr int kItems = 96;  // items of one assembly or finish

int Op::batches() const {
    if (type == kProduct) {
        const int g = groups_of(rows, c1 - c0);
        return 1 + g + ((flags & kTransposed) ? index_batches(g) : 0);
    }
    return 1;
}

// A level's fronts over the warps.  A front of at most 128 rows is one task
// unless its level has too few fronts to fill the CTA and its columns are
// many; other fronts are row chunks x column slices, so that a narrow level at
// the top of the tree keeps every warp busy.
struct Block {
    int front, rows, cols;
    bool kids;
};
void cut_level(const std::vector<Block>& blocks, bool fwd, ClassPlan& P, std::vector<std::vector<Op>>& out) {
    constexpr int kChunk = 128;
    const int nw = (int)out.size();
    // Ends a phase: the warps' last operations carry the barrier.
    std::vector<size_t> begun(nw);
    for (int w = 0; w < nw; ++w) begun[w] = out[w].size();
    auto barrier = [&]() {
        for (int w = 0; w < nw; ++w) {
            if (out[w].size() == begun[w]) {
                Op b{};
                b.type = kNothing;
                out[w].push_back(b);
            }
            out[w].back().flags |= kBar;
            begun[w] = out[w].size();
        }
    };
    auto col_range = [&](const Block& b, int r0, int rows, int& c0, int& c1) {
        // Forward: columns up to the chunk's last row; backward: from its first row.
        c0 = fwd ? 0 : r0;
        c1 = fwd ? std::min(b.cols, r0 + rows) : b.cols;
    };
    auto whole = [&](const Block& b) {
        if (b.rows > kChunk) return false;
        const int g = groups_of(b.rows, b.cols);
        return g <= 8 || ((int)blocks.size() >= 2 * nw && g <= 32);
    };
    // The children's entries of a front beyond two a row, in rounds of two:
    // items that add them to the first (update rows) or to the unknowns.
    // Round 0 of an unknown takes its first two.
    auto rounds = [&](const Block& b) {
        std::vector<std::vector<std::array<int, 4>>> r;
        const int nj = fwd ? b.cols : b.rows, fr = b.front;
        for (int p = 0; p < (int)P.cnt[fr].size(); ++p) {
            const int cnt = P.cnt[fr][p], first = p < nj ? 0 : 2;
            for (int e = first, q = 0; e < cnt; e += 2, ++q) {
                if ((int)r.size() <= q) r.resize(q + 1);
                const int s0 = kSlot + P.slot[fr][p] + e, s1 = e + 1 < cnt ? s0 + 1 : kZero;
                r[q].push_back({p < nj ? P.c0[fr] + p : kSlot + P.slot[fr][p], s0, s1, 0});
            }
        }
        return r;
    };
    auto assembly = [&](const std::vector<std::array<int, 4>>& items, size_t at, size_t n) {
        Op a{};
        a.type = kAssemble;
        a.i0 = (int)P.items.size();
        P.items.insert(P.items.end(), items.begin() + at, items.begin() + std::min(items.size(), at + n));
        a.i1 = (int)P.items.size();
        return a;
    };
    // Inputs of the fronts that several warps read.
    bool split_any = false, split_kids = false;
    long long units = 0;
    for (const Block& b : blocks) {
        if (whole(b)) continue;
        split_any = true;
        split_kids |= fwd && b.kids;
        for (int r0 = 0; r0 < b.rows; r0 += kChunk) {
            int c0, c1;
            col_range(b, r0, std::min(kChunk, b.rows - r0), c0, c1);
            units += groups_of(std::min(kChunk, b.rows - r0), c1 - c0);
        }
    }
    if (split_kids) {
        int w = 0;
        for (const Block& b : blocks) {
            if (whole(b) || !b.kids) continue;
            const auto r = rounds(b);
            if (r.size() == 1) {
                for (size_t i = 0; i < r[0].size(); i += 32) out[w++ % nw].push_back(assembly(r[0], i, 32));
            } else if (!r.empty()) {  // rounds follow one another: one warp
                for (const auto& q : r)
                    for (size_t i = 0; i < q.size(); i += kItems) out[w % nw].push_back(assembly(q, i, kItems));
                ++w;
            }
        }
        barrier();
    }
    // Tasks, the longest first, each to the warp with the least so far.
    struct Task {
        int cost;
        std::vector<Op> ops;
    };
    std::vector<Task> tasks;
    std::vector<Op> fins;
    const int gt = (int)std::min<long long>(8, std::max<long long>(2, (units + nw - 1) / nw));  // step groups per slice
    int po = 0;
    for (const Block& b : blocks) {
        const bool one = whole(b);
        for (int r0 = 0; r0 < b.rows; r0 += kChunk) {
            Op o{};
            o.type = kProduct;
            o.front = b.front;
            o.r0 = r0;
            o.rows = std::min(kChunk, b.rows - r0);
            o.flags = fwd ? 0 : kTransposed;
            o.po = -1;
            const int top = fwd && P.root[b.front] ? kTopRoot : 0;
            int c0, c1;
            col_range(b, r0, o.rows, c0, c1);
            if (one) {
                Task t;
                t.cost = 0;
                if (fwd && b.kids) {
                    const auto r = rounds(b);
                    o.flags |= kPairs;
                    for (size_t q = 0; q < r.size(); ++q) {
                        // A last round of at most 32 items is part of the product.
                        if (q + 1 == r.size() && r[q].size() <= 32) {
                            const Op a = assembly(r[q], 0, 32);
                            o.flags |= kItem;
                            o.i0 = a.i0;
                            o.i1 = a.i1;
                        } else {
                            for (size_t i = 0; i < r[q].size(); i += kItems) t.ops.push_back(assembly(r[q], i, kItems));
                        }
                    }
                }
                o.flags |= top;
                o.c0 = c0;
                o.c1 = c1;
                t.ops.push_back(o);
                for (const Op& q : t.ops) t.cost += q.batches();
                tasks.push_back(std::move(t));
                continue;
            }
            const int all = groups_of(o.rows, c1 - c0), nsl = std::max(1, (all + gt - 1) / gt);
            const int step = ((all + nsl - 1) / nsl) * 4 * (32 >> log2_lanes(o.rows));  // columns per slice
            const int pad = 4 * ((o.rows + 3) / 4);
            int n = 0;
            for (int c = c0; c < c1; c += step, ++n) {
                o.c0 = c;
                o.c1 = std::min(c1, c + step);
                o.po = P.part0 + po + n * pad;
                tasks.push_back({o.batches(), {o}});
            }
            for (int r = 0; r < o.rows; r += 32) {
                Op f{};
                f.type = kFinish;
                f.flags = top;
                f.nsl = n;
                f.stride = pad;
                f.i0 = (int)P.items.size();
                for (int q = r; q < std::min(o.rows, r + 32); ++q) {
                    const int row = r0 + q, fr = b.front;
                    const int cnt = !fwd || row < b.cols ? 0 : P.cnt[fr][row], s0 = cnt > 0 ? kSlot + P.slot[fr][row] : kZero;
                    P.items.push_back({P.part0 + po + q, fwd ? P.dst[fr][row] : P.c0[fr] + row, s0,
                                       cnt > 1 ? s0 + 1 : (int)kZero});
                }
                f.i1 = (int)P.items.size();
                fins.push_back(f);
            }
            po += n * pad;
        }
    }
    P.part_len = std::max(P.part_len, po);
    std::stable_sort(tasks.begin(), tasks.end(), [](const Task& a, const Task& b) { return a.cost > b.cost; });
    std::vector<int> load(nw, 0);
    for (const Task& t : tasks) {
        const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        load[w] += t.cost + 1;
        out[w].insert(out[w].end(), t.ops.begin(), t.ops.end());
    }
    barrier();
    if (split_any) {
        for (size_t i = 0; i < fins.size(); ++i) out[i % nw].push_back(fins[i]);
        barrier();
    }
}

// Schedule of the trees T.trees of factor T.F.  Unknowns are numbered tree by
// tree (a tree's fronts and unknowns are consecutive in the factor's
// post-order); rows outside a tree are its root's update rows, numbered after
// all of them.
void plan_class(const ResidentPlan::Shape& T, int nwarps, ClassPlan& P) {
    const SnFactor& F = *T.F;
    Op end{};
    end.type = kEnd;
    P.fwd.resize(nwarps);
    P.bwd.resize(nwarps);
    std::vector<int> tree_of, tree_base, ext_base, first;
    for (size_t t = 0; t < T.trees.size(); ++t) {
        const int a = T.trees[t].first, b = T.trees[t].last;
        tree_base.push_back(P.n);
        first.push_back((int)P.fronts.size());
        for (int j = a; j <= b; ++j) {
            P.fronts.push_back(j);
            tree_of.push_back((int)t);
            P.n += F.ncol[j];
        }
        const int lo = F.col0[a], hi = F.col0[b] + F.ncol[b];
        for (int i = lo; i < hi; ++i) P.perm.push_back(F.perm[i]);
    }
    for (const auto& t : T.trees) {
        ext_base.push_back(P.n + (int)P.ext.size());
        for (int r : F.rows[t.last]) P.ext.push_back(T.ext_off + r);
    }
    const int ns = (int)P.fronts.size();
    P.zero = P.n + (int)P.ext.size();
    P.none = P.zero + 1;
    P.part0 = P.none + 1;
    if (P.none >= 65536) throw Error(HDD_ERR_INTERNAL, "a resident tree has too many unknowns");
    // Index in the class's vector of row r of a front of tree t.
    auto index_of = [&](int t, int r) {
        const int lo = F.col0[T.trees[t].first], hi = F.col0[T.trees[t].last] + F.ncol[T.trees[t].last];
        if (r >= lo && r < hi) return tree_base[t] + r - lo;
        const std::vector<int>& rr = F.rows[T.trees[t].last];
        const auto it = std::lower_bound(rr.begin(), rr.end(), r);
        if (it == rr.end() || *it != r) throw Error(HDD_ERR_INTERNAL, "a front's row is not among its tree root's");
        return ext_base[t] + (int)(it - rr.begin());
    };
    std::vector<int> parent(ns, -1), height(ns, 0), depth(ns, 0);
    std::vector<std::vector<int>> kids(ns);
    for (int i = 0; i < ns; ++i) {
        const int j = P.fronts[i], t = tree_of[i];
        if (j != T.trees[t].last) parent[i] = first[t] + F.parent[j] - T.trees[t].first;
    }
    for (int i = 0; i < ns; ++i)
        if (parent[i] >= 0) {
            kids[parent[i]].push_back(i);
            height[parent[i]] = std::max(height[parent[i]], height[i] + 1);
        }
    for (int i = ns - 1; i >= 0; --i)
        if (parent[i] >= 0) depth[i] = depth[parent[i]] + 1;
    P.root.assign(ns, 0);
    P.c0.resize(ns);
    P.idx.resize(ns);
    P.dst.resize(ns);
    P.slot.resize(ns);
    P.cnt.resize(ns);
    for (int i = 0; i < ns; ++i) {
        const int j = P.fronts[i], nj = F.ncol[j], nr = (int)F.rows[j].size();
        P.c0[i] = index_of(tree_of[i], F.col0[j]);
        for (int c = 0; c < nj; ++c) P.idx[i].push_back(P.c0[i] + c);
        for (int r : F.rows[j]) P.idx[i].push_back(index_of(tree_of[i], r));
        P.dst[i].assign(nj + nr, P.none);
        for (int c = 0; c < nj; ++c) P.dst[i][c] = P.c0[i] + c;
        P.slot[i].assign(nj + nr, 0);
        P.cnt[i].assign(nj + nr, 0);
        P.coef += 0.5 * nj * (nj + 1.0) + (double)nr * nj;
    }
    const int nh = ns ? *std::max_element(height.begin(), height.end()) + 1 : 0;
    const int nd = ns ? *std::max_element(depth.begin(), depth.end()) + 1 : 0;
    std::vector<std::vector<int>> at_h(nh), at_d(nd);
    for (int i = 0; i < ns; ++i) {
        at_h[height[i]].push_back(i);
        at_d[depth[i]].push_back(i);
    }
    // Update slots: a front's inputs from its children, position by position,
    // child by child, in one interval that is taken at its first child's level
    // and free again after its own.
    std::vector<std::pair<int, int>> room;  // free intervals, by start
    std::vector<int> base(ns, -1), len(ns, 0);
    auto take = [&](int size) {
        for (size_t q = 0; q < room.size(); ++q)
            if (room[q].second - room[q].first >= size) {
                const int at = room[q].first;
                room[q].first += size;
                if (room[q].first == room[q].second) room.erase(room.begin() + q);
                return at;
            }
        int at = P.slots;
        if (!room.empty() && room.back().second == P.slots) {  // grow the last free interval
            at = room.back().first;
            room.pop_back();
        }
        P.slots = at + size;
        return at;
    };
    auto give = [&](int at, int size) {
        auto it = std::lower_bound(room.begin(), room.end(), std::make_pair(at, at));
        it = room.insert(it, {at, at + size});
        const size_t q = it - room.begin();
        if (q + 1 < room.size() && room[q].second == room[q + 1].first) {
            room[q].second = room[q + 1].second;
            room.erase(room.begin() + q + 1);
        }
        if (q > 0 && room[q - 1].second == room[q].first) {
            room[q - 1].second = room[q].second;
            room.erase(room.begin() + q);
        }
    };
    for (int h = 0; h < nh; ++h) {
        for (int i : at_h[h]) {
            const int p = parent[i];
            if (p < 0 || base[p] >= 0) continue;
            // Positions of the children's entries in the parent.
            const int jp = P.fronts[p], nj = F.ncol[jp], pc0 = F.col0[jp];
            std::vector<std::vector<int>> pos(kids[p].size());
            for (size_t c = 0; c < kids[p].size(); ++c)
                for (int r : F.rows[P.fronts[kids[p][c]]]) {
                    int q;
                    if (r >= pc0 && r < pc0 + nj) q = r - pc0;
                    else {
                        const auto it = std::lower_bound(F.rows[jp].begin(), F.rows[jp].end(), r);
                        if (it == F.rows[jp].end() || *it != r) throw Error(HDD_ERR_INTERNAL, "supernode row not in parent front");
                        q = nj + (int)(it - F.rows[jp].begin());
                    }
                    pos[c].push_back(q);
                    ++P.cnt[p][q];
                    ++len[p];
                }
            base[p] = len[p] > 0 ? take(len[p]) : 0;
            int at = base[p];
            for (size_t q = 0; q < P.slot[p].size(); ++q) {
                P.slot[p][q] = at;
                at += P.cnt[p][q];
            }
            std::vector<int> next = P.slot[p];
            for (size_t c = 0; c < kids[p].size(); ++c) {
                const int k = kids[p][c], njk = F.ncol[P.fronts[k]];
                for (size_t q = 0; q < pos[c].size(); ++q) P.dst[k][njk + q] = kSlot + next[pos[c][q]]++;
            }
        }
        for (int i : at_h[h])
            if (len[i] > 0) give(base[i], len[i]);
    }
    for (size_t t = 0; t < T.trees.size(); ++t) {
        const int i = first[t] + T.trees[t].last - T.trees[t].first, nj = F.ncol[T.trees[t].last];
        for (size_t q = 0; q < F.rows[T.trees[t].last].size(); ++q) P.dst[i][nj + q] = -1 - (T.trees[t].top + (int)q);
        P.root[i] = !F.rows[T.trees[t].last].empty();
    }
    for (int h = 0; h < nh; ++h) {
        std::vector<Block> bl;
        for (int i : at_h[h])
            bl.push_back({i, (int)P.idx[i].size(), F.ncol[P.fronts[i]], !kids[i].empty()});
        cut_level(bl, true, P, P.fwd);
    }
    for (int d = 0; d < nd; ++d) {
        std::vector<Block> bl;
        for (int i : at_d[d]) bl.push_back({i, F.ncol[P.fronts[i]], (int)P.idx[i].size(), false});
        cut_level(bl, false, P, P.bwd);
    }
    for (int w = 0; w < nwarps; ++w) {
        P.fwd[w].push_back(end);
        P.bwd[w].push_back(end);
    }
}

// Writes the batches of an operation.
uint32_t* emit(const Op& o, const SnFactor& F, const ClassPlan& P, uint32_t* out) {
    constexpr int L = kLine / 4;  // ints per line
    std::memset(out, 0, kBatchBytes);
    int* h = reinterpret_cast<int*>(out);
    const bool gs = P.slot0 < 0;
    // Destinations: slots are in M, or -1 - slot in global memory.
    auto place = [&](int d) { return d < kZero ? d : (gs ? -1 - (1 + d - kSlot) : P.slot0 + d - kSlot); };
    // Entries of pairs: in M, or slots of global memory after its zero.
    auto entry = [&](int d) { return d == kZero ? (gs ? 0 : P.zero) : (gs ? 1 : P.slot0) + d - kSlot; };
    auto header = [&](int lmq, int count, auto index, int distance) {
        for (int l = 0; l < 32; ++l) {
            h[4 * l] = o.type | lmq << 4 | o.flags << 8;
            h[4 * l + 1] = count;
            h[4 * l + 2] = index(l);
            h[4 * l + 3] = distance;
        }
    };
    auto assemble_entry = [&](int* p, const std::array<int, 4>& t) {
        const bool slot = t[0] >= kSlot;
        p[0] = slot ? entry(t[0]) : t[0];
        p[1] = entry(t[1]);
        p[2] = entry(t[2]);
        p[3] = slot && gs ? 1 : 0;
    };
    if (o.type != kProduct) {
        const int n = o.i1 - o.i0;
        header(0, (n + 31) / 32, [&](int) { return o.nsl; }, o.stride);
        int* p = h + L;
        for (int i = 0; i < kItems; ++i, p += 4) {
            if (i >= n) {
                p[0] = -1;
                continue;
            }
            const std::array<int, 4>& t = P.items[o.i0 + i];
            if (o.type == kAssemble) {
                assemble_entry(p, t);
            } else {
                p[0] = t[0];
                p[1] = place(t[1]);
                p[2] = entry(t[2]);
                p[3] = entry(t[3]);
            }
        }
        return out + kBatch * L;
    }
    const bool tr = (o.flags & kTransposed) != 0;
    const int i = o.front, m = (int)P.idx[i].size();
    const int lmq = log2_lanes(o.rows), mq = 1 << lmq, ns = 32 >> lmq;
    const int groups = groups_of(o.rows, o.c1 - o.c0);
    header(lmq, groups, [&](int l) { return tr ? 0 : P.c0[i] + o.c0 + (l >> lmq); }, ns);
    auto rows_line = [&](int line, auto value) {  // one int per row, four a lane (the first slice's lanes)
        int* p = h + line * L;
        for (int l = 0; l < 32; ++l)
            for (int e = 0; e < 4; ++e) {
                const int q = 4 * (l & (mq - 1)) + e;
                p[4 * l + e] = value(l < mq && q < o.rows ? q : -1);
            }
    };
    rows_line(1, [&](int q) {
        if (q < 0) return P.none;
        if (o.po >= 0) return o.po + q;
        return tr ? P.c0[i] + o.r0 + q : place(P.dst[i][o.r0 + q]);
    });
    if (o.flags & kPairs) {
        const int nj = F.ncol[P.fronts[i]];  // a front's unknowns are assembled before
        rows_line(2, [&](int q) {
            const int cnt = q < 0 || o.r0 + q < nj ? 0 : P.cnt[i][o.r0 + q];
            const int s0 = cnt > 0 ? kSlot + P.slot[i][o.r0 + q] : (int)kZero;
            return entry(s0) | entry(cnt > 1 ? s0 + 1 : (int)kZero) << 16;
        });
    }
    if (o.flags & kItem) {
        int* p = h + 3 * L;
        for (int l = 0; l < 32; ++l, p += 4) {
            if (o.i0 + l < o.i1) assemble_entry(p, P.items[o.i0 + l]);
            else {  // adds zero to the unused entry
                p[0] = P.none;
                p[1] = p[2] = entry(kZero);
                p[3] = 0;
            }
        }
    }
    // Eight steps' column indices, 16 bits each.
    auto index_line = [&](uint32_t* line, int step0) {
        uint16_t* p = reinterpret_cast<uint16_t*>(line);
        for (int l = 0; l < 32; ++l)
            for (int u = 0; u < 8; ++u)
                p[8 * l + u] = (uint16_t)P.idx[i][std::min(o.c1 - 1, o.c0 + (l >> lmq) + (step0 + u) * ns)];
    };
    if (tr) {
        index_line(out + 2 * L, 0);
        index_line(out + 3 * L, 8);
    }
    out += kBatch * L;
    const double* W = F.Fw[P.fronts[i]].data();  // column-major, m rows
    for (int g = 0; g < groups; ++g) {
        if (tr && g >= 4 && (g - 4) % 8 == 0) {
            for (int q = 0; q < 4; ++q) index_line(out + q * L, 4 * g + 8 * q);
            out += kBatch * L;
        }
        for (int u = 0; u < 4; ++u) {
            float* p = reinterpret_cast<float*>(out);
            for (int l = 0; l < 32; ++l) {
                const int c = o.c0 + (l >> lmq) + (4 * g + u) * ns, r = o.r0 + 4 * (l & (mq - 1));
                for (int e = 0; e < 4; ++e) {
                    const bool in = c < o.c1 && r + e < o.r0 + o.rows;
                    p[4 * l + e] = !in ? 0.0f : (float)(tr ? W[(size_t)(r + e) * m + c] : W[(size_t)c * m + r + e]);
                }
            }
            out += L;
        }
    }
    return out;
}

}  // namespace

size_t ResidentPlan::smem_bytes(int entries, int k, int nt) {
    return (size_t)std::max(entries, 1) * k * sizeof(double) + (size_t)(nt / 32) * depth_of(k) * kBatchBytes;
}

bool ResidentPlan::build(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets, cudaStream_t s) {
    release();
    // Classes: members given the same factor.
    std::map<const SnFactor*, int> shape_of;
    std::vector<Shape> shapes;
    std::vector<std::vector<int>> members;
    for (size_t f = 0; f < factors.size(); ++f) {
        const SnFactor* F = factors[f];
        n = std::max(n, offsets[f] + F->n);
        auto it = shape_of.find(F);
        if (it == shape_of.end()) {
            it = shape_of.emplace(F, (int)shapes.size()).first;
            Shape T;
            T.F = F;
            int a = 0;
            for (int j = 0; j < (int)F->col0.size(); ++j)
                if (F->parent[j] < 0) {
                    T.trees.push_back({a, j, -1});
                    a = j + 1;
                }
            shapes.push_back(std::move(T));
            members.emplace_back();
        }
        members[it->second].push_back(offsets[f]);
    }
    cut = false;
    return build_shapes(shapes, members, s);
}

bool ResidentPlan::build_cut(const std::vector<Shape>& shapes, const std::vector<int>& offsets, cudaStream_t s) {
    release();
    std::vector<std::vector<int>> members;
    for (int o : offsets) members.push_back({o});
    cut = true;
    return build_shapes(shapes, members, s);
}

bool ResidentPlan::build_shapes(const std::vector<Shape>& shapes, const std::vector<std::vector<int>>& members,
                                cudaStream_t s) {
    double biggest = 0;
    for (const Shape& T : shapes) {
        if (T.F->Fw.size() != T.F->col0.size()) throw Error(HDD_ERR_INTERNAL, "solve blocks not built");
        double c = 0;
        int len = 0;
        for (const auto& t : T.trees) {
            for (int j = t.first; j <= t.last; ++j) {
                c += 0.5 * T.F->ncol[j] * (T.F->ncol[j] + 1.0) + (double)T.F->rows[j].size() * T.F->ncol[j];
                len += T.F->ncol[j];
            }
            len += (int)T.F->rows[t.last].size();
        }
        biggest = std::max(biggest, c);
        max_n = std::max(max_n, len);
    }
    int dev_id = 0, nsm = 0;
    dev::ck(cudaGetDevice(&dev_id), "cudaGetDevice");
    dev::ck(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev_id), "SM count");
    // Sixteen warps, or four where a tree is a few lines a warp; cut trees that
    // are more than the SMs run two CTAs to an SM.
    if (cut) nt = shapes.size() > (size_t)nsm ? 256 : 512;
    else nt = biggest <= 8192 ? 128 : 512;
    auto groups_for = [&](int k) {
        size_t g = 0;
        for (const auto& m : members) g += (m.size() + k - 1) / k;
        return g;
    };
    std::vector<ClassPlan> cp(shapes.size());
    std::vector<std::string> err(shapes.size());
#pragma omp parallel for schedule(dynamic)
    for (size_t c = 0; c < shapes.size(); ++c) {
        try {
            plan_class(shapes[c], nt / 32, cp[c]);
        } catch (const std::exception& e) { err[c] = e.what(); }
    }
    for (const auto& e : err)
        if (!e.empty()) throw Error(HDD_ERR_INTERNAL, e);

    // Concatenate the classes.
    std::vector<RWarp> warps;
    std::vector<int> off, perm, ext;
    auto fits32 = [](long long v) {
        if (v > (long long)INT32_MAX) throw Error(HDD_ERR_UNSUPPORTED, "solve plan too large for 32-bit indices");
        return (int)v;
    };
    // M's entries with and without the update slots; trees per CTA.
    int bare = 0, all = 0;
    for (const ClassPlan& P : cp) {
        bare = std::max(bare, P.entries() + ClassPlan::kReach);
        all = std::max(all, P.entries() + std::max(P.slots, (int)ClassPlan::kReach));
    }
    km = 1;
    while (!cut && km < 4 && groups_for(km) > (size_t)nsm && smem_bytes(bare, 2 * km, nt) <= kMaxSmem) km *= 2;
    global_slots = !cut && (smem_bytes(all, km, nt) > kMaxSmem || all >= 65536);
    entries = (global_slots ? bare : all) * km;
    smem = smem_bytes(global_slots ? bare : all, km, nt);
    bool fits = smem <= kMaxSmem;
    for (ClassPlan& P : cp) {
        P.slot0 = global_slots ? -1 : P.entries();
        fits &= P.slots + 1 < 65536;
    }
    if (!fits) {  // partial sums or update entries of unusual trees
        release();
        return false;
    }
    struct Item { int c, w; long long at; };  // a warp's stream; its first float
    std::vector<Item> streams;
    std::vector<RGroup> classes(shapes.size());  // the fields of its groups
    long long total = 0;
    for (size_t c = 0; c < shapes.size(); ++c) {
        const ClassPlan& P = cp[c];
        RGroup& C = classes[c];
        C.n = P.n;
        C.perm = fits32(perm.size());
        C.next = (int)P.ext.size();
        C.ext = fits32(ext.size());
        C.warps = fits32(warps.size());
        C.stream = 4 * total;
        perm.insert(perm.end(), P.perm.begin(), P.perm.end());
        ext.insert(ext.end(), P.ext.begin(), P.ext.end());
        long long first = 0;
        for (int w = 0; w < nt / 32; ++w) {
            long long nf = 0, nb = 0;
            for (const Op& o : P.fwd[w]) nf += kBatch * o.batches();
            for (const Op& o : P.bwd[w]) nb += kBatch * o.batches();
            warps.push_back({fits32(first), fits32(nf), fits32(nb), 0});
            streams.push_back({(int)c, w, total});
            first += nf + nb;
            total += (nf + nb) * (kLine / 4);
        }
    }
    // Groups, the longest first (their order does not affect results).
    std::vector<RGroup> groups;
    std::vector<int> order(shapes.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cp[a].coef > cp[b].coef; });
    for (int pass = 0; pass < 2; ++pass)
        for (int c : order)
            for (size_t m = 0; m < members[c].size(); m += km) {
                const int cnt = (int)std::min<size_t>(km, members[c].size() - m);
                if ((cnt > 1) != (pass == 0)) continue;  // full groups take longer than single trees
                RGroup G = classes[c];
                G.member0 = fits32(off.size());
                G.count = cnt;
                G.upd = upd_len;
                G.y = y_len;
                if (cut) y_len += cp[c].n;
                const int kk = cnt > 1 ? km : 1;
                if (global_slots) upd_len += (long long)kk * ((cp[c].slots + 2) & ~1);
                for (int i = 0; i < cnt; ++i) off.push_back(members[c][m + i]);
                groups.push_back(G);
            }
    ngroups = (int)groups.size();
    upd_len = std::max<long long>(upd_len, 2);
    bytes = 0;
    float* d = nullptr;
    // Prefetches run past a stream's end: the last one's into padding.
    const size_t ns = streams.size();
    const long long pad = (long long)depth_of(1) * kBatchBytes / 4;
    streams.push_back({-1, 0, total});
    dev::upload_packed(streams.size(), total + pad, [&](size_t i) { return streams[i].at; },
                       [&](size_t i, float* dst) {
                           if (i == ns) {
                               std::memset(dst, 0, (size_t)pad * 4);
                               return;
                           }
                           const ClassPlan& P = cp[streams[i].c];
                           const SnFactor& F = *shapes[streams[i].c].F;
                           uint32_t* out = reinterpret_cast<uint32_t*>(dst);
                           for (const Op& o : P.fwd[streams[i].w]) out = emit(o, F, P, out);
                           for (const Op& o : P.bwd[streams[i].w]) out = emit(o, F, P, out);
                       },
                       s, d, bytes);
    d_stream = reinterpret_cast<char*>(d);
    auto nonempty = [](std::vector<int>& v) -> const std::vector<int>& {
        if (v.empty()) v.push_back(0);
        return v;
    };
    d_groups = dev::upload(groups, s, bytes);
    d_warps = dev::upload(warps, s, bytes);
    d_off = dev::upload(nonempty(off), s, bytes);
    d_perm = dev::upload(nonempty(perm), s, bytes);
    d_ext = dev::upload(nonempty(ext), s, bytes);
    d_gate = dev::alloc_zero<int>(1, bytes, s);
    // Algorithmic bytes of one solve: each class's coefficients once per
    // direction, b read and x written.
    double unique = 0;
    for (const auto& P : cp) unique += P.coef;
    solve_bytes = 2 * 4.0 * unique + 8.0 * n;
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
                  upd_len, y_len, top.ld_upd, top.ld_x, ld_b, ld_x, ngroups, nrhs, entries, top.ctr, top.n_ctr, d_gate, err,
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
