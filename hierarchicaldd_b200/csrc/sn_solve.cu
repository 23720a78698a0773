// Supernodal triangular solves on the GPU (the device half of the PARDISO
// stand-in; the reference's phase-33 solves are in
// CPU/Interface_Solver/SIGMA_SMOOTHER.cpp:293-324).
//
// Every front J of the nested-dissection forest carries
// Fw = [L_JJ^{-1}; -L_RJ L_JJ^{-1}] (m = nj + nr rows, nj columns), stored once,
// column-major with leading dimension round4(m), so
//   forward   [y_J; v_J] = Fw f_J + [0; f_R]   (f assembled from b and the children's v)
//   backward  x_J        = Fw^T [y_J; x_R]
// are dense products over the same coefficients.  The coefficients are FP32
// (what the HBM stream carries); products are accumulated in FP64 (every
// FP32 x FP32 product is exact in FP64) and the vectors passed between fronts
// (the assembled f, y, x and the update vectors) are FP64, so a solve rounds
// to FP32 once, at its output, like the FP64 substitution it replaces up to
// the rounding of the stored coefficients.
//
// A plan whose trees each fit one CTA is solved by sn_resident.cu alone.
// Otherwise the lower trees of every factor (most of the fronts, little of
// the work each) go there, forward before and backward after the launch of
// this file, which has the fronts above them.
//
// That launch is persistent and does both directions.  Its work is a list of
// tasks in topological order (forward: children before parents; then
// backward: parents before children); CTAs take them by ticket and, before
// starting one, wait on per-front completion counters of the fronts it depends
// on.  A task only ever waits on tasks with smaller tickets.  A CTA takes its
// next ticket while it works on the current one; the smallest unfinished
// ticket is then still the current one of a running CTA, so the walk always
// progresses.  Every wait is bounded anyway and raises the plan's error word
// when it gives up.  Data produced by other CTAs in the same launch is read
// with L2-coherent loads after an acquire of the counter.
//
// Forward tasks are row blocks of up to kRB rows times up to kCC columns (taller
// triangles: several column blocks, whose partial sums the last one to finish
// adds in column order); backward tasks are column blocks, one warp per column
// group, lanes striding down the contiguous columns, tall ones cut into row
// chunks the same way.  So every result is independent of scheduling.
//
// What bounds it: near the top of a tree a few fronts a level follow one
// another, so the time from one front's end to the next one's.  Everything a
// task needs that does not depend on the fronts below (its record, its
// coefficients, the gather indices of its inputs) is loaded before it waits;
// after the wait come one load of the inputs, the products, one reduction and
// the release of its counter.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <exception>
#include <map>
#include <numeric>
#include <string>
#include <vector>

#include "dev_util.h"
#include "sn_streams.h"

namespace hdd {
namespace {

constexpr int kNT = 256;      // threads per CTA
constexpr int kPerSM = 2;     // CTAs per SM the register budget is sized for
constexpr int kRB = 128;      // rows per forward task
constexpr int kCC = 128;      // columns per forward task of a split block
constexpr int kWhole = 256;   // ... and the most columns of an unsplit one
constexpr int kBLoads = 16;   // coefficient quads a lane loads in a backward task
// Backward tasks: 8 warps x kCW columns by kBLoads / kCW row quads per lane:
// 32 columns x 512 rows, or 16 x 1024 for taller fronts, so that a front of up
// to 1024 rows needs no partial sums.
constexpr int kWarps = kNT / 32;
constexpr int kTallRows = 512;
__host__ __device__ constexpr int cols_of(int cw) { return kWarps * cw; }
__host__ __device__ constexpr int rows_of(int cw) { return kBLoads / cw * 128; }
struct PlanView {
    int nsn, n_fwd, ntasks;
    const int* rows;
    const int* child;
    // Gather lists: position p of front J's input vector receives the update
    // entries gent[ge_off[J] + gptr[gp_off[J] + p] .. gptr[gp_off[J] + p + 1])
    // (indices into upd), in child order.
    const int *gptr, *gent;
    const int *ntf, *ntb;
    const int* perm;
    const float* fw;
    const SnTask* tasks;
    const float* b_old;
    float* x_old;
    double* part;
    double* upd;
    double* ynew;
    double* xnew;
    int* ctr;
    int* err;
    long long spin_limit;  // polls before a wait gives up
    // Right-hand side j uses part + j ld_part, upd + j ld_upd, ynew / xnew + j
    // ld_n, ctr + j ld_ctr (the ticket is shared), b_old + j ld_b, x_old + j ld_x.
    long long ld_part, ld_upd, ld_n, ld_ctr, ld_b, ld_x;
    int nrhs;
};

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add_release(int* p) {
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" : : "l"(p) : "memory");
}
__device__ __forceinline__ int add_acq_rel(int* p) {
    int v;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Waits until *p >= target; false when the wait gave up, or soon when an
// earlier wait of this launch already gave up (so one failure cannot turn
// into a long chain of timeouts).
__device__ __noinline__ bool wait_at_least(const int* p, int target, const int* err, long long limit) {
    for (long long i = 0; i < limit; ++i) {
        if (ld_acquire(p) >= target) return true;
        if (i % 16 == 15 && ld_acquire(err) != 0) return false;
    }
    return false;
}

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// Keeps v as FP32 up to here: converted to FP64 before a wait, the preloaded
// coefficients would take twice the registers.
__device__ __forceinline__ void hold(float4& v) {
    asm volatile("" : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w));
}

// Four FP64 fused multiply-adds acc[e] += v.e * x.
__device__ __forceinline__ void fma4(double (&acc)[4], const float4 v, double x) {
    acc[0] = fma((double)v.x, x, acc[0]);
    acc[1] = fma((double)v.y, x, acc[1]);
    acc[2] = fma((double)v.z, x, acc[2]);
    acc[3] = fma((double)v.w, x, acc[3]);
}

// Fw is stored column-major with a leading dimension of round4(m) and
// columns starting on 16-byte boundaries, so four consecutive rows of a column
// are one 16-byte load.  Entries above the diagonal of L_JJ^{-1} and the
// padding rows m .. round4(m) are stored zeros: a load may cover them.

// The vectors of one right-hand side.
struct Vectors {
    double *part, *upd, *y, *x;
    int *done_f, *done_b, *chunk;
    const float* b;
    float* x_old;
};

struct Shared {
    SnTask task[2];
    Vectors vec[2];       // of the task's right-hand side (here to save registers)
    int next[2];          // tickets of task[]
    int last;
    alignas(16) double f[kWhole];  // forward: the task's inputs
    double fr[kRB];                // ... and its update rows' sums of the children's entries
    double red[4 * kNT];           // column-slice partial sums; backward: the input rows
};
static_assert(4 * kNT >= rows_of(2), "backward inputs fit");

template <class Fetch>
__device__ __forceinline__ void forward_task(const PlanView& P, const SnTask& T, Shared& S, const Vectors& V,
                                             Fetch fetch_next) {
    const int tid = threadIdx.x, nj = T.nj;
    // Row quads x column slices: mq lanes on the block's row quads (one
    // 16-byte load per column), ks slices of consecutive columns.
    const int nq = (T.rows + 3) >> 2;
    const int mq = nq <= 8 ? 8 : (nq <= 16 ? 16 : 32);
    const int ks = kNT / mq;
    const int sl = tid / mq, lq = tid - sl * mq;
    const int row = T.r0 + 4 * lq;
    const size_t ld = (size_t)((T.m + 3) & ~3);
    const float* A = P.fw + T.fw + row;
    int cbeg = 0, cend = 0;
    if (lq < nq) {
        const int cs = (T.ncols + ks - 1) / ks;
        cbeg = T.c0 + sl * cs;
        cend = min(T.c0 + T.ncols, cbeg + cs);
        if (row < nj) cend = min(cend, row + 4);  // L_JJ^{-1} is lower triangular
    }
    constexpr int U = 16;
    float4 v[U];
    const float* col = A + (size_t)cbeg * ld;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        v[u] = (cbeg + u < cend) ? ldg4(col) : make_float4(0.f, 0.f, 0.f, 0.f);
        col += ld;
    }
    // The positions this task reads, its columns and its update rows from
    // max(r0, nj) on: b's entry and the gather indices now, the children's
    // update entries after the wait.
    const int rlo = max(T.r0, nj), rend = T.r0 + T.rows;
    const int nneed = T.ncols + max(0, rend - rlo);
    constexpr int Q = (kWhole + kRB + kNT - 1) / kNT;
    double base[Q];
    int e0[Q], e1[Q], first[Q], second[Q];
    const bool kids = T.kids != 0;
#pragma unroll
    for (int h = 0; h < Q; ++h) {
        const int q = tid + h * kNT;
        base[h] = 0.0;
        e0[h] = e1[h] = first[h] = second[h] = 0;
        if (q < nneed) {
            const int p = q < T.ncols ? T.c0 + q : rlo + (q - T.ncols);
            if (q < T.ncols) base[h] = (double)V.b[P.perm[T.col0 + p]];
            if (kids) {
                e0[h] = P.gptr[T.gp + p];
                e1[h] = P.gptr[T.gp + p + 1];
                if (e1[h] > e0[h]) first[h] = P.gent[T.ge + e0[h]];
                if (e1[h] > e0[h] + 1) second[h] = P.gent[T.ge + e0[h] + 1];
            }
        }
    }
    if (kids && tid < 32) {
        bool ok = true;
        for (int c = T.child_b + tid; c < T.child_e; c += 32) {
            const int C = P.child[c];
            ok &= wait_at_least(V.done_f + C, P.ntf[C], P.err, P.spin_limit);
        }
        if (!ok) atomicExch(P.err, 1);
    }
    fetch_next();
    __syncthreads();
    double u0[Q], u1[Q];
#pragma unroll
    for (int h = 0; h < Q; ++h) {
        u0[h] = e1[h] > e0[h] ? __ldcg(V.upd + first[h]) : 0.0;
        u1[h] = e1[h] > e0[h] + 1 ? __ldcg(V.upd + second[h]) : 0.0;
    }
#pragma unroll
    for (int h = 0; h < Q; ++h) {
        const int q = tid + h * kNT;
        if (q >= nneed) continue;
        double s = base[h] + u0[h] + u1[h];
        for (int e = e0[h] + 2; e < e1[h]; ++e) s += __ldcg(V.upd + P.gent[T.ge + e]);
        if (q < T.ncols) S.f[q] = s;
        else S.fr[rlo + (q - T.ncols) - T.r0] = s;
    }
    __syncthreads();
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const double* f = S.f - T.c0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        hold(v[u]);
        if (cbeg + u < cend) fma4(acc, v[u], f[cbeg + u]);
    }
    for (int c = cbeg + U; c < cend; c += 8) {
        float4 w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            w[u] = (c + u < cend) ? ldg4(col) : make_float4(0.f, 0.f, 0.f, 0.f);
            col += ld;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c + u < cend) fma4(acc, w[u], f[c + u]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) S.red[e * kNT + tid] = acc[e];
    __syncthreads();
    // Thread t < rows adds row r0 + t's slices in order.
    const int r = T.r0 + tid;
    double s = 0.0;
    if (tid < T.rows) {
        const double* p = S.red + (tid & 3) * kNT + (tid >> 2);
        s = p[0];
#pragma unroll 8
        for (int q = 1; q < ks; ++q) s += p[q * mq];
    }
    if (T.nk > 1) {
        if (tid < T.rows) V.part[T.part + (size_t)T.k * kRB + tid] = s;
        __syncthreads();
        if (tid == 0) S.last = add_acq_rel(V.chunk + T.chunk) == T.nk - 1;
        __syncthreads();
        if (S.last && tid < T.rows) {
            s = 0.0;
            for (int k = 0; k < T.nk; ++k) s += __ldcg(V.part + T.part + (size_t)k * kRB + tid);
        }
    }
    if (tid < T.rows && (T.nk == 1 || S.last)) {
        if (r < nj) V.y[T.col0 + r] = s;
        else V.upd[T.upd + (r - nj)] = S.fr[tid] + s;
    }
    __syncthreads();
    if (tid == 0) add_release(V.done_f + T.front);
}

// CW columns per warp.
template <int CW, class Fetch>
__device__ __forceinline__ void backward_task(const PlanView& P, const SnTask& T, Shared& S, const Vectors& V,
                                              Fetch fetch_next) {
    constexpr int NI = kBLoads / CW, Q = rows_of(CW) / kNT;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, nj = T.nj;
    // Columns [r0, r0 + rows) of the front; this task's rows [rlo, rhi): all
    // from r0 on (the first any of its columns needs, a multiple of 4), or one
    // chunk of them.
    const int a0 = T.r0, na = T.rows, rlo = T.c0, rhi = T.c0 + T.ncols;
    const size_t ld = (size_t)((T.m + 3) & ~3);
    const float* A = P.fw + T.fw;
    double* g = S.red;  // input rows, entry i - rlo
    float4 v[NI][CW];
    const float* col = A + (size_t)(a0 + w) * ld + rlo + 4 * lane;
#pragma unroll
    for (int j = 0; j < CW; ++j) {
        const bool on = w + kWarps * j < na;
#pragma unroll
        for (int i = 0; i < NI; ++i)
            v[i][j] = (on && rlo + 4 * lane + 128 * i < rhi) ? ldg4(col + 128 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
        col += kWarps * ld;
    }
    int src[Q];
#pragma unroll
    for (int h = 0; h < Q; ++h) {
        const int i = rlo + tid + h * kNT;
        src[h] = (i >= nj && i < rhi) ? P.rows[T.rows_off + (i - nj)] : 0;
    }
    if (tid == 0) {
        // The parent's solution, or (at a root) this front's forward result.
        const bool root = T.parent < 0;
        const int* d = root ? V.done_f + T.front : V.done_b + T.parent;
        const int target = root ? P.ntf[T.front] : P.ntb[T.parent];
        if (!wait_at_least(d, target, P.err, P.spin_limit)) atomicExch(P.err, 1);
    }
    fetch_next();
    __syncthreads();
#pragma unroll
    for (int h = 0; h < Q; ++h) {
        const int i = rlo + tid + h * kNT;
        if (i < nj && i < rhi) g[i - rlo] = __ldcg(V.y + T.col0 + i);
        else if (i < rhi) g[i - rlo] = __ldcg(V.x + src[h]);
        else if (i < rlo + rows_of(CW)) g[i - rlo] = 0.0;  // padding rows
    }
    __syncthreads();
    double s[CW];
#pragma unroll
    for (int j = 0; j < CW; ++j) s[j] = 0.0;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int q = 4 * lane + 128 * i;
        if (rlo + q >= rhi) continue;
        const double2 g0 = *reinterpret_cast<const double2*>(g + q), g1 = *reinterpret_cast<const double2*>(g + q + 2);
#pragma unroll
        for (int j = 0; j < CW; ++j) {
            hold(v[i][j]);
            s[j] = fma((double)v[i][j].x, g0.x, s[j]);
            s[j] = fma((double)v[i][j].y, g0.y, s[j]);
            s[j] = fma((double)v[i][j].z, g1.x, s[j]);
            s[j] = fma((double)v[i][j].w, g1.y, s[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < CW; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
    auto write_x = [&](int a, double x) {
        V.x[T.col0 + a] = x;
        V.x_old[P.perm[T.col0 + a]] = (float)x;
    };
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < CW; ++j) {
            const int a = a0 + w + kWarps * j;
            if (a >= a0 + na) continue;
            if (T.nk == 1) write_x(a, s[j]);
            else V.part[T.part + (size_t)T.k * cols_of(CW) + (a - a0)] = s[j];
        }
    }
    __syncthreads();
    if (T.nk > 1) {
        if (tid == 0) S.last = add_acq_rel(V.chunk + T.chunk) == T.nk - 1;
        __syncthreads();
        if (S.last && tid < na) {
            double x = 0.0;
            for (int k = 0; k < T.nk; ++k) x += __ldcg(V.part + T.part + (size_t)k * cols_of(CW) + tid);
            write_x(a0 + tid, x);
        }
        __syncthreads();
    }
    if (tid == 0) add_release(V.done_b + T.front);
}

__global__ void __launch_bounds__(kNT, kPerSM) sn_task_kernel(PlanView P) {
    __shared__ __align__(16) Shared S;
    const int tid = threadIdx.x, total = P.ntasks * P.nrhs;
    // One warp fetches a ticket and its task's record.
    auto fetch = [&](int slot) {
        int t = 0;
        if ((tid & 31) == 0) t = atomicAdd(P.ctr, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((tid & 31) == 0) {
            S.next[slot] = t;
            const int j = t % P.nrhs;
            int* ctr = P.ctr + 1 + j * P.ld_ctr;
            S.vec[slot] = {P.part + j * P.ld_part, P.upd + j * P.ld_upd, P.ynew + j * P.ld_n, P.xnew + j * P.ld_n,
                           ctr, ctr + P.nsn, ctr + 2 * P.nsn, P.b_old + j * P.ld_b, P.x_old + j * P.ld_x};
        }
        constexpr int N4 = (int)(sizeof(SnTask) / sizeof(int4));
        if (t < total && (tid & 31) < N4)
            reinterpret_cast<int4*>(&S.task[slot])[tid & 31] =
                __ldg(reinterpret_cast<const int4*>(P.tasks + t / P.nrhs) + (tid & 31));
    };
    if (tid < 32) fetch(0);
    __syncthreads();
    for (int cur = 0;; cur ^= 1) {
        const int t = S.next[cur];
        if (t >= total) break;
        // The last warp fetches the next task once this one's loads are issued.
        auto fetch_next = [&]() {
            if (tid >= kNT - 32) fetch(cur ^ 1);
        };
        const SnTask& T = S.task[cur];
        const Vectors& V = S.vec[cur];
        if (t / P.nrhs < P.n_fwd) forward_task(P, T, S, V, fetch_next);
        else if (T.cw == 4) backward_task<4>(P, T, S, V, fetch_next);
        else backward_task<2>(P, T, S, V, fetch_next);
        __syncthreads();  // the records and inputs are reused
    }
}

}  // namespace

void SolvePlan::build(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets, dev::Staging& stage,
                      cudaStream_t s, int* shared_err, double shrink) {
    release();
    const bool verbose = std::getenv("HDD_VERBOSE") != nullptr;
    const auto t_start = std::chrono::steady_clock::now();
    auto stamp = [&](const char* what) {
        if (verbose)
            std::fprintf(stderr, "[hdd setup]   plan (%zu factors): %s at %.3f s\n", factors.size(), what,
                         std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count());
    };
    auto scratch = [&]() {
        PlanScratch sc;
        alloc_scratch(sc, shared_err, s, bytes);
        d_part = sc.part; d_upd = sc.upd; d_ynew = sc.ynew; d_xnew = sc.xnew; d_ctr = sc.ctr;
        d_res = sc.res;
        d_err = sc.err;
        own_err = sc.own_err;
    };
    std::vector<int> base(factors.size() + 1, 0);
    n = 0;
    for (size_t f = 0; f < factors.size(); ++f) {
        if (factors[f]->Fw.size() != factors[f]->col0.size()) throw Error(HDD_ERR_INTERNAL, "solve blocks not built");
        n = std::max(n, offsets[f] + factors[f]->n);
        base[f + 1] = base[f] + (int)factors[f]->col0.size();
    }
    nsn = base.back();
    if (nsn == 0) return;
    double total = 0;
    for (const SnFactor* F : factors) total += tree_weight(*F);
    if (shrink == 1 && resident_plan(factors, total) && res.build(factors, offsets, stage, s)) {
        solve_bytes = res.solve_bytes;
        bytes = res.bytes;
        scratch();
        dev::ck(cudaStreamSynchronize(s), "plan upload");
        stamp("resident plan uploaded");
        return;
    }
    // The lower trees of every factor go to one CTA each (sn_resident.cu); the
    // tasks below are those of the fronts above them.
    // Members given the same factor share its trees' streams and the coefficients
    // of its fronts above.
    std::map<const SnFactor*, FactorCut> cuts;
    for (const SnFactor* F : factors) cuts.emplace(F, FactorCut());
    {
        std::vector<std::pair<const SnFactor* const, FactorCut>*> each;
        for (auto& c : cuts) each.push_back(&c);
        const double cap = cut_weight(total) / shrink;
        std::exception_ptr failed;
#pragma omp parallel for schedule(dynamic)
        for (size_t i = 0; i < each.size(); ++i) {
            try {
                each[i]->second = cut_trees(*each[i]->first, cap);
            } catch (...) {
#pragma omp critical
                failed = std::current_exception();
            }
        }
        if (failed) std::rethrow_exception(failed);
    }
    std::vector<ResidentPlan::Shape> shapes;
    std::vector<std::vector<ResidentPlan::Member>> members;
    std::map<const SnFactor*, size_t> shape0;  // a factor's first shape
    // The fronts above, numbered in post-order, factor by factor.
    struct Front {
        int f, j, nj, nr, col0, parent, height, depth, upd;
        long long fw, rows_off, gp, ge;
        std::vector<int> kids;  // plan fronts (trees' roots among them), in order
        int child_b, child_e, ntf, ntb;
    };
    std::vector<Front> top;
    std::vector<int> top_of(nsn, -1);
    std::vector<int> upd_off(nsn, -1);  // of the fronts above and the trees' roots
    std::vector<int> own;               // fronts whose coefficients are stored
    std::map<const SnFactor*, size_t> first_of;
    long long upd_total = 0, fw_total = 0;
    std::vector<int> rows, perm(n, 0);
    for (size_t f = 0; f < factors.size(); ++f) {
        const SnFactor& F = *factors[f];
        const size_t owner = first_of.emplace(&F, f).first->second;
        const FactorCut& C = cuts.at(&F);
        if (owner == f) {
            shape0[&F] = shapes.size();
            shapes.insert(shapes.end(), C.shapes.begin(), C.shapes.end());
            members.resize(shapes.size());
        }
        if (upd_total + C.upd_len >= (long long)INT32_MAX)
            throw Error(HDD_ERR_UNSUPPORTED, "update vectors too large for 32-bit indices");
        for (size_t i = 0; i < C.shapes.size(); ++i)
            members[shape0[&F] + i].push_back({offsets[f], (int)upd_total});
        for (int i = 0; i < F.n; ++i) perm[offsets[f] + i] = offsets[f] + F.perm[i];
        for (int j = 0; j < (int)F.col0.size(); ++j) {
            const int g = base[f] + j, nr = (int)F.rows[j].size();
            if (C.upd[j] >= 0) upd_off[g] = (int)upd_total + C.upd[j];
            if (C.low[j]) continue;
            Front T{};
            T.f = (int)f; T.j = j; T.nj = F.ncol[j]; T.nr = nr; T.col0 = offsets[f] + F.col0[j]; T.upd = upd_off[g];
            T.rows_off = (long long)rows.size();
            for (int r : F.rows[j]) rows.push_back(offsets[f] + r);
            const long long len = (long long)((T.nj + nr + 3) & ~3) * T.nj;
            if (owner == f) {
                own.push_back((int)top.size());
                T.fw = fw_total;
                fw_total += len;
            } else {
                T.fw = top[top_of[base[owner] + j]].fw;
            }
            top_of[g] = (int)top.size();
            top.push_back(std::move(T));
        }
        for (int j = 0; j < (int)F.col0.size(); ++j) {
            const int p = F.parent[j], g = base[f] + j;
            if (top_of[g] >= 0) top[top_of[g]].parent = p >= 0 ? top_of[base[f] + p] : -1;
            if (p >= 0 && top_of[base[f] + p] >= 0) top[top_of[base[f] + p]].kids.push_back(g);
        }
        upd_total += C.upd_len;
    }
    if (!shapes.empty() && !res.build_cut(shapes, members, stage, s)) {
        // Trees with unusually many update entries: smaller ones, in the end none.
        build(factors, offsets, stage, s, shared_err, shrink * 4);
        return;
    }
    stamp("trees uploaded");
    ntop = (int)top.size();
    for (int t = 0; t < ntop; ++t)
        if (top[t].parent >= 0) top[top[t].parent].height = std::max(top[top[t].parent].height, top[t].height + 1);
    for (int t = ntop - 1; t >= 0; --t)
        if (top[t].parent >= 0) top[t].depth = top[top[t].parent].depth + 1;
    // Tasks in topological order.
    std::vector<int> order(ntop);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return top[a].height < top[b].height; });
    std::vector<SnTask> tasks;
    int nchunk = 0;
    long long part_total = 0;
    auto task_of = [&](int t) {
        const Front& T = top[t];
        SnTask k{};
        k.front = t; k.nj = T.nj; k.m = T.nj + T.nr; k.col0 = T.col0; k.upd = T.upd; k.parent = T.parent;
        k.rows_off = T.rows_off;
        return k;
    };
    for (int t : order) {
        const int nj = top[t].nj, m = nj + top[t].nr;
        for (int r0 = 0; r0 < m; r0 += kRB) {
            const int cend = std::min(nj, r0 + kRB);
            const int nk = cend <= kWhole ? 1 : (cend + kCC - 1) / kCC;
            SnTask k = task_of(t);
            k.r0 = r0; k.rows = std::min(kRB, m - r0); k.nk = nk;
            k.chunk = nk > 1 ? nchunk++ : -1;
            k.part = part_total;
            if (nk > 1) part_total += (long long)nk * kRB;
            for (k.k = 0; k.k < nk; ++k.k) {
                k.c0 = k.k * kCC;
                k.ncols = nk > 1 ? std::min(kCC, cend - k.c0) : cend;
                tasks.push_back(k);
                ++top[t].ntf;
            }
        }
    }
    n_fwd = (int)tasks.size();
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return top[a].depth < top[b].depth; });
    for (int t : order) {
        const int nj = top[t].nj, m = nj + top[t].nr;
        const int cw = m <= kTallRows ? 4 : 2, bc = cols_of(cw), br = rows_of(cw);
        for (int a0 = 0; a0 < nj; a0 += bc) {
            const int nk = (m - a0 + br - 1) / br;
            SnTask k = task_of(t);
            k.r0 = a0; k.rows = std::min(bc, nj - a0); k.nk = nk; k.cw = cw;
            k.chunk = nk > 1 ? nchunk++ : -1;
            k.part = part_total;
            if (nk > 1) part_total += (long long)nk * bc;
            for (k.k = 0; k.k < nk; ++k.k) {
                k.c0 = a0 + k.k * br;
                k.ncols = std::min(br, m - k.c0);
                tasks.push_back(k);
                ++top[t].ntb;
            }
        }
    }
    n_tasks = (int)tasks.size();
    ld_ctr = 2 * ntop + nchunk;
    // Algorithmic bytes: each stored coefficient of L_JJ^{-1} (lower triangle)
    // and of -L_RJ L_JJ^{-1} read once per direction, plus b read and x written.
    double coef = 0;
    for (int t : own) coef += 0.5 * top[t].nj * (top[t].nj + 1.0) + (double)top[t].nr * top[t].nj;
    solve_bytes = 8.0 * coef + 8.0 * n + res.solve_bytes;
    stamp("fronts and tasks");
    // Coefficient blocks (FP64 -> FP32, padding rows zero) of the distinct
    // factors' fronts.
    bytes = res.bytes;
    dev::upload_packed(own.size(), fw_total, [&](size_t i) { return top[own[i]].fw; },
                       [&](size_t i, float* dst) {
                           const Front& T = top[own[i]];
                           const BlockVec& W = factors[T.f]->Fw[T.j];  // m x nj, col-major
                           const int m = T.nj + T.nr, ld = (m + 3) & ~3;
                           for (int c = 0; c < T.nj; ++c) {
                               for (int r = 0; r < m; ++r) dst[(size_t)c * ld + r] = (float)W[(size_t)c * m + r];
                               for (int r = m; r < ld; ++r) dst[(size_t)c * ld + r] = 0.0f;
                           }
                       },
                       stage, s, d_fw, bytes);
    stamp("coefficients packed and uploaded");
    // Gather lists: the children's update entries per position of a front, in
    // child order; and the children it waits for.
    std::vector<int> child, gptr, gent;
    {
        long long np = 0, ne = 0;
        for (Front& T : top) {
            T.gp = np;
            T.ge = ne;
            np += T.nj + T.nr + 1;
            T.child_b = (int)child.size();
            for (int g : T.kids) {
                const size_t f = (size_t)T.f;
                ne += (long long)factors[f]->rows[g - base[f]].size();
                if (top_of[g] >= 0) child.push_back(top_of[g]);
            }
            T.child_e = (int)child.size();
        }
        gptr.resize((size_t)np);
        gent.resize((size_t)ne);
        int bad = 0;
#pragma omp parallel for schedule(dynamic, 8) reduction(| : bad)
        for (int t = 0; t < ntop; ++t) {
            const Front& T = top[t];
            const SnFactor& F = *factors[T.f];
            const int m = T.nj + T.nr, c0 = F.col0[T.j];
            const std::vector<int>& R = F.rows[T.j];
            int* cnt = gptr.data() + T.gp;  // m + 1 entries
            std::fill(cnt, cnt + m + 1, 0);
            std::vector<int> pos;  // position of every child entry, child by child
            for (int g : T.kids)
                for (int r : F.rows[g - base[T.f]]) {
                    int p = 0;
                    if (r >= c0 && r < c0 + T.nj) p = r - c0;
                    else {
                        const auto it = std::lower_bound(R.begin(), R.end(), r);
                        if (it == R.end() || *it != r) bad = 1;
                        else p = T.nj + (int)(it - R.begin());
                    }
                    pos.push_back(p);
                    ++cnt[p + 1];
                }
            for (int q = 0; q < m; ++q) cnt[q + 1] += cnt[q];
            std::vector<int> fill(cnt, cnt + m);
            int* ent = gent.data() + T.ge;
            size_t i = 0;
            for (int g : T.kids)
                for (size_t k = 0; k < F.rows[g - base[T.f]].size(); ++k) ent[fill[pos[i++]]++] = upd_off[g] + (int)k;
        }
        if (bad) throw Error(HDD_ERR_INTERNAL, "supernode row not in parent front");
    }
    for (SnTask& k : tasks) {
        const Front& T = top[k.front];
        k.fw = T.fw;
        k.gp = T.gp;
        k.ge = T.ge;
        k.child_b = T.child_b;
        k.child_e = T.child_e;
        k.kids = T.kids.empty() ? 0 : 1;
    }
    stamp("gather lists");
    std::vector<int> ntf, ntb;
    for (const Front& T : top) {
        ntf.push_back(T.ntf);
        ntb.push_back(T.ntb);
    }
    auto nonempty = [](std::vector<int>& v) -> const std::vector<int>& {
        if (v.empty()) v.push_back(0);
        return v;
    };
    d_rows = dev::upload(nonempty(rows), s, bytes);
    d_child = dev::upload(nonempty(child), s, bytes);
    d_gptr = dev::upload(nonempty(gptr), s, bytes);
    d_gent = dev::upload(nonempty(gent), s, bytes);
    d_ntf = dev::upload(nonempty(ntf), s, bytes);
    d_ntb = dev::upload(nonempty(ntb), s, bytes);
    d_perm = dev::upload(perm, s, bytes);
    if (tasks.empty()) tasks.push_back(SnTask{});
    d_tasks = dev::upload(tasks, s, bytes);
    stamp("uploads issued");
    part_len = std::max<long long>(part_total, 1);
    upd_len = std::max<long long>(upd_total, 1);
    scratch();
    // A front with a child above the trees, for stall_dependency (the wait of its
    // tasks on that child can be made unsatisfiable).
    stall_front = -1;
    for (int t = 0; t < ntop && stall_front < 0; ++t)
        if (top[t].parent >= 0) { stall_front = t; stall_ntf = top[t].ntf; }
    // Persistent grid: as many CTAs as fit on the device; no more than tasks.
    int dev_id = 0, nsm = 0, per_sm = 0;
    dev::ck(cudaGetDevice(&dev_id), "cudaGetDevice");
    dev::ck(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev_id), "SM count");
    dev::ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sn_task_kernel, kNT, 0), "occupancy");
    grid = std::max(1, nsm * std::max(1, per_sm));
    dev::ck(cudaStreamSynchronize(s), "plan upload");
    stamp("uploaded");
}

void SolvePlan::release() {
    dev::release(d_rows); dev::release(d_child); dev::release(d_gptr); dev::release(d_gent);
    dev::release(d_ntf); dev::release(d_ntb); dev::release(d_perm); dev::release(d_tasks); dev::release(d_fw);
    dev::release(d_part); dev::release(d_upd); dev::release(d_ynew); dev::release(d_xnew); dev::release(d_ctr);
    dev::release(d_res.upd); dev::release(d_res.y);
    if (own_err) dev::release(d_err);
    res.release();
    d_err = nullptr;
    own_err = false;
    nsn = ntop = n = n_fwd = n_tasks = ld_ctr = 0;
    part_len = upd_len = 0;
    stall_front = -1;
    bytes = 0;
}

void SolvePlan::alloc_scratch(PlanScratch& sc, int* shared_err, cudaStream_t s, size_t& b, int nrhs) const {
    if (nrhs != 1 && nrhs != 2 && nrhs != 4) throw Error(HDD_ERR_INVALID_ARGUMENT, "right-hand sides per solve: 1, 2 or 4");
    sc.nrhs = nrhs;
    if (res.ngroups > 0) {
        sc.res.upd = dev::alloc_zero<double>(res.upd_len * nrhs, b, s);
        sc.res.y = dev::alloc_zero<double>(res.y_len * nrhs, b, s);
    }
    if (!whole_resident()) {
        sc.part = dev::alloc_zero<double>(part_len * nrhs, b, s);
        sc.upd = dev::alloc_zero<double>(upd_len * nrhs, b, s);
        sc.ynew = dev::alloc_zero<double>((long long)std::max(n, 1) * nrhs, b, s);
        sc.xnew = dev::alloc_zero<double>((long long)std::max(n, 1) * nrhs, b, s);
        sc.ctr = dev::alloc_zero<int>(1 + (size_t)ld_ctr * nrhs, b, s);
    }
    if (shared_err) {
        sc.err = shared_err;
        sc.own_err = false;
    } else {
        sc.err = dev::alloc_zero<int>(1, b, s);
        sc.own_err = true;
    }
}

size_t SolvePlan::scratch_bytes(int nrhs) const {
    if (nsn == 0) return 0;
    size_t t = 4 + (size_t)nrhs * 8 * (size_t)(res.upd_len + res.y_len);
    if (!whole_resident())
        t += (size_t)nrhs * (8 * (size_t)(part_len + upd_len) + 16 * (size_t)std::max(n, 1) + 4 * (size_t)ld_ctr) + 4;
    return t;
}

void SolvePlan::free_scratch(PlanScratch& sc) {
    dev::release(sc.part); dev::release(sc.upd); dev::release(sc.ynew); dev::release(sc.xnew); dev::release(sc.ctr);
    dev::release(sc.res.upd); dev::release(sc.res.y);
    if (sc.own_err) dev::release(sc.err);
    sc.err = nullptr;
    sc.own_err = false;
}

PlanScratch SolvePlan::primary() const {
    PlanScratch sc;
    sc.part = d_part; sc.upd = d_upd; sc.ynew = d_ynew; sc.xnew = d_xnew; sc.ctr = d_ctr; sc.err = d_err;
    sc.res = d_res;
    sc.own_err = false;
    sc.nrhs = 1;
    return sc;
}

void SolvePlan::solve(const float* b_old, float* x_old, cudaStream_t s, long long& launches, PhaseHook* hook) const {
    solve(primary(), b_old, x_old, s, launches, hook);
}

void SolvePlan::solve(const PlanScratch& sc, const float* b_old, float* x_old, cudaStream_t s, long long& launches,
                      PhaseHook* hook, int nrhs, long long ld_b, long long ld_x) const {
    if (nsn == 0) return;
    if ((nrhs != 1 && nrhs != 2 && nrhs != 4) || nrhs > sc.nrhs)
        throw Error(HDD_ERR_INVALID_ARGUMENT, "right-hand sides per solve: 1, 2 or 4, within the scratch");
    if (hook) hook->begin(kPhaseSolve);
    const TopVectors top{sc.upd, sc.xnew, upd_len, (long long)std::max(n, 1), sc.ctr,
                         sc.ctr ? 1 + (long long)ld_ctr * nrhs : 0};
    auto trees = [&](int mode) {
        res.launch(mode, sc.res, top, sc.err, sc.grid_div, spin_limit, b_old, x_old, s, nrhs, ld_b, ld_x);
        ++launches;
    };
    if (whole_resident()) {
        trees(0);
    } else {
        // The forward launch of the trees clears the counters.
        if (res.ngroups > 0) trees(1);
        else dev::ck(cudaMemsetAsync(sc.ctr, 0, sizeof(int) * (size_t)top.n_ctr, s), "reset counters");
        if (n_tasks > 0) {
            const PlanView P{ntop, n_fwd, n_tasks, d_rows, d_child, d_gptr, d_gent, d_ntf, d_ntb, d_perm, d_fw,
                             d_tasks, b_old, x_old, sc.part, sc.upd, sc.ynew, sc.xnew, sc.ctr, sc.err, spin_limit,
                             part_len, upd_len, (long long)std::max(n, 1), ld_ctr, ld_b, ld_x, nrhs};
            const int full = std::min(grid, n_tasks * nrhs);
            const int g = sc.grid_div > 1 ? std::min(full, std::max(1, (grid + sc.grid_div - 1) / sc.grid_div)) : full;
            sn_task_kernel<<<g, kNT, 0, s>>>(P);
            dev::ck(cudaGetLastError(), "sn tasks");
            ++launches;
        }
        if (res.ngroups > 0) trees(2);
    }
    if (hook) hook->end(kPhaseSolve, solve_bytes + 16.0 * n * (nrhs - 1));
}

void SolvePlan::stall_dependency(bool on, cudaStream_t s) {
    if (stall_front < 0) {
        if (res.ngroups > 0) res.set_gate(on ? 1 : 0, s);
        return;
    }
    const int v = on ? stall_ntf + 1 : stall_ntf;
    dev::ck(cudaMemcpyAsync(d_ntf + stall_front, &v, sizeof(int), cudaMemcpyHostToDevice, s), "stall dependency");
    dev::ck(cudaStreamSynchronize(s), "stall dependency");
}

int SolvePlan::error_flag(cudaStream_t s) const {
    if (!d_err) return 0;
    int h = 0;
    dev::ck(cudaMemcpyAsync(&h, d_err, sizeof(int), cudaMemcpyDeviceToHost, s), "read error flag");
    dev::ck(cudaStreamSynchronize(s), "read error flag");
    return h;
}

}  // namespace hdd
