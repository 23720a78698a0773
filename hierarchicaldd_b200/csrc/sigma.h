// Interface (Schur complement, "sigma") solver: host assembly of the
// adaptive-hierarchy Galerkin matrices, supernodal Cholesky factorisations and
// the device-side sigma V-cycle.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstdint>
#include <string>
#include <vector>
#include <utility>
#include <type_traits>
#include <memory>

#include "hdd_common.h"

namespace hdd {

struct DomainLayout;
namespace dev { class Staging; }

struct CsrF {
    int rows = 0, cols = 0;
    std::vector<int> ptr, col;
    std::vector<float> val;
};

// Interface system in the reference's DOF numbering
// (CPU/Interface_Solver/INTERFACE_MATRIX_GENERATOR.h:130-735).
struct InterfaceHost {
    int M = 0, n_sub = 0;
    std::vector<int> n_iface;                       // [level]
    std::vector<std::array<int, 3>> iface_map;      // level-0 interface DOF -> cell
    std::vector<CsrF> Arr, Prr;                     // [level]
    std::vector<std::vector<CsrF>> Aii, Air;        // [level][subdomain]
    // DOF positions in finest-level grid units (used only for the fill-reducing
    // ordering of the factorisations).
    std::vector<std::vector<std::array<int, 3>>> iface_xyz;             // [level][dof]
    std::vector<std::vector<std::vector<std::array<int, 3>>>> aii_xyz;  // [level][subdomain][dof]
};

// Builds the interface system from the caller's flags (before the global
// Domain_Divider pass, as the reference splits first), in parallel over
// subdomains.
void build_interface(const DomainLayout& L, int sigma_levels, InterfaceHost& out);

// Two-level DD: the second-level interface systems of every first-level
// subdomain of sub cells (L.opt.size and L.flags_in are read), stacked into
// one block-diagonal system on boxes of sub/2.
void build_second_level(const DomainLayout& L, const int sub[3], int sigma_levels, InterfaceHost& out);

// Interface dump and reload, the reference's -iomode output / input
// (CPU/SPGrid_Domain_Decomposition_Solver/SPGrid_Domain_Decomposition_Solver.h:121-161);
// host_interface_io.cpp.  read_interface_dir throws HDD_ERR_IO on a missing or
// malformed file; check_interface throws HDD_ERR_INVALID_ARGUMENT when a
// reloaded system does not fit the domain (levels, subdomain count, sizes,
// interface cells).
void write_interface_dir(const InterfaceHost& ih, const std::string& dir);
void read_interface_dir(const std::string& dir, InterfaceHost& ih);
void check_interface(const DomainLayout& L, int sigma_levels, const InterfaceHost& ih);

// Allocator whose resize leaves new elements uninitialised, for blocks that are
// written in full right after (by several threads, instead of one thread
// zeroing them first).
template <class T>
struct NoInitAlloc : std::allocator<T> {
    template <class U>
    struct rebind { using other = NoInitAlloc<U>; };
    NoInitAlloc() = default;
    template <class U>
    NoInitAlloc(const NoInitAlloc<U>&) noexcept {}
    template <class U>
    void construct(U* p) noexcept(std::is_nothrow_default_constructible<U>::value) {
        ::new (static_cast<void*>(p)) U;
    }
    template <class U, class... Args>
    void construct(U* p, Args&&... args) {
        ::new (static_cast<void*>(p)) U(std::forward<Args>(args)...);
    }
};
using BlockVec = std::vector<double, NoInitAlloc<double>>;

// Supernodal Cholesky of (A + eps I) (zero rows get eps), the stand-in for
// the reference's MKL PARDISO phases 11/22 (SIGMA_SMOOTHER.cpp:115-288).
// Supernodes are the fronts of a nested-dissection separator tree.
struct SnFactor {
    int n = 0;
    std::vector<int> perm;                     // new -> old
    std::vector<int> col0, ncol, parent;       // per supernode, post-order
    std::vector<std::vector<int>> rows;        // below-diagonal rows (new indices), sorted
    std::vector<BlockVec> Ljj, Lrj;            // col-major dense blocks (L_JJ: lower triangle only)
    std::vector<BlockVec> Fw;                  // [Linv; -L_RJ Linv], (nj+nr) x nj col-major
    // Nested-dissection ordering and symbolic factorisation.  With DOF
    // positions the separators are planes cut at the median along the axis
    // that gives the smallest separator; without them, breadth-first level sets.
    void analyze(const CsrF& A, const std::vector<std::array<int, 3>>* xyz = nullptr);
    void factor(const CsrF& A, double eps);
    void build_solve_blocks();
    void solve(double* x) const;               // host reference solve (tests)
};

// Optional per-phase device timing: the caller records events around the
// launches of a phase and accumulates the phase's algorithmic bytes.
struct PhaseHook {
    virtual void begin(int phase) = 0;
    virtual void end(int phase, double bytes) = 0;

protected:
    ~PhaseHook() = default;
};

// Timing phase of the supernodal solves (both directions).
constexpr int kPhaseSolve = 6;

// Host reference of a solve plan (sn_plan.cpp): the fronts of a batch of
// independent factorisations with concatenated unknowns and the FP32
// coefficient blocks Fw the device plan stores, solved front by front in
// post-order with FP64 accumulation and FP64 vectors between fronts (the
// device kernels' arithmetic, up to the order of FP64 sums).  Test
// infrastructure for the device plan: CPU tests check it against the FP64
// factorisation, GPU tests check the device solve against it.
struct PlanHost {
    int n = 0, nsn = 0;
    std::vector<int> perm;                        // new -> old (concatenated)
    std::vector<int> col0, ncol, nrow, parent, rows;
    std::vector<long long> rows_off, fw_off;
    std::vector<float> fw;                        // Fw blocks, m x nj col-major, ld round4(m)
    void build(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets);
    void emulate(const float* b_old, float* x_old) const;
};

// DOF positions (for the fill-reducing ordering) of level l's interface
// system and of subdomain sd's interior system, or null when assembly did not
// record them.
const std::vector<std::array<int, 3>>* interface_positions(const InterfaceHost& ih, int l);
const std::vector<std::array<int, 3>>* interior_positions(const InterfaceHost& ih, int l, int sd);

// Subdomains of level l with equal interior systems (matrix and, where known,
// DOF positions relative to the first DOF): entry sd is the first subdomain
// whose system equals sd's.  Equal systems have equal factors.
std::vector<int> interior_classes(const InterfaceHost& ih, int l);

// Factorisations of one interface solve as the sigma solver builds them
// (A + 1e-5 I, ordering from the positions, explicit solve blocks) and the
// plan over them: kind 0 = Arr of level l, kind 1 = Aii of every subdomain of
// level l with the unknowns concatenated in subdomain order.
void interface_solve_plan(const InterfaceHost& ih, int kind, int l, std::vector<SnFactor>& factors, PlanHost& plan);

// One unit of device work of the fronts above a plan's cut trees, taken by a CTA
// of the persistent task kernel (sn_solve.cu), with what the CTA needs of the
// front.  Forward: rows [r0, r0+rows) of front `front` times its columns [c0,
// c0+ncols); backward: columns [r0, r0+rows) over rows [c0, c0+ncols).  A block
// split into nk > 1 tasks writes partial sums to `part`, which the last task to
// finish (counter `chunk`) adds in order.
struct alignas(16) SnTask {
    int front, r0, rows, c0, ncols, k, nk, chunk;
    int nj, m, col0, parent;       // the front's columns, rows, first unknown, parent (-1: root)
    int upd, child_b, child_e;     // its update vector; the children it waits for
    int kids, cw, pad;             // whether it has children at all; backward: columns per warp
    long long part, fw, rows_off, gp, ge;  // offsets of partial sums, coefficients, rows, gather lists
};

// What a ResidentPlan's launches write besides the solution.
struct ResidentScratch {
    double *upd = nullptr, *y = nullptr;
};

// The device buffers one supernodal solve writes (split-block partial sums,
// update vectors, forward and backward results, task counters, error word):
// every solve context of a plan has its own, so solves of one plan on
// different streams can run at the same time.
struct PlanScratch {
    double *part = nullptr, *upd = nullptr, *ynew = nullptr, *xnew = nullptr;
    int* ctr = nullptr;
    ResidentScratch res;
    int* err = nullptr;
    bool own_err = false;
    // The persistent launches use 1/grid_div of the plan's CTAs (rounded up),
    // leaving room on the device for concurrent solves; the results do not
    // depend on it.
    int grid_div = 1;
    int nrhs = 1;  // right-hand sides the buffers hold (1, 2 or 4)
};

struct RGroup;
struct RWarp;

// Cut trees: the update vectors (written going up) and the solution (read
// coming down) of the plan above them; right-hand side j at + j ld.
struct TopVectors {
    double* upd = nullptr;
    const double* x = nullptr;
    long long ld_upd = 0, ld_x = 0;
    int* ctr = nullptr;       // counters that the forward launch clears
    long long n_ctr = 0;
};

// Plan of solves with one CTA per elimination tree, or per group of them
// (sn_resident.cu).
struct ResidentPlan {
    static constexpr size_t kMaxSmem = 226 * 1024;
    // Trees of one factor solved by one CTA: fronts first .. last (the root) of
    // each; top: where the root's update vector goes, from the first of the
    // factor's update vectors in the plan above (-1: the root has none).
    struct Tree { int first, last, top; };
    struct Shape {
        const SnFactor* F = nullptr;
        std::vector<Tree> trees;
    };
    // One use of a shape's factor: offset of its unknowns, and of its update
    // vectors in the plan above.
    struct Member { int off, top; };
    bool cut = false;                   // cut trees: separate forward and backward launches
    int n = 0, max_n = 0, ngroups = 0;  // unknowns; largest vector; CTAs of one solve (0: no plan)
    int km = 1, nt = 256;               // trees per CTA (1, 2 or 4), threads per CTA
    int resident = 1;                   // CTAs that fit on the device
    size_t smem = 0, bytes = 0;         // shared memory per CTA; device bytes
    long long upd_len = 0, y_len = 0;   // doubles of a ResidentScratch's buffers
    double solve_bytes = 0;             // algorithmic bytes of one solve, both directions
    bool global_slots = false;          // update entries in global memory (they do not fit shared memory)
    RGroup* d_groups = nullptr;
    RWarp* d_warps = nullptr;
    int *d_off = nullptr, *d_perm = nullptr, *d_ext = nullptr;
    char* d_stream = nullptr;           // every class's warp streams: coefficients and indices
    int* d_gate = nullptr;
    // Shared memory of the rings and of k trees of `entries` doubles each.
    static size_t smem_bytes(int entries, int k, int nt);
    // Whole factors: factors[i] solves the unknowns from offsets[i] on; members
    // given the same SnFactor form a class that shares its coefficients.  False
    // when a CTA's shared memory does not hold the trees.
    bool build(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets, dev::Staging& stage,
               cudaStream_t s);
    // Cut trees: shapes[i] for each of members[i].
    bool build_cut(const std::vector<Shape>& shapes, const std::vector<std::vector<Member>>& members, dev::Staging& stage,
                   cudaStream_t s);
    void release();
    // mode: 0 whole trees, both directions; 1 / 2 the forward / backward half of cut trees.
    void launch(int mode, const ResidentScratch& sc, const TopVectors& top, int* err, int grid_div,
                long long spin_limit, const float* b_old, float* x_old, cudaStream_t s, int nrhs, long long ld_b,
                long long ld_x) const;
    // Test seam: while nonzero, every solve of whole trees waits for it (bounded) and raises the error word.
    void set_gate(int v, cudaStream_t s);

private:
    bool build_shapes(const std::vector<Shape>& shapes, const std::vector<std::vector<Member>>& members,
                      dev::Staging& stage, cudaStream_t s);
};

// Device plan for a batch of independent supernodal triangular solves.
struct SolvePlan {
    // One CTA per tree: the whole plan, or (cut) the lower trees of a task plan
    // that has the fronts above them.
    ResidentPlan res;
    bool whole_resident() const { return res.ngroups > 0 && !res.cut; }
    int n = 0;                       // total unknowns (concatenated)
    int nsn = 0, ntop = 0;           // fronts; those above the cut trees
    int n_fwd = 0, n_tasks = 0;      // forward tasks, all tasks
    int ld_ctr = 0;                  // ints of one right-hand side's counters
    int grid = 0;                    // persistent CTAs of the task launch
    double solve_bytes = 0;          // algorithmic bytes of one solve, both directions
    int *d_rows = nullptr, *d_child = nullptr;
    int *d_gptr = nullptr, *d_gent = nullptr;  // gather lists (see sn_solve.cu)
    int *d_ntf = nullptr, *d_ntb = nullptr;    // tasks per front, forward / backward
    int* d_perm = nullptr;           // new -> old (concatenated)
    SnTask* d_tasks = nullptr;
    float* d_fw = nullptr;           // Fw blocks of the fronts above
    ResidentScratch d_res;
    double* d_part = nullptr;        // partial sums of split blocks
    double* d_upd = nullptr;         // update vectors
    double* d_ynew = nullptr;        // forward result in new order
    double* d_xnew = nullptr;        // backward result in new order
    int* d_ctr = nullptr;            // ticket, completion and chunk counters
    int* d_err = nullptr;            // set when a bounded wait gives up
    bool own_err = false;            // d_err allocated by this plan (else shared)
    long long spin_limit = 1LL << 22;  // polls of a bounded wait before it gives up
    int stall_front = -1, stall_ntf = 0;  // front used by stall_dependency and its task count
    size_t bytes = 0;
    // shared_err: an error word shared with other plans (owned by the caller),
    // or null for a word of the plan's own.  shrink: divides the size of cut trees.
    void build(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets, dev::Staging& stage,
               cudaStream_t s, int* shared_err = nullptr, double shrink = 1);
    void release();
    long long part_len = 0, upd_len = 0;  // doubles in a scratch's partial-sum and update buffers
    // x_old = (A+eps I)^{-1} b_old (both in the concatenated original order),
    // with the plan's own scratch or a context's.
    void solve(const float* b_old, float* x_old, cudaStream_t s, long long& launches,
               PhaseHook* hook = nullptr) const;
    // With nrhs = 2 or 4 it solves that many systems at once: right-hand side
    // j at b_old + j ld_b, solution at x_old + j ld_x, one system's work beside
    // the other's; each solution is bit-identical to its solve alone.  (Kernels
    // that fed all systems from each coefficient they loaded were slower: whole
    // solves of a batch of four took 70 ms at 64^3, 343 at 128^3 and 1176 at 192^3;
    // these take 30, 122 and 431, and a solve alone 18, 58 and 151.)
    void solve(const PlanScratch& sc, const float* b_old, float* x_old, cudaStream_t s, long long& launches,
               PhaseHook* hook = nullptr, int nrhs = 1, long long ld_b = 0, long long ld_x = 0) const;
    // Scratch for another solve context (error word shared_err, or its own),
    // for up to nrhs right-hand sides per solve.
    void alloc_scratch(PlanScratch& sc, int* shared_err, cudaStream_t s, size_t& bytes, int nrhs = 1) const;
    static void free_scratch(PlanScratch& sc);
    PlanScratch primary() const;
    // Device bytes alloc_scratch takes (without a shared error word).
    size_t scratch_bytes(int nrhs = 1) const;
    int error_flag(cudaStream_t s) const;
    // Test seam: on = raise the forward task count that one front's parent
    // waits for by one, so that wait can never be satisfied and runs into its
    // poll limit; off = restore it.
    void stall_dependency(bool on, cudaStream_t s);
    ~SolvePlan() { release(); }
};

struct DeviceCsr {
    int rows = 0, cols = 0, nnz = 0;
    int *ptr = nullptr, *col = nullptr;
    float* val = nullptr;
    void upload(const CsrF& m, cudaStream_t s);
    void release();
};

struct SigmaLevel {
    int n_iface = 0, n_int = 0;
    DeviceCsr air;      // concatenated Air (rows: interior DOFs of all subdomains)
    DeviceCsr airT;     // its transpose (rows: interface DOFs)
    DeviceCsr arr;      // Arr (for residuals)
    DeviceCsr prr;      // Prr (fine x coarse)
    DeviceCsr prrT;     // Prr^T
    SolvePlan aii, arr_solve;
    float *u = nullptr, *r = nullptr, *b = nullptr, *tmp = nullptr, *vb = nullptr, *vx = nullptr;
};

// The device buffers one sigma V-cycle writes: every level's vectors, the
// scratch of its solve plans, the coarsest level's [0; b] / solution pair and
// the error word.  The solver's first solve context uses the SigmaGpu's own;
// further contexts (concurrent solves of one resident domain) allocate theirs.
struct SigmaScratch {
    // Level vectors for nrhs systems: system j's interface vectors (u, r, b,
    // tmp) at + j * si, its interior vectors (vb, vx) at + j * sn.
    struct Level {
        float *u = nullptr, *r = nullptr, *b = nullptr, *tmp = nullptr, *vb = nullptr, *vx = nullptr;
        size_t si = 0, sn = 0;
        PlanScratch aii, arr;
    };
    int nrhs = 1;
    size_t kbs = 0;  // stride of the coarsest level's [0; b] / solution pair
    std::vector<Level> lv;
    PlanScratch bottom;
    void set_grid_div(int div) {
        for (Level& L : lv) L.aii.grid_div = L.arr.grid_div = div;
        bottom.grid_div = div;
    }
    float *kb = nullptr, *kx = nullptr;
    int* err = nullptr;
    size_t bytes = 0;
    float* b0() const { return lv.empty() ? nullptr : lv[0].b; }
    float* u0() const { return lv.empty() ? nullptr : lv[0].u; }
};

struct SigmaGpu {
    int M = 0, smoothing = 3;
    std::vector<SigmaLevel> lv;
    // Coarsest level: sparse Cholesky of K = [Aii+eps, -Air; -Air^T, Arr+eps]
    // (all subdomain interiors first, then the interface), whose interface block
    // solves the Schur complement S exactly.
    SolvePlan bottom;
    float *kb = nullptr, *kx = nullptr;
    int n_bottom = 0, n_bottom_int = 0;
    double bottom_contraction = 0;   // estimated spectral radius of the bottom smoother
    // True when 200 bottom smoothing steps have converged to S^{-1} b (rho^200 <=
    // 1e-7), so the coarsest level is one solve of K; false runs the 200 steps.
    bool bottom_exact = true;
    static constexpr int kBottomSmoothing = 200;  // SIGMA_MULTIGRID_SOLVER.cpp:43
    size_t device_bytes = 0;
    // Error word shared by every solve plan of this solver: nonzero once a
    // bounded wait gave up (then later waits return at once).
    int* d_err = nullptr;
    // force_exact: solve the coarsest level exactly even where the 200
    // smoothing steps have not converged (HDD_COARSE_EXACT).
    void setup(const InterfaceHost& ih, int smoothing_iterations, cudaStream_t s, bool force_exact = false);
    void release();
    // u[0] = sigma V-cycle(b[0], u[0]) (SIGMA_MULTIGRID_SOLVER.cpp:35-47) in the
    // given scratch (default: the SigmaGpu's own).  u0_zero: the caller has
    // set u[0] = 0.
    void vcycle(bool u0_zero, cudaStream_t s, long long& launches, PhaseHook* hook = nullptr);
    // With sc.nrhs = 2 or 4 it runs that many V-cycles at once (each
    // bit-identical to its V-cycle alone), every supernodal solve taking all
    // right-hand sides in the same launches.
    void vcycle(const SigmaScratch& sc, bool u0_zero, cudaStream_t s, long long& launches, PhaseHook* hook = nullptr);
    SigmaScratch primary() const;
    void alloc_scratch(SigmaScratch& sc, cudaStream_t s, int nrhs = 1) const;
    size_t scratch_bytes(int nrhs = 1) const;
    static void free_scratch(SigmaScratch& sc);
    // Nonzero when a bounded wait inside a supernodal solve gave up.
    int error_flag(cudaStream_t s) const;
    void clear_error(cudaStream_t s);
    static int error_flag(const SigmaScratch& sc, cudaStream_t s);
    static void clear_error(const SigmaScratch& sc, cudaStream_t s);
    // Poll limit of every bounded wait (default 1 << 22).
    void set_wait_limit(long long polls);
    // Test seam (SolvePlan::stall_dependency) on the level-0 interface plan.
    void stall_dependency(bool on, cudaStream_t s);
    float* b0() const { return lv.empty() ? nullptr : lv[0].b; }
    float* u0() const { return lv.empty() ? nullptr : lv[0].u; }
    ~SigmaGpu() { release(); }
};

}  // namespace hdd
