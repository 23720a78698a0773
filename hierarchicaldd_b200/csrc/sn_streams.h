// The schedule of solves with one CTA per elimination tree: the format of the
// warps' streams that sn_resident.cu runs, and the host code that writes them
// (sn_streams.cpp, without CUDA calls, so that CPU tests can walk a schedule).
#pragma once
#include <array>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "sigma.h"

#ifdef __CUDACC__
#define HDD_HD __host__ __device__
#else
#define HDD_HD
#endif

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
    int member0, count;
    int top;                  // cut trees: the member's first update vector in the plan above
};

constexpr int kLine = 512;              // bytes of a line: 16 a lane
constexpr int kBatch = 4;               // lines copied, waited for and released together
constexpr int kBatchBytes = kBatch * kLine;
// Batches in flight per warp (K trees per CTA; the vectors of more leave less room).
HDD_HD constexpr int depth_of(int k) { return k == 1 ? 4 : 2; }

// Operations of a stream.  Each starts with a batch whose first line is the
// header, an int4 for every lane: {type | log2 of the lanes on row quads << 4 |
// flags << 8 | count << 16, ... | CTA barriers after the operation << 20, two
// words of the type}.  The barriers are a count, so that a warp without work in
// a phase needs no operation for it.
enum : int {
    kEnd = 0,
    kNothing = 1,   // barriers only
    // Items on 1 to 3 lines (count), one per lane: {index, first, second entry,
    // 1 when the index is a slot (GS)}: M[index] += the two entries.
    kAssemble = 2,
    // A block of a front times its inputs: count groups of four steps (a batch
    // each).  Header, forward: the lane's first column | distance to its next
    // << 16 (4 bits), and the indices of the last group's four steps (16 bits
    // each).
    // Lines: destinations of four rows a lane; forward the rows' pairs of
    // children's entries (16 bits each) and one item of an assembly before
    // (index -1: none); backward the columns' indices for the first sixteen
    // steps (eight 16-bit indices a lane and line), a batch of four more such
    // lines following every further 32 steps.  Steps past the block's columns
    // read the zero: what lies behind them may be another system's NaN or
    // written by another warp, and zero coefficients do not undo a NaN.
    kProduct = 3,
    // Items on 1 to 3 lines: {first partial sum, destination, first, second
    // entry}.  Header: slices (16 bits), distance between their partial sums.
    kFinish = 4
};
constexpr int kPairs = 1;      // the rows have children's entries
constexpr int kItem = 2;       // the product starts with an assembly
constexpr int kTransposed = 4;
constexpr int kTopRoot = 8;    // destinations -1 - entry are the plan above's update vectors
// Indices are into the CTA's array M: the vector, rows outside cut trees, a
// zero (a pair's missing entries), an unused entry (results of no row, never
// read), partial sums and, where they fit, update slots.  GS: slots are in global memory
// instead (destination -1 - slot; a pair's entries are slots, slot 0 the zero).

// One operation of a warp, before it is written.
struct Op {
    int type, flags, bars;            // bars: barriers after it
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
    int entries() const { return part0 + part_len; }  // of M, without slots
};
// While M is not laid out, slots are numbered from kSlot on and kZero is the zero.
constexpr int kSlot = 0x20000000, kZero = 0x10000000;

// Everything of a ResidentPlan that does not need the device.
struct ResidentSchedule {
    bool cut = false, global_slots = false;
    int max_n = 0, km = 1, nt = 512;
    int entries = 0;                     // entries of M
    size_t smem = 0;                     // shared memory of a CTA
    std::vector<RGroup> groups;
    std::vector<RWarp> warps;
    std::vector<int> off, perm, ext;
    long long upd_len = 0, y_len = 0;    // doubles of the scratch
    double coef = 0;                     // coefficients of one direction, each class's once
    // Schedules shapes[c] for members[c] on a device of nsm SMs; false when a CTA's shared memory does not hold the trees.
    // The shapes are referred to until the streams are written.
    bool plan(const std::vector<ResidentPlan::Shape>& shapes,
              const std::vector<std::vector<ResidentPlan::Member>>& members, bool cut_trees, int nsm);
    // The streams, one per class and warp, in floats: `total` in all (padding
    // that prefetches run into included), stream i from at(i) on.
    size_t streams() const { return stream.size(); }
    long long total() const;
    long long at(size_t i) const { return stream[i].at; }
    void write(size_t i, float* dst) const;

private:
    struct Item { int c, w; long long at; };
    const std::vector<ResidentPlan::Shape>* shape = nullptr;
    std::vector<ClassPlan> cp;
    std::vector<Item> stream;            // the last: padding
};

// Whole factors: a shape per distinct factor, and its members' offsets.
void whole_shapes(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets,
                  std::vector<ResidentPlan::Shape>& shapes, std::vector<std::vector<ResidentPlan::Member>>& members);

// What a factor's trees weigh for the rules below.
double tree_weight(const SnFactor& F);
// Plans solved by one CTA per factor: every factor's unknowns fit a CTA's
// shared memory, and cutting them would not pay.  total: all factors' weight.
bool resident_plan(const std::vector<const SnFactor*>& factors, double total);
// The heaviest tree cut from a plan of weight `total`.
double cut_weight(double total);
// The lower trees of factor F: the largest subtrees of at most weight `cap`;
// consecutive ones share a CTA (a shape) up to that weight.
struct FactorCut {
    std::vector<char> low;            // fronts of the trees
    std::vector<ResidentPlan::Shape> shapes;
    // Offsets of the update vectors of the trees' roots and the fronts above
    // (-1: of the others), and their length in all.
    std::vector<int> upd;
    long long upd_len = 0;
};
FactorCut cut_trees(const SnFactor& F, double cap);

}  // namespace hdd
