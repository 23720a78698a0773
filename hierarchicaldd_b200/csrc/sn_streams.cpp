// Schedules of solves with one CTA per elimination tree (format: sn_streams.h,
// kernel: sn_resident.cu), and the rules for which trees are solved so.
#include "sn_streams.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <numeric>
#include <string>

namespace hdd {

namespace {

// Partial sums a tree may need beside its unknowns.
constexpr int kPartMax = 4096;
// The trees one CTA takes of a cut plan: at most a cut of front_weight() and a
// vector of kCutLen.  A front costs its coefficients and about what 1000
// coefficients do for its operations (the trees of sparse domains are thousands
// of tiny fronts).  The cut grows with the plan so that its trees are about one
// CTA per SM: larger ones would take longer than the task levels they save,
// smaller ones leave more of those.  Measured (us per solve at cuts of total/280
// and at least 16000, total/250 and 36000, total/220 and 48000 (these),
// total/170 and 48000): level-0 interface of 40x36x44, sub 8: 78, 77, 73, 74;
// 64^3, sub 16: 84, 82, 79, 79; 128^3, sub 32: 119, 120, 121, 117; 192^3: 272,
// 271, 272, 273, its second level 160, 159, 164, 159 and third 89, 89, 90, 92;
// second level of sparse 128^3 41, 36, 27, 28; two-level interiors 85, 84, 84, 88.
// Which is best changes by a few per cent; the minimum matters most.
constexpr double kCutMin = 48000, kCutMax = 200000, kCutShare = 220;
// One CTA per whole tree takes as long as its largest tree's weight; cut, about
// as long as kCutCost, and a kCutRate-th of all.  Measured (us per solve, whole
// and cut): a 16^3 domain's interface (564 unknowns) 25 and 35; interiors of
// 40x36x44 (sub 8) 21 and 24, of 64^3 (sub 16) 38 and 49, of 192^3 (216 of 32^3)
// 186 and 356; bubble 48^3 second interface level 133 and 57, sparse 128^3 323 and
// 28; 16 interiors of a two-level domain 158 and 63.  Near the line cutting can win
// on the whole side too: the 64 interiors of 128^3 (sub 32) take 169 and 134.
constexpr double kCutCost = 300000, kCutRate = 80;
constexpr int kCutLen = 8192;

double front_weight(const SnFactor& F, size_t j) {
    return 1000.0 + 0.5 * F.ncol[j] * (F.ncol[j] + 1.0) + (double)F.rows[j].size() * F.ncol[j];
}

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
constexpr int kMaxBars = 4095;

}  // namespace

int Op::batches() const {
    if (type == kProduct) {
        const int g = groups_of(rows, c1 - c0);
        return 1 + g + ((flags & kTransposed) ? index_batches(g) : 0);
    }
    return 1;
}

namespace {

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
    // Ends a phase: a barrier more after the warps' last operations.
    auto barrier = [&]() {
        for (auto& ops : out) {
            if (ops.empty() || ops.back().bars == kMaxBars) {
                Op b{};
                b.type = kNothing;
                ops.push_back(b);
            }
            ++ops.back().bars;
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
        for (int r : F.rows[t.last]) P.ext.push_back(r);
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
    auto header = [&](int lmq, int count, int a = 0, int b = 0) {
        for (int l = 0; l < 32; ++l) {
            h[4 * l] = o.type | lmq << 4 | o.flags << 8 | count << 16;
            h[4 * l + 1] = a | (int)((uint32_t)o.bars << 20);
            h[4 * l + 2] = b;
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
        header(0, (n + 31) / 32, o.nsl, o.stride);
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
    header(lmq, groups);
    // The index of a lane's step: past the block's columns the zero.
    auto input = [&](int l, int step) {
        const int c = o.c0 + (l >> lmq) + step * ns;
        return c < o.c1 ? P.idx[i][c] : P.zero;
    };
    if (!tr)
        for (int l = 0; l < 32; ++l) {
            h[4 * l + 1] |= (P.c0[i] + o.c0 + (l >> lmq)) | ns << 16;
            for (int u = 0; u < 4; ++u) h[4 * l + 2 + u / 2] |= input(l, 4 * (groups - 1) + u) << (u % 2 * 16);
        }
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
            else p[0] = -1;
        }
    }
    // Eight steps' column indices, 16 bits each.
    auto index_line = [&](uint32_t* line, int step0) {
        uint16_t* p = reinterpret_cast<uint16_t*>(line);
        for (int l = 0; l < 32; ++l)
            for (int u = 0; u < 8; ++u) p[8 * l + u] = (uint16_t)input(l, step0 + u);
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

void whole_shapes(const std::vector<const SnFactor*>& factors, const std::vector<int>& offsets,
                  std::vector<ResidentPlan::Shape>& shapes, std::vector<std::vector<ResidentPlan::Member>>& members) {
    std::map<const SnFactor*, int> shape_of;
    for (size_t f = 0; f < factors.size(); ++f) {
        const SnFactor* F = factors[f];
        auto it = shape_of.find(F);
        if (it == shape_of.end()) {
            it = shape_of.emplace(F, (int)shapes.size()).first;
            ResidentPlan::Shape T;
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
        members[it->second].push_back({offsets[f], 0});
    }
}

bool ResidentSchedule::plan(const std::vector<ResidentPlan::Shape>& shapes,
                            const std::vector<std::vector<ResidentPlan::Member>>& members, bool cut_trees, int nsm) {
    cut = cut_trees;
    shape = &shapes;
    double biggest = 0;
    for (const ResidentPlan::Shape& T : shapes) {
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
    // Sixteen warps, or four where a tree is a few lines a warp; cut trees that
    // are more than the SMs run two CTAs to an SM.
    auto groups_for = [&](int k) {
        size_t g = 0;
        for (const auto& m : members) g += (m.size() + k - 1) / k;
        return g;
    };
    if (cut) nt = groups_for(1) > (size_t)nsm ? 256 : 512;
    else nt = biggest <= 8192 ? 128 : 512;
    cp.assign(shapes.size(), ClassPlan());
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
    auto fits32 = [](long long v) {
        if (v > (long long)INT32_MAX) throw Error(HDD_ERR_UNSUPPORTED, "solve plan too large for 32-bit indices");
        return (int)v;
    };
    // M's entries with and without the update slots; trees per CTA.
    int bare = 0, all = 0;
    for (const ClassPlan& P : cp) {
        bare = std::max(bare, P.entries());
        all = std::max(all, P.entries() + P.slots);
    }
    // CTAs of four warps keep their slots in shared memory (there is no kernel
    // of theirs without): one tree's always fit, 8192 coefficients being at most
    // as many unknowns and as many entries.
    const int least = nt == 128 ? all : bare;
    km = 1;
    while (!cut && km < 4 && groups_for(km) > (size_t)nsm &&
           ResidentPlan::smem_bytes(least, 2 * km, nt) <= ResidentPlan::kMaxSmem)
        km *= 2;
    global_slots = !cut && (ResidentPlan::smem_bytes(all, km, nt) > ResidentPlan::kMaxSmem || all >= 65536);
    entries = global_slots ? bare : all;
    smem = ResidentPlan::smem_bytes(entries, km, nt);
    bool fits = smem <= ResidentPlan::kMaxSmem;
    for (ClassPlan& P : cp) {
        P.slot0 = global_slots ? -1 : P.entries();
        fits &= P.slots + 1 < 65536;
    }
    if (!fits) return false;  // partial sums or update entries of unusual trees
    std::vector<RGroup> classes(shapes.size());  // the fields of its groups
    long long at = 0;
    for (size_t c = 0; c < shapes.size(); ++c) {
        const ClassPlan& P = cp[c];
        RGroup& C = classes[c];
        C.n = P.n;
        C.perm = fits32(perm.size());
        C.next = (int)P.ext.size();
        C.ext = fits32(ext.size());
        C.warps = fits32(warps.size());
        C.stream = 4 * at;
        perm.insert(perm.end(), P.perm.begin(), P.perm.end());
        ext.insert(ext.end(), P.ext.begin(), P.ext.end());
        long long first = 0;
        for (int w = 0; w < nt / 32; ++w) {
            long long nf = 0, nb = 0;
            for (const Op& o : P.fwd[w]) nf += kBatch * o.batches();
            for (const Op& o : P.bwd[w]) nb += kBatch * o.batches();
            warps.push_back({fits32(first), fits32(nf), fits32(nb), 0});
            stream.push_back({(int)c, w, at});
            first += nf + nb;
            at += (nf + nb) * (kLine / 4);
        }
        coef += P.coef;
    }
    stream.push_back({-1, 0, at});
    // Groups, the longest first (their order does not affect results).
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
                G.top = members[c][m].top;
                for (int i = 0; i < cnt; ++i) off.push_back(members[c][m + i].off);
                groups.push_back(G);
            }
    upd_len = std::max<long long>(upd_len, 2);
    return true;
}

// Copies run past a stream's end: the last one's into padding.
long long ResidentSchedule::total() const { return stream.back().at + (long long)depth_of(1) * kBatchBytes / 4; }

void ResidentSchedule::write(size_t i, float* dst) const {
    if (stream[i].c < 0) {
        std::memset(dst, 0, (size_t)(total() - stream[i].at) * 4);
        return;
    }
    const ClassPlan& P = cp[stream[i].c];
    const SnFactor& F = *(*shape)[stream[i].c].F;
    uint32_t* out = reinterpret_cast<uint32_t*>(dst);
    for (const Op& o : P.fwd[stream[i].w]) out = emit(o, F, P, out);
    for (const Op& o : P.bwd[stream[i].w]) out = emit(o, F, P, out);
}

double tree_weight(const SnFactor& F) {
    double w = 0;
    for (size_t j = 0; j < F.col0.size(); ++j) w += front_weight(F, j);
    return w;
}

double cut_weight(double total) { return std::min(kCutMax, std::max(kCutMin, total / kCutShare)); }

bool resident_plan(const std::vector<const SnFactor*>& factors, double total) {
    int max_n = 0;
    double largest = 0;
    for (const SnFactor* F : factors) {
        max_n = std::max(max_n, F->n);
        largest = std::max(largest, tree_weight(*F));
    }
    if (max_n == 0 || ResidentPlan::smem_bytes(max_n + kPartMax, 1, 512) > ResidentPlan::kMaxSmem) return false;
    return largest <= kCutCost + total / kCutRate;
}

FactorCut cut_trees(const SnFactor& F, double cap) {
    const int ns = (int)F.col0.size();
    FactorCut C;
    C.low.assign(ns, 0);
    C.upd.assign(ns, -1);
    std::vector<double> weight(ns);
    std::vector<int> size(ns, 1), len(ns);
    for (int j = 0; j < ns; ++j) {
        weight[j] += front_weight(F, j);
        len[j] += F.ncol[j];
        if (F.parent[j] >= 0) {
            weight[F.parent[j]] += weight[j];
            size[F.parent[j]] += size[j];
            len[F.parent[j]] += len[j];
        }
    }
    auto fits = [&](int j) { return weight[j] <= cap && (len[j] + (int)F.rows[j].size()) <= kCutLen; };
    double w = 0;
    int n = 0;
    std::vector<char> root(ns, 0);
    for (int j = 0; j < ns; ++j) {
        if (!fits(j) || (F.parent[j] >= 0 && fits(F.parent[j]))) continue;
        const int vec = len[j] + (int)F.rows[j].size();
        if (C.shapes.empty() || w + weight[j] > cap || n + vec > kCutLen) {
            C.shapes.emplace_back();
            C.shapes.back().F = &F;
            w = 0;
            n = 0;
        }
        w += weight[j];
        n += vec;
        C.shapes.back().trees.push_back({j - size[j] + 1, j, -1});
        root[j] = 1;
        for (int i = j - size[j] + 1; i <= j; ++i) C.low[i] = 1;
    }
    for (int j = 0; j < ns; ++j) {
        if (C.low[j] && !root[j]) continue;
        if (C.upd_len >= (long long)INT32_MAX)
            throw Error(HDD_ERR_UNSUPPORTED, "update vectors too large for 32-bit indices");
        C.upd[j] = (int)C.upd_len;
        C.upd_len += (long long)F.rows[j].size();
    }
    for (ResidentPlan::Shape& S : C.shapes)
        for (ResidentPlan::Tree& T : S.trees)
            if (!F.rows[T.last].empty()) T.top = C.upd[T.last];
    return C;
}

}  // namespace hdd
