// Test shim: the product's host-side setup code (layout, interface assembly,
// supernodal Cholesky) compiled without CUDA device code, so the CPU test suite
// can check it against the oracle.  Built by tests/test_cpu_host.py with g++.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <limits>
#include <map>
#include <random>
#include <string>
#include <vector>

#include "host_setup.h"
#include "sn_streams.h"

using namespace hdd;

namespace {
struct Shim {
    DomainLayout L;
    InterfaceHost ih;
    std::string err;
};
const CsrF* pick(Shim* s, int kind, int level, int sub) {
    if (level < 0 || level >= s->ih.M) return nullptr;
    switch (kind) {
        case 0: return &s->ih.Arr[level];
        case 1: return (sub >= 0 && sub < s->ih.n_sub) ? &s->ih.Aii[level][sub] : nullptr;
        case 2: return (sub >= 0 && sub < s->ih.n_sub) ? &s->ih.Air[level][sub] : nullptr;
        case 3: return level < (int)s->ih.Prr.size() ? &s->ih.Prr[level] : nullptr;
        default: return nullptr;
    }
}

// Walks a schedule of one CTA per tree the way sn_resident.cu runs it, one warp
// after another between two barriers, with every index checked.  The CTA's
// array M starts as NaN (what another system may have left there).
struct StreamWalk {
    const ResidentSchedule& S;
    std::vector<float> words;      // the streams
    long long oob = 0, races = 0;  // accesses out of range; of entries another warp uses in the same phase
    long long ops = 0, barriers = 0;
    explicit StreamWalk(const ResidentSchedule& s) : S(s), words((size_t)s.total()) {
        for (size_t i = 0; i < S.streams(); ++i) S.write(i, words.data() + S.at(i));
    }
    int word(long long line, int i) const {
        int v;
        std::memcpy(&v, &words.at((size_t)(line * (kLine / 4) + i)), 4);
        return v;
    }
    // Entries of M (or update slots in global memory) with their last users.
    struct Memory {
        std::vector<double> v;
        std::vector<int> wp, ww, rp, rw;  // phase and warp of the last write / read (warp -2: several)
        int free_entry = -1;              // results of no row: written by anyone, read by nobody
        StreamWalk* walk = nullptr;
        double dummy = 0;
        void init(StreamWalk* s, long long n) {
            walk = s;
            v.assign((size_t)n, std::numeric_limits<double>::quiet_NaN());
            wp.assign((size_t)n, -1); ww.assign((size_t)n, -1); rp.assign((size_t)n, -1); rw.assign((size_t)n, -1);
        }
        double read(long long i, int warp, int phase) {
            if (i < 0 || i >= (long long)v.size() || i == free_entry) { ++walk->oob; return 0; }
            if (wp[i] == phase && ww[i] != warp) ++walk->races;
            rw[i] = rp[i] == phase && rw[i] != warp ? -2 : warp;
            rp[i] = phase;
            return v[i];
        }
        void write(long long i, double x, int warp, int phase) {
            if (i < 0 || i >= (long long)v.size()) { ++walk->oob; return; }
            if (i == free_entry) return;
            if ((wp[i] == phase && ww[i] != warp) || (rp[i] == phase && rw[i] != warp)) ++walk->races;
            wp[i] = phase;
            ww[i] = warp;
            v[i] = x;
        }
    };
    // mode: 0 whole trees, 1 / 2 the forward / backward half of cut ones.
    void run(int mode, const float* b, float* x, std::vector<double>& y, std::vector<double>& top_upd,
             const std::vector<double>& top_x) {
        const int nw = S.nt / 32;
        for (const RGroup& G : S.groups)
            for (int k = 0; k < G.count; ++k) {  // members side by side never meet
                const int off = S.off.at(G.member0 + k);
                const int zero = G.n + G.next;
                Memory M, U;
                M.init(this, S.entries);
                M.free_entry = zero + 1;
                U.init(this, S.global_slots ? 65536 : 0);
                auto at = [&](long long i, int w, int p) { return M.read(i, w, p); };
                auto slot = [&](long long i, int w, int p) { return S.global_slots ? U.read(i, w, p) : M.read(i, w, p); };
                auto put = [&](int d, double v, int flags, int w, int p) {
                    if (d >= 0) {
                        if (d == zero) ++oob;
                        M.write(d, v, w, p);
                    } else if (S.global_slots) {
                        if (d == -1) ++oob;  // the zero slot
                        U.write(-1 - d, v, w, p);
                    } else if ((flags & kTopRoot) && mode == 1 && G.top - 1 - d < (int)top_upd.size()) {
                        top_upd[G.top - 1 - d] = v;
                    } else {
                        ++oob;
                    }
                };
                auto assemble = [&](const int it[4], int w, int p) {
                    const double s = slot(it[1], w, p) + slot(it[2], w, p);
                    if (it[3] && S.global_slots) U.write(it[0], U.read(it[0], w, p) + s, w, p);
                    else M.write(it[0], at(it[0], w, p) + s, w, p);
                };
                int phase = 0;
                M.write(zero, 0.0, -1, phase);
                if (S.global_slots) U.write(0, 0.0, -1, phase);
                for (int i = 0; i < G.n; ++i)
                    M.write(i, mode == 2 ? y.at(G.y + i) : (double)b[off + S.perm.at(G.perm + i)], -1, phase);
                if (mode == 2)
                    for (int i = 0; i < G.next; ++i) M.write(G.n + i, top_x.at(off + S.ext.at(G.ext + i)), -1, phase);
                for (int pass = mode == 2 ? 1 : 0; pass < (mode == 1 ? 1 : 2); ++pass) {
                    ++phase;
                    std::vector<long long> pos(nw), lim(nw);
                    std::vector<int> owed(nw, 0);  // barriers a warp has still to take
                    for (int w = 0; w < nw; ++w) {
                        const RWarp W = S.warps.at(G.warps + w);
                        pos[w] = G.stream / kLine + W.first + (pass ? W.nf : 0);
                        lim[w] = pos[w] + (pass ? W.nb : W.nf);
                        // Copies run ahead by the ring's depth.
                        if ((lim[w] + (long long)kBatch * depth_of(S.km)) * kLine > (long long)words.size() * 4) ++oob;
                    }
                    for (int ended = 0; ended < nw; ++phase) {
                        ended = 0;
                        int waiting = 0;
                        for (int w = 0; w < nw; ++w) {
                            if (owed[w] > 0) { --owed[w]; ++waiting; continue; }
                            for (;;) {
                                if (pos[w] >= lim[w]) { ++oob; ++ended; break; }
                                const long long h = pos[w];
                                const int type = word(h, 0) & 15;
                                if (type == kEnd) {
                                    if (h + kBatch != lim[w]) ++oob;
                                    ++ended;
                                    break;
                                }
                                ++ops;
                                pos[w] = operation(h, w, phase, M, at, slot, put, assemble);
                                owed[w] = (int)((uint32_t)word(h, 1) >> 20);
                                if (owed[w] > 0) { --owed[w]; ++waiting; break; }
                            }
                        }
                        if (waiting > 0 && ended > 0) { ++oob; break; }  // warps at different barriers
                        if (waiting > 0) ++barriers;
                    }
                }
                if (mode == 1)
                    for (int i = 0; i < G.n; ++i) y.at(G.y + i) = M.v[i];
                else
                    for (int i = 0; i < G.n; ++i) x[off + S.perm.at(G.perm + i)] = (float)M.v[i];
            }
    }
    // One operation from line h on; returns the line behind it.
    template <class At, class Slot, class Put, class Assemble>
    long long operation(long long h, int w, int p, Memory& M, At at, Slot slot, Put put, Assemble assemble) {
        const int type = word(h, 0) & 15, lmq = (word(h, 0) >> 4) & 15, flags = (word(h, 0) >> 8) & 255;
        const int count = word(h, 0) >> 16;
        auto item = [&](long long line, int l, int it[4]) {
            for (int q = 0; q < 4; ++q) it[q] = word(line, 4 * l + q);
            return it[0] >= 0;
        };
        int it[4];
        if (type == kAssemble || type == kFinish) {
            for (int q = 1; q <= count; ++q)
                for (int l = 0; l < 32; ++l) {
                    if (!item(h + q, l, it)) continue;
                    if (type == kAssemble) { assemble(it, w, p); continue; }
                    double t = at(it[0], w, p);
                    for (int s = 1; s < (word(h, 1) & 0xffff); ++s) t += at(it[0] + s * word(h, 2), w, p);
                    put(it[1], (slot(it[2], w, p) + slot(it[3], w, p)) + t, flags, w, p);
                }
            return h + kBatch;
        }
        if (type != kProduct) {
            if (type != kNothing) ++oob;
            return h + kBatch;
        }
        const int mq = 1 << lmq;
        const bool tr = (flags & kTransposed) != 0;
        if (flags & kItem)
            for (int l = 0; l < 32; ++l)
                if (item(h + 3, l, it)) assemble(it, w, p);
        auto half = [](int v, int q) { return q ? (int)((uint32_t)v >> 16) : v & 0xffff; };
        std::vector<double> acc(128, 0.0);
        long long pos = h + kBatch, ix = h + 2;
        for (int g = 0; g < count; ++g) {
            if (tr && g >= 4 && (g - 4) % 8 == 0) { ix = pos; pos += kBatch; }
            const int s0 = 4 * (g < 4 ? g : (g - 4) % 8);
            for (int u = 0; u < 4; ++u, ++pos)
                for (int l = 0; l < 32; ++l) {
                    int j;
                    if (tr) j = half(word(ix + (s0 + u) / 8, 4 * l + (s0 + u) % 8 / 2), u % 2);
                    else if (g + 1 == count) j = half(word(h, 4 * l + 2 + u / 2), u % 2);
                    else j = half(word(h, 4 * l + 1), 0) + (4 * g + u) * (half(word(h, 4 * l + 1), 1) & 15);
                    const double in = at(j, w, p);
                    for (int e = 0; e < 4; ++e)
                        acc[4 * l + e] = std::fma((double)words.at((size_t)(pos * (kLine / 4) + 4 * l + e)), in, acc[4 * l + e]);
                }
        }
        for (int o = 4; o < 32; o <<= 1)
            if (mq <= o) {
                const std::vector<double> a = acc;
                for (int l = 0; l < 32; ++l)
                    for (int e = 0; e < 4; ++e) acc[4 * l + e] = a[4 * l + e] + a[4 * (l ^ o) + e];
            }
        for (int l = 0; l < mq; ++l)
            for (int e = 0; e < 4; ++e) {
                double v = acc[4 * l + e];
                if (flags & kPairs) {
                    const int a = word(h + 2, 4 * l + e);
                    v = (slot(half(a, 0), w, p) + slot(half(a, 1), w, p)) + v;
                }
                put(word(h + 1, 4 * l + e), v, flags, w, p);
            }
        return pos;
    }
};

// The factors of one interface solve with their offsets, as the sigma solver
// passes them to a plan (subdomains with equal systems share a factor).
void plan_factors(const InterfaceHost& ih, int kind, int level, std::vector<SnFactor>& store,
                  std::vector<const SnFactor*>& fs, std::vector<int>& offs) {
    PlanHost ph;
    interface_solve_plan(ih, kind, level, store, ph);
    if (kind == 0) {
        fs.push_back(&store[0]);
        offs.push_back(0);
        return;
    }
    const std::vector<int> rep = interior_classes(ih, level);
    int off = 0;
    for (int sd = 0; sd < ih.n_sub; ++sd) {
        const int n = ih.Aii[level][sd].rows;
        if (n > 0) { fs.push_back(&store[rep[sd]]); offs.push_back(off); }
        off += n;
    }
}
}  // namespace

extern "C" {

// Layout and interface system of a dense flag array; NULL on error (message in err).
void* shim_build(const int size[3], const int sub[3], int vlevels, int sigma_levels, const uint32_t* flags,
                 char* err, int errlen) {
    Shim* s = new Shim();
    try {
        Options o;
        for (int a = 0; a < 3; ++a) { o.size[a] = size[a]; o.sub[a] = sub[a]; }
        o.vlevels = vlevels;
        o.nvcycles = 1;
        o.interior = o.boundary = 1;
        o.sigma_levels = sigma_levels;
        o.sigma_smoothing = 3;
        o.sigma_mg = 1;
        build_layout(o, flags, s->L);
        build_interface(s->L, sigma_levels, s->ih);
        return s;
    } catch (const std::exception& e) {
        if (err && errlen > 0) { std::strncpy(err, e.what(), errlen - 1); err[errlen - 1] = 0; }
        delete s;
        return nullptr;
    }
}

// The product's two-level second-level interface system: every first-level
// subdomain's system (first-level planes made Dirichlet, boxes of sub/2),
// stacked block-diagonally.  NULL on error.
void* shim_build_second_level(const int size[3], const int sub[3], int sigma_levels, const uint32_t* flags,
                              char* err, int errlen) {
    Shim* s = new Shim();
    try {
        for (int a = 0; a < 3; ++a) { s->L.opt.size[a] = size[a]; s->L.opt.sub[a] = sub[a]; }
        s->L.opt.sigma_levels = sigma_levels;
        s->L.flags_in.assign(flags, flags + (size_t)size[0] * size[1] * size[2]);
        build_second_level(s->L, sub, sigma_levels, s->ih);
        return s;
    } catch (const std::exception& e) {
        if (err && errlen > 0) { std::strncpy(err, e.what(), errlen - 1); err[errlen - 1] = 0; }
        delete s;
        return nullptr;
    }
}

// 1 when the layout runs the whole-grid V-cycle (coarse levels couple boxes).
int shim_global_vcycle(void* h) { return static_cast<Shim*>(h)->L.global_vcycle ? 1 : 0; }

// Interface DOF count of a level.
int shim_num_interface(void* h, int level) {
    const InterfaceHost& ih = static_cast<Shim*>(h)->ih;
    return level >= 0 && level < (int)ih.n_iface.size() ? ih.n_iface[level] : -1;
}

void shim_free(void* h) { delete static_cast<Shim*>(h); }

// Factors a matrix of ncomp disconnected path graphs of csize vertices each
// (diagonal 2.5, off-diagonal -1, interleaved so that every component's
// vertices are spread through the numbering) and returns the relative
// residual of one solve; -1 on an exception.  Interface systems of sparse
// domains fall apart into many such pieces.
double shim_factor_components(int ncomp, int csize) {
    try {
        const int n = ncomp * csize;
        CsrF A;
        A.rows = A.cols = n;
        A.ptr.assign(1, 0);
        auto id = [&](int c, int k) { return k * ncomp + c; };  // component c, position k
        std::vector<int> comp_of(n), pos_of(n);
        for (int c = 0; c < ncomp; ++c)
            for (int k = 0; k < csize; ++k) { comp_of[id(c, k)] = c; pos_of[id(c, k)] = k; }
        for (int r = 0; r < n; ++r) {
            const int c = comp_of[r], k = pos_of[r];
            std::vector<std::pair<int, float>> e = {{r, 2.5f}};
            if (k > 0) e.push_back({id(c, k - 1), -1.0f});
            if (k + 1 < csize) e.push_back({id(c, k + 1), -1.0f});
            std::sort(e.begin(), e.end());
            for (auto& t : e) { A.col.push_back(t.first); A.val.push_back(t.second); }
            A.ptr.push_back((int)A.col.size());
        }
        SnFactor F;
        F.analyze(A, nullptr);
        F.factor(A, 1e-5);
        std::vector<double> b(n), x(n);
        for (int i = 0; i < n; ++i) b[i] = std::sin(0.37 * i);
        x = b;
        F.solve(x.data());
        double rn = 0, bn = 0;
        for (int r = 0; r < n; ++r) {
            double ax = 1e-5 * x[r];
            for (int p = A.ptr[r]; p < A.ptr[r + 1]; ++p) ax += (double)A.val[p] * x[A.col[p]];
            rn += (ax - b[r]) * (ax - b[r]);
            bn += b[r] * b[r];
        }
        return std::sqrt(rn / bn);
    } catch (const std::exception&) {
        return -1.0;
    }
}

// FNV-1a digest of everything the GPU plans are built from: the interface
// matrices of every level and subdomain, and the solve blocks and L_RJ of the
// level-0 Arr factorisation and of every level-0 Aii factorisation.  Used to
// check that the host setup gives the same bits for any number of threads.
unsigned long long shim_setup_digest(void* h) {
    Shim* s = static_cast<Shim*>(h);
    unsigned long long d = 1469598103934665603ull;
    auto mix = [&](const void* p, size_t n) {
        const unsigned char* b = static_cast<const unsigned char*>(p);
        for (size_t i = 0; i < n; ++i) d = (d ^ b[i]) * 1099511628211ull;
    };
    auto csr = [&](const CsrF& A) {
        mix(A.ptr.data(), A.ptr.size() * sizeof(int));
        mix(A.col.data(), A.col.size() * sizeof(int));
        mix(A.val.data(), A.val.size() * sizeof(float));
    };
    auto factor = [&](const CsrF& A, const std::vector<std::array<int, 3>>* xyz) {
        if (A.rows == 0) return;
        SnFactor F;
        F.analyze(A, xyz);
        F.factor(A, 1e-5);
        F.build_solve_blocks();
        mix(F.perm.data(), F.perm.size() * sizeof(int));
        for (const auto& v : F.Fw) mix(v.data(), v.size() * sizeof(double));
        for (const auto& v : F.Lrj) mix(v.data(), v.size() * sizeof(double));
    };
    const InterfaceHost& ih = s->ih;
    for (int l = 0; l < ih.M; ++l) {
        csr(ih.Arr[l]);
        if (l < (int)ih.Prr.size()) csr(ih.Prr[l]);
        for (int sd = 0; sd < ih.n_sub; ++sd) { csr(ih.Aii[l][sd]); csr(ih.Air[l][sd]); }
    }
    factor(ih.Arr[0], &ih.iface_xyz[0]);
    for (int sd = 0; sd < ih.n_sub; ++sd) factor(ih.Aii[0][sd], &ih.aii_xyz[0][sd]);
    return d;
}

// SPGrid page scatter / gather (hdd_set_domain_pages); 0 or the hdd_status.
int shim_pages_to_dense(const int size[3], long long n, const int32_t* origin, const uint32_t* flags,
                        const float* vals, uint32_t* dflags, float* dvals, char* err, int errlen) {
    try {
        pages_to_dense(size, n, origin, flags, dflags);
        pages_to_dense(size, n, origin, vals, dvals);
        return 0;
    } catch (const Error& e) {
        if (err && errlen > 0) { std::strncpy(err, e.what(), errlen - 1); err[errlen - 1] = 0; }
        return (int)e.status;
    }
}

int shim_dense_to_pages(const int size[3], long long n, const int32_t* origin, const float* dense, float* vals) {
    try {
        dense_to_pages(size, n, origin, dense, vals);
        return 0;
    } catch (const Error& e) {
        return (int)e.status;
    }
}

// Interface dump / reload (the reference's -iomode): 0 on success, else the
// hdd_status with its message in err.
int shim_write_interface(void* h, const char* dir, char* err, int errlen) {
    try {
        write_interface_dir(static_cast<Shim*>(h)->ih, dir);
        return 0;
    } catch (const Error& e) {
        if (err && errlen > 0) { std::strncpy(err, e.what(), errlen - 1); err[errlen - 1] = 0; }
        return (int)e.status;
    }
}

// A handle holding only a reloaded interface system (NULL on error).
void* shim_read_interface(const char* dir, char* err, int errlen) {
    Shim* s = new Shim();
    try {
        read_interface_dir(dir, s->ih);
        return s;
    } catch (const Error& e) {
        if (err && errlen > 0) { std::strncpy(err, e.what(), errlen - 1); err[errlen - 1] = 0; }
        delete s;
        return nullptr;
    }
}

// Checks the interface system of `sys` against the layout of `dom`.
int shim_check_interface(void* dom, void* sys, int sigma_levels, char* err, int errlen) {
    try {
        check_interface(static_cast<Shim*>(dom)->L, sigma_levels, static_cast<Shim*>(sys)->ih);
        return 0;
    } catch (const Error& e) {
        if (err && errlen > 0) { std::strncpy(err, e.what(), errlen - 1); err[errlen - 1] = 0; }
        return (int)e.status;
    }
}

// Interface DOF positions of level l: n entries (3 ints each) into out when
// out != NULL; sub < 0 selects the interface, else that subdomain's interior.
long long shim_positions(void* h, int l, int sub, int* out) {
    const InterfaceHost& ih = static_cast<Shim*>(h)->ih;
    if (l < 0 || l >= (int)ih.iface_xyz.size()) return -1;
    const std::vector<std::array<int, 3>>& p =
        sub < 0 ? ih.iface_xyz[l] : (sub < (int)ih.aii_xyz[l].size() ? ih.aii_xyz[l][sub] : ih.iface_xyz[l]);
    if (out)
        for (size_t i = 0; i < p.size(); ++i)
            for (int a = 0; a < 3; ++a) out[3 * i + a] = p[i][a];
    return (long long)p.size();
}

// Level-0 interface map: n cells into out (3 ints each) when out != NULL.
long long shim_interface_map(void* h, int* out) {
    const InterfaceHost& ih = static_cast<Shim*>(h)->ih;
    if (out)
        for (size_t i = 0; i < ih.iface_map.size(); ++i)
            for (int a = 0; a < 3; ++a) out[3 * i + a] = ih.iface_map[i][a];
    return (long long)ih.iface_map.size();
}

int shim_num_subdomains(void* h) { return static_cast<Shim*>(h)->ih.n_sub; }

// kind: 0 Arr, 1 Aii, 2 Air, 3 Prr.  shape = {rows, cols, nnz}; returns 0 on success.
int shim_matrix_shape(void* h, int kind, int level, int sub, int* shape) {
    const CsrF* m = pick(static_cast<Shim*>(h), kind, level, sub);
    if (!m) return 1;
    shape[0] = m->rows;
    shape[1] = m->cols;
    shape[2] = (int)m->col.size();
    return 0;
}

int shim_matrix_get(void* h, int kind, int level, int sub, int* ptr, int* col, double* val) {
    const CsrF* m = pick(static_cast<Shim*>(h), kind, level, sub);
    if (!m) return 1;
    for (size_t i = 0; i < m->ptr.size(); ++i) ptr[i] = m->ptr[i];
    for (size_t i = 0; i < m->col.size(); ++i) { col[i] = m->col[i]; val[i] = m->val[i]; }
    return 0;
}

// rep[i]: the first subdomain whose interior system of the level equals i's.
void shim_interior_classes(void* h, int level, int* rep) {
    const std::vector<int> r = interior_classes(static_cast<Shim*>(h)->ih, level);
    for (size_t i = 0; i < r.size(); ++i) rep[i] = r[i];
}

// Factor (A + 1e-5 I) of one matrix with the supernodal Cholesky (geometric
// ordering when positions exist), solve for a random right-hand side on the
// host and return ||(A + 1e-5 I) x - b|| / ||b||; also checks that the explicit
// solve blocks reproduce the same solution (returned in *blocks_diff).
double shim_factor_check(void* h, int kind, int level, int sub, double* blocks_diff) {
    Shim* s = static_cast<Shim*>(h);
    const CsrF* m = pick(s, kind, level, sub);
    if (!m || (kind != 0 && kind != 1) || m->rows == 0) return -1.0;
    const std::vector<std::array<int, 3>>* xyz = nullptr;
    if (kind == 0 && level < (int)s->ih.iface_xyz.size() && (int)s->ih.iface_xyz[level].size() == m->rows)
        xyz = &s->ih.iface_xyz[level];
    if (kind == 1 && (int)s->ih.aii_xyz[level][sub].size() == m->rows) xyz = &s->ih.aii_xyz[level][sub];
    const double eps = 1e-5;
    SnFactor F;
    F.analyze(*m, xyz);
    F.factor(*m, eps);
    F.build_solve_blocks();
    const int n = m->rows;
    std::mt19937 rng(7);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::vector<double> b(n), x(n);
    for (int i = 0; i < n; ++i) b[i] = U(rng);
    x = b;
    F.solve(x.data());
    double rn = 0, bn = 0;
    for (int r = 0; r < n; ++r) {
        double ax = eps * x[r];
        for (int p = m->ptr[r]; p < m->ptr[r + 1]; ++p) ax += (double)m->val[p] * x[m->col[p]];
        rn += (ax - b[r]) * (ax - b[r]);
        bn += b[r] * b[r];
    }
    // Same solve through the explicit blocks Fw = [Linv; -W] the GPU uses:
    // forward [y; v] = Fw f + [0; f_R], backward x_J = Fw^T [y; x_R].
    std::vector<double> f(n), y(n, 0.0), xn(n, 0.0);
    for (int i = 0; i < n; ++i) f[i] = b[F.perm[i]];
    const int ns = (int)F.col0.size();
    std::vector<std::vector<double>> upd(ns);
    std::vector<std::vector<int>> kids(ns);
    for (int j = 0; j < ns; ++j)
        if (F.parent[j] >= 0) kids[F.parent[j]].push_back(j);
    std::vector<int> pos(n, -1);
    for (int j = 0; j < ns; ++j) {
        const int nj = F.ncol[j], nr = (int)F.rows[j].size(), mm = nj + nr;
        std::vector<double> v(mm, 0.0);
        for (int a = 0; a < nj; ++a) { v[a] = f[F.col0[j] + a]; pos[F.col0[j] + a] = a; }
        for (int k = 0; k < nr; ++k) pos[F.rows[j][k]] = nj + k;
        for (int c : kids[j])
            for (size_t k = 0; k < F.rows[c].size(); ++k) v[pos[F.rows[c][k]]] += upd[c][k];
        const BlockVec& W = F.Fw[j];
        for (int r = 0; r < mm; ++r) {
            double acc = 0;
            for (int c = 0; c < nj; ++c) acc += W[(size_t)c * mm + r] * v[c];
            if (r < nj) y[F.col0[j] + r] = acc;
            else upd[j].push_back(v[r] + acc);
        }
    }
    for (int j = ns - 1; j >= 0; --j) {
        const int nj = F.ncol[j], nr = (int)F.rows[j].size(), mm = nj + nr;
        const BlockVec& W = F.Fw[j];
        for (int a = 0; a < nj; ++a) {
            double acc = 0;
            for (int r = 0; r < mm; ++r) {
                const double g = r < nj ? y[F.col0[j] + r] : xn[F.rows[j][r - nj]];
                acc += W[(size_t)a * mm + r] * g;
            }
            xn[F.col0[j] + a] = acc;
        }
    }
    double d = 0, xm = 0;
    for (int i = 0; i < n; ++i) {
        d = std::max(d, std::fabs(xn[i] - x[F.perm[i]]));
        xm = std::max(xm, std::fabs(x[F.perm[i]]));
    }
    *blocks_diff = xm > 0 ? d / xm : d;
    return std::sqrt(rn / bn);
}

// The supernodal solve plan of one interface solve (kind 0: Arr of level l;
// 1: Aii of all subdomains, concatenated), built as the sigma solver builds
// it and solved on the host front by front with the device kernels'
// arithmetic (PlanHost::emulate): x = plan solve of b.  Returns 0, or 1 on an
// exception.
int shim_plan_emulate(void* h, int kind, int level, const float* b, float* x) {
    Shim* s = static_cast<Shim*>(h);
    try {
        if (level < 0 || level >= s->ih.M || (kind != 0 && kind != 1)) return 1;
        std::vector<SnFactor> fs;
        PlanHost plan;
        interface_solve_plan(s->ih, kind, level, fs, plan);
        plan.emulate(b, x);
        return 0;
    } catch (const std::exception&) {
        return 1;
    }
}

// The same solve through the schedule the device runs (sn_streams.h): whole
// trees, or the lower trees of every factor with the fronts above them solved
// front by front.  info: {1 whole / 0 cut, trees per CTA, threads per CTA, 1 when
// update slots are in global memory, CTAs, fronts above, accesses out of range,
// races between warps, operations, barriers, streams of trees (members with the
// same factor share one)}; *bytes: of the streams, *coef: the
// distinct coefficients' of both directions.  Returns 0, or 1 on an exception.
int shim_stream_walk(void* h, int kind, int level, const float* b, float* x, int* info, double* bytes, double* coef) {
    try {
        const InterfaceHost& ih = static_cast<Shim*>(h)->ih;
        if (level < 0 || level >= ih.M || (kind != 0 && kind != 1)) return 1;
        std::vector<SnFactor> store;
        std::vector<const SnFactor*> fs;
        std::vector<int> offs;
        plan_factors(ih, kind, level, store, fs, offs);
        double total = 0;
        for (const SnFactor* F : fs) total += tree_weight(*F);
        std::vector<ResidentPlan::Shape> shapes;
        std::vector<std::vector<ResidentPlan::Member>> members;
        std::vector<double> y, upd, sol;
        ResidentSchedule S;
        constexpr int kSMs = 148;
        bool whole = resident_plan(fs, total);
        if (whole) {
            whole_shapes(fs, offs, shapes, members);
            whole = S.plan(shapes, members, false, kSMs);
        }
        int ntop = 0;
        std::vector<long long> counts(4, 0);
        auto done = [&](const StreamWalk& W) {
            const int v[11] = {whole ? 1 : 0, S.km, S.nt, S.global_slots ? 1 : 0, (int)S.groups.size(), ntop,
                               (int)W.oob, (int)W.races, (int)W.ops, (int)W.barriers, (int)shapes.size()};
            std::copy(v, v + 11, info);
            *bytes = 4.0 * S.total();
            *coef = 8.0 * S.coef;
        };
        if (whole) {
            StreamWalk W(S);
            W.run(0, b, x, y, upd, sol);
            done(W);
            return 0;
        }
        // Update vectors of the fronts above and of the trees' roots, factor by factor.
        std::map<const SnFactor*, FactorCut> cuts;
        std::map<const SnFactor*, size_t> shape0;
        std::vector<long long> first;
        for (size_t f = 0; f < fs.size(); ++f) {
            const auto c = cuts.emplace(fs[f], FactorCut());
            FactorCut& C = c.first->second;
            if (c.second) {
                C = cut_trees(*fs[f], cut_weight(total));
                shape0[fs[f]] = shapes.size();
                shapes.insert(shapes.end(), C.shapes.begin(), C.shapes.end());
                members.resize(shapes.size());
            }
            first.push_back((long long)upd.size());
            for (size_t i = 0; i < C.shapes.size(); ++i) members[shape0[fs[f]] + i].push_back({offs[f], (int)upd.size()});
            upd.resize(upd.size() + (size_t)C.upd_len, std::numeric_limits<double>::quiet_NaN());
        }
        S = ResidentSchedule();
        if (!S.plan(shapes, members, true, kSMs)) return 1;
        StreamWalk W(S);
        y.assign((size_t)S.y_len, 0.0);
        W.run(1, b, x, y, upd, sol);
        int n = 0;
        for (size_t f = 0; f < fs.size(); ++f) n = std::max(n, offs[f] + fs[f]->n);
        sol.assign(n, 0.0);
        for (size_t f = 0; f < fs.size(); ++f) {
            const SnFactor& F = *fs[f];
            const FactorCut& C = cuts.at(fs[f]);
            const int ns = (int)F.col0.size();
            std::vector<std::vector<int>> kids(ns);
            for (int j = 0; j < ns; ++j)
                if (F.parent[j] >= 0) kids[F.parent[j]].push_back(j);
            std::vector<std::vector<double>> yv(ns);
            for (int j = 0; j < ns; ++j) {
                if (C.low[j]) continue;
                ++ntop;
                const int nj = F.ncol[j], nr = (int)F.rows[j].size(), m = nj + nr;
                std::vector<double> v(m, 0.0);
                for (int a = 0; a < nj; ++a) v[a] = b[offs[f] + F.perm[F.col0[j] + a]];
                for (int c : kids[j])
                    for (size_t q = 0; q < F.rows[c].size(); ++q) {
                        const int r = F.rows[c][q];
                        const int i = r < F.col0[j] + nj ? r - F.col0[j]
                                                         : nj + (int)(std::lower_bound(F.rows[j].begin(), F.rows[j].end(), r) -
                                                                      F.rows[j].begin());
                        v[i] += upd.at(first[f] + C.upd[c] + q);
                    }
                for (int r = 0; r < m; ++r) {
                    double s = 0;
                    for (int c = 0; c < nj; ++c) s += (double)(float)F.Fw[j][(size_t)c * m + r] * v[c];
                    if (r < nj) yv[j].push_back(s);
                    else upd.at(first[f] + C.upd[j] + r - nj) = v[r] + s;
                }
            }
            for (int j = ns - 1; j >= 0; --j) {
                if (C.low[j]) continue;
                const int nj = F.ncol[j], m = nj + (int)F.rows[j].size();
                for (int a = 0; a < nj; ++a) {
                    double s = 0;
                    for (int r = 0; r < m; ++r)
                        s += (double)(float)F.Fw[j][(size_t)a * m + r] *
                             (r < nj ? yv[j][r] : sol[offs[f] + F.rows[j][r - nj]]);
                    sol[offs[f] + F.col0[j] + a] = s;
                    x[offs[f] + F.perm[F.col0[j] + a]] = (float)s;
                }
            }
        }
        W.run(2, b, x, y, upd, sol);
        done(W);
        return 0;
    } catch (const std::exception&) {
        return 1;
    }
}

// A forest of ntree trees of two fronts of one column each (child to parent
// -0.5), the same for `members` factors of one class: its schedule, walked.
// info as in shim_stream_walk; returns the largest error of the solution, which
// is known in closed form, or -1 on an exception.
double shim_forest_walk(int ntree, int members, int* info) {
    try {
        SnFactor F;
        F.n = 2 * ntree;
        for (int t = 0; t < ntree; ++t) {
            F.perm.push_back(2 * t);
            F.perm.push_back(2 * t + 1);
            F.col0.push_back(2 * t);
            F.col0.push_back(2 * t + 1);
            F.ncol.insert(F.ncol.end(), {1, 1});
            F.parent.insert(F.parent.end(), {2 * t + 1, -1});
            F.rows.push_back({2 * t + 1});
            F.rows.push_back({});
            for (std::initializer_list<double> w : {std::initializer_list<double>{1.0, -0.5}, {1.0}}) {
                F.Fw.emplace_back(w.size());
                std::copy(w.begin(), w.end(), F.Fw.back().data());
            }
        }
        std::vector<const SnFactor*> fs(members, &F);
        std::vector<int> offs;
        for (int m = 0; m < members; ++m) offs.push_back(m * F.n);
        std::vector<ResidentPlan::Shape> shapes;
        std::vector<std::vector<ResidentPlan::Member>> mem;
        whole_shapes(fs, offs, shapes, mem);
        ResidentSchedule S;
        if (!S.plan(shapes, mem, false, 148)) return -1.0;
        std::vector<float> b((size_t)members * F.n), x(b.size(), 0.0f);
        for (size_t i = 0; i < b.size(); ++i) b[i] = std::sin(0.37 * i);
        std::vector<double> none;
        StreamWalk W(S);
        W.run(0, b.data(), x.data(), none, none, none);
        const int v[10] = {1, S.km, S.nt, S.global_slots ? 1 : 0, (int)S.groups.size(), 0, (int)W.oob, (int)W.races,
                           (int)W.ops, (int)W.barriers};
        std::copy(v, v + 10, info);
        double e = 0;
        for (size_t i = 0; i < b.size(); i += 2) {
            const double root = b[i + 1] - 0.5 * b[i];
            e = std::max({e, std::fabs(x[i + 1] - root), std::fabs(x[i] - (b[i] - 0.5 * root))});
            if (!(x[i] == x[i]) || !(x[i + 1] == x[i + 1])) return -1.0;
        }
        return e;
    } catch (const std::exception&) {
        return -1.0;
    }
}

// A server's estimates of a domain's device bytes, {least, most}.
void shim_estimate(const hdd_options* o, const uint32_t* flags, long long* bytes) {
    const DeviceEstimate e = estimate_device_bytes(*o, flags);
    bytes[0] = e.least;
    bytes[1] = e.most;
}

// Same plan: relative max-norm difference between its host solve (FP32
// coefficients) and the factorisations' own FP64 solve, for a random
// right-hand side; -1 on error.  *n gets the number of unknowns.
double shim_plan_check(void* h, int kind, int level, int* n) {
    Shim* s = static_cast<Shim*>(h);
    try {
        if (level < 0 || level >= s->ih.M || (kind != 0 && kind != 1)) return -1.0;
        std::vector<SnFactor> fs;
        PlanHost plan;
        interface_solve_plan(s->ih, kind, level, fs, plan);
        *n = plan.n;
        std::mt19937 rng(11);
        std::uniform_real_distribution<float> U(-1.0f, 1.0f);
        std::vector<float> b(plan.n), x(plan.n, 0.0f);
        for (float& v : b) v = U(rng);
        plan.emulate(b.data(), x.data());
        std::vector<double> ref(b.begin(), b.end());
        int off = 0;  // unknowns are concatenated in factor order (empty factors add none)
        for (const SnFactor& F : fs) {
            F.solve(ref.data() + off);
            off += F.n;
        }
        double dmax = 0, rmax = 0;
        for (int i = 0; i < plan.n; ++i) {
            dmax = std::max(dmax, std::fabs((double)x[i] - ref[i]));
            rmax = std::max(rmax, std::fabs(ref[i]));
        }
        return rmax > 0 ? dmax / rmax : dmax;
    } catch (const std::exception&) {
        return -1.0;
    }
}
}
