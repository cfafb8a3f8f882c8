// tf_factor_plan.cu -- nested dissection and symbolic factorisation of the Jacobian's block pattern
// (host code; the numeric kernels are in tf_factor.cu). No counterpart in the reference, which
// hands every system to Pardiso (NewtonRaphsonSolver.cpp:498-763).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <exception>
#include <mutex>
#include <numeric>
#include <thread>

#include "tf_factor.cuh"

namespace tfb {
namespace {

struct Node {
    std::vector<int32_t> piv, bnd;  // columns
    int depth = 0;
    int child[2] = {-1, -1};
    int32_t lo = 0, hi = 0;  // its subtree's columns in perm
};

// Operations of a front of p pivots and b boundary unknowns.
double front_flops(double p, double b) { return p * p * p * (2.0 / 3.0) + p * p * b + b * b * p; }

// Operations of the fronts of all tissues, against the limit.
struct Budget {
    double max_flops;
    std::mutex lock;
    double flops = 0.0;
    std::atomic<bool> over{false};

    void add(double more) {
        std::lock_guard<std::mutex> hold(lock);
        flops += more;
        if (flops > max_flops) over = true;
    }
};

// Columns of one tissue: their graph (ptr / adj over local ids), positions, and the dissection.
struct Dissection {
    const int32_t* ptr;
    const int32_t* adj;
    const double* X;  // [n][3]
    int leaf, gd;
    std::vector<Node> nodes;
    std::vector<int32_t> perm, label, match, seen, pos;
    int32_t next_label = 0, stamp = 0;

    // Augmenting path of the bipartite cut graph from a on side A (labels la) to side B (lb).
    bool augment(int32_t a, int32_t lb) {
        for (int32_t k = ptr[a]; k < ptr[a + 1]; ++k) {
            const int32_t b = adj[k];
            if (label[b] != lb || seen[b] == stamp) continue;
            seen[b] = stamp;
            if (match[b] < 0 || augment(match[b], lb)) {
                match[b] = a;
                match[a] = b;
                return true;
            }
        }
        return false;
    }
    // Columns reached from unmatched a by alternating paths (Koenig's construction).
    void reach(int32_t a, int32_t lb) {
        seen[a] = stamp;
        for (int32_t k = ptr[a]; k < ptr[a + 1]; ++k) {
            const int32_t b = adj[k];
            if (label[b] != lb || seen[b] == stamp) continue;
            seen[b] = stamp;
            if (match[b] >= 0 && seen[match[b]] != stamp) reach(match[b], lb);
        }
    }

    // Splits node id's columns perm[lo, hi) in two halves across the longest side of their bounding box; the
    // separator is a smallest set of columns that covers every block between the halves (a minimum vertex
    // cover of the cut edges, from a maximum matching). Its halves are appended to `nodes`.
    void split(int id) {
        const int32_t lo = nodes[id].lo, hi = nodes[id].hi;
        if (hi - lo <= leaf) {
            nodes[id].piv.assign(perm.begin() + lo, perm.begin() + hi);
            return;
        }
        double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
        for (int32_t k = lo; k < hi; ++k)
            for (int d = 0; d < 3; ++d) {
                mn[d] = std::min(mn[d], X[(size_t)perm[k] * 3 + d]);
                mx[d] = std::max(mx[d], X[(size_t)perm[k] * 3 + d]);
            }
        int ax = 0;
        for (int d = 1; d < 3; ++d)
            if (mx[d] - mn[d] > mx[ax] - mn[ax]) ax = d;
        const int32_t mid = lo + (hi - lo) / 2;
        const int a2 = ax == 0 ? 1 : 0;  // columns at the split coordinate are ordered along the cut
        std::nth_element(perm.begin() + lo, perm.begin() + mid, perm.begin() + hi, [&](int32_t u, int32_t v) {
            const double xu = X[(size_t)u * 3 + ax], xv = X[(size_t)v * 3 + ax];
            if (xu != xv) return xu < xv;
            const double yu = X[(size_t)u * 3 + a2], yv = X[(size_t)v * 3 + a2];
            return yu != yv ? yu < yv : u < v;
        });
        const int32_t la = next_label++, lb = next_label++;
        for (int32_t k = lo; k < hi; ++k) {
            label[perm[k]] = k < mid ? la : lb;
            match[perm[k]] = -1;
        }
        std::vector<int32_t> front_a;  // columns of A next to B
        for (int32_t k = lo; k < mid; ++k) {
            const int32_t a = perm[k];
            for (int32_t q = ptr[a]; q < ptr[a + 1]; ++q)
                if (label[adj[q]] == lb) {
                    front_a.push_back(a);
                    break;
                }
        }
        for (int32_t a : front_a)  // greedy matching first, then augmenting paths
            for (int32_t q = ptr[a]; q < ptr[a + 1]; ++q) {
                const int32_t b = adj[q];
                if (label[b] == lb && match[b] < 0) {
                    match[a] = b;
                    match[b] = a;
                    break;
                }
            }
        for (int32_t a : front_a)
            if (match[a] < 0) {
                ++stamp;
                augment(a, lb);
            }
        ++stamp;
        for (int32_t a : front_a)
            if (match[a] < 0 && seen[a] != stamp) reach(a, lb);
        // cover: unreached columns of A, reached columns of B
        const int32_t ls = next_label++;
        std::vector<int32_t> sep;
        for (int32_t a : front_a) {
            if (seen[a] != stamp) sep.push_back(a);
            for (int32_t q = ptr[a]; q < ptr[a + 1]; ++q) {
                const int32_t b = adj[q];
                if (label[b] == lb && seen[b] == stamp) {
                    label[b] = ls;
                    sep.push_back(b);
                }
            }
        }
        for (int32_t v : sep) label[v] = ls;
        const auto ea = std::stable_partition(perm.begin() + lo, perm.begin() + hi, [&](int32_t v) { return label[v] == la; });
        const auto eb = std::stable_partition(ea, perm.begin() + hi, [&](int32_t v) { return label[v] == lb; });
        const int32_t ma = (int32_t)(ea - perm.begin()), mb = (int32_t)(eb - perm.begin());
        nodes[id].piv.assign(eb, perm.begin() + hi);
        // pivots in order along the separator
        std::sort(nodes[id].piv.begin(), nodes[id].piv.end(), [&](int32_t u, int32_t v) {
            const double yu = X[(size_t)u * 3 + a2], yv = X[(size_t)v * 3 + a2];
            return yu != yv ? yu < yv : u < v;
        });
        // A half's boundary: the columns of the enclosing separators, this one's among them, next to it. From the top
        // down the fronts' sizes are known before the fronts below are.
        std::vector<int32_t> out = nodes[id].bnd;
        out.insert(out.end(), nodes[id].piv.begin(), nodes[id].piv.end());
        int n = 0;
        auto half = [&](int32_t a, int32_t z, int32_t l) {
            if (a == z) return;
            nodes[id].child[n++] = (int)nodes.size();
            Node h;
            h.depth = nodes[id].depth + 1;
            h.lo = a;
            h.hi = z;
            // from the separators' side or, where a column of theirs has very many neighbours, from the half's
            int64_t far = 0, near = 0;
            for (int32_t v : out) far += ptr[v + 1] - ptr[v];
            for (int32_t k = a; k < z && near < far; ++k) near += ptr[perm[k] + 1] - ptr[perm[k]];
            ++stamp;
            if (far <= near) {
                for (int32_t v : out)
                    for (int32_t q = ptr[v]; q < ptr[v + 1]; ++q)
                        if (label[adj[q]] == l) {
                            h.bnd.push_back(v);
                            break;
                        }
            } else {
                for (int32_t k = a; k < z; ++k)
                    for (int32_t q = ptr[perm[k]]; q < ptr[perm[k] + 1]; ++q) {
                        const int32_t v = adj[q];
                        if (label[v] == l || seen[v] == stamp) continue;
                        seen[v] = stamp;
                        h.bnd.push_back(v);
                    }
            }
            nodes.push_back(std::move(h));
        };
        half(lo, ma, la);
        half(ma, mb, lb);
    }

    // Elimination positions (children before their parent) and every front's boundary.
    int32_t order(int id, int32_t at) {
        for (int c : nodes[id].child)
            if (c >= 0) at = order(c, at);
        for (int32_t v : nodes[id].piv) pos[v] = at++;
        return at;
    }
    // The nodes in depth-first order from id on, into `to`.
    int renumber(int id, std::vector<Node>& to) {
        const int at = (int)to.size();
        to.push_back(std::move(nodes[id]));
        for (int k = 0; k < 2; ++k)
            if (to[at].child[k] >= 0) {
                const int c = renumber(to[at].child[k], to);
                to[at].child[k] = c;
            }
        return at;
    }

    // Level by level, the largest fronts first: a tissue too large for a factorisation shows after the top two or
    // three of its levels (2,000,000 nodes: after the first cut).
    void run(int32_t n, Budget& budget) {
        perm.resize(n);
        std::iota(perm.begin(), perm.end(), 0);
        label.assign(n, -1);
        match.assign(n, -1);
        seen.assign(n, -1);
        pos.assign(n, 0);
        nodes.emplace_back();
        nodes[0].hi = n;
        double mine = 0.0;  // not in the budget yet: its lock is for shares that matter, not for every front
        for (int id = 0; id < (int)nodes.size() && !budget.over; ++id) {
            split(id);
            const double p = (double)nodes[id].piv.size() * gd, b = (double)nodes[id].bnd.size() * gd;
            if (p > kFcMaxPivots || p + b > kFcMaxFront) budget.over = true;
            mine += front_flops(p, b);
            if (mine * 1024 > budget.max_flops) {
                budget.add(mine);
                mine = 0.0;
            }
        }
        budget.add(mine);
        if (budget.over) return;
        std::vector<Node> sorted;
        sorted.reserve(nodes.size());
        renumber(0, sorted);
        nodes.swap(sorted);
        order(0, 0);
        for (Node& f : nodes) std::sort(f.bnd.begin(), f.bnd.end(), [&](int32_t u, int32_t v) { return pos[u] < pos[v]; });
    }
};

// Fronts that one CTA factorises in shared memory.
bool one_cta(const FcFront& F) { return F.p > 0 && F.p <= kFcTile && F.b <= kFcSmallB; }

// f(0) .. f(n - 1) on up to 16 threads, fewer where no more can be started. What an f throws is thrown here, after
// every thread has ended.
template <class F>
void parallel_items(int n, F f) {
    const int nt = std::min<int>(n, (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency())));
    std::atomic<int> next{0};
    std::exception_ptr thrown;
    std::mutex lock;
    auto work = [&] {
        try {
            for (int i; (i = next.fetch_add(1)) < n;) f(i);
        } catch (...) {
            std::lock_guard<std::mutex> hold(lock);
            if (!thrown) thrown = std::current_exception();
            next = n;
        }
    };
    std::vector<std::thread> th;
    th.reserve(nt);
    try {
        for (int t = 1; t < nt; ++t) th.emplace_back(work);
    } catch (const std::exception&) {
    }
    work();
    for (auto& x : th) x.join();
    if (thrown) std::rethrow_exception(thrown);
}

}  // namespace

void build_factor_plan(int N, int G, const int32_t* rowptr, const int32_t* colidx, const double* X, int T,
                       const int32_t* node0, double max_flops, bool transposed, FcPlan& plan) {
    plan = FcPlan();
    const int nc = N / G, gd = 3 * G;
    plan.gd = gd;
    // a comparison of positions that are not numbers is no order, and std::nth_element may leave its range then
    if (!std::all_of(X, X + (size_t)nc * 3, [](double x) { return std::isfinite(x); })) return;
    // column graph (no self edges), global ids; a tissue's columns are consecutive. By runs of columns, so that a
    // single large tissue has every thread on it.
    std::vector<int32_t> ptr(nc + 1, 0), adj;
    {
        struct Run {
            int t, c0, c1;
            std::vector<int32_t> adj;
        };
        std::vector<Run> runs;
        for (int t = 0; t < T; ++t) {
            const int c0 = node0[t] / G, c1 = node0[t + 1] / G, len = std::max(8192, (c1 - c0 + 15) / 16);
            for (int c = c0; c < c1; c += len) runs.push_back({t, c, std::min(c + len, c1), {}});
        }
        parallel_items((int)runs.size(), [&](int i) {
            Run& r = runs[i];
            const int c0 = node0[r.t] / G, c1 = node0[r.t + 1] / G;
            std::vector<int32_t> mark(c1 - c0, -1);
            for (int c = r.c0; c < r.c1; ++c) {
                const size_t before = r.adj.size();
                for (int i = c * G; i < (c + 1) * G; ++i)
                    for (int32_t k = rowptr[i]; k < rowptr[i + 1]; ++k) {
                        const int32_t d = colidx[k] / G;
                        if (d != c && mark[d - c0] != c) {
                            mark[d - c0] = c;
                            r.adj.push_back(d - c0);
                        }
                    }
                ptr[c + 1] = (int32_t)(r.adj.size() - before);
            }
        });
        for (int c = 0; c < nc; ++c) ptr[c + 1] += ptr[c];
        adj.resize(ptr[nc]);
        parallel_items((int)runs.size(), [&](int i) { std::copy(runs[i].adj.begin(), runs[i].adj.end(), adj.begin() + ptr[runs[i].c0]); });
    }
    std::vector<Dissection> ds(T);
    Budget budget;
    budget.max_flops = max_flops;
    parallel_items(T, [&](int t) {
        const int c0 = node0[t] / G, c1 = node0[t + 1] / G;
        Dissection& d = ds[t];
        std::vector<int32_t> lp(c1 - c0 + 1);
        for (int c = c0; c <= c1; ++c) lp[c - c0] = ptr[c] - ptr[c0];
        d.ptr = lp.data();
        d.adj = adj.data() + ptr[c0];
        d.X = X + (size_t)c0 * 3;
        d.leaf = std::max(1, kFcTile / gd);
        d.gd = gd;
        d.run(c1 - c0, budget);
    });
    plan.flops = budget.flops;
    if (budget.over) return;
    // fronts of all tissues by depth; their operations again, in an order that no thread decides
    int depths = 0;
    plan.flops = 0.0;
    std::vector<std::vector<std::pair<int, int>>> at;  // per depth: (tissue, node)
    for (int t = 0; t < T; ++t)
        for (int k = 0; k < (int)ds[t].nodes.size(); ++k) {
            const Node& f = ds[t].nodes[k];
            if (f.depth >= depths) at.resize(depths = f.depth + 1);
            at[f.depth].push_back({t, k});
            plan.flops += front_flops((double)f.piv.size() * gd, (double)f.bnd.size() * gd);
        }
    std::vector<std::vector<int32_t>> id(T);
    for (int t = 0; t < T; ++t) id[t].resize(ds[t].nodes.size());
    int nf = 0;
    for (auto& level : at)
        for (auto& q : level) id[q.first][q.second] = nf++;
    plan.fronts.resize(nf);
    plan.depths.resize(depths);
    std::vector<std::pair<int, int>> of(nf);
    int64_t n_map = 0, n_vert = 0;
    for (int d = 0; d < depths; ++d) {
        int64_t scratch = 0, contrib = 0;
        for (auto& q : at[d]) {
            const int fi = id[q.first][q.second];
            of[fi] = q;
            const Node& f = ds[q.first].nodes[q.second];
            FcFront& F = plan.fronts[fi];
            const int np = (int)f.piv.size(), nb = (int)f.bnd.size();
            F.p = np * gd;
            F.b = nb * gd;
            F.ldp = (F.p + 1) & ~1;
            F.ldb = (F.b + 1) & ~1;
            F.tissue = q.first;
            F.verts = (int32_t)n_vert;
            n_vert += np + nb;
            for (int k = 0; k < 2; ++k) {
                F.child[k] = f.child[k] >= 0 ? id[q.first][f.child[k]] : -1;
                F.map[k] = (int32_t)n_map;
                if (f.child[k] >= 0) n_map += np + nb;
            }
            F.vec = (int32_t)plan.n_vec;
            F.piv = (int32_t)plan.n_piv;
            plan.n_vec += F.b;
            plan.n_piv += F.ldp;
            F.ent = (int32_t)plan.n_ent;
            plan.n_ent += F.p + F.b;
            F.x11 = plan.n_factor;
            F.w21 = F.x11 + (int64_t)F.p * F.ldp;
            plan.n_factor = F.w21 + (int64_t)F.b * F.ldp;
            if (one_cta(F)) {  // these live in shared memory
                F.a21 = F.l21 = F.lp = scratch;
            } else {
                F.a21 = scratch;
                F.l21 = F.a21 + (int64_t)F.b * F.ldp;
                F.lp = F.l21 + (int64_t)F.b * F.ldp;
                scratch = F.lp + (F.p > kFcTile ? (int64_t)F.p * kFcTile : 0);
            }
            F.c = contrib;
            contrib += (int64_t)F.b * F.ldb;
            if (d == 0) plan.n_root += F.p;
        }
        plan.n_scratch = std::max(plan.n_scratch, scratch);
        plan.n_contrib[d & 1] = std::max(plan.n_contrib[d & 1], contrib);
    }
    for (FcFront& F : plan.fronts)
        for (int k = 0; k < 2; ++k) {
            const FcFront* c = F.child[k] >= 0 ? &plan.fronts[F.child[k]] : nullptr;
            F.child_ldb[k] = c ? c->ldb : 0;
            F.child_vec[k] = c ? c->vec : 0;
            F.child_c[k] = c ? c->c : 0;
        }
    if (n_map > INT32_MAX || n_vert > INT32_MAX || plan.n_ent > INT32_MAX || plan.n_vec > INT32_MAX || plan.n_piv > INT32_MAX) return;
    plan.maps.resize(n_map);
    plan.verts.resize(n_vert);
    // columns, child maps and Jacobian blocks of every front
    std::vector<std::vector<int2>> jb(nf);
    const int step = 64;
    parallel_items((nf + step - 1) / step, [&](int chunk) {
        std::vector<int32_t> where;  // position in the front's column list, by local column
        for (int fi = chunk * step; fi < std::min(nf, (chunk + 1) * step); ++fi) {
            const int t = of[fi].first;
            const Dissection& D = ds[t];
            const Node& f = D.nodes[of[fi].second];
            FcFront& F = plan.fronts[fi];
            const int c0 = node0[t] / G, np = (int)f.piv.size(), nb = (int)f.bnd.size();
            if ((int)where.size() < (int)D.perm.size()) where.resize(D.perm.size());
            for (int k = 0; k < np + nb; ++k) {
                const int32_t v = k < np ? f.piv[k] : f.bnd[k - np];
                plan.verts[F.verts + k] = v + c0;
                where[v] = k;
            }
            for (int q = 0; q < 2; ++q) {
                if (f.child[q] < 0) continue;
                const Node& c = D.nodes[f.child[q]];
                int32_t* m = plan.maps.data() + F.map[q];
                std::fill(m, m + np + nb, -1);
                for (int k = 0; k < (int)c.bnd.size(); ++k) m[where[c.bnd[k]]] = k;
            }
            const int32_t first = np ? D.pos[f.piv[0]] : 0;
            for (int k = 0; k < np; ++k)
                for (int a = 0; a < G; ++a) {
                    const int node = (f.piv[k] + c0) * G + a;
                    for (int32_t e = rowptr[node]; e < rowptr[node + 1]; ++e) {
                        const int32_t other = colidx[e], v = other / G - c0;
                        const int32_t pv = D.pos[v], pk = D.pos[f.piv[k]];
                        if (pv < first || pv < pk || (pv == pk && other < node)) continue;
                        const int row = where[v] * gd + (other % G) * 3, col = k * gd + a * 3;
                        jb[fi].push_back(make_int2(e, (int)((uint32_t)row << 16 | (uint32_t)col)));
                    }
                }
        }
    });
    int64_t nj = 0;
    for (int fi = 0; fi < nf; ++fi) {
        plan.fronts[fi].j0 = (int32_t)nj;
        nj += (int64_t)jb[fi].size();
        plan.fronts[fi].j1 = (int32_t)nj;
    }
    if (nj > INT32_MAX) return;
    plan.jblk.resize(nj);
    if (transposed) plan.jblk_t.resize(nj);
    parallel_items((nf + step - 1) / step, [&](int chunk) {
        for (int fi = chunk * step; fi < std::min(nf, (chunk + 1) * step); ++fi) {
            std::copy(jb[fi].begin(), jb[fi].end(), plan.jblk.begin() + plan.fronts[fi].j0);
            if (!transposed) continue;
            const Dissection& D = ds[of[fi].first];
            const Node& f = D.nodes[of[fi].second];
            const int c0 = node0[of[fi].first] / G;
            for (size_t k = 0; k < jb[fi].size(); ++k) {  // block (node, other) -> (other, node)
                const int e = jb[fi][k].x, col = jb[fi][k].y & 0xffff;
                const int node = (f.piv[col / gd] + c0) * G + (col % gd) / 3, other = colidx[e];
                const int32_t* r0 = colidx + rowptr[other];
                const int32_t* r1 = colidx + rowptr[other + 1];
                plan.jblk_t[plan.fronts[fi].j0 + k] = (int32_t)(std::lower_bound(r0, r1, node) - colidx);
            }
        }
    });
    // task lists, the tasks of a launch by falling front size (the long ones start first)
    auto cdiv = [](int a, int b) { return (a + b - 1) / b; };
    for (int d = 0; d < depths; ++d) {
        FcDepth& L = plan.depths[d];
        std::vector<int32_t> fs;
        for (auto& q : at[d]) fs.push_back(id[q.first][q.second]);
        std::stable_sort(fs.begin(), fs.end(), [&](int32_t a, int32_t b) { return plan.fronts[a].p > plan.fronts[b].p; });
        auto list = [&](FcRange& r, auto emit) {
            r.begin = (int32_t)plan.tasks.size();
            for (int32_t fi : fs) emit(fi, plan.fronts[fi]);
            r.count = (int32_t)plan.tasks.size() - r.begin;
        };
        auto push = [&](int32_t f, int i, int j) { plan.tasks.push_back(FcTask{f, (int16_t)i, (int16_t)j}); };
        std::vector<int32_t> all = fs, rest;
        for (int32_t fi : fs)
            if (!one_cta(plan.fronts[fi])) rest.push_back(fi);
        std::stable_sort(fs.begin(), fs.end(), [&](int32_t a, int32_t b) { return plan.fronts[a].b > plan.fronts[b].b; });
        // in three launches by the shared memory they need, so that two and three small ones share an SM
        // (228 KB, 10 KB of it static per CTA)
        const int bound[4] = {INT32_MAX, 102000, 64000, 0};
        for (int c = 0; c < 3; ++c)
            list(L.small[c], [&](int32_t fi, const FcFront& F) {
                if (!one_cta(F)) return;
                const int bytes = fc_small_smem(F.p, F.b);
                if (bytes <= bound[c] && bytes > bound[c + 1]) push(fi, 0, 0);
            });
        fs = rest;
        list(L.gather, [&](int32_t fi, const FcFront& F) {
            const int rows = F.p > 128 ? 8 : 32;  // long rows: one a warp
            if (F.p > 0)
                for (int i = 0; i < cdiv(F.p + F.b, rows); ++i) push(fi, i, rows);
        });
        list(L.scatter, [&](int32_t fi, const FcFront& F) {
            for (int i = 0; i < cdiv(F.j1 - F.j0, kFcScatter); ++i) push(fi, i, 0);
        });
        list(L.diag, [&](int32_t fi, const FcFront& F) {
            if (F.p > 0) push(fi, 0, 0);
        });
        int np = 0;
        for (int32_t fi : fs) np = std::max(np, cdiv(plan.fronts[fi].p, kFcTile));
        L.panel0 = (int32_t)plan.panels.size();
        L.n_panel = std::max(0, np);
        for (int k = 0; k < np; ++k) {
            FcPanel P;
            // panel k of a front with nt panels: the column below the diagonal block (rows i > k), the
            // inverse's row k (columns j < k); then every tile below row k
            list(P.col, [&](int32_t fi, const FcFront& F) {
                const int nt = cdiv(F.p, kFcTile);
                if (nt <= k) return;
                for (int i = 0; i < nt; ++i)
                    if (i != k) push(fi, i, 0);
            });
            list(P.upd, [&](int32_t fi, const FcFront& F) {
                const int nt = cdiv(F.p, kFcTile);
                // the next diagonal block first: its factorisation is the long one
                if (k + 1 < nt) push(fi, k + 1, k + 1);
                for (int i = k + 1; i < nt; ++i)
                    for (int j = 0; j <= i; ++j)
                        if (!(i == k + 1 && j == k + 1)) push(fi, i, j);
            });
            plan.panels.push_back(P);
        }
        list(L.l21, [&](int32_t fi, const FcFront& F) {
            for (int j = cdiv(F.p, kFcTile) - 1; j >= 0; --j)
                for (int i = 0; i < cdiv(F.b, kFcTile); ++i) push(fi, i, j);
        });
        list(L.schur, [&](int32_t fi, const FcFront& F) {
            // with them, from the same l21, the tiles of w21 (j < 0: column tile -1 - j)
            for (int j = 0; j < cdiv(F.p, kFcTile); ++j)
                for (int i = 0; i < cdiv(F.b, kFcTile); ++i) push(fi, i, -1 - j);
            for (int i = 0; i < cdiv(F.b, kFcTile); ++i)
                for (int j = 0; j <= i; ++j) push(fi, i, j);
        });
        // the longest products first, so that short ones fill the last wave
        auto by_length = [&](const FcTask& a, const FcTask& b) {
            auto length = [&](const FcTask& t) { return plan.fronts[t.front].p - (t.j < 0 ? (-1 - t.j) * kFcTile : 0); };
            return length(a) > length(b);
        };
        std::stable_sort(plan.tasks.begin() + L.schur.begin, plan.tasks.begin() + L.schur.begin + L.schur.count, by_length);
        fs = all;
        std::stable_sort(fs.begin(), fs.end(), [&](int32_t a, int32_t b) {
            return (int64_t)plan.fronts[a].p * plan.fronts[a].b > (int64_t)plan.fronts[b].p * plan.fronts[b].b;
        });
        // Up: rows of [x11; w21] by entries, three tasks an SM where a depth is that large (the tasks of a small
        // depth are latency: 8192 entries each took 2.53 ms a step on 2,713 prisms, 2.33 like this; smaller
        // still, no gain). Down: 64 columns; 32 and more threads where there are many rows, or fewer tasks
        // than SMs (2.33 to 2.25 ms; up to four times the SMs: the wing disc loses 1 %).
        int64_t entries = 0, tiles = 0;
        for (int32_t fi : all) {
            entries += (int64_t)(plan.fronts[fi].p + plan.fronts[fi].b) * plan.fronts[fi].p;
            tiles += cdiv(plan.fronts[fi].p, 64);
        }
        const int per = (int)std::min<int64_t>(kFcRowEntries, std::max<int64_t>(kFcRowEntries / 8, entries / (3 * kFcSms)));
        const bool narrow = tiles < kFcSms;
        list(L.fwd, [&](int32_t fi, const FcFront& F) {
            const int n = F.p + F.b, rows = F.p > 128 ? std::max(8, per / F.p / 8 * 8)
                                                     : std::max(32, per / std::max(F.p, 1) / 32 * 32);
            for (int i = 0; i < cdiv(n, rows); ++i) push(fi, i, std::min(rows, 32736));
            L.fwd_smem = std::max(L.fwd_smem, (int32_t)(F.ldp * sizeof(double)));
        });
        list(L.bwd, [&](int32_t fi, const FcFront& F) {
            const int cols = F.p > 256 || narrow ? 32 : 64, n = F.p + F.b;
            for (int i = 0; i < cdiv(F.p, cols); ++i) push(fi, i, cols);
            L.bwd_smem = std::max(L.bwd_smem, (int32_t)((F.p + F.b) * sizeof(double)));
            if (n > (narrow ? 128 : 300)) L.bwd_threads = std::max(L.bwd_threads, n > (narrow ? 300 : 700) ? 1024 : 512);
        });
    }
    if (plan.tasks.size() > (size_t)INT32_MAX) return;
    plan.ok = true;
}

}  // namespace tfb
