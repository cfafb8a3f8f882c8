// factor_plan_host.cpp -- the host side of the sparse factorisation (tf_factor.cuh) without a GPU, linked
// against libtf_b200.so. tests/test_factor_plan.py builds it with g++ and reads what it prints.
#include <algorithm>
#include <chrono>
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include <sys/resource.h>

#include "tf_factor.cuh"

namespace {

// A sheet of nx x ny columns of G nodes, triangulated: node blocks within a column and between neighbouring
// columns, one layer up or down. star > 0: column 0 has blocks with every star-th column besides.
struct Sheet {
    std::vector<int32_t> rowptr{0}, colidx;
    std::vector<double> X;
    Sheet(int nx, int ny, int G, int star = 0) {
        const int step[7][2] = {{-1, -1}, {-1, 0}, {0, -1}, {0, 0}, {0, 1}, {1, 0}, {1, 1}};
        for (int i = 0; i < nx; ++i)
            for (int j = 0; j < ny; ++j) {
                X.insert(X.end(), {i + 0.013 * (j % 7), 0.9 * j + 0.017 * (i % 5), 0.0});
                for (int k = 0; k < G; ++k) {
                    for (const auto& d : step) {
                        const int a = i + d[0], b = j + d[1];
                        if (a < 0 || b < 0 || a >= nx || b >= ny) continue;
                        for (int l = std::max(k - 1, 0); l <= std::min(k + 1, G - 1); ++l)
                            colidx.push_back((a * ny + b) * G + l);
                    }
                    const int c = i * ny + j;
                    if (star && c == 0)
                        for (int q = star; q < nx * ny; q += star) colidx.push_back(q * G + k);
                    else if (star && c % star == 0)
                        colidx.push_back(k);
                    std::sort(colidx.begin() + rowptr.back(), colidx.end());
                    colidx.erase(std::unique(colidx.begin() + rowptr.back(), colidx.end()), colidx.end());
                    rowptr.push_back((int32_t)colidx.size());
                }
            }
    }
};

uint64_t mix(uint64_t h, const void* p, size_t n) {  // FNV-1a
    for (size_t i = 0; i < n; ++i) h = (h ^ static_cast<const unsigned char*>(p)[i]) * 1099511628211ull;
    return h;
}
template <class T>
uint64_t mix(uint64_t h, const std::vector<T>& v) {
    return mix(h, v.data(), v.size() * sizeof(T));
}

// 0: every column is a pivot of one front, and every front's boundary is what its subtree's columns are next to.
int check(const tfb::FcPlan& P, const Sheet& one, int G) {
    const int nc = ((int)one.rowptr.size() - 1) / G;
    std::vector<int> owner(nc, -1);
    std::vector<std::vector<int32_t>> tree(P.fronts.size());
    for (int f = (int)P.fronts.size() - 1; f >= 0; --f) {  // children have larger numbers
        const tfb::FcFront& F = P.fronts[f];
        const int np = F.p / P.gd, nb = F.b / P.gd;
        std::vector<int32_t>& set = tree[f];
        for (int k = 0; k < np; ++k) {
            const int32_t v = P.verts[F.verts + k];
            if (owner[v] >= 0) return 1;
            owner[v] = f;
            set.push_back(v);
        }
        for (int c : F.child)
            if (c >= 0) set.insert(set.end(), tree[c].begin(), tree[c].end());
        std::vector<char> in(nc, 0);
        for (int32_t v : set) in[v] = 1;
        std::vector<int32_t> next, bnd(P.verts.begin() + F.verts + np, P.verts.begin() + F.verts + np + nb);
        for (int32_t v : set)
            for (int32_t k = one.rowptr[v * G]; k < one.rowptr[(v + 1) * G]; ++k) {
                const int32_t d = one.colidx[k] / G;
                if (!in[d]) {
                    in[d] = 1;
                    next.push_back(d);
                }
            }
        std::sort(next.begin(), next.end());
        std::sort(bnd.begin(), bnd.end());
        if (next != bnd) return 2;
    }
    for (int f : owner)
        if (f < 0) return 3;
    return 0;
}

int run(int argc, char** argv) {
    if (argc == 4 && !std::strcmp(argv[1], "span")) {  // of blocks [a, b)
        const tfb::FcSpan s = tfb::fc_block_span(std::atoi(argv[2]), std::atoi(argv[3]));
        std::printf("%" PRId64 " %" PRId64 "\n", s.begin, s.end);
        return 0;
    }
    if ((argc == 8 || argc == 9) && !std::strcmp(argv[1], "plan")) {  // nx ny G max_flops transposed tissues [kB]
        const int G = std::atoi(argv[4]), T = std::atoi(argv[7]);
        const Sheet one(std::atoi(argv[2]), std::atoi(argv[3]), G);
        const int n = (int)one.rowptr.size() - 1, blocks = one.rowptr.back();
        std::vector<int32_t> rowptr(1, 0), colidx, node0(1, 0);
        std::vector<double> X;
        for (int t = 0; t < T; ++t) {
            for (int i = 1; i <= n; ++i) rowptr.push_back(one.rowptr[i] + t * blocks);
            for (int32_t c : one.colidx) colidx.push_back(c + t * n);
            X.insert(X.end(), one.X.begin(), one.X.end());
            node0.push_back((t + 1) * n);
        }
        if (argc == 9) {  // as much address space besides what the process has by now
            long pages = 0;
            if (FILE* f = std::fopen("/proc/self/statm", "r")) {
                if (std::fscanf(f, "%ld", &pages) != 1) return 3;
                std::fclose(f);
            }
            rlimit lim;
            getrlimit(RLIMIT_AS, &lim);
            lim.rlim_cur = (rlim_t)pages * 4096 + (rlim_t)std::atoi(argv[8]) * 1024;
            if (setrlimit(RLIMIT_AS, &lim)) return 3;
        }
        tfb::FcPlan P;
        const auto t0 = std::chrono::steady_clock::now();
        tfb::build_factor_plan(T * n, G, rowptr.data(), colidx.data(), X.data(), T, node0.data(), std::atof(argv[5]),
                               std::atoi(argv[6]) != 0, P);
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        uint64_t h = 14695981039346656037ull;
        h = mix(mix(mix(mix(mix(mix(h, P.fronts), P.maps), P.verts), P.jblk), P.jblk_t), P.tasks);
        std::printf("%d %.6e %.2f %zu %016" PRIx64 "\n", P.ok ? 1 : 0, P.flops, ms, P.fronts.size(), h);
        return 0;
    }
    if (argc == 5 && !std::strcmp(argv[1], "nan")) {  // nx ny every: each such column's position not a number
        Sheet one(std::atoi(argv[2]), std::atoi(argv[3]), 2);
        for (size_t c = 0; c < one.X.size() / 3; c += std::atoi(argv[4])) one.X[3 * c + c % 3] = std::nan("");
        const int32_t node0[2] = {0, (int32_t)one.rowptr.size() - 1};
        tfb::FcPlan P;
        tfb::build_factor_plan(node0[1], 2, one.rowptr.data(), one.colidx.data(), one.X.data(), 1, node0, 1e13, false, P);
        std::printf("%d\n", P.ok ? 1 : 0);
        return 0;
    }
    if (argc == 6 && !std::strcmp(argv[1], "check")) {  // nx ny G star
        const int G = std::atoi(argv[4]);
        const Sheet one(std::atoi(argv[2]), std::atoi(argv[3]), G, std::atoi(argv[5]));
        const int32_t node0[2] = {0, (int32_t)one.rowptr.size() - 1};
        tfb::FcPlan P;
        tfb::build_factor_plan(node0[1], G, one.rowptr.data(), one.colidx.data(), one.X.data(), 1, node0, 1e13, false, P);
        std::printf("%d %d\n", P.ok ? 1 : 0, P.ok ? check(P, one, G) : -1);
        return 0;
    }
    return 2;
}

}  // namespace

int main(int argc, char** argv) {
    try {
        return run(argc, argv);
    } catch (const std::bad_alloc&) {
        std::printf("bad_alloc\n");
        return 0;
    }
}
