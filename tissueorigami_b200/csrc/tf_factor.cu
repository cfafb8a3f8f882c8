// tf_factor.cu -- numeric multifrontal factorisation of a symmetric J, its solve, and the conjugate
// gradients it preconditions (FP64 throughout). The plan and the notation are in tf_factor.cuh.
//
// Dense work runs on the FP64 tensor instruction (mma.sync m8n8k4; tcgen05 has no FP64 kind): a
// 64 x 64 output tile per CTA. One depth of the dissection tree is
//   k_fc_gather    the front's pivot columns: the children's contributions, gathered (else zero)
//   k_fc_scatter   += its Jacobian blocks
//   k_fc_diag      the first 64 pivots: G^-1 and the signs
//   k_fc_col/upd   per further panel of 64 pivots: L's column panel and the inverse's row panel, then
//                  every tile below (the tile that becomes the next diagonal block factorises it too)
//   k_fc_gemm      l21 = A21 x11^T S, then C = children - l21 S l21^T
#include <math.h>

#include "tf_factor.cuh"

namespace tfb {
namespace {

constexpr int kT = kFcTile;
constexpr int kLd = kT + 4;  // shared leading dimension: 8-byte reads of a fragment hit distinct banks
constexpr int kKc = 16;      // K extent of one stage of the long GEMMs
constexpr int kKld = kKc + 4;
constexpr int kStages = 3;

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// ---- assembly of a front -------------------------------------------------------------------

// Rows [32 i, 32 i + 32) of the front's pivot columns: what its children left there. Rows below p
// need the columns up to the diagonal only.
__global__ void __launch_bounds__(256) k_fc_gather(FcWork w, int begin, int parity) {
    extern __shared__ int2 s_col[];  // per pivot column: its index on either child's boundary
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const double* C[2] = {nullptr, nullptr};
    int ldc[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < 2; ++q)
        if (F.child[q] >= 0) {
            const FcFront& ch = w.fronts[F.child[q]];
            C[q] = w.contrib[parity ^ 1] + ch.c;
            ldc[q] = ch.ldb;
        }
    for (int c = threadIdx.x; c < F.p; c += blockDim.x) {
        const int v = c / w.gd, r = c - v * w.gd;
        int m[2] = {-1, -1};
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (C[q]) {
                const int k = w.maps[F.map[q] + v];
                if (k >= 0) m[q] = k * w.gd + r;
            }
        s_col[c] = make_int2(m[0], m[1]);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r1 = min((tk.i + 1) * kFcGatherRows, F.p + F.b);
    for (int row = tk.i * kFcGatherRows + warp; row < r1; row += 8) {
        const int v = row / w.gd, r = row - v * w.gd;
        const double* R[2] = {nullptr, nullptr};
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (C[q]) {
                const int k = w.maps[F.map[q] + v];
                if (k >= 0) R[q] = C[q] + (size_t)(k * w.gd + r) * ldc[q];
            }
        const int n = row < F.p ? row + 1 : F.p;
        double* out = row < F.p ? w.factor + F.x11 + (size_t)row * F.ldp : w.scratch + F.a21 + (size_t)(row - F.p) * F.ldp;
        for (int c = lane; c < n; c += 32) {
            const int2 m = s_col[c];
            double s = 0.0;
            if (R[0] && m.x >= 0) s = R[0][m.x];
            if (R[1] && m.y >= 0) s += R[1][m.y];
            out[c] = s;
        }
    }
}

// += the front's Jacobian blocks. Block (column k, row i) of the lower triangle is read from row k of
// J, transposed; each lands on entries of its own.
__global__ void __launch_bounds__(256) k_fc_scatter(FcWork w, const double* __restrict__ vals, int begin) {
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int b0 = F.j0 + tk.i * kFcScatter, b1 = min(b0 + kFcScatter, F.j1);
    for (int e = threadIdx.x; e < (b1 - b0) * 9; e += blockDim.x) {
        const int k = e / 9, en = e - k * 9, cc = en / 3, rr = en - cc * 3;
        const int2 jb = w.jblk[b0 + k];
        const int row = (int)((uint32_t)jb.y >> 16) + rr, col = (jb.y & 0xffff) + cc;
        double* out = row < F.p ? w.factor + F.x11 + (size_t)row * F.ldp + col
                                : w.scratch + F.a21 + (size_t)(row - F.p) * F.ldp + col;
        *out += vals[(size_t)jb.x * 9 + en];
    }
}

// ---- pivot block -----------------------------------------------------------------------------

// LDL^T of the 64 x 64 block whose lower triangle is in s (rows / columns from n on: the identity), by
// the row operations that also turn the identity into L^-1, in place: 256 threads, thread 4 r + q holds
// row r, columns q, q + 4, ... A chain of 64 steps (one shared row exchange each) bounds it.
// Writes G^-1 = |D|^-1/2 L^-1 (upper triangle zero) to out and sign(D) to sign.
__device__ void factor_block(double (*s)[kLd], int n, double* out, int ld, double* sign, int32_t* flag) {
    __shared__ double s_row[2][kT];
    __shared__ double s_d[kT];
    const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int c = 4 * k + q;
        v[k] = r < n && c < n ? (c <= r ? s[r][c] : s[c][r]) : (r == c ? 1.0 : 0.0);
    }
    bool bad = false;
#pragma unroll
    for (int jk = 0; jk < 16; ++jk) {
        for (int jq = 0; jq < 4; ++jq) {
            const int j = 4 * jk + jq, buf = j & 1;
            if (r == j) {
#pragma unroll
                for (int k = 0; k < 16; ++k) s_row[buf][4 * k + q] = v[k];
            }
            __syncthreads();
            const double d = s_row[buf][j];
            if (threadIdx.x == 0) s_d[j] = d;
            if (!(fabs(d) > 0.0) || !isfinite(d)) bad = true;
            const double a = __shfl_sync(0xffffffffu, v[jk], (threadIdx.x & 28) | jq);
            if (r > j) {
                const double m = a / d;
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const int c = 4 * k + q;
                    v[k] = c == j ? -m : v[k] - m * s_row[buf][c];
                }
            }
        }
    }
    __syncthreads();
    // row r now holds L^-1 left of the diagonal
    const double d = s_d[r];
    const double g = 1.0 / sqrt(fabs(d));
    if (r < n) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int c = 4 * k + q;
            if (c < n) out[(size_t)r * ld + c] = c < r ? v[k] * g : (c == r ? g : 0.0);
        }
        if (q == 0) sign[r] = d < 0.0 ? -1.0 : 1.0;
    }
    if (bad && threadIdx.x == 0) *flag = 1;
}

__global__ void __launch_bounds__(256) k_fc_diag(FcWork w, int begin) {
    __shared__ double s[kT][kLd];
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    double* A = w.factor + F.x11;
    const int n = min(kT, F.p);
    for (int e = threadIdx.x; e < n * kT; e += blockDim.x) {
        const int r = e / kT, c = e - r * kT;
        if (c <= r) s[r][c] = A[(size_t)r * F.ldp + c];
    }
    __syncthreads();
    factor_block(s, n, A, F.ldp, w.sign + F.piv, w.flags + F.tissue);
}

// A 64 x 64 tile of a matrix with `rows` x `cols` valid entries at src into shared memory (zero
// outside), optionally its columns times sign.
__device__ __forceinline__ void load_tile(double (*s)[kLd], const double* src, int ld, int rows, int cols) {
    for (int e = threadIdx.x; e < kT * kT; e += 256) {
        const int r = e >> 6, c = e & 63;
        s[r][c] = r < rows && c < cols ? src[(size_t)r * ld + c] : 0.0;
    }
}

// 64 x 64 x 64 product of two shared tiles by 8 warps (16 x 32 each): acc = A B^T (BT: B as [col][k]) or
// A B (B as [k][col]).
template <bool BT>
__device__ __forceinline__ void tile_mma(double (*A)[kLd], double (*B)[kLd], double (&acc)[2][4][2]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp >> 1) * 16 + (lane >> 2), c0 = (warp & 1) * 32 + (lane >> 2), kk = lane & 3;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 4
    for (int k = kk; k < kT; k += 4) {
        double a[2], b[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) a[i] = A[r0 + 8 * i][k];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = BT ? B[c0 + 8 * j][k] : B[k][c0 + 8 * j];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_f64(acc[i][j], a[i], b[j]);
    }
}

// Visit the (row, column) of every accumulator of tile_mma.
template <class F>
__device__ __forceinline__ void tile_each(double (&acc)[2][4][2], F f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp >> 1) * 16 + (lane >> 2), c0 = (warp & 1) * 32 + 2 * (lane & 3);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) f(r0 + 8 * i, c0 + 8 * j + h, acc[i][j][h]);
}

constexpr int kPanelSmem = 2 * kT * kLd * (int)sizeof(double);

// Panel k, G_k^-1 known: task i > k: L_ik = A_ik G_k^-T S_k into the panel scratch; i < k: the inverse's
// row panel, X_ki = G_k^-1 X_ki in place.
__global__ void __launch_bounds__(256) k_fc_col(FcWork w, int begin, int k) {
    extern __shared__ double s_dyn[];
    double(*sA)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn);
    double(*sB)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn + kT * kLd);
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    double* X = w.factor + F.x11;
    const int i = tk.i, nk = min(kT, F.p - k * kT), ni = min(kT, F.p - i * kT);
    const double* Gk = X + (size_t)k * kT * F.ldp + k * kT;
    double acc[2][4][2];
    if (i > k) {
        load_tile(sA, X + (size_t)i * kT * F.ldp + k * kT, F.ldp, ni, nk);
        load_tile(sB, Gk, F.ldp, nk, nk);
        __syncthreads();
        tile_mma<true>(sA, sB, acc);
        double* lp = w.scratch + F.lp + (size_t)i * kT * kT;
        const double* sg = w.sign + F.piv + k * kT;
        tile_each(acc, [&](int r, int c, double v) {
            if (r < ni) lp[r * kT + c] = c < nk ? v * sg[c] : 0.0;
        });
    } else {
        double* Xk = X + (size_t)k * kT * F.ldp + i * kT;
        load_tile(sA, Gk, F.ldp, nk, nk);
        load_tile(sB, Xk, F.ldp, nk, kT);
        __syncthreads();
        tile_mma<false>(sA, sB, acc);
        tile_each(acc, [&](int r, int c, double v) {
            if (r < nk) Xk[(size_t)r * F.ldp + c] = v;
        });
    }
}

// Panel k, the tiles below it: A_ij -= L_ik S_k L_jk^T (j > k), X_ik = -L_ik G_k^-1, X_ij -= L_ik X_kj (j < k).
// The tile that is the next diagonal block is factorised at once.
__global__ void __launch_bounds__(256) k_fc_upd(FcWork w, int begin, int k) {
    extern __shared__ double s_dyn[];
    double(*sA)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn);
    double(*sB)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn + kT * kLd);
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    double* X = w.factor + F.x11;
    const int i = tk.i, j = tk.j;
    const int ni = min(kT, F.p - i * kT), nj = min(kT, F.p - j * kT), nk = min(kT, F.p - k * kT);
    const double* lp = w.scratch + F.lp;
    double* out = X + (size_t)i * kT * F.ldp + j * kT;
    double acc[2][4][2];
    load_tile(sA, lp + (size_t)i * kT * kT, kT, ni, nk);
    if (j > k) {
        const double* sg = w.sign + F.piv + k * kT;
        const double* lj = lp + (size_t)j * kT * kT;
        for (int e = threadIdx.x; e < kT * kT; e += 256) {
            const int r = e >> 6, c = e & 63;
            sB[r][c] = r < nj && c < nk ? lj[r * kT + c] * sg[c] : 0.0;
        }
        __syncthreads();
        tile_mma<true>(sA, sB, acc);
        if (i == k + 1 && j == k + 1) {
            __syncthreads();
            tile_each(acc, [&](int r, int c, double v) {
                if (r < ni && c <= r) sA[r][c] = out[(size_t)r * F.ldp + c] - v;
            });
            __syncthreads();
            factor_block(sA, ni, out, F.ldp, w.sign + F.piv + i * kT, w.flags + F.tissue);
        } else {
            tile_each(acc, [&](int r, int c, double v) {
                if (r < ni && c < nj && (i != j || c <= r)) out[(size_t)r * F.ldp + c] -= v;
            });
        }
        return;
    }
    load_tile(sB, X + (size_t)k * kT * F.ldp + j * kT, F.ldp, nk, j == k ? nk : kT);
    __syncthreads();
    tile_mma<false>(sA, sB, acc);
    if (j == k)
        tile_each(acc, [&](int r, int c, double v) {
            if (r < ni && c < nk) out[(size_t)r * F.ldp + c] = -v;
        });
    else
        tile_each(acc, [&](int r, int c, double v) {
            if (r < ni) out[(size_t)r * F.ldp + c] -= v;
        });
}

// ---- boundary GEMMs ---------------------------------------------------------------------------

// 64 x 64 tile of A B^T, both row-major with K contiguous, by 4 warps (32 x 32 each: 16 accumulator
// tiles hide the tensor instruction's latency), K in stages of 16 through a 3-stage cp.async ring.
// a_rows / b_rows: valid rows (0 outside); K: valid columns. SIGN: B's columns times sign.
template <bool SIGN>
__device__ __forceinline__ void gemm_tile(const double* A, int lda, int a_rows, const double* B, int ldb, int b_rows, int K,
                                          const double* sign, double* smem, double (&acc)[4][4][2]) {
    double* sa = smem;
    double* sb = smem + kStages * kT * kKld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_it = (K + kKc - 1) / kKc;
    auto load = [&](int it) {
        const int st = it % kStages, k0 = it * kKc;
#pragma unroll
        for (int e = 0; e < 4; ++e) {  // 64 rows x 8 chunks of two doubles
            const int id = threadIdx.x + e * 128, r = id >> 3, c = (id & 7) * 2, left = K - (k0 + c);
            const int nb = left >= 2 ? 16 : (left > 0 ? 8 : 0);
            const int na_ = r < a_rows ? nb : 0, nb_ = r < b_rows ? nb : 0;
            cp_async16(sa + (st * kT + r) * kKld + c, na_ ? A + (size_t)r * lda + k0 + c : A, na_);
            cp_async16(sb + (st * kT + r) * kKld + c, nb_ ? B + (size_t)r * ldb + k0 + c : B, nb_);
        }
    };
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
    for (int st = 0; st < kStages - 1; ++st) {
        if (st < n_it) load(st);
        cp_commit();
    }
    const int ra = (warp >> 1) * 32 + (lane >> 2), rb = (warp & 1) * 32 + (lane >> 2), kk = lane & 3;
    for (int it = 0; it < n_it; ++it) {
        cp_wait<kStages - 2>();
        __syncthreads();
        if (it + kStages - 1 < n_it) load(it + kStages - 1);
        cp_commit();
        const double* pa = sa + ((it % kStages) * kT + ra) * kKld + kk;
        const double* pb = sb + ((it % kStages) * kT + rb) * kKld + kk;
#pragma unroll
        for (int k = 0; k < kKc; k += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = pa[8 * i * kKld + k];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = pb[8 * j * kKld + k];
            if (SIGN) {
                const int kc = it * kKc + k + kk;
                const double sg = kc < K ? sign[kc] : 0.0;
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] *= sg;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_f64(acc[i][j], a[i], b[j]);
        }
    }
    cp_wait<0>();
}

constexpr int kGemmSmem = 2 * kStages * kT * kKld * (int)sizeof(double);

// l21 tile (i, j) = A21 rows i x (x11 rows j)^T, times S; x11 is lower triangular, so K ends at the tile.
__global__ void __launch_bounds__(128) k_fc_l21(FcWork w, int begin) {
    extern __shared__ __align__(16) double s_dyn[];
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int i = tk.i, j = tk.j, ni = min(kT, F.b - i * kT), nj = min(kT, F.p - j * kT);
    double acc[4][4][2];
    gemm_tile<false>(w.scratch + F.a21 + (size_t)i * kT * F.ldp, F.ldp, ni, w.factor + F.x11 + (size_t)j * kT * F.ldp, F.ldp, nj,
                     min(F.p, (j + 1) * kT), nullptr, s_dyn, acc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp >> 1) * 32 + (lane >> 2), c0 = (warp & 1) * 32 + 2 * (lane & 3);
    double* out = w.factor + F.l21 + (size_t)i * kT * F.ldp + j * kT;
    const double* sg = w.sign + F.piv + j * kT;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * a, c = c0 + 8 * b + h;
                if (r < ni && c < nj) out[(size_t)r * F.ldp + c] = acc[a][b][h] * sg[c];
            }
}

// Contribution tile (i, j <= i): what the children left there minus l21 S l21^T.
__global__ void __launch_bounds__(128) k_fc_schur(FcWork w, int begin, int parity) {
    extern __shared__ __align__(16) double s_dyn[];
    __shared__ int s_map[2][2][kT];  // child, rows / columns
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int i = tk.i, j = tk.j, ni = min(kT, F.b - i * kT), nj = min(kT, F.b - j * kT);
    for (int e = threadIdx.x; e < 4 * kT; e += blockDim.x) {
        const int q = e >> 7, side = (e >> 6) & 1, c = e & 63, idx = (side ? j : i) * kT + c;
        int m = -1;
        if (F.child[q] >= 0 && idx < F.b) {
            const int v = (F.p + idx) / w.gd, r = F.p + idx - v * w.gd;
            const int k = w.maps[F.map[q] + v];
            if (k >= 0) m = k * w.gd + r;
        }
        s_map[q][side][c] = m;
    }
    double acc[4][4][2];
    const double* L = w.factor + F.l21;
    gemm_tile<true>(L + (size_t)i * kT * F.ldp, F.ldp, ni, L + (size_t)j * kT * F.ldp, F.ldp, nj, F.p, w.sign + F.piv, s_dyn, acc);
    __syncthreads();
    const double* C[2] = {nullptr, nullptr};
    int ldc[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < 2; ++q)
        if (F.child[q] >= 0) {
            const FcFront& ch = w.fronts[F.child[q]];
            C[q] = w.contrib[parity ^ 1] + ch.c;
            ldc[q] = ch.ldb;
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp >> 1) * 32 + (lane >> 2), c0 = (warp & 1) * 32 + 2 * (lane & 3);
    double* out = w.contrib[parity] + F.c + (size_t)i * kT * F.ldb + j * kT;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * a, c = c0 + 8 * b + h;
                if (r >= ni || c >= nj || (i == j && c > r)) continue;
                double s = -acc[a][b][h];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int mr = s_map[q][0][r], mc = s_map[q][1][c];
                    if (mr >= 0 && mc >= 0) s += C[q][(size_t)mr * ldc[q] + mc];
                }
                out[(size_t)r * F.ldb + c] = s;
            }
}

// ---- solve -------------------------------------------------------------------------------------

// The children's share of entry `idx` (pivots, then boundary) of a front's right-hand side.
__device__ __forceinline__ double from_children(const FcWork& w, const FcFront& F, int idx) {
    const int v = idx / w.gd, r = idx - v * w.gd;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 2; ++q)
        if (F.child[q] >= 0) {
            const int k = w.maps[F.map[q] + v];
            if (k >= 0) s += w.vec[w.fronts[F.child[q]].vec + k * w.gd + r];
        }
    return s;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// z = x11 v_P for 32 pivots, v_P the right-hand side plus the children's vectors.
__global__ void __launch_bounds__(256) k_fc_fwd1(FcWork w, const double* __restrict__ in, int begin) {
    extern __shared__ double s_v[];
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int r1 = min((tk.i + 1) * kFcRows, F.p);
    for (int c = threadIdx.x; c < r1; c += blockDim.x) {
        const int v = c / w.gd;
        s_v[c] = in[(size_t)w.verts[F.verts + v] * w.gd + (c - v * w.gd)] + from_children(w, F, c);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int r = tk.i * kFcRows + (threadIdx.x >> 5); r < r1; r += 8) {
        const double* X = w.factor + F.x11 + (size_t)r * F.ldp;
        double s = 0.0;
        for (int c = lane; c <= r; c += 32) s += X[c] * s_v[c];
        s = warp_sum(s);
        if (lane == 0) w.z[F.piv + r] = s;
    }
}

// v_B = the children's vectors - l21 z for 32 boundary rows.
__global__ void __launch_bounds__(256) k_fc_fwd2(FcWork w, int begin) {
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int r1 = min((tk.i + 1) * kFcRows, F.b), lane = threadIdx.x & 31;
    const double* z = w.z + F.piv;
    for (int r = tk.i * kFcRows + (threadIdx.x >> 5); r < r1; r += 8) {
        const double* L = w.factor + F.l21 + (size_t)r * F.ldp;
        double s = 0.0;
        for (int c = lane; c < F.p; c += 32) s += L[c] * z[c];
        s = warp_sum(s);
        if (lane == 0) w.vec[F.vec + r] = from_children(w, F, F.p + r) - s;
    }
}

// Partial sums of l21^T x_B: 128 boundary rows (task i) x 64 pivots (task j).
__global__ void __launch_bounds__(256) k_fc_bwd1(FcWork w, const double* __restrict__ x, int begin) {
    __shared__ double s_x[kFcBackRows];
    __shared__ double s_p[4][kT];
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int r0 = tk.i * kFcBackRows, n = min(kFcBackRows, F.b - r0);
    for (int r = threadIdx.x; r < n; r += blockDim.x) {
        const int idx = F.p + r0 + r, v = idx / w.gd;
        s_x[r] = x[(size_t)w.verts[F.verts + v] * w.gd + (idx - v * w.gd)];
    }
    __syncthreads();
    const int c = threadIdx.x & 63, part = threadIdx.x >> 6, col = tk.j * kT + c;
    double s = 0.0;
    if (col < F.p) {
        const double* L = w.factor + F.l21 + (size_t)r0 * F.ldp + col;
#pragma unroll 4
        for (int r = part; r < n; r += 4) s += L[(size_t)r * F.ldp] * s_x[r];
    }
    s_p[part][c] = s;
    __syncthreads();
    if (part == 0 && col < F.p) w.tp[F.tp + (size_t)tk.i * F.ldp + col] = s_p[0][c] + s_p[1][c] + s_p[2][c] + s_p[3][c];
}

// x_P = x11^T (S z - l21^T x_B) for 32 pivots.
__global__ void __launch_bounds__(256) k_fc_bwd2(FcWork w, double* __restrict__ x, int begin) {
    extern __shared__ double s_v[];
    __shared__ double s_p[8][33];
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    if (!w.active[F.tissue]) return;
    const int c0 = tk.i * kFcRows, chunks = (F.b + kFcBackRows - 1) / kFcBackRows;
    for (int c = c0 + threadIdx.x; c < F.p; c += blockDim.x) {
        double t = w.sign[F.piv + c] * w.z[F.piv + c];
        for (int k = 0; k < chunks; ++k) t -= w.tp[F.tp + (size_t)k * F.ldp + c];
        s_v[c - c0] = t;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = c0 + lane;
    double s = 0.0;
    if (col < F.p) {
        const double* X = w.factor + F.x11 + col;
#pragma unroll 4
        for (int r = c0 + warp; r < F.p; r += 8)
            if (r >= col) s += X[(size_t)r * F.ldp] * s_v[r - c0];
    }
    s_p[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && col < F.p) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += s_p[k][lane];
        const int v = col / w.gd;
        x[(size_t)w.verts[F.verts + v] * w.gd + (col - v * w.gd)] = t;
    }
}

// ---- conjugate gradients ------------------------------------------------------------------------

__device__ __forceinline__ double block_total(double v, double* smem) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) smem[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += smem[k];
    return t;
}

// Sum of a tissue's chunk partials, the same in every thread and every CTA.
__device__ __forceinline__ double tissue_total(const FcCg& c, const double* part, int t, double* smem) {
    double s = 0.0;
    for (int k = c.chunk0[t] + threadIdx.x; k < c.chunk0[t + 1]; k += blockDim.x) s += part[k];
    return block_total(s, smem);
}

__global__ void __launch_bounds__(256) k_fc_cg_start(KrylovWork w, FcCg c) {
    __shared__ double smem[8];
    const FcChunk ch = c.chunks[blockIdx.x];
    if (!c.active[ch.tissue]) return;
    double s = 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += blockDim.x) {
        const double b = w.b[i];
        w.x[i] = 0.0;
        w.r[i] = b;
        w.p[i] = 0.0;
        s += b * b;
    }
    s = block_total(s, smem);
    if (threadIdx.x == 0) c.part[2 * c.n_chunks + blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_fc_cg_begin(FcCg c, double rtol, int max_iter) {
    __shared__ double smem[8];
    const int t = blockIdx.x;
    if (!c.active[t]) {
        if (threadIdx.x == 0) c.running[t] = 0;
        return;
    }
    const double bb = tissue_total(c, c.part + 2 * c.n_chunks, t, smem);
    if (threadIdx.x == 0) {
        KrylovScalars& k = c.sc[t];
        k.bb = k.rr = bb;
        k.tol2 = rtol * rtol * bb;
        k.rho = k.rho_prev = 0.0;
        k.iter = 0;
        k.max_iter = max_iter;
        k.method = KM_CG;
        k.status = !isfinite(bb) ? KS_NONFINITE : (bb > 0.0 ? KS_RUNNING : KS_CONVERGED);
        c.running[t] = k.status == KS_RUNNING;
    }
}

__global__ void __launch_bounds__(256) k_fc_cg_dot(KrylovWork w, FcCg c, const double* __restrict__ z) {
    __shared__ double smem[8];
    const FcChunk ch = c.chunks[blockIdx.x];
    if (!c.running[ch.tissue]) return;
    double s = 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += blockDim.x) s += w.r[i] * z[i];
    s = block_total(s, smem);
    if (threadIdx.x == 0) c.part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_fc_cg_p(KrylovWork w, FcCg c, const double* __restrict__ z) {
    __shared__ double smem[8];
    const FcChunk ch = c.chunks[blockIdx.x];
    if (!c.running[ch.tissue]) return;
    const double rho = tissue_total(c, c.part, ch.tissue, smem), old = c.sc[ch.tissue].rho_prev;
    const double beta = old != 0.0 ? rho / old : 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += blockDim.x) w.p[i] = z[i] + beta * w.p[i];
}

// q = J p and the chunk's (p, q); eight lanes a row.
__global__ void __launch_bounds__(256) k_fc_cg_spmv(KrylovWork w, FcCg c, double* __restrict__ q) {
    __shared__ double smem[8];
    const FcChunk ch = c.chunks[blockIdx.x];
    if (!c.running[ch.tissue]) return;
    const int gl = threadIdx.x & 7;
    double dot = 0.0;
    for (int base = ch.row0; base < ch.row1; base += 32) {
        const int row = base + (threadIdx.x >> 3);
        double y0 = 0.0, y1 = 0.0, y2 = 0.0;
        if (row < ch.row1)
            for (int k = w.rowptr[row] + gl; k < w.rowptr[row + 1]; k += 8) {
                const double* B = w.vals + (size_t)k * 9;
                const double* x = w.p + (size_t)w.colidx[k] * 3;
                const double x0 = x[0], x1 = x[1], x2 = x[2];
                y0 += B[0] * x0 + B[1] * x1 + B[2] * x2;
                y1 += B[3] * x0 + B[4] * x1 + B[5] * x2;
                y2 += B[6] * x0 + B[7] * x1 + B[8] * x2;
            }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) {
            y0 += __shfl_xor_sync(0xffffffffu, y0, off);
            y1 += __shfl_xor_sync(0xffffffffu, y1, off);
            y2 += __shfl_xor_sync(0xffffffffu, y2, off);
        }
        if (row < ch.row1 && gl < 3) {
            const double y = gl == 0 ? y0 : (gl == 1 ? y1 : y2);
            q[(size_t)row * 3 + gl] = y;
            dot += y * w.p[(size_t)row * 3 + gl];
        }
    }
    dot = block_total(dot, smem);
    if (threadIdx.x == 0) c.part[c.n_chunks + blockIdx.x] = dot;
}

__global__ void __launch_bounds__(256) k_fc_cg_x(KrylovWork w, FcCg c, const double* __restrict__ q) {
    __shared__ double smem[8];
    const FcChunk ch = c.chunks[blockIdx.x];
    if (!c.running[ch.tissue]) return;
    const double rho = tissue_total(c, c.part, ch.tissue, smem);
    const double pq = tissue_total(c, c.part + c.n_chunks, ch.tissue, smem);
    const double alpha = rho / pq;
    double s = 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += blockDim.x) {
        w.x[i] += alpha * w.p[i];
        const double r = w.r[i] - alpha * q[i];
        w.r[i] = r;
        s += r * r;
    }
    s = block_total(s, smem);
    if (threadIdx.x == 0) c.part[2 * c.n_chunks + blockIdx.x] = s;
}

// The tissue's test: converged, out of iterations, or still running. A step that does not look like
// one of a (nearly) exact preconditioner - (r, z) and (p, J p) of opposite sign, or a residual that
// grows - ends with KS_INDEFINITE, and the caller takes another path.
__global__ void __launch_bounds__(256) k_fc_cg_test(FcCg c) {
    __shared__ double smem[8];
    const int t = blockIdx.x;
    if (!c.running[t]) return;
    const double rho = tissue_total(c, c.part, t, smem), pq = tissue_total(c, c.part + c.n_chunks, t, smem);
    const double rr = tissue_total(c, c.part + 2 * c.n_chunks, t, smem);
    if (threadIdx.x) return;
    KrylovScalars& k = c.sc[t];
    const double before = k.rr;
    k.rr = rr;
    k.rho_prev = rho;
    ++k.iter;
    if (!isfinite(rr) || !isfinite(rho) || !isfinite(pq))
        k.status = KS_NONFINITE;
    else if (rr <= k.tol2)
        k.status = KS_CONVERGED;
    else if (!(rho * pq > 0.0) || rr > before)
        k.status = KS_INDEFINITE;
    else if (k.iter >= k.max_iter)
        k.status = KS_MAXIT;
    if (k.status != KS_RUNNING) c.running[t] = 0;
}

cudaError_t opt_in(const void* f, int bytes) { return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }

}  // namespace

#define FC_CK(call)                                  \
    do {                                             \
        const cudaError_t err_ = (call);             \
        if (err_ != cudaSuccess) return err_;        \
    } while (0)

cudaError_t launch_factor(const FcPlan& plan, const FcWork& w, const double* vals, int64_t* launches, cudaStream_t s) {
    // per-device attributes of the kernels; cheap next to a factorisation
    FC_CK(opt_in((const void*)k_fc_col, kPanelSmem));
    FC_CK(opt_in((const void*)k_fc_upd, kPanelSmem));
    FC_CK(opt_in((const void*)k_fc_l21, kGemmSmem));
    FC_CK(opt_in((const void*)k_fc_schur, kGemmSmem));
    int64_t n = 0;
    for (int d = (int)plan.depths.size() - 1; d >= 0; --d) {
        const FcDepth& L = plan.depths[d];
        if (L.gather.count) {
            const int pmax = plan.fronts[plan.tasks[L.gather.begin].front].p;  // the list starts with the largest
            k_fc_gather<<<L.gather.count, 256, pmax * sizeof(int2), s>>>(w, L.gather.begin, d & 1);
            ++n;
        }
        if (L.scatter.count) {
            k_fc_scatter<<<L.scatter.count, 256, 0, s>>>(w, vals, L.scatter.begin);
            ++n;
        }
        if (L.diag.count) {
            k_fc_diag<<<L.diag.count, 256, 0, s>>>(w, L.diag.begin);
            ++n;
        }
        for (int k = 0; k < L.n_panel; ++k) {
            const FcPanel& P = plan.panels[L.panel0 + k];
            if (P.col.count) {
                k_fc_col<<<P.col.count, 256, kPanelSmem, s>>>(w, P.col.begin, k);
                ++n;
            }
            if (P.upd.count) {
                k_fc_upd<<<P.upd.count, 256, kPanelSmem, s>>>(w, P.upd.begin, k);
                ++n;
            }
        }
        if (L.l21.count) {
            k_fc_l21<<<L.l21.count, 128, kGemmSmem, s>>>(w, L.l21.begin);
            ++n;
        }
        if (L.schur.count) {
            k_fc_schur<<<L.schur.count, 128, kGemmSmem, s>>>(w, L.schur.begin, d & 1);
            ++n;
        }
    }
    *launches += n;
    return cudaGetLastError();
}

cudaError_t launch_factor_solve(const FcPlan& plan, const FcWork& w, const double* in, double* x, int64_t* launches,
                                cudaStream_t s) {
    int64_t n = 0;
    const int depths = (int)plan.depths.size();
    for (int d = depths - 1; d >= 0; --d) {
        const FcDepth& L = plan.depths[d];
        if (L.fwd1.count) {
            const int pmax = plan.fronts[plan.tasks[L.fwd1.begin].front].p;
            k_fc_fwd1<<<L.fwd1.count, 256, pmax * sizeof(double), s>>>(w, in, L.fwd1.begin);
            ++n;
        }
        if (L.fwd2.count) {
            k_fc_fwd2<<<L.fwd2.count, 256, 0, s>>>(w, L.fwd2.begin);
            ++n;
        }
    }
    for (int d = 0; d < depths; ++d) {
        const FcDepth& L = plan.depths[d];
        if (L.bwd1.count) {
            k_fc_bwd1<<<L.bwd1.count, 256, 0, s>>>(w, x, L.bwd1.begin);
            ++n;
        }
        if (L.bwd2.count) {
            const int pmax = plan.fronts[plan.tasks[L.bwd2.begin].front].p;
            k_fc_bwd2<<<L.bwd2.count, 256, pmax * sizeof(double), s>>>(w, x, L.bwd2.begin);
            ++n;
        }
    }
    *launches += n;
    return cudaGetLastError();
}

cudaError_t launch_fc_start(const KrylovWork& w, const FcCg& c, double rtol, int max_iter, cudaStream_t s) {
    k_fc_cg_start<<<c.n_chunks, 256, 0, s>>>(w, c);
    k_fc_cg_begin<<<c.T, 256, 0, s>>>(c, rtol, max_iter);
    return cudaGetLastError();
}

cudaError_t launch_fc_iteration(const KrylovWork& w, const FcCg& c, const double* z, double* q, cudaStream_t s) {
    k_fc_cg_dot<<<c.n_chunks, 256, 0, s>>>(w, c, z);
    k_fc_cg_p<<<c.n_chunks, 256, 0, s>>>(w, c, z);
    k_fc_cg_spmv<<<c.n_chunks, 256, 0, s>>>(w, c, q);
    k_fc_cg_x<<<c.n_chunks, 256, 0, s>>>(w, c, q);
    k_fc_cg_test<<<c.T, 256, 0, s>>>(c);
    return cudaGetLastError();
}

}  // namespace tfb
