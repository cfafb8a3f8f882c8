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
//   k_fc_l21       l21 = A21 x11^T S
//   k_fc_schur     C = children - l21 S l21^T, and w21 = l21 x11
//   k_fc_small     all of it for a front of one panel and a short boundary
// A wing disc of 79,650 prisms (4.3e10 operations): 5.0 ms, of which the Schur and w21 tiles 2.1, the chain of
// 68 panels 1.8, l21 0.7, the gathers 0.3, the small fronts 0.4 behind others; 1.2 ms would be the tensor rate.
// A pass: 0.37 ms for twice the factor's 519 MB (0.16 ms at the copy rate).
#include <math.h>

#include "tf_factor.cuh"

namespace tfb {
namespace {

constexpr int kT = kFcTile;
constexpr int kLd = kT + 4;  // shared leading dimension: 8-byte reads of a fragment hit distinct banks
constexpr int kKc = 16;      // K extent of one stage of the long GEMMs
constexpr int kKld = kKc + 4;
constexpr int kStages = 2;

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// base[off] where ok, else 0, without a branch: a load behind a branch is waited for before the next one
// is issued, and the gathers below live on having all of theirs in flight (base is always readable).
__device__ __forceinline__ double load_if(const double* __restrict__ base, bool ok, size_t off) {
    const double v = base[ok ? off : 0];
    return ok ? v : 0.0;
}

// Programmatic dependent launch: a kernel of a chain lets the next one start when its own CTAs have, and waits
// for the end of the one before it after it has read its part of the plan (which nothing writes) - the launch
// and two or three of the dependent loads of every link then overlap the previous kernel. Every CTA waits, also
// one with nothing to do: the end of a kernel then means the end of all before it. What earlier kernels
// of the chain write is not reached through `const __restrict__`, which would let a load move above the wait.
// Step of a wing disc of 23,876 prisms 7.39 -> 6.69 ms, of a disc of 2,661 2.73 -> 2.53.
__device__ __forceinline__ void chain_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void prefetch(const double* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A parameter's array indexed by a variable is copied to local memory (128 bytes a thread); two of it are not.
__device__ __forceinline__ double* contrib(const FcWork& w, int parity) { return parity ? w.contrib[1] : w.contrib[0]; }

// ---- assembly of a front -------------------------------------------------------------------

// Rows [i j, (i + 1) j) of the front's pivot columns (task j: 8 or 32): what its children left there. Rows below p
// need the columns up to the diagonal only.
__global__ void __launch_bounds__(256) k_fc_gather(FcWork w, int begin, int parity) {
    extern __shared__ int2 s_col[];  // per pivot column: its index on either child's boundary
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    const int2* kids = w.kids + F.ent;
    for (int c = threadIdx.x; c < F.p; c += blockDim.x) s_col[c] = kids[c];
    __syncthreads();
    chain_wait();
    if (!w.active[F.tissue]) return;
    const double* __restrict__ C0 = F.child[0] >= 0 ? contrib(w, parity ^ 1) + F.child_c[0] : w.factor;
    const double* __restrict__ C1 = F.child[1] >= 0 ? contrib(w, parity ^ 1) + F.child_c[1] : w.factor;
    const int ld0 = F.child_ldb[0], ld1 = F.child_ldb[1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r1 = min((tk.i + 1) * tk.j, F.p + F.b);
    for (int row = tk.i * tk.j + warp; row < r1; row += 8) {
        const int2 k = kids[row];
        const double* R0 = C0 + (k.x >= 0 ? (size_t)k.x * ld0 : 0);
        const double* R1 = C1 + (k.y >= 0 ? (size_t)k.y * ld1 : 0);
        const int n = row < F.p ? row + 1 : F.p;
        double* out = row < F.p ? w.factor + F.x11 + (size_t)row * F.ldp : w.scratch + F.a21 + (size_t)(row - F.p) * F.ldp;
        for (int c = lane; c < n; c += 128) {
            double x0[4], x1[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int2 m = c + 32 * u < n ? s_col[c + 32 * u] : make_int2(-1, -1);
                x0[u] = load_if(R0, k.x >= 0 && m.x >= 0, m.x);
                x1[u] = load_if(R1, k.y >= 0 && m.y >= 0, m.y);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c + 32 * u < n) out[c + 32 * u] = x0[u] + x1[u];
        }
    }
}

// Entry (rr, cc) that Jacobian block k (of jblk) adds to a front: the block is read from the earlier pivot's row
// of J, transposed; of an unsymmetric J the mean with its mirror image.
__device__ __forceinline__ double j_entry(const FcWork& w, const double* __restrict__ vals, int k, int block, int cc, int rr) {
    const double v = vals[(size_t)block * 9 + cc * 3 + rr];
    return w.jblk_t ? 0.5 * (v + vals[(size_t)w.jblk_t[k] * 9 + rr * 3 + cc]) : v;
}

// += the front's Jacobian blocks. Block (column k, row i) of the lower triangle is read from row k of
// J, transposed; each lands on entries of its own (one addition each: the order does not matter).
__global__ void __launch_bounds__(256) k_fc_scatter(FcWork w, const double* __restrict__ vals, int begin) {
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    const int b0 = F.j0 + tk.i * kFcScatter, b1 = min(b0 + kFcScatter, F.j1), n9 = (b1 - b0) * 9;
    // all of a thread's entries at once, before the wait (the Jacobian is older than the chain), and added
    // without reading the sums back: one entry after the other took 12.7 us
    constexpr int kPer = kFcScatter * 9 / 256;
    double v[kPer];
    double* out[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int e = min((int)threadIdx.x + u * 256, n9 - 1), k = e / 9, en = e - k * 9, cc = en / 3, rr = en - cc * 3;
        const int2 jb = w.jblk[b0 + k];
        const int row = (int)((uint32_t)jb.y >> 16) + rr, col = (jb.y & 0xffff) + cc;
        double* at = row < F.p ? w.factor + F.x11 + (size_t)row * F.ldp + col
                               : w.scratch + F.a21 + (size_t)(row - F.p) * F.ldp + col;
        // not the upper half of a node's own block
        out[u] = (int)threadIdx.x + u * 256 < n9 && col <= row ? at : nullptr;
        v[u] = j_entry(w, vals, b0 + k, jb.x, cc, rr);
    }
    chain_wait();
    if (!w.active[F.tissue]) return;
#pragma unroll
    for (int u = 0; u < kPer; ++u)
        if (out[u]) atomicAdd(out[u], v[u]);
}

// ---- pivot block -----------------------------------------------------------------------------

// LDL^T of an n x n block (n <= 64, its lower triangle in s, rows of ld), by the row operations that also
// turn the identity into L^-1, in place: 8 warps, warp w holds rows 8 w .. 8 w + 7 as the accumulator
// fragments of eight 8 x 8 tiles. Per block of 8 pivots every warp below it eliminates the pivot tile
// and its own tile of those columns by shuffles (the pivot tile redundantly, so that the 8 steps need no
// barrier), and its other tiles by two tensor instructions each. Returns the rows of
// G^-1 = |D|^-1/2 L^-1 (zero right of the diagonal and outside the block) and writes sign(D). A zero pivot leaves
// non-finite values, which the solve's first residual shows.
// Bound by the chain of 8 steps a block (each a shuffle, a reciprocal and two FP64 operations one after the
// other, 187 to 220 cycles), 350 cycles a pivot with the hand-over and the products: 64 pivots take 22.4 k. A row
// per four threads with the pivot row read from shared memory took 571 cycles a step (64 pivots:
// 36.6 k): 256 threads x 16 entries a step is 256 cycles of shared-memory reads alone.
struct __align__(16) FactorShared {
    double rows[2][8][kLd];
    double d[kT];
};
__device__ __forceinline__ void factor_block(const double* s, int ld, int n, FactorShared& sh, double (&v)[8][2], double* sign,
                                             int32_t* neg) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, lr = lane >> 2, lk = lane & 3, r = 8 * w + lr;
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 8 * t + 2 * lk + h;
            v[t][h] = r < n && c < n ? (c <= r ? s[r * ld + c] : s[c * ld + r]) : (r == c ? 1.0 : 0.0);
        }
#pragma unroll 1  // one copy of the eight steps: eight of them, 64 KB of code, ran from instruction-cache misses
    for (int kb = 0; 8 * kb < n; ++kb) {
        double(*rows)[kLd] = sh.rows[kb & 1];
        if (w == kb) {
#pragma unroll
            for (int t = 0; t < 8; ++t) *reinterpret_cast<double2*>(&rows[lr][8 * t + 2 * lk]) = make_double2(v[t][0], v[t][1]);
        }
        __syncthreads();
        if (w < kb) continue;
        double D[2] = {rows[lr][8 * kb + 2 * lk], rows[lr][8 * kb + 2 * lk + 1]};
        double O[2] = {v[0][0], v[0][1]};
#pragma unroll
        for (int t = 1; t < 8; ++t)
            if (t == kb) {
                O[0] = v[t][0];
                O[1] = v[t][1];
            }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double d = __shfl_sync(0xffffffffu, D[j & 1], 4 * j + (j >> 1));
            const double p0 = __shfl_sync(0xffffffffu, D[0], 4 * j + lk), p1 = __shfl_sync(0xffffffffu, D[1], 4 * j + lk);
            const double aD = __shfl_sync(0xffffffffu, D[j & 1], (lane & 28) + (j >> 1));
            const double aO = __shfl_sync(0xffffffffu, O[j & 1], (lane & 28) + (j >> 1));
            const double inv = __drcp_rn(d);
            const double mD = lr > j ? aD * inv : 0.0, mO = aO * inv;
            O[0] -= mO * p0;
            O[1] -= mO * p1;
            D[0] -= mD * p0;
            D[1] -= mD * p1;
            if (lk == (j >> 1)) {
                O[j & 1] = -mO;
                if (lr > j) D[j & 1] = -mD;
            }
            if (w == kb && lane == 0) sh.d[8 * kb + j] = d;
        }
        if (w == kb) {
            O[0] = D[0];
            O[1] = D[1];
        }
        // the tile as an A fragment: below the pivots minus the multipliers of the published rows; for the pivot
        // rows L^-1 itself (unit diagonal)
        double a[2];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            const int src = (lane & 28) + 2 * f + (lk >> 1), k = 4 * f + lk;
            const double x0 = __shfl_sync(0xffffffffu, O[0], src), x1 = __shfl_sync(0xffffffffu, O[1], src);
            a[f] = lk & 1 ? x1 : x0;
            if (w == kb) a[f] = k < lr ? a[f] : (k == lr ? 1.0 : 0.0);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            if (t == kb) {
                v[t][0] = O[0];
                v[t][1] = O[1];
                continue;
            }
            if (w == kb) v[t][0] = v[t][1] = 0.0;
            mma_f64(v[t], a[0], rows[lk][8 * t + lr]);
            mma_f64(v[t], a[1], rows[4 + lk][8 * t + lr]);
        }
    }
    __syncthreads();
    const double d = r < n ? sh.d[r] : 1.0;
    const double g = r < n ? 1.0 / sqrt(fabs(d)) : 0.0;
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 8 * t + 2 * lk + h;
            v[t][h] = c < r ? v[t][h] * g : (c == r ? g : 0.0);
        }
    if (r < n && lk == 0) {
        sign[r] = d < 0.0 ? -1.0 : 1.0;
        if (d < 0.0) *neg = 1;
    }
}

// factor_block's rows to memory (rows and columns below n).
__device__ __forceinline__ void store_rows(const double (&v)[8][2], int n, double* out, int ld) {
    const int lane = threadIdx.x & 31, r = 8 * (threadIdx.x >> 5) + (lane >> 2);
    if (r >= n) return;
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 8 * t + 2 * (lane & 3) + h;
            if (c < n) out[(size_t)r * ld + c] = v[t][h];
        }
}

// A 64 x 64 tile of a matrix with `rows` x `cols` valid entries at src (its rows 16-byte aligned) into
// shared memory, zero outside, by asynchronous copies of two entries: both tiles of a product are
// in flight together. Follow with tile_wait.
__device__ __forceinline__ void load_tile(double (*s)[kLd], const double* src, int ld, int rows, int cols) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int id = threadIdx.x + e * 256, r = id >> 5, c = (id & 31) * 2, left = r < rows ? cols - c : 0;
        const int bytes = left >= 2 ? 16 : (left > 0 ? 8 : 0);
        cp_async16(&s[r][c], bytes ? src + (size_t)r * ld + c : src, bytes);
    }
}
__device__ __forceinline__ void tile_wait() {
    cp_commit();
    cp_wait<0>();
    __syncthreads();
}

__global__ void __launch_bounds__(256) k_fc_diag(FcWork w, int begin) {
    __shared__ __align__(16) double s[kT][kLd];
    __shared__ FactorShared sh;
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    chain_wait();
    if (!w.active[F.tissue]) return;
    double* A = w.factor + F.x11;
    const int n = min(kT, F.p);
    load_tile(s, A, F.ldp, n, n);  // above the diagonal: not initialised, and not read
    tile_wait();
    double v[8][2];
    factor_block(&s[0][0], kLd, n, sh, v, w.sign + F.piv, w.neg + tk.front);
    store_rows(v, n, A, F.ldp);
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

__device__ __forceinline__ void tile_sub(double (&a)[2][4][2], const double (&b)[2][4][2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) a[i][j][h] -= b[i][j][h];
}

constexpr int kPanelSmem = 2 * kT * kLd * (int)sizeof(double);

// Panel k, G_k^-1 known. Task (i > k, part): 16 rows of L_ik = A_ik G_k^-T S_k into the panel scratch; (i < k, part): 16
// columns of the inverse's row panel, X_ki = G_k^-1 X_ki in place. Quarter tiles: these launches are on the
// critical path with few tiles (22 tiles of the wing disc's second depth: 9.4 us whole).
__global__ void __launch_bounds__(256) k_fc_col(FcWork w, int begin, int k) {
    extern __shared__ double s_dyn[];
    double(*sA)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn);
    double(*sB)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn + kT * kLd);
    chain_go();
    const FcTask tk = w.tasks[begin + (blockIdx.x >> 2)];
    const FcFront F = w.fronts[tk.front];
    chain_wait();
    if (!w.active[F.tissue]) return;
    double* X = w.factor + F.x11;
    const int i = tk.i, part = (blockIdx.x & 3) * 16, nk = min(kT, F.p - k * kT), ni = min(kT, F.p - i * kT);
    const double* Gk = X + (size_t)k * kT * F.ldp + k * kT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lk = lane & 3;
    if (i > k) {
        if (part >= ni) return;
        const double* A = X + ((size_t)i * kT + part) * F.ldp + k * kT;
        {
            const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;  // 16 rows x 64 columns
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int left = part + r < ni ? nk - (c + 2 * h) : 0, bytes = left >= 2 ? 16 : (left > 0 ? 8 : 0);
                cp_async16(&sA[r][c + 2 * h], bytes ? A + (size_t)r * F.ldp + c + 2 * h : A, bytes);
            }
        }
        load_tile(sB, Gk, F.ldp, nk, nk);
        tile_wait();
        double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};  // warp: columns 8 warp .. 8 warp + 7, 16 rows
        const int kend = min(kT, 8 * warp + 8);       // G_k^-1 is lower triangular
        for (int q = lk; q < kend; q += 4) {
            const double b = sB[8 * warp + lr][q];
            mma_f64(acc[0], sA[lr][q], b);
            mma_f64(acc[1], sA[8 + lr][q], b);
        }
        double* lp = w.scratch + F.lp + ((size_t)i * kT + part) * kT;
        const double* sg = w.sign + F.piv + k * kT;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 8 * x + lr, c = 8 * warp + 2 * lk + h;
                if (part + r < ni) lp[r * kT + c] = c < nk ? acc[x][h] * sg[c] : 0.0;
            }
    } else {
        double* Xk = X + (size_t)k * kT * F.ldp + i * kT + part;
        {
            const int r = threadIdx.x >> 2, c = (threadIdx.x & 3) * 4;  // 64 rows x 16 columns
#pragma unroll
            for (int h = 0; h < 2; ++h)
                cp_async16(&sB[r][c + 2 * h], r < nk ? Xk + (size_t)r * F.ldp + c + 2 * h : Xk, r < nk ? 16 : 0);
        }
        load_tile(sA, Gk, F.ldp, nk, nk);
        tile_wait();
        double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};  // warp: rows 8 warp .. 8 warp + 7, 16 columns
        const int kend = min(kT, 8 * warp + 8);
        for (int q = lk; q < kend; q += 4) {
            const double a = sA[8 * warp + lr][q];
            mma_f64(acc[0], a, sB[q][lr]);
            mma_f64(acc[1], a, sB[q][8 + lr]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 8 * warp + lr, c = 8 * x + 2 * lk + h;
                if (r < nk) Xk[(size_t)r * F.ldp + c] = acc[x][h];
            }
    }
}

// Panel k, the tiles below it: A_ij -= L_ik S_k L_jk^T (j > k), X_ik = -L_ik G_k^-1, X_ij -= L_ik X_kj (j < k).
// The tile that is the next diagonal block is factorised at once.
__global__ void __launch_bounds__(256) k_fc_upd(FcWork w, int begin, int k) {
    extern __shared__ double s_dyn[];
    __shared__ FactorShared sh;
    double(*sA)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn);
    double(*sB)[kLd] = reinterpret_cast<double(*)[kLd]>(s_dyn + kT * kLd);
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    chain_wait();
    if (!w.active[F.tissue]) return;
    double* X = w.factor + F.x11;
    const int i = tk.i, j = tk.j;
    const int ni = min(kT, F.p - i * kT), nj = min(kT, F.p - j * kT), nk = min(kT, F.p - k * kT);
    const double* lp = w.scratch + F.lp;
    double* out = X + (size_t)i * kT * F.ldp + j * kT;
    double acc[2][4][2], old[2][4][2];
    tile_each(old, [&](int r, int c, double& v) {  // in flight during the product
        v = j != k && r < ni && c < nj && (i != j || c <= r) ? out[(size_t)r * F.ldp + c] : 0.0;
    });
    load_tile(sA, lp + (size_t)i * kT * kT, kT, ni, nk);
    if (j > k) {
        const double* sg = w.sign + F.piv + k * kT;
        const double sign = (int)threadIdx.x < nk ? sg[threadIdx.x] : 1.0;  // on its way with the tiles
        load_tile(sB, lp + (size_t)j * kT * kT, kT, nj, nk);
        cp_commit();
        cp_wait<0>();
        // Panel k's signs are of an earlier launch. The front's flag is not: the CTA of the next diagonal block sets
        // it in this one, and threads that read it for themselves could part ways around the barrier below.
        if (__syncthreads_or(sign < 0.0)) {
            for (int e = threadIdx.x; e < kT * kT; e += 256) sB[e >> 6][e & 63] *= (e & 63) < nk ? sg[e & 63] : 0.0;
            __syncthreads();
        }
        tile_mma<true>(sA, sB, acc);
        if (i == k + 1 && j == k + 1) {
            __syncthreads();
            tile_sub(old, acc);
            tile_each(old, [&](int r, int c, double v) { sA[r][c] = v; });
            __syncthreads();
            double v[8][2];
            factor_block(&sA[0][0], kLd, ni, sh, v, w.sign + F.piv + i * kT, w.neg + tk.front);
            store_rows(v, ni, out, F.ldp);
        } else {
            tile_sub(old, acc);
            tile_each(old, [&](int r, int c, double v) {
                if (r < ni && c < nj && (i != j || c <= r)) out[(size_t)r * F.ldp + c] = v;
            });
        }
        return;
    }
    load_tile(sB, X + (size_t)k * kT * F.ldp + j * kT, F.ldp, nk, j == k ? nk : kT);
    tile_wait();
    tile_mma<false>(sA, sB, acc);
    if (j == k)
        tile_each(acc, [&](int r, int c, double v) {
            if (r < ni && c < nk) out[(size_t)r * F.ldp + c] = -v;
        });
    else {
        tile_sub(old, acc);
        tile_each(old, [&](int r, int c, double v) {
            if (r < ni) out[(size_t)r * F.ldp + c] = v;
        });
    }
}

// ---- small fronts --------------------------------------------------------------------------------

// A front of at most 64 pivots and kFcSmallB boundary unknowns, all of it in one CTA: its [A11; A21] is
// gathered, completed with the Jacobian's blocks, factorised and turned into l21 in shared memory; w21 and
// the contribution are formed from there. One launch per depth instead of five, and A21 never leaves the
// SM; the bottom half of a tree is made of such fronts.
__global__ void __launch_bounds__(256, 3) k_fc_small(FcWork w, const double* __restrict__ vals, int begin, int parity) {
    extern __shared__ __align__(16) double s_dyn[];
    __shared__ FactorShared sh;
    __shared__ double s_sign[kT];
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    const int p = F.p, b = F.b, n = p + b, ld = fc_small_ld(p), p8r = (p + 7) & ~7, b16 = (b + 15) & ~15;
    double* sX = s_dyn;
    double* sL = sX + p8r * ld;
    int* s_map = reinterpret_cast<int*>(sL + b16 * ld);  // [2][n]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < n; e += 256) {
        const int2 k = w.kids[F.ent + e];
        s_map[e] = k.x;
        s_map[n + e] = k.y;
    }
    for (int e = tid; e < (p8r + b16) * ld; e += 256) s_dyn[e] = 0.0;
    __syncthreads();
    // the Jacobian's entries go straight to their places, in flight while the children's are read
    {
        const int n9 = (F.j1 - F.j0) * 9;
#pragma unroll 4
        for (int e = tid; e < n9; e += 256) {
            const int k = e / 9, en = e - k * 9, cc = en / 3, rr = en - cc * 3;
            const int2 jb = w.jblk[F.j0 + k];
            const int row = (int)((uint32_t)jb.y >> 16) + rr, col = (jb.y & 0xffff) + cc;
            double* dst = (row < p ? sX + row * ld : sL + (row - p) * ld) + col;
            if (w.jblk_t)
                *dst = j_entry(w, vals, F.j0 + k, jb.x, cc, rr);
            else
                cp_async8(dst, vals + (size_t)jb.x * 9 + en);
        }
        cp_commit();
    }
    chain_wait();  // the Jacobian is older than the chain
    if (!w.active[F.tissue]) {
        cp_wait<0>();
        return;
    }
    const double* __restrict__ C0 = F.child[0] >= 0 ? contrib(w, parity ^ 1) + F.child_c[0] : w.factor;
    const double* __restrict__ C1 = F.child[1] >= 0 ? contrib(w, parity ^ 1) + F.child_c[1] : w.factor;
    const int ld0 = F.child_ldb[0], ld1 = F.child_ldb[1];
    if (F.child[0] >= 0) {  // eight rows a warp pass, the loads of all of them in flight
        bool first = true;
        for (int r0 = warp; r0 < n; r0 += 64)
            for (int c = lane; c < ((p + 31) & ~31); c += 32) {
                const int c0 = c < p ? s_map[c] : -1, c1 = c < p ? s_map[n + c] : -1;
                double x[8], y[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int row = min(r0 + 8 * u, n - 1), m0 = s_map[row], m1 = s_map[n + row];
                    const bool in = r0 + 8 * u < n && (row >= p || c <= row);
                    x[u] = load_if(C0, in && m0 >= 0 && c0 >= 0, (size_t)m0 * ld0 + c0);
                    y[u] = load_if(C1, in && m1 >= 0 && c1 >= 0, (size_t)m1 * ld1 + c1);
                }
                if (first) {  // the same pass in every thread: the Jacobian's entries are in place
                    cp_wait<0>();
                    __syncthreads();
                    first = false;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int row = r0 + 8 * u;
                    if (row < n && c < p && (row >= p || c <= row)) (row < p ? sX + row * ld : sL + (row - p) * ld)[c] += x[u] + y[u];
                }
            }
        if (first) {  // a warp without rows
            cp_wait<0>();
            __syncthreads();
        }
    } else {
        cp_wait<0>();
    }
    __syncthreads();
    {
        double v[8][2];
        factor_block(sX, ld, p, sh, v, s_sign, w.neg + tk.front);
        store_rows(v, p, w.factor + F.x11, F.ldp);
        const int r = 8 * warp + (lane >> 2);  // every row of s was read before factor_block's last barrier
        if (r < p8r)
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (8 * t + 2 * (lane & 3) < ld)
                    *reinterpret_cast<double2*>(sX + r * ld + 8 * t + 2 * (lane & 3)) = make_double2(v[t][0], v[t][1]);
        __syncthreads();
        if (tid < p) w.sign[F.piv + tid] = s_sign[tid];
    }
    // l21 = A21 G^-T S, a strip of eight rows per warp: its A21 entries stay in registers, so it is
    // overwritten in place
    const int lr = lane >> 2, lk = lane & 3, p8 = (p + 7) >> 3;
    for (int r0 = warp * 8; r0 < b; r0 += 64) {
        double* strip = sL + (size_t)r0 * ld;
        double a[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) a[k] = 4 * k < p ? strip[lr * ld + 4 * k + lk] : 0.0;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j >= p8) break;
            double d[2] = {0.0, 0.0}, d2[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < 2 * j + 2; k += 2) {
                mma_f64(d, a[k], sX[(8 * j + lr) * ld + 4 * k + lk]);
                mma_f64(d2, a[k + 1], sX[(8 * j + lr) * ld + 4 * k + 4 + lk]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = 8 * j + 2 * lk + h;
                if (c < p) {
                    strip[lr * ld + c] = (d[h] + d2[h]) * s_sign[c];
                }
            }
        }
    }
    // w21 = l21 G^-1 straight to memory, strips again (a warp's own)
    __syncwarp();
    for (int r0 = warp * 8; r0 < b; r0 += 64) {
        const double* strip = sL + (size_t)r0 * ld;
        double a[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) a[k] = 4 * k < p ? strip[lr * ld + 4 * k + lk] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j >= p8) break;
            double d[2] = {0.0, 0.0}, d2[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 2 * j; k < 16; k += 2) {
                if (4 * k >= p) break;
                mma_f64(d, a[k], 4 * k + lk < p ? sX[(4 * k + lk) * ld + 8 * j + lr] : 0.0);
                mma_f64(d2, a[k + 1], 4 * k + 4 + lk < p ? sX[(4 * k + 4 + lk) * ld + 8 * j + lr] : 0.0);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = 8 * j + 2 * lk + h;
                if (c < p && r0 + lr < b) w.factor[F.w21 + (size_t)(r0 + lr) * F.ldp + c] = d[h] + d2[h];
            }
        }
    }
    __syncthreads();
    // contribution, 16 x 16 tiles of the lower triangle
    const bool neg = w.neg[tk.front] != 0;
    double* Cf = contrib(w, parity) + F.c;
    const int nt = b16 >> 4;
    for (int task = warp; task < nt * (nt + 1) / 2; task += 8) {
        int i = (int)((sqrtf(8.0f * task + 1.0f) - 1.0f) * 0.5f);
        while ((i + 1) * (i + 2) / 2 <= task) ++i;
        while (i * (i + 1) / 2 > task) --i;
        const int j = task - i * (i + 1) / 2;
        double acc[2][2][2];  // from minus the children's entries
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = i * 16 + 8 * x + lr, c = j * 16 + 8 * y + 2 * lk + h;
                    const bool in = r < b && c <= r;
                    const int rr = in ? p + r : 0, cc = in ? p + c : 0;
                    const int r0 = s_map[rr], c0 = s_map[cc], r1 = s_map[n + rr], c1 = s_map[n + cc];
                    acc[x][y][h] = -load_if(C0, in && r0 >= 0 && c0 >= 0, (size_t)r0 * ld0 + c0) -
                                   load_if(C1, in && r1 >= 0 && c1 >= 0, (size_t)r1 * ld1 + c1);
                }
        const double* A = sL + (i * 16 + lr) * ld + lk;
        const double* B = sL + (j * 16 + lr) * ld + lk;
#pragma unroll 2
        for (int k = 0; k < p; k += 4) {
            double av[2], bv[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) av[x] = A[8 * x * ld + k];
#pragma unroll
            for (int y = 0; y < 2; ++y) bv[y] = B[8 * y * ld + k];
            if (neg) {
                const double sg = k + lk < p ? s_sign[k + lk] : 0.0;
#pragma unroll
                for (int y = 0; y < 2; ++y) bv[y] *= sg;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y) mma_f64(acc[x][y], av[x], bv[y]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = i * 16 + 8 * x + lr, c = j * 16 + 8 * y + 2 * lk + h;
                    if (r < b && c <= r) Cf[(size_t)r * F.ldb + c] = -acc[x][y][h];
                }
    }
}

// ---- boundary GEMMs ---------------------------------------------------------------------------

// 64 x 64 tile of A B^T (BT: B as [column][k]) or A B (B as [k][column], b_rows columns valid), row-major, by 4 warps (32 x 32 each: 16 accumulator
// tiles hide the tensor instruction's latency), K in stages of 16 through a cp.async ring of two.
// a_rows / b_rows: valid rows (0 outside); K: valid columns; B's columns times sign unless it is null.
template <bool BT, class Init>
__device__ __forceinline__ void gemm_tile(const double* A, int lda, int a_rows, const double* B, int ldb, int b_rows, int K,
                                          const double* sign, double* smem, double (&acc)[4][4][2], Init init) {
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
            const int na_ = r < a_rows ? nb : 0;
            cp_async16(sa + (st * kT + r) * kKld + c, na_ ? A + (size_t)r * lda + k0 + c : A, na_);
            if (BT) {
                const int nb_ = r < b_rows ? nb : 0;
                cp_async16(sb + (st * kT + r) * kKld + c, nb_ ? B + (size_t)r * ldb + k0 + c : B, nb_);
            } else {  // 16 rows x 32 chunks
                const int kr = id >> 5, bc = (id & 31) * 2, bl = k0 + kr < K ? b_rows - bc : 0;
                const int nb_ = bl >= 2 ? 16 : (bl > 0 ? 8 : 0);
                cp_async16(sb + st * kT * kKld + kr * kLd + bc, nb_ ? B + (size_t)(k0 + kr) * ldb + bc : B, nb_);
            }
        }
    };
#pragma unroll
    for (int st = 0; st < kStages - 1; ++st) {
        if (st < n_it) load(st);
        cp_commit();
    }
    init();  // the accumulators, while the first stages are on their way
    const int ra = (warp >> 1) * 32 + (lane >> 2), rb = (warp & 1) * 32 + (lane >> 2), kk = lane & 3;
    for (int it = 0; it < n_it; ++it) {
        cp_wait<kStages - 2>();
        __syncthreads();
        if (it + kStages - 1 < n_it) load(it + kStages - 1);
        cp_commit();
        const double* pa = sa + ((it % kStages) * kT + ra) * kKld + kk;
        const double* pb = BT ? sb + ((it % kStages) * kT + rb) * kKld + kk : sb + (it % kStages) * kT * kKld + kk * kLd + rb;
#pragma unroll
        for (int k = 0; k < kKc; k += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = pa[8 * i * kKld + k];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = BT ? pb[8 * j * kKld + k] : pb[k * kLd + 8 * j];
            if (sign) {
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
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    chain_wait();
    if (!w.active[F.tissue]) return;
    const int i = tk.i, j = tk.j, ni = min(kT, F.b - i * kT), nj = min(kT, F.p - j * kT);
    double acc[4][4][2];
    gemm_tile<true>(w.scratch + F.a21 + (size_t)i * kT * F.ldp, F.ldp, ni, w.factor + F.x11 + (size_t)j * kT * F.ldp, F.ldp, nj,
                     min(F.p, (j + 1) * kT), nullptr, s_dyn, acc, [&] {
#pragma unroll
                 for (int a = 0; a < 4; ++a)
#pragma unroll
                     for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
             });
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp >> 1) * 32 + (lane >> 2), c0 = (warp & 1) * 32 + 2 * (lane & 3);
    double* out = w.scratch + F.l21 + (size_t)i * kT * F.ldp + j * kT;
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

// Contribution tile (i, j <= i): what the children left there minus l21 S l21^T. Or (j < 0) a tile of w21.
__global__ void __launch_bounds__(128, 4) k_fc_schur(FcWork w, int begin, int parity) {
    extern __shared__ __align__(16) double s_dyn[];
    __shared__ int s_map[2][2][kT];  // child, rows / columns
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    chain_wait();
    if (!w.active[F.tissue]) return;
    const int i = tk.i, j = tk.j, ni = min(kT, F.b - i * kT), nj = min(kT, F.b - j * kT);
    const double* L = w.scratch + F.l21;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp >> 1) * 32 + (lane >> 2), c0 = (warp & 1) * 32 + 2 * (lane & 3);
    double acc[4][4][2];
    if (j < 0) {  // w21 tile: l21 x11, x11 lower triangular
        const int k0 = (-1 - j) * kT, np = min(kT, F.p - k0);
        gemm_tile<false>(L + (size_t)i * kT * F.ldp + k0, F.ldp, ni, w.factor + F.x11 + (size_t)k0 * F.ldp + k0, F.ldp, np,
                         F.p - k0, nullptr, s_dyn, acc, [&] {
#pragma unroll
                             for (int a = 0; a < 4; ++a)
#pragma unroll
                                 for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
                         });
        double* out = w.factor + F.w21 + (size_t)i * kT * F.ldp + k0;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = r0 + 8 * a, c = c0 + 8 * b + h;
                    if (r < ni && c < np) out[(size_t)r * F.ldp + c] = acc[a][b][h];
                }
        return;
    }
    for (int e = threadIdx.x; e < 4 * kT; e += blockDim.x) {
        const int q = e >> 7, side = (e >> 6) & 1, c = e & 63, idx = (side ? j : i) * kT + c;
        const int2 k = idx < F.b ? w.kids[F.ent + F.p + idx] : make_int2(-1, -1);
        s_map[q][side][c] = q ? k.y : k.x;
    }
    const double* __restrict__ C0 = F.child[0] >= 0 ? contrib(w, parity ^ 1) + F.child_c[0] : w.factor;
    const double* __restrict__ C1 = F.child[1] >= 0 ? contrib(w, parity ^ 1) + F.child_c[1] : w.factor;
    const int ld0 = F.child_ldb[0], ld1 = F.child_ldb[1];
    // the product accumulates onto minus the children's entries, so that nothing but stores follows it
    gemm_tile<true>(L + (size_t)i * kT * F.ldp, F.ldp, ni, L + (size_t)j * kT * F.ldp, F.ldp, nj, F.p,
              w.neg[tk.front] ? w.sign + F.piv : nullptr, s_dyn, acc, [&] {
                  __syncthreads();  // s_map
#pragma unroll
                  for (int a = 0; a < 4; ++a) {
                      const int r = r0 + 8 * a, m0 = s_map[0][0][r], m1 = s_map[1][0][r];
#pragma unroll
                      for (int b = 0; b < 4; ++b)
#pragma unroll
                          for (int h = 0; h < 2; ++h) {
                              const int c = c0 + 8 * b + h, k0 = s_map[0][1][c], k1 = s_map[1][1][c];
                              const bool in = i != j || c <= r;
                              acc[a][b][h] = -load_if(C0, in && m0 >= 0 && k0 >= 0, (size_t)m0 * ld0 + k0) -
                                             load_if(C1, in && m1 >= 0 && k1 >= 0, (size_t)m1 * ld1 + k1);
                          }
                  }
              });
    double* out = contrib(w, parity) + F.c + (size_t)i * kT * F.ldb + j * kT;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * a, c = c0 + 8 * b + h;
                if (r < ni && c < nj && (i != j || c <= r)) out[(size_t)r * F.ldb + c] = -acc[a][b][h];
            }
}

// ---- solve -------------------------------------------------------------------------------------

__global__ void k_fc_expand(FcWork w, const int32_t* __restrict__ maps, const int32_t* __restrict__ verts) {
    const FcFront F = w.fronts[blockIdx.x];
    for (int e = threadIdx.x; e < F.p + F.b; e += blockDim.x) {
        const int v = e / w.gd, r = e - v * w.gd;
        const int k0 = F.child[0] >= 0 ? maps[F.map[0] + v] : -1, k1 = F.child[1] >= 0 ? maps[F.map[1] + v] : -1;
        w.kids[F.ent + e] = make_int2(k0 >= 0 ? k0 * w.gd + r : -1, k1 >= 0 ? k1 * w.gd + r : -1);
        w.dofs[F.ent + e] = verts[F.verts + v] * w.gd + r;
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Up: rows [i j, (i + 1) j) of [z; v_B] = [x11; children - w21] v_P, v_P the right-hand side plus the children's
// vectors. A row is read by 8 lanes (few pivots) or by a warp, two entries at a time, four such reads in
// flight: one entry at a time both passes were bound by their instructions (58 % issue slots busy).
// Rows are zero from the diagonal to the end of its 64-column block, and in the padding to ldp.
template <int LANES>
__device__ __forceinline__ void up_rows(const FcWork& w, const FcFront& F, const double2* s_v, int r0, int r1) {
    constexpr int PER = 32 / LANES;  // rows of a warp side by side
    const int lane = threadIdx.x & 31, sub = lane % LANES;
    const double* X = w.factor + F.x11;  // rows p .. p + b - 1 of the kept factor are w21
    for (int base = r0 + (threadIdx.x >> 5) * PER; base < r1; base += 8 * PER) {
        const int r = base + lane / LANES;
        const bool in = r < r1;
        const double2* A = reinterpret_cast<const double2*>(X + (size_t)(in ? r : r0) * F.ldp);
        double kid = 0.0;
        if (sub == 0) {
            const int2 q = in && r >= F.p ? w.kids[F.ent + r] : make_int2(-1, -1);
            kid = load_if(w.vec, q.x >= 0, F.child_vec[0] + q.x) + load_if(w.vec, q.y >= 0, F.child_vec[1] + q.y);
        }
        const int n = !in ? 0 : (r < F.p ? min(F.ldp, (r | (kT - 1)) + 1) : F.ldp) >> 1;
        double s = 0.0, s2 = 0.0;
        int c = sub;
        for (; c + 3 * LANES < n; c += 4 * LANES) {
            double2 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = A[c + u * LANES];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double2 v = s_v[c + u * LANES];
                s += x[u].x * v.x;
                s2 += x[u].y * v.y;
            }
        }
        if (c < n) {
            double2 x[3];
#pragma unroll
            for (int u = 0; u < 3; ++u) x[u] = A[min(c + u * LANES, n - 1)];
#pragma unroll
            for (int u = 0; u < 3; ++u)
                if (c + u * LANES < n) {
                    const double2 v = s_v[c + u * LANES];
                    s += x[u].x * v.x;
                    s2 += x[u].y * v.y;
                }
        }
        s += s2;
#pragma unroll
        for (int off = LANES / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (sub == 0 && in) *(r < F.p ? w.z + F.piv + r : w.vec + F.vec + r - F.p) = r < F.p ? s : kid - s;
    }
}

__global__ void __launch_bounds__(256) k_fc_up(FcWork w, const double* in, int begin) {
    extern __shared__ __align__(16) double s_vec[];  // v_P, padded with zero
    double* s_v = s_vec;
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    const int r0 = tk.i * tk.j, r1 = min(r0 + tk.j, F.p + F.b);
    int2 k[4];
    int d[4];
    auto entries = [&](int c0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = min(c0 + u * 256, F.p - 1);
            k[u] = w.kids[F.ent + c];
            d[u] = w.dofs[F.ent + c];
        }
    };
    if ((int)threadIdx.x < F.p) entries(threadIdx.x);
    // the factor is older than the chain: its rows may be on their way into L2 before the wait
    for (int o = threadIdx.x * 16; o < (r1 - r0) * F.ldp; o += 256 * 16) prefetch(w.factor + F.x11 + (size_t)r0 * F.ldp + o);
    chain_wait();
    if (!w.active[F.tissue]) return;
    for (int c0 = threadIdx.x; c0 < F.p; c0 += 4 * 256) {
        double x[4], y[4], z[4];
        if (c0 != (int)threadIdx.x) entries(c0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            x[u] = in[d[u]];
            y[u] = load_if(w.vec, k[u].x >= 0, F.child_vec[0] + k[u].x);
            z[u] = load_if(w.vec, k[u].y >= 0, F.child_vec[1] + k[u].y);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + u * 256 < F.p) s_v[c0 + u * 256] = x[u] + y[u] + z[u];
    }
    if (threadIdx.x == 0 && (F.p & 1)) s_v[F.p] = 0.0;
    __syncthreads();
    if (F.p <= 128)
        up_rows<8>(w, F, reinterpret_cast<const double2*>(s_v), r0, r1);
    else
        up_rows<32>(w, F, reinterpret_cast<const double2*>(s_v), r0, r1);
}

// Down: columns [i j, (i + 1) j) of x_P = [x11; w21]^T [S z; -x_B], j = 64 or 32: two columns a lane, one or two
// rows a warp at a time, the warps splitting the rows.
template <int COLS>
__device__ __forceinline__ void down_columns(const double* X, int ldp, const double* s_u, int rows, double* s_p) {
    constexpr int PER = 64 / COLS;  // rows of a warp side by side
    const int lane = threadIdx.x & 31, col = 2 * (lane % (COLS / 2)), group = (threadIdx.x >> 5) * PER + lane / (COLS / 2);
    const int step = (blockDim.x >> 5) * PER;
    const double* A = X + col + (size_t)group * ldp;
    const size_t hop = (size_t)step * ldp;
    double sa = 0.0, sb = 0.0;
    int r = group;
    for (; r + 3 * step < rows; r += 4 * step, A += 4 * hop) {
        double2 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = *reinterpret_cast<const double2*>(A + u * hop);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double v = s_u[r + u * step];
            sa += x[u].x * v;
            sb += x[u].y * v;
        }
    }
    if (r < rows) {
        double2 x[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) x[u] = *reinterpret_cast<const double2*>(r + u * step < rows ? A + u * hop : A);
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (r + u * step < rows) {
                const double v = s_u[r + u * step];
                sa += x[u].x * v;
                sb += x[u].y * v;
            }
    }
    *reinterpret_cast<double2*>(s_p + group * COLS + col) = make_double2(sa, sb);
}

__global__ void __launch_bounds__(1024) k_fc_down(FcWork w, double* x, int begin) {
    extern __shared__ double s_u[];  // [S z; -x_B] from row c0 on
    __shared__ __align__(16) double s_p[32 * 64];
    __shared__ double s_q[4][64];
    chain_go();
    const FcTask tk = w.tasks[begin + blockIdx.x];
    const FcFront F = w.fronts[tk.front];
    const int cols = tk.j, c0 = tk.i * cols, n = F.p + F.b, nt = blockDim.x;
    int d[4];
    auto entries = [&](int r) {
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = w.dofs[F.ent + F.p + min(r + u * nt, F.b - 1)];
    };
    if ((int)threadIdx.x < F.b) entries(threadIdx.x);
    for (int o = threadIdx.x; o < (n - c0) * (cols / 16); o += nt)
        prefetch(w.factor + F.x11 + (size_t)(c0 + o / (cols / 16)) * F.ldp + c0 + o % (cols / 16) * 16);
    chain_wait();
    if (!w.active[F.tissue]) return;
    for (int r = c0 + threadIdx.x; r < F.p; r += nt) s_u[r - c0] = w.sign[F.piv + r] * w.z[F.piv + r];
    for (int r = threadIdx.x; r < F.b; r += 4 * nt) {
        if (r != (int)threadIdx.x) entries(r);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double v = x[d[u]];
            if (r + u * nt < F.b) s_u[F.p + r + u * nt - c0] = -v;
        }
    }
    __syncthreads();
    // x11 is lower triangular, and zero above its diagonal within the 64 x 64 diagonal blocks; columns past the
    // last one read the next rows' entries (the last row's: the padding behind the factors) and are dropped
    const double* X = w.factor + F.x11 + (size_t)c0 * F.ldp + c0;
    if (cols == 64)
        down_columns<64>(X, F.ldp, s_u, n - c0, s_p);
    else
        down_columns<32>(X, F.ldp, s_u, n - c0, s_p);
    __syncthreads();
    const int groups = nt / cols * 2, c = threadIdx.x % cols, part = threadIdx.x / cols;
    if (part < 4) {
        double t = 0.0;
        for (int k = part; k < groups; k += 4) t += s_p[k * cols + c];
        s_q[part][c] = t;
    }
    __syncthreads();
    if (part == 0 && c0 + c < F.p) x[w.dofs[F.ent + c0 + c]] = s_q[0][c] + s_q[1][c] + s_q[2][c] + s_q[3][c];
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
    for (int k = c.chunk0[t] + threadIdx.x; k < c.chunk0[t + 1]; k += blockDim.x) s += __ldcg(part + k);
    return block_total(s, smem);
}
// Of the first two kinds of partials at once.
__device__ __forceinline__ double2 tissue_totals(const FcCg& c, int t, double* smem) {
    double s = 0.0, u = 0.0;
    for (int k = c.chunk0[t] + threadIdx.x; k < c.chunk0[t + 1]; k += blockDim.x) {
        s += __ldcg(c.part + k);
        u += __ldcg(c.part + c.n_chunks + k);
    }
    s = warp_sum(s);
    u = warp_sum(u);
    if ((threadIdx.x & 31) == 0) {
        smem[threadIdx.x >> 5] = s;
        smem[8 + (threadIdx.x >> 5)] = u;
    }
    __syncthreads();
    double2 r = make_double2(0.0, 0.0);
    for (int k = 0; k < 8; ++k) {
        r.x += smem[k];
        r.y += smem[8 + k];
    }
    __syncthreads();
    return r;
}

// True in every thread of the last CTA of the tissue to arrive, after all partials are visible.
__device__ __forceinline__ bool last_of_tissue(const FcCg& c, int t) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t n = (uint32_t)(c.chunk0[t + 1] - c.chunk0[t]);
        last = atomicAdd(&c.sc[t].ticket[0], 1u) == n - 1;
        if (last) c.sc[t].ticket[0] = 0u;
        __threadfence();
    }
    __syncthreads();
    return last;
}

__global__ void __launch_bounds__(256) k_fc_cg_start(KrylovWork w, FcCg c, double rtol, int max_iter) {
    __shared__ double smem[8];
    chain_go();
    const FcChunk ch = c.chunks[blockIdx.x];
    const int t = ch.tissue;
    chain_wait();
    if (!c.active[t]) {
        if (threadIdx.x == 0 && (int)blockIdx.x == c.chunk0[t]) c.running[t] = 0;
        return;
    }
    double s = 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += 256) {
        const double b = w.b[i];
        w.x[i] = 0.0;
        w.r[i] = b;
        s += b * b;
    }
    s = block_total(s, smem);
    if (threadIdx.x == 0) c.part[2 * c.n_chunks + blockIdx.x] = s;
    if (!last_of_tissue(c, t)) return;
    const double bb = tissue_total(c, c.part + 2 * c.n_chunks, t, smem);
    if (threadIdx.x == 0) {
        KrylovScalars& k = c.sc[t];
        k.bb = k.rr = bb;
        k.tol2 = rtol * rtol * bb;
        k.rho = k.rho_prev = 0.0;
        k.iter = 0;
        k.max_iter = max_iter;
        k.method = c.minres ? KM_MINIMAL_RESIDUAL : KM_CG;
        k.status = !isfinite(bb) ? KS_NONFINITE : (bb > 0.0 ? KS_RUNNING : KS_CONVERGED);
        c.running[t] = k.status == KS_RUNNING;
        c.host[t] = k;
    }
}

__global__ void __launch_bounds__(256) k_fc_cg_dot(KrylovWork w, FcCg c, const double* z) {
    __shared__ double smem[8];
    chain_go();
    const FcChunk ch = c.chunks[blockIdx.x];
    chain_wait();
    if (!c.running[ch.tissue]) return;
    double s = 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += 256) s += w.r[i] * z[i];
    s = block_total(s, smem);
    if (threadIdx.x == 0) c.part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_fc_cg_p(KrylovWork w, FcCg c, const double* z) {
    __shared__ double smem[8];
    chain_go();
    const FcChunk ch = c.chunks[blockIdx.x];
    chain_wait();
    if (!c.running[ch.tissue]) return;
    const double beta = tissue_total(c, c.part, ch.tissue, smem) / c.sc[ch.tissue].rho_prev;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += 256) w.p[i] = z[i] + beta * w.p[i];
}

// q = J p and the chunk's (p, q); eight lanes a row. FIRST: the first iteration, p = z, and (r, z) as
// well, so that it needs no kernel before this one. The minimal residual iteration is all first ones, with
// (r, q) and (q, q).
template <bool FIRST>
__global__ void __launch_bounds__(256) k_fc_cg_spmv(KrylovWork w, FcCg c, const double* z, double* q) {
    __shared__ double smem[8];
    chain_go();
    const FcChunk ch = c.chunks[blockIdx.x];
    const FcSpan js = fc_block_span(w.rowptr[ch.row0], w.rowptr[ch.row1]);
    for (int64_t o = js.begin + threadIdx.x * 16; o < js.end; o += 256 * 16) prefetch(w.vals + o);  // J is older than the chain
    chain_wait();
    if (!c.running[ch.tissue]) return;
    const double* pv = FIRST ? z : w.p;
    const int gl = threadIdx.x & 7;
    double dot = 0.0, rho = 0.0;
    for (int base = ch.row0; base < ch.row1; base += 32) {
        const int row = base + (threadIdx.x >> 3);
        double y0 = 0.0, y1 = 0.0, y2 = 0.0;
        if (row < ch.row1)
            for (int k = w.rowptr[row] + gl; k < w.rowptr[row + 1]; k += 8) {
                const double* B = w.vals + (size_t)k * 9;
                const double* x = pv + (size_t)w.colidx[k] * 3;
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
            const size_t i = (size_t)row * 3 + gl;
            const double p = pv[i];
            q[i] = y;
            if (FIRST) {
                const double m = c.minres ? y : p;
                w.p[i] = p;
                dot += y * m;
                rho += w.r[i] * m;
            } else {
                dot += y * p;
            }
        }
    }
    dot = block_total(dot, smem);
    if (FIRST) rho = block_total(rho, smem);
    if (threadIdx.x == 0) {
        c.part[c.n_chunks + blockIdx.x] = dot;
        if (FIRST) c.part[blockIdx.x] = rho;
    }
}

// x += alpha p, r -= alpha q, and the tissue's test by the last of its CTAs: converged, out of
// iterations, or still running. A step that does not look like one of a (nearly) exact preconditioner
// - (r, z) and (p, J p) of opposite sign, or a residual that does not fall - ends with KS_INDEFINITE,
// and the caller takes another path.
__global__ void __launch_bounds__(256) k_fc_cg_x(KrylovWork w, FcCg c, const double* q) {
    __shared__ double smem[16];
    chain_go();
    const FcChunk ch = c.chunks[blockIdx.x];
    const int t = ch.tissue;
    chain_wait();
    if (!c.running[t]) return;
    const double2 both = tissue_totals(c, t, smem);
    const double rho = both.x, pq = both.y, alpha = rho / pq;
    double s = 0.0;
    for (int i = 3 * ch.row0 + threadIdx.x; i < 3 * ch.row1; i += 256) {
        w.x[i] += alpha * w.p[i];
        const double r = w.r[i] - alpha * q[i];
        w.r[i] = r;
        s += r * r;
    }
    s = block_total(s, smem);
    if (threadIdx.x == 0) c.part[2 * c.n_chunks + blockIdx.x] = s;
    if (!last_of_tissue(c, t)) return;
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
    else if (!(rho * pq > 0.0) || rr > (c.minres ? 0.25 * before : before))
        k.status = KS_INDEFINITE;
    else if (k.iter >= k.max_iter)
        k.status = KS_MAXIT;
    if (k.status != KS_RUNNING) c.running[t] = 0;
    c.host[t] = k;
}

// Launches kernels of a stream one after the other, each but the first as a link of a chain.
struct Chain {
    cudaStream_t stream;
    bool linked = false;
    template <class... P, class... A>
    cudaError_t operator()(void (*kernel)(P...), int grid, int threads, size_t smem, A... args) {
        cudaLaunchAttribute a{};
        a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        a.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t c{};
        c.gridDim = dim3((unsigned)grid);
        c.blockDim = dim3((unsigned)threads);
        c.dynamicSmemBytes = smem;
        c.stream = stream;
        c.attrs = &a;
        c.numAttrs = linked ? 1 : 0;
        linked = true;
        return cudaLaunchKernelEx(&c, kernel, P(args)...);
    }
};

cudaError_t opt_in(const void* f, int bytes) { return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }

}  // namespace

#define FC_CK(call)                                  \
    do {                                             \
        const cudaError_t err_ = (call);             \
        if (err_ != cudaSuccess) return err_;        \
    } while (0)

cudaError_t launch_factor(const FcPlan& plan, const FcWork& w, const double* vals, int64_t* launches, const FcStreams& st) {
    // per-device attributes of the kernels; cheap next to a factorisation
    FC_CK(opt_in((const void*)k_fc_small, fc_small_smem(kT, kFcSmallB)));
    FC_CK(opt_in((const void*)k_fc_col, kPanelSmem));
    FC_CK(opt_in((const void*)k_fc_upd, kPanelSmem));
    FC_CK(opt_in((const void*)k_fc_l21, kGemmSmem));
    FC_CK(opt_in((const void*)k_fc_schur, kGemmSmem));
    int64_t n = 0;
    Chain chain{st.main};
    for (int d = (int)plan.depths.size() - 1; d >= 0; --d) {
        const FcDepth& L = plan.depths[d];
        // The fronts of a depth do not depend on each other: each size of small fronts and the chain of the
        // others has a stream of its own, else a depth takes the sum of their latencies (a wing disc of
        // 23,876 prisms: 11 launches of small fronts, 35 to 120 us each, on 5 depths; 8.15 ms a
        // step like that, 7.39 side by side).
        bool main_free = L.gather.count == 0;
        bool forked[3] = {};
        FC_CK(cudaEventRecord(st.fork, st.main));
        for (int c = 0; c < 3; ++c) {
            const FcRange& r = L.small[c];
            if (r.count) {
                cudaStream_t s = st.main;
                if (!main_free) {
                    s = st.side[c];
                    forked[c] = true;
                    FC_CK(cudaStreamWaitEvent(s, st.fork, 0));
                }
                main_free = false;
                int smem = 0;
                for (int k = 0; k < r.count; ++k) {
                    const FcFront& F = plan.fronts[plan.tasks[r.begin + k].front];
                    smem = smem < fc_small_smem(F.p, F.b) ? fc_small_smem(F.p, F.b) : smem;
                }
                Chain alone{s};
                FC_CK((forked[c] ? alone : chain)(k_fc_small, r.count, 256, smem, w, vals, r.begin, d & 1));
                ++n;
                if (forked[c]) FC_CK(cudaEventRecord(st.join[c], s));
            }
        }
        if (L.gather.count) {
            const int pmax = plan.fronts[plan.tasks[L.gather.begin].front].p;  // the list starts with the largest
            FC_CK(chain(k_fc_gather, L.gather.count, 256, pmax * sizeof(int2), w, L.gather.begin, d & 1));
            ++n;
        }
        if (L.scatter.count) {
            FC_CK(chain(k_fc_scatter, L.scatter.count, 256, 0, w, vals, L.scatter.begin));
            ++n;
        }
        if (L.diag.count) {
            FC_CK(chain(k_fc_diag, L.diag.count, 256, 0, w, L.diag.begin));
            ++n;
        }
        for (int k = 0; k < L.n_panel; ++k) {
            const FcPanel& P = plan.panels[L.panel0 + k];
            if (P.col.count) {
                FC_CK(chain(k_fc_col, 4 * P.col.count, 256, kPanelSmem, w, P.col.begin, k));
                ++n;
            }
            if (P.upd.count) {
                FC_CK(chain(k_fc_upd, P.upd.count, 256, kPanelSmem, w, P.upd.begin, k));
                ++n;
            }
        }
        if (L.l21.count) {
            FC_CK(chain(k_fc_l21, L.l21.count, 128, kGemmSmem, w, L.l21.begin));
            ++n;
        }
        if (L.schur.count) {
            FC_CK(chain(k_fc_schur, L.schur.count, 128, kGemmSmem, w, L.schur.begin, d & 1));
            ++n;
        }
        for (int c = 0; c < 3; ++c)
            if (forked[c]) {
                FC_CK(cudaStreamWaitEvent(st.main, st.join[c], 0));
                chain.linked = false;
            }
    }
    *launches += n;
    return cudaGetLastError();
}

cudaError_t launch_factor_expand(const FcPlan& plan, const FcWork& w, const int32_t* maps, const int32_t* verts,
                                 cudaStream_t s) {
    k_fc_expand<<<(unsigned)plan.fronts.size(), 128, 0, s>>>(w, maps, verts);
    return cudaGetLastError();
}

cudaError_t launch_fc_iteration(const FcPlan& plan, const FcWork& f, const KrylovWork& w, const FcCg& c, bool first, double rtol,
                                int max_iter, double* z, double* q, int64_t* launches, cudaStream_t s) {
    FC_CK(opt_in((const void*)k_fc_down, kFcMaxFront * (int)sizeof(double)));
    int64_t n = 0;
    Chain chain{s};
    if (first) {
        FC_CK(chain(k_fc_cg_start, c.n_chunks, 256, 0, w, c, rtol, max_iter));
        ++n;
    }
    const int depths = (int)plan.depths.size();
    for (int d = depths - 1; d >= 0; --d) {
        const FcDepth& L = plan.depths[d];
        if (!L.fwd.count) continue;
        FC_CK(chain(k_fc_up, L.fwd.count, 256, L.fwd_smem, f, w.r, L.fwd.begin));
        ++n;
    }
    for (int d = 0; d < depths; ++d) {
        const FcDepth& L = plan.depths[d];
        if (!L.bwd.count) continue;
        FC_CK(chain(k_fc_down, L.bwd.count, L.bwd_threads, L.bwd_smem, f, z, L.bwd.begin));
        ++n;
    }
    if (first || c.minres) {
        FC_CK(chain(k_fc_cg_spmv<true>, c.n_chunks, 256, 0, w, c, z, q));
    } else {
        FC_CK(chain(k_fc_cg_dot, c.n_chunks, 256, 0, w, c, z));
        FC_CK(chain(k_fc_cg_p, c.n_chunks, 256, 0, w, c, z));
        FC_CK(chain(k_fc_cg_spmv<false>, c.n_chunks, 256, 0, w, c, z, q));
        n += 2;
    }
    FC_CK(chain(k_fc_cg_x, c.n_chunks, 256, 0, w, c, q));
    *launches += n + 2;
    return cudaGetLastError();
}

}  // namespace tfb
