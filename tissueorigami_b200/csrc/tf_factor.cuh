// tf_factor.cuh -- plan and kernel entry points of the sparse factorisation of a symmetric J.
//
// A tissue's unknowns are ordered by nested dissection: a small set of prism columns (a separator)
// splits the mesh in two halves that share no Jacobian block, each half is split again, and so on.
// Every separator (and every undivided piece at the bottom) is a front: its own unknowns, the
// pivots, and the boundary, the unknowns of enclosing separators its subtree touches. A front's
// dense matrix is its share of J plus what its (at most two) children left on their boundaries;
// eliminating its pivots leaves a matrix on the boundary for its parent. All fronts of one depth
// of the tree are processed together, the deepest first.
//
// With the front's matrix [A11 A21^T; A21 A22], A11 = G S G^T (G lower triangular, S = diag(+-1)):
//   x11 = G^-1 (p x p, lower), l21 = A21 G^-T S (b x p), contribution C = A22 - l21 S l21^T,
//   w21 = l21 x11 = A21 A11^-1 (b x p), kept in l21's place.
// A solve is then one pass up the tree, z = x11 v_P and v_B -= w21 v_P, and one down,
// x_P = x11^T S z - w21^T x_B: matrix-vector products whose rows (columns) do not wait for each other,
// one launch per depth and pass.
#pragma once

#include <vector>

#include "tf_internal.cuh"

namespace tfb {

constexpr int kFcTile = 64;        // pivot panel width and GEMM tile
constexpr int kFcScatter = 256;    // Jacobian blocks per assembly task
constexpr int kFcSmallB = 288;     // boundary unknowns up to which a one-panel front is one CTA's
constexpr int kFcRowEntries = 8192; // most entries of [x11; w21] per task of the upward pass
constexpr int kFcSms = 148;
constexpr int kFcMaxPivots = 5000; // pivots of one front, and unknowns of one front: the passes stage
constexpr int kFcMaxFront = 24000; // vectors of them in shared memory

struct FcFront {
    int32_t p, b;          // pivot and boundary unknowns
    int32_t ldp, ldb;      // leading dimensions (even): rows of x11 / l21 / a21, rows of c
    int32_t tissue;
    int32_t child[2];      // fronts one depth below, or -1
    int32_t child_ldb[2], child_vec[2];  // the children's ldb and vec, and below their c: one load away
    int32_t map[2];        // offsets into maps: per column of this front, its index on the child's boundary
    int32_t verts;         // offset into verts: the pivots' columns, then the boundary's
    int32_t j0, j1;        // its Jacobian blocks in jblk
    int32_t ent;           // offset of its p + b entries in kids / dofs
    int32_t vec, piv;      // offsets of the boundary vector (b) and of z / the signs (p)
    int64_t x11, w21;      // kept factors
    int64_t a21, l21, lp;  // scratch of the front's depth: A21, l21 and the current panel of L11 (p x 64)
    int64_t c;             // contribution (b x b, lower), in the scratch of the depth's parity
    int64_t child_c[2];
};

struct FcTask {
    int32_t front;
    int16_t i, j;
};

// One-CTA fronts keep [A11; A21] in shared memory: leading dimension (4 mod 8: the fragments' reads hit
// distinct banks) and bytes, with the two children's maps.
__host__ __device__ inline int fc_small_ld(int p) {
    const int l = (p + 3) & ~3;
    return l % 8 ? l : l + 4;
}
__host__ __device__ inline int fc_small_smem(int p, int b) {
    return (((p + 7) & ~7) + ((b + 15) & ~15)) * fc_small_ld(p) * 8 + 2 * (p + b) * 4;
}

struct FcRange {
    int32_t begin = 0, count = 0;
};

struct FcPanel {
    FcRange col, upd;
};

struct FcDepth {
    FcRange small[3], gather, scatter, diag, l21, schur;  // small: fronts factorised by one CTA each, by size
    FcRange fwd, bwd;  // tasks (i, j): rows [i j, (i + 1) j); columns [i j, (i + 1) j)
    int32_t fwd_smem = 0, bwd_smem = 0, bwd_threads = 256;  // bytes; threads of a downward CTA
    int32_t panel0 = 0, n_panel = 0;
};

// Host side of a factorisation: the symbolic result, laid out for the device.
struct FcPlan {
    int gd = 3;  // unknowns per column (three per node)
    std::vector<FcFront> fronts;
    std::vector<int32_t> maps, verts;
    std::vector<int2> jblk;  // {block, row << 16 | column} in the front's [x11; a21] rows
    std::vector<int32_t> jblk_t;  // the transposed block of each, for an unsymmetric J (else empty)
    std::vector<FcTask> tasks;
    std::vector<FcDepth> depths;  // 0: the roots
    std::vector<FcPanel> panels;
    int64_t n_factor = 0, n_scratch = 0, n_contrib[2] = {0, 0};  // doubles
    int64_t n_vec = 0, n_piv = 0, n_ent = 0;
    int64_t n_root = 0;   // pivots of the root fronts
    double flops = 0.0;   // multiplications and additions of one factorisation
    bool ok = false;
};

// Symbolic factorisation of the block pattern (G consecutive nodes form one column with in-plane
// position X[3 column]); tissue t owns nodes [node0[t], node0[t+1]). plan.ok = false when a front
// is too large for the kernels, the operation count exceeds max_flops or a position is not a finite number.
// transposed: with jblk_t, so that the symmetric part (J + J^T) / 2 of an unsymmetric J is factorised. Throws
// std::bad_alloc.
void build_factor_plan(int N, int G, const int32_t* rowptr, const int32_t* colidx, const double* X, int T,
                       const int32_t* node0, double max_flops, bool transposed, FcPlan& plan);

// Device side.
struct FcWork {
    int gd;
    const FcFront* fronts;
    int2* kids;     // [n_ent] every entry's index on the boundary of either child, or -1
    int32_t* dofs;  // [n_ent] every entry's unknown
    const int2* jblk;
    const int32_t* jblk_t;  // NULL: J is symmetric
    const FcTask* tasks;
    const int32_t* active;  // [T]
    double* factor;
    double* scratch;
    double* contrib[2];
    double* vec;
    double* z;
    double* sign;    // [n_piv] +1 / -1
    int32_t* neg;    // [fronts] 1: the front has negative pivots
};

// kids and dofs of every front from the plan's columns (maps, verts on the device)
cudaError_t launch_factor_expand(const FcPlan& plan, const FcWork& w, const int32_t* maps, const int32_t* verts,
                                 cudaStream_t s);
// Streams of a factorisation: the side streams start after and end before what is on `main`.
struct FcStreams {
    cudaStream_t main = nullptr, side[3] = {};
    cudaEvent_t fork = nullptr, join[3] = {};
};
// Numeric factorisation of J (vals: the full BSR3 values; block (row, column) is read from the row of
// the earlier pivot, transposed). Returns the kernels launched in *launches.
cudaError_t launch_factor(const FcPlan& plan, const FcWork& w, const double* vals, int64_t* launches, const FcStreams& st);
// Preconditioned iterations with the factor as preconditioner, one kernel per phase, every tissue with its
// own scalars: conjugate gradients, or for an unsymmetric J the minimal residual iteration (p = z,
// alpha = (r, q) / (q, q)), which the factor of the symmetric part contracts by the asymmetry. A chunk is a run of rows of one tissue; the dot products are summed
// per chunk and then per tissue in chunk order.
struct FcChunk {
    int32_t tissue, row0, row1;
};
// Rows of a chunk: two chunks per SM, between 32 (one pass of a CTA's 8-lane rows) and 256 (few partial sums).
inline int fc_chunk_rows(int n_nodes) {
    const int r = (n_nodes / 296 + 31) / 32 * 32;
    return r < 32 ? 32 : (r > 256 ? 256 : r);
}

// The doubles [begin, end) of the Jacobian blocks [k0, k1). In 64 bits: 32 end at 238.6 million blocks, a batch
// of 243 full wing discs (17 GB of values beside 126 GB of factors).
struct FcSpan {
    int64_t begin, end;
};
__host__ __device__ inline FcSpan fc_block_span(int32_t k0, int32_t k1) { return {(int64_t)k0 * 9, (int64_t)k1 * 9}; }

struct FcCg {
    int n_chunks;
    const FcChunk* chunks;
    const int32_t* chunk0;  // [T+1]
    KrylovScalars* sc;      // [T]
    KrylovScalars* host;    // [T] page-locked: sc after the start and after every iteration
    const int32_t* active;  // [T] tissues of this solve
    int32_t* running;       // [T] still iterating (the preconditioner's active flags)
    double* part;           // [3][n_chunks]: (r, z), (p, J p), (r, r) / (b, b)
    int32_t minres;         // 1: the minimal residual iteration (part: (r, q), (q, q), (r, r))
};
// One iteration: z = M^-1 r (a pass up and down the tree with the factor; every unknown is a pivot of one
// front), p = z + beta p (p = z in the first), q = J p, x += alpha p, r -= alpha q, and the test. Before the
// first: x = 0, r = b; every active tissue running (unless b = 0).
cudaError_t launch_fc_iteration(const FcPlan& plan, const FcWork& f, const KrylovWork& w, const FcCg& c, bool first, double rtol,
                                int max_iter, double* z, double* q, int64_t* launches, cudaStream_t s);

}  // namespace tfb
