// Coarsest-level direct solve (SetupSolver.m:257-259, Vcycle.m:22-23): the
// reference factors the assembled free-DOF matrix with a sparse Cholesky and
// applies two triangular solves per V-cycle.  Here the free DOFs are numbered
// node by node in slot order, so the matrix is banded; with blocks of order
// B >= the half bandwidth it is block tridiagonal,
//     A = tridiag(A_(i,i-1), A_ii, A_(i,i-1)^T),   i = 0..nb-1.
// It is factored from both ends towards a middle block k ("twisted" block
// LDL^T): from the top
//     S_0 = A_00,  G_i = A_(i,i-1) S_(i-1)^-1,  S_i = A_ii - G_i A_(i,i-1)^T   (i < k)
// from the bottom
//     T_(nb-1) = A_(nb-1,nb-1),  H_i = A_(i+1,i)^T T_(i+1)^-1,
//     T_i = A_ii - H_i A_(i+1,i)                                             (i > k)
// and in the middle M = A_kk - G_k A_(k,k-1)^T - H_k A_(k+1,k).  A x = r is
//     c_i = r_i - G_i c_(i-1) (i = 1..k-1),  c_i = r_i - H_i c_(i+1) (i = nb-2..k+1)
//     c_k = r_k - G_k c_(k-1) - H_k c_(k+1)
//     x_i = D_i^-1 c_i for every block (D = S, T or M)
//     x_i -= G_(i+1)^T x_(i+1) (i = k-1..0),  x_i -= H_(i-1)^T x_(i-1) (i = k+1..nb-1)
// so both sequential sweeps run as two independent chains of about nb/2
// steps, and the two halves of the factorisation run on two streams.
//
// Each D_i^-1 comes from a recursive blocked Cholesky that also forms L^-1 (no
// pivoting: every D_i is SPD), then D^-1 = L^-T L^-1.
//
// Every sum is a chain of multiply-adds in ascending order from zero, grouped
// by the recursion and, in the solve, by 16 columns and 64-column tiles: the
// results do not depend on how the launches tile the work.  The mixed path
// rounds the solution to FP32 each V-cycle, and on an ill-conditioned coarsest
// level another order changes some of those roundings and through them the
// stresses in the eighth digit (an inverse by Gauss-Jordan block sweeps, with
// half the operations, was as accurate and 0.1 ms per block faster, and is not
// used for that reason).
//
// A warp's FP64 instruction takes the SM's one FP64 unit for 19 clocks (64 for
// a single warp) however many of its lanes are active (measured), so the work
// is spread over many SMs and small launches, and operations are avoided:
//   - the couplings A_(i,i-1) hold about 20 non-zeros per row (27-point
//     coupling); the products with them skip the zeros (172 and 118 us per
//     block of order 448 as dense products, 14 and 13 us so)
//   - the 32 x 32 Cholesky leaf spent two thirds of its 43 us in the square
//     root and the division of each column; it forms both from one FP32
//     reciprocal square root, while the other warps update
//   - L^-T L^-1 is symmetric: half of its tiles are computed
// Measured for 15 blocks of order 448: factorisation 14 -> 8.0 ms; the solve's
// launches 8 -> 4 us each (a warp per row instead of 64 x 64 tiles with partial
// sums in memory and arrival counters).
#include "setup.cuh"
#include "sqrt_reciprocal.h"

namespace gmgs {

namespace {

enum : int { TRI_A_LOWER = 1, TRI_A_UPPER = 2, TRI_B_LOWER = 4, TRI_B_UPPER = 8 };
enum : int { OUT_ALL = 0, OUT_LOWER = 1, OUT_MIRROR = 2 };

// C = alpha op(A) op(B) + beta C, column-major, m, n, k multiples of 16, one
// output per thread on 16 x 8 tiles (the smallest products of the recursion are
// 32^3: small tiles put them on more SMs).  TRI marks operands known to be
// triangular so the k-loop skips their zero tiles (exact zeros).  OUT_LOWER
// skips output tiles strictly above the diagonal (their values are never
// read), OUT_MIRROR computes a symmetric product's lower half and stores both.
constexpr int GR = 16, GC = 8, GK = 16, GT = GR * GC;
template <bool TA, bool TB, int TRI, int OUT>
__global__ void __launch_bounds__(GT) k_dgemm(int k, double alpha, const double* A, int lda, const double* B, int ldb, double beta,
                                              double* C, int ldc) {
    pdl_begin();
    pdl_wait();
    const int r0 = blockIdx.x * GR, c0 = blockIdx.y * GC;
    if (OUT != OUT_ALL && r0 + GR <= c0) return;
    __shared__ double As[2][GK][GR + 1];   // As[.][l][i] = op(A)(r0 + i, k0 + l)
    __shared__ double Bs[2][GK][GC + 1];   // Bs[.][l][j] = op(B)(k0 + l, c0 + j)
    const int t = threadIdx.x, tx = t % GR, ty = t / GR;
    int kb = 0, ke = k;
    if (TRI & TRI_A_LOWER) ke = min(ke, r0 + GR);
    if (TRI & TRI_A_UPPER) kb = max(kb, r0);
    if (TRI & TRI_B_LOWER) kb = max(kb, c0 & ~(GK - 1));
    if (TRI & TRI_B_UPPER) ke = min(ke, (c0 & ~(GK - 1)) + GK);
    double ra[2], rb;
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int e = t + q * GT;
            ra[q] = TA ? A[(int64_t)(r0 + e / GK) * lda + k0 + e % GK] : A[(int64_t)(k0 + e / GR) * lda + r0 + e % GR];
        }
        rb = TB ? B[(int64_t)(k0 + t / GC) * ldb + c0 + t % GC] : B[(int64_t)(c0 + t / GK) * ldb + k0 + t % GK];
    };
    double acc = 0.0;
    if (kb < ke) load(kb);
    int buf = 0;
    for (int k0 = kb; k0 < ke; k0 += GK, buf ^= 1) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int e = t + q * GT;
            if (TA) As[buf][e % GK][e / GK] = ra[q];
            else As[buf][e / GR][e % GR] = ra[q];
        }
        if (TB) Bs[buf][t / GC][t % GC] = rb;
        else Bs[buf][t % GK][t / GK] = rb;
        __syncthreads();
        if (k0 + GK < ke) load(k0 + GK);
#pragma unroll
        for (int l = 0; l < GK; ++l) acc = fma(As[buf][l][tx], Bs[buf][l][ty], acc);
    }
    const int r = r0 + tx, c = c0 + ty;
    if (OUT == OUT_MIRROR) {
        if (r < c) return;
        C[(int64_t)c * ldc + r] = alpha * acc;
        C[(int64_t)r * ldc + c] = alpha * acc;
        return;
    }
    double* cp = C + (int64_t)c * ldc + r;
    *cp = beta == 0.0 ? alpha * acc : fma(alpha, acc, beta * *cp);
}
template <bool TA, bool TB, int TRI, int OUT>
void gemm(Ctx& c, int m, int n, int k, double alpha, const double* A, int lda, const double* B, int ldb, double beta,
          double* C, int ldc) {
    if (m <= 0 || n <= 0) return;
    launch_chain(c, k_dgemm<TA, TB, TRI, OUT>, dim3(m / GR, n / GC), GT, 0, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// sqrt(d) and its reciprocal, both correctly rounded, for a positive d: from one
// FP32 reciprocal square root, outside the FP32 range by the library
__device__ __forceinline__ void pivot_root(double d, double& s, double& r) {
    const int e = (__double2hiint(d) >> 20) - 1023;
    if (e < -120 || e > 120) {
        s = sqrt(d);
        r = 1.0 / s;
        return;
    }
    sqrt_reciprocal(d, f2d_int(rsqrtf(d2f_int(d))), s, r);
}

// Cholesky of a 32 x 32 SPD tile (lower triangle of A, in place) and the
// inverse of its factor into Li (zeros above the diagonal), one column per
// step: the pivot's square root and reciprocal, column j of L, row j of L^-1
// (forward substitution of L X = I carried along: X(j, c) is final once
// scaled by 1 / L(j,j)), then the rank-1 updates of the rows below j of A and
// of X.  Warp 0 updates row j + 1 first and goes on to its square root while
// the warps of the other three quarters of the SM update the rest (warp 4
// shares warp 0's quarter and would hold its chain up).  A pivot that is not positive sets *info and
// is replaced by 1 so the arithmetic stays finite.
__global__ void __launch_bounds__(256) k_chol_inv32(double* A, int lda, double* Li, int ldl, int* __restrict__ info) {
    pdl_begin();
    pdl_wait();
    __shared__ double a[32][33];   // a[c][r] = A(r, c), becomes L
    __shared__ double x[32][33];   // x[c][r] = X(r, c), becomes L^-1
    __shared__ double s_piv, s_inv;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int e = t; e < 1024; e += 256) {
        const int cc = e >> 5, r = e & 31;
        a[cc][r] = A[(int64_t)cc * lda + r];
        x[cc][r] = r == cc ? 1.0 : 0.0;
    }
    auto pivot = [&](double d) {
        const int hi = __double2hiint(d);
        const bool ok = hi >= 0 && hi < 0x7ff00000 && (hi | __double2loint(d)) != 0;    // positive and finite
        if (!ok) atomicExch(info, 1);
        double s = 1.0, r = 1.0;
        if (ok) pivot_root(d, s, r);
        s_piv = s;
        s_inv = r;
    };
    __syncthreads();
    if (t == 0) pivot(a[0][0]);
#pragma unroll 1
    for (int j = 0; j < 32; ++j) {
        __syncthreads();
        const double dinv = s_inv;
        if (w == 0) {
            if (lane == j) a[j][j] = s_piv;
            if (lane > j) a[j][lane] *= dinv;               // L(r, j)
        } else if (w == 1 && lane <= j) {
            x[lane][j] *= dinv;                             // X(j, c), c <= j
        }
        __syncthreads();
        auto row = [&](int r) {
            double v = 0.0;
            if (lane > j) {
                if (r >= lane) a[lane][r] = v = fma(-a[j][r], a[j][lane], a[lane][r]);
            } else {
                x[lane][r] = fma(-a[j][r], x[lane][j], x[lane][r]);
            }
            return v;
        };
        if (w == 0) {
            if (j + 1 < 32) {
                const double d = row(j + 1);
                if (lane == j + 1) pivot(d);
            }
        } else if (w != 4) {
            for (int r = j + 1 + (w < 4 ? w : w - 1); r < 32; r += 6) row(r);
        }
    }
    __syncthreads();
    for (int e = t; e < 1024; e += 256) {
        const int cc = e >> 5, r = e & 31;
        if (r >= cc) A[(int64_t)cc * lda + r] = a[cc][r];
        Li[(int64_t)cc * ldl + r] = x[cc][r];
    }
}

// The non-zeros E'(row, c0 .. c0 + 255) of one row of E' (E, or its transpose)
// into shared memory in column order; returns their number.  E column-major.
__device__ __forceinline__ int row_nonzeros(int B, const double* __restrict__ E, bool trans, int row, int c0, double* val,
                                            int* idx, int* cnt) {
    const int t = threadIdx.x, c = c0 + t;
    double v = 0.0;
    if (c < B) v = trans ? E[(int64_t)row * B + c] : E[(int64_t)c * B + row];
    const unsigned m = __ballot_sync(0xffffffffu, v != 0.0);
    __syncthreads();                                  // the previous chunk's readers are done
    if ((t & 31) == 0) cnt[t >> 5] = __popc(m);
    __syncthreads();
    int at = 0, n = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w == (t >> 5)) at = n;
        n += cnt[w];
    }
    if (v != 0.0) {
        at += __popc(m & ((1u << (t & 31)) - 1u));
        val[at] = v;
        idx[at] = c;
    }
    __syncthreads();
    return n;
}

// G = E' X with X symmetric (both triangles): one CTA per row and 256 columns;
// G row-major to gt, column-major to gc
__global__ void __launch_bounds__(256) k_sparse_left(int B, const double* __restrict__ E, int trans, const double* __restrict__ X,
                                                     double* __restrict__ gt, double* __restrict__ gc) {
    __shared__ double val[256];
    __shared__ int idx[256], cnt[8];
    const int row = blockIdx.x, j = blockIdx.y * 256 + threadIdx.x;
    double acc = 0.0;
    for (int c0 = 0; c0 < B; c0 += 256) {
        const int n = row_nonzeros(B, E, trans != 0, row, c0, val, idx, cnt);
        if (j < B)
            for (int q = 0; q < n; ++q) acc = fma(val[q], X[(int64_t)idx[q] * B + j], acc);
    }
    if (j < B) {
        gt[(int64_t)row * B + j] = acc;
        gc[(int64_t)j * B + row] = acc;
    }
}

// D -= G E'^T on the lower triangle, G column-major: one CTA per column of D
// and 256 rows
__global__ void __launch_bounds__(256) k_sparse_update(int B, const double* __restrict__ E, int trans,
                                                       const double* __restrict__ gc, double* __restrict__ D) {
    __shared__ double val[256];
    __shared__ int idx[256], cnt[8];
    const int j = blockIdx.x, i = blockIdx.y * 256 + threadIdx.x;
    if ((int)blockIdx.y * 256 + 255 < j) return;      // above the diagonal, uniform across the CTA
    double acc = 0.0;
    for (int c0 = 0; c0 < B; c0 += 256) {
        const int n = row_nonzeros(B, E, trans != 0, j, c0, val, idx, cnt);
        if (i < B)
            for (int q = 0; q < n; ++q) acc = fma(val[q], gc[(int64_t)idx[q] * B + i], acc);
    }
    if (i < B && i >= j) D[(int64_t)j * B + i] -= acc;
}

// scratch of one chain of the factorisation
struct Chain {
    DevBuf li, l, t, g;      // L^-1, the off-diagonal parts of L, a product, G column-major (B x B each)
    void alloc(int B) {
        for (DevBuf* d : {&li, &l, &t, &g}) *d = dalloc((size_t)B * B * sizeof(double));
    }
};

// L^-1 (into Li, whose part above the diagonal must be zero on entry) of the
// n x n SPD matrix A (overwritten), n a multiple of 32, by halves:
// L11 = chol(A11), L21 = A21 L11^-T, L22 = chol(A22 - L21 L21^T),
// L^-1_21 = -L22^-1 L21 L11^-1.  L21 goes to the same place of Lo; T: scratch.
void chol_inv(Ctx& c, double* A, double* Li, double* Lo, int n, int ld, double* T, int* info) {
    if (n == 32) {
        launch_chain(c, k_chol_inv32, 1, 256, 0, A, ld, Li, ld, info);
        return;
    }
    const int n1 = 32 * ((n / 32) / 2), n2 = n - n1;
    const int64_t at22 = (int64_t)n1 * ld + n1;
    double* L21 = Lo + n1;
    chol_inv(c, A, Li, Lo, n1, ld, T, info);
    gemm<false, true, TRI_B_UPPER, OUT_ALL>(c, n2, n1, n1, 1.0, A + n1, ld, Li, ld, 0.0, L21, ld);
    gemm<false, true, 0, OUT_LOWER>(c, n2, n2, n1, -1.0, L21, ld, L21, ld, 1.0, A + at22, ld);
    chol_inv(c, A + at22, Li + at22, Lo + at22, n2, ld, T, info);
    gemm<false, false, TRI_B_LOWER, OUT_ALL>(c, n2, n1, n1, 1.0, L21, ld, Li, ld, 0.0, T, n2);          // L21 L11^-1
    gemm<false, false, TRI_A_LOWER, OUT_ALL>(c, n2, n1, n2, -1.0, Li + at22, ld, T, n2, 0.0, Li + n1, ld);
}

// D^-1 of the SPD block D (lower triangle in, both triangles out): 68 dependent
// launches per block of order 448, as programmatic dependents of each other (15
// blocks 8.0 ms, as plain launches 8.7 ms)
void inv_spd(Ctx& c, double* D, int B, Chain& s, int* info) {
    double* li = s.li.as<double>();
    GMGS_CUDA(cudaMemsetAsync(li, 0, (size_t)B * B * sizeof(double), c.stream));
    chol_inv(c, D, li, s.l.as<double>(), B, B, s.t.as<double>(), info);
    gemm<true, false, TRI_A_UPPER | TRI_B_LOWER, OUT_MIRROR>(c, B, B, B, 1.0, li, B, li, B, 0.0, D, B);
}
void sparse_left(Ctx& c, int B, const double* E, bool trans, const double* X, double* gt, double* gc) {
    k_sparse_left<<<dim3(B, (B + 255) / 256), 256, 0, c.stream>>>(B, E, trans, X, gt, gc);
    GMGS_LAUNCHED(c);
}
void sparse_update(Ctx& c, int B, const double* E, bool trans, const double* gc, double* D) {
    k_sparse_update<<<dim3(B, (B + 255) / 256), 256, 0, c.stream>>>(B, E, trans, gc, D);
    GMGS_LAUNCHED(c);
}

// ---------------------------------------------------------------------------
// the solve: launches of independent jobs y = base - sum_s M_s v_s (base null:
// the sum itself), M_s B x B with its rows contiguous
// ---------------------------------------------------------------------------
constexpr int STEP_ROWS = 8;      // rows (warps) per CTA
constexpr int CH = 16;            // columns per lane: the sums' first grouping
constexpr int PART = 32 * CH;     // columns a warp takes at a time
constexpr int MAX_JOBS = 4;
struct StepJob {
    const double* M[2];
    const double* v[2];
    const double* base;
    double* y;
    int nseg;
    int out;             // y is final: its first row in the solution, else -1
};
struct StepJobs {
    StepJob j[MAX_JOBS];
    CoarseOut out;
    int n = 0;
    void add(double* y, const double* base, const double* M0, const double* v0, const double* M1 = nullptr,
             const double* v1 = nullptr) {
        j[n++] = {{M0, M1}, {v0, v1}, base, y, M1 ? 2 : 1, -1};
    }
    void add_final(int row, double* y, const double* base, const double* M0, const double* v0) {
        add(y, base, M0, v0);
        j[n - 1].out = row;
    }
};

// Rows in the order k_rows reads them: of each 512 columns lane L takes the
// columns 16 L .. 16 L + 15, stored as pairs, pair u of all lanes together.  In
// place, one CTA per row; z: the three families of matrices.
__global__ void __launch_bounds__(128) k_order_rows(int B, double* m0, double* m1, double* m2) {
    __shared__ double part[PART];
    double* m = (blockIdx.z == 0 ? m0 : (blockIdx.z == 1 ? m1 : m2)) + ((int64_t)blockIdx.y * B + blockIdx.x) * B;
    for (int p0 = 0; p0 < B; p0 += PART, m += PART) {
        const int n = min(PART, B - p0), nl = n / CH;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) part[i] = m[i];
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int u = i / (2 * nl), l = i % (2 * nl) / 2;
            m[i] = part[CH * l + 2 * u + (i & 1)];
        }
    }
}

// One warp per row, eight rows per CTA: a matrix-vector product has to be
// spread over all SMs (an SM does 1.7 FP64 multiply-adds per clock), and a row
// per warp needs no partial sums through memory.  Launched as a programmatic
// dependent of the previous kernel in the stream: a row's first 512 entries are
// loaded while that kernel finishes, then the hardware grid dependency is
// waited for, and only then are vectors read or written.
// Order of a row's sum: 16 columns in sequence, (s0 + s1) + (s2 + s3) of four
// such groups, then the 64-column tiles (of both segments) in sequence; the
// tiles of the CTA's rows are summed by one warp, a lane per row.
__global__ void __launch_bounds__(32 * STEP_ROWS) k_rows(int B, const __grid_constant__ StepJobs jobs) {
    pdl_begin();
    __shared__ double vs[17 * 32];                        // 512 entries of v, 17 places per 16
    __shared__ double tile[8][STEP_ROWS];
    const StepJob& J = jobs.j[blockIdx.y];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, row = blockIdx.x * STEP_ROWS + w;
    const int nl0 = min(32, B / CH);
    double2 m[2][CH / 2];
#pragma unroll
    for (int s = 0; s < 2; ++s)
        if (s < J.nseg && lane < nl0) {
            const double2* r = reinterpret_cast<const double2*>(J.M[s] + (int64_t)row * B);
#pragma unroll
            for (int u = 0; u < CH / 2; ++u) m[s][u] = r[u * nl0 + lane];
        }
    pdl_wait();
    double sum = 0.0;                                     // lanes of warp 0: the row's tiles so far
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        if (s >= J.nseg) break;
        for (int p0 = 0; p0 < B; p0 += PART) {
            const int n = min(PART, B - p0), nl = n / CH;
            for (int i = t; i < n; i += 32 * STEP_ROWS) vs[i + i / CH] = J.v[s][p0 + i];
            __syncthreads();                              // also: the tile sums before these are taken
            double acc = 0.0;
            if (lane < nl) {
                const double2* r = reinterpret_cast<const double2*>(J.M[s] + (int64_t)row * B + p0);
                const double* v = vs + 17 * lane;
#pragma unroll
                for (int u = 0; u < CH / 2; ++u) {
                    const double2 e = p0 == 0 ? m[s][u] : r[u * nl + lane];
                    acc = fma(e.x, v[2 * u], acc);
                    acc = fma(e.y, v[2 * u + 1], acc);
                }
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            if ((lane & 3) == 0 && lane < nl) tile[lane / 4][w] = acc;
            __syncthreads();
            if (w == 0 && lane < STEP_ROWS)
                for (int k = 0; k < n / 64; ++k) sum += tile[k][lane];
        }
    }
    if (w == 0 && lane < STEP_ROWS) {
        const int r = blockIdx.x * STEP_ROWS + lane;
        const double y = J.base ? J.base[r] - sum : sum;
        J.y[r] = y;
        if (J.out >= 0 && J.out + r < jobs.out.n) {         // to the level's vector (a scatter launch less)
            const int32_t slot = jobs.out.idx[J.out + r];
            if (jobs.out.f) jobs.out.f[slot] = (float)y;
            else jobs.out.d[slot] = y;
        }
    }
}

void launch_step(Ctx& c, int B, const StepJobs& jobs) {
    if (jobs.n == 0) return;
    launch_chain(c, k_rows, dim3(B / STEP_ROWS, jobs.n, 1), dim3(32 * STEP_ROWS, 1, 1), 0, B, jobs);
}

int coarse_middle(int nb) { return (nb - 1) / 2; }

}  // namespace

int coarse_block_order(int n, int half_bandwidth) {
    constexpr int Q = 64;         // the solve's tiles
    const int want = std::max(half_bandwidth, 1);
    return std::max(Q, (std::min(want, n) + Q - 1) / Q * Q);
}

void factor_coarse(Ctx& c, CoarseBlocks& cb, const std::function<void()>& overlap) {
    const int B = cb.B, nb = cb.nb, k = coarse_middle(nb);
    const int64_t B2 = (int64_t)B * B;
    double* D = cb.sinv.as<double>();   // A_ii on entry
    double* E = cb.g.as<double>();      // E_i = A_(i,i-1) on entry (i >= 1)
    if (cb.gt.bytes < (size_t)nb * B2 * sizeof(double)) cb.gt = dalloc((size_t)nb * B2 * sizeof(double));
    auto Db = [&](int i) { return D + i * B2; };
    auto Eb = [&](int i) { return E + i * B2; };
    auto Gt = [&](int i) { return cb.gt.as<double>() + i * B2; };
    // the two halves run on their own streams, forked from and joined to c.stream
    cudaStream_t st[2] = {nullptr, nullptr};
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    struct Res {
        cudaStream_t* s; cudaEvent_t* e;
        ~Res() {
            for (int i = 0; i < 2; ++i) if (s[i]) cudaStreamDestroy(s[i]);
            for (int i = 0; i < 3; ++i) if (e[i]) cudaEventDestroy(e[i]);
        }
    } res{st, ev};
    for (int i = 0; i < 2; ++i) GMGS_CUDA(cudaStreamCreateWithFlags(&st[i], cudaStreamNonBlocking));
    for (int i = 0; i < 3; ++i) GMGS_CUDA(cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming));
    DevBuf info = dalloc(2 * sizeof(int));
    GMGS_CUDA(cudaMemsetAsync(info.p, 0, 2 * sizeof(int), c.stream));
    Chain chain[2];
    for (int h = 0; h < 2; ++h) chain[h].alloc(B);
    GMGS_CUDA(cudaEventRecord(ev[0], c.stream));
    Ctx half[2] = {c, c};
    for (int h = 0; h < 2; ++h) {
        half[h].stream = st[h];
        half[h].prof = false;
        half[h].trace = false;
        half[h].launches = 0;
        GMGS_CUDA(cudaStreamWaitEvent(st[h], ev[0], 0));
    }
    int* inf = info.as<int>();
    auto keep_g = [&](Ctx& h, Chain& s, int i) {     // G column-major takes the coupling's place
        GMGS_CUDA(cudaMemcpyAsync(Eb(i), s.g.p, B2 * sizeof(double), cudaMemcpyDeviceToDevice, h.stream));
    };
    // block by block from both ends (interleaved, so both streams have work
    // from the start): top S_i^-1 (i < k) with G_i, then G_k; bottom T_i^-1
    // (i > k) with H_i in the place of E_(i+1), then H_k.  The middle block's
    // couplings stay in place until both have reached it.
    for (int step = 0; step <= std::max(k, nb - 1 - k); ++step) {
        if (step <= k) {
            const int i = step;
            Ctx& h = half[0];
            if (i > 0) sparse_left(h, B, Eb(i), false, Db(i - 1), Gt(i), chain[0].g.as<double>());
            if (i < k) {
                if (i > 0) {
                    sparse_update(h, B, Eb(i), false, chain[0].g.as<double>(), Db(i));
                    keep_g(h, chain[0], i);
                }
                inv_spd(h, Db(i), B, chain[0], inf);
            }
        }
        if (nb - 1 - step >= k) {
            const int i = nb - 1 - step;
            Ctx& h = half[1];
            if (i < nb - 1) sparse_left(h, B, Eb(i + 1), true, Db(i + 1), Gt(i + 1), chain[1].g.as<double>());
            if (i > k) {
                if (i < nb - 1) {
                    sparse_update(h, B, Eb(i + 1), true, chain[1].g.as<double>(), Db(i));
                    keep_g(h, chain[1], i + 1);
                }
                inv_spd(h, Db(i), B, chain[1], inf + 1);
            }
        }
    }
    if (overlap) overlap();
    c.trace_point("bc: work buffers (beside the factorisation)");
    for (int h = 0; h < 2; ++h) {
        GMGS_CUDA(cudaEventRecord(ev[1 + h], st[h]));
        GMGS_CUDA(cudaStreamWaitEvent(c.stream, ev[1 + h], 0));
        c.launches += half[h].launches;
    }
    // the middle block: M = A_kk - G_k A_(k,k-1)^T - H_k A_(k+1,k), then M^-1
    if (k >= 1) {
        sparse_update(c, B, Eb(k), false, chain[0].g.as<double>(), Db(k));
        keep_g(c, chain[0], k);
    }
    if (k + 1 <= nb - 1) {
        sparse_update(c, B, Eb(k + 1), true, chain[1].g.as<double>(), Db(k));
        keep_g(c, chain[1], k + 1);
    }
    inv_spd(c, Db(k), B, chain[0], inf);
    // rows into the solve's order: D^-1 (symmetric), G^T (the columns of G) and G
    k_order_rows<<<dim3(B, nb, 3), 128, 0, c.stream>>>(B, D, E, cb.gt.as<double>());
    GMGS_LAUNCHED(c);
    c.trace_point("bc: coarsest block LDL^T");
    int h_info[2] = {0, 0};
    GMGS_CUDA(cudaMemcpyAsync(h_info, info.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    if (h_info[0] || h_info[1]) throw Error(GMGS_ERR_NOT_SPD, "coarsest-level matrix is not positive definite");
}

void launch_coarse_solve(Ctx& c, const CoarseBlocks& cb, double* cvec, double* x, const CoarseOut& out) {
    const int B = cb.B, nb = cb.nb, k = coarse_middle(nb);
    if (nb <= 0) return;
    const int64_t B2 = (int64_t)B * B;
    auto Db = [&](int i) { return cb.sinv.as<double>() + i * B2; };    // symmetric; rows in k_rows' order
    auto G = [&](int i) { return cb.gt.as<double>() + i * B2; };       // rows of G
    auto GT = [&](int i) { return cb.g.as<double>() + i * B2; };       // rows of G^T
    auto cv = [&](int i) { return cvec + (int64_t)i * B; };
    auto xv = [&](int i) { return x + (int64_t)i * B; };
    // Forward chains, in place on cvec: top i = 1..k-1, bottom i = nb-2..k+1.
    // x_i = D_i^-1 c_i of the blocks that the previous launch finished rides
    // along (one launch of its own for all blocks would wait for them all and
    // read every D_i^-1 at once).
    const int top = k, bot = nb - 1 - k;      // blocks above and below the middle
    const int steps = std::max(top, bot);
    for (int step = 0; step < steps; ++step) {
        StepJobs J;
        J.out = out;
        if (step == steps - 1) {              // the middle block's right-hand side: both chains have ended
            if (top > 0 && bot > 0) J.add(cv(k), cv(k), G(k), cv(k - 1), G(k + 1), cv(k + 1));
            else J.add(cv(k), cv(k), G(bot > 0 ? k + 1 : k), cv(bot > 0 ? k + 1 : k - 1));
        }
        if (step < top) {
            J.add(xv(step), nullptr, Db(step), cv(step));
            if (step + 1 < top) J.add(cv(step + 1), cv(step + 1), G(step + 1), cv(step));
        }
        if (step < bot) {
            const int i = nb - 1 - step;
            J.add(xv(i), nullptr, Db(i), cv(i));
            if (step + 1 < bot) J.add(cv(i - 1), cv(i - 1), G(i), cv(i));
        }
        launch_step(c, B, J);
    }
    {
        StepJobs J;
        J.out = out;
        J.add_final(k * B, xv(k), nullptr, Db(k), cv(k));
        launch_step(c, B, J);
    }
    // backward chains, in place on x: top i = k-1..0, bottom i = k+1..nb-1
    for (int s = 0; s < steps; ++s) {
        StepJobs J;
        J.out = out;
        if (s < top) J.add_final((k - 1 - s) * B, xv(k - 1 - s), xv(k - 1 - s), GT(k - s), xv(k - s));
        if (s < bot) J.add_final((k + 1 + s) * B, xv(k + 1 + s), xv(k + 1 + s), GT(k + 1 + s), xv(k + s));
        launch_step(c, B, J);
    }
}

}  // namespace gmgs
