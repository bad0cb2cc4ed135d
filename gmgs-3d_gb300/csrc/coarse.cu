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
// Everything runs in FP64 (about 2 lanes per clock per SM on GB300), so the
// factorisation is organised to do few operations on many SMs:
//   - each D_i^-1 by symmetric block sweeps (Gauss-Jordan on the lower
//     triangle, 32 pivots at a time, no pivoting: every D_i is SPD), B^3 / 2
//     multiply-adds in B/32 pairs of launches.  A recursive Cholesky with the
//     inverse factor and L^-T L^-1 took B^3 and spent 43 us in each of its
//     B/32 single-CTA leaves: 1.45 ms per block of order 448
//   - the couplings A_(i,i-1) hold about 20 non-zeros per row (27-point
//     coupling), so the products with them are sparse: 5 % of the dense ones'
//     operations (172 and 118 us per block)
// Measured for 15 blocks of order 448: factorisation 14 -> 5.7 ms, solve 15
// launches of a 64 x 64-tile product with partial sums and arrival counters
// (about 8 us each in the stream) -> 15 launches of a warp per row.
// The errors of the solve are the same (5.9e-15 for both on a 6315-DOF
// coarsest level, 1.5e-10 against 2.2e-10 on a long column of condition 2e7).
#include "setup.cuh"

namespace gmgs {

namespace {

constexpr int PB = 32;       // pivots per panel
constexpr int PH = 16;       // pivots swept one by one
constexpr int PR = 8;        // rows per panel CTA

// 1 / d of a positive normal d from an FP32 reciprocal by one third-order step
// (Halley's iteration for the reciprocal: relative error e -> e^3, 2^-24 ->
// rounding): three FP64 operations instead of the division's dozen; outside
// the FP32 range the division.
__device__ __forceinline__ double reciprocal(double d) {
    const int e = (__double2hiint(d) >> 20) - 1023;
    if (e < -120 || e > 120) return 1.0 / d;
    const double r = f2d_int(__frcp_rn(d2f_int(d)));
    const double h = fma(-d, r, 1.0);
    return fma(r, fma(h, h, h), r);
}

// Sweeps of the 16 x 16 SPD block at (o, o) of A (lower triangle) one pivot at
// a time; its inverse into the same place of Pm, both triangles.  256 threads;
// ends with a barrier.  A pivot that is not positive sets *info and is replaced
// by 1 so the arithmetic stays finite.
struct SweepShared {
    double col[2][PH], rp[2], ws[PH];
};
__device__ __forceinline__ void invert16(const double (*A)[PB + 1], double (*Pm)[PB + 1], int o, SweepShared& sh, int* info) {
    constexpr int NO = PH * (PH - 1) / 2;                // elements below the diagonal: threads 0..119
    const int t = threadIdx.x;
    int i = -1, j = -1;
    if (t >= 128 && t < 128 + PH) {
        i = j = t - 128;
    } else if (t < NO) {                                 // i > j: t = i (i - 1) / 2 + j
        i = (int)((sqrtf(8.f * (float)t + 1.f) + 1.f) * 0.5f);
        while (i * (i + 1) / 2 <= t) ++i;
        while (i * (i - 1) / 2 > t) --i;
        j = t - i * (i - 1) / 2;
    }
    double a = i >= 0 ? A[o + i][o + j] : 0.0;
    auto publish = [&](int s) {     // the pivot column of sweep s and the reciprocal of its pivot
        if (i == s || j == s) sh.col[s & 1][i == s ? j : i] = a;
        if (i == s && j == s) {
            const int hi = __double2hiint(a);
            const bool ok = hi >= 0x00100000 && hi < 0x7ff00000;      // positive, normal, finite
            if (!ok) atomicExch(info, 1);
            sh.rp[s & 1] = ok ? reciprocal(a) : 1.0;
        }
    };
    publish(0);
#pragma unroll 1
    for (int s = 0; s < PH; ++s) {
        __syncthreads();
        const double r = sh.rp[s & 1];
        if (t < PH) sh.ws[t] = sh.col[s & 1][t] * r;
        __syncthreads();
        if (i == s || j == s) a = i == j ? -r : sh.ws[i == s ? j : i];
        else if (i >= 0) a = fma(-sh.ws[i], sh.col[s & 1][j], a);
        if (s + 1 < PH) publish(s + 1);
    }
    if (i >= 0) Pm[o + i][o + j] = Pm[o + j][o + i] = -a;
    __syncthreads();
}

// Inverse P of the 32 x 32 pivot block and W = C P for 8 rows of the panel C
// (the pivot columns of the symmetric matrix, of which D holds the lower
// triangle).  Every CTA inverts the pivot block for itself: that is a
// dependent chain, so sharing one inverse would only add a launch between it
// and the panel.  A warp's FP64 instruction takes the SM's FP64 unit for 19
// clocks (64 for a single warp) however many of its lanes are active
// (measured), so the cost of a sweep is its number of warp instructions: 17
// warps for one element per thread of a 32 x 32 triangle, 5 for 16 x 16.  The
// block is therefore inverted by halves, each half swept pivot by pivot and
// the rest products with one output per thread:
//   P22 = (A22 - W A21^T)^-1,  W = A21 A11^-1,  P21 = -P22 W,  P11 = A11^-1 + W^T P22 W
// (32 sweeps of the whole block took 32 to 43 us per launch: a division per
// sweep, 2 x 2 pivots, or a common factor in place of the divisions.)
constexpr int PT = 256;
__global__ void __launch_bounds__(PT) k_sweep_panel(int B, const double* D, int k0, double* W, double* C, double* P,
                                                    int* __restrict__ info) {
    __shared__ double A[PB][PB + 1], Ps[PB][PB + 1], Wh[PH][PH + 1], Xh[PH][PH + 1], Cs[PR][PB + 1];
    __shared__ SweepShared sh;
    const int t = threadIdx.x;
    const int r0 = blockIdx.x * PR;
    const bool pivot_rows = r0 >= k0 && r0 < k0 + PB, below = r0 > k0;
#pragma unroll
    for (int q = 0; q < PB * PB / PT; ++q) {
        const int r = t % PB, c = t / PB + q * (PT / PB);
        if (r >= c) A[r][c] = D[(int64_t)(k0 + c) * B + k0 + r];
    }
    // above the pivot block the column is held as a row of the lower triangle
    const int rr = below ? t % PR : t / PB, cc = below ? t / PR : t % PB;
    if (!pivot_rows) Cs[rr][cc] = below ? D[(int64_t)(k0 + cc) * B + r0 + rr] : D[(int64_t)(r0 + rr) * B + k0 + cc];
    __syncthreads();
    invert16(A, Ps, 0, sh, info);
    const int x = t / PH, y = t % PH;
    {
        double w0 = 0.0, w1 = 0.0;
#pragma unroll
        for (int m = 0; m < PH; m += 2) {
            w0 = fma(A[PH + x][m], Ps[m][y], w0);
            w1 = fma(A[PH + x][m + 1], Ps[m + 1][y], w1);
        }
        Wh[x][y] = w0 + w1;
    }
    __syncthreads();
    if (x >= y) {
        double s0 = A[PH + x][PH + y], s1 = 0.0;
#pragma unroll
        for (int m = 0; m < PH; m += 2) {
            s0 = fma(-Wh[x][m], A[PH + y][m], s0);
            s1 = fma(-Wh[x][m + 1], A[PH + y][m + 1], s1);
        }
        A[PH + x][PH + y] = s0 + s1;
    }
    __syncthreads();
    invert16(A, Ps, PH, sh, info);
    {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int m = 0; m < PH; m += 2) {
            s0 = fma(Ps[PH + x][PH + m], Wh[m][y], s0);
            s1 = fma(Ps[PH + x][PH + m + 1], Wh[m + 1][y], s1);
        }
        Xh[x][y] = s0 + s1;
        Ps[PH + x][y] = Ps[y][PH + x] = -(s0 + s1);
    }
    __syncthreads();
    {
        double s0 = Ps[x][y], s1 = 0.0;
#pragma unroll
        for (int m = 0; m < PH; m += 2) {
            s0 = fma(Wh[m][x], Xh[m][y], s0);
            s1 = fma(Wh[m + 1][x], Xh[m + 1][y], s1);
        }
        Ps[x][y] = s0 + s1;
    }
    __syncthreads();
    const int r = t % PR, c = t / PR;
    if (pivot_rows) {
        P[(r + r0 - k0) * PB + c] = Ps[r + r0 - k0][c];
        return;
    }
    double w0 = 0.0, w1 = 0.0;
#pragma unroll 8
    for (int m = 0; m < PB; m += 2) {
        w0 = fma(Cs[r][m], Ps[m][c], w0);
        w1 = fma(Cs[r][m + 1], Ps[m + 1][c], w1);
    }
    W[(int64_t)c * B + r0 + r] = w0 + w1;
    C[(int64_t)c * B + r0 + r] = Cs[r][c];
}

// The sweep's update of a 32 x 16 half of a tile of the lower triangle: A_ij -=
// W_i C_j^T off the pivots, A_ik = W_i, A_kk = -P.  After the last pivots the
// matrix is -D^-1: that launch changes the sign and fills both triangles.
// (Half tiles: the two chains' 420 CTAs of 4 us balance over the SMs where 210
// of 8 us leave some of them a round behind.)
constexpr int UT = 128, UC = 16;
__global__ void __launch_bounds__(UT) k_sweep_update(int B, double* D, int k0, const double* W, const double* C,
                                                     const double* P, int last) {
    __shared__ double Ws[PB][PB + 1], Cs[PB][UC + 1];   // [pivot][row], [pivot][column]
    const int tile = (int)blockIdx.x >> 1, half = (int)blockIdx.x & 1;
    int ti = (int)((sqrtf(8.f * (float)tile + 1.f) - 1.f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= tile) ++ti;
    while (ti * (ti + 1) / 2 > tile) --ti;
    const int tj = tile - ti * (ti + 1) / 2, kt = k0 / PB;
    const int t = threadIdx.x, x = t & 15, y = t >> 4, ri = ti * PB, cj = tj * PB + half * UC;
    double v[2][2];
    if (ti == kt || tj == kt) {
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = x + 16 * p, c = half * UC + y + 8 * q;
                v[p][q] = ti == tj ? -P[r * PB + c] : (tj == kt ? W[(int64_t)c * B + ri + r] : W[(int64_t)r * B + tj * PB + c]);
            }
    } else {
#pragma unroll
        for (int q = 0; q < PB * PB / UT; ++q) {
            const int e = t + q * UT, m = e / PB, r = e % PB;
            Ws[m][r] = W[(int64_t)m * B + ri + r];
        }
#pragma unroll
        for (int q = 0; q < PB * UC / UT; ++q) {
            const int e = t + q * UT, m = e / UC, c = e % UC;
            Cs[m][c] = C[(int64_t)m * B + cj + c];
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q) v[p][q] = D[(int64_t)(cj + y + 8 * q) * B + ri + x + 16 * p];
        __syncthreads();
#pragma unroll 8
        for (int m = 0; m < PB; ++m) {
            const double w0 = Ws[m][x], w1 = Ws[m][x + 16], c0 = Cs[m][y], c1 = Cs[m][y + 8];
            v[0][0] = fma(-w0, c0, v[0][0]);
            v[1][0] = fma(-w1, c0, v[1][0]);
            v[0][1] = fma(-w0, c1, v[0][1]);
            v[1][1] = fma(-w1, c1, v[1][1]);
        }
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = ri + x + 16 * p, c = cj + y + 8 * q;
            if (!last) {
                D[(int64_t)c * B + r] = v[p][q];
            } else if (ti != tj || r >= c) {        // a diagonal tile's lower half, mirrored
                D[(int64_t)c * B + r] = -v[p][q];
                D[(int64_t)r * B + c] = -v[p][q];
            }
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
    DevBuf w, c, p, g;      // panels W and C (PB columns), pivot inverse, G column-major
    void alloc(int B) {
        w = dalloc((size_t)PB * B * sizeof(double));
        c = dalloc((size_t)PB * B * sizeof(double));
        p = dalloc((size_t)PB * PB * sizeof(double));
        g = dalloc((size_t)B * B * sizeof(double));
    }
};

// D^-1 of the SPD block D (lower triangle in, both triangles out).  Plain
// launches: as programmatic dependents the two chains hold each other up (8.4
// instead of 5.7 ms for 15 blocks of order 448).
void inv_spd(Ctx& c, double* D, int B, Chain& s, int* info) {
    const int tiles = B / PB;
    for (int k0 = 0; k0 < B; k0 += PB) {
        k_sweep_panel<<<B / PR, PT, 0, c.stream>>>(B, D, k0, s.w.as<double>(), s.c.as<double>(), s.p.as<double>(), info);
        GMGS_LAUNCHED(c);
        k_sweep_update<<<tiles * (tiles + 1), UT, 0, c.stream>>>(B, D, k0, s.w.as<double>(), s.c.as<double>(),
                                                                 s.p.as<double>(), k0 + PB == B ? 1 : 0);
        GMGS_LAUNCHED(c);
    }
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
constexpr int STEP_ROWS = 4;      // rows (warps) per CTA
constexpr int MAX_JOBS = 4;
struct StepJob {
    const double* M[2];
    const double* v[2];
    const double* base;
    double* y;
    int nseg;
};
struct StepJobs {
    StepJob j[MAX_JOBS];
    int n = 0;
    void add(double* y, const double* base, const double* M0, const double* v0, const double* M1 = nullptr,
             const double* v1 = nullptr) {
        j[n++] = {{M0, M1}, {v0, v1}, base, y, M1 ? 2 : 1};
    }
};

// One warp per row, four rows per CTA: at 2 FP64 lanes per clock per SM a
// matrix-vector product has to be spread over all SMs, and a row per warp
// needs no partial sums through memory.  Launched as a programmatic dependent
// of the previous kernel in the stream: the first 16 entries per lane (rows of
// up to 512) are loaded while that kernel finishes, then the hardware grid
// dependency is waited for, and only then are vectors read or written.
__global__ void __launch_bounds__(32 * STEP_ROWS) k_rows(int B, const __grid_constant__ StepJobs jobs) {
    pdl_begin();
    const StepJob& J = jobs.j[blockIdx.y];
    const int lane = threadIdx.x & 31, row = blockIdx.x * STEP_ROWS + (threadIdx.x >> 5);
    constexpr int PRE = 8;        // double2 per lane
    double2 m[2][PRE];
#pragma unroll
    for (int s = 0; s < 2; ++s)
        if (s < J.nseg) {
            const double2* r = reinterpret_cast<const double2*>(J.M[s] + (int64_t)row * B);
#pragma unroll
            for (int q = 0; q < PRE; ++q)
                if (64 * q < B) m[s][q] = r[32 * q + lane];
        }
    pdl_wait();
    const double b = (lane == 0 && J.base) ? J.base[row] : 0.0;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int s = 0; s < 2; ++s)
        if (s < J.nseg) {
            const double2* v = reinterpret_cast<const double2*>(J.v[s]);
#pragma unroll
            for (int q = 0; q < PRE; ++q)
                if (64 * q < B) {
                    const double2 u = v[32 * q + lane];
                    s0 = fma(m[s][q].x, u.x, s0);
                    s1 = fma(m[s][q].y, u.y, s1);
                }
            const double2* r = reinterpret_cast<const double2*>(J.M[s] + (int64_t)row * B);
            for (int q = PRE; 64 * q < B; ++q) {
                const double2 u = v[32 * q + lane], w = r[32 * q + lane];
                s0 = fma(w.x, u.x, s0);
                s1 = fma(w.y, u.y, s1);
            }
        }
    double s = s0 + s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) J.y[row] = J.base ? b - s : s;
}

void launch_step(Ctx& c, int B, const StepJobs& jobs) {
    if (jobs.n == 0) return;
    launch_chain(c, k_rows, dim3(B / STEP_ROWS, jobs.n, 1), dim3(32 * STEP_ROWS, 1, 1), 0, B, jobs);
}

int coarse_middle(int nb) { return (nb - 1) / 2; }

}  // namespace

int coarse_block_order(int n, int half_bandwidth) {
    constexpr int Q = 64;         // a lane of k_rows reads double2: rows of 64 entries
    const int want = std::max(half_bandwidth, 1);
    return std::max(Q, (std::min(want, n) + Q - 1) / Q * Q);
}

void factor_coarse(Ctx& c, CoarseBlocks& cb, const std::function<void()>& overlap) {
    const int B = cb.B, nb = cb.nb, k = coarse_middle(nb);
    const int64_t B2 = (int64_t)B * B;
    double* D = cb.sinv.as<double>();   // A_ii on entry
    double* E = cb.g.as<double>();      // E_i = A_(i,i-1) on entry (i >= 1)
    cb.gt = dalloc((size_t)nb * B2 * sizeof(double));
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
    c.trace_point("bc: coarsest block LDL^T");
    int h_info[2] = {0, 0};
    GMGS_CUDA(cudaMemcpyAsync(h_info, info.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    if (h_info[0] || h_info[1]) throw Error(GMGS_ERR_NOT_SPD, "coarsest-level matrix is not positive definite");
}

void launch_coarse_solve(Ctx& c, const CoarseBlocks& cb, double* cvec, double* x) {
    const int B = cb.B, nb = cb.nb, k = coarse_middle(nb);
    if (nb <= 0) return;
    const int64_t B2 = (int64_t)B * B;
    auto Db = [&](int i) { return cb.sinv.as<double>() + i * B2; };    // symmetric
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
        J.add(xv(k), nullptr, Db(k), cv(k));
        launch_step(c, B, J);
    }
    // backward chains, in place on x: top i = k-1..0, bottom i = k+1..nb-1
    for (int s = 0; s < steps; ++s) {
        StepJobs J;
        if (s < top) J.add(xv(k - 1 - s), xv(k - 1 - s), GT(k - s), xv(k - s));
        if (s < bot) J.add(xv(k + 1 + s), xv(k + 1 + s), GT(k + 1 + s), xv(k + s));
        launch_step(c, B, J);
    }
}

}  // namespace gmgs
