// Per-level helpers of the V-cycle PCG: trilinear restriction, deterministic
// dot products and the compact <-> dense conversions (K*x, the prolongation and the CG updates are in fine.cu and
// fine64.cu).  All kernels work on the dense slot grids described in
// gmgs_internal.cuh and are free of atomics on data (reruns are bitwise equal).
#include <type_traits>

#include "fixed96.cuh"
#include "gmgs_internal.cuh"

namespace gmgs {

static dim3 node_grid(const Grid& g, dim3 blk) {
    return dim3((g.ny + 1 + blk.x - 1) / blk.x, (g.nx + 1 + blk.y - 1) / blk.y, g.nz + 1);
}

static int ew_blocks(const Ctx& c, int64_t n) {
    int64_t b = (n + 255) / 256;
    int64_t cap = (int64_t)c.num_sms * 16;
    return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

// ---------------------------------------------------------------------------
// trilinear transfers (RestrictResidual.m, InterpolationDeviation.m)
//
// With zero values on non-solid fine nodes, the reference's restriction
// (divide by the multiplicity, gather 27 nodes per non-empty coarse element,
// weight by RI, scatter to 8 corners) equals sum_k w(k - 2C) r_f(k) over the
// 27 fine nodes around coarse node C, w = prod(1 - |d|/2); its interpolation
// equals the trilinear interpolant restricted to solid fine nodes.
// ---------------------------------------------------------------------------
// one line of the restriction stencil, (w/2 a + b) + w/2 c with w = 1, and one
// weighted accumulation (weight 1 when `centre`, else 1/2); the roundings are
// explicit so that every kernel summing in this order gives the same bits
__device__ __forceinline__ float restrict_line(float a, float b, float c) {
    return __fmaf_rn(0.5f, c, __fmaf_rn(0.5f, a, b));
}
__device__ __forceinline__ double restrict_line(double a, double b, double c) {
    return __fma_rn(0.5, c, __fma_rn(0.5, a, b));
}
__device__ __forceinline__ float restrict_acc(float acc, float v, bool centre) {
    return centre ? __fadd_rn(acc, v) : __fmaf_rn(0.5f, v, acc);
}
__device__ __forceinline__ double restrict_acc(double acc, double v, bool centre) {
    return centre ? __dadd_rn(acc, v) : __fma_rn(0.5, v, acc);
}

// the 27 values in y, x, z order
template <typename T>
__device__ __forceinline__ T restrict_lines(const T (&v)[27]) {
    T accz = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        T accx = 0;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const T* l = v + 9 * c + 3 * b;
            accx = restrict_acc(accx, restrict_line(l[0], l[1], l[2]), b == 1);
        }
        accz = restrict_acc(accz, accx, c == 1);
    }
    return accz;
}
__device__ __forceinline__ float restrict_sum(const float (&v)[27]) { return restrict_lines(v); }
// In FP64 the 30 operations of each component bound the kernel (the FP64 unit
// takes 19 clocks of the SM per warp instruction), so they are integer
// additions (190 -> 87 us at 6.4M fine nodes); the lines remain for zeros,
// infinities, NaN and values near the ends of the exponent range.  27 random
// terms: at most 2.4 2^-53 of the largest value off, FP64 in sequence 14 2^-53.
__device__ __forceinline__ double restrict_sum(const double (&v)[27]) {
    int h = 0;
#pragma unroll
    for (int k = 0; k < 27; ++k) h = max(h, abs_hi(v[k]));
    const int E = h >> 20;
    if (!sum64_holds(E)) return restrict_lines(v);
    long long t = 0;
#pragma unroll
    for (int k = 0; k < 27; ++k) t += sum64_term(v[k], E, (k % 3 != 1) + (k / 3 % 3 != 1) + (k / 9 != 1));
    return sum64_value(t, E, 0);
}

// FREE: onto the coarsest level's free DOFs, cvec[rank of the DOF] in FP64,
// instead of its dense vector (a gather launch less per V-cycle)
template <typename T, bool FREE>
__global__ void k_restrict(Grid gf, Grid gc, const uint8_t* __restrict__ nflag_c, const T* rf, T* rc,
                           const int32_t* __restrict__ rank, double* cvec) {
    const int Iy = blockIdx.x * blockDim.x + threadIdx.x;
    const int Ix = blockIdx.y * blockDim.y + threadIdx.y;
    const int Iz = blockIdx.z;
    pdl_begin();
    if (Iy > gc.ny || Ix > gc.nx) return;
    const int64_t cs = gc.slot(Iy, Ix, Iz);
    const int64_t Sf = gf.slots, Sc = gc.slots, sx = gf.sx(), sz = gf.sz();
    constexpr int R = chk::RESTRICT;
    pdl_wait();
    if (!(chk::ld(nflag_c, cs, Sc, R) & NF_SOLID)) {
        if (FREE) return;
        chk::st(rc, cs, 3 * Sc, R, 0);
        chk::st(rc, cs + Sc, 3 * Sc, R, 0);
        chk::st(rc, cs + 2 * Sc, 3 * Sc, R, 0);
        return;
    }
    const int64_t f0 = gf.slot(2 * Iy, 2 * Ix, 2 * Iz);
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
        T v[27];
#pragma unroll
        for (int k = 0; k < 27; ++k)
            v[k] = chk::ld(rf, comp * Sf + f0 + (k / 3 % 3 - 1) * sx + (k / 9 - 1) * sz + (k % 3 - 1), 3 * Sf, R);
        const T accz = restrict_sum(v);
        if (FREE) {
            const int at = chk::ld(rank, cs + comp * Sc, 3 * Sc, R);
            if (at >= 0) cvec[at] = (double)accz;
        } else {
            chk::st(rc, cs + comp * Sc, 3 * Sc, R, accz);
        }
    }
}

template <typename T>
void launch_restrict(Ctx& c, const Grid& gf, const Grid& gc, const uint8_t* nflag_c, const T* rf, T* rc) {
    dim3 blk(32, 4, 1);
    launch_chain(c, k_restrict<T, false>, node_grid(gc, blk), blk, 0, gf, gc, nflag_c, rf, rc, nullptr, nullptr);
}
template <typename T>
void launch_restrict_free(Ctx& c, const Grid& gf, const Grid& gc, const uint8_t* nflag_c, const T* rf, const int32_t* rank,
                          double* cvec) {
    dim3 blk(32, 4, 1);
    launch_chain(c, k_restrict<T, true>, node_grid(gc, blk), blk, 0, gf, gc, nflag_c, rf, nullptr, rank, cvec);
}
template void launch_restrict<double>(Ctx&, const Grid&, const Grid&, const uint8_t*, const double*, double*);
template void launch_restrict<float>(Ctx&, const Grid&, const Grid&, const uint8_t*, const float*, float*);
template void launch_restrict_free<double>(Ctx&, const Grid&, const Grid&, const uint8_t*, const double*, const int32_t*,
                                           double*);
template void launch_restrict_free<float>(Ctx&, const Grid&, const Grid&, const uint8_t*, const float*, const int32_t*,
                                          double*);

// ---------------------------------------------------------------------------
// deterministic dot product: fixed grid-stride partition, fixed-order block
// reduction, and the last block to finish sums the partials in index order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    v = 0;
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;   // valid in thread 0
}

template <typename Ta, typename Tb>
__global__ void __launch_bounds__(256) k_dot(int64_t n, const Ta* __restrict__ a, const Tb* __restrict__ b,
                                             double* __restrict__ partials, unsigned int* ticket,
                                             double* __restrict__ out) {
    __shared__ double sh[32];
    __shared__ bool last;
    double s = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += (double)a[i] * (double)b[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) {
        __threadfence();
        double t = 0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) t += ((volatile double*)partials)[i];
        t = block_sum(t, sh);
        if (threadIdx.x == 0) {
            *out = t;
            *ticket = 0;
        }
    }
}

template <typename Ta, typename Tb>
void launch_dot(Ctx& c, const DotScratch& s, int64_t n, const Ta* a, const Tb* b, double* out) {
    k_dot<Ta, Tb><<<s.blocks, 256, 0, c.stream>>>(n, a, b, s.partials, s.ticket, out);
    GMGS_LAUNCHED(c);
}
template void launch_dot<double, double>(Ctx&, const DotScratch&, int64_t, const double*, const double*, double*);

// ---------------------------------------------------------------------------
// compact interleaved <-> dense planes
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_c2d(int64_t nn, int64_t S, const int32_t* __restrict__ ns, const double* __restrict__ src,
                      T* __restrict__ dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = ns[i];
        dst[s] = (T)src[3 * i];
        dst[s + S] = (T)src[3 * i + 1];
        dst[s + 2 * S] = (T)src[3 * i + 2];
    }
}
template <typename T>
__global__ void k_d2c(int64_t nn, int64_t S, const int32_t* __restrict__ ns, const T* __restrict__ src,
                      double* __restrict__ dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = ns[i];
        dst[3 * i] = (double)src[s];
        dst[3 * i + 1] = (double)src[s + S];
        dst[3 * i + 2] = (double)src[s + 2 * S];
    }
}
template <typename T>
void launch_compact_to_dense(Ctx& c, int64_t nn, int64_t S, const int32_t* ns, const double* src, T* dst) {
    k_c2d<T><<<ew_blocks(c, nn), 256, 0, c.stream>>>(nn, S, ns, src, dst);
    GMGS_LAUNCHED(c);
}
template <typename T>
void launch_dense_to_compact(Ctx& c, int64_t nn, int64_t S, const int32_t* ns, const T* src, double* dst) {
    k_d2c<T><<<ew_blocks(c, nn), 256, 0, c.stream>>>(nn, S, ns, src, dst);
    GMGS_LAUNCHED(c);
}
template void launch_compact_to_dense<double>(Ctx&, int64_t, int64_t, const int32_t*, const double*, double*);
template void launch_compact_to_dense<float>(Ctx&, int64_t, int64_t, const int32_t*, const double*, float*);
template void launch_dense_to_compact<double>(Ctx&, int64_t, int64_t, const int32_t*, const double*, double*);
template void launch_dense_to_compact<float>(Ctx&, int64_t, int64_t, const int32_t*, const float*, double*);

}  // namespace gmgs
