// FP64 streaming operator kernels of the default path.
//
// GB300 issues FP64 arithmetic at about 2 lanes per clock per SM, 1/64 of its
// FP32 rate: every FP64 operation per node costs as much time as moving 11
// bytes per node through HBM, so these kernels are organised to spend as few
// FP64 operations as possible and to let everything else (loads, shared
// memory, integer work) hide behind that pipe.
//
// K x on interior nodes of a uniform level: the trilinear box element's
// stencil is a sum of tensor products of 1-D operators (Coef64), so it is
// applied axis by axis (z in registers, x and y through shared memory), 66
// operations per node instead of the 117 of the assembled 27-point pairs or
// the 576 of the element form.  The 1-D second differences annihilate
// constants exactly, so the result is also more accurate than the assembled
// sum (2.6e-14 against 3.8e-14 relative on a smooth field, where |K x| is
// small against |K||x|).  The integer units do those operations on 96-bit fixed
// point, exactly and four times as fast, wherever that is the more accurate
// form (fixed96.cuh, k_fine64); FP64 arithmetic remains for the rest.
//
// Solid nodes with void elements around them take the assembled stencil of
// their own set of solid elements (256 precomputed sets, 4 lanes per node), nodes
// on elements with stored matrices the element sum (8 lanes per node), both from
// compact node lists; a level with an element scale (density) takes the element form in
// modal coordinates (k_modal64).  All parts of one K x run in one launch: the
// list blocks first, then the tiles.
//
// The vector operations around K x (Jacobi step, CG direction, CG update,
// residuals, dot products) are fused into it as in the mixed path (fine.cu).
//
// Measured at 6.4M nodes (169 x 147 x 256 elements): K x alone took 4.1 ms as
// a thread per node on the assembled pairs and eight element rows.  Axis by
// axis in FP64, with the Jacobi step and the residual in the same launch, it
// took 1.44 ms, with the CG update 1.80 ms, at 80 % of the FP64 unit; with the
// stencil on integers 0.70 and 1.14 ms; K x alone 0.64 ms since the columns of
// a warp avoid bank conflicts and the halo is spread over all warps.  No one
// unit bounds them then (FP64 unit about a third, issue slots about half,
// shared-memory pipe 40 % busy): two CTAs of 128 registers per SM do.
// A PCG iteration went from 16.9 to 2.9 ms.
#include <algorithm>
#include <atomic>

#include "element_host.h"
#include "fine.cuh"
#include "fine64.cuh"
#include "fixed96.cuh"

namespace gmgs {

namespace {

constexpr int TY = 16, TX = 16;
constexpr int NT = TY * TX;
constexpr int HY = TY + 2, HX = TX + 2;
constexpr int NP = HY * HX;          // points of a tile plane with its one-node halo
constexpr int NHALO = NP - NT;       // 68
constexpr int NXP = HY * TX;         // points of the x stage: the tile's columns with the y halo
constexpr int BND_LANES = 4;         // lanes per boundary node
constexpr int ELEM_LANES = 8;        // lanes per node on stored matrices

__host__ __device__ constexpr int field_arrays64(int mode) {
    return mode == M64_PLAIN ? 1 : (mode == M64_CG_UPDATE_JACOBI ? 3 : 2);
}
__host__ __device__ constexpr bool has_dot(int mode) { return mode == M64_CG_UPDATE_JACOBI || mode == M64_CG_DIRECTION; }

// input arrays of the field, in the order form() takes them
template <int MODE>
__device__ __forceinline__ const double* field_array(const Args64& a, int j) {
    if (MODE == M64_PLAIN) return a.v;
    if (MODE == M64_VCYCLE_DOWN) return j == 0 ? a.r : a.w;
    if (MODE == M64_CG_UPDATE_JACOBI) return j == 0 ? a.r : (j == 1 ? a.w : a.q);
    return j == 0 ? a.z : a.pold;
}

// one component of the field from its inputs; s: what the epilogue needs of
// them at the node itself (r of the down-sweep, r_m of the update)
template <int MODE>
__device__ __forceinline__ void form(double f0, double f1, double f2, double ab, int first, double& v, double& s) {
    s = 0.0;
    if (MODE == M64_PLAIN) {
        v = f0;
    } else if (MODE == M64_VCYCLE_DOWN) {
        s = f0;
        v = f0 * f1;
    } else if (MODE == M64_CG_UPDATE_JACOBI) {
        s = first ? f0 : fma(-ab, f2, f0);
        v = s * f1;
    } else {
        v = first ? f0 : fma(ab, f1, f0);
    }
}
template <int MODE>
__device__ __forceinline__ void form_at(const Args64& a, int64_t i, int64_t n3, double ab, double& v, double& s) {
    constexpr int F = chk::F64_FIELD;
    const double f0 = chk::ld(field_array<MODE>(a, 0), i, n3, F);
    double f1 = 0.0, f2 = 0.0;
    const bool need1 = MODE == M64_VCYCLE_DOWN || MODE == M64_CG_UPDATE_JACOBI || (MODE == M64_CG_DIRECTION && !a.first);
    if (need1) f1 = chk::ld(field_array<MODE>(a, 1), i, n3, F);
    if (MODE == M64_CG_UPDATE_JACOBI && !a.first) f2 = chk::ld(field_array<MODE>(a, 2), i, n3, F);
    form<MODE>(f0, f1, f2, ab, a.first, v, s);
}

// outputs of one DOF from y = (A v), already zeroed on fixed DOFs; px, xx: p
// and x of the node (update only)
template <int MODE>
__device__ __forceinline__ void finish_dof(const Args64& a, int64_t i, int64_t n3, double y, double v, double s, double px,
                                           double xx, double ab, double& dot) {
    constexpr int O = chk::F64_OUT;
    if (MODE == M64_PLAIN) {
        chk::st(a.out, i, n3, O, y);
    } else if (MODE == M64_VCYCLE_DOWN) {
        chk::st(a.out, i, n3, O, s - y);
    } else if (MODE == M64_CG_UPDATE_JACOBI) {
        // x += alpha p + dx; r = r_m - A dx; the caller removes the last dx
        // (of an iteration that does not run) when the solve stops
        chk::st(a.x, i, n3, O, xx + (a.first ? v : fma(ab, px, v)));
        chk::st(a.out, i, n3, O, s - y);
        dot = fma(s, s, dot);
    } else {
        chk::st(a.pout, i, n3, O, v);
        chk::st(a.out, i, n3, O, y);
        dot = fma(v, y, dot);
    }
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// beta = r.z / r_old.z_old of the direction, alpha = r.z / p.q of the update:
// one division per CTA
template <int MODE>
__device__ __forceinline__ double step_length(const Args64& a) {
    if (!has_dot(MODE) || a.first) return 0.0;
    __shared__ double s_ab;
    if (threadIdx.x == 0) s_ab = a.scal[a.cur] / a.scal[MODE == M64_CG_DIRECTION ? (a.cur ^ 1) : 2];
    __syncthreads();
    return s_ab;
}

// sum over the N lanes of a list node
template <int N>
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
    for (int o = 1; o < N; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A boundary node, 4 lanes: the assembled stencil of its solid elements, lane
// j taking the j-th, j+4-th, ... of the offsets those elements reach (18 of 27
// on a face).  Fewer lanes per node spend fewer FP64 operations on the sum
// across them (8 lanes over all 27 offsets: 560 lane operations per node of
// the update; 4 over the reached ones: 330).
// A node on stored matrices, 8 lanes: the element sum, lane j taking the
// coupling to element node j.
template <int MODE, bool BND>
__device__ void list_node(const Level64& L, const Args64& a, int at, int j, double& dot) {
    const Grid& g = L.g;
    const int64_t S = g.slots, n3 = 3 * S, sx = g.sx(), sz = g.sz();
    const int count = BND ? L.n_bnd : L.n_perel;
    const bool active = at < count;
    const int64_t n = active ? chk::ld(BND ? L.bnd : L.perel, at, count, chk::F64_LIST) : 0;
    double y[3] = {0.0, 0.0, 0.0};
    // the 8 elements around the node, all loads in flight together: -1 void, 0 uniform, k the stored matrix k - 1
    int type[8];
    uint32_t mask = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int64_t es = n - (e & 1) - ((e >> 1) & 1) * sx - (e >> 2) * sz;
        type[e] = -1;
        if (active && chk::ld(L.emask, es, S, chk::F64_LIST)) {
            mask |= 1u << e;
            type[e] = !BND && L.etype ? chk::ld(L.etype, es, S, chk::F64_LIST) : 0;
            if (type[e] > 0 && !chk::ok(type[e] - 1, L.nK, chk::F64_LIST)) type[e] = -1;
        }
    }
    pdl_wait();                      // the lists, masks and types above do not change during a solve
    const double ab = step_length<MODE>(a);
    if (BND) {
        const MaskStencil& T = L.mask_stencil[mask];      // mask 0 (idle lanes): no offsets
        for (int t = j; t < T.n; t += BND_LANES) {
            const int k = T.k[t];
            const int64_t m = n + off_y(k) + off_x(k) * sx + off_z(k) * sz;
            double v[3], s;
#pragma unroll
            for (int b = 0; b < 3; ++b) form_at<MODE>(a, m + b * S, n3, ab, v[b], s);
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int b = 0; b < 3; ++b) y[c] = fma(T.S[t][3 * c + b], v[b], y[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) y[c] = L.kscale * lanes_sum<BND_LANES>(y[c]);
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (type[e] < 0) continue;                    // uniform across the node's lanes
            const int A = e & 1, B = (e >> 1) & 1, C = e >> 2;
            const int64_t m = n - A - B * sx - C * sz + corner_y(j) + corner_x(j) * sx + corner_z(j) * sz;
            const double* K = (type[e] > 0 ? L.Ks + (int64_t)(type[e] - 1) * KE : L.ke0) + 3 * corner_of(A, B, C) * 24 + 3 * j;
            const double k = type[e] > 0 ? 1.0 : L.kscale;
            double v[3], s;
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                form_at<MODE>(a, m + b * S, n3, ab, v[b], s);
                v[b] *= k;
            }
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int b = 0; b < 3; ++b) y[c] = fma(K[24 * c + b], v[b], y[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) y[c] = lanes_sum<ELEM_LANES>(y[c]);
    }
    if (active && j < 3) {
        const uint32_t f = chk::ld(L.nflag, n, S, chk::F64_LIST);
        const int64_t i = n + j * S;
        double v, s, px = 0.0, xx = 0.0;
        form_at<MODE>(a, i, n3, ab, v, s);
        if (MODE == M64_CG_UPDATE_JACOBI) {
            xx = chk::ld((const double*)a.x, i, n3, chk::F64_FIELD);
            if (!a.first) px = chk::ld(a.pold, i, n3, chk::F64_FIELD);
        }
        double yj = j == 0 ? y[0] : (j == 1 ? y[1] : y[2]);
        if (f & (NF_FIX_X << j)) yj = 0.0;
        finish_dof<MODE>(a, i, n3, yj, v, s, px, xx, ab, dot);
    }
}

template <int MODE>
__device__ __forceinline__ void dot_finish(double dot, const Args64& a, double* sh) {
    if (has_dot(MODE)) grid_dot_finish(dot, DotOut{a.dot.partials, a.dot.ticket, a.dot.out}, sh);
}

// A warp holds the y columns x and x + 8 of the tile: at the planes' pitch of
// 18 their 16 words each fall into opposite halves of the 32 banks (columns x
// and x + 1 would share two banks, a second pass for every access: 44 M of 100 M
// shared-memory wavefronts of a down-sweep at 6.4M nodes).
__device__ __forceinline__ int tile_y(int tid) { return tid & (TY - 1); }
__device__ __forceinline__ int tile_x(int tid) { return (tid >> 5) + 8 * ((tid >> 4) & 1); }
static_assert(TY == 16 && TX == 16 && HY == 18, "two columns 8 apart are 16 banks apart");

// this thread's points of a tile plane: its own node and point k of the
// one-node halo (none for k >= NHALO)
struct Points {
    int pc, ph;             // index in the (HX x HY) plane
    int64_t cbase, hbase;   // slot at z = 0
    bool cok, hok;          // inside the allocated grid
    int cy, cx;
    __device__ Points(const Grid& g, int y0, int x0, int tid, int k) {
        const int ly = tile_y(tid), lx = tile_x(tid);
        cy = y0 + ly;
        cx = x0 + lx;
        pc = (ly + 1) + (lx + 1) * HY;
        cok = cy <= g.ny + 1 && cx <= g.nx + 1;
        cbase = g.slot(cy, cx, 0);
        ph = 0;
        hbase = 0;
        hok = false;
        if (k < NHALO) {
            int hy, hx;
            if (k < 2 * TY) { hx = k < TY ? 0 : HX - 1; hy = 1 + (k & (TY - 1)); }            // x faces: whole rows
            else { hy = (k & 1) ? HY - 1 : 0; hx = (k - 2 * TY) >> 1; }                       // y faces with the corners
            ph = hy + hx * HY;
            const int gy = y0 - 1 + hy, gx = x0 - 1 + hx;
            hok = gy <= g.ny + 1 && gx <= g.nx + 1;
            hbase = g.slot(gy, gx, 0);
        }
    }
};

// the z and x stages' fields (9 each, three words a value), the field inputs of a plane
template <int MODE>
constexpr size_t fine64_smem() {
    return 12 * (9 * NP + 9 * NXP) + sizeof(double) * (3 * field_arrays64(MODE) * NP);
}

// The three stages run on 96-bit integers (fixed96.cuh) where that is at least
// as accurate as FP64 arithmetic at every node.  The values of the three planes
// are multiples of 2^-82 of the largest one: exact down to 2^-30 of it, all sums
// are exact, and the products with the coefficients (exact as fractions) drop
// less than 3 units each, about 70 units of a row in all.  A row of FP64 rounds
// its terms at 2^-53, so integers lose nothing
//   - in a window whose non-zero components all reach 2^-23 of its largest value:
//     every row then has a term of that size or none at all
//   - elsewhere, if every row's largest term (own component: 27 neighbours;
//     another one: the 12 whose 3 x 3 block couples the two) reaches 2^-20 of the
//     largest value or all are zero: what is cut off the smaller values, at most
//     240 units, is less than that term's rounding.  A component at rounding
//     level, as on a symmetry plane, fails the first test and passes this one
//     (rows_hold: 27 loads of packed exponents a node, in such windows only).
// Both limits shrink by the spread of the coefficients.  A point's largest
// component does not do as a test: u = (2^-60, 0, 1) at one node has an x row of
// 2^-60, which the z component does not couple into.  Other windows, those with
// infinities or NaN, or near the ends of the exponent range take the same stages in
// FP64, as do voxels so flat that a coefficient is below 2^-11 of the largest one.
constexpr int FIXED_RANGE = 23, FIXED_ROW_MARGIN = 3;

// how far a value lies below the largest exponent E, in binary orders; 255: zero
// (a subnormal, which to_fixed drops, lies at the exponent 0)
__device__ __forceinline__ uint32_t below_top(double v, int E) {
    const int h = abs_hi(v);
    return h | __double2loint(v) ? (uint32_t)min(E - (h >> 20), 254) : 255u;
}

// Whether every row of this node reaches the limit: a component's own term at
// any of the 27 points, another component's where both axes differ (x and y for
// the pair of components x, y).  k: below_top of the three components, a byte
// each, for the planes iz - 1, iz, iz + 1; pc: the node's point.
__device__ __forceinline__ bool rows_hold(const uint32_t* k, int pc, int limit) {
    uint32_t best = 0xffffffffu;
#pragma unroll 1
    for (int dz = -1; dz <= 1; ++dz)                      // not unrolled: no registers of the walk spill
#pragma unroll
        for (int o = 0; o < 9; ++o) {
            const int dy = o % 3 - 1, dx = o / 3 - 1;
            const uint32_t w = chk::ld(k, (dz + 1) * NP + pc + dy + dx * HY, 3 * NP, chk::F64_TILE) | 0xff000000u;
            best = __vminu4(best, w);
            if (dx && dy) best = __vminu4(best, __byte_perm(w, 0xffffffffu, 0x4401));         // (y, x, -)
            if (dx && dz) best = __vminu4(best, __byte_perm(w, 0xffffffffu, 0x4042));         // (z, -, x)
            if (dy && dz) best = __vminu4(best, __byte_perm(w, 0xffffffffu, 0x4124));         // (-, z, y)
        }
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int b = (int)((best >> (8 * c)) & 0xffu);
        ok = ok && (b <= limit || b == 255);
    }
    return ok;
}

// ---------------------------------------------------------------------------
// K x with the uniform matrix, axis by axis.  A CTA owns a 16 (y) x 16 (x)
// column of nodes and walks a chunk of z planes.  Per plane:
//   - the field of plane z + 1 is formed from its inputs, which cp.async has
//     brought to this thread's own places in shared memory one plane ahead
//     (each thread reads back only what it copied: no barrier)
//   - z stage: m, k and d along z at the tile's nodes and halo, from the three
//     planes in registers                                  (12 operations)
//   - x stage: sums P, Q, R of the y operators m, k, d at the tile's columns
//     and their y halo                                     (33 operations)
//   - both halos by components: a thread holds one component of one point of
//     the z halo (10 points a warp), three warps one component each of the x
//     stage's.  With all three components on the first threads, their warps did
//     twice the work of the others between two barriers (K x at 6.4M nodes 683
//     -> 639 us)
//   - y stage and the mode's vector updates at the interior nodes
// Three barriers per plane; two CTAs per SM keep the FP64 pipe fed across them.
// One buffer of field inputs, refilled right after it was read: with two, the
// CG update's CTAs took 112 KB each and left the L1 cache next to nothing (its
// loads then waited in the memory pipeline; solve 169 x 147 x 256 90.8 -> 83.3 ms).
// The square tile wastes fewer lanes than 32 x 8 on grids a little over a
// multiple of 32 (84 x 73 x 128: 82 against 74 % of the tile's nodes used).
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(NT, 2) k_fine64(Level64 L, const __grid_constant__ Coef64 cf, Args64 a, int zc, int nb_bnd,
                                                  int nb_list, int tiles_y, int tiles_x) {
    __shared__ double sh[32];
    extern __shared__ double dyn[];
    const int tid = threadIdx.x;
    const Grid& g = L.g;
    pdl_begin();
    double dot = 0.0;
    if ((int)blockIdx.x < nb_list) {
        if ((int)blockIdx.x < nb_bnd)
            list_node<MODE, true>(L, a, (int)blockIdx.x * (NT / BND_LANES) + tid / BND_LANES, tid % BND_LANES, dot);
        else
            list_node<MODE, false>(L, a, ((int)blockIdx.x - nb_bnd) * (NT / ELEM_LANES) + tid / ELEM_LANES, tid % ELEM_LANES,
                                   dot);
        dot_finish<MODE>(dot, a, sh);
        return;
    }
    const int bid = (int)blockIdx.x - nb_list;
    const int bty = bid % tiles_y, btx = bid / tiles_y % tiles_x, btz = bid / (tiles_y * tiles_x);
    const int y0 = bty * TY, x0 = btx * TX;
    const int zb = btz * zc, ze = min(zb + zc, g.nz + 1);       // node planes [zb, ze)
    uint32_t occ = 0;                                           // planes of the chunk (at most 32) with a solid node in the tile
    for (int iz = zb; iz < ze; ++iz)
        occ |= L.tile_occ[((int64_t)iz * tiles_x + btx) * tiles_y + bty] != 0 ? 1u << (iz - zb) : 0u;
    const int64_t S = g.slots, n3 = 3 * S, sz = g.sz();
    const int lane = tid & 31, hcmp = lane % 3, hk = lane < 30 ? (tid >> 5) * 10 + lane / 3 : NHALO;
    const Points p(g, y0, x0, tid, hk);                         // one component of a halo point per thread
    const int64_t hbase = p.hbase + hcmp * S;
    const bool own = p.cy <= g.ny && p.cx <= g.nx;
    uint32_t f_next = own ? chk::ld(L.nflag, p.cbase + zb * sz, S, chk::F64_FIELD) : 0u;
    pdl_wait();                                                 // occupancy and flags do not change during a solve
    if (!occ) {                                                 // uniform across the CTA
        dot_finish<MODE>(0.0, a, sh);
        return;
    }
    const double ab = step_length<MODE>(a);
    constexpr int NA = field_arrays64(MODE);
    constexpr int R = chk::F64_TILE;
    double* const stage = dyn;                    // [NA * 3][NP] field inputs of a plane
    double* const Zb = stage + NA * 3 * NP;   // 9 fields of the z stage: m, k, d of the three components
    double* const Xb = Zb + 9 * NP * 3 / 2;       // 9 fields of the x stage: P, Q, R
    uint32_t* const Zw = reinterpret_cast<uint32_t*>(Zb);      // the same as three words a value
    uint32_t* const Xw = reinterpret_cast<uint32_t*>(Xb);
    const int narr = ((MODE == M64_CG_UPDATE_JACOBI || MODE == M64_CG_DIRECTION) && a.first) ? NA - 1 : NA;

    // field inputs of plane iz to this thread's places of st
    auto issue = [&](int iz, double* st) {
#pragma unroll
        for (int j = 0; j < NA; ++j) {
            if (j >= narr) break;
            const double* src = field_array<MODE>(a, j);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int64_t ic = p.cbase + iz * sz + c * S;
                if (p.cok && chk::ok(ic, n3, chk::F64_FIELD)) cp_async8(st + (j * 3 + c) * NP + p.pc, src + ic);
            }
            const int64_t ih = hbase + iz * sz;
            if (p.hok && chk::ok(ih, n3, chk::F64_FIELD)) cp_async8(st + (j * 3 + hcmp) * NP + p.ph, src + ih);
        }
    };
    auto formed_one = [&](const double* st, int pt, int c, bool ok, double& v, double& s) {
        v = s = 0.0;
        if (ok) {
            const double f0 = chk::ld(st, c * NP + pt, NA * 3 * NP, R);
            double f1 = 0.0, f2 = 0.0;
            if (NA > 1 && narr > 1) f1 = chk::ld(st, (3 + c) * NP + pt, NA * 3 * NP, R);
            if (NA > 2 && narr > 2) f2 = chk::ld(st, (6 + c) * NP + pt, NA * 3 * NP, R);
            form<MODE>(f0, f1, f2, ab, a.first, v, s);
        }
    };
    auto formed = [&](const double* st, double v[3], double s[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) formed_one(st, p.pc, c, p.cok, v[c], s[c]);
    };
    double vm[3], vc[3], vp[3], hm, hc, hp, sc[3], sp[3], unused[3], unused_h;
    // of a formed plane, over the CTA: the largest biased exponent, and in the
    // upper half 2047 minus the smallest one of a non-zero component
    __shared__ uint32_t s_exp[2][NT / 32];
    auto put_exp = [&](int par, const double* u, double h) {
        int top = 0, low = 0;
        auto take = [&](double v) {
            const int a = abs_hi(v), e = a >> 20;
            top = max(top, e);
            low = max(low, a | __double2loint(v) ? 2047 - e : 0);
        };
        take(h);
#pragma unroll
        for (int c = 0; c < 3; ++c) take(u[c]);
        top = __reduce_max_sync(0xffffffffu, top);
        low = __reduce_max_sync(0xffffffffu, low);
        if ((tid & 31) == 0) s_exp[par][tid >> 5] = (uint32_t)(top | low << 16);
    };
    auto get_exp = [&](int par) {
        uint32_t e = s_exp[par][0];
#pragma unroll
        for (int w = 1; w < NT / 32; ++w) e = __vmaxu2(e, s_exp[par][w]);
        return e;
    };
    // the first two planes pass through the stages' buffers, all three in flight together
    static_assert(12 * 9 * NXP >= 8 * 3 * NA * NP && NXP <= NP, "a plane's field inputs fit");
    issue(zb - 1, Zb);
    cp_async_commit();
    issue(zb, Xb);
    cp_async_commit();
    issue(zb + 1, stage);
    cp_async_commit();
    cp_async_wait<2>();
    formed(Zb, vm, unused);
    formed_one(Zb, p.ph, hcmp, p.hok, hm, unused_h);
    cp_async_wait<1>();
    formed(Xb, vc, sc);
    formed_one(Xb, p.ph, hcmp, p.hok, hc, unused_h);
    put_exp(0, vm, hm);
    put_exp(1, vc, hc);
    __syncthreads();
    uint32_t em = get_exp(0), ec = get_exp(1);
    __syncthreads();

    auto z_one = [&](int pt, int c, double um, double u, double up) {
        const double s = um + up;
        chk::st(Zb, c * NP + pt, 9 * NP, R, fma(4.0, u, s));
        chk::st(Zb, (3 + c) * NP + pt, 9 * NP, R, fma(2.0, u, -s));
        chk::st(Zb, (6 + c) * NP + pt, 9 * NP, R, up - um);
    };
    // P, Q, R of component c at plane point (yy, x column): operands at pt - HY, pt, pt + HY
    auto x_one = [&](int pt, int c, double& P, double& Q, double& Rr) {
        auto zf = [&](int f, int o) { return chk::ld((const double*)Zb, f * NP + pt + o * HY, 9 * NP, R); };
        auto mx = [&](int f) { return fma(4.0, zf(f, 0), zf(f, -1) + zf(f, 1)); };
        auto dx = [&](int f) { return zf(f, 1) - zf(f, -1); };
        const double u = zf(c, 0), s = zf(c, -1) + zf(c, 1), kM = fma(2.0, u, -s);
        Q = fma(4.0, u, s);
        P = fma(cf.az[c], mx(3 + c), cf.ax[c] * kM);
        if (c != 1) P = fma(cf.gxz, dx(c == 0 ? 8 : 6), P);
        Rr = c == 0 ? dx(1) : (c == 1 ? fma(cf.gyz, mx(8), cf.gxy * dx(0)) : mx(7));
    };
    // the same stages on 96-bit integers, all values multiples of 2^(E - 1105)
    auto put_w = [](uint32_t* w, int n, int k, int pt, const I96& x) {
        chk::st(w, (3 * k + 0) * n + pt, 27 * n, R, x.a);
        chk::st(w, (3 * k + 1) * n + pt, 27 * n, R, x.b);
        chk::st(w, (3 * k + 2) * n + pt, 27 * n, R, x.c);
    };
    auto get_w = [](const uint32_t* w, int n, int k, int pt) {
        return I96{chk::ld(w, (3 * k + 0) * n + pt, 27 * n, R), chk::ld(w, (3 * k + 1) * n + pt, 27 * n, R),
                   chk::ld(w, (3 * k + 2) * n + pt, 27 * n, R)};
    };
    auto z_one_i = [&](int pt, int c, double um, double u, double up, int E) {
        const I96 l = to_fixed(um, E), m = to_fixed(u, E), r = to_fixed(up, E), t = l + r;
        put_w(Zw, NP, c, pt, t + shl<2>(m));
        put_w(Zw, NP, 3 + c, pt, shl<1>(m) - t);
        put_w(Zw, NP, 6 + c, pt, r - l);
    };
    auto x_one_i = [&](int pt, int c, I96& P, I96& Q, I96& Rr) {
        auto zf = [&](int k, int o) { return get_w(Zw, NP, k, pt + o * HY); };
        auto mx = [&](int k) { return zf(k, -1) + zf(k, 1) + shl<2>(zf(k, 0)); };
        auto dx = [&](int k) { return zf(k, 1) - zf(k, -1); };
        const I96 u = zf(c, 0), t = zf(c, -1) + zf(c, 1);
        Q = t + shl<2>(u);
        P = mul_frac(shl<1>(u) - t, cf.fax[c]) + mul_frac(mx(3 + c), cf.faz[c]);
        if (c != 1) P = P - mul_frac(dx(c == 0 ? 8 : 6), cf.fgxz);
        Rr = c == 0 ? dx(1) : (c == 1 ? mul_frac(dx(0), cf.fgxy) + mul_frac(mx(8), cf.fgyz) : mx(7));
    };
    const int xc = p.pc - HY;                // own point of the x stage
    // the y halo of the x stage: a component to each of the last three warps
    const int hx_c = (tid >> 5) - (NT / 32 - 3), hyy = (lane & 1) ? HY - 1 : 0;
    const int hz_pt = hyy + ((lane >> 1) + 1) * HY, hx_pt = hyy + (lane >> 1) * HY;
    static_assert(2 * TX == 32 && NHALO <= 10 * (NT / 32), "points of the y halo and of the z halo by warps");

#pragma unroll 1
    for (int iz = zb; iz < ze; ++iz) {
        const int64_t n = p.cbase + iz * sz;
        const uint32_t f = f_next;              // loaded a plane ahead: the x and p loads below depend on it
        if (own && iz + 1 < ze) f_next = chk::ld(L.nflag, n + sz, S, chk::F64_FIELD);
        const bool node = (f & NF_INTERIOR) != 0;
        double xx[3] = {0.0, 0.0, 0.0}, px[3] = {0.0, 0.0, 0.0};
        if (MODE == M64_CG_UPDATE_JACOBI && node) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xx[c] = chk::ld((const double*)a.x, n + c * S, n3, chk::F64_FIELD);
                if (!a.first) px[c] = chk::ld(a.pold, n + c * S, n3, chk::F64_FIELD);
            }
        }
        cp_async_wait<0>();
        formed(stage, vp, sp);
        formed_one(stage, p.ph, hcmp, p.hok, hp, unused_h);
        put_exp((iz - zb) & 1, vp, hp);
        __syncthreads();
        if (iz + 1 < ze) issue(iz + 2, stage);                   // the places just read
        cp_async_commit();
        const uint32_t ep = get_exp((iz - zb) & 1), ew = __vmaxu2(em, __vmaxu2(ec, ep));
        const int E = (int)(ew & 0xffffu);
        em = ec;
        ec = ep;
        const bool here = (occ >> (iz - zb)) & 1u;               // uniform across the CTA, as the next ones
        bool fixed = here && cf.fixed && E > 1023 - 700 && E < 1023 + 700;
        if (fixed && E - 2047 + (int)(ew >> 16) > cf.fixed) {
            auto put_k = [&](int plane, const double* u, double h) {
                chk::st(Zw, plane * NP + p.pc, 3 * NP, R, below_top(u[0], E) | below_top(u[1], E) << 8 | below_top(u[2], E) << 16);
                if (hk < NHALO)
                    chk::st(reinterpret_cast<uint8_t*>(Zw), 4 * (plane * NP + p.ph) + hcmp, 12 * NP, R, below_top(h, E));
            };
            put_k(0, vm, hm);
            put_k(1, vc, hc);
            put_k(2, vp, hp);
            __syncthreads();
            fixed = __syncthreads_and(!node || rows_hold(Zw, p.pc, cf.fixed - FIXED_ROW_MARGIN));
        }
        if (!here) {
        } else if (fixed) {
#pragma unroll
            for (int c = 0; c < 3; ++c) z_one_i(p.pc, c, vm[c], vc[c], vp[c], E);
            if (hk < NHALO) z_one_i(p.ph, hcmp, hm, hc, hp, E);
            __syncthreads();
            I96 P[3], Q[3], Rr[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (hx_c == c) {                                 // uniform across the warp
                    I96 hP, hQ, hR;
                    x_one_i(hz_pt, c, hP, hQ, hR);
                    put_w(Xw, NXP, c, hx_pt, hP);
                    put_w(Xw, NXP, 3 + c, hx_pt, hQ);
                    put_w(Xw, NXP, 6 + c, hx_pt, hR);
                }
            }
            // a warp holds whole y columns of the tile, so its x stage is read by its own y stage alone
            if (__any_sync(0xffffffffu, node)) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    x_one_i(p.pc, c, P[c], Q[c], Rr[c]);
                    put_w(Xw, NXP, c, xc, P[c]);
                    put_w(Xw, NXP, 3 + c, xc, Q[c]);
                    put_w(Xw, NXP, 6 + c, xc, Rr[c]);
                }
            }
            __syncthreads();
            if (node) {
                const int ex = E - 1105 + cf.cexp + 1023 + 95;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    auto xf = [&](int k, int o) { return get_w(Xw, NXP, 3 * k + c, xc + o); };
                    const I96 mP = xf(0, -1) + xf(0, 1) + shl<2>(P[c]);
                    const I96 kQ = shl<1>(Q[c]) - (xf(1, -1) + xf(1, 1));
                    I96 dR = xf(2, 1) - xf(2, -1);
                    if (c != 1) dR = mul_frac(dR, c == 0 ? cf.fgxy : cf.fgyz);
                    double y = to_double(mP + mul_frac(kQ, cf.fay[c]) + dR, ex);
                    if (f & (NF_FIX_X << c)) y = 0.0;
                    finish_dof<MODE>(a, n + c * S, n3, y, vc[c], sc[c], px[c], xx[c], ab, dot);
                }
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) z_one(p.pc, c, vm[c], vc[c], vp[c]);
            if (hk < NHALO) z_one(p.ph, hcmp, hm, hc, hp);
            __syncthreads();
            double P[3], Q[3], Rr[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (hx_c == c) {
                    double hP, hQ, hR;
                    x_one(hz_pt, c, hP, hQ, hR);
                    chk::st(Xb, c * NXP + hx_pt, 9 * NXP, R, hP);
                    chk::st(Xb, (3 + c) * NXP + hx_pt, 9 * NXP, R, hQ);
                    chk::st(Xb, (6 + c) * NXP + hx_pt, 9 * NXP, R, hR);
                }
            }
            // a warp holds whole y columns of the tile, so its x stage is read by its own y stage alone
            if (__any_sync(0xffffffffu, node)) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    x_one(p.pc, c, P[c], Q[c], Rr[c]);
                    chk::st(Xb, c * NXP + xc, 9 * NXP, R, P[c]);
                    chk::st(Xb, (3 + c) * NXP + xc, 9 * NXP, R, Q[c]);
                    chk::st(Xb, (6 + c) * NXP + xc, 9 * NXP, R, Rr[c]);
                }
            }
            __syncthreads();
            if (node) {
                const double gr[3] = {cf.gxy, 1.0, cf.gyz};
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    auto xf = [&](int k, int o) { return chk::ld((const double*)Xb, (3 * k + c) * NXP + xc + o, 9 * NXP, R); };
                    const double mP = fma(4.0, P[c], xf(0, -1) + xf(0, 1));
                    const double kQ = fma(2.0, Q[c], -(xf(1, -1) + xf(1, 1)));
                    const double dR = xf(2, 1) - xf(2, -1);
                    double y = fma(cf.ay[c], kQ, mP);
                    y = c == 1 ? y + dR : fma(gr[c], dR, y);
                    if (f & (NF_FIX_X << c)) y = 0.0;
                    finish_dof<MODE>(a, n + c * S, n3, y, vc[c], sc[c], px[c], xx[c], ab, dot);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            vm[c] = vc[c];
            vc[c] = vp[c];
            sc[c] = sp[c];
        }
        hm = hc;
        hc = hp;
    }
    cp_async_wait<0>();
    dot_finish<MODE>(dot, a, sh);
}

// ---------------------------------------------------------------------------
// K x with a scale per element (density), element form in modal coordinates.
// With the sums s = u0 + u1 and differences e = u1 - u0 along each axis, the
// 1-D element operators are diagonal or have one entry (mass: h/4 s s' +
// h/12 e e'; stiffness: e e'/h; derivative: e s'/2), so the 24 x 24 element
// matrix becomes 45 multiplications, and the transforms along z and their
// sums at the nodes are shared between neighbouring elements: about 235
// operations per node against 600 for eight elements' rows.  Rigid
// translations (the all-s modes) drop out exactly.
// Walk as in k_fine64; layer l lies between the node planes l and l + 1.
// ---------------------------------------------------------------------------
constexpr int EY = TY + 1, EX = TX + 1, NE = EY * EX;      // elements of a layer that touch the tile
constexpr size_t MODAL_SMEM = sizeof(double) * (6 * NP + 24 * NE);

// coefficients of the modal element matrix
struct Modal {
    double m[3][2];           // mass per axis (x, y, z): [0] sum mode, [1] difference mode
    double k[3];              // stiffness per axis on the difference mode
    double lam4, mu4, lam, mu, sgn_xy, sgn_xz, sgn_yz;
};
__device__ __forceinline__ Modal modal_coefs(const Coef64& cf) {
    Modal c;
    const double h[3] = {cf.hx, cf.hy, cf.hz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        c.m[d][0] = 0.25 * h[d];
        c.m[d][1] = h[d] / 12.0;
        c.k[d] = 1.0 / h[d];
    }
    c.lam = cf.lam;
    c.mu = cf.mu;
    c.lam4 = 0.25 * cf.lam;
    c.mu4 = 0.25 * cf.mu;
    c.sgn_xy = -1.0;          // physical y runs against the node index
    c.sgn_xz = 1.0;
    c.sgn_yz = -1.0;
    return c;
}

// the constants of the 45 products, formed once per thread
struct ModalK {
    double d[3][8];           // diagonal, component c, mode bits x = 1, y = 2, z = 4
    double l_xy[2], u_xy[2];  // lambda and mu couplings of the axes (x, y) by the third axis' mode
    double l_xz[2], u_xz[2];
    double l_yz[2], u_yz[2];
};
__device__ __forceinline__ void modal_k(const Coef64& cf, double* out) {
    const Modal c = modal_coefs(cf);
    ModalK k;
#pragma unroll
    for (int comp = 0; comp < 3; ++comp)
#pragma unroll
        for (int md = 0; md < 8; ++md) {
            double v = 0.0;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                const int o1 = ax == 0 ? 1 : 0, o2 = ax == 2 ? 1 : 2;
                if (!((md >> ax) & 1)) continue;
                const double e = ax == comp ? c.lam + 2.0 * c.mu : c.mu;
                v += e * c.k[ax] * c.m[o1][(md >> o1) & 1] * c.m[o2][(md >> o2) & 1];
            }
            k.d[comp][md] = v;
        }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        k.l_xy[t] = c.sgn_xy * c.lam4 * c.m[2][t];
        k.u_xy[t] = c.sgn_xy * c.mu4 * c.m[2][t];
        k.l_xz[t] = c.sgn_xz * c.lam4 * c.m[1][t];
        k.u_xz[t] = c.sgn_xz * c.mu4 * c.m[1][t];
        k.l_yz[t] = c.sgn_yz * c.lam4 * c.m[0][t];
        k.u_yz[t] = c.sgn_yz * c.mu4 * c.m[0][t];
    }
    double* o = out;
    for (int comp = 0; comp < 3; ++comp)
        for (int md = 0; md < 8; ++md) *o++ = k.d[comp][md];
    for (int t = 0; t < 2; ++t) {
        *o++ = k.l_xy[t]; *o++ = k.u_xy[t];
        *o++ = k.l_xz[t]; *o++ = k.u_xz[t];
        *o++ = k.l_yz[t]; *o++ = k.u_yz[t];
    }
}
constexpr int NMODAL = 36;

template <int MODE>
__global__ void __launch_bounds__(NT, 2) k_modal64(Level64 L, const __grid_constant__ Coef64 cf, Args64 a, int zc, int tiles_y,
                                                   int tiles_x) {
    __shared__ double sh[32], mk[NMODAL];
    extern __shared__ double dyn[];
    const int tid = threadIdx.x;
    const Grid& g = L.g;
    pdl_begin();
    pdl_wait();
    const double ab = step_length<MODE>(a);
    const int bty = blockIdx.x % tiles_y, btx = blockIdx.x / tiles_y % tiles_x, btz = blockIdx.x / (tiles_y * tiles_x);
    const int y0 = bty * TY, x0 = btx * TX;
    const int zb = btz * zc, ze = min(zb + zc, g.nz + 1);
    double dot = 0.0;
    {
        bool any = false;
        for (int iz = zb; iz < ze; ++iz) any |= L.tile_occ[((int64_t)iz * tiles_x + btx) * tiles_y + bty] != 0;
        if (!any) {
            dot_finish<MODE>(0.0, a, sh);
            return;
        }
    }
    if (tid == 0) modal_k(cf, mk);
    const int64_t S = g.slots, n3 = 3 * S, sx = g.sx(), sz = g.sz();
    const Points p(g, y0, x0, tid, tid);
    const bool own = p.cy <= g.ny && p.cx <= g.nx;
    constexpr int R = chk::F64_TILE;
    double* const Zb = dyn;               // s (0..2) and e (3..5) along z of the three components
    double* const Eb = Zb + 6 * NP;       // per element: component, z mode, (y, x) corner
    auto field = [&](int iz, int64_t base, bool ok, double v[3], double s[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = s[c] = 0.0;
            if (ok) form_at<MODE>(a, base + iz * sz + c * S, n3, ab, v[c], s[c]);
        }
    };
    double vc[3], vp[3], hc[3], hp[3], sc[3], sp[3], unused[3];
    double carry[3] = {0.0, 0.0, 0.0};    // A v at plane l from layer l - 1
    const int l0 = max(zb - 1, 0);
    field(l0, p.cbase, p.cok, vc, sc);
    field(l0, p.hbase, p.hok, hc, unused);
#pragma unroll 1
    for (int l = l0; l < ze; ++l) {       // layer l, then node plane l
        double y[3] = {carry[0], carry[1], carry[2]};
        const int64_t n = p.cbase + l * sz;
        const uint32_t f = own && l >= zb ? chk::ld(L.nflag, n, S, chk::F64_FIELD) : 0u;
        double xx[3] = {0.0, 0.0, 0.0}, px[3] = {0.0, 0.0, 0.0};
        if (MODE == M64_CG_UPDATE_JACOBI && (f & NF_SOLID)) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xx[c] = chk::ld((const double*)a.x, n + c * S, n3, chk::F64_FIELD);
                if (!a.first) px[c] = chk::ld(a.pold, n + c * S, n3, chk::F64_FIELD);
            }
        }
        if (l < g.nz) {
            field(l + 1, p.cbase, p.cok, vp, sp);
            field(l + 1, p.hbase, p.hok, hp, unused);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                chk::st(Zb, c * NP + p.pc, 6 * NP, R, vp[c] + vc[c]);
                chk::st(Zb, (3 + c) * NP + p.pc, 6 * NP, R, vp[c] - vc[c]);
                if (tid < NHALO) {
                    chk::st(Zb, c * NP + p.ph, 6 * NP, R, hp[c] + hc[c]);
                    chk::st(Zb, (3 + c) * NP + p.ph, 6 * NP, R, hp[c] - hc[c]);
                }
            }
            __syncthreads();
            for (int e = tid; e < NE; e += NT) {
                const int ey = e % EY, ex = e / EY, gy = y0 - 1 + ey, gx = x0 - 1 + ex;
                double sc_e = 0.0;
                if (gy >= 0 && gx >= 0 && gy < g.ny && gx < g.nx) {
                    const int64_t es = g.slot(gy, gx, l);
                    if (chk::ld(L.emask, es, S, chk::F64_FIELD)) sc_e = L.kscale * chk::ld(L.escale, es, S, chk::F64_FIELD);
                }
                if (sc_e != 0.0) {
                    // modes u[c][mode], bits x = 1, y = 2, z = 4
                    double u[3][8];
                    const int pt = ey + ex * HY;
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int zm = 0; zm < 2; ++zm) {
                            auto zf = [&](int o) { return chk::ld((const double*)Zb, (3 * zm + c) * NP + pt + o, 6 * NP, R); };
                            const double a00 = zf(0), a10 = zf(1), a01 = zf(HY), a11 = zf(HY + 1);   // (y, x)
                            const double s0 = a10 + a00, e0 = a10 - a00, s1 = a11 + a01, e1 = a11 - a01;
                            u[c][4 * zm + 0] = s1 + s0;
                            u[c][4 * zm + 1] = s1 - s0;
                            u[c][4 * zm + 2] = e1 + e0;
                            u[c][4 * zm + 3] = e1 - e0;
                        }
                    const double* D = mk;
                    const double *c0 = mk + 24, *c1 = mk + 30;   // couplings by the third axis' mode: l_xy u_xy l_xz u_xz l_yz u_yz
                    double t[3][8];
                    t[0][1] = fma(c0[2], u[2][4], fma(c0[0], u[1][2], D[1] * u[0][1]));
                    t[0][2] = fma(c0[1], u[1][1], D[2] * u[0][2]);
                    t[0][4] = fma(c0[3], u[2][1], D[4] * u[0][4]);
                    t[0][3] = fma(c1[2], u[2][6], D[3] * u[0][3]);
                    t[0][5] = fma(c1[0], u[1][6], D[5] * u[0][5]);
                    t[0][6] = fma(c1[3], u[2][3], fma(c1[1], u[1][5], D[6] * u[0][6]));
                    t[0][7] = D[7] * u[0][7];
                    t[1][2] = fma(c0[4], u[2][4], fma(c0[0], u[0][1], D[8 + 2] * u[1][2]));
                    t[1][1] = fma(c0[1], u[0][2], D[8 + 1] * u[1][1]);
                    t[1][4] = fma(c0[5], u[2][2], D[8 + 4] * u[1][4]);
                    t[1][3] = fma(c1[4], u[2][5], D[8 + 3] * u[1][3]);
                    t[1][6] = fma(c1[0], u[0][5], D[8 + 6] * u[1][6]);
                    t[1][5] = fma(c1[5], u[2][3], fma(c1[1], u[0][6], D[8 + 5] * u[1][5]));
                    t[1][7] = D[8 + 7] * u[1][7];
                    t[2][4] = fma(c0[4], u[1][2], fma(c0[2], u[0][1], D[16 + 4] * u[2][4]));
                    t[2][1] = fma(c0[3], u[0][4], D[16 + 1] * u[2][1]);
                    t[2][2] = fma(c0[5], u[1][4], D[16 + 2] * u[2][2]);
                    t[2][5] = fma(c1[4], u[1][3], D[16 + 5] * u[2][5]);
                    t[2][6] = fma(c1[2], u[0][3], D[16 + 6] * u[2][6]);
                    t[2][3] = fma(c1[5], u[1][5], fma(c1[3], u[0][6], D[16 + 3] * u[2][3]));
                    t[2][7] = D[16 + 7] * u[2][7];
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int zm = 0; zm < 2; ++zm) {
                            // transposed transforms along x and y; mode 0 carries no force
                            const double m0 = zm ? sc_e * t[c][4] : 0.0, m1 = sc_e * t[c][4 * zm + 1],
                                         m2 = sc_e * t[c][4 * zm + 2], m3 = sc_e * t[c][4 * zm + 3];
                            const double s0 = m0 - m1, s1 = m0 + m1, e0 = m2 - m3, e1 = m2 + m3;   // x = 0, 1
                            constexpr int N = 24 * NE;
                            const int b = ((c * 2 + zm) * 4) * NE + e;
                            chk::st(Eb, b, N, R, s0 - e0);                // (y, x) = (0, 0)
                            chk::st(Eb, b + NE, N, R, s0 + e0);           // (1, 0)
                            chk::st(Eb, b + 2 * NE, N, R, s1 - e1);       // (0, 1)
                            chk::st(Eb, b + 3 * NE, N, R, s1 + e1);       // (1, 1)
                        }
                } else {
#pragma unroll
                    for (int k = 0; k < 24; ++k) chk::st(Eb, k * NE + e, 24 * NE, R, 0.0);
                }
            }
            __syncthreads();
            const int ly = tile_y(tid), lx = tile_x(tid);
            const int e00 = ly + lx * EY;      // the element with this node at its (1, 1) corner
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double fz[2];
#pragma unroll
                for (int zm = 0; zm < 2; ++zm) {
                    const int b = ((c * 2 + zm) * 4) * NE + e00;
                    auto E = [&](int i) { return chk::ld((const double*)Eb, b + i, 24 * NE, R); };
                    fz[zm] = (E(3 * NE) + E(2 * NE + 1)) + (E(NE + EY) + E(EY + 1));
                }
                y[c] += fz[0] - fz[1];
                carry[c] = fz[0] + fz[1];
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) carry[c] = vp[c] = hp[c] = sp[c] = 0.0;
        }
        if (f & NF_SOLID) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
                finish_dof<MODE>(a, n + c * S, n3, (f & (NF_FIX_X << c)) ? 0.0 : y[c], vc[c], sc[c], px[c], xx[c], ab, dot);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            vc[c] = vp[c];
            hc[c] = hp[c];
            sc[c] = sp[c];
        }
    }
    dot_finish<MODE>(dot, a, sh);
}

// z planes per CTA: about 12 waves of two resident CTAs per SM on large grids
// (169 x 147 x 256 solve with 12 / 8 / 6 / 4 planes, 8 of them by this rule: 84.3 /
// 84.0 / 85.6 / 87.6 ms), at least 2 where that gives every SM two CTAs (each
// chunk forms two planes beyond its own; 42 x 37 x 64 solve with 1 / 2 / 3 / 4 / 6
// planes on its finest level: 23.3 / 22.1 / 22.9 / 24.5 / 27.2 ms), else zmin: a
// plane per CTA for the factorised form (its coarse levels at 1 / 2 / 3 / 4 planes:
// 22.1 / 21.6 / 21.3 / 21.9 ms), 2 for the modal one, whose chunks compute a layer
// more (density gradient at 42 x 37 x 64 with 2 / 3 / 4 / 5 planes: 20.7 / 22.9 /
// 23.6 / 25.6 ms)
int pick_zc64(const Grid& g, const Ctx& c, int zmin) {
    const int64_t cols = (int64_t)((g.ny + 1 + TY - 1) / TY) * ((g.nx + 1 + TX - 1) / TX);
    const int64_t want = (int64_t)c.num_sms * 2 * 12;
    int64_t zc = (cols * (g.nz + 1) + want - 1) / want;
    if (zc < 2) zc = cols * ((g.nz + 1 + 1) / 2) >= 2 * (int64_t)c.num_sms ? 2 : zmin;
    return (int)std::min<int64_t>(zc, 32);
}

template <typename K>
void opt_in_smem(K kernel, size_t bytes, std::atomic<unsigned long long>& opted) {
    if (bytes <= 48 * 1024) return;
    int dev = 0;
    GMGS_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (opted.load() & bit) return;
    GMGS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    opted.fetch_or(bit);
}

}  // namespace

Coef64 make_coef64(double E, double nu, const double ele[3]) {
    double D[6][6];
    hooke(E, nu, D);
    const double a = D[0][0], lam = D[0][1], mu = D[3][3];
    const double x = ele[0], y = ele[1], z = ele[2];
    const double cx = y * z / (36.0 * x), cy = x * z / (36.0 * y), cz = x * y / (36.0 * z);
    Coef64 c;
    for (int k = 0; k < 3; ++k) {
        c.ax[k] = (k == 0 ? a : mu) * cx;
        c.ay[k] = (k == 1 ? a : mu) * cy;
        c.az[k] = (k == 2 ? a : mu) * cz;
    }
    c.gxy = (lam + mu) * z / 24.0;       // physical y runs against the node index: the sign of the
    c.gxz = -(lam + mu) * y / 24.0;      // (x, y) and (y, z) terms is the opposite of (x, z)'s
    c.gyz = (lam + mu) * x / 24.0;
    c.lam = lam;
    c.mu = mu;
    c.hx = x;
    c.hy = y;
    c.hz = z;
    return c;
}

// occupied tiles: one block per (y tile, x tile, z plane)
__global__ void k_tile_occ64(Grid g, const uint8_t* __restrict__ nflag, uint8_t* __restrict__ occ) {
    const int iy = blockIdx.x * TY + threadIdx.x % TY, ix = blockIdx.y * TX + threadIdx.x / TY, iz = blockIdx.z;
    const bool solid = iy <= g.ny && ix <= g.nx && (nflag[g.slot(iy, ix, iz)] & NF_SOLID);
    const int any = __syncthreads_or(solid);
    if (threadIdx.x == 0) occ[((int64_t)iz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = any ? 1 : 0;
}
size_t tile_occ64_bytes(const Grid& g) {
    return (size_t)((g.ny + 1 + TY - 1) / TY) * ((g.nx + 1 + TX - 1) / TX) * (g.nz + 1);
}
void launch_tile_occ64(Ctx& c, const Grid& g, const uint8_t* nflag, uint8_t* occ) {
    const dim3 grid((g.ny + 1 + TY - 1) / TY, (g.nx + 1 + TX - 1) / TX, g.nz + 1);
    k_tile_occ64<<<grid, NT, 0, c.stream>>>(g, nflag, occ);
    GMGS_LAUNCHED(c);
}

__global__ void k_mask_stencils(const double* __restrict__ ke0, MaskStencil* __restrict__ table) {
    MaskStencil& T = table[blockIdx.x];
    const int mask = blockIdx.x, k = threadIdx.x;          // one warp, lane = offset
    // the solid elements that hold both the node and its neighbour at offset k
    auto holds = [&](int e, int& cn, int& cm) {
        const int A = e & 1, B = (e >> 1) & 1, C = e >> 2;                  // node = element origin + (A, B, C)
        const int my = A + off_y(k), mx = B + off_x(k), mz = C + off_z(k);  // neighbour relative to the origin
        if (!((mask >> e) & 1) || my < 0 || my > 1 || mx < 0 || mx > 1 || mz < 0 || mz > 1) return false;
        cn = corner_of(A, B, C);
        cm = corner_of(my, mx, mz);
        return true;
    };
    int cn = 0, cm = 0;
    bool any = false;
    if (k < 27)
        for (int e = 0; e < 8; ++e) any = holds(e, cn, cm) || any;
    const unsigned reach = __ballot_sync(0xffffffffu, any);
    if (k == 0) T.n = __popc(reach);
    if (!any) return;
    const int t = __popc(reach & ((1u << k) - 1u));
    T.k[t] = k;
    for (int i = 0; i < 9; ++i) {
        double v = 0.0;
        for (int e = 0; e < 8; ++e)
            if (holds(e, cn, cm)) v += ke0[(3 * cn + i / 3) * 24 + 3 * cm + i % 3];
        T.S[t][i] = v;
    }
}
void launch_mask_stencils(Ctx& c, const double* ke0, MaskStencil* table) {
    k_mask_stencils<<<256, 32, 0, c.stream>>>(ke0, table);
    GMGS_LAUNCHED(c);
}

void set_fixed_coefs(Coef64& c) {
    const double g[12] = {c.ax[0], c.ax[1], c.ax[2], c.ay[0], c.ay[1], c.ay[2],
                          c.az[0], c.az[1], c.az[2], c.gxy, -c.gxz, c.gyz};
    uint2* f[12] = {&c.fax[0], &c.fax[1], &c.fax[2], &c.fay[0], &c.fay[1], &c.fay[2],
                    &c.faz[0], &c.faz[1], &c.faz[2], &c.fgxy, &c.fgxz, &c.fgyz};
    const double big = *std::max_element(g, g + 12), small = *std::min_element(g, g + 12);
    c.fixed = 0;
    if (!(small > 0) || !std::isfinite(big)) return;
    std::frexp(big, &c.cexp);                       // big < 2^cexp
    // below 2^-11 of the largest a coefficient's 53 bits would not fit the fraction
    if (small < std::ldexp(big, -11) || c.cexp < -100 || c.cexp > 100) return;
    for (int k = 0; k < 12; ++k) {
        const uint64_t C = (uint64_t)std::ldexp(g[k], 64 - c.cexp);
        *f[k] = make_uint2((uint32_t)C, (uint32_t)(C >> 32));
    }
    // the largest coefficient of the row with the smallest terms, against 2^cexp
    double row = std::min({c.gxy, -c.gxz, c.gyz});
    for (int k = 0; k < 3; ++k) row = std::min(row, std::max({c.ax[k], c.ay[k], c.az[k]}));
    c.fixed = FIXED_RANGE - (c.cexp - 1 - std::ilogb(row));
}

template <int MODE>
void launch_fine64(Ctx& c, const Level64& L, const Coef64& cf0, const Args64& a) {
    const int ty = (L.g.ny + 1 + TY - 1) / TY, tx = (L.g.nx + 1 + TX - 1) / TX;
    static std::atomic<unsigned long long> opted_m{0}, opted_f{0};
    if (L.escale) {
        opt_in_smem(k_modal64<MODE>, MODAL_SMEM, opted_m);
        const int zc = pick_zc64(L.g, c, 2);
        const int blocks = ty * tx * ((L.g.nz + 1 + zc - 1) / zc);
        launch_chain(c, k_modal64<MODE>, blocks, NT, MODAL_SMEM, L, cf0, a, zc, ty, tx);
        return;
    }
    Coef64 cf = cf0;
    for (int k = 0; k < 3; ++k) {
        cf.ax[k] *= L.kscale;
        cf.ay[k] *= L.kscale;
        cf.az[k] *= L.kscale;
    }
    cf.gxy *= L.kscale;
    cf.gxz *= L.kscale;
    cf.gyz *= L.kscale;
    set_fixed_coefs(cf);
    opt_in_smem(k_fine64<MODE>, fine64_smem<MODE>(), opted_f);
    constexpr int per_b = NT / BND_LANES, per_e = NT / ELEM_LANES;
    const int nb_bnd = (L.n_bnd + per_b - 1) / per_b, nb_list = nb_bnd + (L.n_perel + per_e - 1) / per_e;
    const int zc = pick_zc64(L.g, c, 1);
    // a level whose nodes are all on the lists has no tiles to walk
    const int tiles = L.n_bnd + (int64_t)L.n_perel < L.n_node ? ty * tx * ((L.g.nz + 1 + zc - 1) / zc) : 0;
    launch_chain(c, k_fine64<MODE>, nb_list + tiles, NT, fine64_smem<MODE>(), L, cf, a, zc, nb_bnd, nb_list, ty, tx);
}
template void launch_fine64<M64_PLAIN>(Ctx&, const Level64&, const Coef64&, const Args64&);
template void launch_fine64<M64_VCYCLE_DOWN>(Ctx&, const Level64&, const Coef64&, const Args64&);
template void launch_fine64<M64_CG_UPDATE_JACOBI>(Ctx&, const Level64&, const Coef64&, const Args64&);
template void launch_fine64<M64_CG_DIRECTION>(Ctx&, const Level64&, const Coef64&, const Args64&);


// ---------------------------------------------------------------------------
// up-sweep (Vcycle.m:27-32): one thread per (y, x) column of a 32 x 8 tile
// (a warp holds one x, so the parity of x is uniform in it),
// walking a chunk of z planes.  omega / diagonal is stored, so no division is
// left, and the trilinear sum (in FP64: coarse planes first, then x, then y, 3.5
// additions per DOF on average) is one of 64-bit integers (fixed96.cuh): FP64
// operations bound the kernel (7.5 per DOF with the dot product, 3 now) and one
// of them costs the issue slots of 75 integer ones.  At 6.4M nodes 414 -> 264 us;
// on small grids the shorter chain of 64-clock operations counts as well (solve
// 42 x 37 x 64 35.1 -> 25.5 ms together with k_restrict).
// ---------------------------------------------------------------------------
constexpr int UY = 32, UX = 8;
template <bool DOT>
__global__ void __launch_bounds__(UY * UX, 2) k_up64(Grid gf, Grid gc, const uint8_t* __restrict__ nflag, int zc,
                                                const double* __restrict__ w, const double* r, const double* rp, const double* xc, double* xf,
                                                int zero_fixed, DotOut64 dout) {
    __shared__ double sh[32];
    pdl_begin();
    pdl_wait();
    const int64_t Sf = gf.slots, Sc = gc.slots, csx = gc.sx(), csz = gc.sz(), fsz = gf.sz();
    const int iy = blockIdx.x * UY + threadIdx.x, ix = blockIdx.y * UX + threadIdx.y;
    const int zb = blockIdx.z * zc, ze = min(zb + zc, gf.nz + 1);
    double dot = 0.0;
    if (iy <= gf.ny && ix <= gf.nx) {
        const bool oy = iy & 1, ox = ix & 1;            // ox is uniform across a warp
        const double wyx = (oy ? 0.5 : 1.0) * (ox ? 0.5 : 1.0);
        const int kyx = (oy ? 1 : 0) + (ox ? 1 : 0), drop_y = oy ? 0 : SUM64_DROP;
        const int64_t fcol = gf.slot(iy, ix, 0), ccol = gc.slot(iy >> 1, ix >> 1, 0);
        constexpr int U = chk::UP_FINE, UC = chk::UP_COARSE;
        double qa[3][4], qb[3][4];
        int qa_z = -1;
        auto load_q = [&](int Z, double (&q)[3][4]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int64_t x = c * Sc + ccol + Z * csz;
                q[c][0] = chk::ld(xc, x, 3 * Sc, UC);
                q[c][1] = chk::ld(xc, x + 1, 3 * Sc, UC);
                q[c][2] = ox ? chk::ld(xc, x + csx, 3 * Sc, UC) : 0.0;
                q[c][3] = ox ? chk::ld(xc, x + csx + 1, 3 * Sc, UC) : 0.0;
            }
        };
        for (int iz = zb; iz < ze; ++iz) {
            const int64_t fs = fcol + iz * fsz;
            const uint32_t fl = chk::ld(nflag, fs, Sf, U);
            if (!(fl & NF_SOLID)) continue;
            double wv[3], rv[3], pv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                wv[c] = chk::ld(w, fs + c * Sf, 3 * Sf, U);
                rv[c] = chk::ld(r, fs + c * Sf, 3 * Sf, U);
                pv[c] = chk::ld(rp, fs + c * Sf, 3 * Sf, U);
            }
            const int Iz = iz >> 1;
            const bool oz = iz & 1;                     // uniform across the CTA
            if (qa_z != Iz) load_q(Iz, qa);
            if (oz) load_q(Iz + 1, qb);
            const double wt = wyx * (oz ? 0.5 : 1.0);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double e0 = qa[c][0], e1 = qa[c][1], e2 = qa[c][2], e3 = qa[c][3], t;
                int h = max(abs_hi(e0), oy ? abs_hi(e1) : 0);
                if (ox) h = max(h, max(abs_hi(e2), oy ? abs_hi(e3) : 0));
                if (oz) {
                    h = max(h, max(abs_hi(qb[c][0]), oy ? abs_hi(qb[c][1]) : 0));
                    if (ox) h = max(h, max(abs_hi(qb[c][2]), oy ? abs_hi(qb[c][3]) : 0));
                }
                const int E = h >> 20;
                if (sum64_holds(E)) {
                    long long n = sum64_term(e0, E, 0) + sum64_term(e1, E, drop_y);
                    if (ox) n += sum64_term(e2, E, 0) + sum64_term(e3, E, drop_y);
                    if (oz) {
                        n += sum64_term(qb[c][0], E, 0) + sum64_term(qb[c][1], E, drop_y);
                        if (ox) n += sum64_term(qb[c][2], E, 0) + sum64_term(qb[c][3], E, drop_y);
                    }
                    t = sum64_value(n, E, kyx + (oz ? 1 : 0));
                } else {                                // zeros, infinities, NaN, the ends of the range
                    if (oz) {
                        e0 += qb[c][0];
                        e1 += qb[c][1];
                        if (ox) { e2 += qb[c][2]; e3 += qb[c][3]; }
                    }
                    if (ox) { e0 += e2; e1 += e3; }
                    t = wt * (oy ? e0 + e1 : e0);
                }
                double out = fma(wv[c], rv[c] + pv[c], t);
                if (zero_fixed && (fl & (NF_FIX_X << c))) out = 0.0;
                chk::st(xf, fs + c * Sf, 3 * Sf, chk::UP_OUT, out);
                if (DOT) dot = fma(rv[c], out, dot);
            }
            qa_z = Iz;
            if (oz) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int k = 0; k < 4; ++k) qa[c][k] = qb[c][k];
                qa_z = Iz + 1;
            }
        }
    }
    if (DOT) grid_dot_finish(dot, DotOut{dout.partials, dout.ticket, dout.out}, sh);
}

void launch_up64(Ctx& c, const Grid& gf, const Grid& gc, const uint8_t* nflag, const double* w, const double* r,
                 const double* rp, const double* xc, double* xf, bool zero_fixed, const DotOut64* dot) {
    const int ty = (gf.ny + 1 + UY - 1) / UY, tx = (gf.nx + 1 + UX - 1) / UX;
    const int64_t want = (int64_t)c.num_sms * 2 * 12;
    const int zc = (int)std::min<int64_t>(32, std::max<int64_t>(2, ((int64_t)ty * tx * (gf.nz + 1) + want - 1) / want));
    const dim3 grid(ty, tx, (gf.nz + 1 + zc - 1) / zc);
    const dim3 blk(UY, UX, 1);
    launch_chain(c, dot ? k_up64<true> : k_up64<false>, grid, blk, 0, gf, gc, nflag, zc, w, r, rp, xc, xf,
                 zero_fixed ? 1 : 0, dot ? *dot : DotOut64{});
}

// upper bound over the z-chunk choices
int dot64_blocks(const Grid& g, int64_t n_list) {
    const int64_t a = (int64_t)((g.ny + 1 + TY - 1) / TY) * ((g.nx + 1 + TX - 1) / TX);
    const int64_t b = (int64_t)((g.ny + 1 + UY - 1) / UY) * ((g.nx + 1 + UX - 1) / UX);
    const int64_t tiles = std::max(a, b) * (g.nz + 1);
    return (int)(tiles + n_list / (NT / ELEM_LANES) + 2);
}

// x -= dx, dx = w (r - alpha q) as the fused update added it
__global__ void k_drop_last_dx64(int64_t n, double* __restrict__ x, const double* __restrict__ r, const double* __restrict__ q,
                                 const double* __restrict__ w, const double* __restrict__ scal, int cur) {
    const double alpha = scal[cur] / scal[2];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] -= fma(-alpha, q[i], r[i]) * w[i];
}
void launch_drop_last_dx64(Ctx& c, int64_t n, double* x, const double* r, const double* q, const double* w,
                           const double* scal, int cur) {
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)c.num_sms * 16);
    k_drop_last_dx64<<<blocks, 256, 0, c.stream>>>(n, x, r, q, w, scal, cur);
    GMGS_LAUNCHED(c);
}

__global__ void k_wdinv64(int64_t n, const double* __restrict__ d, double omega, double* __restrict__ w) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        w[i] = d[i] != 0.0 ? omega / d[i] : 0.0;
}
void launch_wdinv64(Ctx& c, int64_t n, const double* d, double omega, double* w) {
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)c.num_sms * 16);
    k_wdinv64<<<blocks, 256, 0, c.stream>>>(n, d, omega, w);
    GMGS_LAUNCHED(c);
}

}  // namespace gmgs
