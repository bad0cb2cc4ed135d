// V-cycle preconditioner and the outer PCG (src/kernel/Vcycle.m:1-36,
// src/kernel/CG_solver.m:1-56, src/kernel/JacobiSmoother.m:1-10).
//
// The FP64 path runs every vector and operator in double precision on the
// kernels of fine64.cu.  The mixed path keeps x and r as double-float vectors
// and the coarsest solve in FP64 and runs everything else in FP32 on the
// kernels of fine.cu.  Both fuse the vector updates into the operator.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>

#include "setup.cuh"

namespace gmgs {

enum { SC_RZ0 = 0, SC_RZ1 = 1, SC_PQ = 2, SC_RR = 3, SC_BB = 5, SC_TC = 4, SC_N = 8 };   // SC_TC: the wait-error flag (an int), beside SC_RR: one copy fetches both

static void zalloc(Ctx& c, DevBuf& b, size_t bytes) {
    if (b.bytes < bytes) b = dalloc(bytes);
    GMGS_CUDA(cudaMemsetAsync(b.p, 0, bytes, c.stream));
}

// what the FP64 operator needs of a level beyond the hierarchy: the occupied
// tiles and the list of its boundary nodes (an FP64 handle builds them with
// its work buffers, a mixed one when an FP64 operator is first applied)
static void prepare_fp64_level(Model& M, int l) {
    Ctx& c = M.ctx;
    Level& lv = M.levels[l];
    if (!M.mask_stencil.p) {
        M.mask_stencil = dalloc(256 * sizeof(MaskStencil));
        launch_mask_stencils(c, M.ke0_dev.as<double>(), M.mask_stencil.as<MaskStencil>());
    }
    if (lv.n_bnd >= 0) return;
    if (lv.tile_occ64.bytes < tile_occ64_bytes(lv.g)) lv.tile_occ64 = dalloc(tile_occ64_bytes(lv.g));
    launch_tile_occ64(c, lv.g, lv.nflag.as<uint8_t>(), lv.tile_occ64.as<uint8_t>());
    if (l == 0 && lv.escale64.p) lv.n_bnd = 0;   // every node takes the scaled elements
    else build_boundary_list(M, l);
}

static Level64 level64(const Model& M, const Level& lv) {
    Level64 f;
    f.g = lv.g;
    f.emask = lv.emask.as<uint8_t>();
    f.nflag = lv.nflag.as<uint8_t>();
    f.tile_occ = lv.tile_occ64.as<uint8_t>();
    f.etype = lv.etype.as<int32_t>();
    f.Ks = lv.Ks64.as<double>();
    f.nK = lv.Ks64.p ? lv.nK : 0;
    f.ke0 = M.ke0_dev.as<double>();
    f.kscale = lv.kscale;
    f.escale = lv.escale64.as<double>();
    f.mask_stencil = M.mask_stencil.as<MaskStencil>();
    f.bnd = lv.bnd_nodes.as<int32_t>();
    f.n_bnd = (int)lv.n_bnd;
    f.perel = lv.perel_nodes.as<int32_t>();
    f.n_perel = (int)lv.n_perel;
    f.n_node = lv.n_node;
    return f;
}

void alloc_work(Model& M) {
    Ctx& c = M.ctx;
    ++M.gen;   // buffers and operators may move: captured graphs are stale
    const bool mixed = M.prm.precision == GMGS_MIXED;
    const size_t T = mixed ? sizeof(float) : sizeof(double);
    const int L = M.num_levels;
    for (int l = 0; l < L; ++l) {
        Level& lv = M.levels[l];
        const size_t n3 = 3 * (size_t)lv.g.slots;
        if (l > 0) zalloc(c, lv.vr, n3 * T);
        if (l > 0) zalloc(c, lv.vx, n3 * T);
        if (!mixed) prepare_fp64_level(M, l);
        if (l < L - 1) {
            zalloc(c, lv.vrp, n3 * T);
            if (!mixed) {
                if (lv.wdinv64.bytes < n3 * 8) lv.wdinv64 = dalloc(n3 * 8);
                launch_wdinv64(c, (int64_t)n3, lv.diag64.as<double>(), M.prm.omega, lv.wdinv64.as<double>());
            } else {
                if (lv.wdinv32.bytes < n3 * 4) lv.wdinv32 = dalloc(n3 * 4);
                launch_wdinv(c, (int64_t)n3, lv.diag64.as<double>(), M.prm.omega, lv.wdinv32.as<float>());
                if (lv.emask8.bytes < (size_t)lv.g.slots) lv.emask8 = dalloc(lv.g.slots);
                launch_emask8(c, lv.g, lv.emask.as<uint8_t>(), lv.emask8.as<uint8_t>());
                if (lv.tile_occ.bytes < tile_occ_bytes(lv.g)) lv.tile_occ = dalloc(tile_occ_bytes(lv.g));
                launch_tile_occ(c, lv.g, lv.nflag.as<uint8_t>(), lv.tile_occ.as<uint8_t>());
                if (lv.tc_occ.bytes < tc_tile_occ_bytes(lv.g)) lv.tc_occ = dalloc(tc_tile_occ_bytes(lv.g));
                launch_tc_tile_occ(c, lv.g, lv.nflag.as<uint8_t>(), lv.tc_occ.as<uint8_t>());
            }
        }
    }
    const size_t n3 = 3 * (size_t)M.levels[0].g.slots;
    zalloc(c, M.cg_r, n3 * 8);
    if (mixed) {
        zalloc(c, M.cg_x, n3 * 8);
        zalloc(c, M.cg_r32b, n3 * 4);
        zalloc(c, M.cg_pa, n3 * 4);
        zalloc(c, M.cg_pb, n3 * 4);
        zalloc(c, M.cg_q32, n3 * 4);
        zalloc(c, M.cg_z32, n3 * 4);
        zalloc(c, M.cg_r32, n3 * 4);
    } else {
        zalloc(c, M.cg_rb, n3 * 8);
        zalloc(c, M.cg_p, n3 * 8);
        zalloc(c, M.cg_p2, n3 * 8);
        zalloc(c, M.cg_q64, n3 * 8);
        zalloc(c, M.cg_z64, n3 * 8);
    }
    zalloc(c, M.scal, SC_N * sizeof(double));
    M.dot_blocks = M.ctx.num_sms * 4;
    const Level& l0 = M.levels[0];
    const int maxb = mixed ? std::max({M.dot_blocks, fine_grid_blocks(l0.g), up32_grid_blocks(l0.g)})
                           : std::max(M.dot_blocks, dot64_blocks(l0.g, l0.n_bnd + l0.n_perel));
    zalloc(c, M.dot_partials, (size_t)maxb * sizeof(double));
    zalloc(c, M.dot_ticket, sizeof(unsigned int));
    if (const size_t planes = mixed ? dot_split_planes(l0.g, c.num_sms) : 0) {
        if (M.dot_prod.bytes < planes * DOT_PLANE * sizeof(float)) M.dot_prod = dalloc(planes * DOT_PLANE * sizeof(float));
        zalloc(c, M.dot_chunk, planes * sizeof(unsigned int));
    }
    if (!M.scal_host) GMGS_CUDA(cudaMallocHost(&M.scal_host, SC_N * sizeof(double)));
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
}

static int* wait_error(Model& M) { return reinterpret_cast<int*>(M.scal.as<double>() + SC_TC); }

static DotScratch dots(Model& M) {
    return DotScratch{M.dot_partials.as<double>(), M.dot_ticket.as<unsigned int>(), M.dot_blocks};
}

// V-cycle down-sweeps on the tensor cores when the environment sets GMGS_TC=1
static bool tc_enabled() {
    const char* e = std::getenv("GMGS_TC");
    return e && e[0] == '1';
}

// A kernel whose bounded wait ran out (a tensor-core kernel waiting for its
// MMA, or the CG update waiting for its TMA-staged operands) sets the device
// flag; the solve reports it instead of returning a result computed without
// the data it waited for.
static void check_tc(Model& M) {
    int flag = 0;
    GMGS_CUDA(cudaMemcpyAsync(&flag, wait_error(M), sizeof(int), cudaMemcpyDeviceToHost, M.ctx.stream));
    GMGS_CUDA(cudaStreamSynchronize(M.ctx.stream));
    if (flag) {
        GMGS_CUDA(cudaMemsetAsync(wait_error(M), 0, sizeof(int), M.ctx.stream));
        throw Error(GMGS_ERR_CUDA, "a kernel's bounded wait for its tensor-core MMA or staged operands timed out");
    }
}

static DotOut64 dot_out64(Model& M, int slot) {
    DotOut64 d;
    d.partials = M.dot_partials.as<double>();
    d.ticket = M.dot_ticket.as<unsigned int>();
    d.out = M.scal.as<double>() + slot;
    return d;
}

// One V(1,1) cycle in FP64, Vcycle.m:1-36: down-sweep Jacobi with residual
// update and restriction, coarsest direct solve, up-sweep prolongation +
// Jacobi with the pre-smoothing residual, fixed DOFs of the finest level
// zeroed.  The finest up-sweep also accumulates r . z into scal[dot_slot].
static void vcycle64(Model& M, const double* r0, double* z, bool with_dot, int dot_slot) {
    Ctx& c = M.ctx;
    c.mark(PK_VCYCLE, false);
    const int L = M.num_levels;
    for (int l = 0; l < L - 1; ++l) {
        Level& lv = M.levels[l];
        Level& lc = M.levels[l + 1];
        Args64 a;
        a.r = l == 0 ? r0 : lv.vr.as<double>();
        a.w = lv.wdinv64.as<double>();
        a.out = lv.vrp.as<double>();
        if (l == 0) c.mark(PK_FINE_MATVEC, false);
        launch_fine64<M64_VCYCLE_DOWN>(c, level64(M, lv), M.coef64, a);
        if (l == 0) c.mark(PK_FINE_MATVEC, true, (double)lv.n_node * 3 * 24 + (double)lv.n_elem);
        if (l + 1 < L - 1) launch_restrict<double>(c, lv.g, lc.g, lc.nflag.as<uint8_t>(), lv.vrp.as<double>(), lc.vr.as<double>());
        else launch_restrict_free<double>(c, lv.g, lc.g, lc.nflag.as<uint8_t>(), lv.vrp.as<double>(), M.free_rank.as<int32_t>(),
                                         M.cvec_in.as<double>());
    }
    Level& lc = M.levels[L - 1];
    launch_coarse_solve(c, M.cb, M.cvec_in.as<double>(), M.cvec_out.as<double>(),
                        CoarseOut{M.free_idx.as<int32_t>(), nullptr, lc.vx.as<double>(), M.nfree});
    for (int l = L - 2; l >= 0; --l) {
        Level& lv = M.levels[l];
        const DotOut64 d = dot_out64(M, dot_slot);
        launch_up64(c, lv.g, M.levels[l + 1].g, lv.nflag.as<uint8_t>(), lv.wdinv64.as<double>(),
                    l == 0 ? r0 : lv.vr.as<double>(), lv.vrp.as<double>(), M.levels[l + 1].vx.as<double>(),
                    l == 0 ? z : lv.vx.as<double>(), l == 0, (l == 0 && with_dot) ? &d : nullptr);
    }
    c.mark(PK_VCYCLE, true);
}

static void vcycle32(Model& M, const float* r32, float* z, bool with_dot, int dot_slot);

// The operator handles work in the handle's own CG and V-cycle vectors, which
// are idle between solves and rewritten by the next one: three cudaMalloc /
// cudaFree pairs per call cost 0.2 to 0.4 ms (K x at 42 x 37 x 64: 264 us with
// them, of which the launches take about 60).
void vcycle_apply(Model& M, const double* r, double* z) {
    Ctx& c = M.ctx;
    const Level& l0 = M.levels[0];
    const int64_t nn = l0.n_node, S = l0.g.slots;
    const int32_t* ns = l0.node_slot.as<int32_t>();
    if (M.prm.precision == GMGS_MIXED) {
        M.use_tc = tc_enabled();
        launch_compact_to_dense<float>(c, nn, S, ns, r, M.cg_r32.as<float>());
        vcycle32(M, M.cg_r32.as<float>(), M.cg_z32.as<float>(), false, 0);
        launch_dense_to_compact<float>(c, nn, S, ns, M.cg_z32.as<float>(), z);
        check_tc(M);
    } else {
        launch_compact_to_dense<double>(c, nn, S, ns, r, M.cg_p.as<double>());
        vcycle64(M, M.cg_p.as<double>(), M.cg_z64.as<double>(), false, 0);
        launch_dense_to_compact<double>(c, nn, S, ns, M.cg_z64.as<double>(), z);
    }
}

void operator_apply(Model& M, int level, const double* x, double* y) {
    Ctx& c = M.ctx;
    prepare_fp64_level(M, level);
    const Level& lv = M.levels[level];
    const int64_t nn = lv.n_node, S = lv.g.slots;
    const int32_t* ns = lv.node_slot.as<int32_t>();
    Args64 a;
    double* v;
    if (M.prm.precision == GMGS_MIXED) {
        // the double-float CG state: 3 S doubles each, cleared by the next solve
        v = M.cg_x.as<double>();
        a.out = M.cg_r.as<double>();
        GMGS_CUDA(cudaMemsetAsync(v, 0, 3 * S * sizeof(double), c.stream));
    } else if (level == 0) {
        v = M.cg_p.as<double>();
        a.out = M.cg_q64.as<double>();
    } else {
        v = lv.vr.as<double>();
        a.out = lv.vx.as<double>();
    }
    launch_compact_to_dense<double>(c, nn, S, ns, x, v);
    a.v = v;
    launch_fine64<M64_PLAIN>(c, level64(M, lv), M.coef64, a);
    launch_dense_to_compact<double>(c, nn, S, ns, a.out, y);
}


// ---------------------------------------------------------------------------
// mixed path: FP32 V-cycle on the fused tiled kernels
// ---------------------------------------------------------------------------
static FineLevel fine_level(const Level& lv) {
    FineLevel f;
    f.g = lv.g;
    f.emask = lv.emask.as<uint8_t>();
    f.nflag = lv.nflag.as<uint8_t>();
    f.emask8 = lv.emask8.as<uint8_t>();
    f.etype = lv.etype.as<int32_t>();
    f.Ks = lv.Ks32.as<float>();
    f.nK = lv.Ks32.p ? lv.nK : 0;
    f.escale = lv.escale32.as<float>();
    f.kscale = (float)lv.kscale;
    f.tile_occ = lv.tile_occ.as<uint8_t>();
    return f;
}

template <int MODE>
static void launch_l0(Model& M, const FineLevel& f, const FineArgs& a) {
    launch_fine<MODE>(M.ctx, f, M.coef, a);
}

static DotOut dot_out(Model& M, int slot) {
    DotOut d;
    d.partials = M.dot_partials.as<double>();
    d.ticket = M.dot_ticket.as<unsigned int>();
    d.out = M.scal.as<double>() + slot;
    return d;
}

// z = V(r32); the level-1 up-sweep also accumulates r32 . z into scal[dot_slot]
static void vcycle32(Model& M, const float* r32, float* z, bool with_dot, int dot_slot) {
    Ctx& c = M.ctx;
    const int L = M.num_levels;
    c.mark(PK_VCYCLE, false);
    for (int l = 0; l < L - 1; ++l) {
        Level& lv = M.levels[l];
        Level& lc = M.levels[l + 1];
        FineArgs a;
        a.r32 = l == 0 ? r32 : lv.vr.as<float>();
        a.wdinv = lv.wdinv32.as<float>();
        a.out32 = lv.vrp.as<float>();
        // r, omega/diag, r' per node; element masks
        const double bytes = (double)lv.n_node * 3 * 12 + (double)lv.n_elem;
        if (l == 0) {
            c.mark(PK_FINE_MATVEC, false);
            c.mark(PK_VDOWN0, false);
        }
        if (l == 1) c.mark(PK_COARSE, false);
        const FineLevel fl = fine_level(lv);
        a.perel = lv.perel_nodes.as<int32_t>();
        a.n_perel = (int)lv.n_perel;
        if (M.use_tc && lv.n_perel < lv.n_node) {
            FineLevel ft = fl;
            ft.tile_occ = lv.tc_occ.as<uint8_t>();
            launch_tc_vdown(c, ft, M.tcoef, a.r32, a.wdinv, a.out32, wait_error(M));
            if (lv.n_perel > 0) launch_perel_vdown(c, fl, M.coef, a);
        } else if (lv.n_perel < lv.n_node) {
            launch_fine<FM_VCYCLE_DOWN>(c, fl, M.coef, a);
        } else {
            launch_perel_vdown(c, fl, M.coef, a);
        }
        if (l == 0) {
            c.mark(PK_FINE_MATVEC, true, bytes);
            c.mark(PK_VDOWN0, true, bytes);
        }
        if (l + 1 < L - 1) launch_restrict<float>(c, lv.g, lc.g, lc.nflag.as<uint8_t>(), lv.vrp.as<float>(), lc.vr.as<float>());
        else launch_restrict_free<float>(c, lv.g, lc.g, lc.nflag.as<uint8_t>(), lv.vrp.as<float>(), M.free_rank.as<int32_t>(),
                                         M.cvec_in.as<double>());
    }
    if (L == 2) c.mark(PK_COARSE, false);
    Level& lc = M.levels[L - 1];
    launch_coarse_solve(c, M.cb, M.cvec_in.as<double>(), M.cvec_out.as<double>(),
                        CoarseOut{M.free_idx.as<int32_t>(), lc.vx.as<float>(), nullptr, M.nfree});
    for (int l = L - 2; l >= 0; --l) {
        Level& lv = M.levels[l];
        const DotOut d = dot_out(M, dot_slot);
        if (l == 0) {
            c.mark(PK_COARSE, true);
            c.mark(PK_UP0, false);
        }
        launch_up32(c, lv.g, M.levels[l + 1].g, lv.nflag.as<uint8_t>(), lv.tile_occ.as<uint8_t>(),
                    lv.wdinv32.as<float>(),
                    l == 0 ? r32 : lv.vr.as<float>(), lv.vrp.as<float>(), M.levels[l + 1].vx.as<float>(),
                    l == 0 ? z : lv.vx.as<float>(), l == 0, (l == 0 && with_dot) ? &d : nullptr);
        if (l == 0) c.mark(PK_UP0, true, (double)lv.n_node * 3 * 20);
    }
    c.mark(PK_VCYCLE, true);
}

static bool graphs_enabled() {
    const char* e = std::getenv("GMGS_GRAPH");
    return e && e[0] && e[0] != '0';
}

void reset_graphs(Model& M) {
    for (auto& g : M.cg_graph) {
        if (g) cudaGraphExecDestroy(g);
        g = nullptr;
    }
    M.cg_graph_x = nullptr;
}

// Capture the iteration body for both parities (its = 2 and 3) without
// running it.  Returns false (nothing captured) when capture or
// instantiation fails; the caller restores its pointer state and launches
// eagerly.
template <class Body>
static bool capture_iteration_graphs(Model& M, Body& body) {
    Ctx& c = M.ctx;
    reset_graphs(M);
    for (int k = 0; k < 2; ++k) {
        const int its = 2 + k;
        cudaGraph_t g = nullptr;
        if (cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            reset_graphs(M);
            return false;
        }
        bool ok = true;
        const int64_t l0 = c.launches;
        try {
            body(its);
        } catch (const Error&) {
            ok = false;
        }
        M.cg_graph_kernels[its & 1] = c.launches - l0;   // recorded, not run
        c.launches = l0;
        const cudaError_t e = cudaStreamEndCapture(c.stream, &g);
        cudaGraphExec_t ex = nullptr;
        if (ok && e == cudaSuccess && g && cudaGraphInstantiate(&ex, g, 0) == cudaSuccess) M.cg_graph[its & 1] = ex;
        else ok = false;
        cudaGetLastError();
        if (g) cudaGraphDestroy(g);
        if (!ok) {
            reset_graphs(M);
            return false;
        }
    }
    return true;
}

static int pcg_mixed(Model& M, const double* b, double* x, int32_t* iters_out, double* relres_out, double* hist) {
    Ctx& c = M.ctx;
    M.use_tc = tc_enabled();
    Level& l0 = M.levels[0];
    const int64_t n3 = 3 * l0.g.slots;
    double* scal = M.scal.as<double>();
    const DotScratch ds = dots(M);
    // double-float state: x = x_hi + x_lo in the two halves of cg_x, r = r32 + r_lo
    // (the high part double-buffered, the low part in the first half of cg_r)
    float* x_hi = M.cg_x.as<float>();
    float* x_lo = x_hi + n3;
    float* r_lo = M.cg_r.as<float>();
    float* r32a = M.cg_r32.as<float>();
    float* r32b = M.cg_r32b.as<float>();
    float* pa = M.cg_pa.as<float>();
    float* pb = M.cg_pb.as<float>();
    float* q = M.cg_q32.as<float>();
    const FineLevel f0 = fine_level(l0);

    launch_dot<double, double>(c, ds, n3, b, b, scal + SC_BB);
    GMGS_CUDA(cudaMemcpyAsync(M.scal_host + SC_BB, scal + SC_BB, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    GMGS_CUDA(cudaMemsetAsync(x_hi, 0, 2 * n3 * sizeof(float), c.stream));
    launch_df_split(c, n3, b, r32a, r_lo);     // r = b - A*0
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    const double normB = std::sqrt(M.scal_host[SC_BB]);
    if (normB == 0.0) {
        GMGS_CUDA(cudaMemsetAsync(x, 0, n3 * sizeof(double), c.stream));
        GMGS_CUDA(cudaStreamSynchronize(c.stream));
        if (iters_out) *iters_out = 0;
        if (relres_out) *relres_out = 0;
        M.last_iters = 0;
        M.last_relres = 0;
        return GMGS_OK;
    }
    if (!std::isfinite(normB)) throw Error(GMGS_ERR_NONFINITE, "non-finite load vector");
    // algorithmic bytes per node: r (high part read + write, low part rw), q, p, wdinv, x (both parts rw)
    const double jbytes = (double)l0.n_node * 3 * (8 + 8 + 4 + 4 + 4 + 16) + 2.0 * (double)l0.n_node;
    const double pbytes = (double)l0.n_node * 3 * (4 + 4 + 4 + 4) + 2.0 * (double)l0.n_node;

    // Fused kernel: the previous iteration's update (x += alpha p, r -= alpha q,
    // |r|^2 for its convergence test) followed by the next iteration's Jacobi
    // step (x += dx, r -= A dx).  When the solve stops, the last dx (which
    // belongs to an iteration that does not run) is removed from x again.
    auto update_jacobi = [&](int first, int cur) {
        FineArgs a;
        a.r32 = r32a;
        a.r_lo = r_lo;
        a.q32 = q;
        a.pold = pa;
        a.wdinv = l0.wdinv32.as<float>();
        a.x_hi = x_hi;
        a.x_lo = x_lo;
        a.r32out = r32b;
        a.scal = scal;
        a.cur = cur;
        a.first = first;
        a.dot = dot_out(M, SC_RR);
        a.prod = M.dot_prod.as<float>();
        a.chunk = M.dot_chunk.as<unsigned int>();
        a.err = wait_error(M);
        c.mark(PK_FINE_MATVEC, false);
        c.mark(PK_UPDATE_JACOBI, false);
        launch_l0<FM_CG_UPDATE_JACOBI>(M, f0, a);
        c.mark(PK_FINE_MATVEC, true, jbytes);
        c.mark(PK_UPDATE_JACOBI, true, jbytes);
        std::swap(r32a, r32b);
    };

    // one PCG iteration: V-cycle, direction + A p, update + next Jacobi step;
    // the double buffers swap, so the launches repeat with period two
    auto body = [&](int its) {
        const int cur = its & 1;
        vcycle32(M, r32a, M.cg_z32.as<float>(), true, cur);     // z2 = PtV(r1), r1'z2   (CG_solver.m:21,26)
        {   // p2 = z2 + beta p1; q = A p2; p2'q   (CG_solver.m:23-31)
            FineArgs a;
            a.z32 = M.cg_z32.as<float>();
            a.pold = pa;
            a.pout = pb;
            a.scal = scal;
            a.cur = cur;
            a.first = its == 1;
            a.out32 = q;
            a.dot = dot_out(M, SC_PQ);
            a.prod = M.dot_prod.as<float>();
            a.chunk = M.dot_chunk.as<unsigned int>();
            c.mark(PK_FINE_MATVEC, false);
            c.mark(PK_DIRECTION, false);
            launch_l0<FM_CG_DIRECTION>(M, f0, a);
            c.mark(PK_FINE_MATVEC, true, pbytes);
            c.mark(PK_DIRECTION, true, pbytes);
            std::swap(pa, pb);
        }
        update_jacobi(0, cur);     // x += alpha p2; r2 = r1 - alpha q; |r2|; next Jacobi step
    };
    // With GMGS_GRAPH=1 the body is replayed from the second iteration on as
    // a CUDA graph (one per parity, captured once per model and solution
    // buffer): one launch per iteration instead of ~50.  Measured on the
    // 153M-DOF model it gives the same solve time as eager launches (the host
    // enqueues far ahead of the GPU and the in-iteration gaps are short) and
    // its capture + instantiation costs ~55 ms on the first solve, so eager
    // launches are the default.  Profiled runs always launch eagerly.
    const bool use_graph = !c.prof && graphs_enabled();
    bool graphs_ok = use_graph && M.cg_graph[0] && M.cg_graph[1] && M.cg_graph_x == x && M.cg_graph_gen == M.gen;

    const auto t0 = std::chrono::steady_clock::now();
    int its = 0, nhist = 0;
    double resnorm = INFINITY;
    int status = GMGS_ERR_MAX_ITERATIONS;
    update_jacobi(1, 0);          // [x, r1] = JacobiSmoother(var) of the first iteration (CG_solver.m:18-19)
    while (its <= M.prm.max_it) {
        c.mark(PK_CG_ITER, false);
        ++its;
        if (its >= 2 && use_graph && !graphs_ok) {
            float *sa = r32a, *sb = r32b, *qa = pa, *qb = pb;
            graphs_ok = capture_iteration_graphs(M, body);
            r32a = sa; r32b = sb; pa = qa; pb = qb;
            if (graphs_ok) {
                M.cg_graph_x = x;
                M.cg_graph_gen = M.gen;
            }
        }
        if (its >= 2 && graphs_ok) {
            GMGS_CUDA(cudaGraphLaunch(M.cg_graph[its & 1], c.stream));
            c.launches += M.cg_graph_kernels[its & 1];
            std::swap(pa, pb);     // the swaps the replayed body made
            std::swap(r32a, r32b);
        } else {
            body(its);
        }
        c.mark(PK_CG_ITER, true);
        static_assert(SC_TC == SC_RR + 1, "the residual and the flag in one copy");
        GMGS_CUDA(cudaMemcpyAsync(M.scal_host + SC_RR, scal + SC_RR, 2 * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
        GMGS_CUDA(cudaStreamSynchronize(c.stream));
        if (*reinterpret_cast<const int*>(M.scal_host + SC_TC)) break;   // check_tc reports it
        resnorm = std::sqrt(M.scal_host[SC_RR]) / normB;
        if (M.prm.verbose) std::printf(" It.: %4d Res.: %16.6e\n", its, resnorm);
        if (!std::isfinite(resnorm)) {
            status = GMGS_ERR_NONFINITE;
            break;
        }
        if (resnorm < M.prm.tol) {
            status = GMGS_OK;
            if (M.prm.verbose)
                std::printf("CG solver converged at iteration%5d to a solution with relative residual%16.6e\n", its,
                            resnorm);
            break;
        }
        if (hist) {
            const double t = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
            hist[3 * nhist + 0] = its;
            hist[3 * nhist + 1] = t;
            hist[3 * nhist + 2] = resnorm;
        }
        ++nhist;
    }
    // the last fused launch already applied the Jacobi step of an iteration
    // that does not run; its inputs (r32 it read, q, alpha) are still in place
    launch_drop_last_dx(c, n3, x, x_hi, x_lo, r32b, q, l0.wdinv32.as<float>(), scal, its & 1, 0);
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    check_tc(M);
    if (status == GMGS_ERR_MAX_ITERATIONS && M.prm.verbose) std::printf("Exceed the maximum iterate numbers\n");
    if (iters_out) *iters_out = its;
    if (relres_out) *relres_out = resnorm;
    M.last_iters = its;
    M.last_relres = resnorm;
    return status;
}

// CG_solver.m:1-56 with the Jacobi step before each preconditioner call.
static int pcg_fp64(Model& M, const double* b, double* x, int32_t* iters_out, double* relres_out, double* hist) {
    Ctx& c = M.ctx;
    Level& l0 = M.levels[0];
    const int64_t n3 = 3 * l0.g.slots;
    double* scal = M.scal.as<double>();
    const DotScratch ds = dots(M);
    const double* r = b;                      // r = b - A*0; then alternately in the two buffers
    double* rbuf[2] = {M.cg_r.as<double>(), M.cg_rb.as<double>()};
    int rnext = 0;
    double* pa = M.cg_p.as<double>();
    double* pb = M.cg_p2.as<double>();
    double* q = M.cg_q64.as<double>();
    double* z = M.cg_z64.as<double>();
    const double* w = l0.wdinv64.as<double>();
    const Level64 f0 = level64(M, l0);

    launch_dot<double, double>(c, ds, n3, b, b, scal + SC_BB);
    GMGS_CUDA(cudaMemcpyAsync(M.scal_host + SC_BB, scal + SC_BB, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    GMGS_CUDA(cudaMemsetAsync(x, 0, n3 * sizeof(double), c.stream));
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    const double normB = std::sqrt(M.scal_host[SC_BB]);
    if (normB == 0.0) {
        // zero load: the reference would divide 0/0; the solution is zero
        if (iters_out) *iters_out = 0;
        if (relres_out) *relres_out = 0;
        M.last_iters = 0;
        M.last_relres = 0;
        return GMGS_OK;
    }
    if (!std::isfinite(normB)) throw Error(GMGS_ERR_NONFINITE, "non-finite load vector");
    // algorithmic bytes per node: r read and written, x read and written, q, p, w; z, p read, p, q written
    const double jbytes = (double)l0.n_node * 3 * 8 * 7 + 2.0 * (double)l0.n_node;
    const double pbytes = (double)l0.n_node * 3 * 8 * 4 + 2.0 * (double)l0.n_node;
    const double* r_read = b;
    // the previous iteration's update and the next iteration's Jacobi step in
    // one pass, as in the mixed path
    auto update_jacobi = [&](int first, int cur) {
        Args64 a;
        a.r = r;
        a.w = w;
        a.q = q;
        a.pold = pa;
        a.x = x;
        a.out = rbuf[rnext];
        a.scal = scal;
        a.cur = cur;
        a.first = first;
        a.dot = dot_out64(M, SC_RR);
        c.mark(PK_FINE_MATVEC, false);
        c.mark(PK_UPDATE_JACOBI, false);
        launch_fine64<M64_CG_UPDATE_JACOBI>(c, f0, M.coef64, a);
        c.mark(PK_FINE_MATVEC, true, jbytes);
        c.mark(PK_UPDATE_JACOBI, true, jbytes);
        r_read = r;
        r = rbuf[rnext];
        rnext ^= 1;
    };

    const auto t0 = std::chrono::steady_clock::now();
    int its = 0, nhist = 0;
    double resnorm = INFINITY;
    int status = GMGS_ERR_MAX_ITERATIONS;
    update_jacobi(1, 0);          // [x, r1] = JacobiSmoother(var) of the first iteration (CG_solver.m:18-19)
    while (its <= M.prm.max_it) {
        c.mark(PK_CG_ITER, false);
        ++its;
        const int cur = its & 1;
        vcycle64(M, r, z, true, cur);      // z2 = PtV(r1), r1'z2   (CG_solver.m:21,26)
        {   // p2 = z2 + beta p1; q = A p2; p2'q   (CG_solver.m:23-31)
            Args64 a;
            a.z = z;
            a.pold = pa;
            a.pout = pb;
            a.out = q;
            a.scal = scal;
            a.cur = cur;
            a.first = its == 1;
            a.dot = dot_out64(M, SC_PQ);
            c.mark(PK_FINE_MATVEC, false);
            c.mark(PK_DIRECTION, false);
            launch_fine64<M64_CG_DIRECTION>(c, f0, M.coef64, a);
            c.mark(PK_FINE_MATVEC, true, pbytes);
            c.mark(PK_DIRECTION, true, pbytes);
            std::swap(pa, pb);
        }
        update_jacobi(0, cur);    // x += alpha p2; r2 = r1 - alpha q; |r2|; next Jacobi step
        c.mark(PK_CG_ITER, true);
        GMGS_CUDA(cudaMemcpyAsync(M.scal_host + SC_RR, scal + SC_RR, sizeof(double), cudaMemcpyDeviceToHost,
                                  c.stream));
        GMGS_CUDA(cudaStreamSynchronize(c.stream));
        resnorm = std::sqrt(M.scal_host[SC_RR]) / normB;
        if (M.prm.verbose) std::printf(" It.: %4d Res.: %16.6e\n", its, resnorm);
        if (!std::isfinite(resnorm)) {
            status = GMGS_ERR_NONFINITE;
            break;
        }
        if (resnorm < M.prm.tol) {
            status = GMGS_OK;
            if (M.prm.verbose)
                std::printf("CG solver converged at iteration%5d to a solution with relative residual%16.6e\n", its,
                            resnorm);
            break;
        }
        if (hist) {
            const double t = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
            hist[3 * nhist + 0] = its;
            hist[3 * nhist + 1] = t;
            hist[3 * nhist + 2] = resnorm;
        }
        ++nhist;
    }
    launch_drop_last_dx64(c, n3, x, r_read, q, w, scal, its & 1);
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    if (status == GMGS_ERR_MAX_ITERATIONS && M.prm.verbose) std::printf("Exceed the maximum iterate numbers\n");
    if (iters_out) *iters_out = its;
    if (relres_out) *relres_out = resnorm;
    M.last_iters = its;
    M.last_relres = resnorm;
    return status;
}

double load_work(Model& M) {
    Ctx& c = M.ctx;
    double* out = M.scal.as<double>() + SC_N - 1;
    launch_dot<double, double>(c, dots(M), 3 * M.levels[0].g.slots, M.F.as<double>(), M.U.as<double>(), out);
    double v = 0;
    GMGS_CUDA(cudaMemcpyAsync(&v, out, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    GMGS_CUDA(cudaStreamSynchronize(c.stream));
    return v;
}

int pcg_solve(Model& M, const double* b, double* x, int32_t* iters_out, double* relres_out, double* hist) {
    return M.prm.precision == GMGS_MIXED ? pcg_mixed(M, b, x, iters_out, relres_out, hist)
                                         : pcg_fp64(M, b, x, iters_out, relres_out, hist);
}

}  // namespace gmgs
