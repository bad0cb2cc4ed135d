// The state behind one gmgs_handle and the setup / solve entry points used by
// the C ABI (api.cu).
#pragma once

#include "fine.cuh"
#include "fine64.cuh"
#include "gmgs_internal.cuh"

namespace gmgs {

struct Model {
    gmgs_params prm{};
    int nely = 0, nelx = 0, nelz = 0;   // unpadded voxel grid
    int ny = 0, nx = 0, nz = 0;         // padded finest grid
    double ele[3] = {1, 1, 1};
    int num_levels = 0;
    bool has_density = false;
    bool density_built = false;   // levels and operators stand for a density field
    double penal = 3.0;
    std::vector<Level> levels;
    Ctx ctx;
    bool own_stream = false;
    double ke0_rows[KE];   // Ke0 with row = output DOF
    DevBuf ke0_dev;
    DevBuf galerkin_child; // 8 x 24x24: P_j^T Ke0 P_j per child position j
    DevBuf galerkin_grand; // 64 x 24x24: the same over two levels (mixed precision + density)
    bool lean_level1 = false; // level-2 (index 1) matrices kept in FP32 only (mixed precision + density)
    Coef64 coef64{};       // factorised FP64 stencil of this handle's material and voxel
    DevBuf mask_stencil;   // its 256 boundary stencils
    DevBuf rho;            // compact density (double), extension
    // boundary conditions and solution (finest level, FP64, 3 planes)
    DevBuf F, U;
    // coarsest level
    int nfree = 0;
    DevBuf free_idx, free_rank;           // free DOF -> slot and slot -> free DOF (-1: none)
    DevBuf cvec_in, cvec_out;             // coarse vectors (cb.nb * cb.B long)
    CoarseBlocks cb;
    // outer CG work vectors
    DevBuf cg_x, cg_r;                                         // mixed path: hi / lo parts; cg_r also FP64
    DevBuf cg_rb, cg_p, cg_p2, cg_q64, cg_z64;                 // FP64 path (r and p double-buffered)
    DevBuf cg_q32, cg_z32, cg_r32;                             // mixed path
    DevBuf cg_r32b, cg_pa, cg_pb;                              // mixed path double buffers
    Coef32 coef{};                                             // FP32 stencil + element matrix
    TcCoef tcoef{};                                            // Ke as the tensor cores' B operand
    bool use_tc = false;   // V-cycle down-sweeps on the tensor cores (environment GMGS_TC)
    DevBuf scal;           // device scalars (see solver.cu)
    DevBuf dot_partials, dot_ticket;
    DevBuf dot_prod, dot_chunk;   // split dot products of small grids (mixed path)
    // CUDA graphs of the mixed PCG iteration body (one per parity), valid for
    // the solution buffer and the work-buffer generation they were captured with
    cudaGraphExec_t cg_graph[2] = {nullptr, nullptr};
    int64_t cg_graph_kernels[2] = {0, 0};
    const double* cg_graph_x = nullptr;
    uint64_t cg_graph_gen = 0, gen = 0;
    double* scal_host = nullptr;   // pinned
    int dot_blocks = 0;
    bool bc_set = false, coarse_ready = false, solved = false, ops_ready = false;
    bool loads_solved = false;   // U belongs to the loads in F (set_bc replaces them)
    // diagnostics
    double t_create_ms = 0, t_bc_ms = 0, t_solve_ms = 0, t_stress_ms = 0;
    int last_iters = 0;
    double last_relres = 0;
    std::string err;
};

DevBuf dalloc(size_t bytes);
int64_t exclusive_scan(Ctx& c, int32_t* d, int64_t n);

void element_stiffness(double E, double nu, const double ele[3], double Ke[KE]);
// Isotropic Hooke coefficients (d11, d12, d44) and reciprocal element edges
// (1/dx, 1/dy, 1/dz) for the stress kernels.
void stress_coefficients(double E, double nu, const double ele[3], double c[6]);

// setup.cu
void build_levels(Model& M, const int32_t* occ_dev);
void build_operators(Model& M, bool values_only = false);
void build_boundary_list(Model& M, int l);
void apply_bc(Model& M, const int32_t* fixed, int64_t nfixed, const double* loads, int64_t nload);
// overlap: see factor_coarse
void build_coarse_bc(Model& M, const std::function<void()>& overlap = {});
void set_density_dev(Model& M, const double* rho_dev, double penal);

// solver.cu
void alloc_work(Model& M);
void reset_graphs(Model& M);   // destroy the captured PCG iteration graphs
int pcg_solve(Model& M, const double* b_dense, double* x_dense, int32_t* iters, double* relres, double* hist);
// on compact interleaved device vectors (in place allowed); level 0-based
void vcycle_apply(Model& M, const double* r, double* z);
void operator_apply(Model& M, int level, const double* x, double* y);

// post.cu
void stress_dev(Model& M, const double* U_dense, double* nodal_compact, float* per_voxel_compact);
double load_work(Model& M);   // F . U of the last solve
void grad_dev(Model& M, const double* U_dense, const double* lam_dense, double* dJdrho_compact);

}  // namespace gmgs
