// FP64 operator kernels of the default path (fine64.cu).
#pragma once

#include "gmgs_internal.cuh"

namespace gmgs {

// The assembled interior stencil of the uniform box element as sums of tensor
// products of the 1-D operators m = [1 4 1], k = [-1 2 -1], d = [-1 0 1]
// (mass h/6 m, stiffness k/h, derivative d/2 of linear elements), times the
// level's kscale:
//   y_c = ax[c] kx my mz u_c + ay[c] mx ky mz u_c + az[c] mx my kz u_c
//         + the mixed terms  gxy dx dy mz, gxz dx my dz, gyz mx dy dz
//           between the components of the two axes
struct Coef64 {
    double ax[3], ay[3], az[3];
    double gxy, gxz, gyz;
    // modal form of one element (fine64.cu): diagonal and coupling coefficients
    double lam, mu;             // Lame constants
    double hx, hy, hz;
    // the stencil's coefficients as fractions C / 2^64 of 2^cexp (Coef64's
    // signs: gxz is negative, the others positive); fixed: 0 if they are not exact,
    // else the binary orders below its largest value that a window may reach
    uint2 fax[3], fay[3], faz[3], fgxy, fgxz, fgyz;
    int cexp = 0, fixed = 0;
};
void set_fixed_coefs(Coef64& c);   // from ax .. gyz
Coef64 make_coef64(double E, double nu, const double ele[3]);
// The assembled stencil of one set of solid elements around a node, on the
// uniform element matrix: the offsets the elements reach and their 3 x 3 blocks
struct MaskStencil {
    int n;
    int k[27];
    double S[27][9];
};
void launch_mask_stencils(Ctx& c, const double* ke0, MaskStencil* table);   // for the 256 sets

// one level as the FP64 kernels see it
struct Level64 {
    Grid g;
    const uint8_t* emask;
    const uint8_t* nflag;
    const uint8_t* tile_occ;      // per (z plane, x tile, y tile): any solid node
    const int32_t* etype;
    const double* Ks;
    int64_t nK;
    const double* ke0;            // Ke0, row = output DOF
    double kscale;
    const double* escale;         // finest-level element scale or null
    const MaskStencil* mask_stencil;   // one per set of solid elements
    const int32_t* bnd;           // solid nodes with a void element around them and no stored matrix
    int n_bnd;
    const int32_t* perel;         // nodes touching an element with its own stored matrix
    int n_perel;
    int64_t n_node;
};

enum Mode64 {
    M64_PLAIN = 0,            // y = A v                              (AtX.m)
    M64_VCYCLE_DOWN = 1,      // v = w r, out = r - A v               (Vcycle.m:14, JacobiSmoother.m:5-9)
    M64_CG_UPDATE_JACOBI = 2, // previous CG update r_m = r - alpha q, x += alpha p, r_m.r_m; then the
                              // Jacobi step v = w r_m, x += v, r = r_m - A v      (CG_solver.m:31-35, 18-19)
    M64_CG_DIRECTION = 3      // v = z + beta p_old, p = v, q = A v, p.q           (CG_solver.m:23-31)
};

struct DotOut64 {
    double* partials = nullptr;   // one per block (dot64_blocks)
    unsigned int* ticket = nullptr;
    double* out = nullptr;
};

struct Args64 {
    const double* v = nullptr;     // M64_PLAIN input
    const double* r = nullptr;     // residual (read on the halo)
    const double* w = nullptr;     // omega / diagonal
    const double* q = nullptr;     // M64_CG_UPDATE_JACOBI: A p of the previous iteration
    const double* z = nullptr;     // M64_CG_DIRECTION
    const double* pold = nullptr;  // previous direction
    double* out = nullptr;         // y / r' / the updated residual / q (must not alias the inputs)
    double* pout = nullptr;        // new direction (must not alias pold)
    double* x = nullptr;           // solution (owned nodes, in place)
    const double* scal = nullptr;  // CG scalars: [0],[1] r.z by parity, [2] p.q
    int cur = 0, first = 0;
    DotOut64 dot;
};

template <int MODE>
void launch_fine64(Ctx& c, const Level64& L, const Coef64& cf, const Args64& a);
size_t tile_occ64_bytes(const Grid& g);
void launch_tile_occ64(Ctx& c, const Grid& g, const uint8_t* nflag, uint8_t* occ);
// upper bound of the blocks (dot partials) of launch_fine64 and launch_up64
int dot64_blocks(const Grid& g, int64_t n_list);

// z = w (r + r') + P x_c on solid nodes (Vcycle.m:27-32), optionally the fixed
// DOFs zeroed and the dot r . z accumulated
void launch_up64(Ctx& c, const Grid& gf, const Grid& gc, const uint8_t* nflag, const double* w, const double* r,
                 const double* rp, const double* xc, double* xf, bool zero_fixed, const DotOut64* dot);
// x -= the last Jacobi step w (r - alpha q)
void launch_drop_last_dx64(Ctx& c, int64_t n, double* x, const double* r, const double* q, const double* w,
                           const double* scal, int cur);
// w = omega / d, 0 where the diagonal is 0
void launch_wdinv64(Ctx& c, int64_t n, const double* d, double omega, double* w);

}  // namespace gmgs
