// mg.hpp -- multilevel (coarse-space) correction for the SIPG block-Jacobi PCG.
//
// Preconditioner  z = B r + P V(P^T r):  B the block-Jacobi inverse, P the
// prolongation of continuous piecewise-linear functions on the mesh vertices
// into the DG space (exact: P1 is inside P_N), V one symmetric V(1,1) cycle
// on the Galerkin coarse operator A_1 = P^T S P (assembled in closed form: for
// continuous P1 functions the interior-face terms of SIPG vanish, leaving the
// P1 stiffness, the Nitsche terms of the fixed-value boundary faces and the
// Helmholtz mass term), weighted-Jacobi smoothing, coarser levels by greedy
// vertex aggregation with piecewise-constant transfer, the coarsest (at most
// 500 unknowns) solved by a dense inverse.  Everything is linear and symmetric, so plain PCG applies.
#pragma once

#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "dg_basis.hpp"
#include "ipdg.hpp"

namespace dgk {

constexpr int kMgMaxLevels = 10;

// A level as its cycle uses it.  The sweep down starts from x = D r (D =
// omega / diag A) and the sweep up ends with one Jacobi step, so with R the
// sum over aggregates and P = R^T its transpose the level's work is linear in
// r and in the coarse result:
//   r_c = B r,            B = R (I - A D)
//   x   = w + B^T x_c,    w = M r,  M = 2 D - D A D
// (B^T = (I - D A) P).  The sparse matrices B, B^T and M are formed once, so
// a level is one launch down (B r and M r) and one up.
struct MgLevel {
    int n = 0;
    const int *bptr = nullptr, *bcol = nullptr;  // B in CSR, nc rows
    const double* bval = nullptr;
    const int *tptr = nullptr, *tcol = nullptr;  // B^T in CSR, n rows
    const double* tval = nullptr;
    const int *mptr = nullptr, *mcol = nullptr;  // M in CSR, n rows
    const double* mval = nullptr;
    double* r = nullptr;  // work vectors of the cycle
    double* x = nullptr;
    double* w = nullptr;
};

struct MgLevels {
    int nl = 0;                    // lv[0] (P1 on the vertices) .. lv[nl-1], the level held as a dense matrix
    MgLevel lv[kMgMaxLevels];
    const double* V = nullptr;     // dense cycle operator of lv[nl-1] (row-major, symmetric)
    int K = 0, Np = 0;
    const int* etov = nullptr;     // [K][3] vertex ids
    const double* lam = nullptr;   // [Np][3] barycentric coordinates of the nodes (ring order)
    const int* vptr = nullptr;     // vertex -> incident element corners k*3+c (CSR)
    const int* vinc = nullptr;
};

// host-side levels
struct MgCsr {
    std::vector<int> ptr, col;
    std::vector<double> val;
};

struct MgBuild {
    struct Level {
        int n = 0;
        MgCsr A;
        std::vector<double> dinv;  // omega / diag A
        std::vector<int> agg;      // coarse index of each unknown (empty on the coarsest level)
        MgCsr B, Bt, M;            // B of the sparse levels only
    };
    std::vector<int> vptr, vinc;
    std::vector<double> lam;
    std::vector<Level> levels;  // levels[0]: P1 on the vertices
    int nd = 0;                 // levels[nd] is held as its dense cycle operator, those below go into it
};

// Builds the levels; "" on success.  etov: [K][3] vertex ids, geo: [K][4]
// metrics, conn: packed neighbours (negative: boundary slot), fc: the face
// coefficients as built (tau/2 and sJ per element face), btype: per
// boundary slot (0: fixed value, Nitsche terms; otherwise none), mass_coef:
// Helmholtz coefficient.
std::string mg_build(int K, int N, int Np, const int* etov, const double* geo, const int* conn,
                     const std::vector<double>& fc, const std::vector<int>& btype, double mass_coef,
                     const dgb::RefOps& ops, MgBuild& out);

// The dense cycle operator of levels[nd] from the levels nd .. coarsest
// (count of them, lv[0] = levels[nd]): B^T and M of each in CSR, for the coarsest
// its operator A in place of M.  work holds mg_dense_work doubles (sizes n[0..count-1]);
// the n[0]^2 result is at its start.  *status (0 before) becomes 1 where the
// coarsest operator is not positive definite.
struct MgDenseLevel {
    int n = 0;
    const int *tptr = nullptr, *tcol = nullptr;
    const double* tval = nullptr;
    const int *mptr = nullptr, *mcol = nullptr;
    const double* mval = nullptr;
};
size_t mg_dense_work(const int* n, int count);
cudaError_t launch_mg_dense(const MgDenseLevel* lv, int count, double* work, int* status, cudaStream_t s);

// z = zb + P V(P^T r) and r.z (mode: 1 init -> S->rz, 2 refresh -> S->rz, 3
// iteration -> pcg_finish); dz (mixed precision) is completed as an offset
// mirror.  zb_summed: S->rzb holds r.zb, so that r.z = rzb + (P^T r).V(P^T r)
// comes out of the cycle; otherwise r.z is summed over the rows.
cudaError_t launch_mg_correction(const MgLevels& m, const double* r, const double* zb, double* z, float* dz, int mode,
                                 bool zb_summed, PcgScalars* S, double* part, int grid, cudaStream_t s);

}  // namespace dgk
