// mg.cu -- multilevel coarse-space correction of the SIPG PCG (see mg.hpp):
// host construction of the sparse levels, device construction of the dense cycle
// operator, and the device V-cycle.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "euler_flux.cuh"
#include "f64split.cuh"
#include "ipdg_rows.cuh"
#include "mg.hpp"
#include "pcg_reduce.cuh"
#include "pdl.cuh"

namespace dgk {

namespace {

constexpr double kOmega = 0.6;  // weighted-Jacobi factor of the smoother
constexpr int kCoarsest = 500;  // largest operator solved by its dense inverse
// Largest level whose whole cycle is held as one dense matrix.  A product with
// it costs its n^2 doubles from L2 (33 MB at 2000: 5 us) where the levels it
// stands for cost two launches each (4 us and up).
constexpr int kDense = 2000;

void jacobi_of(MgBuild::Level& L) {
    L.dinv.assign(L.n, 0.0);
    for (int i = 0; i < L.n; i++)
        for (int q = L.A.ptr[i]; q < L.A.ptr[i + 1]; q++)
            if (L.A.col[q] == i) L.dinv[i] = kOmega / L.A.val[q];
}

// greedy aggregation on the matrix graph: each unassigned unknown opens an
// aggregate with its unassigned neighbours
int aggregate(const MgBuild::Level& L, std::vector<int>& agg) {
    agg.assign(L.n, -1);
    int na = 0;
    for (int i = 0; i < L.n; i++) {
        if (agg[i] >= 0) continue;
        agg[i] = na;
        for (int q = L.A.ptr[i]; q < L.A.ptr[i + 1]; q++)
            if (agg[L.A.col[q]] < 0) agg[L.A.col[q]] = na;
        na++;
    }
    return na;
}

// rows built one after another from (column, value) contributions; columns
// sorted, values summed in the order they come
struct RowBuilder {
    std::vector<int> at, cols;  // at[c]: 1 + place of column c in this row
    std::vector<double> vals;
    explicit RowBuilder(int ncols) : at(ncols, 0) {}
    void add(int c, double v) {
        if (at[c] == 0) {
            cols.push_back(c);
            vals.push_back(v);
            at[c] = (int)cols.size();
        } else {
            vals[at[c] - 1] += v;
        }
    }
    void finish(MgCsr& m) {
        // insertion sort: rows are short
        for (size_t i = 1; i < cols.size(); i++)
            for (size_t j = i; j > 0 && cols[j - 1] > cols[j]; j--) {
                std::swap(cols[j - 1], cols[j]);
                std::swap(vals[j - 1], vals[j]);
            }
        for (size_t i = 0; i < cols.size(); i++) {
            at[cols[i]] = 0;
            m.col.push_back(cols[i]);
            m.val.push_back(vals[i]);
        }
        m.ptr.push_back((int)m.col.size());
        cols.clear();
        vals.clear();
    }
};

MgCsr transpose(const MgCsr& a, int rows, int cols) {
    MgCsr t;
    t.ptr.assign(cols + 1, 0);
    for (int c : a.col) t.ptr[c + 1]++;
    for (int c = 0; c < cols; c++) t.ptr[c + 1] += t.ptr[c];
    t.col.resize(a.col.size());
    t.val.resize(a.col.size());
    std::vector<int> fill(t.ptr.begin(), t.ptr.end() - 1);
    for (int i = 0; i < rows; i++)
        for (int q = a.ptr[i]; q < a.ptr[i + 1]; q++) {
            const int p = fill[a.col[q]]++;
            t.col[p] = i;
            t.val[p] = a.val[q];
        }
    return t;
}

// B^T = (I - D A) P and M = 2 D - D A D of a level
void cycle_matrices(MgBuild::Level& F, int nc) {
    F.Bt = MgCsr();
    F.Bt.ptr.reserve(F.n + 1);
    F.Bt.ptr.push_back(0);
    RowBuilder rb(nc);
    for (int i = 0; i < F.n; i++) {
        rb.add(F.agg[i], 1.0);
        for (int q = F.A.ptr[i]; q < F.A.ptr[i + 1]; q++) rb.add(F.agg[F.A.col[q]], -F.dinv[i] * F.A.val[q]);
        rb.finish(F.Bt);
    }
    F.M.ptr = F.A.ptr;
    F.M.col = F.A.col;
    F.M.val.resize(F.A.val.size());
    for (int i = 0; i < F.n; i++)
        for (int q = F.A.ptr[i]; q < F.A.ptr[i + 1]; q++) {
            const int j = F.A.col[q];
            F.M.val[q] = (i == j ? 2.0 * F.dinv[i] : 0.0) - F.dinv[i] * F.A.val[q] * F.dinv[j];
        }
}

}  // namespace

std::string mg_build(int K, int N, int Np, const int* etov, const double* geo, const int* conn,
                     const std::vector<double>& fc, const std::vector<int>& btype, double mass_coef,
                     const dgb::RefOps& ops, MgBuild& out) {
    out = MgBuild();
    int nv = 0;
    for (int q = 0; q < 3 * K; q++) nv = std::max(nv, etov[q] + 1);
    if (nv <= 0) return "no vertices";
    // barycentric coordinates of the nodes, ring order
    out.lam.resize((size_t)Np * 3);
    for (int p = 0; p < Np; p++) {
        const double r = ops.r[ops.ring[p]], s = ops.s[ops.ring[p]];
        out.lam[p * 3 + 0] = -(r + s) / 2;
        out.lam[p * 3 + 1] = (1 + r) / 2;
        out.lam[p * 3 + 2] = (1 + s) / 2;
    }
    // vertex -> element corners
    out.vptr.assign(nv + 1, 0);
    for (int q = 0; q < 3 * K; q++) out.vptr[etov[q] + 1]++;
    for (int v = 0; v < nv; v++) out.vptr[v + 1] += out.vptr[v];
    out.vinc.assign(3 * K, 0);
    {
        std::vector<int> fill(out.vptr.begin(), out.vptr.end() - 1);
        for (int q = 0; q < 3 * K; q++) out.vinc[fill[etov[q]]++] = q;
    }
    // level 0: P^T S P for continuous P1 functions, element matrices first
    std::vector<double> ea((size_t)9 * K);
    for (int k = 0; k < K; k++) {
        const double* g = geo + 4 * (size_t)k;
        const double rx = g[0], sx = g[1], ry = g[2], sy = g[3];
        const double J = 1.0 / (rx * sy - sx * ry);
        const double area = 2.0 * J;
        const double gx[3] = {-0.5 * (rx + sx), 0.5 * rx, 0.5 * sx};
        const double gy[3] = {-0.5 * (ry + sy), 0.5 * ry, 0.5 * sy};
        double a[3][3];
        for (int c = 0; c < 3; c++)
            for (int d = 0; d < 3; d++) {
                a[c][d] = area * (gx[c] * gx[d] + gy[c] * gy[d]);
                if (mass_coef != 0.0) a[c][d] += mass_coef * area / 12.0 * (c == d ? 2.0 : 1.0);
            }
        for (int f = 0; f < 3; f++) {
            const int cn = conn[(size_t)k * 3 + f];
            if (cn >= 0 || btype[-1 - cn] != 0) continue;
            // Nitsche terms of a fixed-value face: tau int u v - int (du/dn v + u dv/dn)
            const double* fk = &fc[((size_t)k * 3 + f) * kFaceCoef];
            const double tau = 2.0 * fk[4], len = 2.0 * fk[5];
            double nx, ny, fsc;
            face_normal(f, rx, sx, ry, sy, nx, ny, fsc);
            double dn[3], m1[3] = {0, 0, 0}, mf[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            for (int c = 0; c < 3; c++) dn[c] = nx * gx[c] + ny * gy[c];
            const int fa = f, fb = (f + 1) % 3;
            m1[fa] = m1[fb] = len / 2;
            mf[fa][fa] = mf[fb][fb] = len / 3;
            mf[fa][fb] = mf[fb][fa] = len / 6;
            for (int c = 0; c < 3; c++)
                for (int d = 0; d < 3; d++) a[c][d] += tau * mf[c][d] - (dn[c] * m1[d] + m1[c] * dn[d]);
        }
        for (int c = 0; c < 3; c++)
            for (int d = 0; d < 3; d++) ea[(size_t)9 * k + 3 * c + d] = a[c][d];
    }
    out.levels.emplace_back();
    {
        MgBuild::Level& L = out.levels.back();
        L.n = nv;
        L.A.ptr.reserve(nv + 1);
        L.A.ptr.push_back(0);
        L.A.col.reserve((size_t)8 * nv);
        L.A.val.reserve((size_t)8 * nv);
        RowBuilder rb(nv);
        for (int v = 0; v < nv; v++) {
            for (int q = out.vptr[v]; q < out.vptr[v + 1]; q++) {
                const int k = out.vinc[q] / 3, c = out.vinc[q] - 3 * k;
                for (int d = 0; d < 3; d++) rb.add(etov[3 * (size_t)k + d], ea[(size_t)9 * k + 3 * c + d]);
            }
            rb.finish(L.A);
        }
        jacobi_of(L);
    }
    // aggregation levels
    while (out.levels.back().n > kCoarsest) {
        if ((int)out.levels.size() >= kMgMaxLevels) return "too many levels";
        MgBuild::Level& F = out.levels.back();
        const int na = aggregate(F, F.agg);
        if (na > F.n * 9 / 10) return "aggregation does not coarsen";
        // Galerkin operator: rows of one aggregate after another
        std::vector<int> cptr(na + 1, 0), cmem(F.n);
        for (int i = 0; i < F.n; i++) cptr[F.agg[i] + 1]++;
        for (int a = 0; a < na; a++) cptr[a + 1] += cptr[a];
        {
            std::vector<int> fill(cptr.begin(), cptr.end() - 1);
            for (int i = 0; i < F.n; i++) cmem[fill[F.agg[i]]++] = i;
        }
        MgBuild::Level C;
        C.n = na;
        C.A.ptr.push_back(0);
        RowBuilder rb(na);
        for (int a = 0; a < na; a++) {
            for (int p = cptr[a]; p < cptr[a + 1]; p++)
                for (int q = F.A.ptr[cmem[p]]; q < F.A.ptr[cmem[p] + 1]; q++) rb.add(F.agg[F.A.col[q]], F.A.val[q]);
            rb.finish(C.A);
        }
        jacobi_of(C);
        cycle_matrices(F, na);
        out.levels.push_back(std::move(C));
    }
    out.nd = (int)out.levels.size() - 1;
    while (out.nd > 0 && out.levels[out.nd - 1].n <= kDense) out.nd--;
    for (int l = 0; l < out.nd; l++) out.levels[l].B = transpose(out.levels[l].Bt, out.levels[l].n, out.levels[l + 1].n);
    (void)N;
    return "";
}

// ---------------------------------------------------------------------------
// Dense cycle operator: the coarsest operator is inverted in place and carried
// up through the dense levels, V = M + B^T Vc B.  On one host core the
// inverse and the products were 5.6 ms of the 11.6 ms of a rebuild at 16,641
// vertices (289 and 1089 dense unknowns), and their result 9.5 MB of upload.  Now 0.4 ms;
// projection steps that rebuild the operator: K = 32768, N = 2 36.0 -> 29.5 ms.
//
// Inverse: Gauss-Jordan without pivoting on blocks of 16 rows (the pivots are
// the Cholesky ones of an SPD matrix).  A step is two launches: the panel kernel
// inverts the diagonal block in every block of the grid, multiplies the block
// row by it and sets the block column aside; the update kernel subtracts their
// product.  Bound by the serial chain of pivots (16 divisions a step); tiles of
// 16 x 32 keep the FP64 work of a step, n^2 16 multiplications, spread over the chip.
constexpr int kGj = 16;

__global__ void __launch_bounds__(256) mg_gj_panel_kernel(int n, int p0, const double* __restrict__ A, double* __restrict__ Rp,
                                                          double* __restrict__ Cp, int* status) {
    __shared__ double D[kGj][kGj + 1], inv;
    const int t = threadIdx.x, i = t / kGj, j = t % kGj, nb = min(kGj, n - p0);
    D[i][j] = i < nb && j < nb ? A[(size_t)(p0 + i) * n + p0 + j] : (i == j ? 1.0 : 0.0);
    for (int k = 0; k < nb; k++) {
        __syncthreads();
        if (t == 0) {
            const double d = D[k][k];
            if (!(d > 0) && blockIdx.x == 0) *status = 1;
            inv = 1.0 / d;
        }
        __syncthreads();
        const double f = D[i][k], r = D[k][j] * inv;
        const double w = i == k ? (j == k ? inv : r) : (j == k ? -f * inv : D[i][j] - f * r);
        __syncthreads();
        D[i][j] = w;
    }
    __syncthreads();
    // 64 columns of the block row, 64 rows of the block column
    const int c = blockIdx.x * 64 + t % 64;
    if (c < n) {
        const bool in = c >= p0 && c < p0 + nb;
        for (int r = t / 64; r < nb; r += 4) {
            double s = 0;
            for (int m = 0; m < nb; m++) s += D[r][m] * A[(size_t)(p0 + m) * n + c];
            Rp[(size_t)r * n + c] = in ? D[r][c - p0] : s;
        }
    }
    for (int q = t; q < 64 * kGj; q += 256) {
        const int r = blockIdx.x * 64 + q / kGj, m = q % kGj;
        if (r < n && m < nb) Cp[(size_t)r * kGj + m] = A[(size_t)r * n + p0 + m];
    }
}

__global__ void __launch_bounds__(128) mg_gj_update_kernel(int n, int p0, double* __restrict__ A, const double* __restrict__ Rp,
                                                           const double* __restrict__ Cp) {
    __shared__ double R[kGj][32], C[16][kGj];
    const int t = threadIdx.x, nb = min(kGj, n - p0), r0 = blockIdx.y * 16, c0 = blockIdx.x * 32;
    for (int q = t; q < kGj * 32; q += 128) {
        const int m = q / 32, c = c0 + q % 32;
        R[m][q % 32] = m < nb && c < n ? Rp[(size_t)m * n + c] : 0.0;
    }
    for (int q = t; q < 16 * kGj; q += 128) {
        const int r = r0 + q / kGj, m = q % kGj;
        C[q / kGj][m] = m < nb && r < n ? Cp[(size_t)r * kGj + m] : 0.0;
    }
    __syncthreads();
    const int c = c0 + t % 32;
    if (c >= n) return;
    for (int l = t / 32; l < 16; l += 4) {
        const int r = r0 + l;
        if (r >= n) return;
        double* a = A + (size_t)r * n + c;
        if (r >= p0 && r < p0 + nb) {
            *a = R[r - p0][t % 32];
            continue;
        }
        double s0 = 0, s1 = 0;
#pragma unroll
        for (int m = 0; m < kGj; m += 2) {
            s0 += C[l][m] * R[m][t % 32];
            s1 += C[l][m + 1] * R[m + 1][t % 32];
        }
        *a = (c >= p0 && c < p0 + nb ? 0.0 : *a) - (s0 + s1);
    }
}

// dense rows of a CSR matrix (one warp a row)
__global__ void __launch_bounds__(256) mg_scatter_kernel(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                                                         const double* __restrict__ val, double* __restrict__ A) {
    const int row = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (row >= n) return;
    for (int j = lane; j < n; j += 32) A[(size_t)row * n + j] = 0.0;
    __syncwarp();
    for (int q = ptr[row] + lane; q < ptr[row + 1]; q += 32) A[(size_t)row * n + col[q]] = val[q];
}

// T = Vc B, [nc][n]
__global__ void __launch_bounds__(256) mg_dense_t_kernel(MgDenseLevel F, int nc, const double* __restrict__ Vc,
                                                         double* __restrict__ T) {
    const int i = blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
    if (i >= F.n) return;
    double s = 0;
    for (int q = F.tptr[i]; q < F.tptr[i + 1]; q++) s += F.tval[q] * Vc[(size_t)c * nc + F.tcol[q]];
    T[(size_t)c * F.n + i] = s;
}

// V = M + B^T T, a block a row
__global__ void __launch_bounds__(256) mg_dense_v_kernel(MgDenseLevel F, const double* __restrict__ T, double* __restrict__ V) {
    const int i = blockIdx.x;
    double* v = V + (size_t)i * F.n;
    const int q0 = F.tptr[i], q1 = F.tptr[i + 1];
    for (int j = threadIdx.x; j < F.n; j += 256) {
        double s = 0;
        for (int q = q0; q < q1; q++) s += F.tval[q] * T[(size_t)F.tcol[q] * F.n + j];
        v[j] = s;
    }
    __syncthreads();
    for (int q = F.mptr[i] + threadIdx.x; q < F.mptr[i + 1]; q += 256) v[F.mcol[q]] += F.mval[q];
}

// the preconditioner has to be symmetric: both halves become their mean
__global__ void __launch_bounds__(256) mg_symmetrise_kernel(int n, double* __restrict__ A) {
    const int i = blockIdx.y, j = blockIdx.x * 256 + threadIdx.x;
    if (j >= i) return;
    const double a = 0.5 * (A[(size_t)i * n + j] + A[(size_t)j * n + i]);
    A[(size_t)i * n + j] = A[(size_t)j * n + i] = a;
}

size_t mg_dense_work(const int* n, int count) {
    size_t w = 2 * kGj * (size_t)n[count - 1];
    for (int l = count - 1; l >= 0; l--) w += (size_t)n[l] * n[l] + (l > 0 ? (size_t)n[l] * n[l - 1] : 0);
    return w;
}

// lv[0] is the top, lv[count - 1] the coarsest; the result is at the start of work
cudaError_t launch_mg_dense(const MgDenseLevel* lv, int count, double* work, int* status, cudaStream_t s) {
    double* X[kMgMaxLevels];
    for (int l = 0; l < count; l++) {
        X[l] = work;
        work += (size_t)lv[l].n * lv[l].n;
    }
    const MgDenseLevel& C = lv[count - 1];
    double *Rp = work, *Cp = Rp + (size_t)kGj * C.n, *T = Cp + (size_t)kGj * C.n;
    auto symmetrise = [&](int n, double* A) {
        mg_symmetrise_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)n), 256, 0, s>>>(n, A);
    };
    double* A = X[count - 1];
    mg_scatter_kernel<<<(C.n + 7) / 8, 256, 0, s>>>(C.n, C.mptr, C.mcol, C.mval, A);
    for (int p = 0; p < C.n; p += kGj) {
        mg_gj_panel_kernel<<<(C.n + 63) / 64, 256, 0, s>>>(C.n, p, A, Rp, Cp, status);
        mg_gj_update_kernel<<<dim3((unsigned)((C.n + 31) / 32), (unsigned)((C.n + 15) / 16)), 128, 0, s>>>(C.n, p, A, Rp, Cp);
    }
    symmetrise(C.n, A);
    for (int l = count - 2; l >= 0; l--) {
        const int n = lv[l].n, nc = lv[l + 1].n;
        mg_dense_t_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)nc), 256, 0, s>>>(lv[l], nc, X[l + 1], T);
        mg_dense_v_kernel<<<n, 256, 0, s>>>(lv[l], T, X[l]);
        symmetrise(n, X[l]);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// device cycle: the DG-to-P1 restriction, one launch per sparse level down,
// one dense product, one launch per level up, and the collect kernel.  Every
// launch is a few microseconds of dependent L2 reads on vectors that fit L2, so
// their number is what the cycle costs (three a level down and two up, before
// the level's matrices were multiplied out).  Measured per application, kernel
// times with cold caches: K = 32768 (16,641 vertices) 16 launches, 83 us ->
// 6 launches, 38 us; K = 101,246 (51,000 vertices) 61 us now.  One cluster of
// 16 blocks for the whole cycle took 41 and 111 us (too few SMs for the first
// level) and was left out.  Solves: K = 101,246, N = 4, mixed 38.8 -> 31.3 ms;
// building the levels 95 -> 30 ms there (rows merged in place instead of
// sorted triplets, a vectorised inverse, one upload).

// r1 = P^T r, and for the collect kernel whether this iteration still runs (S
// is null outside the iterations); eight lanes per vertex, one incident element corner each,
// summed in a fixed order
__global__ void __launch_bounds__(256) mg_restrict_dg_kernel(MgLevels m, const double* __restrict__ r,
                                                             double* __restrict__ r1, PcgScalars* S) {
    dependency_wait();
    if (S) {
        const int done = S->done;
        if (blockIdx.x == 0 && threadIdx.x == 0) S->skip = done;
        if (done) return;
    }
    __shared__ double lam[36 * 3];
    for (int i = threadIdx.x; i < 3 * m.Np; i += blockDim.x) lam[i] = m.lam[i];
    __syncthreads();
    const int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, l8 = threadIdx.x & 7;
    const bool ok = v < m.lv[0].n;
    double s = 0;
    if (ok) {
        const int q1 = m.vptr[v + 1];
        for (int q = m.vptr[v] + l8; q < q1; q += 8) {
            const int c = m.vinc[q], k = c / 3, lv = c - 3 * k;
            const double* rk = r + (size_t)k * m.Np;
#pragma unroll 6
            for (int i = 0; i < m.Np; i++) s += lam[i * 3 + lv] * rk[i];
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
    if (ok && l8 == 0) r1[v] = s;
}

// sum of a CSR row over LANES lanes (all of a warp's lanes call it); valid in lane 0 of the row's group
template <int LANES>
__device__ __forceinline__ double row_dot(const int* __restrict__ ptr, const int* __restrict__ col,
                                          const double* __restrict__ val, const double* __restrict__ x, int row, bool ok,
                                          int l) {
    double s = 0;
    if (ok) {
        const int q1 = ptr[row + 1];
        for (int q = ptr[row] + l; q < q1; q += LANES) s += val[q] * x[col[q]];
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
    return s;
}

constexpr int kDownLanes = 16, kMLanes = 4, kUpLanes = 4;  // lanes per row: about a third of its entries each

// r_c = B r (blocks [0, bblocks)) and w = M r (the others)
__global__ void __launch_bounds__(256) mg_down_kernel(MgLevel a, int nc, int bblocks, const double* __restrict__ r,
                                                      double* __restrict__ rc, const int* __restrict__ done) {
    dependency_wait();
    if (done && *done) return;
    if ((int)blockIdx.x < bblocks) {
        const int t = blockIdx.x * blockDim.x + threadIdx.x, row = t / kDownLanes, l = t % kDownLanes;
        const double s = row_dot<kDownLanes>(a.bptr, a.bcol, a.bval, r, row, row < nc, l);
        if (row < nc && l == 0) rc[row] = s;
    } else {
        const int t = (blockIdx.x - bblocks) * blockDim.x + threadIdx.x, row = t / kMLanes, l = t % kMLanes;
        const double s = row_dot<kMLanes>(a.mptr, a.mcol, a.mval, r, row, row < a.n, l);
        if (row < a.n && l == 0) a.w[row] = s;
    }
}

// x = w + B^T x_c
__global__ void __launch_bounds__(256) mg_up_kernel(MgLevel a, const double* __restrict__ xc, const int* __restrict__ done) {
    dependency_wait();
    if (done && *done) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, row = t / kUpLanes, l = t % kUpLanes;
    const double s = row_dot<kUpLanes>(a.tptr, a.tcol, a.tval, xc, row, row < a.n, l);
    if (row < a.n && l == 0) a.x[row] = a.w[row] + s;
}

// x = V r, one warp per row, r staged in shared memory
__global__ void __launch_bounds__(256) mg_dense_kernel(int n, const double* __restrict__ V, const double* __restrict__ r,
                                                       double* __restrict__ x, const int* __restrict__ done) {
    __shared__ double rs[kDense];
    dependency_wait();
    if (done && *done) return;
    for (int j = threadIdx.x; j < n; j += blockDim.x) rs[j] = r[j];
    __syncthreads();
    const int row = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (row >= n) return;
    const double* v = V + (size_t)row * n;
    double s0 = 0, s1 = 0;
    int j = lane;
#pragma unroll 4
    for (; j + 32 < n; j += 64) {
        s0 += v[j] * rs[j];
        s1 += v[j + 32] * rs[j + 32];
    }
    if (j < n) s0 += v[j] * rs[j];
    s0 += s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    if (lane == 0) x[row] = s0;
}

// z = zb + P x1, and dz from the mirror of zb to that of z: z - z0 = (zb - zb0) +
// (c - c0).  Bound by the FP64 pipe: three operations for c, one each for z and
// c - c0, which is rounded to FP32 by integer operations.  What the correction adds
// to r.z is r1.x1 with r1 = P^T r and x1 the cycle's result: the first kDotBlocks
// blocks sum it over the vertices beside the others and finish the iteration, or
// leave rz, from S->rzb = r.zb.  DOT (the learned forms, whose r.zb nobody has
// summed): r.z over all rows instead, finishing like the learned preconditioner's
// collect.  K = 101,246, N = 4: 34 us with the sum over all rows, 22 us with
// the vertices' sum in the kernel before (and 8 us there), 22 us with it here.
constexpr int kDotBlocks = 64;

template <int NP, bool DOT>
__global__ void __launch_bounds__(RowDims<NP>::THREADS) mg_collect_kernel(MgLevels m, const double* __restrict__ zb,
                                                                          const double* __restrict__ x1,
                                                                          const double* __restrict__ r, double* __restrict__ z,
                                                                          float* __restrict__ dz, int mode, PcgScalars* S,
                                                                          double* part) {
    using R = RowDims<NP>;
    dependency_wait();
    if (mode == 3 && S->skip) return;  // not S->done: this launch's own blocks may set that while others start
    int e, i;
    row_of<NP>(e, i);
    const bool lane_ok = e < R::EB;
    if (!DOT && blockIdx.x < kDotBlocks) {
        const MgLevel& a = m.lv[0];
        double dot = 0;
        for (int v = blockIdx.x * R::THREADS + threadIdx.x; v < a.n; v += kDotBlocks * R::THREADS) dot += a.x[v] * a.r[v];
        double val[1] = {dot}, tot[1];
        if (grid_sum<1>(val, part, kDotBlocks, &S->counter, tot) && threadIdx.x == 0) {
            const double rz = S->rzb + tot[0];
            if (mode == 3) pcg_finish(S, rz, 0.0, S->rr);
            else S->rz = rz;
        }
        return;
    }
    const int blk = blockIdx.x - (DOT ? 0 : kDotBlocks), nblk = gridDim.x - (DOT ? 0 : kDotBlocks);
    const double l0 = m.lam[3 * i], l1 = m.lam[3 * i + 1], l2 = m.lam[3 * i + 2];
    __shared__ double c0s[R::WA ? 1 : R::EB];
    double rz = 0;
    for (int grp = blk; grp < row_groups<NP>(m.K); grp += nblk) {
        const int k = grp * R::EB + e;
        const bool act = lane_ok && k < m.K;
        const size_t t = (size_t)k * NP + i;
        double c = 0, zv = 0;
        float d = 0.f;
        if (act) {
            const int* ev = m.etov + 3 * (size_t)k;
            zv = zb[t];
            if (dz) d = dz[t];
            c = l0 * x1[ev[0]] + l1 * x1[ev[1]] + l2 * x1[ev[2]];
            zv += c;
            z[t] = zv;
            if (DOT) rz += r[t] * zv;
        }
        if (dz) {
            double c0;
            if constexpr (R::WA) {
                c0 = __shfl_sync(0xffffffffu, c, (threadIdx.x & 31) - i);
            } else {
                __syncthreads();
                if (act && i == 0) c0s[e] = c;
                __syncthreads();
                c0 = act ? c0s[e] : 0.0;
            }
            if (act) dz[t] = d + f64s::minus_f32(c - c0, 0.f);
        }
    }
    if (DOT) {
        double val[1] = {rz}, tot[1];
        if (grid_sum<1>(val, part, gridDim.x, &S->counter, tot) && threadIdx.x == 0) {
            if (mode == 3) pcg_finish(S, tot[0], 0.0, S->rr);
            else S->rz = tot[0];
        }
    }
}

template <int NP>
static cudaError_t launch_collect(const MgLevels& m, const double* zb, const double* r, double* z, float* dz, int mode,
                                  bool zb_summed, PcgScalars* S, double* part, int grid, cudaStream_t s) {
    const int groups = row_groups<NP>(m.K);
    if (zb_summed)
        return launch_dependent(mg_collect_kernel<NP, false>, groups + kDotBlocks, RowDims<NP>::THREADS, s, m, zb, m.lv[0].x, r, z, dz, mode,
                                S, part);
    return launch_dependent(mg_collect_kernel<NP, true>, std::min(groups, grid), RowDims<NP>::THREADS, s, m, zb, m.lv[0].x, r,
                            z, dz, mode, S, part);
}

static unsigned nb256(int n) { return (unsigned)((n + 255) / 256); }

cudaError_t launch_mg_correction(const MgLevels& m, const double* r, const double* zb, double* z, float* dz, int mode,
                                 bool zb_summed, PcgScalars* S, double* part, int grid, cudaStream_t s) {
    const int L = m.nl;
    const int* done = mode == 3 ? &S->done : nullptr;  // a stopped iteration leaves every vector as it is
    cudaError_t e = launch_dependent(mg_restrict_dg_kernel, nb256(8 * m.lv[0].n), 256, s, m, r, m.lv[0].r, mode == 3 ? S : nullptr);
    for (int l = 0; l + 1 < L && e == cudaSuccess; l++) {
        const int nc = m.lv[l + 1].n, bblocks = (int)nb256(kDownLanes * nc);
        e = launch_dependent(mg_down_kernel, bblocks + nb256(kMLanes * m.lv[l].n), 256, s, m.lv[l], nc, bblocks, m.lv[l].r,
                             m.lv[l + 1].r, done);
    }
    const MgLevel& c = m.lv[L - 1];
    if (e == cudaSuccess) e = launch_dependent(mg_dense_kernel, (c.n + 7) / 8, 256, s, c.n, m.V, c.r, c.x, done);
    for (int l = L - 2; l >= 0 && e == cudaSuccess; l--)
        e = launch_dependent(mg_up_kernel, nb256(kUpLanes * m.lv[l].n), 256, s, m.lv[l], m.lv[l + 1].x, done);
    if (e != cudaSuccess) return e;
    switch (m.Np) {
        case 3: return launch_collect<3>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        case 6: return launch_collect<6>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        case 10: return launch_collect<10>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        case 15: return launch_collect<15>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        case 21: return launch_collect<21>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        case 28: return launch_collect<28>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        case 36: return launch_collect<36>(m, zb, r, z, dz, mode, zb_summed, S, part, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace dgk
