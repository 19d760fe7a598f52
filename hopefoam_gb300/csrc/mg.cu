// mg.cu -- multilevel coarse-space correction of the SIPG PCG (see mg.hpp):
// host construction of the levels and the device V-cycle.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "euler_flux.cuh"
#include "mg.hpp"
#include "pcg_reduce.cuh"

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

// B^T = (I - D A) P, its transpose B, and M = 2 D - D A D of a level
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
    F.B = transpose(F.Bt, F.n, nc);
    F.M.ptr = F.A.ptr;
    F.M.col = F.A.col;
    F.M.val.resize(F.A.val.size());
    for (int i = 0; i < F.n; i++)
        for (int q = F.A.ptr[i]; q < F.A.ptr[i + 1]; q++) {
            const int j = F.A.col[q];
            F.M.val[q] = (i == j ? 2.0 * F.dinv[i] : 0.0) - F.dinv[i] * F.A.val[q] * F.dinv[j];
        }
}

// dense inverse of an SPD matrix in place (Gauss-Jordan without pivoting: the
// pivots are the Cholesky ones); false if not positive definite
bool spd_inverse(int n, std::vector<double>& A) {
    for (int k = 0; k < n; k++) {
        double* rk = &A[(size_t)k * n];
        const double d = rk[k];
        if (!(d > 0)) return false;
        const double inv = 1.0 / d;
        rk[k] = 1.0;
        for (int j = 0; j < n; j++) rk[j] *= inv;
        for (int i = 0; i < n; i++) {
            if (i == k) continue;
            double* ri = &A[(size_t)i * n];
            const double f = ri[k];
            if (f == 0.0) continue;
            ri[k] = 0.0;
            for (int j = 0; j < n; j++) ri[j] -= f * rk[j];
        }
    }
    for (int i = 0; i < n; i++)  // the preconditioner has to be symmetric
        for (int j = 0; j < i; j++) A[(size_t)i * n + j] = A[(size_t)j * n + i] = 0.5 * (A[(size_t)i * n + j] + A[(size_t)j * n + i]);
    return true;
}

// dense cycle operator of a level from the next one's: V = M + B^T Vc B
std::vector<double> dense_cycle(const MgBuild::Level& F, int nc, const std::vector<double>& Vc) {
    const int n = F.n;
    std::vector<double> T((size_t)nc * n, 0.0), V((size_t)n * n, 0.0);  // T = Vc B
    for (int c = 0; c < nc; c++) {
        double* t = &T[(size_t)c * n];
        const double* v = &Vc[(size_t)c * nc];
        for (int i = 0; i < n; i++) {
            double s = 0;
            for (int q = F.Bt.ptr[i]; q < F.Bt.ptr[i + 1]; q++) s += F.Bt.val[q] * v[F.Bt.col[q]];
            t[i] = s;
        }
    }
    for (int i = 0; i < n; i++) {
        double* v = &V[(size_t)i * n];
        for (int q = F.Bt.ptr[i]; q < F.Bt.ptr[i + 1]; q++) {
            const double f = F.Bt.val[q];
            const double* t = &T[(size_t)F.Bt.col[q] * n];
            for (int j = 0; j < n; j++) v[j] += f * t[j];
        }
        for (int q = F.M.ptr[i]; q < F.M.ptr[i + 1]; q++) v[F.M.col[q]] += F.M.val[q];
    }
    for (int i = 0; i < n; i++)
        for (int j = 0; j < i; j++) V[(size_t)i * n + j] = V[(size_t)j * n + i] = 0.5 * (V[(size_t)i * n + j] + V[(size_t)j * n + i]);
    return V;
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
    // coarsest: dense inverse; then the dense cycle operators of the levels above it
    out.nd = (int)out.levels.size() - 1;
    {
        const MgBuild::Level& C = out.levels.back();
        out.V.assign((size_t)C.n * C.n, 0.0);
        for (int i = 0; i < C.n; i++)
            for (int q = C.A.ptr[i]; q < C.A.ptr[i + 1]; q++) out.V[(size_t)i * C.n + C.A.col[q]] = C.A.val[q];
        if (!spd_inverse(C.n, out.V)) return "coarse operator is not positive definite";
    }
    while (out.nd > 0 && out.levels[out.nd - 1].n <= kDense) {
        out.V = dense_cycle(out.levels[out.nd - 1], out.levels[out.nd].n, out.V);
        out.nd--;
    }
    (void)N;
    return "";
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

// r1 = P^T r; eight lanes per vertex, one incident element corner each,
// summed in a fixed order
__global__ void __launch_bounds__(256) mg_restrict_dg_kernel(MgLevels m, const double* __restrict__ r,
                                                             double* __restrict__ r1, const int* __restrict__ done) {
    if (done && *done) return;
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
    if (done && *done) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, row = t / kUpLanes, l = t % kUpLanes;
    const double s = row_dot<kUpLanes>(a.tptr, a.tcol, a.tval, xc, row, row < a.n, l);
    if (row < a.n && l == 0) a.x[row] = a.w[row] + s;
}

// x = V r, one warp per row, r staged in shared memory
__global__ void __launch_bounds__(256) mg_dense_kernel(int n, const double* __restrict__ V, const double* __restrict__ r,
                                                       double* __restrict__ x, const int* __restrict__ done) {
    __shared__ double rs[kDense];
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

// z = zb + P x1; r.z; dz mirror; finish like the learned preconditioner's collect
__global__ void mg_collect_kernel(MgLevels m, const double* __restrict__ zb, const double* __restrict__ x1,
                                  const double* __restrict__ r, double* __restrict__ z, float* __restrict__ dz,
                                  int mode, PcgScalars* S, double* part) {
    __shared__ double c0s[256];
    if (mode == 3 && S->done) return;
    const int Np = m.Np, EB = 256 / Np;
    const int e = threadIdx.x / Np, q = threadIdx.x - e * Np;
    const int ngroups = (m.K + EB - 1) / EB;
    double rz = 0;
    for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const int k = grp * EB + e;
        const bool act = e < EB && k < m.K;
        double c = 0;
        if (act) {
            const size_t t = (size_t)k * Np + q;
            c = m.lam[q * 3 + 0] * x1[m.etov[3 * (size_t)k]] + m.lam[q * 3 + 1] * x1[m.etov[3 * (size_t)k + 1]] +
                m.lam[q * 3 + 2] * x1[m.etov[3 * (size_t)k + 2]];
            const double zv = zb[t] + c;
            z[t] = zv;
            rz += r[t] * zv;
            if (q == 0) c0s[e] = c;
        }
        if (dz) {
            // dz enters as the offset mirror of zb: z - z0 = (zb - zb0) + (c - c0)
            __syncthreads();
            if (act) {
                const size_t t = (size_t)k * Np + q;
                dz[t] = dz[t] + (float)(c - c0s[e]);
            }
            __syncthreads();
        }
    }
    double val[1] = {rz}, tot[1];
    if (grid_sum<1>(val, part, gridDim.x, &S->counter, tot) && threadIdx.x == 0) {
        if (mode == 3) pcg_finish(S, tot[0], 0.0, S->rr);
        else S->rz = tot[0];
    }
}

static unsigned nb256(int n) { return (unsigned)((n + 255) / 256); }

cudaError_t launch_mg_correction(const MgLevels& m, const double* r, const double* zb, double* z, float* dz,
                                 int mode, PcgScalars* S, double* part, int grid, cudaStream_t s) {
    const int L = m.nl;
    const int* done = mode == 3 ? &S->done : nullptr;  // a stopped iteration leaves every vector as it is
    mg_restrict_dg_kernel<<<nb256(8 * m.lv[0].n), 256, 0, s>>>(m, r, m.lv[0].r, done);
    for (int l = 0; l + 1 < L; l++) {
        const int nc = m.lv[l + 1].n, bblocks = (int)nb256(kDownLanes * nc);
        mg_down_kernel<<<bblocks + nb256(kMLanes * m.lv[l].n), 256, 0, s>>>(m.lv[l], nc, bblocks, m.lv[l].r, m.lv[l + 1].r,
                                                                            done);
    }
    const MgLevel& c = m.lv[L - 1];
    mg_dense_kernel<<<(c.n + 7) / 8, 256, 0, s>>>(c.n, m.V, c.r, c.x, done);
    for (int l = L - 2; l >= 0; l--) mg_up_kernel<<<nb256(kUpLanes * m.lv[l].n), 256, 0, s>>>(m.lv[l], m.lv[l + 1].x, done);
    const int EB = 256 / m.Np;
    const int ngroups = (m.K + EB - 1) / EB;
    mg_collect_kernel<<<std::min(ngroups, grid), 256, 0, s>>>(m, zb, m.lv[0].x, r, z, dz, mode, S, part);
    return cudaGetLastError();
}

}  // namespace dgk
