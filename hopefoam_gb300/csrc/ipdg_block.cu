// ipdg_block.cu -- the SIPG operator as assembled block rows, for the FP64
// iterations of the PCG (sm_103a).
//
// Element k's row of S couples it to itself and to its three face
// neighbours, four dense Np x Np blocks.  Matrix-free, the FP64 apply spends
// most of its operations on traces and normal derivatives of both sides of
// every face and is bound by the FP64 pipe (two operations per clock per SM).
// With the blocks formed once per operator a row is 4 Np + 12 FP64 operations
// and 32 Np bytes.  Per apply: K = 101,246, N = 4 665 -> about 230 us (FP64
// pipe 173, memory 107); K = 32,768, N = 2 76 -> 26 us; K = 1,152, N = 3
// 19.6 -> 12.9 us.  The element matrices are formed by one CTA per element
// from its traces and derivatives in shared memory; the diagonal blocks of the
// block-Jacobi preconditioner come from the same kernel.
//
// As in the matrix-free apply the input enters as offsets from each
// element's first-node value (d = u - u_0), so that constants, which the
// gradients annihilate, do not cost digits.  With w_f = O_f 1 the row sums of a
// neighbour block and wb those of the boundary and mass terms, D 1 = wb - sum
// w_f and
//   (S u)_k = D d + sum_f [ O_f d_f + w_f (u_f0 - u_0) ] + wb u_0.
//
// Blocks (the formulas of ipdg.cu with basis functions for u): with T the
// trace and dm the own normal derivative of the basis at a face's Gauss
// points, up, dp the neighbour's at the same points with this element's normal,
//   D   = J (c_rr Srr + c_rs Srs2 + c_ss Sss) + mass
//         + sum wJ [ T (a tau/2 T - a/2 dm)^T - a/2 dm T^T ],  a = 1 inside, 2 on a Dirichlet face
//   O_f = sum wJ [ -T (tau/2 up + dp/2)^T + dm up^T / 2 ].
#include <algorithm>

#include "dg_internal.hpp"
#include "ipdg.hpp"
#include "ipdg_rows.cuh"
#include "pcg_reduce.cuh"
#include "pdl.cuh"

namespace dgk {

namespace {

// sblocks: per group of elements (ipdg_rows.cuh) 4 Np columns (own block, then
// the neighbours') and four more of w_0, w_1, w_2, wb, each EB Np doubles
template <int NP>
constexpr int kRowCols = 4 * NP + 4;

// blocks of one element, one CTA; D row-major to `diag` (when set), everything
// to the grouped storage `sb` (when set)
template <int N, typename T>
__global__ void __launch_bounds__(128) ipdg_blocks_kernel(IpdgArgs a, double* __restrict__ diag, T* __restrict__ sb) {
    constexpr int Np = Dims<N>::Np, Nfp = Dims<N>::Nfp, Nfq = Dims<N>::Nfq, NF = 3 * Nfq, NB = 3 * N;
    using R = RowDims<Np>;
    const IpdgOps<double>& o = a.o64;
    __shared__ double tr[NF][Np];  // trace of the basis (zero off the face)
    __shared__ double dm[NF][Np];  // own normal derivative
    __shared__ double up[NF][Np];  // neighbour's trace and derivative at the same points
    __shared__ double dp[NF][Np];
    __shared__ double wJ[NF], tau2[3];
    __shared__ int cn[3];
    for (int k = blockIdx.x; k < a.K; k += gridDim.x) {
        const double* fck = o.fc + (size_t)k * 3 * kFaceCoef;
        if (threadIdx.x < 3) {
            cn[threadIdx.x] = a.conn[(size_t)k * 3 + threadIdx.x];
            tau2[threadIdx.x] = fck[threadIdx.x * kFaceCoef + 4];
        }
        if (threadIdx.x < NF) wJ[threadIdx.x] = fck[threadIdx.x / Nfq * kFaceCoef + 5] * o.fw[threadIdx.x % Nfq];
        __syncthreads();
        for (int t = threadIdx.x; t < NF * Np; t += blockDim.x) {
            const int fg = t / Np, p = t - fg * Np, f = fg / Nfq, g = fg - f * Nfq;
            const double* fc = fck + f * kFaceCoef;
            auto trace = [&](int face, int gq) {  // basis p on `face` at its Gauss point gq
                if (p >= NB) return 0.0;
                const int d = (p - face * N + NB) % NB;
                return d <= N ? o.If[gq * Nfp + d] : 0.0;
            };
            tr[fg][p] = trace(f, g);
            dm[fg][p] = fc[0] * o.Drf[(size_t)fg * Np + p] + fc[1] * o.Dsf[(size_t)fg * Np + p];
            double u = 0.0, d = 0.0;
            if (cn[f] >= 0) {
                const int fn = cn[f] & 3, g2 = ((cn[f] >> 2) & 1) ? Nfq - 1 - g : g, fg2 = fn * Nfq + g2;
                u = trace(fn, g2);
                d = fc[2] * o.Drf[(size_t)fg2 * Np + p] + fc[3] * o.Dsf[(size_t)fg2 * Np + p];
            }
            up[fg][p] = u;
            dp[fg][p] = d;
        }
        __syncthreads();
        const double vrr = o.vc[(size_t)k * 3], vrs = o.vc[(size_t)k * 3 + 1], vss = o.vc[(size_t)k * 3 + 2];
        const double mc = a.mass_coef * a.J[k];
        const int grp = k / R::EB, e = k - grp * R::EB;
        T* col0 = sb ? sb + (size_t)grp * kRowCols<Np> * R::EB * Np + e * Np : nullptr;
        constexpr size_t CS = (size_t)R::EB * Np;  // column stride
        for (int t = threadIdx.x; t < Np * Np; t += blockDim.x) {
            const int j = t / Np, i = t - j * Np;
            double v = vrr * o.Srr[j * Np + i] + vrs * o.Srs2[j * Np + i] + vss * o.Sss[j * Np + i] + mc * o.Mr[j * Np + i];
#pragma unroll
            for (int f = 0; f < 3; f++) {
                const double h = cn[f] >= 0 ? 0.5 : 1.0;  // a / 2
                double vo = 0.0;
#pragma unroll
                for (int g = 0; g < Nfq; g++) {
                    const int fg = f * Nfq + g;
                    const double ti = wJ[fg] * tr[fg][i], di = wJ[fg] * dm[fg][i];
                    v += ti * (2.0 * h * tau2[f] * tr[fg][j] - h * dm[fg][j]) - h * di * tr[fg][j];
                    vo += 0.5 * di * up[fg][j] - ti * (tau2[f] * up[fg][j] + 0.5 * dp[fg][j]);
                }
                if (col0) col0[((size_t)(f + 1) * Np + j) * CS + i] = (T)vo;
            }
            if (col0) col0[(size_t)j * CS + i] = (T)v;
            if (diag) diag[((size_t)k * Np + i) * Np + j] = v;
        }
        if (col0)
            for (int i = threadIdx.x; i < Np; i += blockDim.x) {
                double wb = mc * o.mrow[i];
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    double s = 0.0;
#pragma unroll
                    for (int g = 0; g < Nfq; g++) {
                        const int fg = f * Nfq + g;
                        s += wJ[fg] * (tau2[f] * tr[fg][i] - 0.5 * dm[fg][i]);
                    }
                    // inside: row sums of the neighbour block; Dirichlet: twice the term, on u_0
                    col0[((size_t)4 * Np + f) * CS + i] = cn[f] >= 0 ? (T)-s : (T)0;
                    if (cn[f] < 0) wb += 2.0 * s;
                }
                col0[((size_t)4 * Np + 3) * CS + i] = (T)wb;
            }
        __syncthreads();
    }
}

// y = S u (or, in the PCG, y = S p with p = z + beta p_old formed here, its
// rows written out, and p.y summed grid-wide): one lane per row; the element's
// own and its neighbours' values reach the rows by shuffles (through shared
// memory at N = 7).  The block columns are coalesced 8-byte reads.
template <int NP>
__global__ void __launch_bounds__(RowDims<NP>::THREADS, 3) block_apply_kernel(IpdgArgs a, const double* __restrict__ u,
                                                                             double* __restrict__ y, ApplyPcg pc) {
    using R = RowDims<NP>;
    constexpr int EB = R::EB, CS = EB * NP;
    dependency_wait();
    double beta = 0.0;
    if (pc.S) {
        if (pc.S->done) return;
        beta = pc.S->beta;
    }
    const bool has_beta = beta != 0.0;
    int e, i;
    row_of<NP>(e, i);
    const int ngroups = row_groups<NP>(a.K);
    auto value = [&](size_t idx) { return has_beta ? fma(beta, pc.p_old[idx], u[idx]) : u[idx]; };
    double dot = 0;
    __shared__ double sm[R::WA ? 1 : EB][4][NP];
    for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const int k = grp * EB + e;
        const bool act = e < EB && k < a.K;
        const size_t idx = (size_t)k * NP + i;
        double v[4] = {0, 0, 0, 0};  // own value, neighbours' (zero across a boundary)
        if (act) {
            int c[3];
#pragma unroll
            for (int f = 0; f < 3; f++) c[f] = a.conn[(size_t)k * 3 + f];
            v[0] = value(idx);
#pragma unroll
            for (int f = 0; f < 3; f++)
                if (c[f] >= 0) v[f + 1] = value((size_t)(c[f] >> 3) * NP + i);
            if (pc.p_new) pc.p_new[idx] = v[0];
        }
        const double* col = a.sblocks + (size_t)grp * kRowCols<NP> * CS + (act ? e * NP + i : 0);
        double s = 0;
        if constexpr (R::WA) {
            const int lb = (threadIdx.x & 31) - i;  // lane of the element's row 0
            double first[4];
#pragma unroll
            for (int b = 0; b < 4; b++) first[b] = __shfl_sync(0xffffffffu, v[b], lb);
            if (act) {
                s = col[(size_t)(4 * NP + 3) * CS] * first[0];
#pragma unroll
                for (int f = 0; f < 3; f++) s = fma(col[(size_t)(4 * NP + f) * CS], first[f + 1] - first[0], s);
            }
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const double d = v[b] - first[b];
#pragma unroll
                for (int j = 0; j < NP; j++) {
                    const double dj = __shfl_sync(0xffffffffu, d, lb + j);
                    if (act) s = fma(__ldg(col + (size_t)(b * NP + j) * CS), dj, s);
                }
            }
        } else {
            __syncthreads();
            if (act)
#pragma unroll
                for (int b = 0; b < 4; b++) sm[e][b][i] = v[b];
            __syncthreads();
            double first[4] = {0, 0, 0, 0};
            if (act) {
#pragma unroll
                for (int b = 0; b < 4; b++) first[b] = sm[e][b][0];
                s = col[(size_t)(4 * NP + 3) * CS] * first[0];
#pragma unroll
                for (int f = 0; f < 3; f++) s = fma(col[(size_t)(4 * NP + f) * CS], first[f + 1] - first[0], s);
            }
            __syncthreads();
            if (act)
#pragma unroll
                for (int b = 0; b < 4; b++) sm[e][b][i] = v[b] - first[b];
            __syncthreads();
            if (act)
                for (int b = 0; b < 4; b++)
#pragma unroll 12
                    for (int j = 0; j < NP; j++) s = fma(__ldg(col + (size_t)(b * NP + j) * CS), sm[e][b][j], s);
        }
        if (act) {
            y[idx] = s;
            dot += s * v[0];
        }
    }
    if (pc.S) {
        // the halving tree wants a power of two of threads: N = 7 runs 256 too
        double val[1] = {dot}, tot[1];
        if (grid_sum<1>(val, pc.part, gridDim.x, &pc.S->counter, tot) && threadIdx.x == 0) {
            const double pap = tot[0];
            pc.S->pap = pap;
            pc.S->alpha = pc.S->rz / pap;
            if (!(pap > 0.0) || !(pc.S->alpha == pc.S->alpha)) pc.S->done = 2;
        }
    }
}

template <int N, typename T>
cudaError_t blocks_n(const IpdgArgs& a, double* diag, T* sb, cudaStream_t s) {
    ipdg_blocks_kernel<N, T><<<std::min(a.K, 16 * a.sms), 128, 0, s>>>(a, diag, sb);
    return cudaGetLastError();
}

template <typename T>
cudaError_t blocks_dispatch(const IpdgArgs& a, double* diag, T* sb, cudaStream_t s) {
    switch (a.N) {
        case 1: return blocks_n<1, T>(a, diag, sb, s);
        case 2: return blocks_n<2, T>(a, diag, sb, s);
        case 3: return blocks_n<3, T>(a, diag, sb, s);
        case 4: return blocks_n<4, T>(a, diag, sb, s);
        case 5: return blocks_n<5, T>(a, diag, sb, s);
        case 6: return blocks_n<6, T>(a, diag, sb, s);
        case 7: return blocks_n<7, T>(a, diag, sb, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_ipdg_diag(const IpdgArgs& a, double* blocks, cudaStream_t s) { return blocks_dispatch<double>(a, blocks, nullptr, s); }
cudaError_t launch_block_rows(const IpdgArgs& a, double* sblocks, cudaStream_t s) { return blocks_dispatch<double>(a, nullptr, sblocks, s); }
cudaError_t launch_block_rows(const IpdgArgs& a, float* sblocks, cudaStream_t s) { return blocks_dispatch<float>(a, nullptr, sblocks, s); }

size_t block_rows_size(int K, int Np) {
    auto n = [&](auto tag) {
        constexpr int NP = decltype(tag)::value;
        return (size_t)row_groups<NP>(K) * kRowCols<NP> * RowDims<NP>::EB * NP;
    };
    switch (Np) {
        case 3: return n(std::integral_constant<int, 3>());
        case 6: return n(std::integral_constant<int, 6>());
        case 10: return n(std::integral_constant<int, 10>());
        case 15: return n(std::integral_constant<int, 15>());
        case 21: return n(std::integral_constant<int, 21>());
        case 28: return n(std::integral_constant<int, 28>());
        case 36: return n(std::integral_constant<int, 36>());
        default: return 0;
    }
}

template <int NP>
static cudaError_t block_apply_n(const IpdgArgs& a, const double* u, double* y, const ApplyPcg& pc, cudaStream_t s) {
    const int grid = std::max(1, std::min(row_groups<NP>(a.K), 3 * a.sms));
    return launch_dependent(block_apply_kernel<NP>, grid, RowDims<NP>::THREADS, s, a, u, y, pc);
}

cudaError_t launch_block_apply(const IpdgArgs& a, const double* u, double* y, const ApplyPcg& pc, cudaStream_t s) {
    switch (a.Np) {
        case 3: return block_apply_n<3>(a, u, y, pc, s);
        case 6: return block_apply_n<6>(a, u, y, pc, s);
        case 10: return block_apply_n<10>(a, u, y, pc, s);
        case 15: return block_apply_n<15>(a, u, y, pc, s);
        case 21: return block_apply_n<21>(a, u, y, pc, s);
        case 28: return block_apply_n<28>(a, u, y, pc, s);
        case 36: return block_apply_n<36>(a, u, y, pc, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace dgk
