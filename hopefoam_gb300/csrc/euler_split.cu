// euler_split.cu -- split-precision fused DG Euler stage on the tcgen05 tensor
// cores (sm_103a).
//
// Arithmetic: the two contractions of the quadrature-form DG right-hand side
// run as TF32 GEMMs with 3-pass split products (hi*hi + lo*hi + hi*lo) and
// FP32 accumulation in tensor memory, on deltas against a per-element
// reference state qb (the row mean):
//   GEMM1 (cubature interpolation, dgGaussField.C:193-202):
//     dQg[r][g] = sum_p dQ[r][p] Vg[g][p],      M = 128 rows r = 4 e + v
//                                               (32 elements x 4 variables),
//                                               N = Ng padded, K = Np padded
//   GEMM2 (volume term + surface lift with the affine mass inverse folded in,
//          defaultConvectionScheme.C:79-128, defaultGrad.C:120-165,
//          defaultDivScheme.C:118-165):
//     R[r][p] = sum_g dFr[r][g] Sr[p][g] + dFs[r][g] Ss[p][g]
//             + sum_c (-sJ/J dF*)[r][c] Lift[p][c],   N = Np padded
// with dF = F(qb + dQ) - F(qb) and dF* = n.F*(q-, q+) - n.F(qb) evaluated
// point-wise in FP32 in cancellation-free product-rule form (euler_flux.cuh).
// Because the weak divergence of a constant flux cancels against its own
// surface term, R is unchanged by the shift, but the FP32 round-off now
// scales with the variation inside an element instead of with |F| N^2 / h.
// The state q stays FP64 in HBM; dQ = q - qb (and the neighbour traces' deltas)
// is one FP64 subtraction and conversion per value (at N = 7 it is formed from
// q's bits with integer and FP32 operations, f64split.cuh); the low-storage RK
// register is FP32 (it carries dt*R, whose own precision is FP32); q += b*res
// is the only other FP64 arithmetic per value.
//
// The kernel is in euler_split_pipe.cu; here are its operands' images, set-up and
// launch.  Persistent CTAs take tiles of 32 elements.  Per tile: q (FP64 tile in shared
// memory) -> reference state, FP32 deltas, TF32 hi/lo in the canonical no-swizzle
// K-major layout (umma.cuh) -> GEMM1 -> face fluxes in lane segments, one per (element,
// face) (Gauss interpolation and wave-speed max by shuffles); per chunk of 16 cubature
// points: tensor memory -> registers, the 4 variables of a point exchanged by a
// two-stage butterfly of warp shuffles within the element's 4 lanes -> FP32 delta
// flux -> TF32 split into a chunk operand -> GEMM2 MMAs for that K chunk -> epilogue:
// tensor memory -> shared -> coalesced LSERK update.  At N = 7 the volume
// operator is streamed from L2 per chunk and the tile is not copied to shared
// memory (SplitDims::STREAM).
#include <cstring>
#include <vector>

#include "../../include/dgcu.h"
#include "dg_ctx.hpp"
#include "euler_split.cuh"
#include "umma.cuh"

namespace dgk {

static inline float tf32_rna(float x) {
    uint32_t u;
    memcpy(&u, &x, 4);
    u = (u + 0x1000u) & 0xFFFFE000u;
    float r;
    memcpy(&r, &u, 4);
    return r;
}

// canonical K-major image of an (rows x KP) operand given by f(row, k) (double),
// hi part then lo part
template <typename F>
static std::vector<float> operand_image(int rows, int KP, F f) {
    std::vector<float> img((size_t)2 * rows * KP, 0.f);
    const size_t lo = (size_t)rows * KP;
    for (int r = 0; r < rows; r++)
        for (int k = 0; k < KP; k++) {
            const double x = f(r, k);
            const float hi = tf32_rna((float)x);
            const float l = (float)(x - (double)hi);
            const size_t off = umma::kmajor_offset(r, k, KP) >> 2;
            img[off] = hi;
            img[lo + off] = l;
        }
    return img;
}

template <int N>
static int setup_n(dg_ctx* c) {
    using D = SplitDims<N>;
    const dgb::RefOps& o = c->ops;
    const int Np = D::Np, Ng = D::Ng, Nfq = D::Nfq, NG = D::NG;
    std::vector<float> b1 = operand_image(D::NG, D::KP1, [&](int g, int p) {
        return (g < Ng && p < Np) ? o.dVg[(size_t)g * Np + p] : 0.0;
    });
    std::vector<float> b2;
    if (D::STREAM) {
        // lift image (resident), then one [Sr 16 | Ss 16] image per chunk (streamed)
        b2 = operand_image(D::NP2, D::NF, [&](int p, int cc) {
            return (p < Np && cc < 3 * Nfq) ? o.dLift[(size_t)p * 3 * Nfq + cc] : 0.0;
        });
        for (int ch = 0; ch < D::NCH; ch++) {
            std::vector<float> bc = operand_image(D::NP2, D::KC, [&](int p, int k) {
                const int g = ch * D::CH + (k < D::CH ? k : k - D::CH);
                if (p >= Np || g >= Ng) return 0.0;
                return k < D::CH ? o.dSr[(size_t)p * Ng + g] : o.dSs[(size_t)p * Ng + g];
            });
            b2.insert(b2.end(), bc.begin(), bc.end());
        }
    } else {
        b2 = operand_image(D::NP2, D::KP2, [&](int p, int k) {
            if (p >= Np) return 0.0;
            if (k < NG) return k < Ng ? o.dSr[(size_t)p * Ng + k] : 0.0;
            if (k < 2 * NG) return (k - NG) < Ng ? o.dSs[(size_t)p * Ng + (k - NG)] : 0.0;
            const int cc = k - 2 * NG;
            return cc < 3 * Nfq ? o.dLift[(size_t)p * 3 * Nfq + cc] : 0.0;
        });
    }
    std::vector<float> if32(o.If.begin(), o.If.end());  // Nfq x Nfp
    size_t bytes = (b1.size() + b2.size() + if32.size()) * sizeof(float);
    float* d = nullptr;
    if (cudaMalloc(&d, bytes) != cudaSuccess) return DG_ERR_NOMEM;
    cudaMemcpy(d, b1.data(), b1.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d + b1.size(), b2.data(), b2.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d + b1.size() + b2.size(), if32.data(), if32.size() * 4, cudaMemcpyHostToDevice);
    c->split.d_ops = d;
    c->split.ops_bytes = bytes;
    c->split.b2_offset = b1.size();
    c->split.if32_offset = b1.size() + b2.size();
    if (cudaMalloc(&c->split.d_status, sizeof(int)) != cudaSuccess) return DG_ERR_NOMEM;
    cudaMemset(c->split.d_status, 0, sizeof(int));
    if (cudaMalloc(&c->split.d_res32, (size_t)c->K * 4 * Np * sizeof(float)) != cudaSuccess) return DG_ERR_NOMEM;
    cudaMemset(c->split.d_res32, 0, (size_t)c->K * 4 * Np * sizeof(float));
    if (setup_split_pipe<N>() != cudaSuccess) return DG_ERR_CUDA;
    if (!D::STREAM && setup_split_batch() != cudaSuccess) return DG_ERR_CUDA;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    c->split.sms = sms;
    c->split.N = N;
    c->split.ready = true;
    return DG_OK;
}

int split_fill_args(const EulerArgs& a, const SplitPlan& plan, SplitArgs* sa) {
    sa->e = a;
    sa->res32 = plan.d_res32;
    sa->res32_out = plan.d_res32;
    sa->b1 = static_cast<const float*>(plan.d_ops);
    sa->b2 = static_cast<const float*>(plan.d_ops) + plan.b2_offset;
    sa->status = plan.d_status;
    sa->qbulk = (reinterpret_cast<uintptr_t>(a.qin) & 15u) == 0;
    sa->If32 = static_cast<const float*>(plan.d_ops) + plan.if32_offset;
    sa->dtk32 = a.dtk ? a.dtk32 : nullptr;
    sa->rkaf = (float)a.rka;
    sa->rkbf = (float)a.rkb;
    sa->dtf = (float)a.dt;
    sa->first = a.rka == 0.0;
    return DG_OK;
}

template <int N>
static cudaError_t launch_split_n(const EulerArgs& a, const SplitPlan& plan, cudaStream_t s) {
    using D = SplitDims<N>;
    SplitArgs sa;
    split_fill_args(a, plan, &sa);
    const int ntiles = (a.K + D::E - 1) / D::E;
    if (!D::STREAM && !sa.qbulk) return cudaErrorMisalignedAddress;  // the tile copies want 16 bytes
    const int sms = (plan.sm_budget > 0 && plan.sm_budget < plan.sms) ? plan.sm_budget : plan.sms;
    return launch_split_pipe<N>(sa, ntiles < sms ? ntiles : sms, s);
}

cudaError_t launch_euler_split(int N, const EulerArgs& a, const SplitPlan& plan, cudaStream_t s) {
    if (!plan.ready || plan.N != N) return cudaErrorNotSupported;
    switch (N) {
        case 1: return launch_split_n<1>(a, plan, s);
        case 2: return launch_split_n<2>(a, plan, s);
        case 3: return launch_split_n<3>(a, plan, s);
        case 4: return launch_split_n<4>(a, plan, s);
        case 5: return launch_split_n<5>(a, plan, s);
        case 6: return launch_split_n<6>(a, plan, s);
        case 7: return launch_split_n<7>(a, plan, s);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace dgk

int split_setup(dg_ctx* c) {
    c->split.ready = false;
    switch (c->N) {
        case 1: return dgk::setup_n<1>(c);
        case 2: return dgk::setup_n<2>(c);
        case 3: return dgk::setup_n<3>(c);
        case 4: return dgk::setup_n<4>(c);
        case 5: return dgk::setup_n<5>(c);
        case 6: return dgk::setup_n<6>(c);
        case 7: return dgk::setup_n<7>(c);
        default: return DG_ERR_UNSUPPORTED;
    }
}

void split_teardown(dg_ctx* c) {
    if (c->split.d_ops) cudaFree(c->split.d_ops);
    if (c->split.d_status) cudaFree(c->split.d_status);
    if (c->split.d_res32) cudaFree(c->split.d_res32);
    c->split.d_ops = nullptr;
    c->split.d_status = nullptr;
    c->split.d_res32 = nullptr;
    c->split.ready = false;
}
