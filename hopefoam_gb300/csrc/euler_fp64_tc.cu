// euler_fp64_tc.cu -- FP64 Euler stage with its contractions on the tensor
// cores (sm_103a).
//
// GB300 retires two FP64 operations per clock per SM, and of the ~21,000 an
// element needs per stage at N = 5 the contractions (interpolation to the
// cubature and face points, weak derivative, lift) are 18,400.  Here those
// run as exact integer products on tcgen05 (ozaki.cuh: seven base-256
// digits per value, FP16 operands, FP32 accumulators that hold exact
// integers), with an error against 64 bits below the FMA chain's; the FP64
// pipe keeps the point-wise fluxes (25 operations per cubature point with
// reciprocals from FP32 seeds) and the Runge-Kutta update.
//
// One CTA per SM walks tiles of 32 elements (128 operand rows).  Warps
// 0-15 compute: warp w owns the eight elements 8 (w % 4) .. + 7, the ones
// whose tensor-memory lanes it can read, and quarter w / 4 of the points, so
// only the four warps of one such group ever wait for each other (named
// barriers); warp 16 feeds the tensor core (operator pieces arrive by bulk
// copies in a ring, consumed in a fixed order) and all hand-overs are
// mbarriers, so warps in their integer phases overlap warps in their FP64
// phase.  Per tile:
//   1. own nodes and neighbour face nodes -> digit operands;
//   2. traces at the face points (two products), numerical flux, digits;
//   3. per chunk of 16 cubature points: state at the points (product),
//      fluxes, digits, product into the result accumulators;
//   4. result rows -> FP64, stage update.
// The digits of a row share one exponent.  For the nodal rows it is the row's
// own; for the flux rows it comes from the face fluxes and from a bound on
// the volume fluxes formed from the element's nodal extremes.  An element
// whose fluxes leave that bound, or with values that are not finite or
// outside the FP32 exponent range, is recomputed by its warps in plain FP64,
// as euler_fp64.cu does it (plain_element).  All of this is per element:
// results do not depend on an element's place in the mesh.
//
// Measured, LSERK4 step with the state's layout changes, against the kernel of
// euler_fp64.cu: K = 32768, N = 5, LF 13.36 -> 2.13 ms; K = 9798, N = 7, Roe
// 13.14 -> 1.10 ms; K = 3200, N = 3, LF 392 -> 139 us; SSP-RK2 step at
// K = 512, N = 2 42 -> 31 us.  So it is taken at every order and size.
// Right-hand sides against 80-bit arithmetic: 2.7e-13 relative at N = 5, both.
//
// Every mbarrier wait is bounded; on a timeout the CTA stops waiting, sets
// the status word, lets its copies and MMAs in flight end, frees its tensor
// memory and exits.
#include <cstring>

#include "dg_ctx.hpp"
#include "euler_flux.cuh"
#include "euler_fp64_tc.cuh"
#include "euler_split.cuh"
#include "umma.cuh"

namespace dgk {

namespace {

constexpr int kOzThreads = 544;

struct OzArgs {
    EulerArgs e;
    const unsigned char* image;
    const int* eb;
    int* status;
};

__device__ __forceinline__ uint32_t idesc_f16(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (8u << 24);  // D F32, A = B = F16, M = 128
}

__device__ __forceinline__ double shfl_x(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

// 4 x 4 transpose between lanes l, l ^ 8, l ^ 16, l ^ 24: lane 8 v + e holds
// variable v of four points, afterwards the four variables of point v
__device__ __forceinline__ void transpose4(double x[4], int lane) {
    const bool b1 = lane & 16, b0 = lane & 8;
#pragma unroll
    for (int p = 0; p < 2; p++) {
        const double r = shfl_x(b1 ? x[p] : x[p + 2], 16);
        if (b1) x[p] = r;
        else x[p + 2] = r;
    }
#pragma unroll
    for (int v = 0; v < 4; v += 2) {
        const double r = shfl_x(b0 ? x[v] : x[v + 1], 8);
        if (b0) x[v] = r;
        else x[v + 1] = r;
    }
}

// four consecutive columns of seven digit groups (stride P) -> FP64 values
// of the lane's row
template <int P>
__device__ __forceinline__ void load7(uint32_t taddr, int ebab, double x[4]) {
    float d[7][4];
#pragma unroll
    for (int s = 0; s < 7; s++) umma::tmem_ld4(taddr + s * P, d[s]);
    umma::tmem_ld_wait();
#pragma unroll
    for (int c = 0; c < 4; c++)
        x[c] = oz::combine7(oz::acc_int22(d[0][c]), oz::acc_int22(d[1][c]), oz::acc_int22(d[2][c]),
                            oz::acc_int22(d[3][c]), oz::acc_int22(d[4][c]), oz::acc_int22(d[5][c]),
                            oz::acc_int22(d[6][c]), ebab);
}

struct FaceSide {
    double r, u, v, p, mn;
};
__device__ __forceinline__ FaceSide face_side(double g1, double nx, double ny, const double q[4]) {
    FaceSide s;
    s.r = oz::rcp64(q[0]);
    s.u = q[1] * s.r;
    s.v = q[2] * s.r;
    s.p = g1 * fma(-0.5, fma(q[1], s.u, q[2] * s.v), q[3]);
    s.mn = fma(nx, q[1], ny * q[2]);
    return s;
}

// Roe flux, euler_flux.cuh's roe_flux with reciprocals
__device__ __forceinline__ void roe_flux_fast(double g1, double nx, double ny, const double qO[4], const double qN[4],
                                              double F[4]) {
    const double QP2 = fma(nx, qN[1], ny * qN[2]), QM2 = fma(nx, qO[1], ny * qO[2]);
    const double QP3 = fma(nx, qN[2], -ny * qN[1]), QM3 = fma(nx, qO[2], -ny * qO[1]);
    const double rP = oz::rcp64(qN[0]), rM = oz::rcp64(qO[0]);
    const double uM = QM2 * rM, uP = QP2 * rP, vM = QM3 * rM, vP = QP3 * rP;
    const double pM = g1 * fma(-0.5, fma(QM2, uM, QM3 * vM), qO[3]);
    const double pP = g1 * fma(-0.5, fma(QP2, uP, QP3 * vP), qN[3]);
    const double eM = qO[3] + pM, eP = qN[3] + pP;
    double fr = QM2 + QP2;
    double fu = fma(QM2, uM, pM) + fma(QP2, uP, pP);
    double fv = fma(QM3, uM, QP3 * uP);
    double fe = fma(uM, eM, uP * eP);
    const double sM = oz::sqrt64(qO[0]), sP = oz::sqrt64(qN[0]);
    const double rhob = sM * sP, w = oz::rcp64(sM + sP);
    const double aM = sM * w, aP = sP * w;
    const double u = fma(aM, uM, aP * uP), v = fma(aM, vM, aP * vP);
    const double H = fma(aM, eM * rM, aP * (eP * rP));
    const double ke = fma(u, u, v * v);
    const double c2 = g1 * fma(-0.5, ke, H);
    const double ic = oz::rsqrt64(fabs(c2));
    const double c = fabs(c2) * ic;
    const double jp = pP - pM;
    const double a = 0.5 * rhob * (uP - uM) * ic, jc = jp * copysign(ic * ic, c2), b = 0.5 * jc;
    const double um = u - c, up = u + c;
    const double dw1 = (b - a) * fabs(um);
    const double dw2 = ((qN[0] - qO[0]) - jc) * fabs(u);
    const double dw3 = rhob * (vP - vM) * fabs(u);
    const double dw4 = (a + b) * fabs(up);
    const double dr = dw1 + dw2 + dw4;
    fr -= dr;
    fu -= fma(dw1, um, fma(dw2, u, dw4 * up));
    fv -= fma(dr, v, dw3);
    const double uc = u * c;
    fe -= fma(dw1, H - uc, fma(dw2, 0.5 * ke, fma(dw3, v, dw4 * (H + uc))));
    F[0] = 0.5 * fr;
    F[1] = 0.5 * fma(nx, fu, -ny * fv);
    F[2] = 0.5 * fma(ny, fu, nx * fv);
    F[3] = 0.5 * fe;
}

__device__ __forceinline__ void group_sync(int sub) { asm volatile("bar.sync %0, 128;" ::"r"(sub + 1) : "memory"); }

// place of scratch value i of element group `sub` in an operand whose slices
// are `stride` bytes and hold `per` bytes of the group's rows each
__device__ __forceinline__ double* striped(unsigned char* base, int sub, int i, int stride, int per) {
    const int n = per >> 3, s = i / n;
    return reinterpret_cast<double*>(base + (size_t)s * stride + (size_t)sub * per) + (i - s * n);
}

// Right-hand side of element k in plain FP64 by the 128 threads of its group,
// operation for operation as euler_stage_fp64_kernel forms it
template <int N, typename Sc, typename Out>
__device__ __noinline__ void plain_element(const EulerArgs& a, int k, int t, int sub, Sc sc, Out out) {
    using D = OzDims<N>;
    constexpr int Np = D::Np, Ng = D::Ng, Nfp = D::Nfp, Nfq = D::Nfq, NB = D::NB, NF = D::NF;
    const double* qe = a.qin + (size_t)k * 4 * Np;
    const double* gk = a.geo + (size_t)k * 4;
    const double rx = gk[0], sx = gk[1], ry = gk[2], sy = gk[3], gamma = a.gamma;
    for (int g = t; g < Ng; g += 128) {
        double q[4] = {0, 0, 0, 0}, fx[4], fy[4];
        for (int p = 0; p < Np; p++) {
            const double w = a.ops.Vg[g * Np + p];
            for (int v = 0; v < 4; v++) q[v] += w * qe[v * Np + p];
        }
        euler_phys_flux(gamma, q, fx, fy);
        for (int v = 0; v < 4; v++) {
            *sc(v * Ng + g) = rx * fx[v] + ry * fy[v];
            *sc((4 + v) * Ng + g) = sx * fx[v] + sy * fy[v];
        }
    }
    if (t < 3) {
        const int f = t, c = a.conn[(size_t)k * 3 + f];
        double nx, ny, fsc, lam = 0;
        face_normal(f, rx, sx, ry, sy, nx, ny, fsc);
        auto side = [&](int i, double qm[4], double qp[4]) {
            for (int v = 0; v < 4; v++) {
                double m = 0, p = 0;
                for (int j = 0; j < Nfp; j++) {
                    const double w = a.ops.If[i * Nfp + j];
                    m += w * qe[v * Np + (f * N + j) % NB];
                    double o;
                    if (c >= 0) {
                        const int fn = c & 3, jj = ((c >> 2) & 1) ? (N - j) : j;
                        o = a.qin[((size_t)(c >> 3) * 4 + v) * Np + (fn * N + jj) % NB];
                    } else {
                        o = a.btrace[((size_t)(-1 - c) * 4 + v) * Nfp + j];
                    }
                    p += w * o;
                }
                qm[v] = m;
                qp[v] = p;
            }
        };
        if (a.flux != 1)
            for (int i = 0; i < Nfq; i++) {
                double qm[4], qp[4];
                side(i, qm, qp);
                lam = fmax(lam, wave_speed(gamma, nx, ny, qm));
                lam = fmax(lam, wave_speed(gamma, nx, ny, qp));
            }
        for (int i = 0; i < Nfq; i++) {
            double qm[4], qp[4], F[4];
            side(i, qm, qp);
            if (a.flux == 1) roe_flux(gamma, nx, ny, qm, qp, F);
            else lf_flux(gamma, nx, ny, lam, qm, qp, F);
            for (int v = 0; v < 4; v++) *sc(8 * Ng + v * NF + f * Nfq + i) = fsc * F[v];
        }
    }
    group_sync(sub);
    for (int it = t; it < 4 * Np; it += 128) {
        const int v = it / Np, p = it - v * Np;
        double acc = 0, acc2 = 0, accf = 0;
        for (int g = 0; g < Ng; g++) {
            acc += a.ops.Sr[p * Ng + g] * *sc(v * Ng + g);
            acc2 += a.ops.Ss[p * Ng + g] * *sc((4 + v) * Ng + g);
        }
        acc += acc2;
        for (int q = 0; q < NF; q++) accf += a.ops.Lift[p * NF + q] * *sc(8 * Ng + v * NF + q);
        *out(it) = acc - accf;
    }
    group_sync(sub);
}

}  // namespace

template <int N>
__global__ void __launch_bounds__(kOzThreads, 1) euler_stage_fp64_tc_kernel(OzArgs oa) {
    using D = OzDims<N>;
    constexpr int Np = D::Np, Ng = D::Ng, Nfp = D::Nfp, Nfq = D::Nfq, NB = D::NB, NF = D::NF, K1 = D::K1;
    const EulerArgs& a = oa.e;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* A1 = smem + D::OFF_A1;
    unsigned char* A2 = smem + D::OFF_A2;
    double* lamS = reinterpret_cast<double*>(smem + D::OFF_LAM);
    double* geoS = reinterpret_cast<double*>(smem + D::OFF_GEO);
    double* nrmS = reinterpret_cast<double*>(smem + D::OFF_NRM);
    int* connS = reinterpret_cast<int*>(smem + D::OFF_CONN);
    uint32_t* maxq = reinterpret_cast<uint32_t*>(smem + D::OFF_MAXQ);
    int* minr = reinterpret_cast<int*>(smem + D::OFF_MINR);
    int* e3S = reinterpret_cast<int*>(smem + D::OFF_E3);
    uint32_t* maxf = reinterpret_cast<uint32_t*>(smem + D::OFF_MAXF);
    uint32_t* flagS = reinterpret_cast<uint32_t*>(smem + D::OFF_FLAG);
    int* ebS = reinterpret_cast<int*>(smem + D::OFF_EB);
    volatile int* dead = reinterpret_cast<volatile int*>(smem + D::OFF_DEAD);
    uint32_t* tmemS = reinterpret_cast<uint32_t*>(smem + D::OFF_TMEM);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + D::OFF_BAR);
    uint64_t *bAready = bars, *bTrFull = bars + 1, *bTrRead = bars + 2, *bA2w = bars + 3, *bA2free = bars + 4,
             *bD1full = bars + 5, *bD1read = bars + 6, *bFin = bars + 7, *bFull = bars + 8, *bEmpty = bFull + D::NSLOT;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        umma::mbar_init(bAready, 16);
        umma::mbar_init(bTrFull, 1);
        umma::mbar_init(bTrRead, 16);
        umma::mbar_init(bA2w, 16);
        umma::mbar_init(bA2free, 1);
        umma::mbar_init(bD1full, 1);
        umma::mbar_init(bD1read, 16);
        umma::mbar_init(bFin, 1);
        for (int i = 0; i < D::NSLOT; i++) {
            umma::mbar_init(bFull + i, 1);
            umma::mbar_init(bEmpty + i, 1);
        }
        umma::fence_mbar_init();
        *dead = 0;
    }
    for (int i = threadIdx.x; i < D::NP2 + 2; i += kOzThreads) ebS[i] = oa.eb[i];
    if (warp == 16) umma::tmem_alloc(tmemS, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmemS;
    const int ntiles = (a.K + 31) / 32;

    auto wait = [&](uint64_t* bar, uint32_t phase) {
        if (*dead) return;
        if (!umma::mbar_wait(bar, phase, kWaitLimit)) *dead = 1;
    };

    if (warp == 16) {
        // -------------------------------------------------------------- tensor-core feeder
        if (lane == 0) {
            const int mine = (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
            const long long total = (long long)mine * D::PIECES;
            long long nload = 0, nuse = 0;
            int loadp = 0;
            size_t loado = 0;
            auto load = [&]() {
                if (nload >= total || *dead) return;
                const int s = (int)(nload % D::NSLOT);
                if (nload >= D::NSLOT) wait(bEmpty + s, (uint32_t)((nload / D::NSLOT - 1) & 1));
                if (*dead) return;
                const uint32_t n = loadp == 0 ? D::B1F : loadp == 1 ? D::B3 : loadp == 2 ? D::B1
                                   : loadp == 3 || loadp == D::PIECES - 1 ? D::B2 : (loadp & 1) ? D::B2 : D::B1;
                umma::mbar_arrive_expect_tx(bFull + s, n);
                umma::bulk_g2s(smem + D::OFF_RING + s * D::SLOT, oa.image + loado, n, bFull + s);
                loado += n;
                if (++loadp == D::PIECES) {
                    loadp = 0;
                    loado = 0;
                }
                nload++;
            };
            for (int i = 0; i < D::NSLOT - 1; i++) load();
            auto take = [&]() {  // the next piece, landed
                const int s = (int)(nuse % D::NSLOT);
                wait(bFull + s, (uint32_t)((nuse / D::NSLOT) & 1));
                return umma::smem_u32(smem + D::OFF_RING + s * D::SLOT);
            };
            auto done = [&]() {  // its MMAs are issued
                umma::commit(bEmpty + (int)(nuse % D::NSLOT));
                nuse++;
                load();
            };
            // digit product of a nodal operand (slice stride AS, reduction KP) with P points
            auto product = [&](uint32_t d, uint32_t as, int AS, int KP, uint32_t bs, int P) {
                const uint32_t sbo = (uint32_t)(KP >> 3) << 7;
                for (int i = 0; i < oz::kSlices; i++) {
                    const uint32_t id = idesc_f16((oz::kSlices - i) * P);
                    for (int ks = 0; ks < KP / 16; ks++)
                        umma::mma_bf16(d + i * P, umma::smem_desc(as + i * AS + ks * 256, 128, sbo),
                                       umma::smem_desc(bs + ks * 256, 128, sbo), id, i + ks > 0 ? 1u : 0u);
                }
            };
            // flux operand times a B2 piece into the result groups (pairs i + j <= 7;
            // digit block 7 of the operator is zero and starts every group)
            auto product2 = [&](uint32_t bs, bool first) {
                const uint32_t as = umma::smem_u32(A2), sbo = 4u << 7;
                for (int i = 0; i < oz::kSlices; i++) {
                    const int nj = i == 0 ? 8 : 8 - i;
                    const int n = (nj * D::NP2 + 15) & ~15;
                    for (int ks = 0; ks < 2; ks++)
                        for (int n0 = 0; n0 < n; n0 += 256) {
                            const int nn = n - n0 < 256 ? n - n0 : 256;
                            umma::mma_bf16(tmem + D::T_RES + i * D::NP2 + n0,
                                           umma::smem_desc(as + i * D::A2S + ks * 256, 128, sbo),
                                           umma::smem_desc(bs + (uint32_t)(n0 >> 3) * sbo + ks * 256, 128, sbo), idesc_f16(nn),
                                           first && i + ks == 0 ? 0u : 1u);
                        }
                }
            };
            uint32_t phA = 0, phTR = 0, phW = 0, phR = 0;
            for (int tile = blockIdx.x; tile < ntiles && !*dead; tile += gridDim.x) {
                wait(bAready, phA);
                phA ^= 1;
                uint32_t b = take();
                if (*dead) break;
                umma::fence_after_sync();
                product(tmem + D::T_OWN, umma::smem_u32(A1), D::A1S, K1, b, 32);
                done();
                b = take();
                if (*dead) break;
                product(tmem + D::T_NBR, umma::smem_u32(A2), D::A2S, 32, b, 32);
                umma::commit(bTrFull);
                done();
                wait(bTrRead, phTR);
                phTR ^= 1;
                b = take();
                if (*dead) break;
                umma::fence_after_sync();
                product(tmem + D::T_CUB, umma::smem_u32(A1), D::A1S, K1, b, 16);
                umma::commit(bD1full);
                done();
                wait(bA2w, phW);
                phW ^= 1;
                b = take();
                if (*dead) break;
                umma::fence_after_sync();
                product2(b, true);
                umma::commit(bA2free);
                done();
                for (int c = 0; c < D::NC; c++) {
                    wait(bD1read, phR);
                    phR ^= 1;
                    if (c + 1 < D::NC) {
                        b = take();
                        if (*dead) break;
                        umma::fence_after_sync();
                        product(tmem + D::T_CUB, umma::smem_u32(A1), D::A1S, K1, b, 16);
                        umma::commit(bD1full);
                        done();
                    }
                    wait(bA2w, phW);
                    phW ^= 1;
                    b = take();
                    if (*dead) break;
                    umma::fence_after_sync();
                    product2(b, false);
                    umma::commit(bA2free);
                    done();
                }
            }
            // everything issued ends before the CTA does
            umma::commit(bFin);
            umma::mbar_wait(bFin, 0, kWaitLimit);
            if (*dead) {
                for (long long n = nuse; n < nload; n++)
                    umma::mbar_wait(bFull + (int)(n % D::NSLOT), (uint32_t)((n / D::NSLOT) & 1), kWaitLimit);
                *reinterpret_cast<volatile int*>(oa.status) = 1;
                __threadfence_system();
            }
        }
        __syncwarp();
    } else {
        // -------------------------------------------------------------- compute warps
        const int sub = warp & 3, cg = warp >> 2, t = cg * 32 + lane;  // t: thread within the element group
        const int el = lane & 7, jv = lane >> 3;                       // element of the group; variable, then point
        const int e = 8 * sub + el;
        const uint32_t tlane = tmem + ((uint32_t)(32 * sub) << 16);
        const int ebV = ebS[D::NP2], ebI = ebS[D::NP2 + 1];
        const double g1 = a.gamma - 1.0;
        const float g1f = fabsf((float)g1);
        uint32_t phT = 0, phD = 0, phF = 0;
        auto waitw = [&](uint64_t* bar, uint32_t phase) {
            wait(bar, phase);
            __syncwarp();
        };
        auto arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(bar);
        };
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int k0 = tile * 32;
            const int gk0 = k0 + 8 * sub;  // the group's elements
            // ---- 1. geometry, digits of the nodal rows
            if (t < 24) {
                const int e8 = t / 3, f = t - 3 * e8, k = min(gk0 + e8, a.K - 1);
                const double* gk = a.geo + (size_t)k * 4;
                double* nr = nrmS + (8 * sub + e8) * 9 + f * 3;
                face_normal(f, gk[0], gk[1], gk[2], gk[3], nr[0], nr[1], nr[2]);
                connS[(8 * sub + e8) * 3 + f] = a.conn[(size_t)k * 3 + f];
            } else if (t >= 32 && t < 64) {
                const int i = t - 32;
                geoS[sub * 32 + i] = a.geo[(size_t)min(gk0 + (i >> 2), a.K - 1) * 4 + (i & 3)];
            } else if (t >= 64 && t < 96) {
                maxf[sub * 32 + t - 64] = 0u;
            } else if (t == 96) {
                flagS[sub] = 0u;
            }
            constexpr int LPR = D::LPR, RPW = 32 / LPR;  // rows per warp pass
#pragma unroll
            for (int pass = 0; pass < 8 / RPW; pass++) {
                const int i = pass * RPW + lane / LPR, kb = lane % LPR, v = cg;
                const bool in = gk0 + i < a.K;
                const double* src = a.qin + ((size_t)(gk0 + i) * 4 + v) * Np + 8 * kb;
                double x[8];
                uint32_t mx = 0;
                int mn = 0x7FF00000;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    x[j] = 0.0;
                    if (in && 8 * kb + j < Np) {
                        x[j] = src[j];
                        mn = min(mn, __double2hiint(x[j]));
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) mx = max(mx, oz::mag_hi(x[j]));
#pragma unroll
                for (int o = 1; o < LPR; o <<= 1) {
                    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                }
                const int eb = oz::row_bound(mx);
                if (kb == 0) {
                    maxq[(8 * sub + i) * 4 + v] = mx;
                    if (v == 0) minr[8 * sub + i] = mn;
                }
                if (kb < D::KB1) {
                    uint64_t y[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) y[j] = oz::biased(x[j], eb);
                    unsigned char* dst = A1 + (((4 * sub + v) * D::KB1 + kb) << 7) + (i << 4);
#pragma unroll
                    for (int s = 0; s < oz::kSlices; s++)
                        *reinterpret_cast<uint4*>(dst + s * D::A1S) =
                            make_uint4(oz::digit_pair(y[0], y[1], s), oz::digit_pair(y[2], y[3], s),
                                       oz::digit_pair(y[4], y[5], s), oz::digit_pair(y[6], y[7], s));
                }
            }
            group_sync(sub);
            {   // neighbour traces: 4 lanes per row, 8 face nodes each
                const int i = lane >> 2, kb = lane & 3, v = cg;
                const bool in = gk0 + i < a.K;
                double x[8];
                uint32_t mx = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int k = 8 * kb + j, f = k / Nfp, jn = k - f * Nfp;
                    x[j] = 0.0;
                    if (in && k < D::NT) {
                        const int c = connS[(8 * sub + i) * 3 + f];
                        if (c >= 0) {
                            const int fn = c & 3, jj = ((c >> 2) & 1) ? (N - jn) : jn;
                            int pos = fn * N + jj;
                            if (pos >= NB) pos -= NB;
                            x[j] = a.qin[((size_t)(c >> 3) * 4 + v) * Np + pos];
                        } else {
                            x[j] = a.btrace[((size_t)(-1 - c) * 4 + v) * Nfp + jn];
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) mx = max(mx, oz::mag_hi(x[j]));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const int eb = oz::row_bound(mx);
                if (kb == 0) {
                    e3S[(8 * sub + i) * 4 + v] = eb;
                    if (!oz::row_ok(mx) || !oz::row_ok(maxq[(8 * sub + i) * 4 + v])) atomicOr(flagS + sub, 1u << i);
                }
                uint64_t y[8];
#pragma unroll
                for (int j = 0; j < 8; j++) y[j] = oz::biased(x[j], eb);
                unsigned char* dst = A2 + (((4 * sub + v) * 4 + kb) << 7) + (i << 4);
#pragma unroll
                for (int s = 0; s < oz::kSlices; s++)
                    *reinterpret_cast<uint4*>(dst + s * D::A2S) =
                        make_uint4(oz::digit_pair(y[0], y[1], s), oz::digit_pair(y[2], y[3], s),
                                   oz::digit_pair(y[4], y[5], s), oz::digit_pair(y[6], y[7], s));
            }
            umma::fence_async_smem();
            arrive(bAready);
            // a bound on the volume flux rows of element e from its nodal extremes (FP32)
            const bool live = k0 + e < a.K;
            const double rx = geoS[e * 4], sx = geoS[e * 4 + 1], ry = geoS[e * 4 + 2], sy = geoS[e * 4 + 3];
            float est[4];
            {
                auto up = [](uint32_t h) { return oz::trunc32(__hiloint2double((int)h, -1)); };
                const float rmax = up(maxq[e * 4]), m = up(maxq[e * 4 + 1]), n = up(maxq[e * 4 + 2]),
                            E = up(maxq[e * 4 + 3]);
                const float ir = __fdividef(1.f, fmaxf(oz::trunc32(__hiloint2double(minr[e], 0)), 1e-3f * rmax));
                const float frx = fabsf(oz::trunc32(rx)), fry = fabsf(oz::trunc32(ry)), fsx = fabsf(oz::trunc32(sx)),
                            fsy = fabsf(oz::trunc32(sy));
                const float Mr = frx * m + fry * n, Ms = fsx * m + fsy * n, M = fmaxf(Mr, Ms);
                const float p = g1f * E;
                est[0] = M;
                est[1] = M * (m * ir) + fmaxf(frx, fsx) * p;
                est[2] = M * (n * ir) + fmaxf(fry, fsy) * p;
                est[3] = M * ((E + p) * ir);
            }
            // ---- 2. face fluxes
            waitw(bTrFull, phT);
            phT ^= 1;
            umma::fence_after_sync();
            const int ownrow = e * 4 + jv;
            const int eb1 = oz::row_bound(maxq[ownrow]);
            constexpr int GR = (D::NG4 + 3) / 4;  // rounds of 4-point groups per warp
            double qm[GR][4], qp[GR][4];
#pragma unroll
            for (int r = 0; r < GR; r++) {
                const int gi = cg + 4 * r;
                if (gi < D::NG4) {
                    load7<32>(tlane + D::T_OWN + 4 * gi, eb1 + ebI, qm[r]);
                    load7<32>(tlane + D::T_NBR + 4 * gi, e3S[ownrow] + ebI, qp[r]);
                }
            }
            umma::fence_before_sync();
            arrive(bTrRead);
#pragma unroll
            for (int r = 0; r < GR; r++)
                if (cg + 4 * r < D::NG4) {
                    transpose4(qm[r], lane);
                    transpose4(qp[r], lane);
                }
            uint32_t bad = 0;
            double F[GR][4];
            if (a.flux == 1) {
#pragma unroll
                for (int r = 0; r < GR; r++) {
                    const int pt = 4 * (cg + 4 * r) + jv;
                    if (cg + 4 * r < D::NG4) {
                        const int f = min(pt, NF - 1) / Nfq;
                        const double* nr = nrmS + e * 9 + f * 3;
                        roe_flux_fast(g1, nr[0], nr[1], qm[r], qp[r], F[r]);
#pragma unroll
                        for (int v = 0; v < 4; v++) F[r][v] = pt < NF && live ? nr[2] * F[r][v] : 0.0;
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < GR; r++) {
                    const int pt = 4 * (cg + 4 * r) + jv;
                    if (cg + 4 * r < D::NG4) {
                        const int f = min(pt, NF - 1) / Nfq;
                        const double nx = nrmS[e * 9 + f * 3], ny = nrmS[e * 9 + f * 3 + 1];
                        const FaceSide m = face_side(g1, nx, ny, qm[r]), p = face_side(g1, nx, ny, qp[r]);
                        const double um = m.mn * m.r, up = p.mn * p.r;
                        const double wm = fabs(um) + oz::sqrt64(fabs(a.gamma * m.p * m.r));
                        const double wp = fabs(up) + oz::sqrt64(fabs(a.gamma * p.p * p.r));
                        // magnitudes compare as integers (a NaN is the largest)
                        const long long wmi = __double_as_longlong(wm) & 0x7FFFFFFFFFFFFFFFll,
                                        wpi = __double_as_longlong(wp) & 0x7FFFFFFFFFFFFFFFll;
                        if (pt < NF) lamS[e * NF + pt] = __longlong_as_double(wmi > wpi ? wmi : wpi);
                        F[r][0] = m.mn + p.mn;
                        F[r][1] = fma(qm[r][1], um, fma(qp[r][1], up, nx * (m.p + p.p)));
                        F[r][2] = fma(qm[r][2], um, fma(qp[r][2], up, ny * (m.p + p.p)));
                        F[r][3] = fma(qm[r][3] + m.p, um, (qp[r][3] + p.p) * up);
                    }
                }
                group_sync(sub);
#pragma unroll
                for (int r = 0; r < GR; r++) {
                    const int pt = 4 * (cg + 4 * r) + jv;
                    if (cg + 4 * r < D::NG4) {
                        const int f = min(pt, NF - 1) / Nfq;
                        long long l = 0;
#pragma unroll
                        for (int i = 0; i < Nfq; i++) {
                            const long long w = __double_as_longlong(lamS[e * NF + f * Nfq + i]);
                            l = w > l ? w : l;
                        }
                        const double lam = __longlong_as_double(l), h = 0.5 * nrmS[e * 9 + f * 3 + 2];
#pragma unroll
                        for (int v = 0; v < 4; v++)
                            F[r][v] = pt < NF && live ? h * fma(lam, qm[r][v] - qp[r][v], F[r][v]) : 0.0;
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < GR; r++)
                if (cg + 4 * r < D::NG4) {
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const uint32_t h = oz::mag_hi(F[r][v]);
                        if (h >= 0x7FF00000u) bad = 1u;
                        else atomicMax(maxf + e * 4 + v, h);
                    }
                }
            if (bad) atomicOr(flagS + sub, 1u << el);
            group_sync(sub);
            int eb2[4];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                // one bit above the estimate for points between the nodes
                const float b = fminf(2.f * est[v], 1e38f);
                const int ee = b > 0.f ? (int)(__float_as_uint(b) >> 23) - 127 + 1 + 1022 : 0;
                eb2[v] = max(oz::row_bound(maxf[e * 4 + v]), ee);
                if (eb2[v] > 1700 || (eb2[v] != 0 && eb2[v] < 300)) bad = 1u;
            }
#pragma unroll
            for (int r = 0; r < GR; r++) {
                const int gi = cg + 4 * r, pt = 4 * gi + jv;
                if (gi < D::NG4) {
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const uint64_t y = oz::biased(F[r][v], eb2[v]);
                        unsigned char* dst = A2 + (((4 * sub + v) * 4 + (pt >> 3)) << 7) + (el << 4) + ((pt & 7) << 1);
#pragma unroll
                        for (int s = 0; s < oz::kSlices; s++)
                            *reinterpret_cast<uint16_t*>(dst + s * D::A2S) = (uint16_t)oz::digit_pair(y, y, s);
                    }
                }
            }
            umma::fence_async_smem();
            arrive(bA2w);
            // ---- 3. volume fluxes, 16 cubature points per chunk
            for (int c = 0; c < D::NC; c++) {
                const int p0 = 16 * c + 4 * cg, pt = p0 + jv;
                waitw(bD1full, phD);
                phD ^= 1;
                umma::fence_after_sync();
                double q[4];
                if (p0 < Ng) load7<16>(tlane + D::T_CUB + 4 * cg, eb1 + ebV, q);
                umma::fence_before_sync();
                arrive(bD1read);
                uint64_t yr[4], ys[4];
                if (p0 < Ng) {
                    transpose4(q, lane);
                    const double r = oz::rcp64(q[0]);
                    const double u = q[1] * r, v = q[2] * r;
                    const double p = g1 * fma(-0.5, fma(q[1], u, q[2] * v), q[3]);
                    const double H = (q[3] + p) * r;
                    const double Mr = fma(rx, q[1], ry * q[2]), Ms = fma(sx, q[1], sy * q[2]);
                    double Fr[4] = {Mr, fma(Mr, u, rx * p), fma(Mr, v, ry * p), Mr * H};
                    double Fs[4] = {Ms, fma(Ms, u, sx * p), fma(Ms, v, sy * p), Ms * H};
                    const bool ok = live && pt < Ng;
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        if (!ok) Fr[w] = Fs[w] = 0.0;
                        const uint32_t h = max(oz::mag_hi(Fr[w]), oz::mag_hi(Fs[w]));
                        if (oz::row_bound(h) > eb2[w]) bad = 1u;
                        yr[w] = oz::biased(Fr[w], eb2[w]);
                        ys[w] = oz::biased(Fs[w], eb2[w]);
                    }
                }
                waitw(bA2free, phF);  // the previous product has read the operand
                phF ^= 1;
                if (p0 < Ng) {
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        unsigned char* dst = A2 + (((4 * sub + w) * 4 + cg) << 7) + (el << 4) + (jv << 2);
#pragma unroll
                        for (int s = 0; s < oz::kSlices; s++)
                            *reinterpret_cast<uint32_t*>(dst + s * D::A2S) = oz::digit_pair(yr[w], ys[w], s);
                    }
                }
                umma::fence_async_smem();
                arrive(bA2w);
            }
            if (bad) atomicOr(flagS + sub, 1u << el);
            // ---- 4. result rows
            waitw(bA2free, phF);
            phF ^= 1;
            umma::fence_after_sync();
            int ebr = 0;
#pragma unroll
            for (int v = 0; v < 4; v++) ebr = jv == v ? eb2[v] : ebr;
            auto R = [&](int i) { return striped(A2, sub, i, D::A2S, 2048); };
#pragma unroll
            for (int n0 = 0; n0 < D::NP2; n0 += 16) {
                const int n4 = n0 + 4 * cg;
                if (n4 < Np) {
                    float d[8][4];
#pragma unroll
                    for (int s = 0; s < 8; s++) umma::tmem_ld4(tlane + D::T_RES + s * D::NP2 + n4, d[s]);
                    umma::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (n4 + j < Np) {
                            int ds[8];
#pragma unroll
                            for (int s = 0; s < 8; s++) ds[s] = oz::acc_int24(d[s][j]);
                            *R((el * 4 + jv) * Np + n4 + j) = oz::combine8(ds, ebr + ebS[n4 + j]);
                        }
                }
            }
            umma::fence_before_sync();
            group_sync(sub);
            for (uint32_t fl = flagS[sub]; fl; fl &= fl - 1) {
                const int i = __ffs((int)fl) - 1;
                if (gk0 + i < a.K)
                    plain_element<N>(a, gk0 + i, t, sub,
                                     [&](int j) { return striped(A1, sub, j, D::A1S, 32 * K1 * 2); },
                                     [&](int j) { return R(i * 4 * Np + j); });
            }
            const int nval = max(0, min(8, a.K - gk0)) * 4 * Np;
            for (int i = t; i < nval; i += 128) {
                const double Rv = *R(i);
                const size_t idx = (size_t)gk0 * 4 * Np + i;
                const double dt = a.dtk ? a.dt * a.dtk[gk0 + i / (4 * Np)] : a.dt;
                switch (a.mode) {
                    case MODE_RHS: a.rhs[idx] = Rv; break;
                    case MODE_LSERK: {
                        const double r = a.rka * a.res[idx] + dt * Rv;
                        a.res[idx] = r;
                        a.qout[idx] = a.qin[idx] + a.rkb * r;
                    } break;
                    case MODE_EULER: a.qout[idx] = a.qin[idx] + dt * Rv; break;
                    default: a.qout[idx] = 0.5 * a.qold[idx] + 0.5 * (a.qin[idx] + dt * Rv); break;
                }
            }
            group_sync(sub);  // staging, flags and geometry are rewritten by the next tile
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 16) {
        umma::fence_after_sync();
        umma::tmem_relinquish();
        umma::tmem_dealloc(tmem, 512);
    }
}

template <int N>
static cudaError_t setup_tc(const dgb::RefOps& ops, OzPlan& plan) {
    const OzImage im = oz_build<N>(ops);
    if (!im.exact) return cudaSuccess;  // not representable: the plain kernel stays
    cudaError_t e = cudaFuncSetAttribute(euler_stage_fp64_tc_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         OzDims<N>::SMEM);
    int dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&plan.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaHostAlloc((void**)&plan.h_status, sizeof(int), cudaHostAllocMapped);
    if (e == cudaSuccess) {
        *plan.h_status = 0;
        e = cudaHostGetDevicePointer((void**)&plan.status, plan.h_status, 0);
    }
    if (e == cudaSuccess) e = cudaMalloc(&plan.d_image, im.bytes.size() + im.eb.size() * sizeof(int));
    if (e != cudaSuccess) return e;
    plan.d_eb = reinterpret_cast<int*>((unsigned char*)plan.d_image + im.bytes.size());
    e = cudaMemcpy(plan.d_image, im.bytes.data(), im.bytes.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(plan.d_eb, im.eb.data(), im.eb.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) plan.ready = true;
    return e;
}

cudaError_t setup_euler_fp64_tc(int N, const dgb::RefOps& ops, OzPlan& plan) {
    switch (N) {
        case 1: return setup_tc<1>(ops, plan);
        case 2: return setup_tc<2>(ops, plan);
        case 3: return setup_tc<3>(ops, plan);
        case 4: return setup_tc<4>(ops, plan);
        case 5: return setup_tc<5>(ops, plan);
        case 6: return setup_tc<6>(ops, plan);
        case 7: return setup_tc<7>(ops, plan);
        default: return cudaErrorInvalidValue;
    }
}

void teardown_euler_fp64_tc(OzPlan& plan) {
    if (plan.d_image) cudaFree(plan.d_image);
    if (plan.h_status) cudaFreeHost(plan.h_status);
    plan = OzPlan();
}

template <int N>
static cudaError_t launch_tc(const OzArgs& oa, const OzPlan& plan, cudaStream_t s) {
    const int ntiles = (oa.e.K + 31) / 32;
    euler_stage_fp64_tc_kernel<N><<<std::min(ntiles, plan.sms), kOzThreads, OzDims<N>::SMEM, s>>>(oa);
    return cudaGetLastError();
}

cudaError_t launch_euler_fp64_tc(int N, const EulerArgs& a, const OzPlan& plan, cudaStream_t s) {
    const OzArgs oa{a, (const unsigned char*)plan.d_image, plan.d_eb, plan.status};
    switch (N) {
        case 1: return launch_tc<1>(oa, plan, s);
        case 2: return launch_tc<2>(oa, plan, s);
        case 3: return launch_tc<3>(oa, plan, s);
        case 4: return launch_tc<4>(oa, plan, s);
        case 5: return launch_tc<5>(oa, plan, s);
        case 6: return launch_tc<6>(oa, plan, s);
        case 7: return launch_tc<7>(oa, plan, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace dgk
