// euler_fp64_tc.cu -- FP64 Euler stage with its contractions on the tensor
// cores (sm_103a).
//
// GB300 retires two FP64 operations per clock per SM, and of the ~21,000 an
// element needs per stage at N = 5 the contractions (interpolation to the
// cubature and face points, weak derivative, lift) are 18,400.  Here those
// run as exact integer products on tcgen05 (ozaki.cuh: seven base-256
// digits per value, FP16 operands, FP32 accumulators that hold exact
// integers), with an error against extended precision no larger than the FMA
// chain's (kFluxSlack); the FP64 pipe keeps the point-wise fluxes (25 operations per cubature point with
// reciprocals from FP32 seeds) and the Runge-Kutta update.
//
// One CTA per SM walks tiles of 32 elements (128 operand rows).  Warps
// 0-15 compute: warp w owns the eight elements 8 (w % 4) .. + 7, the ones
// whose tensor-memory lanes it can read, and quarter w / 4 of the points, so
// only the four warps of one such group ever wait for each other (named
// barriers); warp 16 feeds the tensor core (operator pieces arrive by bulk
// copies in a ring, consumed in a fixed order) and all hand-overs are
// mbarriers.  Per tile:
//   1. own nodes and neighbour face nodes -> digit operands;
//   2. traces at the face points (two products), numerical flux, digits;
//   3. per chunk of 16 cubature points: state at the points (product),
//      fluxes, digits, product into the result accumulators;
//   4. result rows -> FP64, stage update.
// The metrics carry the element's time step, so the results are dt R.
// The digits of a row share one exponent.  For the nodal rows it is the row's
// own (for neighbour traces each face's own); for the flux rows it comes from the
// face fluxes and from the volume fluxes at the nodes, in FP32, doubled.  An element
// whose fluxes leave that bound or stay too far below it, whose density or
// energy varies too much (kFluxSlack, kRhoDepth, kEnergyDepth), or with values that
// are not finite or outside the FP32 exponent range, is left to plain FP64 after the
// tiles, as euler_fp64.cu does it (plain_elements).  All of this is per element:
// results do not depend on an element's place in the mesh.
//
// Measured, LSERK4 stage in a queue of steps, against the kernel of euler_fp64.cu: K = 32768,
// N = 5, LF 2.66 ms -> 399 us; K = 9794, N = 7, Roe 2.62 ms -> 197 us;
// K = 3200, N = 3, LF 78 -> 26 us; so it is taken at every order and size.
// What bounds it now: the FP64 pipe is busy half of the time (58,000 of
// 117,000 cycles per tile at N = 5: 25,000 in the face fluxes, 30,000 in the
// volume fluxes); the four warps of a scheduler run their integer phases
// (digits, sums) in step, and the pipe idles through them.  Measured and left
// out: a second flux operand with the next tile's operands made during this
// tile's last product (400 us), the next chunk's sums interleaved with this
// chunk's fluxes (400 us), MMA issue in rolled loops (456 us: one thread
// issues them, and at 100 cycles an MMA the products fell behind).
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

// What an element may lose to the common exponents of its rows, in bits; beyond, it
// is left to plain FP64.  A value is cut at 2^-56 of its row's bound, FP64 arithmetic rounds
// at 2^-53 of the value.  kFluxSlack: how far the bound of a flux row may lie above
// the largest flux that it held.  kRhoDepth, kEnergyDepth: how far a density or an
// energy at a point may lie below the row's largest nodal value.  With these, the
// error of the right-hand side against extended precision has, over random elements of
// one kind, a median of 0.5 to 1.1 of the plain kernel's (N = 1 .. 7, both fluxes, density,
// pressure or velocity varying by 1.5, 10, 25, 100 and 900 inside an element, neighbours up
// to 900 times apart), and single elements no more than twice its.  Densities 25 times
// below, without that limit: twice the error in an ill-conditioned element at N = 7; 100 times: 1.3 as
// the median at N = 4.  The exponent from products of nodal extremes in place of nodal fluxes,
// which this kernel used before: 2.5 at contrast 10, 20 at 100, 200 at 900.
constexpr int kFluxSlack = 3, kRhoDepth = 4, kEnergyDepth = 9;

struct OzArgs {
    EulerArgs e;
    const unsigned char* image;
    const int* eb;
    int* status;
    unsigned char* flags;  // per group of 8 elements, those left to plain FP64
    int groups;            // groups of 8 elements per tile, 1 .. 4
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

// waits for the columns requested into d; their uses stay behind the wait
// because the values pass through it
template <int R>
__device__ __forceinline__ void arrived(float (&d)[R][4]) {
    umma::tmem_ld_wait();
#pragma unroll
    for (int s = 0; s < R; s++) asm volatile("" : "+f"(d[s][0]), "+f"(d[s][1]), "+f"(d[s][2]), "+f"(d[s][3]));
}

// four consecutive columns of eight digit groups (stride P) -> FP64 values
// of the lane's row; ebab(c): the bounds of both rows added
template <int P, typename E>
__device__ __forceinline__ void load8(uint32_t taddr, E ebab, double x[4]) {
    float d[8][4];
#pragma unroll
    for (int s = 0; s < 8; s++) umma::tmem_ld4(taddr + s * P, d[s]);
    arrived(d);
#pragma unroll
    for (int c = 0; c < 4; c++)
        x[c] = oz::combine_nodal(oz::acc_int22(d[0][c]), oz::acc_int22(d[1][c]), oz::acc_int22(d[2][c]), oz::acc_int22(d[3][c]),
                                 oz::acc_int22(d[4][c]), oz::acc_int22(d[5][c]), oz::acc_int22(d[6][c]), oz::acc_int22(d[7][c]),
                                 ebab(c));
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

// bounded wait on an mbarrier phase
__device__ __forceinline__ bool bounded_wait(uint64_t* bar, uint32_t phase) {
    uint32_t left;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mov.u32 %0, %3;\n\t"
        "OZ_POLL:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra OZ_DONE;\n\t"
        "sub.u32 %0, %0, 1;\n\t"
        "setp.ne.u32 p, %0, 0;\n\t"
        "@p bra OZ_POLL;\n\t"
        "OZ_DONE:\n\t}"
        : "=&r"(left)
        : "r"(umma::smem_u32(bar)), "r"(phase), "n"(kWaitLimit)
        : "memory");
    return left != 0u;
}

__device__ __forceinline__ void group_sync(int sub) { asm volatile("bar.sync %0, 128;" ::"r"(sub + 1) : "memory"); }

// One operator piece: operand slices at `as` (AS bytes apart, reduction KP)
// times the piece's digit blocks of P rows, digit pairs i + j = s <= 7 into columns
// d + P s (the zero block 7 of the operator starts every group).  Unrolled: one
// thread issues every MMA, and their rate is the piece's latency.
template <int AS, int KP, int P>
__device__ __forceinline__ void digit_product(uint32_t d, uint32_t as, uint32_t bs, bool start) {
    constexpr uint32_t SBO = (uint32_t)(KP / 8) << 7;
    const uint64_t ad = umma::smem_desc(as, 128, SBO), bd = umma::smem_desc(bs, 128, SBO);
#pragma unroll
    for (int i = 0; i < oz::kSlices; i++) {
        const int n = ((oz::kSlices + 1 - i) * P + 15) & ~15;
#pragma unroll
        for (int ks = 0; ks < KP / 16; ks++)
#pragma unroll
            for (int n0 = 0; n0 < n; n0 += 256)
                umma::mma_bf16(d + i * P + n0, ad + (uint32_t)((i * AS + ks * 256) >> 4),
                               bd + (uint32_t)(((n0 >> 3) * SBO + ks * 256) >> 4), idesc_f16(n - n0 < 256 ? n - n0 : 256),
                               i + ks > 0 || !start ? 1u : 0u);
    }
}

// place of scratch value i of element group `sub` in an operand whose slices
// are `stride` bytes and hold `per` bytes of the group's rows each
__device__ __forceinline__ double* striped(unsigned char* base, int sub, int i, int stride, int per) {
    const int n = per >> 3, s = i / n;
    return reinterpret_cast<double*>(base + (size_t)s * stride + (size_t)sub * per) + (i - s * n);
}

// factor of the fluxes: the element's time step (1 for a right-hand side)
__device__ __forceinline__ double step_of(const EulerArgs& a, int k) {
    return a.mode == MODE_RHS ? 1.0 : a.dtk ? a.dt * a.dtk[k] : a.dt;
}

// the stage's update of one value: right-hand side times the step, state q0,
// and the RK register or the old state o0
__device__ __forceinline__ void stage_update(const EulerArgs& a, size_t idx, double dR, double q0, double o0) {
    if (a.mode == MODE_RHS) {
        a.rhs[idx] = dR;
    } else if (a.mode == MODE_LSERK) {
        const double r = fma(a.rka, o0, dR);
        a.res[idx] = r;
        a.qout[idx] = fma(a.rkb, r, q0);
    } else if (a.mode == MODE_EULER) {
        a.qout[idx] = q0 + dR;
    } else {
        a.qout[idx] = 0.5 * (o0 + (q0 + dR));
    }
}

// Stage of nb <= D::PB elements of a group in plain FP64 by its 128 threads,
// operation for operation as euler_stage_fp64_kernel forms it; element b is
// gk0 + ((list >> 4 b) & 7), sc(i) scratch value i.  Several at once: at low orders one
// element leaves most threads idle.  With every element on this route (K = 32768,
// N = 1, 3, 5; K = 9800, N = 7, a right-hand side): 980, 1736, 3516, 3683 us one at a time with
// rolled loops, 398, 1020, 2293, 2098 so; euler_fp64.cu 168, 817, 2616, 2256.
template <int N, typename Sc>
__device__ __forceinline__ void plain_elements(const EulerArgs& a, int gk0, uint32_t list, int nb, int t, int sub, Sc sc) {
    using D = OzDims<N>;
    constexpr int Np = D::Np, Ng = D::Ng, Nfp = D::Nfp, Nfq = D::Nfq, NB = D::NB, NF = D::NF, SS = D::PLAIN_SCRATCH;
    const double gamma = a.gamma;
    auto element = [&](int b) { return gk0 + (int)((list >> (4 * b)) & 7u); };
#pragma unroll 1
    for (int it = t; it < nb * Ng; it += 128) {
        const int b = it / Ng, g = it - b * Ng, k = element(b);
        const double *qe = a.qin + (size_t)k * 4 * Np, *gk = a.geo + (size_t)k * 4;
        double q[4] = {0, 0, 0, 0}, fx[4], fy[4];
#pragma unroll 3
        for (int p = 0; p < Np; p++) {
            const double w = __ldg(a.ops.Vg + g * Np + p);
#pragma unroll
            for (int v = 0; v < 4; v++) q[v] += w * __ldg(qe + v * Np + p);
        }
        euler_phys_flux(gamma, q, fx, fy);
        const double rx = gk[0], sx = gk[1], ry = gk[2], sy = gk[3];
#pragma unroll
        for (int v = 0; v < 4; v++) {
            *sc(b * SS + v * Ng + g) = rx * fx[v] + ry * fy[v];
            *sc(b * SS + (4 + v) * Ng + g) = sx * fx[v] + sy * fy[v];
        }
    }
    // face fluxes, a thread a point; the wave speeds of a face meet in the scratch
    const int b = t / NF, fq = t - b * NF, f = fq / Nfq, i = fq - f * Nfq;
    const bool face = t < nb * NF;
    double nx = 0, ny = 0, fsc = 0, qm[4] = {0, 0, 0, 0}, qp[4] = {0, 0, 0, 0};
    if (face) {
        const int k = element(b), c = a.conn[(size_t)k * 3 + f];
        const double *qe = a.qin + (size_t)k * 4 * Np, *gk = a.geo + (size_t)k * 4;
        face_normal(f, gk[0], gk[1], gk[2], gk[3], nx, ny, fsc);
        const int fn = c & 3;
        const bool turned = (c >> 2) & 1;
        const double* qn = c >= 0 ? a.qin + (size_t)(c >> 3) * 4 * Np : a.btrace + (size_t)(-1 - c) * 4 * Nfp;
        const int stride = c >= 0 ? Np : Nfp;
#pragma unroll 2
        for (int j = 0; j < Nfp; j++) {
            const double w = __ldg(a.ops.If + i * Nfp + j);
            const int own = (f * N + j) % NB, other = c >= 0 ? (fn * N + (turned ? N - j : j)) % NB : j;
#pragma unroll
            for (int v = 0; v < 4; v++) {
                qm[v] += w * __ldg(qe + v * Np + own);
                qp[v] += w * __ldg(qn + v * stride + other);
            }
        }
        if (a.flux != 1) *sc(b * SS + 8 * Ng + 4 * NF + fq) = fmax(wave_speed(gamma, nx, ny, qm), wave_speed(gamma, nx, ny, qp));
    }
    if (a.flux != 1) group_sync(sub);
    if (face) {
        double F[4], lam = 0;
        if (a.flux == 1) {
            roe_flux(gamma, nx, ny, qm, qp, F);
        } else {
#pragma unroll 1
            for (int j = 0; j < Nfq; j++) lam = fmax(lam, *sc(b * SS + 8 * Ng + 4 * NF + f * Nfq + j));
            lf_flux(gamma, nx, ny, lam, qm, qp, F);
        }
#pragma unroll
        for (int v = 0; v < 4; v++) *sc(b * SS + 8 * Ng + v * NF + fq) = fsc * F[v];
    }
    group_sync(sub);
#pragma unroll 1
    for (int it = t; it < nb * 4 * Np; it += 128) {
        const int b = it / (4 * Np), r = it - b * 4 * Np, v = r / Np, p = r - v * Np, k = element(b);
        double acc = 0, acc2 = 0, accf = 0;
#pragma unroll 4
        for (int g = 0; g < Ng; g++) {
            acc += __ldg(a.ops.Sr + p * Ng + g) * *sc(b * SS + v * Ng + g);
            acc2 += __ldg(a.ops.Ss + p * Ng + g) * *sc(b * SS + (4 + v) * Ng + g);
        }
        acc += acc2;
#pragma unroll 3
        for (int q = 0; q < NF; q++) accf += __ldg(a.ops.Lift + p * NF + q) * *sc(b * SS + 8 * Ng + v * NF + q);
        const size_t idx = (size_t)k * 4 * Np + r;
        stage_update(a, idx, step_of(a, k) * (acc - accf), a.qin[idx],
                     a.mode == MODE_LSERK ? a.res[idx] : a.mode == MODE_SSP2 ? a.qold[idx] : 0.0);
    }
    group_sync(sub);
}

// The elements of the block's tiles that are left to plain FP64 (none, as a rule), by one
// group's threads.  The group's flags are thread 0's stores, the last tile's with no
// barrier behind it yet: every thread must read the same, since plain_elements has the
// group's barriers inside.  A call, after the tiles, so that it costs their loop no registers.
template <int N>
__device__ __noinline__ void plain_pass(const OzArgs& oa, unsigned char* smem, int t, int sub) {
    using D = OzDims<N>;
    const int tile_elems = 8 * oa.groups, K = oa.e.K;
    group_sync(sub);
    for (int k0 = (int)blockIdx.x * tile_elems; k0 < K; k0 += (int)gridDim.x * tile_elems) {
        const int gk0 = k0 + 8 * sub;
        uint32_t fl = oa.flags[gk0 >> 3] & ((1u << max(0, min(8, K - gk0))) - 1u);
        while (fl) {
            uint32_t list = 0;
            int nb = 0;
            for (; fl && nb < D::PB; fl &= fl - 1) list |= (uint32_t)(__ffs((int)fl) - 1) << (4 * nb++);
            plain_elements<N>(oa.e, gk0, list, nb, t, sub, [&](int j) {
                return j < D::A1_SCRATCH ? striped(smem + D::OFF_A1, sub, j, D::A1S, 32 * D::K1 * 2)
                                         : striped(smem + D::OFF_A2, sub, j - D::A1_SCRATCH, D::A2S, 2048);
            });
        }
    }
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
    uint32_t* h3S = reinterpret_cast<uint32_t*>(smem + D::OFF_H3);
    uint32_t* estS = reinterpret_cast<uint32_t*>(smem + D::OFF_EST);
    uint32_t* maxf = reinterpret_cast<uint32_t*>(smem + D::OFF_MAXF);
    uint32_t* flagS = reinterpret_cast<uint32_t*>(smem + D::OFF_FLAG);
    uint32_t* reachS = reinterpret_cast<uint32_t*>(smem + D::OFF_REACH);
    int* ebS = reinterpret_cast<int*>(smem + D::OFF_EB);
    volatile int* dead = reinterpret_cast<volatile int*>(smem + D::OFF_DEAD);
    uint32_t* tmemS = reinterpret_cast<uint32_t*>(smem + D::OFF_TMEM);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + D::OFF_BAR);
    uint64_t *bOwn = bars, *bTrFull = bars + 1, *bTrRead = bars + 2, *bD1full = bars + 3, *bD1read = bars + 4,
             *bFin = bars + 5, *bA2w = bars + 6, *bA2free = bars + 7, *bFull = bars + 8, *bEmpty = bFull + D::NSLOT;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        umma::mbar_init(bOwn, 4 * oa.groups);
        umma::mbar_init(bTrFull, 1);
        umma::mbar_init(bTrRead, 4 * oa.groups);
        umma::mbar_init(bD1full, 1);
        umma::mbar_init(bD1read, 4 * oa.groups);
        umma::mbar_init(bFin, 1);
        umma::mbar_init(bA2w, 4 * oa.groups);
        umma::mbar_init(bA2free, 1);
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
    const int tile_elems = 8 * oa.groups, ntiles = (a.K + tile_elems - 1) / tile_elems;

    auto wait = [&](uint64_t* bar, uint32_t phase) {
        if (*dead) return;
        if (!bounded_wait(bar, phase)) *dead = 1;
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
                const uint32_t n = loadp == 0 ? D::B1F : loadp == 1 ? D::B3 : D::piece_flux(loadp) ? D::B2 : D::B1;
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
            const uint32_t a1 = umma::smem_u32(A1), a2 = umma::smem_u32(A2);
            uint32_t phO = 0, phTR = 0, phR = 0, phW = 0;
#pragma unroll 1
            for (int tile = blockIdx.x; tile < ntiles && !*dead; tile += gridDim.x)
#pragma unroll 1
                for (int p = 0; p < D::PIECES; p++) {
                    const bool last = p == D::PIECES - 1, flux = D::piece_flux(p);
                    if (p == 0) {
                        wait(bOwn, phO);
                        phO ^= 1;
                    } else if (p == 2) {
                        wait(bTrRead, phTR);
                        phTR ^= 1;
                    } else if (p > 3 && (!flux || last)) {
                        wait(bD1read, phR);
                        phR ^= 1;
                    }
                    if (flux || p == 1) {
                        wait(bA2w, phW);
                        phW ^= 1;
                    }
                    const uint32_t b = take();
                    if (*dead) break;
                    umma::fence_after_sync();
                    if (flux) digit_product<D::A2S, 32, D::NP2>(tmem + D::T_RES, a2, b, p == 3);
                    else if (p == 0) digit_product<D::A1S, K1, 32>(tmem + D::T_OWN, a1, b, true);
                    else if (p == 1) digit_product<D::A2S, 32, 32>(tmem + D::T_NBR, a2, b, true);
                    else digit_product<D::A1S, K1, 16>(tmem + D::T_CUB, a1, b, true);
                    if (flux || p == 1) umma::commit(bA2free);
                    if (p == 1) umma::commit(bTrFull);
                    else if (!flux && p > 1) umma::commit(bD1full);
                    done();
                }
            // everything issued ends before the CTA does
            umma::commit(bFin);
            if (!umma::mbar_wait(bFin, 0, kWaitLimit)) *dead = 1;
            if (*dead)
                for (long long n = nuse; n < nload; n++)
                    umma::mbar_wait(bFull + (int)(n % D::NSLOT), (uint32_t)((n / D::NSLOT) & 1), kWaitLimit);
        }
        __syncwarp();
    } else if ((warp & 3) < oa.groups) {
        // -------------------------------------------------------------- compute warps
        const int sub = warp & 3, cg = warp >> 2, t = cg * 32 + lane;  // t: thread within the element group
        const int el = lane & 7, jv = lane >> 3;                       // element of the group; variable, then point
        const int e = 8 * sub + el;
        const uint32_t tlane = tmem + ((uint32_t)(32 * sub) << 16);
        const int ebV = ebS[D::NP2], ebI = ebS[D::NP2 + 1];
        const double g1 = a.gamma - 1.0;
        const float g1f = (float)g1;
        constexpr int IT = (32 * Np + 127) / 128;
        uint32_t phT = 0, phD = 0;
        int use = 0;
        auto waitw = [&](uint64_t* bar, uint32_t phase) {
            wait(bar, phase);
            __syncwarp();
        };
        auto arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(bar);
        };
        // The second operand (neighbour traces, face fluxes, then each chunk's fluxes)
        // has one buffer: free once its last product is done, and handed over
        auto flux_free = [&]() {
            if (use) waitw(bA2free, (uint32_t)(use - 1) & 1u);
        };
        auto flux_written = [&]() {
            umma::fence_async_smem();
            arrive(bA2w);
            use++;
        };
#pragma unroll 1
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int gk0 = tile * tile_elems + 8 * sub;  // the group's elements
            const int nval = max(0, min(8, a.K - gk0)) * 4 * Np;
            const size_t g0 = (size_t)gk0 * 4 * Np;
            double q0[IT], o0[IT];
            int eb2[4];
            // ---- 1. geometry, digits of the nodal rows
            group_sync(sub);
            if (t < 24) {
                const int e8 = t / 3, f = t - 3 * e8, k = min(gk0 + e8, a.K - 1);
                const double* gk = a.geo + (size_t)k * 4;
                double* nr = nrmS + (8 * sub + e8) * 9 + f * 3;
                const double gx = f == 0 ? -gk[1] : f == 1 ? gk[0] + gk[1] : -gk[0];
                const double gy = f == 0 ? -gk[3] : f == 1 ? gk[2] + gk[3] : -gk[2];
                const double s2 = fma(gx, gx, gy * gy), is = oz::rsqrt64(s2);
                nr[0] = gx * is;
                nr[1] = gy * is;
                nr[2] = s2 * is * step_of(a, k);
                connS[(8 * sub + e8) * 3 + f] = a.conn[(size_t)k * 3 + f];
            } else if (t >= 32 && t < 64) {
                const int i = t - 32, k = min(gk0 + (i >> 2), a.K - 1);
                geoS[sub * 32 + i] = a.geo[(size_t)k * 4 + (i & 3)] * step_of(a, k);
            } else if (t >= 64 && t < 96) {
                maxf[sub * 32 + t - 64] = 0u;
            } else if (t == 96) {
                flagS[sub] = 0u;
                reachS[sub] = 0u;
            }
            constexpr int LPR = D::LPR, RPW = 32 / LPR;  // rows per warp pass
#pragma unroll 1
            for (int pass = 0; pass < 8 / RPW; pass++) {
                const int i = pass * RPW + lane / LPR, kb = lane % LPR, v = cg;
                const bool in = gk0 + i < a.K;
                const double* src = a.qin + ((size_t)(gk0 + i) * 4 + v) * Np + 8 * kb;
                double x[8];
                uint32_t mx = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) x[j] = in && 8 * kb + j < Np ? src[j] : 0.0;
#pragma unroll
                for (int j = 0; j < 8; j++) mx = max(mx, oz::mag_hi(x[j]));
#pragma unroll
                for (int o = 1; o < LPR; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const int eb = oz::row_bound(mx);
                if (kb == 0) maxq[(8 * sub + i) * 4 + v] = mx;
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
            umma::fence_async_smem();
            arrive(bOwn);
            group_sync(sub);
            {
                const int i = lane >> 2, kb = lane & 3, v = cg;  // neighbour traces: 4 lanes per row, 8 face nodes each
                const bool in = gk0 + i < a.K;
                double x[8];
                const double* src[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int k = 8 * kb + j, f = k / Nfp, jn = k - f * Nfp;
                    src[j] = nullptr;
                    if (in && k < D::NT) {
                        const int c = connS[(8 * sub + i) * 3 + f];
                        const int fn = c & 3, jj = ((c >> 2) & 1) ? (N - jn) : jn;
                        int pos = fn * N + jj;
                        if (pos >= NB) pos -= NB;
                        src[j] = c >= 0 ? a.qin + ((size_t)(c >> 3) * 4 + v) * Np + pos
                                        : a.btrace + ((size_t)(-1 - c) * 4 + v) * Nfp + jn;
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    x[j] = 0.0;
                    if (src[j]) x[j] = *src[j];
                }
                uint32_t mx[3] = {0, 0, 0};  // a face point takes its own face's nodes only: a bound per face
                flux_free();
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int f = (8 * kb + j) / Nfp;
                    const uint32_t h = oz::mag_hi(x[j]);
#pragma unroll
                    for (int g = 0; g < 3; g++) mx[g] = max(mx[g], f == g ? h : 0u);
                }
#pragma unroll
                for (int g = 0; g < 3; g++) {
                    mx[g] = max(mx[g], __shfl_xor_sync(0xffffffffu, mx[g], 1));
                    mx[g] = max(mx[g], __shfl_xor_sync(0xffffffffu, mx[g], 2));
                }
                if (kb == 0) {
#pragma unroll
                    for (int g = 0; g < 3; g++) h3S[((8 * sub + i) * 4 + v) * 3 + g] = mx[g];
                    if (!oz::row_ok(mx[0]) || !oz::row_ok(mx[1]) || !oz::row_ok(mx[2]) ||
                        !oz::row_ok(maxq[(8 * sub + i) * 4 + v]))
                        atomicOr(flagS + sub, 1u << i);
                }
                uint64_t y[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int f = (8 * kb + j) / Nfp;
                    y[j] = oz::biased(x[j], oz::row_bound(f == 0 ? mx[0] : f == 1 ? mx[1] : mx[2]));
                }
                unsigned char* dst = A2 + (((4 * sub + v) * 4 + kb) << 7) + (i << 4);
#pragma unroll
                for (int s = 0; s < oz::kSlices; s++)
                    *reinterpret_cast<uint4*>(dst + s * D::A2S) =
                        make_uint4(oz::digit_pair(y[0], y[1], s), oz::digit_pair(y[2], y[3], s),
                                   oz::digit_pair(y[4], y[5], s), oz::digit_pair(y[6], y[7], s));
                flux_written();
            }
            // the largest volume flux at the nodes (FP32), two elements a warp: what the
            // exponent of the flux rows comes from
#pragma unroll 1
            for (int u = 0; u < 2; u++) {
                const int i = 2 * cg + u;
                const double* gk = geoS + (8 * sub + i) * 4;
                const float rx = oz::trunc32(gk[0]), sx = oz::trunc32(gk[1]), ry = oz::trunc32(gk[2]), sy = oz::trunc32(gk[3]);
                float mf[4] = {0.f, 0.f, 0.f, 0.f};
                for (int n = lane; n < Np && gk0 + i < a.K; n += 32) {
                    float q[4];
#pragma unroll
                    for (int v = 0; v < 4; v++) q[v] = oz::trunc32(a.qin[((size_t)(gk0 + i) * 4 + v) * Np + n]);
                    const float ir = __fdividef(1.f, q[0]), uf = q[1] * ir, vf = q[2] * ir;
                    const float p = g1f * (q[3] - 0.5f * (q[1] * uf + q[2] * vf)), H = (q[3] + p) * ir;
                    const float Mr = rx * q[1] + ry * q[2], Ms = sx * q[1] + sy * q[2];
                    mf[0] = fmaxf(mf[0], fmaxf(fabsf(Mr), fabsf(Ms)));
                    mf[1] = fmaxf(mf[1], fmaxf(fabsf(Mr * uf + rx * p), fabsf(Ms * uf + sx * p)));
                    mf[2] = fmaxf(mf[2], fmaxf(fabsf(Mr * vf + ry * p), fabsf(Ms * vf + sy * p)));
                    mf[3] = fmaxf(mf[3], fmaxf(fabsf(Mr * H), fabsf(Ms * H)));
                }
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(mf[v]));
                    if (lane == 0) estS[(8 * sub + i) * 4 + v] = m;
                }
            }
            const bool live = gk0 + el < a.K;
            const double rx = geoS[e * 4], sx = geoS[e * 4 + 1], ry = geoS[e * 4 + 2], sy = geoS[e * 4 + 3];
            // a density or an energy whose digits lie too far below its row's largest value
            auto deep = [](double rho, uint32_t rmax, double E, uint32_t emax) {
                return oz::mag_hi(rho) + ((uint32_t)kRhoDepth << 20) < rmax || oz::mag_hi(E) + ((uint32_t)kEnergyDepth << 20) < emax;
            };
            // ---- 2. face fluxes
            waitw(bTrFull, phT);
            phT ^= 1;
            umma::fence_after_sync();
            const int ownrow = e * 4 + jv;
            const int eb1 = oz::row_bound(maxq[ownrow]);
            // A warp takes the 4-point groups cg and cg + 4 (when there are more than
            // four).  The rounds are rolled loops that shift their results (F, and the
            // jump for the Lax-Friedrichs flux) from one register set to the other.
            constexpr int GR = (D::NG4 + 3) / 4;
            double F[4], J[4], F0[4] = {0, 0, 0, 0}, J0[4] = {0, 0, 0, 0};
            uint32_t bad = 0;
#pragma unroll 1
            for (int r = 0; r < GR; r++) {
                const int gi = cg + 4 * r, pt = 4 * gi + jv;
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    F0[v] = F[v];
                    J0[v] = J[v];
                }
                if (gi < D::NG4) {
                    double qm[4], qp[4];
                    load8<32>(tlane + D::T_OWN + 4 * gi, [&](int) { return eb1 + ebI; }, qm);
                    load8<32>(tlane + D::T_NBR + 4 * gi,
                              [&](int c) { return oz::row_bound(h3S[ownrow * 3 + min(4 * gi + c, NF - 1) / Nfq]) + ebI; }, qp);
                    transpose4(qm, lane);
                    transpose4(qp, lane);
                    const int f = min(pt, NF - 1) / Nfq;
                    if (pt < NF && (deep(qm[0], maxq[e * 4], qm[3], maxq[e * 4 + 3]) ||
                                    deep(qp[0], h3S[e * 12 + f], qp[3], h3S[e * 12 + 9 + f])))
                        bad = 1u;
                    const double* nr = nrmS + e * 9 + f * 3;
                    if (a.flux == 1) {
                        roe_flux_fast(g1, nr[0], nr[1], qm, qp, F);
#pragma unroll
                        for (int v = 0; v < 4; v++) F[v] = pt < NF && live ? nr[2] * F[v] : 0.0;
                    } else {
                        // half the scaled normal in place of the normal: every term of the
                        // flux and the wave speeds carry the factor h = sJ/J / 2
                        const double h = 0.5 * nr[2], nx = h * nr[0], ny = h * nr[1], gh = a.gamma * (h * h);
                        const FaceSide m = face_side(g1, nx, ny, qm), p = face_side(g1, nx, ny, qp);
                        const double um = m.mn * m.r, up = p.mn * p.r, ps = m.p + p.p;
                        const double wm = fabs(um) + oz::sqrt64(fabs(gh * m.p * m.r));
                        const double wp = fabs(up) + oz::sqrt64(fabs(gh * p.p * p.r));
                        // magnitudes compare as integers (a NaN is the largest)
                        const long long wmi = __double_as_longlong(wm) & 0x7FFFFFFFFFFFFFFFll,
                                        wpi = __double_as_longlong(wp) & 0x7FFFFFFFFFFFFFFFll;
                        if (pt < NF) lamS[e * NF + pt] = __longlong_as_double(wmi > wpi ? wmi : wpi);
                        F[0] = m.mn + p.mn;
                        F[1] = fma(qm[1], um, fma(qp[1], up, nx * ps));
                        F[2] = fma(qm[2], um, fma(qp[2], up, ny * ps));
                        F[3] = fma(qm[3] + m.p, um, (qp[3] + p.p) * up);
#pragma unroll
                        for (int v = 0; v < 4; v++) J[v] = qm[v] - qp[v];
                    }
                }
            }
            umma::fence_before_sync();
            arrive(bTrRead);
            if (a.flux != 1) group_sync(sub);
#pragma unroll 1
            for (int r = 0; r < GR; r++) {
                const int gi = cg + 4 * (GR - 1 - r), pt = 4 * gi + jv;  // last round first
                if (gi < D::NG4) {
                    if (a.flux != 1) {
                        const int f = min(pt, NF - 1) / Nfq;
                        long long l = 0;
#pragma unroll
                        for (int i = 0; i < Nfq; i++) {
                            const long long w = __double_as_longlong(lamS[e * NF + f * Nfq + i]);
                            l = w > l ? w : l;
                        }
                        const double lam = __longlong_as_double(l);
#pragma unroll
                        for (int v = 0; v < 4; v++) F[v] = pt < NF && live ? fma(lam, J[v], F[v]) : 0.0;
                    }
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const uint32_t h = oz::mag_hi(F[v]);
                        if (h >= 0x7FF00000u) bad = 1u;
                        else atomicMax(maxf + e * 4 + v, h);
                    }
                }
                if (GR == 2) {
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const double w = F[v];
                        F[v] = F0[v];
                        F0[v] = w;
                        J[v] = J0[v];
                    }
                }
            }
            if (bad) atomicOr(flagS + sub, 1u << el);
            group_sync(sub);
            uint32_t reach = 0;
#pragma unroll
            for (int v = 0; v < 4; v++) {
                // one bit above the nodes' largest for points between them
                const float b = fminf(2.f * __uint_as_float(estS[e * 4 + v]), 1e38f);
                const int ee = b > 0.f ? (int)(__float_as_uint(b) >> 23) - 127 + 1 + 1022 : 0;
                const int ef = oz::row_bound(maxf[e * 4 + v]);
                eb2[v] = max(ef, ee);
                if (eb2[v] > 1700 || (eb2[v] != 0 && eb2[v] < 300)) bad = 1u;
                if (ef + kFluxSlack >= eb2[v]) reach |= 1u << v;
            }
            flux_free();
#pragma unroll 1
            for (int r = 0; r < GR; r++) {
                const int gi = cg + 4 * (GR - 1 - r), pt = 4 * gi + jv;
                if (gi < D::NG4) {
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const uint64_t y = oz::biased(F[v], eb2[v]);
                        unsigned char* dst = A2 + (((4 * sub + v) * 4 + (pt >> 3)) << 7) + (el << 4) + ((pt & 7) << 1);
#pragma unroll
                        for (int s = 0; s < oz::kSlices; s++)
                            *reinterpret_cast<uint16_t*>(dst + s * D::A2S) = (uint16_t)oz::digit_pair(y, y, s);
                    }
                }
                if (GR == 2) {
#pragma unroll
                    for (int v = 0; v < 4; v++) F[v] = F0[v];
                }
            }
            flux_written();
            // ---- 3. volume fluxes, 16 cubature points per chunk
#pragma unroll 1
            for (int c = 0; c < D::NC; c++) {
                const int p0 = 16 * c + 4 * cg, pt = p0 + jv;
                waitw(bD1full, phD);
                phD ^= 1;
                umma::fence_after_sync();
                double q[4];
                if (p0 < Ng) load8<16>(tlane + D::T_CUB + 4 * cg, [&](int) { return eb1 + ebV; }, q);
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
                    if (ok && deep(q[0], maxq[e * 4], q[3], maxq[e * 4 + 3])) bad = 1u;
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        if (!ok) Fr[w] = Fs[w] = 0.0;
                        const int b = oz::row_bound(max(oz::mag_hi(Fr[w]), oz::mag_hi(Fs[w])));
                        if (b > eb2[w]) bad = 1u;
                        if (b + kFluxSlack >= eb2[w]) reach |= 1u << w;
                        yr[w] = oz::biased(Fr[w], eb2[w]);
                        ys[w] = oz::biased(Fs[w], eb2[w]);
                    }
                }
                flux_free();
                if (p0 < Ng) {
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        unsigned char* dst = A2 + (((4 * sub + w) * 4 + cg) << 7) + (el << 4) + (jv << 2);
#pragma unroll
                        for (int s = 0; s < oz::kSlices; s++)
                            *reinterpret_cast<uint32_t*>(dst + s * D::A2S) = oz::digit_pair(yr[w], ys[w], s);
                    }
                }
                flux_written();
            }
            if (bad) atomicOr(flagS + sub, 1u << el);
            reach |= __shfl_xor_sync(0xffffffffu, reach, 8);
            reach |= __shfl_xor_sync(0xffffffffu, reach, 16);
            if (jv == 0) atomicOr(reachS + sub, reach << (4 * el));
            // ---- 4. result rows; the update's operands are on their way meanwhile
            const double* other = a.mode == MODE_LSERK ? a.res : a.mode == MODE_SSP2 ? a.qold : nullptr;
#pragma unroll
            for (int it = 0; it < IT; it++) {
                const int i = t + 128 * it;
                q0[it] = i < nval && a.mode != MODE_RHS ? a.qin[g0 + i] : 0.0;
                o0[it] = i < nval && other ? other[g0 + i] : 0.0;
            }
            flux_free();
            umma::fence_after_sync();
            int ebr = 0;
#pragma unroll
            for (int v = 0; v < 4; v++) ebr = jv == v ? eb2[v] : ebr;
#pragma unroll 1
            for (int n0 = 0; n0 < D::NP2; n0 += 16) {
                const int n4 = n0 + 4 * cg;
                if (n4 < Np) {
                    float d[8][4];
#pragma unroll
                    for (int s = 0; s < 8; s++) umma::tmem_ld4(tlane + D::T_RES + s * D::NP2 + n4, d[s]);
                    arrived(d);
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (n4 + j < Np) {
                            int ds[8];
#pragma unroll
                            for (int s = 0; s < 8; s++) ds[s] = oz::acc_int24(d[s][j]);
                            *striped(A2, sub, (el * 4 + jv) * Np + n4 + j, D::A2S, 2048) = oz::combine8(ds, ebr + ebS[n4 + j]);
                        }
                }
            }
            umma::fence_before_sync();
            group_sync(sub);
            uint32_t fl = flagS[sub];
            const uint32_t far = ~reachS[sub];  // a flux row whose bound its fluxes stayed far below
#pragma unroll
            for (int i = 0; i < 8; i++) fl |= ((far >> (4 * i)) & 15u) ? 1u << i : 0u;
            if (t == 0) oa.flags[gk0 >> 3] = (unsigned char)fl;
            // stage update, coalesced
#pragma unroll
            for (int it = 0; it < IT; it++) {
                const int i = t + 128 * it;
                if (i < nval && !((fl >> (i / (4 * Np))) & 1u)) {
                    const double Rv = *striped(A2, sub, i, D::A2S, 2048);
                    const size_t idx = g0 + i;
                    stage_update(a, idx, Rv, q0[it], o0[it]);
                }
            }
        }
        plain_pass<N>(oa, smem, t, sub);
    }
    umma::fence_before_sync();
    __syncthreads();
    // whoever gave up, and whenever
    if (threadIdx.x == 0 && *dead) {
        *reinterpret_cast<volatile int*>(oa.status) = 1;
        __threadfence_system();
    }
    if (warp == 16) {
        umma::fence_after_sync();
        umma::tmem_relinquish();
        umma::tmem_dealloc(tmem, 512);
    }
}

template <int N>
static cudaError_t setup_tc(const dgb::RefOps& ops, int K, OzPlan& plan) {
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
    if (e == cudaSuccess) e = cudaMalloc(&plan.d_image, im.bytes.size() + im.eb.size() * sizeof(int) + (size_t)K / 8 + 4);
    if (e != cudaSuccess) return e;
    plan.d_eb = reinterpret_cast<int*>((unsigned char*)plan.d_image + im.bytes.size());
    plan.d_flags = reinterpret_cast<unsigned char*>(plan.d_eb + im.eb.size());
    e = cudaMemcpy(plan.d_image, im.bytes.data(), im.bytes.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(plan.d_eb, im.eb.data(), im.eb.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(plan.d_flags, 0, (size_t)K / 8 + 4);
    if (e == cudaSuccess) plan.ready = true;
    return e;
}

cudaError_t setup_euler_fp64_tc(int N, const dgb::RefOps& ops, int K, OzPlan& plan) {
    switch (N) {
        case 1: return setup_tc<1>(ops, K, plan);
        case 2: return setup_tc<2>(ops, K, plan);
        case 3: return setup_tc<3>(ops, K, plan);
        case 4: return setup_tc<4>(ops, K, plan);
        case 5: return setup_tc<5>(ops, K, plan);
        case 6: return setup_tc<6>(ops, K, plan);
        case 7: return setup_tc<7>(ops, K, plan);
        default: return cudaErrorInvalidValue;
    }
}

void teardown_euler_fp64_tc(OzPlan& plan) {
    if (plan.d_image) cudaFree(plan.d_image);
    if (plan.h_status) cudaFreeHost(plan.h_status);
    plan = OzPlan();
}

// Groups of 8 elements per tile.  A tile of fewer groups is quicker, but not in
// proportion, since the chain of products and barriers stays: with 1, 2, 3 groups
// a tile takes 0.67, 0.76, 0.87 of the time of one with 4, within 0.07 at
// N = 1 .. 7 with either flux (N = 5, Lax-Friedrichs: 39, 43, 49, 55 us).  A small
// problem is that chain and nothing else, so its tiles are as small as half of
// the SMs allow (K = 512, N = 2, Roe: 39 -> 26 us).  Beyond that the SM time counts, for the
// stages of other contexts run beside this one: at K = 3200, N = 3, tiles of 3
// groups on 134 SMs are quicker alone (41 -> 37 us) and slower with others (28 -> 29).
static int tile_groups(int K, int sms) {
    for (int g = 1; g < 4; g++)
        if ((K + 8 * g - 1) / (8 * g) <= sms / 2) return g;
    return 4;
}

template <int N>
static cudaError_t launch_tc(const OzArgs& oa, const OzPlan& plan, cudaStream_t s) {
    const int ntiles = (oa.e.K + 8 * oa.groups - 1) / (8 * oa.groups);
    euler_stage_fp64_tc_kernel<N><<<std::min(ntiles, plan.sms), kOzThreads, OzDims<N>::SMEM, s>>>(oa);
    return cudaGetLastError();
}

cudaError_t launch_euler_fp64_tc(int N, const EulerArgs& a, const OzPlan& plan, cudaStream_t s) {
    const OzArgs oa{a, (const unsigned char*)plan.d_image, plan.d_eb, plan.status, plan.d_flags, tile_groups(a.K, plan.sms)};
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
