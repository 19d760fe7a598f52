// euler_flux.cuh -- point-wise Euler fluxes (device), templated on the
// arithmetic type (double for the FP64 path, float for the split path).
#pragma once

namespace dgk {

// physical flux at a point; p = (gamma-1)(E - rho |U|^2 / 2) as gther_p of
// tutorials/DG/2D/isentropicVortex/dgEulerFoam/dgEulerFoam.C:81-82
template <typename T>
__device__ __forceinline__ void euler_phys_flux(T gamma, const T q[4], T fx[4], T fy[4]) {
    const T rho = q[0];
    const T u = q[1] / rho, v = q[2] / rho;
    const T p = (gamma - T(1)) * (q[3] - T(0.5) * (rho * (u * u + v * v)));
    fx[0] = q[1];
    fx[1] = u * q[1] + p;
    fx[2] = u * q[2];
    fx[3] = u * (q[3] + p);
    fy[0] = q[2];
    fy[1] = v * q[1];
    fy[2] = v * q[2] + p;
    fy[3] = v * (q[3] + p);
}

// outward unit normal and sJ/J of local face f of an affine triangle from its
// metrics (face 0: s = -1, face 1: r + s = 0, face 2: r = -1); equals the
// reference's faceNx / fscale (gaussTriangleIntegration.C:153-192,
// triangleBaseFunction.C:393-419) for straight edges.
__host__ __device__ __forceinline__ void face_normal(int f, double rx, double sx, double ry, double sy, double& nx,
                                                     double& ny, double& fsc) {
    double gx, gy;
    if (f == 0) { gx = -sx; gy = -sy; }
    else if (f == 1) { gx = rx + sx; gy = ry + sy; }
    else { gx = -rx; gy = -ry; }
    fsc = sqrt(gx * gx + gy * gy);
    nx = gx / fsc;
    ny = gy / fsc;
}

// FP32 version for the split path (GB300 runs FP64 sqrt/divide as long DFMA
// sequences at 1/70 of the FP32 rate)
__device__ __forceinline__ void face_normal_f(int f, float rx, float sx, float ry, float sy, float& nx, float& ny,
                                              float& fsc) {
    float gx, gy;
    if (f == 0) { gx = -sx; gy = -sy; }
    else if (f == 1) { gx = rx + sx; gy = ry + sy; }
    else { gx = -rx; gy = -ry; }
    fsc = sqrtf(fmaf(gy, gy, __fmul_rn(gx, gx)));
    const float inv = 1.f / fsc;
    nx = __fmul_rn(gx, inv);
    ny = __fmul_rn(gy, inv);
}

template <typename T>
__device__ __forceinline__ T wave_speed(T gamma, T nx, T ny, const T q[4]) {
    const T rho = q[0], u = q[1] / rho, v = q[2] / rho;
    const T p = (gamma - T(1)) * (q[3] - T(0.5) * rho * (u * u + v * v));
    const T c = sqrt(fabs(gamma * p / rho));
    return fabs(u * nx + v * ny) + c;
}

// Euler Lax-Friedrichs (Rusanov): n.F* = 1/2 (F- + F+).n + 1/2 lam (q- - q+)
template <typename T>
__device__ __forceinline__ void lf_flux(T gamma, T nx, T ny, T lam, const T qm[4], const T qp[4], T F[4]) {
    T fxa[4], fya[4], fxb[4], fyb[4];
    euler_phys_flux(gamma, qm, fxa, fya);
    euler_phys_flux(gamma, qp, fxb, fyb);
#pragma unroll
    for (int v = 0; v < 4; v++)
        F[v] = T(0.5) * ((fxa[v] + fxb[v]) * nx + (fya[v] + fyb[v]) * ny) + T(0.5) * lam * (qm[v] - qp[v]);
}

// Roe flux in the face-normal frame, entropy fix 0
// (DG/godunovFlux/fluxSchemes/scheme/RoeFlux/RoeFlux.C:129-178).
template <typename T>
__device__ __forceinline__ void roe_flux(T gamma, T nx, T ny, const T qO[4], const T qN[4], T F[4]) {
    const T QP2 = nx * qN[1] + ny * qN[2], QM2 = nx * qO[1] + ny * qO[2];
    const T QP3 = nx * qN[2] - ny * qN[1], QM3 = nx * qO[2] - ny * qO[1];
    const T rhoP = qN[0], rhoM = qO[0];
    const T uM = QM2 / rhoM, uP = QP2 / rhoP, vM = QM3 / rhoM, vP = QP3 / rhoP;
    const T pM = (gamma - T(1)) * (qO[3] - T(0.5) * (QM2 * uM + QM3 * vM));
    const T pP = (gamma - T(1)) * (qN[3] - T(0.5) * (QP2 * uP + QP3 * vP));
    const T HM = (qO[3] + pM) / rhoM, HP = (qN[3] + pP) / rhoP;
    T fr = (QM2 + QP2) / T(2);
    T fu = (QM2 * uM + pM + QP2 * uP + pP) / T(2);
    T fv = (QM3 * uM + QP3 * uP) / T(2);
    T fe = (uM * (qO[3] + pM) + uP * (qN[3] + pP)) / T(2);
    const T rhoMs = sqrt(rhoM), rhoPs = sqrt(rhoP);
    const T rhob = rhoMs * rhoPs;
    const T u = (rhoMs * uM + rhoPs * uP) / (rhoMs + rhoPs);
    const T v = (rhoMs * vM + rhoPs * vP) / (rhoMs + rhoPs);
    const T H = (rhoMs * HM + rhoPs * HP) / (rhoMs + rhoPs);
    const T c2 = (gamma - T(1)) * (H - T(0.5) * (u * u + v * v));
    const T c = sqrt(fabs(c2));
    const T dw1 = (T(-0.5) * rhob * (uP - uM) / c + T(0.5) * (pP - pM) / c2) * fabs(u - c);
    const T dw2 = ((rhoP - rhoM) - (pP - pM) / c2) * fabs(u);
    const T dw3 = (rhob * (vP - vM)) * fabs(u);
    const T dw4 = (T(0.5) * rhob * (uP - uM) / c + T(0.5) * (pP - pM) / c2) * fabs(u + c);
    fr -= (dw1 + dw2 + dw4) / T(2);
    fu -= (dw1 * (u - c) + dw2 * u + dw4 * (u + c)) / T(2);
    fv -= (dw1 * v + dw2 * v + dw3 + dw4 * v) / T(2);
    fe -= (dw1 * (H - u * c) + dw2 * (u * u + v * v) / T(2) + dw3 * v + dw4 * (H + u * c)) / T(2);
    F[0] = fr;
    F[1] = nx * fu - ny * fv;
    F[2] = ny * fu + nx * fv;
    F[3] = fe;
}

// ---------------------------------------------------------------------------
// Delta (product-rule) forms used by the split-precision path (FP32; the
// divisions use the fast approximate form: their results carry FP32-level
// relative error, inside the path's error budget).  With a
// per-element reference state qb and q = qb + dq, the weak right-hand side
// satisfies R(F) = R(F - F(qb)) exactly (the discrete divergence of a
// constant flux cancels against its own surface term), so the kernels feed the
// contractions with dF = F(qb + dq) - F(qb).  Written as below, dF carries
// FP32 round-off relative to |dq| instead of |q|: no cancellation.
//
// Every sum of products below says which product is rounded (__fmul_rn) and
// which goes into an FMA.  Left to the compiler, that choice differs between
// the inlined copies of the same source (a block's first tile and its others,
// one order's kernel and the mixed-order one), and results would depend on a tile's place.

struct RefState {
    float rho, m, n, E, u, v, p, H;  // H = E + p
};

__device__ __forceinline__ RefState make_ref(float gamma, const float qb[4]) {
    RefState b;
    b.rho = qb[0];
    b.m = qb[1];
    b.n = qb[2];
    b.E = qb[3];
    const float ir = __fdividef(1.f, b.rho);
    b.u = __fmul_rn(b.m, ir);
    b.v = __fmul_rn(b.n, ir);
    b.p = __fmul_rn(gamma - 1.f, fmaf(-0.5f, fmaf(b.n, b.v, __fmul_rn(b.m, b.u)), b.E));
    b.H = b.E + b.p;
    return b;
}

// full velocities and pressure delta of q = qb + dq (helpers shared by the fluxes)
struct DeltaPrim {
    float rho, u, v, du, dv, dp, E;
};

__device__ __forceinline__ DeltaPrim delta_prim(float gamma, const RefState& b, const float dq[4]) {
    DeltaPrim d;
    d.rho = b.rho + dq[0];
    const float m = b.m + dq[1], n = b.n + dq[2];
    const float ir = __fdividef(1.f, d.rho);
    d.du = __fmul_rn(fmaf(-b.u, dq[0], dq[1]), ir);
    d.dv = __fmul_rn(fmaf(-b.v, dq[0], dq[2]), ir);
    d.u = b.u + d.du;
    d.v = b.v + d.dv;
    // twice the kinetic part, from the products and sums that flux_delta needs as well (as FMAs the
    // N = 5 stage spills in its face phase: 307 us a stage for 297)
    const float dK2 = ((__fmul_rn(dq[1], b.u) + __fmul_rn(m, d.du)) + __fmul_rn(dq[2], b.v)) + __fmul_rn(n, d.dv);
    d.dp = __fmul_rn(gamma - 1.f, fmaf(-0.5f, dK2, dq[3]));
    d.E = b.E + dq[3];
    return d;
}

__device__ __forceinline__ void flux_delta(const RefState& b, const float dq[4], const DeltaPrim& d, float dFx[4],
                                           float dFy[4]) {
    const float m = b.m + dq[1], n = b.n + dq[2];
    const float dH = dq[3] + d.dp;
    dFx[0] = dq[1];
    dFx[1] = (__fmul_rn(dq[1], b.u) + __fmul_rn(m, d.du)) + d.dp;
    dFx[2] = fmaf(n, d.du, __fmul_rn(dq[2], b.u));
    dFx[3] = fmaf(d.u, dH, __fmul_rn(d.du, b.H));
    dFy[0] = dq[2];
    dFy[1] = fmaf(m, d.dv, __fmul_rn(dq[1], b.v));
    dFy[2] = (__fmul_rn(dq[2], b.v) + __fmul_rn(n, d.dv)) + d.dp;
    dFy[3] = fmaf(d.v, dH, __fmul_rn(d.dv, b.H));
}

__device__ __forceinline__ float wave_speed_delta(float gamma, float nx, float ny, const RefState& b, const DeltaPrim& d) {
    const float p = b.p + d.dp;
    return fabsf(fmaf(d.v, ny, __fmul_rn(d.u, nx))) + sqrtf(fabsf(__fdividef(__fmul_rn(gamma, p), d.rho)));
}

// twice the mean normal flux of the two sides
__device__ __forceinline__ float normal_sum(float nx, float ny, float xm, float xp, float ym, float yp) {
    return fmaf(ym + yp, ny, __fmul_rn(xm + xp, nx));
}

// 2 (n.F*(q-, q+) - n.F(qb)), Lax-Friedrichs
__device__ __forceinline__ void lf_flux_delta(float nx, float ny, float lam, const RefState& b, const float dm[4],
                                              const DeltaPrim& pm, const float dpq[4], const DeltaPrim& pp, float F[4]) {
    float fxm[4], fym[4], fxp[4], fyp[4];
    flux_delta(b, dm, pm, fxm, fym);
    flux_delta(b, dpq, pp, fxp, fyp);
#pragma unroll
    for (int v = 0; v < 4; v++) F[v] = fmaf(lam, dm[v] - dpq[v], normal_sum(nx, ny, fxm[v], fxp[v], fym[v], fyp[v]));
}

// 2 (n.F*(q-, q+) - n.F(qb)), Roe (RoeFlux.C:129-178 rearranged: central part in
// delta form, wave strengths from side-to-side jumps of the deltas)
__device__ __forceinline__ void roe_flux_delta(float gamma, float nx, float ny, const RefState& b, const float dm[4],
                                               const DeltaPrim& pm, const float dpq[4], const DeltaPrim& pp,
                                               float F[4]) {
    float fxm[4], fym[4], fxp[4], fyp[4];
    flux_delta(b, dm, pm, fxm, fym);
    flux_delta(b, dpq, pp, fxp, fyp);
    const float unM = fmaf(ny, pm.v, __fmul_rn(nx, pm.u)), unP = fmaf(ny, pp.v, __fmul_rn(nx, pp.u));
    const float utM = fmaf(-ny, pm.u, __fmul_rn(nx, pm.v)), utP = fmaf(-ny, pp.u, __fmul_rn(nx, pp.v));
    const float pM = b.p + pm.dp, pP = b.p + pp.dp;
    const float HM = (pm.E + pM) / pm.rho, HP = (pp.E + pP) / pp.rho;
    const float sM = sqrtf(pm.rho), sP = sqrtf(pp.rho);
    const float rhob = __fmul_rn(sM, sP);
    const float inv = 1.f / (sM + sP);
    const float u = __fmul_rn(fmaf(sP, unP, __fmul_rn(sM, unM)), inv);
    const float v = __fmul_rn(fmaf(sP, utP, __fmul_rn(sM, utM)), inv);
    const float H = __fmul_rn(fmaf(sP, HP, __fmul_rn(sM, HM)), inv);
    const float ke2 = fmaf(u, u, __fmul_rn(v, v));
    const float c2 = __fmul_rn(gamma - 1.f, fmaf(-0.5f, ke2, H));
    const float c = sqrtf(fabsf(c2));
    const float jr = dpq[0] - dm[0];
    const float jdu = pp.du - pm.du, jdv = pp.dv - pm.dv;
    const float jun = fmaf(ny, jdv, __fmul_rn(nx, jdu)), jut = fmaf(-ny, jdu, __fmul_rn(nx, jdv));
    const float jp = pp.dp - pm.dp;
    const float wu = __fmul_rn(__fmul_rn(0.5f, rhob), jun) / c, wp = __fmul_rn(0.5f, jp) / c2;
    const float dw1 = __fmul_rn(wp - wu, fabsf(u - c));
    const float dw2 = __fmul_rn(jr - jp / c2, fabsf(u));
    const float dw3 = __fmul_rn(__fmul_rn(rhob, jut), fabsf(u));
    const float dw4 = __fmul_rn(wu + wp, fabsf(u + c));
    const float dr = dw1 + dw2 + dw4;
    const float du = fmaf(dw4, u + c, fmaf(dw2, u, __fmul_rn(dw1, u - c)));
    const float dv = fmaf(dr, v, dw3);
    const float de = fmaf(dw4, fmaf(u, c, H),
                          fmaf(dw3, v, fmaf(__fmul_rn(dw2, ke2), 0.5f, __fmul_rn(dw1, fmaf(-u, c, H)))));
    const float d[4] = {dr, fmaf(-ny, dv, __fmul_rn(nx, du)), fmaf(nx, dv, __fmul_rn(ny, du)), de};
#pragma unroll
    for (int w = 0; w < 4; w++) F[w] = normal_sum(nx, ny, fxm[w], fxp[w], fym[w], fyp[w]) - d[w];
}

}  // namespace dgk
