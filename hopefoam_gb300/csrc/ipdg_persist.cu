// ipdg_persist.cu -- PCG iterations of small problems in one cooperative
// launch (sm_103a).
//
// Up to a few thousand elements every kernel of a PCG iteration is a few
// microseconds of latency: launches, a trip through memory for each vector,
// and two grid-wide sums with their own arrival logic (29 us per iteration
// at K = 4228, N = 4 with block Jacobi; 42 us at K = 1152, N = 3 with the
// coarse space).  Here one lane owns one row for the whole launch: its
// entries of x, r, z, p, its block row of S (ipdg_block.cu, 4 Np values) and its
// row of the block-Jacobi inverse stay in registers and shared memory, and what crosses
// elements is the preconditioned residual.  The neighbours' search directions
// are not exchanged: every lane carries its neighbours' through the same
// recurrence p = z + beta p.  An iteration is two grid barriers, each with its
// sum (p.Ap; r.z and r.r); with the coarse space (a level held as one dense
// matrix, mg.hpp) two more.  Scalars are computed by every block from the
// same partial sums in the same order, so they agree and solves are
// reproducible.
//
// Measured at persist_fits.  Waits are bounded (co-residency comes from the
// cooperative launch); a block whose wait gave up sets the status word and
// leaves, and the others follow.
#include <algorithm>
#include <type_traits>

#include "ipdg.hpp"
#include "ipdg_rows.cuh"
#include "mg.hpp"

namespace dgk {

namespace {

constexpr unsigned kSpinLimit = 1u << 21;  // polls of about a microsecond

template <typename T>
struct PersistDims {
    // warps per block: 128 registers a thread at 16, 255 at 8
    __host__ __device__ static constexpr int warps(int np) { return sizeof(T) == 4 && np <= 15 ? 16 : 8; }
    // of a row's four blocks of S, how many stay in shared memory with the row of
    // the block-Jacobi inverse: registers that spill come back through L2, since
    // every exchange's fence drops the L1
    __host__ __device__ static constexpr int shared_blocks(int np) { return sizeof(T) == 4 && np <= 15 ? np / 7 : 0; }
    __host__ __device__ static constexpr size_t shared_bytes(int np, int threads) {
        return (size_t)threads * (sizeof(double) + sizeof(T) * (np + 4 + shared_blocks(np) * np));
    }
    __host__ __device__ static constexpr bool fits(int np) { return sizeof(T) == 4 ? np <= 21 : np <= 15; }
};

struct PersistArgs {
    IpdgArgs a;
    PcgVecs v;
    MgLevels m;
    const void* rows;  // block rows in the arithmetic type
    double* corner;    // [3 K] corner sums of the coarse restriction, in the order of the vertices' lists
    int parity, count;
    ulonglong2* slots;  // of the exchanges
    unsigned long long exchanges;  // before this launch
    int owners;        // warps of a block that own rows; the others help with the coarse space
    int vrows;         // rows of the dense cycle a block holds at most
};

// Sums over a warp of NV values; with two, each half of the warp finishes one.
// The sums are right in lane 0 (first value) and lane 16 (second).
template <int NV>
__device__ __forceinline__ double warp_sums(const double (&a)[2], int lane) {
    double s = a[0];
    if (NV == 2) {
        const bool hi = lane & 16;
        s = (hi ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[1], 16);
    } else {
        s += __shfl_xor_sync(0xffffffffu, s, 16);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Grid-wide sums through tagged words.  A value travels as a pair (bits, bits
// ^ tag of this exchange), so arrival and data are one trip.  Blocks post to
// the leader of their group of 13, which sums them and posts the group's sum
// to a line of every block; every block sums the groups in the same order.
// Bound by the trips through L2 and the chain of FP64 additions.  Against
// other schemes, per iteration of 151 blocks: an arrival counter with partial
// sums (a release, an atomic, a poll, a read) 1.05 times as long; every block
// polling every post 1.5 times (23 thousand reads a poll delay the posts); one
// block summing and one line polled by all 1.4 times.
// Two sets of slots alternate: a slot is rewritten two exchanges later, after
// everyone who reads it has taken part in the exchange between.
constexpr int kMaxBlocks = 160, kGroup = 13, kSetSlots = 2 * 16 * 16 + 2 * 16 * kMaxBlocks;

__device__ __forceinline__ void post(ulonglong2* slot, double a, unsigned long long tag) {
    const unsigned long long w = (unsigned long long)__double_as_longlong(a);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(w), "l"(w ^ tag) : "memory");
}

__device__ __forceinline__ bool peek(const ulonglong2* slot, double& a, unsigned long long tag) {
    unsigned long long w, x;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w), "=l"(x) : "l"(slot) : "memory");
    a = __longlong_as_double((long long)w);
    return (w ^ tag) == x;
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

struct Exchange {
    ulonglong2* slots;     // [2][kSetSlots]
    unsigned long long n;  // exchanges so far, over all launches

    // By warp 0 of every block: sums over lanes and blocks of NV values, turned by
    // scalars(sums, tot) into every block's tot.  PUB: what the block's threads
    // wrote before its last __syncthreads is visible to every block after the
    // next.  False when a wait gave up.
    template <int NV, bool PUB, typename F>
    __device__ __forceinline__ bool run(const double (&s)[2], double* tot, int lane, F scalars) {
        constexpr int NQ = NV > 1 ? 2 : 1;
        const unsigned long long tag = (n + 1) * 0x9E3779B97F4A7C15ull;
        ulonglong2* set = slots + (n & 1) * kSetSlots;
        n++;
        const int q = lane >> 4, m = lane & 15, grid = gridDim.x;
        const int grp = blockIdx.x / kGroup, first = grp * kGroup, groups = (grid + kGroup - 1) / kGroup;
        double a = 0;
        if (NV > 0) a = warp_sums<NQ>(s, lane);
        if (PUB) fence_gpu();
        if (m == 0 && q < NQ) post(set + (q * 16 + grp) * 16 + blockIdx.x - first, a, tag);
        unsigned tries = 0;
        bool all;
        if (blockIdx.x == first) {
            const int members = min(kGroup, grid - first);
            do {
                all = true;
                a = 0;
                if (q < NQ && m < members) all = peek(set + (q * 16 + grp) * 16 + m, a, tag);
                all = __all_sync(0xffffffffu, all);
            } while (!all && ++tries < kSpinLimit);
            if (!all) return false;
            if (NV > 0)
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (PUB) fence_gpu();
            if (q < NQ)
#pragma unroll
                for (int u = 0; u < 10; u++) {
                    const int c = m + 16 * u;
                    if (c < grid) post(set + 512 + (c * 2 + q) * 16 + grp, a, tag);
                }
        }
        do {
            all = true;
            a = 0;
            if (q < NQ && m < groups) all = peek(set + 512 + (blockIdx.x * 2 + q) * 16 + m, a, tag);
            all = __all_sync(0xffffffffu, all);
        } while (!all && ++tries < kSpinLimit);
        if (PUB) fence_gpu();
        if (!all) return false;
        if (NV > 0) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            const double t[2] = {a, __shfl_sync(0xffffffffu, a, 16)};
            if (lane == 0) scalars(t, tot);
        }
        return true;
    }
};

template <int NP, typename T, bool MG>
__global__ void __launch_bounds__(32 * PersistDims<T>::warps(NP), 1) pcg_persist_kernel(const __grid_constant__ PersistArgs A) {
    using R = RowDims<NP>;
    constexpr int EW = R::EW, EB = R::EB, CS = EB * NP;
    constexpr bool F32 = sizeof(T) == 4;
    constexpr int MAXT = 32 * PersistDims<T>::warps(NP);
    __shared__ double red[2][MAXT];
    __shared__ double tot[3];
    __shared__ int dead;
    __shared__ double lamS[MG ? 3 * NP : 1];
    // per thread: x, its row of the block-Jacobi inverse, face weights, maybe a block
    // of S; then the coarse residual, the block's rows of the dense cycle, vertex pointers
    extern __shared__ double dyn[];
    constexpr int SH = PersistDims<T>::shared_blocks(NP);
    const int OT = 32 * A.owners, ot = threadIdx.x;
    double* xs = dyn;
    T* sP = reinterpret_cast<T*>(xs + OT);
    T* sW = sP + NP * OT;
    T* sR = sW + 4 * OT;
    double* coarse = reinterpret_cast<double*>(sR + SH * NP * OT);
    const PcgVecs& v = A.v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const bool owner = warp < A.owners;
    const int le = lane / NP, i = lane - le * NP, lb = le * NP;
    const int k = (blockIdx.x * A.owners + warp) * EW + le;
    const bool act = owner && le < EW && k < A.a.K;
    const size_t idx = (size_t)k * NP + i;
    if (threadIdx.x == 0) dead = 0;
    if (v.S->done) return;  // the same for every block
    const int n0 = MG ? A.m.lv[0].n : 0;
    double *r1s = coarse, *Vs = coarse + n0;
    int* vptr = reinterpret_cast<int*>(Vs + (size_t)A.vrows * n0);
    if (MG) {
        for (int t = threadIdx.x; t < 3 * NP; t += blockDim.x) lamS[t] = A.m.lam[t];
        for (int t = threadIdx.x; t <= n0; t += blockDim.x) vptr[t] = A.m.vptr[t];
        for (int m = warp, q = blockIdx.x + warp * gridDim.x; q < n0; m += nw, q += nw * gridDim.x)
            for (int j = lane; j < n0; j += 32) Vs[(size_t)m * n0 + j] = A.m.V[(size_t)q * n0 + j];
        __syncthreads();
    }
    Exchange ex{A.slots, A.exchanges};
    // Sums of one or two values per owner thread; `scalars` turns them into what
    // every thread reads from tot.  Within the block warp 0 sums columns of the
    // staged values, a third of the FP64 additions of warp butterflies.
    auto reduce = [&](double a0, double a1, auto nv, auto scalars) {
        constexpr int NV = decltype(nv)::value;
        if (owner) {
            red[0][threadIdx.x] = a0;
            if (NV == 2) red[1][threadIdx.x] = a1;
        }
        __syncthreads();
        if (warp == 0) {
            double s[2] = {0, 0};
#pragma unroll
            for (int q = 0; q < NV; q++) {
                double u[4] = {0, 0, 0, 0};
#pragma unroll
                for (int w = 0; w < MAXT / 32; w++)
                    if (w < A.owners) u[w & 3] += red[q][32 * w + lane];
                s[q] = (u[0] + u[1]) + (u[2] + u[3]);
            }
            if (!ex.template run<NV, NV == 2>(s, tot, lane, scalars) && lane == 0) dead = 1;
        }
        __syncthreads();
        return dead == 0;
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    auto barrier = [&]() {
        __syncthreads();
        if (warp == 0) {
            const double none[2] = {0, 0};
            if (!ex.template run<0, true>(none, tot, lane, [](const double*, double*) {}) && lane == 0) dead = 1;
        }
        __syncthreads();
        return dead == 0;
    };

    // state of the row
    constexpr int RB = 4 - SH;  // blocks 4 - SH .. 3 are in shared memory
    T row[RB * NP];
    int nb[3] = {-1, -1, -1}, ev[3] = {0, 0, 0};
    double r = 0, z = 0, p = 0;
    double pn[3] = {0, 0, 0};               // FP64: row i of the neighbours' p
    double pf = 0;                          // FP32: lane i < 3 carries neighbour i's first value of p
    int nf = -1;                            //       and its element
    float dz = 0, dp = 0, dn[3] = {0, 0, 0};  // FP32: offsets of z, p and the neighbours' p
    const double* p_old = v.p[A.parity];
    const float* dp_old = F32 ? v.dp[A.parity] : nullptr;
#pragma unroll
    for (int j = 0; j < RB * NP; j++) row[j] = 0;
    if (owner) {
        xs[ot] = 0;
        for (int j = 0; j < NP; j++) sP[j * OT + ot] = 0;
        for (int j = 0; j < SH * NP; j++) sR[j * OT + ot] = 0;
        for (int j = 0; j < 4; j++) sW[j * OT + ot] = 0;
    }
    double beta = v.S->beta;
    if (act) {
        const int grp = k / EB, e = k - grp * EB;
        const T* col = static_cast<const T*>(A.rows) + (size_t)grp * (4 * NP + 4) * CS + e * NP + i;
#pragma unroll
        for (int j = 0; j < RB * NP; j++) row[j] = col[(size_t)j * CS];
#pragma unroll
        for (int j = 0; j < SH * NP; j++) sR[j * OT + ot] = col[(size_t)(RB * NP + j) * CS];
#pragma unroll
        for (int f = 0; f < 4; f++) sW[f * OT + ot] = col[(size_t)(4 * NP + f) * CS];
        const size_t pb = (size_t)grp * NP * CS + e * NP + i;
#pragma unroll
        for (int j = 0; j < NP; j++) sP[j * OT + ot] = F32 ? (T)v.P32[pb + (size_t)j * CS] : (T)v.P64[pb + (size_t)j * CS];
        xs[ot] = v.x[idx];
        r = v.r[idx];
        z = v.z[idx];
        if (beta != 0.0) p = p_old[idx];
        if (F32) {
            dz = v.dz[idx];
            if (beta != 0.0) dp = dp_old[idx];
        }
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const int c = A.a.conn[(size_t)k * 3 + f];
            nb[f] = c >= 0 ? c >> 3 : -1;
            if (nb[f] >= 0 && beta != 0.0) {
                if (F32) dn[f] = dp_old[(size_t)nb[f] * NP + i];
                else pn[f] = p_old[(size_t)nb[f] * NP + i];
            }
            if (i == f) nf = nb[f];
            if (MG) ev[f] = A.m.etov[(size_t)k * 3 + f];
        }
        if (F32 && nf >= 0 && beta != 0.0) pf = p_old[(size_t)nf * NP];
    }
    int cpos = 0;  // place of corner i < 3 of the element in the vertices' lists
    if (MG && act && i < 3) {
        cpos = A.m.vptr[i == 0 ? ev[0] : i == 1 ? ev[1] : ev[2]];
        while (A.m.vinc[cpos] != 3 * k + i) cpos++;
    }
    double rz = v.S->rz, rr = v.S->rr, pap = v.S->pap, alpha = v.S->alpha;
    int done = 0, it = v.S->it, n = 0;
    const double tol2 = v.S->tol2;
    bool ok = true;
    for (; n < A.count && !done; n++) {
        double Ap = 0;
        if (owner) {
            // p = z + beta p, the neighbours' likewise
            const bool hb = beta != 0.0;
            const float bf = (float)beta;
            double zn[3] = {0, 0, 0}, zf = 0;
            float dzn[3] = {0, 0, 0};
#pragma unroll
            for (int f = 0; f < 3; f++)
                if (nb[f] >= 0) {
                    if (F32) dzn[f] = __ldcg(v.dz + (size_t)nb[f] * NP + i);
                    else zn[f] = __ldcg(v.z + (size_t)nb[f] * NP + i);
                }
            if (F32 && nf >= 0) zf = __ldcg(v.z + (size_t)nf * NP);
            p = hb ? fma(beta, p, z) : z;
            const double p0 = __shfl_sync(0xffffffffu, p, lb);
            // Ap, row by row (ipdg_block.cu), the four blocks in sums of their own
            T s[4] = {0, 0, 0, 0}, d[4];
            if (F32) {
                dp = hb ? fmaf(bf, dp, dz) : dz;
                d[0] = (T)dp;
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    dn[f] = hb ? fmaf(bf, dn[f], dzn[f]) : dzn[f];
                    d[f + 1] = (T)dn[f];
                }
                // first-node differences: lane f < 3 forms neighbour f's, lane 3 (a cast of
                // its own at N = 1) passes the own value on
                pf = hb ? fma(beta, pf, zf) : zf;
                const float df = (float)(i < 3 ? pf - p0 : p0);
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    const float w = __shfl_sync(0xffffffffu, df, lb + f);
                    if (nb[f] >= 0) s[f + 1] = sW[f * OT + ot] * (T)w;
                }
                s[0] = sW[3 * OT + ot] * (T)(NP > 3 ? __shfl_sync(0xffffffffu, df, lb + 3) : (float)p0);
            } else {
                d[0] = (T)(p - p0);
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    pn[f] = hb ? fma(beta, pn[f], zn[f]) : zn[f];
                    const double q0 = __shfl_sync(0xffffffffu, pn[f], lb);
                    d[f + 1] = (T)(pn[f] - q0);
                    if (nb[f] >= 0) s[f + 1] = sW[f * OT + ot] * (T)(q0 - p0);
                }
                s[0] = sW[3 * OT + ot] * (T)p0;
            }
#pragma unroll
            for (int j = 0; j < NP; j++)
#pragma unroll
                for (int b = 0; b < 4; b++)
                    s[b] += (b < RB ? row[(b < RB ? b : 0) * NP + j] : sR[((b - RB) * NP + j) * OT + ot]) * __shfl_sync(0xffffffffu, d[b], lb + j);
            Ap = act ? (double)((s[0] + s[1]) + (s[2] + s[3])) : 0.0;
        }
        if (!(ok = reduce(Ap * p, 0.0, One{}, [&](const double* t, double* out) {
                  out[0] = t[0];
                  out[1] = rz / t[0];
              })))
            break;
        pap = tot[0];
        alpha = tot[1];
        if (!(pap > 0.0) || !(alpha == alpha)) {
            done = 2;
            break;
        }
        if (owner) {
            // x, r, and the block-Jacobi product
            xs[ot] += alpha * p;
            r -= alpha * Ap;
            if (!act) r = 0.0;
            const T rt = (T)r;
            T z0 = 0, z1 = 0;
#pragma unroll
            for (int j = 0; j < NP; j += 2) {
                z0 += sP[j * OT + ot] * __shfl_sync(0xffffffffu, rt, lb + j);
                if (j + 1 < NP) z1 += sP[(j + 1) * OT + ot] * __shfl_sync(0xffffffffu, rt, lb + j + 1);
            }
            z0 += z1;
            z = (double)z0;
            if (F32) dz = (float)z0 - __shfl_sync(0xffffffffu, (float)z0, lb);
        }
        if (MG) {
            if (owner) {
                // corner sums of the restriction, lane i < 3 corner i
                double c0 = 0, c1 = 0;
                const int cc = i % 3;
#pragma unroll
                for (int j = 0; j < NP; j += 2) {
                    c0 += lamS[3 * j + cc] * __shfl_sync(0xffffffffu, r, lb + j);
                    if (j + 1 < NP) c1 += lamS[3 * (j + 1) + cc] * __shfl_sync(0xffffffffu, r, lb + j + 1);
                }
                if (act && i < 3) __stcg(A.corner + cpos, c0 + c1);
            }
            if (!(ok = barrier())) break;
            // every block sums the vertices, then takes its rows of the dense cycle
            for (int q = threadIdx.x; q < n0; q += blockDim.x) {
                double t = 0;
                const int w1 = vptr[q + 1];
                for (int w = vptr[q]; w < w1; w += 8) {
                    double g[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) g[u] = w + u < w1 ? __ldcg(A.corner + w + u) : 0.0;
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        if (w + u < w1) t += g[u];
                }
                r1s[q] = t;
            }
            __syncthreads();
            for (int m = warp, q = blockIdx.x + warp * gridDim.x; q < n0; m += nw, q += nw * gridDim.x) {
                const double* V = Vs + (size_t)m * n0;
                double t0 = 0, t1 = 0;
                int j = lane;
#pragma unroll 4
                for (; j + 32 < n0; j += 64) {
                    t0 += V[j] * r1s[j];
                    t1 += V[j + 32] * r1s[j + 32];
                }
                if (j < n0) t0 += V[j] * r1s[j];
                t0 += t1;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t0 += __shfl_xor_sync(0xffffffffu, t0, o);
                if (lane == 0) __stcg(A.m.lv[0].x + q, t0);
            }
            if (!(ok = barrier())) break;
            if (owner) {
                double cz = 0;
                if (act)
                    cz = lamS[3 * i] * __ldcg(A.m.lv[0].x + ev[0]) + lamS[3 * i + 1] * __ldcg(A.m.lv[0].x + ev[1]) +
                         lamS[3 * i + 2] * __ldcg(A.m.lv[0].x + ev[2]);
                z += cz;
                if (F32) {
                    const double c0 = __shfl_sync(0xffffffffu, cz, lb);
                    dz += (float)(cz - c0);
                }
            }
        }
        if (act) {
            // what the neighbours need of z
            if (F32) {
                __stcg(v.dz + idx, dz);
                if (i == 0) __stcg(v.z + idx, z);
            } else {
                __stcg(v.z + idx, z);
            }
        }
        if (!(ok = reduce(act ? r * z : 0.0, r * r, Two{}, [&](const double* t, double* out) {
                  out[0] = t[0];
                  out[1] = t[1];
                  out[2] = t[0] / rz;
              })))
            break;
        const double rzn = tot[0];
        rr = tot[1];
        if (!(rr == rr) || !(rzn == rzn) || rz == 0.0) done = 2;
        else if (rr <= tol2) done = 1;
        beta = tot[2];
        rz = rzn;
        it++;
    }
    // back to memory: the direction of iteration j goes where the next one reads it
    if (act) {
        v.x[idx] = xs[ot];
        v.r[idx] = r;
        v.z[idx] = z;
        const int par = (A.parity + n) & 1;
        v.p[par][idx] = p;
        if (F32) {
            v.dz[idx] = dz;
            v.dp[par][idx] = dp;
        }
    }
    if (!ok && threadIdx.x == 0) atomicExch(&v.S->gaveup, 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        PcgScalars* S = v.S;
        S->pap = pap;
        S->alpha = alpha;
        S->beta = beta;
        S->rz = rz;
        S->rr = rr;
        S->it = it;
        if (done) S->done = done;
    }
}

// warps per block that own rows, and blocks
void persist_shape(const IpdgArgs& a, int* owners, int* grid) {
    const int ew = 32 / a.Np, nwarps = (a.K + ew - 1) / ew, sms = std::min(a.sms, kMaxBlocks);
    *owners = (nwarps + sms - 1) / sms;
    *grid = (nwarps + *owners - 1) / *owners;
}

size_t coarse_smem(const MgLevels& m, int grid, int* vrows) {
    const int n0 = m.lv[0].n;
    *vrows = (n0 + grid - 1) / grid;
    return sizeof(double) * (size_t)n0 * (1 + *vrows) + sizeof(int) * (size_t)(n0 + 1);
}

template <int NP, typename T, bool MG>
cudaError_t launch_p(PersistArgs& A, cudaStream_t s) {
    int grid;
    persist_shape(A.a, &A.owners, &grid);
    // the coarse space is shared by eight warps a block, however few own rows
    const int nw = MG ? std::max(A.owners, 8) : A.owners;
    const size_t smem = PersistDims<T>::shared_bytes(NP, 32 * A.owners) + (MG ? coarse_smem(A.m, grid, &A.vrows) : 0);
    auto kernel = pcg_persist_kernel<NP, T, MG>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    void* args[] = {&A};
    return cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(32 * nw), args, smem, s);
}

template <int NP, typename T>
cudaError_t launch_t(PersistArgs& A, bool mg, cudaStream_t s) {
    return mg ? launch_p<NP, T, true>(A, s) : launch_p<NP, T, false>(A, s);
}

}  // namespace

// As many elements as the chip's registers hold: 152 blocks of 16 warps (FP32
// up to N = 4) or 8 warps, 32/Np elements a warp.  Where it fits it is the faster
// way at every size, so the line is the capacity.  Per iteration, one launch
// against the kernels of ipdg_block.cu / ipdg.cu: K = 4228, N = 4, FP32, block
// Jacobi 12 us (29 us); K = 1152, N = 3, FP64, coarse space of 617 vertices
// 23 us (37 us).  Bound by the latency of the exchanges (5 k cycles each: two
// trips through L2 of 1.2 k, three chains of FP64 additions) and by the FP64 pipe
// for a dozen FP64 operations per row.
bool persist_fits(const IpdgArgs& a, const PcgVecs& v, bool fp32) {
    if (v.zl || v.r32 || (v.zb && !v.mg)) return false;  // learned forms
    if (v.mg && v.mg->nl != 1) return false;
    const bool np = fp32 ? PersistDims<float>::fits(a.Np) : PersistDims<double>::fits(a.Np);
    if (!np) return false;
    int owners, grid, vrows;
    persist_shape(a, &owners, &grid);
    if (owners > (fp32 ? PersistDims<float>::warps(a.Np) : PersistDims<double>::warps(a.Np))) return false;
    const size_t own = fp32 ? PersistDims<float>::shared_bytes(a.Np, 32 * owners) : PersistDims<double>::shared_bytes(a.Np, 32 * owners);
    return own + (v.mg ? coarse_smem(*v.mg, grid, &vrows) : 0) <= 216 * 1024;
}

size_t persist_slots() { return sizeof(ulonglong2) * 2 * kSetSlots; }

cudaError_t launch_pcg_persistent(const IpdgArgs& a, const PcgVecs& v, bool fp32, const void* rows, double* corner,
                                  void* slots, unsigned long long* exchanges, int parity, int count, cudaStream_t s) {
    PersistArgs A{a, v, v.mg ? *v.mg : MgLevels(), rows, corner, parity, count, static_cast<ulonglong2*>(slots), *exchanges, 0, 0};
    *exchanges += 4ull * count + 4;  // at most four an iteration
    const bool mg = v.mg != nullptr;
    switch (a.Np) {
        case 3: return fp32 ? launch_t<3, float>(A, mg, s) : launch_t<3, double>(A, mg, s);
        case 6: return fp32 ? launch_t<6, float>(A, mg, s) : launch_t<6, double>(A, mg, s);
        case 10: return fp32 ? launch_t<10, float>(A, mg, s) : launch_t<10, double>(A, mg, s);
        case 15: return fp32 ? launch_t<15, float>(A, mg, s) : launch_t<15, double>(A, mg, s);
        case 21: return fp32 ? launch_t<21, float>(A, mg, s) : cudaErrorInvalidValue;
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace dgk
