// euler_split_pipe.cu -- the split-precision fused DG Euler stage,
// software-pipelined across tiles (sm_103a).  Arithmetic and operands: euler_split.cu.
//
// The FP64-pipe work of staging (one FP64 subtraction and conversion per staged value;
// GB300 retires two FP64 operations per clock per SM) and the memory latency of the
// epilogue leave the other pipes idle.  So tile t+1's phases are interleaved with tile
// t's, and no phase ends in a CTA barrier: sixteen compute warps hand over through
// mbarriers, each waiting only for what it is about to read or overwrite, and
// one thread of a warp of its own issues every MMA and bulk copy.
//
//   compute warps, prologue:  stage(t0); faces(t0)
//   per tile t (t+1 = the CTA's next tile):
//     wait GEMM1(t)
//     volume passes of t (TMEM -> FP32 flux -> chunk operand), with stage(t+1)
//       in slices between them: pass 0 waits for every warp to be through the
//       end of tile t-1 and forms t+1's reference state and metrics (after its
//       FP64 tile copy has landed), the later passes its FP32 deltas and TF32
//       operand
//     faces(t+1) up to the fluxes, wait GEMM2(t), the fluxes into the lift operand
//     R(t) TMEM -> shared, epilogue(t) (LSERK update, global stores), within the
//       four warps of 8 elements
//   issuer:  per volume pass of t its GEMM2 MMAs, the lift's with the last; once
//     t+1 is staged GEMM1(t+1) and the bulk copy of t+2's FP64 tile
//   the three warps beside the issuer:  t+1's neighbour traces (cp.async) when
//     the face phase of t has read its own
//
// The reference state, its FP64 copy and the metrics are double-buffered by
// tile parity; the FP64 tile buffer, the FP32 deltas, the GEMM1 operand and
// the neighbour traces are single-buffered because their readers (faces and
// GEMM1 of t) have finished before stage(t+1) writes them.  The stage input
// is re-read from L2 in the epilogue.  At N = 7 there is no FP64 tile buffer
// and no buffer of deltas (SplitDims): a volume pass reads what it stages from
// memory ahead of its fluxes, the face phase takes the deltas from the GEMM1
// operand, and the issuer streams the volume operator's slices.
//
// What bounds it: latency at 16 warps per SM.  With every computation, load and
// store taken out and only the hand-overs left, the stage with CTA barriers and an
// issuing thread among the compute warps took 214 of its 358 us (N = 5, K =
// 131,072, Lax-Friedrichs).  Per stage, K = 131,072, N = 1 .. 6, Lax-Friedrichs:
// 119, 156, 209, 277, 358, 451 us so; with an issuing warp and mbarriers 116, 144,
// 202, 277, 330, 410; with the wait for the other warps' face phase moved behind
// the first fluxes 111, 136, 199, 257, 307, 407; with the face fluxes in the
// wait for GEMM2 107, 130, 184, 236, 309, 395; with the traces requested by other
// warps (N <= 5) 105, 131, 181, 234, 296.  N = 7, K = 320,000, against a
// kernel with the phases one after another: Roe 1609 -> 1430, Lax-Friedrichs 1523 -> 1346.  Measured and left out: face fluxes
// in three warps of their own beside the issuer (359 us at N = 5, 320 at N = 4:
// a face is a long chain, and three warps do not keep up).
//
// Every mbarrier wait is bounded; after a timeout nobody waits any more, the
// status word is set, and the CTA lets its copies and MMAs in flight end before
// it frees tensor memory and returns.
#include <algorithm>
#include <cstdio>

#include "../../include/dgcu.h"
#include "euler_flux.cuh"
#include "euler_split.cuh"
#include "f64split.cuh"
#include "umma.cuh"

namespace dgk {

// Sixteen compute warps and a warpgroup whose first warp issues and whose others
// request the neighbour traces.  A launch gives
// every warp 96 registers; the compute warps take 104, which the second
// warpgroup leaves them: 16 * 104 + 4 * 64 = 20 * 96.
constexpr int kPipeThreads = 640, kComputeRegs = 104, kIssuerRegs = 64, kTraceWarps = 3;

template <int N>
struct PipeDims {
    using S = SplitDims<N>;
    static constexpr int al(int x) { return (x + 1023) / 1024 * 1024; }  // tensor-core operands
    static constexpr int a128(int x) { return (x + 127) / 128 * 128; }    // everything else
    static constexpr int OFF_B1 = 0;
    static constexpr int OFF_B2 = OFF_B1 + al(S::SZ_B1);
    static constexpr int OFF_BC = OFF_B2 + al(S::SZ_B2);  // N = 7: streamed [Sr | Ss] slices
    static constexpr int OFF_A1 = OFF_BC + (S::STREAM ? S::NBUF * S::AL_BC : 0);
    static constexpr int OFF_AC = OFF_A1 + al(S::SZ_A1);
    static constexpr int OFF_AF = OFF_AC + S::NBUF * S::AL_AC;
    static constexpr int OFF_QF = OFF_AF + al(S::SZ_AF);
    static constexpr int OFF_Q64 = OFF_QF + a128(S::SZ_QF);
    // per tile parity: reference state FP32 [ROWS], FP64 [ROWS], metrics FP32 [E][4]
    static constexpr int SZ_QB = S::ROWS * 4 + S::ROWS * 8 + S::E * 16;
    static constexpr int QB_STRIDE = (SZ_QB + 127) / 128 * 128;
    static constexpr int OFF_QB = OFF_Q64 + a128(S::SZ_Q64);
    static constexpr int OFF_NB = OFF_QB + 2 * QB_STRIDE;
    static constexpr bool GATHER = OFF_NB + a128(S::SZ_NB_FULL) + 128 <= 232448;
    static constexpr int SZ_NB = GATHER ? S::SZ_NB_FULL : 0;
    static constexpr int OFF_BAR = OFF_NB + a128(SZ_NB);
    static constexpr int SMEM = OFF_BAR + 128;
    static_assert(SMEM <= 232448, "shared memory budget");
    // volume passes (two chunks per pass where there are two chunk buffers)
    static constexpr int NPASS = S::PAIR ? (S::NCH + 1) / 2 : S::NCH;
    // FP32 deltas of a tile per thread, and how they are spread over the passes
    // one core matrix of the GEMM1 operand per warp and step: warp w holds
    // rows 8w .. 8w + 7, lane = 4 (row % 8) + (k % 4), KP1 / 4 steps along K
    static constexpr int NDQ = S::KP1 / 4;
    static_assert(S::THREADS == 512 && S::ROWS == 128, "16 warps x 8 rows");
    static_assert(!S::STREAM || (S::NBUF == 2 && S::NCH % 2 == 0), "slices alternate like the chunk buffers");
    static constexpr int DQ_SLICES = NPASS > 1 ? NPASS - 1 : 1;
    static constexpr int DQ_PER = (NDQ + DQ_SLICES - 1) / DQ_SLICES;
};

// The stage for the tiles bid, bid + nblk, ... of one context (a CTA of
// kPipeThreads threads); the single-context kernel runs it with its own block index and
// grid size, the mixed-order batch kernel with its share of the grid.
template <int N>
__device__ __forceinline__ void pipe_body(const SplitArgs& sa, const int bid, const int nblk) {
    using S = SplitDims<N>;
    using D = PipeDims<N>;
    constexpr int Np = S::Np, Ng = S::Ng, Nfp = S::Nfp, Nfq = S::Nfq, E = S::E;
    constexpr int KP1 = S::KP1, NG = S::NG, NF = S::NF, NP2 = S::NP2, KP2 = S::KP2, CH = S::CH, KC = S::KC;
    constexpr int NB = 3 * N;
    extern __shared__ __align__(1024) unsigned char smem[];
    float* sB1 = reinterpret_cast<float*>(smem + D::OFF_B1);
    float* sB2 = reinterpret_cast<float*>(smem + D::OFF_B2);
    float* sA1 = reinterpret_cast<float*>(smem + D::OFF_A1);
    float* sAF = reinterpret_cast<float*>(smem + D::OFF_AF);
    float* sQF = reinterpret_cast<float*>(smem + D::OFF_QF);
    double* sQ64 = reinterpret_cast<double*>(smem + D::OFF_Q64);
    double* sNB = reinterpret_cast<double*>(smem + D::OFF_NB);
    float* sRS = reinterpret_cast<float*>(smem + D::OFF_AC);  // after GEMM2 completed
    uint64_t* bar1 = reinterpret_cast<uint64_t*>(smem + D::OFF_BAR);  // GEMM1 done
    uint64_t* bar2 = bar1 + 1;     // [NBUF] the chunk's MMAs done
    uint64_t* bq = bar1 + 3;       // the FP64 tile copy has landed
    uint64_t* bready = bar1 + 4;   // [2] a volume pass is in the chunk buffers (N = 7: in chunk buffer b)
    uint64_t* bstaged = bar1 + 6;  // the next tile is staged; its predecessor's D1 and the tile copy are read
    uint64_t* bfaces = bar1 + 7;   // the tile's face fluxes are in place; traces, deltas and staged results are read
    uint64_t* bfin = bar1 + 8;
    uint64_t* bfull = bar1 + 9;    // [2] N = 7: the operator slice has landed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar1 + 11);
    volatile int* dead = reinterpret_cast<volatile int*>(bar1 + 12);  // a wait timed out: nobody waits any more
    // reference state / metrics of tile parity b
    auto qbf = [&](int b) { return reinterpret_cast<float*>(smem + D::OFF_QB + b * D::QB_STRIDE); };
    auto qbd = [&](int b) {
        return reinterpret_cast<double*>(smem + D::OFF_QB + b * D::QB_STRIDE + S::ROWS * 4);
    };
    auto geo = [&](int b) {
        return reinterpret_cast<float*>(smem + D::OFF_QB + b * D::QB_STRIDE + S::ROWS * 12);
    };

    const EulerArgs& a = sa.e;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = (a.K + E - 1) / E;
    const float gamma = (float)a.gamma;
    const int G = nblk;

    auto wait = [&](uint64_t* bar, uint32_t phase) {
        if (*dead) return;
        if (!umma::mbar_wait(bar, phase, kWaitLimit)) *dead = 1;
    };
    auto arrive = [&](uint64_t* bar) {
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(bar);
    };

    // neighbour traces of a tile's faces into sNB by 8-byte asynchronous copies
    // (the neighbour element's node in its own face order with the rotation
    // applied, or the boundary slot's trace); cn[j]: the face link of this
    // thread's task j, loaded ahead
    constexpr int FT = 32 * kTraceWarps, GT = (3 * E * Nfp + FT - 1) / FT;
    const int ft = tid - 17 * 32;
    int cn[GT];
    auto load_links = [&](int t) {
#pragma unroll
        for (int j = 0; j < GT; j++) {
            const int i = ft + j * FT;
            cn[j] = (t < ntiles && i < 3 * min(E, a.K - t * E) * Nfp) ? __ldg(a.conn + (size_t)t * E * 3 + i / Nfp) : 0;
        }
    };
    auto gather = [&](int t) {
        const int kt = t * E;
        const int nt = 3 * min(E, a.K - kt) * Nfp;
#pragma unroll
        for (int j = 0; j < GT; j++) {
            const int i = ft + j * FT;
            if (i >= nt) break;
            const int ef = i / Nfp, ii = i - ef * Nfp;
            const int c = cn[j];
            const double* src;
            int vstride;
            if (c >= 0) {
                const int nb = c >> 3, fn = c & 3, rot = (c >> 2) & 1;
                const int jj = rot ? (N - ii) : ii;
                src = a.qin + (size_t)nb * 4 * Np + (fn * N + jj) % NB;
                vstride = Np;
            } else {
                src = a.btrace + (size_t)(-1 - c) * 4 * Nfp + ii;
                vstride = Nfp;
            }
            double* dst = sNB + (size_t)i * 4;
#pragma unroll
            for (int v = 0; v < 4; v++) umma::cp_async8(dst + v, src + v * vstride);
        }
    };

    // N = 7: no FP64 tile copy; what a volume pass stages is read from memory ahead
    // of its fluxes
    double pre[S::STREAM ? (D::DQ_PER > 3 ? D::DQ_PER : 3) : 1];
    float pgeo = 0.f;
    // the rows and K offsets of this thread in the core-matrix mapping
    const int cm_r = 8 * warp + (lane >> 2), cm_k = lane & 3;
    auto fetch_ref = [&](int t) {
        if constexpr (S::STREAM) {
            const int k0t = t * E, net = min(E, a.K - k0t), r = 8 * warp + (lane & 7);
            if (lane < 8 && (r >> 2) < net) {
                const double* row = a.qin + (size_t)k0t * 4 * Np + (size_t)r * Np;
#pragma unroll
                for (int j = 0; j < 3; j++) pre[j] = __ldg(row + j * N);
            } else if (lane >= 8 && lane < 16 && (r >> 2) < net) {
                pgeo = (float)a.geo[(size_t)(k0t + (r >> 2)) * 4 + (r & 3)];
            }
        }
    };
    auto fetch_dq = [&](int t, int j0, int j1) {
        if constexpr (S::STREAM) {
            const int net = min(E, a.K - t * E);
            const double* src = a.qin + (size_t)t * E * 4 * Np + (size_t)cm_r * Np + cm_k;
#pragma unroll
            for (int j = 0; j < D::DQ_PER; j++)
                if (j0 + j < j1 && cm_r < 4 * net && 4 * (j0 + j) + cm_k < Np) pre[j] = __ldg(src + 4 * (j0 + j));
        }
    };
    // stage, part 1: the reference state (mean of the three vertex values,
    // FP32 and its FP64 copy) and FP32 metrics of the warp's two elements of tile t
    // into parity b; the tile's FP64 copy must have landed
    auto stage_ref = [&](int t, int b) {
        const int k0t = t * E, net = min(E, a.K - k0t);
        if (lane < 8) {
            const int r = 8 * warp + lane, e = r >> 2;
            float qb = 1.f;
            if (e < net) {
                if constexpr (S::STREAM) {
                    qb = (f64s::trunc_f32(pre[0]) + f64s::trunc_f32(pre[1]) + f64s::trunc_f32(pre[2])) * (1.f / 3.f);
                } else {
                    const double* row = sQ64 + r * Np;  // ring order: vertices at 0, N, 2N
                    qb = (float)((row[0] + row[N] + row[2 * N]) * (1.0 / 3.0));
                }
            }
            qbf(b)[r] = qb;
            if constexpr (!S::STREAM) qbd(b)[r] = (double)qb;
        } else if (lane < 16) {
            const int i = 8 * warp + lane - 8, e = i >> 2;
            if constexpr (S::STREAM) geo(b)[i] = e < net ? pgeo : 0.f;
            else geo(b)[i] = e < net ? (float)a.geo[(size_t)(k0t + e) * 4 + (i & 3)] : 0.f;
        }
        __syncwarp();
    };
    // stage, part 2: FP32 deltas (this thread's items j0 <= j < j1) into sQF and
    // their TF32 hi / lo into the GEMM1 operand (N = 7: only there, hi + lo is exact;
    // by integer and FP32 operations, f64split.cuh)
    constexpr uint32_t LO_A1 = 128 * KP1 * 4;
    auto stage_dq = [&](int t, int b, int j0, int j1) {
        const int net = min(E, a.K - t * E);
        if (cm_r >= 4 * net) return;  // rows of a missing element (tail tile)
        float* dst = sA1 + (warp * (KP1 / 4)) * 32 + lane;
        if constexpr (S::STREAM) {
            const float qr = qbf(b)[cm_r];
#pragma unroll
            for (int j = 0; j < D::DQ_PER; j++)
                if (j0 + j < j1 && 4 * (j0 + j) + cm_k < Np) {
                    float hi, lo;
                    umma::split_tf32(f64s::minus_f32(pre[j], qr), hi, lo);
                    dst[32 * (j0 + j)] = hi;
                    dst[32 * (j0 + j) + LO_A1 / 4] = lo;
                }
        } else {
            const double qr = qbd(b)[cm_r];
            const double* src = sQ64 + cm_r * Np + cm_k;
            float* qf = sQF + cm_r * Np + cm_k;
#pragma unroll
            for (int j = j0; j < j1; j++) {
                if (j < D::NDQ && 4 * j + cm_k < Np) {
                    const float d = (float)(src[4 * j] - qr);
                    qf[4 * j] = d;
                    float hi, lo;
                    umma::split_tf32(d, hi, lo);
                    dst[32 * j] = hi;
                    dst[32 * j + LO_A1 / 4] = lo;
                }
            }
        }
    };

    // constant operands and zero padding, once per CTA
    {
        const int4* src1 = reinterpret_cast<const int4*>(sa.b1);
        int4* dst1 = reinterpret_cast<int4*>(sB1);
        for (int i = tid; i < S::SZ_B1 / 16; i += blockDim.x) dst1[i] = src1[i];
        const int4* src2 = reinterpret_cast<const int4*>(sa.b2);
        int4* dst2 = reinterpret_cast<int4*>(sB2);
        for (int i = tid; i < S::SZ_B2 / 16; i += blockDim.x) dst2[i] = src2[i];
        for (int i = tid; i < S::SZ_A1 / 4; i += blockDim.x) sA1[i] = 0.f;
        for (int i = tid; i < S::SZ_AF / 4; i += blockDim.x) sAF[i] = 0.f;
    }
    const int t0 = bid;
    if (tid == 0) {
        umma::mbar_init(bar1, 1);
        for (int b = 0; b < S::NBUF; b++) umma::mbar_init(bar2 + b, 1);
        umma::mbar_init(bq, 1);
        for (int b = 0; b < 2; b++) {
            umma::mbar_init(bready + b, 16);
            umma::mbar_init(bfull + b, 1);
        }
        umma::mbar_init(bstaged, 16 + (D::GATHER ? kTraceWarps : 0));
        umma::mbar_init(bfaces, 16);
        umma::mbar_init(bfin, 1);
        *dead = 0;
        umma::fence_mbar_init();
    }
    if (warp == 16) {
        umma::tmem_alloc(tmem_slot, S::TMEM_COLS);
        umma::tmem_relinquish();
    }
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tD1 = tmem, tD2 = tmem + S::D2_COL;
    const uint32_t idesc1 = umma::idesc_tf32(128, NG);
    const uint32_t idesc2 = umma::idesc_tf32(128, NP2);
    const uint32_t aB1 = umma::smem_u32(sB1), aB2 = umma::smem_u32(sB2);
    const uint32_t aA1 = umma::smem_u32(sA1), aAF = umma::smem_u32(sAF);
    const uint32_t aAC = umma::smem_u32(smem + D::OFF_AC);
    const uint32_t aBC = umma::smem_u32(smem + D::OFF_BC);
    constexpr uint32_t LO_B1 = NG * KP1 * 4, LO_B2 = S::SZ_B2 / 2, LO_AC = 128 * KC * 4, LO_AF = 128 * NF * 4,
                       STRIDE_AC = S::AL_AC;
    const int qd = warp & 3, sub = warp >> 2;
    const int my_e = 8 * qd + (lane >> 2), my_v = lane & 3;

    // face fluxes of tile t (reference state / metrics of parity b) into the
    // lift operand sAF; the neighbour traces are in sNB (GATHER) or are loaded
    // here; operand_free() before the first store
    auto faces = [&](int t, int b, auto operand_free) {
        const int k0 = t * E, ne = min(E, a.K - k0);
        const float* sQB = qbf(b);
        const double* sQBd = qbd(b);
        const float* sGeo = geo(b);
        if constexpr (S::FP == 2) {
            // N = 4..6: one (element, face) per segment of FW = ceil(Nfq / 2)
            // lanes; lane li = face nodes li, li + FW and Gauss points li, li + FW
            constexpr int FW = S::FW, FPW = S::FPW;
            const int seg = lane / FW, li = lane - seg * FW;  // lanes with seg >= FPW idle
            const int sbase = (seg < FPW ? seg : 0) * FW;
            const int Gf = warp * FPW + seg;
            const bool gok = seg < FPW && Gf < 3 * E;
            const int Gc = gok ? Gf : min(warp * FPW, 3 * E - 1);
            const int e = Gc / 3, f = Gc - 3 * e;
            const bool valid = gok && e < ne;
            [[maybe_unused]] const int k = k0 + (valid ? e : 0);
            float qbv[4];
            double qbdv[4];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                qbv[v] = sQB[4 * (valid ? e : 0) + v];
                qbdv[v] = S::STREAM ? 0.0 : sQBd[4 * (valid ? e : 0) + v];
            }
            float own[2][4], nbr[2][4];
#pragma unroll
            for (int sl = 0; sl < 2; sl++) {
                const int i = li + sl * FW;
#pragma unroll
                for (int v = 0; v < 4; v++) own[sl][v] = nbr[sl][v] = 0.f;
                if (valid && i < Nfp) {
                    const int pos = (f * N + i) % NB;
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        if constexpr (S::STREAM) {
                            const uint32_t off = umma::kmajor_offset(4 * e + v, pos, KP1) >> 2;
                            own[sl][v] = sA1[off] + sA1[off + LO_A1 / 4];
                        } else {
                            own[sl][v] = sQF[e * 4 * Np + v * Np + pos];
                        }
                    }
                    if constexpr (D::GATHER) {
                        const double* nv = sNB + (size_t)((3 * e + f) * Nfp + i) * 4;
#pragma unroll
                        for (int v = 0; v < 4; v++) nbr[sl][v] = f64s::minus_f32(nv[v], qbv[v]);
                    } else {
                        const int c = __ldg(a.conn + (size_t)k * 3 + f);
                        const double* src;
                        int vs;
                        if (c >= 0) {
                            const int nb = c >> 3, fn = c & 3, rot = (c >> 2) & 1;
                            const int jj = rot ? (N - i) : i;
                            src = a.qin + (size_t)nb * 4 * Np + (fn * N + jj) % NB;
                            vs = Np;
                        } else {
                            src = a.btrace + (size_t)(-1 - c) * 4 * Nfp + i;
                            vs = Nfp;
                        }
#pragma unroll
                        for (int v = 0; v < 4; v++)
                            nbr[sl][v] = S::STREAM ? f64s::minus_f32(__ldg(src + v * vs), qbv[v])
                                                   : (float)(__ldg(src + v * vs) - qbdv[v]);
                    }
                }
            }
            float dm[2][4], dp[2][4];
            int gi[2];
#pragma unroll
            for (int sl = 0; sl < 2; sl++) {
                gi[sl] = (li + sl * FW < Nfq) ? li + sl * FW : 0;
#pragma unroll
                for (int v = 0; v < 4; v++) dm[sl][v] = dp[sl][v] = 0.f;
            }
#pragma unroll
            for (int jn = 0; jn < Nfp; jn++) {
                const int src = sbase + jn % FW;
                const float w0 = __ldg(sa.If32 + gi[0] * Nfp + jn);
                const float w1 = __ldg(sa.If32 + gi[1] * Nfp + jn);
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const float om = __shfl_sync(0xffffffffu, own[jn / FW][v], src);
                    const float op = __shfl_sync(0xffffffffu, nbr[jn / FW][v], src);
                    dm[0][v] = fmaf(w0, om, dm[0][v]);
                    dp[0][v] = fmaf(w0, op, dp[0][v]);
                    dm[1][v] = fmaf(w1, om, dm[1][v]);
                    dp[1][v] = fmaf(w1, op, dp[1][v]);
                }
            }
            const float* gk = sGeo + 4 * (valid ? e : 0);
            float nx, ny, fsc;
            face_normal_f(f, gk[0], gk[1], gk[2], gk[3], nx, ny, fsc);
            const RefState rb = make_ref(gamma, qbv);
            DeltaPrim pm[2], pp[2];
#pragma unroll
            for (int sl = 0; sl < 2; sl++) {
                pm[sl] = delta_prim(gamma, rb, dm[sl]);
                pp[sl] = delta_prim(gamma, rb, dp[sl]);
            }
            float F[2][4];
            if (a.flux == 1) {
#pragma unroll
                for (int sl = 0; sl < 2; sl++) roe_flux_delta(gamma, nx, ny, rb, dm[sl], pm[sl], dp[sl], pp[sl], F[sl]);
            } else {
                float lam = 0.f;
#pragma unroll
                for (int sl = 0; sl < 2; sl++)
                    if (li + sl * FW < Nfq)
                        lam = fmaxf(lam, fmaxf(wave_speed_delta(gamma, nx, ny, rb, pm[sl]),
                                               wave_speed_delta(gamma, nx, ny, rb, pp[sl])));
                float m = lam;
#pragma unroll
                for (int j = 0; j < FW; j++) m = fmaxf(m, __shfl_sync(0xffffffffu, lam, sbase + j));
#pragma unroll
                for (int sl = 0; sl < 2; sl++) lf_flux_delta(nx, ny, m, rb, dm[sl], pm[sl], dp[sl], pp[sl], F[sl]);
            }
            operand_free();
#pragma unroll
            for (int sl = 0; sl < 2; sl++) {
                const int g = li + sl * FW;
                if (valid && g < Nfq) {
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        float hi, lo;
                        umma::split_tf32(__fmul_rn(-0.5f * fsc, F[sl][v]), hi, lo);
                        const uint32_t off = umma::kmajor_offset(g2row(e, v), f * Nfq + g, NF) >> 2;
                        sAF[off] = hi;
                        sAF[off + LO_AF / 4] = lo;
                    }
                }
            }
        } else {
            // one (element, face) per segment of SW lanes, lane i = face node i
            // (gather) and face Gauss point i (flux)
            constexpr int SW = S::SW, SPW = S::SPW;
            const int seg = lane / SW, i = lane - seg * SW;  // lanes with seg >= SPW idle
            const int sbase = (seg < SPW ? seg : 0) * SW;
            static_assert(S::THREADS / 32 * SPW >= 3 * E, "one pass over the faces");
            {
                const int gbase = warp * SPW < 3 * E ? warp * SPW : 3 * E - 1;
                const int Gf = gbase + seg;
                const bool gok = seg < SPW && Gf < 3 * E && warp * SPW < 3 * E;
                const int Gc = gok ? Gf : gbase;
                const int e = Gc / 3, f = Gc - 3 * e;
                const bool valid = gok && e < ne;
                [[maybe_unused]] const int k = k0 + (valid ? e : 0);
                float own[4] = {0.f, 0.f, 0.f, 0.f}, nbr[4] = {0.f, 0.f, 0.f, 0.f};
                float qbv[4];
                double qbdv[4];
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    qbv[v] = sQB[4 * (valid ? e : 0) + v];
                    qbdv[v] = sQBd[4 * (valid ? e : 0) + v];
                }
                if (valid && i < Nfp) {
                    const int pos = (f * N + i) % NB;
#pragma unroll
                    for (int v = 0; v < 4; v++) own[v] = sQF[e * 4 * Np + v * Np + pos];
                    if constexpr (D::GATHER) {
                        const double* nv = sNB + (size_t)((3 * e + f) * Nfp + i) * 4;
#pragma unroll
                        for (int v = 0; v < 4; v++) nbr[v] = f64s::minus_f32(nv[v], qbv[v]);
                    } else {
                        const int c = __ldg(a.conn + (size_t)k * 3 + f);
                        if (c >= 0) {
                            const int nb = c >> 3, fn = c & 3, rot = (c >> 2) & 1;
                            const int jj = rot ? (N - i) : i;
                            const double* qn = a.qin + (size_t)nb * 4 * Np + (fn * N + jj) % NB;
#pragma unroll
                            for (int v = 0; v < 4; v++) nbr[v] = (float)(__ldg(qn + v * Np) - qbdv[v]);
                        } else {
                            const double* bt = a.btrace + (size_t)(-1 - c) * 4 * Nfp + i;
#pragma unroll
                            for (int v = 0; v < 4; v++) nbr[v] = (float)(__ldg(bt + v * Nfp) - qbdv[v]);
                        }
                    }
                }
                float dm[4] = {0.f, 0.f, 0.f, 0.f}, dp[4] = {0.f, 0.f, 0.f, 0.f};
                const int gi = i < Nfq ? i : 0;
#pragma unroll
                for (int jn = 0; jn < Nfp; jn++) {
                    const float w = __ldg(sa.If32 + gi * Nfp + jn);
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        if constexpr (S::PACKED) {
                            dm[v] = fmaf(w, __shfl_sync(0xffffffffu, own[v], sbase + jn), dm[v]);
                            dp[v] = fmaf(w, __shfl_sync(0xffffffffu, nbr[v], sbase + jn), dp[v]);
                        } else {
                            dm[v] = fmaf(w, __shfl_sync(0xffffffffu, own[v], jn, SW), dm[v]);
                            dp[v] = fmaf(w, __shfl_sync(0xffffffffu, nbr[v], jn, SW), dp[v]);
                        }
                    }
                }
                const float* gk = sGeo + 4 * (valid ? e : 0);
                float nx, ny, fsc;
                face_normal_f(f, gk[0], gk[1], gk[2], gk[3], nx, ny, fsc);
                const RefState rb = make_ref(gamma, qbv);
                const DeltaPrim pm = delta_prim(gamma, rb, dm), pp = delta_prim(gamma, rb, dp);
                float F[4];
                if (a.flux == 1) {
                    roe_flux_delta(gamma, nx, ny, rb, dm, pm, dp, pp, F);
                } else {
                    float lam = (i < Nfq) ? fmaxf(wave_speed_delta(gamma, nx, ny, rb, pm),
                                                  wave_speed_delta(gamma, nx, ny, rb, pp))
                                          : 0.f;
                    if constexpr (S::PACKED) {
                        float m = lam;
#pragma unroll
                        for (int j = 0; j < Nfq; j++) m = fmaxf(m, __shfl_sync(0xffffffffu, lam, sbase + j));
                        lam = m;
                    } else {
#pragma unroll
                        for (int o = 1; o < SW; o <<= 1) lam = fmaxf(lam, __shfl_xor_sync(0xffffffffu, lam, o, SW));
                    }
                    lf_flux_delta(nx, ny, lam, rb, dm, pm, dp, pp, F);
                }
                operand_free();
                if (valid && i < Nfq) {
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        float hi, lo;
                        umma::split_tf32(__fmul_rn(-0.5f * fsc, F[v]), hi, lo);
                        const uint32_t off = umma::kmajor_offset(g2row(e, v), f * Nfq + i, NF) >> 2;
                        sAF[off] = hi;
                        sAF[off + LO_AF / 4] = lo;
                    }
                }
            }
        }
    };

    if (warp >= 16) {
        // ------------------------------------------------------------ tensor-core issuer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssuerRegs));
        if (warp > 16) {
            // ---------------------------------------------------- neighbour traces
            if constexpr (D::GATHER) {
                uint32_t phf = 0;
                if (t0 < ntiles) {
                    load_links(t0);
                    gather(t0);
                    load_links(t0 + G);
                    umma::cp_async_wait_all();
                    arrive(bstaged);
                }
#pragma unroll 1
                for (int tn = t0 + G; tn < ntiles; tn += G) {
                    // every warp has read the traces of the tile before; these land during
                    // its volume phase
                    wait(bfaces, phf);
                    phf ^= 1;
                    gather(tn);
                    load_links(tn + G);
                    umma::cp_async_wait_all();
                    arrive(bstaged);
                }
            }
        } else if (lane == 0) {
            auto issue_gemm1 = [&]() {
#pragma unroll
                for (int s = 0; s < KP1 / 8; s++) {
                    const uint64_t ah = umma::smem_desc(aA1 + s * 256, 128, (KP1 / 4) * 128);
                    const uint64_t al = umma::smem_desc(aA1 + LO_A1 + s * 256, 128, (KP1 / 4) * 128);
                    const uint64_t bh = umma::smem_desc(aB1 + s * 256, 128, (KP1 / 4) * 128);
                    const uint64_t bl = umma::smem_desc(aB1 + LO_B1 + s * 256, 128, (KP1 / 4) * 128);
                    umma::mma_tf32(tD1, ah, bh, idesc1, s > 0);
                    umma::mma_tf32(tD1, al, bh, idesc1, 1);
                    umma::mma_tf32(tD1, ah, bl, idesc1, 1);
                }
                umma::commit(bar1);
            };
            auto issue_mma = [&](int ch, int buf, int slice) {
                constexpr uint32_t sboA = (KC / 4) * 128, sboB = (KP2 / 4) * 128;
                const uint32_t aC = aAC + buf * STRIDE_AC;
#pragma unroll
                for (int s = 0; s < KC / 8; s++) {
                    const uint64_t ah = umma::smem_desc(aC + s * 256, 128, sboA);
                    const uint64_t al = umma::smem_desc(aC + LO_AC + s * 256, 128, sboA);
                    uint64_t bh, bl;
                    if constexpr (S::STREAM) {
                        // the streamed slice has the chunk's own K layout [Sr 16 | Ss 16]
                        const uint32_t bC = aBC + slice * S::AL_BC;
                        bh = umma::smem_desc(bC + s * 256, 128, sboA);
                        bl = umma::smem_desc(bC + S::SZ_BC / 2 + s * 256, 128, sboA);
                    } else {
                        const int kb = (s < CH / 8) ? (ch * CH + 8 * s) : (NG + ch * CH + 8 * (s - CH / 8));
                        bh = umma::smem_desc(aB2 + kb * 32, 128, sboB);
                        bl = umma::smem_desc(aB2 + LO_B2 + kb * 32, 128, sboB);
                    }
                    const uint32_t acc = (ch > 0 || s > 0) ? 1u : 0u;
                    umma::mma_tf32(tD2, ah, bh, idesc2, acc);
                    umma::mma_tf32(tD2, al, bh, idesc2, 1);
                    umma::mma_tf32(tD2, ah, bl, idesc2, 1);
                }
                if (ch == S::NCH - 1) {
                    constexpr uint32_t sboF = (NF / 4) * 128;
#pragma unroll
                    for (int s = 0; s < NF / 8; s++) {
                        // lift part: k = 2 NG + 8 s of the resident image, or k = 8 s of the lift's own
                        const int kb = S::STREAM ? 8 * s : 2 * NG + 8 * s;
                        constexpr uint32_t sbo = S::STREAM ? sboF : sboB;
                        const uint64_t ah = umma::smem_desc(aAF + s * 256, 128, sboF);
                        const uint64_t al = umma::smem_desc(aAF + LO_AF + s * 256, 128, sboF);
                        const uint64_t bh = umma::smem_desc(aB2 + kb * 32, 128, sbo);
                        const uint64_t bl = umma::smem_desc(aB2 + LO_B2 + kb * 32, 128, sbo);
                        umma::mma_tf32(tD2, ah, bh, idesc2, 1);
                        umma::mma_tf32(tD2, al, bh, idesc2, 1);
                        umma::mma_tf32(tD2, ah, bl, idesc2, 1);
                    }
                }
                umma::commit(bar2 + buf);
            };
            int nq = 0;  // tile copies issued
            auto issue_q = [&](int t) {
                if (S::STREAM || t >= ntiles || *dead) return;
                const int k0t = t * E;
                const uint32_t bytes = (uint32_t)min(E, a.K - k0t) * 4u * (uint32_t)Np * 8u;
                umma::mbar_arrive_expect_tx(bq, bytes);
                umma::bulk_g2s(sQ64, a.qin + (size_t)k0t * 4 * Np, bytes, bq);
                nq++;
            };
            uint32_t phr = 0, phs = 0;
            // the staged tile's GEMM1; the tile after it into the FP64 buffer
            auto next = [&](int t) {
                wait(bstaged, phs);
                phs ^= 1;
                if (*dead) return;
                umma::fence_after_sync();
                issue_gemm1();
                issue_q(t + G);
            };
            // N = 7: slices of the operator, one per chunk and again for every tile, in two
            // buffers; g counts them
            const int mine = t0 < ntiles ? (ntiles - t0 + G - 1) / G * S::NCH : 0;
            int nsl = 0;
            uint32_t ph2i = 0;
            auto issue_slice = [&]() {
                if (nsl >= mine || *dead) return;
                const int b = nsl & 1;
                umma::mbar_arrive_expect_tx(bfull + b, S::SZ_BC);
                umma::bulk_g2s(smem + D::OFF_BC + b * S::AL_BC, sa.b2 + S::SZ_B2 / 4 + (size_t)(nsl % S::NCH) * (S::SZ_BC / 4),
                               S::SZ_BC, bfull + b);
                nsl++;
            };
            issue_q(t0);
            if constexpr (S::STREAM) {
                issue_slice();
                issue_slice();
            }
            if (t0 < ntiles) next(t0);
            int g = 0;
#pragma unroll 1
            for (int tile = t0; tile < ntiles && !*dead; tile += G) {
#pragma unroll 1
                for (int p = 0; p < D::NPASS; p++) {
                    const int buf = S::STREAM ? p & 1 : 0;
                    wait(bready + buf, (phr >> buf) & 1u);
                    phr ^= 1u << buf;
                    if constexpr (S::STREAM) wait(bfull + (g & 1), (uint32_t)(g >> 1) & 1u);
                    if (*dead) break;
                    umma::fence_after_sync();
                    if constexpr (S::PAIR) {
                        issue_mma(2 * p, 0, 0);
                        if (2 * p + 1 < S::NCH) issue_mma(2 * p + 1, 1, 0);
                    } else {
                        issue_mma(p, buf, S::STREAM ? g & 1 : 0);
                    }
                    if constexpr (S::STREAM) {
                        // the MMAs before these are through with their slice: the next one into its place
                        if (g > 0) {
                            const int o = buf ^ 1;
                            wait(bar2 + o, (ph2i >> o) & 1u);
                            ph2i ^= 1u << o;
                            issue_slice();
                        }
                        g++;
                    }
                }
                if (tile + G < ntiles) next(tile + G);
            }
            // everything issued ends before the CTA does
            umma::commit(bfin);
            if (!umma::mbar_wait(bfin, 0, kWaitLimit)) *dead = 1;
            if (*dead) {
                if (nq) umma::mbar_wait(bq, (uint32_t)(nq - 1) & 1u, kWaitLimit);
                for (int q = max(0, nsl - 2); q < nsl; q++) umma::mbar_wait(bfull + (q & 1), (uint32_t)(q >> 1) & 1u, kWaitLimit);
            }
        }
        __syncwarp();
    } else {
    // ---------------------------------------------------------------- compute warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kComputeRegs));
    uint32_t pq = 0, ph1 = 0, phs = 0, phf = 0;
    uint32_t ph2 = 0;  // bit b: phase parity of chunk buffer b's MMA barrier
    // tile t is staged: its operand, deltas and traces
    auto staged = [&]() {
        umma::fence_async_smem();
        umma::fence_before_sync();
        arrive(bstaged);
    };
    auto face_phase = [&](int t, int b, auto operand_free) {
        wait(bstaged, phs);
        phs ^= 1;
        faces(t, b, operand_free);
        umma::fence_async_smem();
    };
    // ---- prologue: stage and face fluxes of the first tile
    if (t0 < ntiles) {
        if constexpr (S::STREAM) {
            fetch_ref(t0);
            stage_ref(t0, 0);
#pragma unroll 1
            for (int j = 0; j < D::NDQ; j += D::DQ_PER) {
                fetch_dq(t0, j, min(D::NDQ, j + D::DQ_PER));
                stage_dq(t0, 0, j, min(D::NDQ, j + D::DQ_PER));
            }
        } else {
            wait(bq, pq);
            pq ^= 1;
            stage_ref(t0, 0);
            stage_dq(t0, 0, 0, D::NDQ);
        }
        staged();
        face_phase(t0, 0, []() {});
        arrive(bfaces);
    }

    int par = 0;  // parity of the current tile's reference-state buffer
#pragma unroll 1
    for (int tile = t0; tile < ntiles; tile += G, par ^= 1) {
        const int k0 = tile * E;
        const int ne = min(E, a.K - k0);
        const int tn = tile + G;  // this CTA's next tile
        const bool has_next = tn < ntiles;
        // ---- GEMM1(t)
        wait(bar1, ph1);
        ph1 ^= 1;
        umma::fence_after_sync();
        // per-thread element data for the volume flux
        float qbe[4];
#pragma unroll
        for (int v = 0; v < 4; v++) qbe[v] = qbf(par)[4 * my_e + v];
        const RefState bref = make_ref(gamma, qbe);
        const float* gcur = geo(par);
        const float rx = gcur[4 * my_e], sx = gcur[4 * my_e + 1], ry = gcur[4 * my_e + 2], sy = gcur[4 * my_e + 3];

        auto vol_flux = [&](const float* x, int ch, float* fr, float* fs) {
            // the 4 variables at point (sub*4 + my_v): a 4 x 4 transpose across the
            // element's 4 lanes in two butterfly stages (lane bit 1, then bit 0)
            float dq[4] = {x[0], x[1], x[2], x[3]};
            {
                const bool bb = (my_v & 2) != 0;
                const float r0 = __shfl_xor_sync(0xffffffffu, bb ? dq[0] : dq[2], 2);
                const float r1 = __shfl_xor_sync(0xffffffffu, bb ? dq[1] : dq[3], 2);
                dq[0] = bb ? r0 : dq[0];
                dq[1] = bb ? r1 : dq[1];
                dq[2] = bb ? dq[2] : r0;
                dq[3] = bb ? dq[3] : r1;
            }
            {
                const bool bb = (my_v & 1) != 0;
                const float r0 = __shfl_xor_sync(0xffffffffu, bb ? dq[0] : dq[1], 1);
                const float r1 = __shfl_xor_sync(0xffffffffu, bb ? dq[2] : dq[3], 1);
                dq[0] = bb ? r0 : dq[0];
                dq[2] = bb ? r1 : dq[2];
                dq[1] = bb ? dq[1] : r0;
                dq[3] = bb ? dq[3] : r1;
            }
            const int g = ch * CH + sub * 4 + my_v;
            if (g < Ng && my_e < ne) {
                const DeltaPrim d = delta_prim(gamma, bref, dq);
                float fx[4], fy[4];
                flux_delta(bref, dq, d, fx, fy);
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    fr[v] = fmaf(ry, fy[v], __fmul_rn(rx, fx[v]));
                    fs[v] = fmaf(sy, fy[v], __fmul_rn(sx, fx[v]));
                }
            } else {
#pragma unroll
                for (int v = 0; v < 4; v++) fr[v] = fs[v] = 0.f;
            }
        };
        // this thread's slots in a chunk operand: rows g2row(my_e, v) are one
        // 8-row group apart per v (KC * 8 floats), the Fs columns CH / 4 core
        // matrices after the Fr ones, so every store is a fixed offset from one base
        float* const sAC0 =
            reinterpret_cast<float*>(smem + D::OFF_AC) + (umma::kmajor_offset(g2row(my_e, 0), sub * 4 + my_v, KC) >> 2);
        auto store_chunk = [&](int buf, const float* fr, const float* fs) {
            constexpr int VSTR = KC * 8, FSO = CH * 8, LO = LO_AC / 4;
            float* const b = sAC0 + buf * (STRIDE_AC / 4);
#pragma unroll
            for (int v = 0; v < 4; v++) {
                float hi, lo;
                umma::split_tf32(fr[v], hi, lo);
                b[v * VSTR] = hi;
                b[v * VSTR + LO] = lo;
                umma::split_tf32(fs[v], hi, lo);
                b[v * VSTR + FSO] = hi;
                b[v * VSTR + FSO + LO] = lo;
            }
        };
        // the slice of stage(tn) that goes with volume pass p
        const int pn = par ^ 1;
        auto stage_slice = [&](int p) {
            if (!has_next) return;
            if (p == 0) {
                // tn's FP64 tile (issued after stage(t)) has landed by now
                if constexpr (!S::STREAM) {
                    wait(bq, pq);
                    pq ^= 1;
                }
                stage_ref(tn, pn);
            } else if (D::NPASS > 1) {
                const int j0 = (p - 1) * D::DQ_PER;
                const int j1 = min(D::NDQ, j0 + D::DQ_PER);
                if (j0 < j1) stage_dq(tn, pn, j0, j1);
            }
        };

        // ---- (C) volume phase of t, stage(tn) in slices
        auto chunk_free = [&](int b) {
            wait(bar2 + b, (ph2 >> b) & 1u);
            ph2 ^= 1u << b;
        };
        constexpr int CPP = S::PAIR ? 2 : 1;  // chunks per pass
        [[maybe_unused]] int prev_n = 0;
#pragma unroll 1
        for (int p = 0; p < D::NPASS; p++) {
            const int ch0 = CPP * p;
            const int n = (S::NCH - ch0 >= CPP) ? CPP : 1;
            float x0[4], x1[4];
            umma::tmem_ld4(tD1 + ((uint32_t)(32 * qd) << 16) + ch0 * CH + sub * 4, x0);
            if (n == 2) umma::tmem_ld4(tD1 + ((uint32_t)(32 * qd) << 16) + (ch0 + 1) * CH + sub * 4, x1);
            if (has_next) {
                if (p == 0) fetch_ref(tn);
                else fetch_dq(tn, (p - 1) * D::DQ_PER, min(D::NDQ, p * D::DQ_PER));
            }
            umma::tmem_ld_wait();
            float fr0[4], fs0[4], fr1[4], fs1[4];
            vol_flux(x0, ch0, fr0, fs0);
            if (n == 2) vol_flux(x1, ch0 + 1, fr1, fs1);
            if (p == 0) {
                // every warp is through its face phase of t: the traces, the deltas and the
                // staged results in chunk buffer 0 are read
                wait(bfaces, phf);
                phf ^= 1;
            }
            stage_slice(p);
            if constexpr (S::STREAM) {
                if (p >= 2) chunk_free(p & 1);
                store_chunk(p & 1, fr0, fs0);
                umma::fence_async_smem();
                umma::fence_before_sync();
                arrive(bready + (p & 1));
            } else {
                for (int b = 0; b < prev_n; b++) chunk_free(b);
                store_chunk(0, fr0, fs0);
                if (n == 2) store_chunk(1, fr1, fs1);
                umma::fence_async_smem();
                umma::fence_before_sync();
                arrive(bready);
                prev_n = n;
            }
        }
        if (has_next) {
            if constexpr (D::NPASS == 1) stage_dq(tn, pn, 0, D::NDQ);
            staged();
        }
        // the group's 8 elements (the four warps of one tensor-memory quarter): RK
        // register values and stage input (L2), loaded while the last MMAs run
        constexpr int EPI = (8 * 4 * Np + 127) / 128;
        const bool first = sa.first != 0;
        const int gt = sub * 32 + lane, nv = max(0, min(8, ne - 8 * qd)) * 4 * Np;
        const size_t base = (size_t)(k0 + 8 * qd) * 4 * Np;
        float* const sR = sRS + qd * 8 * 4 * Np;
        float resp[EPI];
        double q0v[EPI];
        auto gemm2_done = [&]() {
            const bool need = a.mode == MODE_LSERK && !first;
            const bool needq = a.mode != MODE_RHS;
#pragma unroll
            for (int j = 0; j < EPI; j++) {
                const int i = gt + j * 128;
                resp[j] = (need && i < nv) ? __ldg(sa.res32 + base + i) : 0.f;
                q0v[j] = (needq && i < nv) ? __ldg(a.qin + base + i) : 0.0;
            }
            if constexpr (S::STREAM) {
                chunk_free(0);
                chunk_free(1);
            } else {
                for (int b = 0; b < prev_n; b++) chunk_free(b);
            }
        };
        // ---- face fluxes of tn while the last MMAs of t run; those read the operand
        // that the fluxes go to
        if (has_next) face_phase(tn, pn, gemm2_done);
        else gemm2_done();
        umma::fence_after_sync();
        // ---- (D) R (tensor memory) -> staging, in chunk buffer 0
        {
            const int e8 = lane & 7, v2 = lane >> 3;  // this lane's GEMM2 row (g2row)
#pragma unroll
            for (int col = sub * 8; col < NP2; col += 32) {
                float val[8];
                umma::tmem_ld8(tD2 + ((uint32_t)(32 * qd) << 16) + col, val);
                umma::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int p = col + j;
                    if (p < Np) sR[(4 * e8 + v2) * Np + p] = val[j];
                }
            }
        }
        umma::fence_before_sync();
        asm volatile("bar.sync %0, 128;" ::"r"(qd + 1) : "memory");
        // ---- epilogue of t
        {
            const float rka = sa.rkaf, dtf0 = sa.dtf, rkb = sa.rkbf;
            if (a.mode == MODE_LSERK && !sa.dtk32) {
#pragma unroll
                for (int j = 0; j < EPI; j++) {
                    const int i = gt + j * 128;
                    if (i < nv) {
                        const float R = sR[i];
                        const float r = first ? dtf0 * R : fmaf(rka, resp[j], dtf0 * R);
                        sa.res32_out[base + i] = r;
                        a.qout[base + i] = q0v[j] + (double)(rkb * r);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < EPI; j++) {
                    const int i = gt + j * 128;
                    if (i >= nv) break;
                    const float R = sR[i];
                    const double q0 = q0v[j];
                    const size_t idx = base + i;
                    const float dtf = sa.dtk32 ? dtf0 * sa.dtk32[k0 + 8 * qd + i / (4 * Np)] : dtf0;
                    switch (a.mode) {
                        case MODE_RHS: a.rhs[idx] = (double)R; break;
                        case MODE_LSERK: {
                            const float r = first ? dtf * R : fmaf(rka, resp[j], dtf * R);
                            sa.res32_out[idx] = r;
                            a.qout[idx] = q0 + (double)(rkb * r);
                        } break;
                        case MODE_EULER: a.qout[idx] = q0 + (double)(dtf * R); break;
                        default: a.qout[idx] = 0.5 * a.qold[idx] + 0.5 * (q0 + (double)(dtf * R)); break;
                    }
                }
            }
        }
        arrive(bfaces);
    }
    if constexpr (D::GATHER) umma::cp_async_wait_all();
    }
    umma::fence_before_sync();
    __syncthreads();
    if (tid == 0 && *dead) atomicExch(sa.status, 1);  // whoever gave up, and whenever
    if (warp == 16) umma::tmem_dealloc(tmem, S::TMEM_COLS);
}

template <int N>
__global__ void __launch_bounds__(kPipeThreads, 1) euler_stage_split_pipe_kernel(SplitArgs sa) {
    pipe_body<N>(sa, blockIdx.x, gridDim.x);
}

// One stage of several contexts of orders 1..6 in one launch: blocks
// [cta_end[g-1], cta_end[g]) run group g's tiles with its order's body.
__global__ void __launch_bounds__(kPipeThreads, 1) euler_stage_split_batch_kernel(const __grid_constant__ SplitBatchArgs P) {
    int g = 0;
    while (g + 1 < P.ngroups && (int)blockIdx.x >= P.cta_end[g]) g++;
    const int begin = g ? P.cta_end[g - 1] : 0;
    const int bid = (int)blockIdx.x - begin, nblk = P.cta_end[g] - begin;
    switch (P.order[g]) {
        case 1: pipe_body<1>(P.sa[g], bid, nblk); break;
        case 2: pipe_body<2>(P.sa[g], bid, nblk); break;
        case 3: pipe_body<3>(P.sa[g], bid, nblk); break;
        case 4: pipe_body<4>(P.sa[g], bid, nblk); break;
        case 5: pipe_body<5>(P.sa[g], bid, nblk); break;
        case 6: pipe_body<6>(P.sa[g], bid, nblk); break;
        default: break;
    }
}

// the register split (kComputeRegs, kIssuerRegs) draws on what a block is launched
// with; a build that launches with less must not run
static cudaError_t check_registers(const void* kernel) {
    cudaFuncAttributes at;
    const cudaError_t e = cudaFuncGetAttributes(&at, kernel);
    if (e != cudaSuccess) return e;
    return (at.numRegs + 7) / 8 * 8 * (kPipeThreads / 32) >= 16 * kComputeRegs + 4 * kIssuerRegs ? cudaSuccess : cudaErrorInvalidConfiguration;
}

static int batch_smem(int N) {
    switch (N) {
        case 1: return PipeDims<1>::SMEM;
        case 2: return PipeDims<2>::SMEM;
        case 3: return PipeDims<3>::SMEM;
        case 4: return PipeDims<4>::SMEM;
        case 5: return PipeDims<5>::SMEM;
        case 6: return PipeDims<6>::SMEM;
        default: return 0;
    }
}

cudaError_t setup_split_batch() {
    int smax = 0;
    for (int n = 1; n <= 6; n++) smax = std::max(smax, batch_smem(n));
    const cudaError_t e = check_registers((const void*)euler_stage_split_batch_kernel);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(euler_stage_split_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
}

cudaError_t launch_split_batch(const SplitBatchArgs& P, cudaStream_t s) {
    if (P.ngroups < 1 || P.ngroups > SplitBatchArgs::MAXG) return cudaErrorInvalidValue;
    int smax = 0;
    for (int g = 0; g < P.ngroups; g++) {
        const int sm = batch_smem(P.order[g]);
        if (sm == 0) return cudaErrorInvalidValue;
        smax = std::max(smax, sm);
    }
    euler_stage_split_batch_kernel<<<P.cta_end[P.ngroups - 1], kPipeThreads, smax, s>>>(P);
    return cudaGetLastError();
}

template <int N>
cudaError_t setup_split_pipe() {
    const cudaError_t e = check_registers((const void*)euler_stage_split_pipe_kernel<N>);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(euler_stage_split_pipe_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                PipeDims<N>::SMEM);
}

template <int N>
cudaError_t launch_split_pipe(const SplitArgs& sa, int grid, cudaStream_t s) {
    euler_stage_split_pipe_kernel<N><<<grid, kPipeThreads, PipeDims<N>::SMEM, s>>>(sa);
    return cudaGetLastError();
}

template cudaError_t setup_split_pipe<1>();
template cudaError_t setup_split_pipe<2>();
template cudaError_t setup_split_pipe<3>();
template cudaError_t setup_split_pipe<4>();
template cudaError_t setup_split_pipe<5>();
template cudaError_t setup_split_pipe<6>();
template cudaError_t setup_split_pipe<7>();
template cudaError_t launch_split_pipe<1>(const SplitArgs&, int, cudaStream_t);
template cudaError_t launch_split_pipe<2>(const SplitArgs&, int, cudaStream_t);
template cudaError_t launch_split_pipe<3>(const SplitArgs&, int, cudaStream_t);
template cudaError_t launch_split_pipe<4>(const SplitArgs&, int, cudaStream_t);
template cudaError_t launch_split_pipe<5>(const SplitArgs&, int, cudaStream_t);
template cudaError_t launch_split_pipe<6>(const SplitArgs&, int, cudaStream_t);
template cudaError_t launch_split_pipe<7>(const SplitArgs&, int, cudaStream_t);

}  // namespace dgk
