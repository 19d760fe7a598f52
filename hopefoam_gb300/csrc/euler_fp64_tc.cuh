// euler_fp64_tc.cuh -- operator images and sizes of the tensor-core FP64 Euler
// stage (euler_fp64_tc.cu), shared with the host code that builds them.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "dg_basis.hpp"
#include "dg_internal.hpp"
#include "ozaki.cuh"

namespace dgk {

// Sizes of one order.  M = 128 operand rows are 32 elements x 4 variables,
// row = 32 (e / 8) + 8 v + e % 8: tensor-memory lanes 32 s .. 32 s + 31 (the
// ones a warp w with w % 4 == s can read) hold the four variables of eight
// elements.
template <int N>
struct OzDims {
    static constexpr int Np = Dims<N>::Np, Ng = Dims<N>::Ng, Nfp = Dims<N>::Nfp, Nfq = Dims<N>::Nfq;
    static constexpr int NF = 3 * Nfq, NB = 3 * N, NT = 3 * Nfp;
    static constexpr int K1 = (Np + 15) / 16 * 16;       // reduction length of the interpolation
    static constexpr int KB1 = K1 / 8;
    static constexpr int LPR = KB1 <= 4 ? 4 : 8;         // lanes per operand row while it is cut into digits
    static constexpr int NP2 = N == 5 ? 24 : (Np + 15) / 16 * 16;  // result columns per digit group
    static constexpr int NC = (Ng + 15) / 16;            // chunks of 16 cubature points
    static constexpr int NG4 = (NF + 3) / 4;             // groups of 4 face points
    static_assert(NF <= 32 && NT <= 32 && NG4 <= 8, "face operand sizes");
    // operator pieces in the order they are consumed per tile
    // (seven digit blocks and a block of zeros, which starts the eighth accumulator)
    static constexpr int B1F = (oz::kSlices + 1) * 32 * K1 * 2;   // own nodes -> face points
    static constexpr int B3 = (oz::kSlices + 1) * 32 * 32 * 2;    // neighbour face nodes -> face points
    static constexpr int B1 = (oz::kSlices + 1) * 16 * K1 * 2;    // own nodes -> one chunk of cubature points
    static constexpr int B2 = (oz::kSlices + 1) * NP2 * 32 * 2;   // one chunk's fluxes (or the face fluxes) -> nodes
    // order: own traces, neighbour traces, chunk 0's interpolation, face fluxes,
    // then per chunk c the interpolation of chunk c + 1 and the fluxes of chunk c
    static constexpr int PIECES = 2 * NC + 3;
    OZ_HD static constexpr bool piece_flux(int p) {
        return p == 3 || p == PIECES - 1 || (p > 3 && (p & 1));
    }
    static constexpr int piece_b1(int c) { return c == 0 ? 2 : 4 + 2 * (c - 1); }
    static constexpr int piece_b2(int c) { return c == NC - 1 ? PIECES - 1 : 5 + 2 * c; }
    static constexpr int piece_bytes(int p) { return p == 0 ? B1F : p == 1 ? B3 : piece_flux(p) ? B2 : B1; }
    static constexpr size_t piece_off(int i) {
        size_t o = 0;
        for (int j = 0; j < i; j++) o += piece_bytes(j);
        return o;
    }
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    static constexpr int SLOT = cmax(cmax(B1F, B3), cmax(B1, B2));
    static constexpr int NSLOT = N == 7 ? 3 : 4;
    // tensor memory columns, eight digit groups each: face traces (own, neighbour), then
    // the result groups and the cubature accumulators over them
    static constexpr int T_OWN = 0, T_NBR = 256, T_RES = 0, T_CUB = 384;
    static_assert(8 * NP2 <= T_CUB && T_CUB + 8 * 16 <= 512 && T_NBR + 8 * 32 <= 512, "tensor memory");
    // shared memory
    static constexpr int A1S = 128 * K1 * 2, A2S = 128 * 32 * 2;  // one digit slice of each operand
    static constexpr int OFF_A1 = 0;
    static constexpr int OFF_A2 = OFF_A1 + oz::kSlices * A1S;
    static constexpr int OFF_RING = OFF_A2 + oz::kSlices * A2S;
    static constexpr int OFF_LAM = OFF_RING + NSLOT * SLOT;       // [32][NF] wave speeds
    static constexpr int OFF_GEO = OFF_LAM + 32 * NF * 8;         // [32][4]
    static constexpr int OFF_NRM = OFF_GEO + 32 * 4 * 8;          // [32][3][3] nx, ny, sJ/J
    static constexpr int OFF_CONN = OFF_NRM + 32 * 9 * 8;         // [32][3]
    static constexpr int OFF_MAXQ = OFF_CONN + 32 * 3 * 4;        // [32][4] high word of max |q|
    static constexpr int OFF_H3 = OFF_MAXQ + 128 * 4;             // [32][4][3] the same of a face's neighbour trace
    static constexpr int OFF_EST = OFF_H3 + 384 * 4;              // [32][4] max |volume flux| at the nodes (FP32)
    static constexpr int OFF_MAXF = OFF_EST + 128 * 4;            // [32][4] high word of max |face flux|
    static constexpr int OFF_FLAG = OFF_MAXF + 128 * 4;           // [4] elements left to plain FP64
    static constexpr int OFF_REACH = OFF_FLAG + 4 * 4;            // [4] flux rows that came near their bound, 4 bits an element
    static constexpr int OFF_EB = OFF_REACH + 4 * 4;              // [NP2 + 2] operator bounds
    static constexpr int OFF_DEAD = OFF_EB + (NP2 + 2) * 4;
    static constexpr int OFF_TMEM = OFF_DEAD + 4;
    static constexpr int OFF_BAR = (OFF_TMEM + 4 + 7) / 8 * 8;    // mbarriers
    static constexpr int SMEM = OFF_BAR + (8 + 2 * NSLOT) * 8;
    static_assert(SMEM <= 232448, "shared memory");
    // the plain route: scratch values per element, those of a group in the first operand and
    // in both, and how many elements it takes at once
    static constexpr int PLAIN_SCRATCH = 8 * Ng + 5 * NF;
    static constexpr int A1_SCRATCH = oz::kSlices * 32 * K1 * 2 / 8, A12_SCRATCH = A1_SCRATCH + oz::kSlices * 2048 / 8;
    static constexpr int cmin(int a, int b) { return a < b ? a : b; }
    static constexpr int PB = cmin(8, cmin(128 / NF, A12_SCRATCH / PLAIN_SCRATCH));
    static_assert(PB >= 1 && PB * NF <= 128 && PB * PLAIN_SCRATCH <= A12_SCRATCH, "scratch of the plain route");
    static_assert(32 * Np * 8 <= oz::kSlices * 2048, "result staging");
};

struct OzImage {
    std::vector<unsigned char> bytes;  // operator pieces, in consumption order
    std::vector<int> eb;               // [NP2] bounds of the result rows, then of Vg and of If
    bool exact = false;                // every accumulator and 64-bit sum is provably exact
};

// byte offset of (row, k) in the K-major no-swizzle operand layout (8 rows x
// 16 bytes per core matrix), 2-byte elements
inline size_t oz_off(int r, int k, int KP) { return (size_t)(((r >> 3) * (KP >> 3) + (k >> 3)) << 7) + ((r & 7) << 4) + ((k & 7) << 1); }

template <int N>
OzImage oz_build(const dgb::RefOps& o) {
    using D = OzDims<N>;
    OzImage im;
    im.bytes.assign(D::piece_off(D::PIECES), 0);
    auto bound = [](const std::vector<double>& v, size_t i0, size_t n) {
        uint32_t m = 0;
        for (size_t i = i0; i < i0 + n; i++) m = std::max(m, oz::mag_hi(v[i]));
        return oz::row_bound(m);
    };
    const int ebV = bound(o.dVg, 0, o.dVg.size()), ebI = bound(o.If, 0, o.If.size());
    im.eb.assign(D::NP2 + 2, 0);
    for (int n = 0; n < D::Np; n++)
        im.eb[n] = std::max(std::max(bound(o.dSr, (size_t)n * D::Ng, D::Ng), bound(o.dSs, (size_t)n * D::Ng, D::Ng)),
                            bound(o.dLift, (size_t)n * D::NF, D::NF));
    im.eb[D::NP2] = ebV;
    im.eb[D::NP2 + 1] = ebI;
    // FP16 bits of every digit, and where the pieces are
    uint16_t half[257];
    for (int d = -128; d <= 128; d++) half[d + 128] = oz::half_bits(d);
    size_t at[D::PIECES];
    for (size_t i = 0, o = 0; i < (size_t)D::PIECES; o += D::piece_bytes((int)i++)) at[i] = o;
    // digits of one operator value into a piece; |digit| into the sums of its result column, by digit
    auto put = [&](int piece, int P, int KP, int n, int k, double v, int eb, std::vector<int>& sum) {
        unsigned char* base = im.bytes.data() + at[piece];
        const uint64_t y = oz::biased(v, eb);
        for (int j = 0; j < oz::kSlices; j++) {
            const int d = oz::digit(y, j);
            memcpy(base + oz_off(j * P + n, k, KP), &half[d + 128], 2);
            sum[(size_t)j * P + n] += d < 0 ? -d : d;
        }
    };
    // largest possible |accumulator| over the columns and digit groups i + j = s, the
    // activation digits at their largest (128): |a| sum |b|
    auto worst = [&](const std::vector<int>& sum, int P) {
        long long m = 0;
        for (int n = 0; n < P; n++)
            for (int s = 0; s < 8; s++) {
                long long t = 0;
                for (int j = std::max(0, s - oz::kSlices + 1); j <= std::min(s, oz::kSlices - 1); j++) t += sum[(size_t)j * P + n];
                m = std::max(m, 128 * t);
            }
        return m;
    };
    long long worst1 = 0;
    std::vector<int> sum2((size_t)oz::kSlices * D::NP2, 0);
    // own nodes -> face points; neighbour face nodes -> face points
    {
        std::vector<int> s1((size_t)oz::kSlices * 32, 0), s3((size_t)oz::kSlices * 32, 0);
        for (int f = 0; f < 3; f++)
            for (int i = 0; i < D::Nfq; i++)
                for (int j = 0; j < D::Nfp; j++) {
                    const double v = o.If[(size_t)i * D::Nfp + j];
                    put(0, 32, D::K1, f * D::Nfq + i, (f * N + j) % D::NB, v, ebI, s1);
                    put(1, 32, 32, f * D::Nfq + i, f * D::Nfp + j, v, ebI, s3);
                }
        worst1 = std::max(worst(s1, 32), worst(s3, 32));
    }
    for (int c = 0; c < D::NC; c++) {
        std::vector<int> s1((size_t)oz::kSlices * 16, 0);
        for (int p = 0; p < 16 && 16 * c + p < D::Ng; p++) {
            const int g = 16 * c + p;
            for (int k = 0; k < D::Np; k++) put(D::piece_b1(c), 16, D::K1, p, k, o.dVg[(size_t)g * D::Np + k], ebV, s1);
            for (int n = 0; n < D::Np; n++) {
                put(D::piece_b2(c), D::NP2, 32, n, 2 * p, o.dSr[(size_t)n * D::Ng + g], im.eb[n], sum2);
                put(D::piece_b2(c), D::NP2, 32, n, 2 * p + 1, o.dSs[(size_t)n * D::Ng + g], im.eb[n], sum2);
            }
        }
        worst1 = std::max(worst1, worst(s1, 16));
    }
    for (int n = 0; n < D::Np; n++)
        for (int q = 0; q < D::NF; q++) put(3, D::NP2, 32, n, q, -o.dLift[(size_t)n * D::NF + q], im.eb[n], sum2);
    const long long worst2 = worst(sum2, D::NP2);
    bool fits = true;
    auto ratio = [](double v, int eb) { return std::ldexp(std::fabs(v), 1022 - eb); };
    for (int g = 0; g < D::Ng; g++) {
        double s = 0;
        for (int k = 0; k < D::Np; k++) s += ratio(o.dVg[(size_t)g * D::Np + k], ebV);
        fits = fits && s < 31.0;
    }
    for (int i = 0; i < D::Nfq; i++) {
        double s = 0;
        for (int j = 0; j < D::Nfp; j++) s += ratio(o.If[(size_t)i * D::Nfp + j], ebI);
        fits = fits && s < 31.0;
    }
    for (int n = 0; n < D::Np; n++) {
        double s = 0;
        for (int g = 0; g < D::Ng; g++)
            s += ratio(o.dSr[(size_t)n * D::Ng + g], im.eb[n]) + ratio(o.dSs[(size_t)n * D::Ng + g], im.eb[n]);
        for (int q = 0; q < D::NF; q++) s += ratio(o.dLift[(size_t)n * D::NF + q], im.eb[n]);
        fits = fits && s < 127.0;
    }
    im.exact = fits && worst1 < (1ll << 22) && worst2 < (1ll << 24);
    return im;
}

}  // namespace dgk
