// ipdg_rows.cuh -- element-aligned thread layout shared by the SIPG row kernels
// (block Jacobi, PCG updates, the block apply).
#pragma once

namespace dgk {

// Element-aligned kernels: a group of EB = 256 / Np whole elements, one
// thread per (element, row), Np a compile-time constant so that the block
// products unroll (Np independent loads in flight per thread).  Persistent
// CTAs (a few per SM) stride over the groups, so each grid-wide sum has one
// arrival per CTA.  The inverse diagonal blocks are stored grouped: for group
// g and column j the EB x Np entries (element, row) are contiguous,
//   Pg[((g Np + j) EB + e) Np + i] = P_{g EB + e}[i][j],
// so the CTA's loads for one column form a single contiguous read.
//
// Up to Np = 32 (N <= 6) an element's rows never straddle a warp: each warp
// holds EW = 32 / Np whole elements (WA), so the rows of an element exchange
// their values by warp shuffles and the kernels need no CTA barrier per
// group.  N = 7 (Np = 36) keeps one shared-memory exchange per group.
template <int NP>
struct RowDims {
    static constexpr bool WA = NP <= 32;
    static constexpr int EW = WA ? 32 / NP : 0;  // elements per warp
    static constexpr int EB = WA ? 8 * EW : 256 / NP;
    static constexpr int THREADS = WA ? 256 : (EB * NP + 31) / 32 * 32;  // extra lanes idle but join the reductions
};

// this thread's (element in the group, row) and its slot in the grouped layout
template <int NP>
__device__ __forceinline__ void row_of(int& e, int& i) {
    if constexpr (RowDims<NP>::WA) {
        const int lane = threadIdx.x & 31;
        e = (threadIdx.x >> 5) * RowDims<NP>::EW + lane / NP;
        i = lane % NP;
        if (lane >= RowDims<NP>::EW * NP) e = RowDims<NP>::EB;  // idle lane
    } else {
        e = threadIdx.x / NP;
        i = threadIdx.x - e * NP;
    }
}

template <int NP>
__host__ __device__ constexpr int row_groups(int K) { return (K + RowDims<NP>::EB - 1) / RowDims<NP>::EB; }

}  // namespace dgk
