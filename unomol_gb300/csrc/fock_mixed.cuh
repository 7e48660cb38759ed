// Kernels of the mixed-precision build whose work lists hold an FP64 and an FP32 part.
#pragma once
#include "fock_df64.cuh"

namespace ugb {

// Lanes per quartet of the FP64 part (2: 157.1, 4: 160.2, 8: 157.0 builds/s on 32 waters).
constexpr int FP64_PARTS = 4;

// FP64 part of a mixed build with FP64_PARTS lanes per quartet: the warp holds the 32 / FP64_PARTS items from
// g0.  The work lists put a quartet in the FP64 part when its Schwarz bound times the largest |P| of the whole
// density reaches the FP32 cut; a quartet whose bound times the largest |P| of its own six blocks (the density
// elements it is contracted with) is below that cut runs in FP32 here (with the FP32 part's arguments A32),
// under the same per-quartet error bound as the FP32 part's own quartets.  Of the others, those below SPLIT_CUT
// are left to fock_jk_df64_part unless the part is small, and the rest (few, and the costliest of the build: one
// lane each would leave most of the issue slots idle) run in FP64; classes of few quartets in all leave both to
// fock_jk_group, a warp per quartet (full-density build of a water in STO-3G 1.01 -> 0.27 ms, of five in 6-31G 2.44 -> 1.17 ms).
template <int LA, int LB, int LC, int LD, bool UHF>
__device__ __forceinline__ void fock_group_fp64_part(const FockArgs& A64, const FockArgs& A32, const NormTable& nt,
                                                     const double* __restrict__ rys64, const float* __restrict__ rys32,
                                                     long long g0) {
    constexpr int NP = FP64_PARTS;
    const int lane = threadIdx.x & 31, sub = lane / NP, part = lane % NP;
    const unsigned gmask = ((1u << NP) - 1u) << (sub * NP);
    int bi, ki;
    if (!decode_warp_items<true>(A64, g0, sub, bi, ki)) return;  // warp-collective; uniform over a group
    const ShellPair bra = A64.pairs[bi];
    const ShellPair ket = A64.pairs[ki];
    const float bound = quartet_bound(A64, bra, ket);
    if (bound < A64.skip_cut32) {
        if (A64.counters && part == 0) count_screened(A64);
        return;
    }
    if (bound < A64.fp32_cut32) {
        if (A64.counters && part == 0) count_demoted(A64);
        quartet_item_group<LA, LB, LC, LD, UHF, float, NP>(A32, nt, rys32, bra, ket, bi == ki, part, gmask);
    } else if (bra.qf * ket.qf < A64.split_cut32) {
        if (A64.only_demoted || *A64.dyn_total > A64.df_group_max) return;  // fock_jk_group, fock_jk_df64_part
        quartet_item_group_df<LA, LB, LC, LD, UHF, NP>(A64, nt, bra, ket, bi, ki, part, gmask);
    } else if (!A64.only_demoted) {
        quartet_item_group<LA, LB, LC, LD, UHF, double, NP>(A64, nt, rys64, bra, ket, bi == ki, part, gmask);
    }
}

// The FP64 part of a mixed build of one class (a kernel of its own: the FP32 part runs at the FP32 code's
// register count): a fixed grid whose warps step over the part's quartets.
template <int LA, int LB, int LC, int LD, bool UHF>
__global__ void __launch_bounds__(128) fock_jk_fp64_part(const FockArgs A64, const FockArgs A32, const NormTable nt,
                                                         const double* __restrict__ rys64, const float* __restrict__ rys32) {
    const long long per_warp = 32 / FP64_PARTS;
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long total = *A64.dyn_total;
    for (long long wi = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); wi * per_warp < total; wi += nwarps)
        fock_group_fp64_part<LA, LB, LC, LD, UHF>(A64, A32, nt, rys64, rys32, wi * per_warp);
}

// The quartets of the FP64 part that take pairs of floats, one lane each, stepping over the part's list.  A
// kernel beside the group kernel above, because one lane per quartet keeps the warps full where the quartets
// are many (in the group kernel, four lanes each: 8.7 against 7.7 ms per build of 32 waters, 42.0 against 31.4
// ms for 256 molecules; all in FP64 10.0 and 68.9 ms).
template <int LA, int LB, int LC, int LD, bool UHF>
__global__ void __launch_bounds__(128, LA + LB + LC + LD <= 1 ? 8 : 1) fock_jk_df64_part(const FockArgs A, const NormTable nt) {
    if (*A.dyn_total <= A.df_group_max) return;  // the group kernel's
    const long long total = *A.dyn_total, step = (long long)gridDim.x * blockDim.x;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g - (threadIdx.x & 31) < total; g += step)
        df_item<LA, LB, LC, LD, UHF>(A, nt, g);
}

}  // namespace ugb
