// The class-templated kernels of the mixed build's FP64 part.
#include <algorithm>

#include "fock_mixed.cuh"
#include "fock_dispatch.cuh"

namespace ugb {

template <int BC, int KC, bool UHF>
static cudaError_t launch_fp64_part(const FockArgs& A64, const FockArgs& A32, const NormTable& nt, const double* rys64,
                                    const float* rys32, int grid, cudaStream_t s) {
    constexpr int LA = pc_la(BC), LB = pc_lb(BC), LC = pc_la(KC), LD = pc_lb(KC);
    if (A64.nwork <= 0) return cudaSuccess;
    if constexpr (QClass<LA, LB, LC, LD>::NF <= 81) {
        const long long blocks = std::min<long long>((A64.nwork + FOCK_THREADS - 1) / FOCK_THREADS, grid);
        fock_jk_fp64_part<LA, LB, LC, LD, UHF><<<(unsigned)blocks, FOCK_THREADS, 0, s>>>(A64, A32, nt, rys64, rys32);
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int BC, int KC, bool UHF>
static cudaError_t launch_df_part(const FockArgs& A, const NormTable& nt, int grid, cudaStream_t s) {
    constexpr int LA = pc_la(BC), LB = pc_lb(BC), LC = pc_la(KC), LD = pc_lb(KC);
    if (A.nwork <= 0) return cudaSuccess;
    if constexpr (QClass<LA, LB, LC, LD>::NF <= 81) {
        const long long blocks = std::min<long long>((A.nwork + FOCK_THREADS - 1) / FOCK_THREADS, grid);
        fock_jk_df64_part<LA, LB, LC, LD, UHF><<<(unsigned)blocks, FOCK_THREADS, 0, s>>>(A, nt);
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

#define UGB_CASE(BC, KC)                                                                      \
    case (BC) * 8 + (KC):                                                                     \
        return uhf ? launch_df_part<BC, KC, true>(A, nt, grid, stream)                        \
                   : launch_df_part<BC, KC, false>(A, nt, grid, stream);

cudaError_t launch_fock_df64_part(int bc, int kc, bool uhf, const FockArgs& A, const NormTable& nt, int grid,
                                  cudaStream_t stream) {
    switch (bc * 8 + kc) {
#include "fock_cases.inc"
        default:
            return cudaErrorInvalidValue;
    }
}

bool fock_split_class(int bc, int kc) {
    const int la = pc_la(bc), lb = pc_lb(bc), lc = pc_la(kc), ld = pc_lb(kc);
    return bc < NTMPLCLASS && kc < NTMPLCLASS &&
           ncart(la) * ncart(lb) * ncart(lc) * ncart(ld) <= 81;
}

#undef UGB_CASE
#define UGB_CASE(BC, KC)                                                                      \
    case (BC) * 8 + (KC):                                                                     \
        return uhf ? launch_fp64_part<BC, KC, true>(A64, A32, nt, rys64, rys32, grid, stream) \
                   : launch_fp64_part<BC, KC, false>(A64, A32, nt, rys64, rys32, grid, stream);

cudaError_t launch_fock_fp64_part(int bc, int kc, bool uhf, const FockArgs& A64, const FockArgs& A32, const NormTable& nt,
                                  const double* rys64, const float* rys32, int grid, cudaStream_t stream) {
    switch (bc * 8 + kc) {
#include "fock_cases.inc"
        default:
            return cudaErrorInvalidValue;
    }
}

cudaError_t launch_mixed_fp64(int bc, int kc, bool uhf, FockArgs A, const FockArgs& A32, const NormTable& nt,
                              const double* rys64, const float* rys32, int nsm, int ctas64, int ctasdf, bool demotes,
                              cudaStream_t s, int* launches) {
    const long long few = (long long)nsm * 32;
    // below eight times that many quartets in the part (known to the device only) four lanes per quartet fill the
    // SMs better than one
    A.df_group_max = 8 * few;
    cudaError_t e = cudaSuccess;
    if (A.nwork <= few) {
        for (bool df : {false, true})
            if (e == cudaSuccess) e = launch_fock_group(bc, kc, uhf, A, A.nwork, df, 32, nt, rys64, s);
        *launches += 2;
        A.only_demoted = 1;
        if (e != cudaSuccess || !(demotes || A.counters)) return e;
    }
    e = launch_fock_fp64_part(bc, kc, uhf, A, A32, nt, rys64, rys32, nsm * ctas64, s);
    ++*launches;
    if (e == cudaSuccess && A.nwork > A.df_group_max) {
        e = launch_fock_df64_part(bc, kc, uhf, A, nt, nsm * ctasdf, s);
        ++*launches;
    }
    return e;
}

}  // namespace ugb
