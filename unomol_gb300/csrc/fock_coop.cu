// Launches of the warp-per-quartet kernels (fock_coop.cuh).
#include "fock_coop.cuh"
#include "fock_dispatch.cuh"

namespace ugb {
namespace {

// The same limit on every launch, the largest of all classes ((dd|dd): 69768 bytes): it is the kernel's, not the
// launch's, so one set to a smaller class's need would fail another thread's launch of a larger one.
constexpr size_t COOP_SMEM = 72 * 1024;

// Four quartets to a CTA; above 2^21 quartets the CTAs are laid out in rows, which keeps the grid's first dimension inside
// its limit for lists of up to 1.4e11 (a single row ended at 8.6e9).
constexpr long long COOP_ROW = 1 << 19;

template <int KF>
cudaError_t launch(const FockArgs& A, const NormTable& nt, const double* rys, const CoopShape& q, cudaStream_t s) {
    const size_t bytes = sizeof(double) * (q.per_cta + (size_t)COOP_WARPS * q.per_warp);
    if (bytes > COOP_SMEM) return cudaErrorInvalidValue;
    if (bytes > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(fock_jk_coop<KF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)COOP_SMEM);
        if (e != cudaSuccess) return e;
    }
    const long long ctas = (A.nwork + COOP_WARPS - 1) / COOP_WARPS, cols = ctas < COOP_ROW ? ctas : COOP_ROW;
    const dim3 grid((unsigned)cols, (unsigned)((ctas + cols - 1) / cols));
    fock_jk_coop<KF><<<grid, 32 * COOP_WARPS, bytes, s>>>(A, nt, rys, q.la, q.lb, q.lc, q.ld);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_fock_coop(int la, int lb, int lc, int ld, const FockArgs& A, const NormTable& nt, const double* rys,
                             cudaStream_t s) {
    if (A.nwork <= 0) return cudaSuccess;
    const CoopShape q(la, lb, lc, ld);
    if (la + lb + lc + ld > 8) return cudaErrorInvalidValue;
    // function quartets per lane: the next of a few register budgets
    if (q.nf <= 4 * 32) return launch<4>(A, nt, rys, q, s);
    if (q.nf <= 7 * 32) return launch<7>(A, nt, rys, q, s);
    if (q.nf <= 12 * 32) return launch<12>(A, nt, rys, q, s);
    if (q.nf <= 21 * 32) return launch<21>(A, nt, rys, q, s);
    if (q.nf <= 41 * 32) return launch<41>(A, nt, rys, q, s);
    return cudaErrorInvalidValue;
}

}  // namespace ugb
