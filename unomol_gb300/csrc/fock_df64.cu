// Kernels of the split FP64 build: the quartets below SPLIT_CUT in pairs of floats, the others in FP64, with
// several lanes per quartet where they are few.
#include "fock_df64.cuh"
#include "fock_dispatch.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace ugb {

template <int BC, int KC, bool UHF>
static cudaError_t launch_df(const FockArgs& A, long long items, const NormTable& nt, cudaStream_t s) {
    constexpr int LA = pc_la(BC), LB = pc_lb(BC), LC = pc_la(KC), LD = pc_lb(KC);
    if (items <= 0) return cudaSuccess;
    if constexpr (QClass<LA, LB, LC, LD>::NF <= 81) {
        fock_jk_df64<LA, LB, LC, LD, UHF><<<(unsigned)((items + FOCK_THREADS - 1) / FOCK_THREADS), FOCK_THREADS, 0, s>>>(A, nt);
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int BC, int KC>
static cudaError_t launch_persist(const FockArgs& A, const NormTable& nt, int grid, int block, cudaStream_t s) {
    constexpr int LA = pc_la(BC), LB = pc_lb(BC), LC = pc_la(KC), LD = pc_lb(KC);
    if constexpr (QClass<LA, LB, LC, LD>::NF <= 81) {
        fock_jk_df64_persistent<LA, LB, LC, LD, false><<<grid, block, 0, s>>>(A, nt);
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int BC, int KC, bool UHF>
static cudaError_t launch_group(const FockArgs& A, long long items, bool pairs_of_floats, int lanes, const NormTable& nt,
                                const double* rys, cudaStream_t s) {
    constexpr int LA = pc_la(BC), LB = pc_lb(BC), LC = pc_la(KC), LD = pc_lb(KC);
    if (items <= 0) return cudaSuccess;
    if constexpr (QClass<LA, LB, LC, LD>::NF <= 81) {
        const unsigned blocks = (unsigned)((items * lanes + FOCK_THREADS - 1) / FOCK_THREADS);
        if (lanes == 32) {
            const size_t bytes = sizeof(double) * (FOCK_THREADS / 32) * group_smem<LA, LB, LC, LD>();
            if (pairs_of_floats) fock_jk_group<LA, LB, LC, LD, UHF, 32, true><<<blocks, FOCK_THREADS, bytes, s>>>(A, nt, rys);
            else fock_jk_group<LA, LB, LC, LD, UHF, 32, false><<<blocks, FOCK_THREADS, bytes, s>>>(A, nt, rys);
        } else {
            if (pairs_of_floats) fock_jk_group<LA, LB, LC, LD, UHF, 4, true><<<blocks, FOCK_THREADS, 0, s>>>(A, nt, rys);
            else fock_jk_group<LA, LB, LC, LD, UHF, 4, false><<<blocks, FOCK_THREADS, 0, s>>>(A, nt, rys);
        }
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

#define UGB_CASE(BC, KC)                                                              \
    case (BC) * 8 + (KC):                                                             \
        return uhf ? launch_df<BC, KC, true>(A, items, nt, stream)              \
                   : launch_df<BC, KC, false>(A, items, nt, stream);

cudaError_t launch_fock_df64(int bc, int kc, bool uhf, const FockArgs& A, long long items, const NormTable& nt,
                             cudaStream_t stream) {
    switch (bc * 8 + kc) {
#include "fock_cases.inc"
        default:
            return cudaErrorInvalidValue;
    }
}

#undef UGB_CASE
#define UGB_CASE(BC, KC)  \
    case (BC) * 8 + (KC): \
        return launch_persist<BC, KC>(A, nt, grid, block, stream);

cudaError_t launch_fock_df64_persistent(int bc, int kc, const FockArgs& A, const NormTable& nt, int grid, int block,
                                        cudaStream_t stream) {
    switch (bc * 8 + kc) {
#include "fock_cases.inc"
        default:
            return cudaErrorInvalidValue;
    }
}

#undef UGB_CASE
#define UGB_CASE(BC, KC)                                                              \
    case (BC) * 8 + (KC):                                                             \
        return uhf ? launch_group<BC, KC, true>(A, items, pairs_of_floats, lanes, nt, rys, stream) \
                   : launch_group<BC, KC, false>(A, items, pairs_of_floats, lanes, nt, rys, stream);

cudaError_t launch_fock_group(int bc, int kc, bool uhf, const FockArgs& A, long long items, bool pairs_of_floats, int lanes,
                              const NormTable& nt, const double* rys, cudaStream_t stream) {
    switch (bc * 8 + kc) {
#include "fock_cases.inc"
        default:
            return cudaErrorInvalidValue;
    }
}

// The tables of df_roots, from the FP64 ones (rys_tables.inc); the second two-root block holds, for the
// intervals in (15, 40], degree-7 fits of the reference's large-T nodes and weights (Rys.cpp:611-623, as
// rys2_reference_regime writes them), which are smooth there: the fit is good to 1e-17.
std::vector<float> df_rys_tables() {
    std::vector<float> t(DF_TABLE_LEN, 0.f);
    auto put = [&](size_t row, int k, double v) {
        t[row * DF_STRIDE + k] = (float)v;
        t[row * DF_STRIDE + 8 + k] = (float)(v - (double)(float)v);
    };
    const size_t rows = RYS_TABLE_SIZE / (RYS_DEG + 1);
    for (size_t r = 0; r < rows; ++r)
        for (int d = 0; d <= RYS_DEG; ++d) put(r, d, RYS_TABLE_H[r * (RYS_DEG + 1) + d]);
    const size_t row2 = rys_off(2, DF_STRIDE, RYS_H) / DF_STRIDE, n2 = rys_off(3, DF_STRIDE, RYS_H) / DF_STRIDE - row2;
    const size_t rowc = DF_COMPAT2 / DF_STRIDE;
    std::copy(t.begin() + row2 * DF_STRIDE, t.begin() + (row2 + n2) * DF_STRIDE, t.begin() + rowc * DF_STRIDE);
    constexpr int NC = 16;  // Chebyshev nodes of the fit
    for (int k = int(15 / RYS_H); k < int(40 / RYS_H); ++k) {
        double f[4][NC];
        for (int j = 0; j < NC; ++j) {
            const double y = std::cos(M_PI * (j + 0.5) / NC), T = (k + 0.5 * (y + 1.0)) * RYS_H;
            const double r12 = .275255128608411, r22 = 2.72474487139158, w22 = .0917517095361369;
            const double g = std::exp(-T), w0 = std::sqrt(.785398163397448 / T);
            const double u0 = (T * -.87894730749888 + 10.9243702330261) * g + r12 / (T - r12);
            const double u1 = (T * -9.28903924275977 + 81.0642367843811) * g + r22 / (T - r22);
            const double w1 = (T * 4.468573893084 - 77.9250653461045) * g + w22 * w0;
            f[0][j] = u0 / (1.0 + u0);
            f[1][j] = w0 - w1;
            f[2][j] = u1 / (1.0 + u1);
            f[3][j] = w1;
        }
        for (int q = 0; q < 4; ++q) {
            double c[RYS_DEG + 1], mono[RYS_DEG + 1] = {0};
            for (int n = 0; n <= RYS_DEG; ++n) {
                double s = 0;
                for (int j = 0; j < NC; ++j) s += f[q][j] * std::cos(M_PI * n * (j + 0.5) / NC);
                c[n] = s * (n ? 2.0 : 1.0) / NC;
            }
            // Chebyshev to monomials: T_{n+1} = 2 y T_n - T_{n-1}
            double a[RYS_DEG + 1] = {1}, b[RYS_DEG + 1] = {0, 1};
            for (int n = 0; n <= RYS_DEG; ++n) {
                for (int i = 0; i <= RYS_DEG; ++i) mono[i] += c[n] * a[i];
                double nx[RYS_DEG + 1];
                for (int i = 0; i <= RYS_DEG; ++i) nx[i] = (i ? 2.0 * b[i - 1] : 0.0) - a[i];
                for (int i = 0; i <= RYS_DEG; ++i) {
                    a[i] = b[i];
                    b[i] = nx[i];
                }
            }
            for (int i = 0; i <= RYS_DEG; ++i) put(rowc + (size_t)k * 4 + q, RYS_DEG - i, mono[i]);
        }
    }
    for (int n = 0; n < 5; ++n)
        for (int i = 0; i < 5; ++i) {
            const double v[2] = {RYS_HERMITE_X_H[n][i], RYS_HERMITE_W_H[n][i]};
            for (int q = 0; q < 2; ++q) {
                float* o = &t[DF_HERMITE + 2 * (25 * q + 5 * n + i)];
                o[0] = (float)v[q];
                o[1] = (float)(v[q] - (double)o[0]);
            }
        }
    return t;
}

}  // namespace ugb
