// Shell-quartet integrals in pairs of floats (df64.cuh), for the quartets of the FP64 build whose Schwarz
// bound lies below SPLIT_CUT (1/16).  Their integrals come out within about 2^-50 of the bound (rms, s and p
// shells), that is 2^-54, less than an FP64 evaluation of the quartets of order one is off; G keeps its error
// (SPLIT_CUT's comment has the figures).  The quartets above the cut are evaluated in FP64, and the density
// contraction and the accumulation are FP64 for all of them.
//
// What bounds it: the FP64 kernels keep the FP64 pipe (2 lanes per clock and SM) 88 % busy; the same
// primitive quartet of (ps|ss) is about 65 FP64 instructions (1040 SM clocks per warp) or about 350 FP32
// ones (88 clocks at full issue).  Here issue is 47-67 % active, the L1 data pipe 35-72 % and the FP64 pipe
// (the density contraction) 16-36 %, with the loads the leading stall.  One build, GB300: 32 waters 6-31G
// 79.3 -> 21.9 ms, n-decane cation UHF 12.2 -> 3.2 ms (with the group kernels below).
// Measured beside it: look-ahead for the next surviving primitive quartet (as the FP64 kernels) instead of
// plain loops, kept for la+lb+lc+ld = 2 only ((ps|ps) 3.9 against 4.2 ms, (ps|ss) 7.6 against 6.9); 64
// registers for (ss|ss) and (ps|ss) (25.3 -> 24.0 ms for the build).
#pragma once
#include <type_traits>

#include "df64.cuh"
#include "fock_kernels.cuh"
// (after load_row)
#include "df_roots.cuh"

namespace ugb {

// rys_axis (fock_kernels.cuh) in double-float.  UNIT: the axis starts from 1 (its factor sits on the z
// axis), so products with element (0, 0) fall away.
template <int LA, int LB, int LC, int LD, bool UNIT>
__device__ __forceinline__ void df_axis(df g00, df C, df Cp, df B00, df B1, df B1p, df AB, df CD,
                                        df (&I)[(LA + 1) * (LB + 1) * (LC + 1) * (LD + 1)]) {
    constexpr int L12 = LA + LB, L34 = LC + LD;
    // a x + y with x element (ix) of the recurrence, which is 1 for UNIT at index 0
    auto mad = [](bool one, df a, df x, df y) { return (UNIT && one) ? df_add(y, a) : df_fma(a, x, y); };
    auto prod = [](bool one, df a, df x) { return (UNIT && one) ? a : df_mul(a, x); };
    df G[L12 + 1][L34 + 1];
    G[0][0] = g00;
    if constexpr (L12 > 0) G[1][0] = prod(true, C, g00);
#pragma unroll
    for (int i = 1; i < L12; ++i) {
        const df b = i == 1 ? B1 : df_mulf(B1, float(i));
        G[i + 1][0] = mad(i == 1, b, G[i - 1][0], df_mul(C, G[i][0]));
    }
#pragma unroll
    for (int j = 0; j < L34; ++j) {
#pragma unroll
        for (int i = 0; i <= L12; ++i) {
            df v = prod(i == 0 && j == 0, Cp, G[i][j]);
            if (j > 0) v = mad(i == 0 && j == 1, j == 1 ? B1p : df_mulf(B1p, float(j)), G[i][j - 1], v);
            if (i > 0) v = mad(i == 1 && j == 0, i == 1 ? B00 : df_mulf(B00, float(i)), G[i - 1][j], v);
            G[i][j + 1] = v;
        }
    }
    df X[LB + 1][L12 + 1][L34 + 1];
#pragma unroll
    for (int a = 0; a <= L12; ++a)
#pragma unroll
        for (int j = 0; j <= L34; ++j) X[0][a][j] = G[a][j];
#pragma unroll
    for (int b = 1; b <= LB; ++b)
#pragma unroll
        for (int a = 0; a <= L12 - b; ++a)
#pragma unroll
            for (int j = 0; j <= L34; ++j)
                X[b][a][j] = mad(b == 1 && a == 0 && j == 0, AB, X[b - 1][a][j], X[b - 1][a + 1][j]);
#pragma unroll
    for (int a = 0; a <= LA; ++a)
#pragma unroll
        for (int b = 0; b <= LB; ++b) {
            df Y[LD + 1][L34 + 1];
#pragma unroll
            for (int c = 0; c <= L34; ++c) Y[0][c] = X[b][a][c];
#pragma unroll
            for (int d = 1; d <= LD; ++d)
#pragma unroll
                for (int c = 0; c <= L34 - d; ++c)
                    Y[d][c] = mad(a == 0 && b == 0 && c == 0 && d == 1, CD, Y[d - 1][c], Y[d - 1][c + 1]);
#pragma unroll
            for (int c = 0; c <= LC; ++c)
#pragma unroll
                for (int d = 0; d <= LD; ++d) I[((a * (LB + 1) + b) * (LC + 1) + c) * (LD + 1) + d] = Y[d][c];
        }
}

// FP32 -> FP64 through the integer pipe as f32_to_f64, with infinities and NaN kept
__device__ __forceinline__ double df_to_f64(df a) {
    auto cvt = [](float f) {
        const unsigned u = __float_as_uint(f);
        const unsigned e = (u >> 23) & 0xffu;
        const unsigned ex = e == 0xffu ? 0x7ffu : e + 896u;
        const unsigned hi = (u & 0x80000000u) | (e ? ((ex << 20) | ((u >> 3) & 0xfffffu)) : 0u);
        return __hiloint2double((int)hi, (int)(e ? (u << 29) : 0u));
    };
    return cvt(a.h) + cvt(a.l);
}

// SRTERM E_ab E_cd / sqrt(p + q) > PRIM_CUT on all 48 bits
__device__ __forceinline__ bool df_passes(df p, df Eab, df q, df Ecd) {
    const float sh = float(SRTERM), sl = float(SRTERM - double(float(SRTERM)));
    const float ch = float(PRIM_CUT), cl = float(PRIM_CUT - double(float(PRIM_CUT)));
    const df v = df_mul(df_mul({sh, sl}, df_mul(Eab, Ecd)), df_rsqrt(df_add(p, q)));
    return __fadd_rn(__fsub_rn(v.h, ch), __fsub_rn(v.l, cl)) > 0.f;
}

__device__ __forceinline__ df pair_ab(const ShellPair& p, int k) {
    return {p.ABf[k], k == 0 ? p.ABl0 : k == 1 ? p.ABl1 : p.ABl2};
}

// A - C of a quartet's bra and ket
__device__ __forceinline__ void centre_diff(const PairCentre& a, const PairCentre& c, df (&AC)[3]) {
    AC[0] = df_triple_diff(a.x.x, a.x.y, a.x.z, c.x.x, c.x.y, c.x.z);
    AC[1] = df_triple_diff(a.y.x, a.y.y, a.y.z, c.y.x, c.y.y, c.y.z);
    AC[2] = df_triple_diff(a.z.x, a.z.y, a.z.z, c.z.x, c.z.y, c.z.z);
}

// Contracted integrals of one shell quartet as shell_quartet_eri<..., double>, in double-float: the same
// primitive quartets (prefactor screen on floats, decided in double-float within 0.1 % of the cut).
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void shell_quartet_df64(const ShellPair& bra, const ShellPair& ket, const df (&AC)[3],
                                                   const PrimPairDF* __restrict__ prims, const float* __restrict__ tab,
                                                   float prim_cut32, bool compat, df (&acc)[QClass<LA, LB, LC, LD>::NF],
                                                   unsigned* npass, int part = 0, int nparts = 1) {
    using Q = QClass<LA, LB, LC, LD>;
    constexpr int NR = Q::NR;
    constexpr int L12 = LA + LB, L34 = LC + LD;
#pragma unroll
    for (int f = 0; f < Q::NF; ++f) acc[f] = {0.f, 0.f};
    const PrimPairDF* pb = prims + bra.prim_begin;
    const PrimPairDF* pk = prims + ket.prim_begin;
    const int nb = bra.nprim, nk = ket.nprim, sb = bra.prim_stride, sk = ket.prim_stride;
    const float lo32 = prim_cut32 * 0.999f, hi32 = prim_cut32 * 1.001f;
    // the prefactor screen on floats; in the band around the cut on all 48 bits (TwoElectronInts.cpp:478-479)
    auto passes = [&](const df& bp_p, const df& bp_E, const df& kp_p, const df& kp_E) {
        const float v32 = float(SRTERM) * bp_E.h * kp_E.h * rsqrtf(bp_p.h + kp_p.h);
        if (v32 < lo32) return false;
        if (v32 <= hi32 && !df_passes(bp_p, bp_E, kp_p, kp_E)) return false;
        return true;
    };
    // P - Q = AC + (P - A) - (Q - C), normalised before it is squared; AC with the record of the outer loop in `base`
    auto with_bra = [&](const PrimPairDF& bp, df (&base)[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) base[k] = df_add(AC[k], bp.PA[k]);
    };
    auto primitive = [&](const PrimPairDF& bp, const PrimPairDF& kp, const df& PQx, const df& PQy, const df& PQz) {
        if (npass) ++*npass;
        const df rs = df_rsqrt(df_add(bp.p, kp.p));
        // the factors that the rest is made of are normalised: the error of an integral falls from 15 to 11 (ss|ss), 12
        // to 7 (ps|ss) and 11 to 6 (ps|ps) units of 2^-53 of the bound (rms over random primitives)
        const df sr = df_muln(df_muln(bp.Ecc, kp.Ecc), rs);
        const df rpq = df_norm(df_sqr(rs));
        const df R2 = df_norm(df_add(df_add(df_sqr(PQx), df_sqr(PQy)), df_sqr(PQz)));
        const df T = df_mul(df_muln(df_muln(bp.p, kp.p), rpq), R2);
        df x[NR], w[NR];
        df_roots<NR, L12 + L34 != 0>(T, tab, compat, x, w);
        if constexpr (L12 + L34 == 0) {
            acc[0] = df_fma(df_norm(w[0]), sr, acc[0]);
        } else {
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const df fff = df_muln(df_norm(x[r]), rpq);  // t^2 / (p + q)   (Rys.hpp:126-129)
                const df zero = {0.f, 0.f};
                const df qf = L12 > 0 ? df_mul(kp.p, fff) : zero, pf = L34 > 0 ? df_mul(bp.p, fff) : zero;
                const df B00 = (L12 > 0 && L34 > 0) ? df_half(fff) : zero;
                // (1/2 - q B00) / p = (1 - q t^2 / (p + q)) / 2 p
                const df B1 = L12 > 1 ? df_half(df_mul(df_rsubf(1.f, qf), bp.rp)) : zero;
                const df B1p = L34 > 1 ? df_half(df_mul(df_rsubf(1.f, pf), kp.rp)) : zero;
                df Ix[Q::NI], Iy[Q::NI], Iz[Q::NI];
                const df nqf = df_neg(qf);
                auto axis = [&](int k, const df& PQ, auto unit, df g, df(&I)[Q::NI]) {
                    const df C = L12 > 0 ? df_norm(df_fma(nqf, PQ, bp.PA[k])) : zero;
                    const df Cp = L34 > 0 ? df_norm(df_fma(pf, PQ, kp.PA[k])) : zero;
                    const df AB = LB > 0 ? pair_ab(bra, k) : zero, CD = LD > 0 ? pair_ab(ket, k) : zero;
                    df_axis<LA, LB, LC, LD, decltype(unit)::value>(g, C, Cp, B00, B1, B1p, AB, CD, I);
                };
                axis(0, PQx, std::true_type{}, df{1.f, 0.f}, Ix);
                axis(1, PQy, std::true_type{}, df{1.f, 0.f}, Iy);
                axis(2, PQz, std::false_type{}, df_muln(df_norm(w[r]), sr), Iz);
#pragma unroll
                for (int ia = 0; ia < Q::NA; ++ia)
#pragma unroll
                    for (int ibb = 0; ibb < Q::NB; ++ibb)
#pragma unroll
                        for (int ic = 0; ic < Q::NC; ++ic)
#pragma unroll
                            for (int id = 0; id < Q::ND; ++id) {
                                const int f = ((ia * Q::NB + ibb) * Q::NC + ic) * Q::ND + id;
                                const int jx = Q::iidx(cart_lx(LA, ia), cart_lx(LB, ibb), cart_lx(LC, ic), cart_lx(LD, id));
                                const int jy = Q::iidx(cart_ly(LA, ia), cart_ly(LB, ibb), cart_ly(LC, ic), cart_ly(LD, id));
                                const int jz = Q::iidx(cart_lz(LA, ia), cart_lz(LB, ibb), cart_lz(LC, ic), cart_lz(LD, id));
                                // element 0 of the x and y axes is 1
                                if (jx == 0 && jy == 0) acc[f] = df_add(acc[f], Iz[jz]);
                                else if (jx == 0) acc[f] = df_fma(Iy[jy], Iz[jz], acc[f]);
                                else if (jy == 0) acc[f] = df_fma(Ix[jx], Iz[jz], acc[f]);
                                else acc[f] = df_fma(df_mul(Ix[jx], Iy[jy]), Iz[jz], acc[f]);
                            }
            }
        }
    };
    if (nparts > 1) {  // the caller's lanes split the quartet (as shell_quartet_eri)
        for (int t = part; t < nb * nk; t += nparts) {
            const int ib = t / nk, ik = t - ib * nk;
            const PrimPairDF bp = pb[ib * sb];
            const PrimPairDF kp = pk[ik * sk];
            if (!passes(bp.p, bp.E, kp.p, kp.E)) continue;
            df base[3];
            with_bra(bp, base);
            primitive(bp, kp, df_diff(base[0], kp.PA[0]), df_diff(base[1], kp.PA[1]), df_diff(base[2], kp.PA[2]));
        }
        return;
    }
    if constexpr (L12 + L34 == 2) {
        int ib = 0, ik = 0, cb = -1;
        float rowf = 0.f;  // bound of SRTERM E_ab / sqrt(p + q) over the kets
        PrimPairDF bp = pb[0];
        df base[3];
        with_bra(bp, base);
        for (;;) {
            PrimPairDF kp;
            bool found = false;
            while (ib < nb) {
                if (ib != cb) {
                    bp = pb[ib * sb];
                    cb = ib;
                    rowf = float(SRTERM) * bp.E.h * rsqrtf(bp.p.h);
                    with_bra(bp, base);
                }
                kp = pk[ik * sk];
                if (rowf * kp.E.h < lo32) {  // E_cd descends: no later ket primitive passes either
                    ik = 0;
                    ++ib;
                    continue;
                }
                if (++ik == nk) {
                    ik = 0;
                    ++ib;
                }
                if (!passes(bp.p, bp.E, kp.p, kp.E)) continue;
                found = true;
                break;
            }
            if (!found) break;
            primitive(bp, kp, df_diff(base[0], kp.PA[0]), df_diff(base[1], kp.PA[1]), df_diff(base[2], kp.PA[2]));
        }
    } else {
        for (int ik = 0; ik < nk; ++ik) {
            const PrimPairDF kp = pk[ik * sk];
            const float colf = float(SRTERM) * kp.E.h * rsqrtf(kp.p.h);
            df base[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) base[k] = df_sub(AC[k], kp.PA[k]);
            for (int ib = 0; ib < nb; ++ib) {
                const PrimPairDF bp = pb[ib * sb];
                if (colf * bp.E.h < lo32) break;  // E_ab descends: no later bra primitive passes either
                if (!passes(bp.p, bp.E, kp.p, kp.E)) continue;
                primitive(bp, kp, df_norm(df_add(base[0], bp.PA[0])), df_norm(df_add(base[1], bp.PA[1])),
                          df_norm(df_add(base[2], bp.PA[2])));
            }
        }
    }
}

// One quartet: integrals in pairs of floats, density contraction and scatter in FP64 as the FP64 kernels.
template <int LA, int LB, int LC, int LD, bool UHF>
__device__ __forceinline__ void df_item(const FockArgs& A, const NormTable& nt, long long g) {
    using Q = QClass<LA, LB, LC, LD>;
    int bi, ki;
    if (!decode_work_warp<true>(A, g, bi, ki)) return;
    const ShellPair bra = A.pairs[bi];
    const ShellPair ket = A.pairs[ki];
    if (A.mode == 1) {  // the FP64 part of a mixed build: the others are the group kernel's
        if (!(bra.qf * ket.qf < A.split_cut32)) return;
        const float bound = quartet_bound(A, bra, ket);
        if (bound < A.skip_cut32 || bound < A.fp32_cut32) return;
    }
    unsigned npass = 0;
    double v[Q::NF];
    {
        df acc[Q::NF], AC[3];
        centre_diff(A.pcen[bi], A.pcen[ki], AC);
        shell_quartet_df64<LA, LB, LC, LD>(bra, ket, AC, A.primsdf, A.rysdf, A.prim_cut32, A.rys_compat != 0, acc,
                                           A.counters ? &npass : nullptr);
#pragma unroll
        for (int f = 0; f < Q::NF; ++f) v[f] = df_to_f64(acc[f]);
    }
    digest_jk<LA, LB, LC, LD, UHF, double>(A, bra, ket, bi == ki, v, nt);
    if (A.counters) count_flush(A, npass);
}

// The quartets below SPLIT_CUT of one class (its split list).
template <int LA, int LB, int LC, int LD, bool UHF>
__global__ void __launch_bounds__(128, LA + LB + LC + LD <= 1 ? 8 : 1) fock_jk_df64(const FockArgs A, const NormTable nt) {
    df_item<LA, LB, LC, LD, UHF>(A, nt, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// The same for batches of molecules: a fixed grid pulling tiles (as fock_jk_persistent).
template <int LA, int LB, int LC, int LD, bool UHF>
__global__ void __launch_bounds__(256, LA + LB + LC + LD <= 1 ? 4 : 1) fock_jk_df64_persistent(const FockArgs A, const NormTable nt) {
    __shared__ long long tile;
    const long long end = *A.dyn_total;
    for (;;) {
        if (threadIdx.x == 0) tile = (long long)atomicAdd(A.tile_counter, 1ull);
        __syncthreads();
        const long long g0 = tile * blockDim.x;
        __syncthreads();
        if (g0 >= end) return;
        df_item<LA, LB, LC, LD, UHF>(A, nt, g0 + threadIdx.x);
    }
}

// Sums of the 32 lanes' acc[0..N), scattered: the lane ends with the sums of elements first .. first + count - 1
// in acc[0 ..].  Halving exchanges: in each the lane keeps one half of its elements and adds its partner's.
__device__ __forceinline__ double sum_exchange(double keep, double send, int o) {
    return keep + __shfl_xor_sync(0xffffffffu, send, o);
}
__device__ __forceinline__ df sum_exchange(df keep, df send, int o) {
    return df_add(keep, {__shfl_xor_sync(0xffffffffu, send.h, o), __shfl_xor_sync(0xffffffffu, send.l, o)});
}
template <int N, int O, class T, int M>
__device__ __forceinline__ void reduce_scatter(T (&acc)[M], int& first, int& count) {
    constexpr int H = (N + 1) / 2;
    const bool upper = threadIdx.x & O;
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const T lo = acc[i], hi = i + H < N ? acc[i + H < N ? i + H : 0] : T{};
        acc[i] = sum_exchange(upper ? hi : lo, upper ? lo : hi, O);
    }
    first += upper ? H : 0;
    count = upper ? max(count - H, 0) : min(count, H);
    if constexpr (O > 1) reduce_scatter<H, O / 2>(acc, first, count);
}
__host__ __device__ constexpr int scatter_left(int n) {  // elements per lane after the five exchanges
    for (int k = 0; k < 5; ++k) n = (n + 1) / 2;
    return n;
}
// Shared memory of the contraction by a warp, in doubles: the integrals (odd row stride) and the density blocks.
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr int group_smem() {
    using Q = QClass<LA, LB, LC, LD>;
    return Q::NA * Q::NB * ((Q::NC * Q::ND) | 1) + Q::NA * Q::NB + Q::NC * Q::ND + (Q::NA + Q::NB) * (Q::NC + Q::ND);
}

// quartet_item_group (fock_kernels.cuh) in pairs of floats.
template <int LA, int LB, int LC, int LD, bool UHF, int NP>
__device__ __forceinline__ void quartet_item_group_df(const FockArgs& A, const NormTable& nt, const ShellPair& bra,
                                                      const ShellPair& ket, int bi, int ki, int part, unsigned gmask) {
    using Q = QClass<LA, LB, LC, LD>;
    unsigned npass = 0;
    double v[Q::NF];
    {
        df acc[Q::NF], AC[3];
        centre_diff(A.pcen[bi], A.pcen[ki], AC);
        shell_quartet_df64<LA, LB, LC, LD>(bra, ket, AC, A.primsdf, A.rysdf, A.prim_cut32, A.rys_compat != 0, acc,
                                           A.counters ? &npass : nullptr, part, NP);
#pragma unroll
        for (int o = 1; o < NP; o <<= 1)
#pragma unroll
            for (int f = 0; f < Q::NF; ++f)
                acc[f] = df_add(acc[f], {__shfl_xor_sync(gmask, acc[f].h, o), __shfl_xor_sync(gmask, acc[f].l, o)});
#pragma unroll
        for (int f = 0; f < Q::NF; ++f) v[f] = df_to_f64(acc[f]);
    }
    if (part == 0) digest_jk<LA, LB, LC, LD, UHF, double>(A, bra, ket, bi == ki, v, nt);
    if (A.counters) count_flush(A, npass);
}

// One quartet of a split list (or, mode 0, of the class's whole list) on NP lanes, each summing every NP-th primitive quartet: where a launch holds few
// quartets, one lane each leaves the GPU idle behind a serial chain of primitive quartets (water in STO-3G, 81
// of them per quartet: 1.36 -> 0.17 ms per build with a warp each).  DF: in pairs of floats (below SPLIT_CUT),
// otherwise in FP64 (the others: few, and the costliest of the build).
template <int LA, int LB, int LC, int LD, bool UHF, int NP, bool DF>
__global__ void __launch_bounds__(128) fock_jk_group(const FockArgs A, const NormTable nt, const double* __restrict__ rys) {
    using Q = QClass<LA, LB, LC, LD>;
    const int lane = threadIdx.x & 31, sub = lane / NP, part = lane % NP;
    const unsigned gmask = NP == 32 ? 0xffffffffu : ((1u << (NP & 31)) - 1u) << (sub * NP);
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int bi, ki;
    const long long g0 = warp * (32 / NP);
    if (!(A.mode == 0 ? decode_warp_items<false>(A, g0, sub, bi, ki) : decode_warp_items<true>(A, g0, sub, bi, ki))) return;
    const ShellPair bra = A.pairs[bi];
    const ShellPair ket = A.pairs[ki];
    if (A.mode == 1) {  // the FP64 part of a mixed build: the quartets on this kernel's side of SPLIT_CUT that stay in it
        if ((bra.qf * ket.qf < A.split_cut32) != DF) return;
        const float bound = quartet_bound(A, bra, ket);
        if (bound < A.skip_cut32 || bound < A.fp32_cut32) return;
    }
    if constexpr (NP == 32) {
        // the lanes' partial sums scattered over the warp (81 elements: 82 additions per lane, 405 where every lane
        // gets every sum), then the contraction by all lanes: (pp|pp) of water in STO-3G 112 -> 68 us, four waters
        // with d shells 1.15 -> 0.75 ms per build
        extern __shared__ double smem[];
        constexpr int VS = (Q::NC * Q::ND) | 1;
        double* V = smem + (threadIdx.x >> 5) * group_smem<LA, LB, LC, LD>();
        unsigned npass = 0;
        std::conditional_t<DF, df, double> acc[Q::NF];
        if constexpr (DF) {
            df AC[3];
            centre_diff(A.pcen[bi], A.pcen[ki], AC);
            shell_quartet_df64<LA, LB, LC, LD>(bra, ket, AC, A.primsdf, A.rysdf, A.prim_cut32, A.rys_compat != 0, acc,
                                               A.counters ? &npass : nullptr, part, NP);
        } else
            shell_quartet_eri<LA, LB, LC, LD, double, PrimPair>(bra, ket, A.prims, rys, A.prim_cut, A.prim_cut32, A.rys_compat != 0,
                                                                acc, A.counters ? &npass : nullptr, part, NP);
        int first = 0, count = Q::NF;
        reduce_scatter<Q::NF, 16>(acc, first, count);
        const int ndeg = (bra.same() ? 1 : 0) + (ket.same() ? 1 : 0) + (bi == ki ? 1 : 0);
        constexpr int LEFT = scatter_left(Q::NF);
#pragma unroll
        for (int i = 0; i < LEFT; ++i)
            if (i < count) {
                const int f = first + i, ab = f / (Q::NC * Q::ND), cd = f - ab * (Q::NC * Q::ND);
                double v;
                if constexpr (DF) v = df_to_f64(acc[i]);
                else v = acc[i];
                if constexpr (LA > 1 || LB > 1 || LC > 1 || LD > 1)
                    v *= nt.v[LA][ab / Q::NB] * nt.v[LB][ab % Q::NB] * nt.v[LC][cd / Q::ND] * nt.v[LD][cd % Q::ND];
                V[ab * VS + cd] = above_cut(v, A.thr_int) ? scale_pow2(v, -ndeg) : 0.0;
            }
        digest_shared(A, bra, ket, V, Q::NA, Q::NB, Q::NC, Q::ND, VS);
        if (A.counters) count_flush(A, npass);
    } else if constexpr (!DF) {
        quartet_item_group<LA, LB, LC, LD, UHF, double, NP>(A, nt, rys, bra, ket, bi == ki, part, gmask);
    } else {
        quartet_item_group_df<LA, LB, LC, LD, UHF, NP>(A, nt, bra, ket, bi, ki, part, gmask);
    }
}

}  // namespace ugb
