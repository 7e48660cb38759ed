// Rys nodes and weights in pairs of floats.  The includer provides load_row (eight consecutive floats).
#pragma once
#include "df64.cuh"
#include "rys_layout.cuh"

namespace ugb {

// Rows of the root tables: 8 leading parts (highest power first), then the 8 remainders.
constexpr int DF_STRIDE = 16;
constexpr int DF_ROWS_END = rys_off(RYS_NMAX + 1, DF_STRIDE, RYS_H);
// a second two-root block whose intervals in (15, 40] hold the reference's own large-T form
constexpr int DF_COMPAT2 = DF_ROWS_END;
constexpr int DF_HERMITE = DF_COMPAT2 + rys_off(3, DF_STRIDE, RYS_H) - rys_off(2, DF_STRIDE, RYS_H);
constexpr int DF_TABLE_LEN = DF_HERMITE + 100;  // x[5][5] (h, l), w[5][5] (h, l)
static_assert(RYS_DEG == 7 && RYS_H == 0.25, "the double-float table rows and the index below");

// One table polynomial at y = yh + yl.  Coefficient k is about 0.125^k / k! of the first, so the three
// highest powers need only floats: their rounding lies below 2^-50 of the value.
__device__ __forceinline__ df df_poly(const float* __restrict__ c, float yh, float yl) {
    float h[8], l[8];
    load_row(c, h);
    load_row(c + 8, l);
    float v = __fmaf_rn(h[0], yh, h[1]);
    // power 5: its own leading part, everything above it in the remainder
    df r = {h[2], __fmaf_rn(v, yh, l[2])};
#pragma unroll
    for (int k = 3; k < 8; ++k) {
        const float p = __fmul_rn(r.h, yh);
        float e = __fmaf_rn(r.h, yh, -p);
        e = __fmaf_rn(r.l, yh, e);
        e = __fmaf_rn(r.h, yl, e);
        const df t = df_add({h[k], l[k]}, {p, e});
        r = t;
    }
    return r;
}

// Interval k and local coordinate y = yh + yl = 2 (T / H - k) - 1 of a normalised T below the table's end.
// above: intervals (k H, (k + 1) H], for the two-root tables (the reference's form starts above T = 15 and
// ends at T = 40); else [k H, (k + 1) H).
__device__ __forceinline__ int df_index(bool above, df T, float& yh, float& yl) {
    const float f = 4.0f * T.h;
    int k;
    if (above) {
        const float c = ceilf(f);
        k = max((int)c - ((c == f && T.l > 0.f) ? 0 : 1), 0);
    } else {
        k = max((int)f, 0);
    }
    // 8 T - (2 k + 1); the leading part rounds only below T = 1/8
    const float T8 = 8.0f * T.h, m = float(2 * k + 1);
    yh = __fsub_rn(T8, m);
    yl = __fmaf_rn(8.0f, T.l, __fsub_rn(T8, __fadd_rn(yh, m)));
    return k;
}

// Rys nodes and weights in double-float, as rys_roots.  compat: the two-root block with the reference's form
// in 15 < T <= 40.  T comes in unnormalised; its leading part as the rounded sum decides the range and the
// interval alike, and with the sign of the rest the side of 15: a leading part a few ulps off the sum would
// pass the test at the table's end with an interval past it, or take the other side of 15.
template <int NR, bool NEED_X>
__device__ __forceinline__ void df_roots(df T, const float* __restrict__ tab, bool compat, df* x, df* w) {
    constexpr float TMAX = float(rys_tmax(NR));
    T = df_norm(T);
    if (T.h < TMAX) {
        float yh, yl;
        const int k = df_index(NR == 2, T, yh, yl);
        const float* blk = tab + (NR == 2 && compat ? DF_COMPAT2 : rys_off(NR, DF_STRIDE, RYS_H)) + k * (2 * NR * DF_STRIDE);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            if (NEED_X) x[i] = df_poly(blk + 2 * i * DF_STRIDE, yh, yl);
            w[i] = df_poly(blk + (2 * i + 1) * DF_STRIDE, yh, yl);
        }
    } else {
        const float2* herm = reinterpret_cast<const float2*>(tab + DF_HERMITE);
        const df s = df_rsqrt(T);
        const df r = df_sqr(s);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const float2 hx = __ldg(herm + (NR - 1) * 5 + i), hw = __ldg(herm + 25 + (NR - 1) * 5 + i);
            if (NEED_X) x[i] = df_mul({hx.x, hx.y}, r);
            w[i] = df_mul({hw.x, hw.y}, s);
        }
    }
}

}  // namespace ugb
