// Layout of the root tables (rys_tables.inc) on the device.
#pragma once
#include "rys_tables.inc"

namespace ugb {

template <typename R> struct RysDeg;
template <> struct RysDeg<double> { static constexpr int value = RYS_DEG; };
template <> struct RysDeg<float> { static constexpr int value = RYS32_DEG; };
// Row length of one polynomial in the device tables: the coefficients padded to a multiple of 16
// bytes, so that a row is read with 16-byte loads (FP64: 10 doubles; FP32: 6 floats padded to 8).
template <typename R> struct RysStride;
template <> struct RysStride<double> { static constexpr int value = (RYS_DEG + 2) / 2 * 2; };
template <> struct RysStride<float> { static constexpr int value = (RYS32_DEG + 4) / 4 * 4; };
// Interval width in T of each precision's table (a power of two: T / H is exact).
template <typename R> struct RysH;
template <> struct RysH<double> { static constexpr double value = RYS_H; };
template <> struct RysH<float> { static constexpr double value = RYS32_H; };

__host__ __device__ constexpr double rys_tmax(int n) {
    return n == 1 ? RYS_TMAX_1 : n == 2 ? RYS_TMAX_2 : n == 3 ? RYS_TMAX_3 : n == 4 ? RYS_TMAX_4 : RYS_TMAX_5;
}
// Offset of the n-root block in a table of interval width h whose polynomial rows hold `stride`
// coefficients (rys_tables.inc with stride = degree + 1; the device tables with the padded strides of
// RysStride).
__host__ __device__ constexpr int rys_off(int n, int stride, double h) {
    int o = 0;
    for (int m = 1; m < n; ++m) o += int(rys_tmax(m) / h) * 2 * m * stride;
    return o;
}
// Size of a device table: polynomial blocks, then hermite x[5][5] and w[5][5].
__host__ __device__ constexpr int rys_table_len(int stride, double h) { return rys_off(RYS_NMAX + 1, stride, h) + 50; }

}  // namespace ugb
