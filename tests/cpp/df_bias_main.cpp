// Mean relative errors of the pairs of floats (df64.cuh) on the host, in units of 2^-53: squares of normalised values,
// and the square of the reciprocal square root.
#include <cmath>
#include <cstdio>
#include <random>

#include <cuda_runtime.h>

static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static std::mt19937_64 coin(9);
static inline float rsqrtf(float a) {  // within the two ulps that CUDA documents: one either way in half of the calls
    const float r = (float)(1.0 / std::sqrt((double)a));
    const int k = coin() % 4;
    return k == 0 ? std::nextafterf(r, 0.f) : k == 1 ? std::nextafterf(r, 1e30f) : r;
}

#include "df64.cuh"

using namespace ugb;

int main() {
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> u(-5.0, 5.0);
    const int n = 2000000;
    double sq = 0.0, rq = 0.0;
    for (int i = 0; i < n; ++i) {
        const double v = std::exp(u(rng));
        const df a = {(float)v, (float)(v - (double)(float)v)};
        // error of p + e against a^2, term by term: the differences of products below are exact in doubles
        const df s = df_sqr(a);
        const double exact_hh = (double)a.h * a.h, rest = 2.0 * (double)a.h * a.l + (double)a.l * a.l;
        sq += (((double)s.h - exact_hh) + ((double)s.l - rest)) / exact_hh;
        const df r = df_sqr(df_rsqrt(a));  // 1 / a: r a - 1
        const double ph = (double)r.h * a.h;
        rq += (ph - 1.0) + ((double)r.h * a.l + (double)r.l * a.h + (double)r.l * a.l);
    }
    std::printf("%.4f %.4f\n", sq / n * 0x1p53, rq / n * 0x1p53);
    return 0;
}
