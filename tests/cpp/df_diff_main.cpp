// Squared differences of close values in pairs of floats (df64.cuh), on the host.  Prints the number of values
// looked at and of wrong ones.
#include <cmath>
#include <cstdio>
#include <random>

#include <cuda_runtime.h>

static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static inline float rsqrtf(float a) { return (float)(1.0 / std::sqrt((double)a)); }

#include "df64.cuh"

using namespace ugb;

int main() {
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    long long looked = 0, wrong = 0;
    for (double far : {1.0, 15.0, 60.0, 2000.0})
        for (double near : {1e-3, 0.1, 1.0, 10.0})
            for (int n = 0; n < 20000; ++n) {
                auto split = [](double v) {
                    const float h = (float)v;
                    return df{h, (float)(v - (double)h)};
                };
                const double x = far * u(rng);
                const df a = split(x), b = split(x + near * u(rng));
                const double d = ((double)a.h - (double)b.h) + ((double)a.l - (double)b.l);
                const df s = df_sqr(df_diff(a, b));
                // the difference to a few 2^-48 of the values that enter, its square to a few 2^-48 of itself
                const double tol = 2.0 * std::fabs(d) * 0x1p-46 * (far + near) + 0x1p-45 * d * d + 0x1p-92 * (far + near) * (far + near);
                ++looked;
                if (!(std::fabs(((double)s.h + s.l) - d * d) <= tol)) ++wrong;
            }
    std::printf("%lld %lld\n", looked, wrong);
    return 0;
}
