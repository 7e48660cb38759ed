// df_roots.cuh on the host: the CUDA intrinsics by their IEEE meaning, and a table whose polynomial of interval
// k is T itself, (k + 1/2) H + (H / 2) y, with NaN wherever no interval of the block lies.  What comes back for
// T must be T below the table's end and the Hermite form (nodes 1 / T, weights 1 / sqrt(T)) from it on.  Prints
// the number of values looked at and of wrong ones.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include <cuda_runtime.h>

static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static inline float rsqrtf(float a) { return (float)(1.0 / std::sqrt((double)a)); }
template <class T> static inline T __ldg(const T* p) { return *p; }
static inline int max(int a, int b) { return a > b ? a : b; }
static inline void load_row(const float* c, float (&v)[8]) { std::memcpy(v, c, sizeof(v)); }

#include "df_roots.cuh"

using namespace ugb;

static long long looked = 0, wrong = 0;

template <int NR>
void check(float h, float l, const std::vector<float>& tab, bool compat) {
    df x[NR], w[NR];
    df_roots<NR, true>({h, l}, tab.data(), compat, x, w);
    const double T = (double)h + (double)l;
    const bool table = (float)T < (float)rys_tmax(NR);
    for (int i = 0; i < NR; ++i) {
        const double gx = (double)x[i].h + x[i].l, gw = (double)w[i].h + w[i].l;
        const double ex = table ? T : 1.0 / T, ew = table ? T : 1.0 / std::sqrt(T);
        ++looked;
        // a handful of operations of 2^-47 each, of the value or of the table's terms (up to H / 2)
        const double tol = table ? 0x1p-43 * (T + RYS_H) : 0x1p-43 * ew;
        if (!(std::fabs(gx - ex) <= tol) || !(std::fabs(gw - ew) <= tol)) {
            if (++wrong <= 5) std::printf("NR %d compat %d T %.17g (%a + %a): %.17g %.17g\n", NR, compat, T, h, l, gx, gw);
        }
    }
}

int main() {
    std::vector<float> tab(DF_TABLE_LEN, std::numeric_limits<float>::quiet_NaN());
    auto block = [&](int off, int nr) {
        for (int k = 0; k < int(rys_tmax(nr) / RYS_H); ++k)
            for (int r = 0; r < 2 * nr; ++r) {
                float* c = &tab[off + (k * 2 * nr + r) * DF_STRIDE];
                for (int d = 0; d < 16; ++d) c[d] = 0.f;
                c[6] = (float)(RYS_H / 2);
                c[7] = (float)((k + 0.5) * RYS_H);
            }
    };
    for (int nr = 1; nr <= 3; ++nr) block(rys_off(nr, DF_STRIDE, RYS_H), nr);
    block(DF_COMPAT2, 2);
    for (int i = 0; i < 50; ++i) {
        tab[DF_HERMITE + 2 * i] = 1.f;
        tab[DF_HERMITE + 2 * i + 1] = 0.f;
    }
    std::mt19937_64 rng(7);
    auto both = [&](float h, float l) {
        check<1>(h, l, tab, false);
        check<2>(h, l, tab, false);
        check<2>(h, l, tab, true);
        check<3>(h, l, tab, false);
    };
    // on both sides of the two-root form's edges and of every table's end, leading parts up to 16 ulps off the sum
    for (double edge : {0.25, 15.0, 15.25, 40.0, 41.0, 48.0, 55.0, 62.0, 68.0})
        for (int n = 0; n < 20000; ++n) {
            const double T = edge * (1.0 + (double)((long long)(rng() % 2048) - 1024) * 0x1p-32 * (n & 1 ? 1.0 : 64.0));
            const float ulp = std::nextafterf((float)edge, 100.f) - (float)edge;
            const float h = (float)((float)T + ulp * (float)((long long)(rng() % 33) - 16));
            both(h, (float)(T - (double)h));
        }
    for (int n = 0; n < 200000; ++n) {  // and anywhere
        const double T = std::exp(std::uniform_real_distribution<double>(std::log(1e-3), std::log(200.0))(rng));
        const float h = (float)(T * (1.0 + 0x1p-24 * (double)((long long)(rng() % 17) - 8)));
        both(h, (float)(T - (double)h));
    }
    std::printf("%lld %lld\n", looked, wrong);
    return 0;
}
