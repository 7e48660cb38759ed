// Fock kernels of the classes without a template (more than 81 function quartets, f and g shells;
// la+lb+lc+ld <= 8): one warp per shell quartet.  Per primitive quartet the lanes share out the roots, the
// recurrence (one lane per root and axis), the two horizontal transfers (element by element) and the function
// quartets, of which each lane keeps every 32nd in registers; the 1D tables pass through shared memory.  The
// contraction with the density then goes output by output: the quartet's integrals and its six density blocks
// in shared memory, one lane per J or K element, one atomic per element of T.
//
// Why this form: with one thread per quartet the runtime-L arrays (up to 1296 integrals and the transfer
// tables) live in local memory and five atomics per function quartet go to L2; four waters with d shells took
// 18 ms that way (6.3 ms with three such builds in flight) and take 1.4 ms (0.71), of which these kernels are a
// fifth; the chain of barriers and shared-memory loads of a quartet is what bounds them now.
//
// All in FP64: with the quartets below a bound in pairs of floats (fock_df64.cuh) the build takes 1.38 ms
// against 1.34, because the FP64 pipe does not bind it, and with the cut of the templated classes the error of
// G grows threefold where f and g shells take part.  References as fock_kernels.cuh.
#pragma once
#include "fock_kernels.cuh"

namespace ugb {

// One root's node and weight at T: the lane's own rows of the tables of rys_roots.
__device__ __forceinline__ void coop_root(int nr, int r, double T, const double* __restrict__ tab, bool compat, double& x, double& w) {
    if (nr == 2 && compat && T > 15.0 && T <= 40.0) {
        double xs[2], ws[2];
        rys2_reference_regime(T, xs, ws);
        x = r ? xs[1] : xs[0];
        w = r ? ws[1] : ws[0];
        return;
    }
    constexpr int ST = RysStride<double>::value;
    int k, off = 0;
    double tmax = 0.0, y;
#pragma unroll
    for (int n = 1; n <= RYS_NMAX; ++n)
        if (n == nr) {
            off = rys_off(n, ST, RYS_H);
            tmax = rys_tmax(n);
        }
    if (rys_index64(T, tmax, k, y)) {
        const double* c = tab + off + (k * nr + r) * (2 * ST);
        double cx[ST], cw[ST];
        load_row(c, cx);
        load_row(c + ST, cw);
        x = cx[0];
        w = cw[0];
#pragma unroll
        for (int d = 1; d <= RYS_DEG; ++d) {
            x = fma(x, y, cx[d]);
            w = fma(w, y, cw[d]);
        }
    } else {
        const double* herm = tab + rys_table_len(ST, RYS_H) - 50;
        const double rT = 1.0 / T, s = sqrt(rT);
        x = __ldg(herm + (nr - 1) * 5 + r) * rT;
        w = __ldg(herm + 25 + (nr - 1) * 5 + r) * s;
    }
}

// Sizes of one class and its shared-memory layout (host and device).
struct CoopShape {
    int la, lb, lc, ld, l12, l34, nr, na, nb, nc, nd, nab, ncd, nf, ng, nhb, ni;
    int vs, pblk;   // row stride of the integrals in shared memory; density elements
    int per_warp;   // 8-byte words per warp
    int per_cta;    // 8-byte words shared by the CTA: function indices, transfer indices, norms
    __host__ __device__ CoopShape(int a, int b, int c, int d) : la(a), lb(b), lc(c), ld(d) {
        l12 = la + lb, l34 = lc + ld, nr = (l12 + l34) / 2 + 1;
        na = ncart(la), nb = ncart(lb), nc = ncart(lc), nd = ncart(ld);
        nab = na * nb, ncd = nc * nd, nf = nab * ncd;
        ng = (l12 + 1) * (l34 + 1);
        nhb = lb > 0 ? (la + 1) * (lb + 1) * (l34 + 1) : ld > 0 ? ng : 0;  // no bra transfer: the recurrence itself
        ni = (la + 1) * (lb + 1) * (lc + 1) * (ld + 1);
        vs = ncd | 1;  // odd: the lanes of a column of ab hit different banks
        pblk = nab + ncd + na * nc + na * nd + nb * nc + nb * nd;
        const int tables = 3 * nr * ((ng > ni ? ng : ni) + nhb) + 2 * nr + 90;  // 90: transfer coefficients
        const int fin = nab * vs + pblk;
        per_warp = tables > fin ? tables : fin;
        per_cta = (nf + 1) / 2 + (ni + 1) / 2 + nab + ncd;
    }
};

constexpr int COOP_WARPS = 4;

// KF: function quartets per lane.  The work list is the class's own (mode 0) or a screened build's FP64 part (1).
template <int KF>
__global__ void __launch_bounds__(32 * COOP_WARPS) fock_jk_coop(const FockArgs A, const NormTable nt, const double* __restrict__ rys,
                                                                int la, int lb, int lc, int ld) {
    extern __shared__ double smem[];
    const long long cta = (long long)blockIdx.y * gridDim.x + blockIdx.x;
    if (A.mode != 0 && cta * COOP_WARPS >= *A.dyn_total) return;  // past a screened list's end
    const CoopShape q(la, lb, lc, ld);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // CTA tables: per function quartet its element of the three axes, per transfer element (a, b, c, d), norms
    unsigned* fidx = reinterpret_cast<unsigned*>(smem);
    unsigned* tidx = reinterpret_cast<unsigned*>(smem + (q.nf + 1) / 2);
    double* nab = smem + (q.nf + 1) / 2 + (q.ni + 1) / 2;
    double* ncd = nab + q.nab;
    for (int f = threadIdx.x; f < q.nf; f += blockDim.x) {
        const int id = f % q.nd, ic = f / q.nd % q.nc, ib = f / q.ncd % q.nb, ia = f / (q.ncd * q.nb);
        auto at = [&](int a, int b, int c, int d) { return ((a * (lb + 1) + b) * (lc + 1) + c) * (ld + 1) + d; };
        fidx[f] = at(cart_lx(la, ia), cart_lx(lb, ib), cart_lx(lc, ic), cart_lx(ld, id)) |
                  at(cart_ly(la, ia), cart_ly(lb, ib), cart_ly(lc, ic), cart_ly(ld, id)) << 8 |
                  at(cart_lz(la, ia), cart_lz(lb, ib), cart_lz(lc, ic), cart_lz(ld, id)) << 16;
    }
    for (int e = threadIdx.x; e < q.ni; e += blockDim.x) {
        const int d = e % (ld + 1), c = e / (ld + 1) % (lc + 1), ab = e / ((ld + 1) * (lc + 1));
        tidx[e] = d | c << 8 | ab << 16;
    }
    for (int e = threadIdx.x; e < q.nab; e += blockDim.x) nab[e] = nt.v[la][e / q.nb] * nt.v[lb][e % q.nb];
    for (int e = threadIdx.x; e < q.ncd; e += blockDim.x) ncd[e] = nt.v[lc][e / q.nd] * nt.v[ld][e % q.nd];
    __syncthreads();
    const long long w = cta * COOP_WARPS + wid;
    int bi, ki;
    if (!(A.mode == 0 ? decode_warp_items<false>(A, w, 0, bi, ki) : decode_warp_items<true>(A, w, 0, bi, ki))) return;
    const ShellPair bra = A.pairs[bi];
    const ShellPair ket = A.pairs[ki];
    if (A.mode == 1 && quartet_bound(A, bra, ket) < A.skip_cut32) {
        if (A.counters && lane == 0) count_screened(A);
        return;
    }
    double* base = smem + q.per_cta + (size_t)wid * q.per_warp;
    double* Ht = base;                                    // bra transfer [root, axis][nhb]
    double* It = Ht + 3 * q.nr * q.nhb;                   // recurrence, then ket transfer [root, axis][max(ng, ni)]
    const int ist = q.ng > q.ni ? q.ng : q.ni;
    double* xw = It + 3 * q.nr * ist;
    double* cab = xw + 2 * q.nr;                          // binom(b, k) AB^(b - k) at [axis][b (b + 1) / 2 + k]
    double* ccd = cab + 45;
    // the recurrence G where the next step does not write: in It before a bra transfer (and as the result when
    // there is no transfer at all), in Ht when the ket transfer reads it
    double* Gt = lb == 0 && ld > 0 ? Ht : It;
    const int gst = lb == 0 && ld > 0 ? q.nhb : ist;
    for (int e = lane; e < 90; e += 32) {
        const bool isk = e >= 45;
        const int ax = e % 45 / 15, t = e % 15;
        const int b = (t >= 1) + (t >= 3) + (t >= 6) + (t >= 10), k = t - b * (b + 1) / 2;
        const double X = (isk ? ket : bra).AB[ax];
        float bin = 1.f;
        for (int i = 1; i <= k; ++i) bin = bin * float(b - k + i) / float(i);
        double v = double(bin);
        for (int i = 0; i < b - k; ++i) v = v * X;
        cab[e] = v;
    }
    double acc[KF];
#pragma unroll
    for (int k = 0; k < KF; ++k) acc[k] = 0.0;
    const PrimPair* pb = A.prims + bra.prim_begin;
    const PrimPair* pk = A.prims + ket.prim_begin;
    const int nk = ket.nprim, np = bra.nprim * nk, sb = bra.prim_stride, sk = ket.prim_stride;
    const float lo32 = A.prim_cut32 * 0.999f, hi32 = A.prim_cut32 * 1.001f;
    const bool compat = A.rys_compat != 0;
    unsigned npass = 0;
    for (int t0 = 0; t0 < np; t0 += 32) {
        // 32 primitive quartets screened at once (TwoElectronInts.cpp:478-479)
        bool ok = false;
        if (t0 + lane < np) {
            const int ib = (t0 + lane) / nk, ik = (t0 + lane) - ib * nk;
            const PrimPair &b = pb[ib * sb], &k = pk[ik * sk];
            const float v32 = float(SRTERM) * b.Ef * k.Ef * rsqrtf(b.pf + k.pf);
            ok = !(v32 < lo32) && (v32 > hi32 || above_cut(SRTERM * b.E * k.E * rsqrt(b.p + k.p), PRIM_CUT));
        }
        for (unsigned m = __ballot_sync(0xffffffffu, ok); m; m &= m - 1) {
            const int t = t0 + __ffs(m) - 1, ib = t / nk, ik = t - ib * nk;
            const PrimPair bp = pb[ib * sb], kp = pk[ik * sk];
            ++npass;
            const double rs = rsqrt(bp.p + kp.p), rpq = rs * rs;
            double PQ[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) PQ[k] = bp.P[k] - kp.P[k];
            const double T = bp.p * kp.p * rpq * fma(PQ[0], PQ[0], fma(PQ[1], PQ[1], PQ[2] * PQ[2]));
            __syncwarp();  // the previous primitive quartet's tables have been read
            if (lane < q.nr) {
                double x, wt;
                coop_root(q.nr, lane, T, rys, compat, x, wt);
                xw[lane] = x;
                xw[q.nr + lane] = wt * (bp.Ecc * kp.Ecc * rs);
            }
            __syncwarp();
            if (lane < 3 * q.nr) {  // lane = root and axis: the 2D recurrence (Rys.hpp:85-150)
                const int r = lane / 3, ax = lane - 3 * r;
                const double fff = xw[r] * rpq, qf = kp.p * fff, pf = bp.p * fff;
                const double B00 = fff * 0.5;
                const double B1 = 0.5 * (1.0 - qf) * bp.rp, B1p = 0.5 * (1.0 - pf) * kp.rp;
                const double pq = ax == 0 ? PQ[0] : ax == 1 ? PQ[1] : PQ[2];
                const double pa = ax == 0 ? bp.PA[0] : ax == 1 ? bp.PA[1] : bp.PA[2], qc = ax == 0 ? kp.PA[0] : ax == 1 ? kp.PA[1] : kp.PA[2];
                const double C = pa - qf * pq, Cp = fma(pf, pq, qc);
                double* G = Gt + lane * gst;
                const int w1 = q.l34 + 1;
                double g0 = ax == 2 ? xw[q.nr + r] : 1.0, gm = 0.0;
                G[0] = g0;
                for (int i = 0; i < q.l12; ++i) {  // G(i + 1, 0)
                    double v = C * g0;
                    if (i > 0) v = fma(B1 * double(i), gm, v);
                    G[(i + 1) * w1] = v;
                    gm = g0;
                    g0 = v;
                }
                for (int j = 0; j < q.l34; ++j) {
                    double left = 0.0;
                    for (int i = 0; i <= q.l12; ++i) {
                        const double g = G[i * w1 + j];
                        double v = Cp * g;
                        if (j > 0) v = fma(B1p * double(j), G[i * w1 + j - 1], v);
                        if (i > 0) v = fma(B00 * double(i), left, v);
                        G[i * w1 + j + 1] = v;
                        left = g;
                    }
                }
            }
            __syncwarp();
            const int w1 = q.l34 + 1;
            const double* src = Gt;
            int sst = gst;
            if (lb > 0) {  // bra transfer: sum_k binom(b, k) AB^(b - k) G(a + k, j)
                const int n = 3 * q.nr * q.nhb;
                for (int e = lane; e < n; e += 32) {
                    const int ra = e / q.nhb, i = e - ra * q.nhb, j = i % w1, ab = i / w1, b = ab % (lb + 1), a = ab / (lb + 1);
                    const double* c = cab + (ra % 3) * 15 + b * (b + 1) / 2;
                    const double* g = Gt + ra * gst + a * w1 + j;
                    double v = g[b * w1];
                    for (int k = 0; k < b; ++k) v = fma(c[k], g[k * w1], v);
                    Ht[e] = v;
                }
                __syncwarp();
                src = Ht;
                sst = q.nhb;
            }
            if (ld > 0) {  // ket transfer, Ht to It
                const int n = 3 * q.nr * q.ni;
                for (int e = lane; e < n; e += 32) {
                    const int ra = e / q.ni, i = e - ra * q.ni;
                    const unsigned u = tidx[i];
                    const int d = u & 0xff, c = u >> 8 & 0xff, ab = u >> 16;
                    const double* cc = ccd + (ra % 3) * 15 + d * (d + 1) / 2;
                    const double* g = src + ra * sst + ab * w1 + c;
                    double v = g[d];
                    for (int k = 0; k < d; ++k) v = fma(cc[k], g[k], v);
                    It[ra * ist + i] = v;
                }
                __syncwarp();
                src = It;
                sst = ist;
            }
            // products over the axes, summed over the roots (Rys.hpp:152-170)
#pragma unroll
            for (int k = 0; k < KF; ++k) {
                const int f = lane + 32 * k;
                if (f < q.nf) {
                    const unsigned u = fidx[f];
                    const double *X = src + (u & 0xff), *Y = src + sst + (u >> 8 & 0xff), *Z = src + 2 * sst + (u >> 16);
                    for (int r = 0; r < q.nr; ++r) {
                        const int o = 3 * sst * r;
                        acc[k] = fma(X[o] * Y[o], Z[o], acc[k]);
                    }
                }
            }
        }
    }
    __syncwarp();
    // the integrals, normalised, cut and with the degeneracy factor, to shared memory for the contraction
    const int ndeg = (bra.same() ? 1 : 0) + (ket.same() ? 1 : 0) + (bi == ki ? 1 : 0);
    double* V = base;
#pragma unroll
    for (int k = 0; k < KF; ++k) {
        const int f = lane + 32 * k;
        if (f < q.nf) {
            const int ab = f / q.ncd, cd = f - ab * q.ncd;
            double v = acc[k] * (nab[ab] * ncd[cd]);
            V[ab * q.vs + cd] = above_cut(v, A.thr_int) ? scale_pow2(v, -ndeg) : 0.0;
        }
    }
    digest_shared(A, bra, ket, V, q.na, q.nb, q.nc, q.nd, q.vs);
    if (A.counters && lane == 0) count_flush(A, npass);
}

}  // namespace ugb
