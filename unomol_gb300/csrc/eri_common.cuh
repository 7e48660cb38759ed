// Shared device/host definitions of the direct Fock build: data layout of shell pairs and primitive
// pairs in HBM, Cartesian component tables, and the Rys root/weight evaluation.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "df64.cuh"

namespace ugb {

constexpr int LMAX = 4;                 // largest shell angular momentum (g; Basis.hpp:222)
constexpr int LTMPL = 2;                // shells up to d have class-templated Rys kernels
constexpr int NPAIRCLASS = (LMAX + 1) * (LMAX + 2) / 2;  // (la >= lb) pair classes
constexpr int NTMPLCLASS = (LTMPL + 1) * (LTMPL + 2) / 2;
constexpr double SRTERM = 34.9868366552497250;  // 2 pi^{5/2} (TwoElectronInts.cpp:427)
constexpr double PRIM_CUT = 1.e-12;     // primitive prefactor cut (TwoElectronInts.cpp:428,478-479)
constexpr double STORE_CUT = 1.e-14;    // integral storage cut (TwoElectronInts.cpp:517,668)

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int pair_class(int la, int lb) { return la * (la + 1) / 2 + lb; }

// Cartesian exponents of component c of a shell with angular momentum l, in the reference's order:
// lx descending, then ly descending (AuxFunctions.hpp:35-43).
// Closed form (components with lx = l - i form the i-th block of i+1 entries, ly descending), so
// that unrolled kernels fold it to constants without evaluating loops.
__host__ __device__ constexpr int cart_blk(int c) { return (c >= 1) + (c >= 3) + (c >= 6) + (c >= 10); }
__host__ __device__ constexpr int cart_lx(int l, int c) { return l - cart_blk(c); }
__host__ __device__ constexpr int cart_ly(int l, int c) {
    return cart_blk(c) - (c - cart_blk(c) * (cart_blk(c) + 1) / 2);
}
__host__ __device__ constexpr int cart_lz(int l, int c) { return l - cart_lx(l, c) - cart_ly(l, c); }

// One primitive pair of a shell pair (a has the larger L after the swap of
// TwoElectronInts.cpp:563-579); the kernels read it through the read-only path.  The records of a shell
// pair are in descending E (k_interleave_prims), so that a loop over them ends at the first one whose
// prefactor can no longer pass the screen (plain FP64 build of 32 waters 21.8 -> 21.4 ms).
struct __align__(16) PrimPair {
    double p;          // alpha_a + alpha_b
    double rp;         // 1 / p
    double P[3];       // Gaussian product centre
    double PA[3];      // P - A
    double E;          // exp(-alpha_a alpha_b |AB|^2 / p) / p, coefficient free (prefactor screen)
    double cc;         // c_a c_b, times 2 for the i != j half of a same-shell pair
                       // (TwoElectronInts.cpp:444-449)
    double Ecc;        // sqrt(2 pi^{5/2}) E cc: a primitive quartet's prefactor is Ecc_ab Ecc_cd / sqrt(p + q)
    float pf, Ef;      // p and E in FP32, for a cheap pre-screen (96 bytes: six 16-byte loads)
};

struct __align__(16) PrimPair32 {
    float p, rp, P[3], PA[3], E, cc;
    float Ecc;      // sqrt(2 pi^{5/2}) E cc, as PrimPair::Ecc
    float pad_;     // 48 bytes: three 16-byte loads
};

// The record in pairs of floats (48 bits, df64.cuh), for the quartets below SPLIT_CUT.  It holds no product
// centre: P - Q is A - C + (P - A) - (Q - C), whose rounding follows the distances inside the quartet and not
// the molecule's extent.
struct __align__(16) PrimPairDF {
    df p, E;        // first 16-byte load: the prefactor screen
    df Ecc, rp;
    df PA[3];       // 64 bytes: four 16-byte loads
};

// Centre A of a shell pair as sums of three floats, per axis h + m + l: h a multiple of the molecule's centre
// step, m of 2^-24 of it, so that differences of the first two are exact (setup.cu: centre_step).
struct __align__(16) PairCentre {
    float4 x, y, z;  // .w unused
};

// Schwarz bound from which a quartet of the FP64 build is evaluated in FP64; below it, in pairs of floats
// (fock_df64.cuh), whose integrals are off by about 2^-50 of the bound (rms; s and p shells).  Chosen as the largest
// for which the error of G stays what the all-FP64 build had with one accumulator per element.  Error of G against the
// oracle in long double (rms, 1e-15; that build / a cut of 1/16 / of 1/8), densities of the core Hamiltonian: 6-31G
// ethane 1.00 / 1.23 / 2.76, n-butane 2.38 / 2.14 / 4.64, five waters 2.31 / 1.89 / 2.50; STO-3G n-heptane
// 3.09 / 2.90 / 5.44.  Time, 32 waters / n-decane UHF: 1/32 25.4 / 3.7 ms, 1/16 25.1 / 3.1, 1/8 23.9 / 2.7.
// Builds with an FP32 part, whose error the caller sets, split their FP64 part at MIXED_SPLIT_CUT (32 waters, full
// density: 9.45 ms at 1/16, 8.84 at 1/8).
constexpr double SPLIT_CUT = 0.0625;
constexpr double MIXED_SPLIT_CUT = 0.125;

constexpr double SQRT_SRTERM = 5.914967172795613;  // sqrt(2 pi^{5/2})
static_assert(SQRT_SRTERM * SQRT_SRTERM - SRTERM < 1e-13 && SRTERM - SQRT_SRTERM * SQRT_SRTERM < 1e-13, "sqrt of SRTERM");

// One shell pair, sorted into blocks of equal (class, primitive-pair count), within a block by
// descending Schwarz bound.
struct __align__(8) ShellPair {
    // the first and the third 32-byte sector are what the FP32 kernels read, in 8-byte loads (the fields one
    // by one cost those kernels 2 %)
    int a_off, b_off;      // first AO of shell a (larger L) and of shell b
    int prim_begin, nprim; // primitive pair ik of this pair at prim_begin + ik * prim_stride
    int prim_stride;       // pairs of one block (equal nprim) interleave their primitive pairs: the
                           // stride is the block's pair count, so consecutive pairs' records are adjacent
    int flags;             // bit 0: ish == jsh; la << 8, lb << 16 (la >= lb)
    int pad;               // the molecule of a batch
    float ABl0;            // ABl0..2: what A - B leaves over its FP32 copy, for the pairs-of-floats kernels
    double AB[3];          // A - B
    double q;              // Schwarz bound: max over functions of sqrt|(ab|ab)|
    int ish, jsh;          // shell indices (ish >= jsh)
    float ABl1, ABl2;
    float ABf[3];          // A - B and q in FP32, for the FP32 kernels (no FP64 work or conversion there)
    float qf;
    __host__ __device__ bool same() const { return flags & 1; }
    __host__ __device__ int la() const { return (flags >> 8) & 0xff; }
    __host__ __device__ int lb() const { return (flags >> 16) & 0xff; }
};

static_assert(sizeof(ShellPair) == 96, "three 32-byte sectors a pair");

// A rectangle (or triangle, when bra block == ket block) of quartets between two pair blocks,
// trimmed by the Schwarz staircase: bra pair i pairs with the first cnt[i] ket pairs of its block.
struct BlockPair {
    int bra_begin, bra_count;   // pair index range of the bra block
    int ket_begin, ket_count;   // pair index range of the ket block
    int triangle;               // bra block == ket block: ket index <= bra index
    int prefix_off;             // offset of this block pair's prefix array (bra_count + 1 entries)
    int prim_quartets;          // primitive quartets of each of its shell quartets (nprim bra x nprim ket)
    long long work_begin;       // first work item (multiple of 32, so warps never straddle)
    long long work_count;       // quartets in this block pair
};

// Copies of the J/K accumulators that the CTAs share out; the fold adds them.  Why: each diagonal element of T takes one
// addition per surviving ket pair (10^5 for 32 waters), each rounded at the running sum, and that, not the integrals, is
// most of the error of G.  With c copies a copy takes 1/c of the additions at 1/c of the sum, and the errors add up to
// 1/sqrt(c).  Against the oracle in long double (rms over G, 1e-15): 16 waters 8.2 with one copy, 3.8 with four, 3.4 with
// eight (5.0 for one copy with the light classes first, when the large integrals come last); 32 waters 23.6, 7.6, 5.5
// (10.4).  Fewer CTAs meet on an address, too: 32 waters 26.4 -> 23.9 ms.  Up to 1 GiB for all copies, then fewer.
constexpr int ACC_COPIES = 8;
inline int acc_copies(long long elements, long long room = 1ll << 27) {
    int c = ACC_COPIES;
    while (c > 1 && c * elements > room) c /= 2;
    return c;
}

// Kernel arguments shared by every class instance.
struct FockArgs {
    const ShellPair* pairs;
    const PrimPair* prims;
    const PrimPair32* prims32;
    const PrimPairDF* primsdf;
    const PairCentre* pcen;
    const float* rysdf;         // root tables of the pairs-of-floats kernels
    const BlockPair* bps;
    const long long* prefix;    // concatenated staircase prefix sums
    int nbp;                    // block pairs of this launch
    long long nwork;            // work items of this launch (padded)
    int nbf;
    const double* Pa;           // full N x N density (RHF: P; UHF: Pa)
    const double* Pb;           // UHF: Pb; RHF: nullptr
    const float* Pa32;          // FP32 copies of Pa / Pb for the FP32 kernels' density contraction
    const float* Pb32;
    const float* pmax;          // shell-pair max |P| (nshell x nshell), for density screening
    double* Ta;                 // N x N accumulators; G = T + T^T
    double* Tb;                 // UHF beta accumulator
    int tmask;                  // copies of the accumulators less one (acc_copies), tstride elements apart, taken
    long long tstride;          // by the CTAs in turn
    double thr_int;             // per-integral cut (1e-14)
    double prim_cut;            // primitive prefactor cut (1e-12)
    float thr_int32, prim_cut32, skip_cut32;  // the same cuts in FP32, for the FP32 kernels
    float split_cut32;          // FP64 part of a screened build: quartets with a Schwarz bound below this in pairs of floats
    int only_demoted;           // FP64 part of a mixed build: only its FP32 quartets (the others have a launch of their own)
    long long df_group_max;     // and up to this many quartets in the part it also takes the pairs-of-floats ones
    float fp32_cut32;           // mixed mode: a quartet with bound * max|P| of its blocks below this runs in FP32
    double fp32_cut;            // mixed mode: bound * max|P| below this -> FP32 part, else FP64 part
    int mode;                   // 0 all quartets; 1 only "large" (FP64 part); 2 only "small" (FP32 part);
                                // 3 / 4 the parts above / below SPLIT_CUT of an FP64 build
    int nshell;
    int rys_compat;             // reference-compatible two-root Rys regime (FP64 only)
    unsigned long long* counters;  // optional: primitive quartets past the prefactor cut, 32 slots per launch
    int counter_base;           // first slot of this launch (class id * 32)
    // density-screened / mixed-precision builds (mode 1 = FP64 part, mode 2 = FP32 part): per-build
    // work lists made on the device (split_rows + scan_rows)
    const long long* dyn_prefix;  // per bra row, exclusive prefix of this part's quartets (prefix layout)
    const long long* dyn_count;   // per block pair of this launch: quartets of this part
    const long long* dyn_begin;   // per block pair of this launch: its first item in this part's compact
                                  // numbering (counts rounded up to 32 and summed over the launch)
    const long long* dyn_total;   // [0]: items of this part in the launch (the compact numbering's end)
    const int* dyn_mseg;          // per bra row: length of its FP64 segment (the FP32 segment follows it)
    const float* dmax;            // [0]: max |P| over all shell-pair blocks
    double skip_cut;              // quartets with bound * max|P| below this are skipped
    // batches of molecules: ShellPair::pad holds the molecule; its dense P / T start at mol_base and
    // have mol_nbf rows (nullptr: one molecule, A.nbf rows at offset 0)
    const int* mol_nbf;
    const long long* mol_base;
    const int* mol_nshell;        // batches in the screened build: shells of the molecule and the first
    const long long* mol_pmax;    // entry of its shell-pair max|P| blocks in pmax
    unsigned long long* tile_counter;  // persistent launches: next tile of this launch
    int* status;                // device error flag
};

}  // namespace ugb
