// Launch table of the class-templated Fock kernels.  Pair class c = la(la+1)/2 + lb (la >= lb);
// quartet classes are (bra class >= ket class).  One translation unit per kind of kernel instantiates all of
// them.
#pragma once
#include <vector>

#include "eri_common.cuh"

namespace ugb {

struct NormTable;

__host__ __device__ constexpr int pc_la(int c) { return (c >= 1) + (c >= 3) + (c >= 6) + (c >= 10); }
__host__ __device__ constexpr int pc_lb(int c) { return c - pc_la(c) * (pc_la(c) + 1) / 2; }

// The FP32 Fock kernel of quartet class (bc | kc) over `A.nwork` work items on `stream`.
cudaError_t launch_fock_fp32(int bc, int kc, bool uhf, const FockArgs& A, const NormTable& nt,
                             const float* rys, cudaStream_t stream);
// Whether a class has the templated kernels of the split builds (s, p and d shells, at most 81 function
// quartets).
bool fock_split_class(int bc, int kc);
// The FP64 part of a mixed build of one class alone (fock_split_class), on a grid of
// at most `grid` CTAs whose warps step over the part's quartets (NP lanes per quartet).
cudaError_t launch_fock_fp64_part(int bc, int kc, bool uhf, const FockArgs& A64, const FockArgs& A32, const NormTable& nt,
                                  const double* rys64, const float* rys32, int grid, cudaStream_t stream);
// That part's quartets in pairs of floats as a kernel of their own.
cudaError_t launch_fock_df64_part(int bc, int kc, bool uhf, const FockArgs& A, const NormTable& nt, int grid,
                                  cudaStream_t stream);
// The whole FP64 part of one class of a mixed build on stream s: classes of up to 32 quartets per SM with a warp per
// quartet (plus four lanes for those that run in FP32), the others as the two kernels above.
cudaError_t launch_mixed_fp64(int bc, int kc, bool uhf, FockArgs A, const FockArgs& A32, const NormTable& nt,
                              const double* rys64, const float* rys32, int nsm, int ctas64, int ctasdf, bool demotes,
                              cudaStream_t s, int* launches);
cudaError_t launch_schwarz(int pc, const ShellPair* pairs, const PrimPair* prims, int begin, int count,
                           const NormTable& nt, const double* rys, double* q_out, cudaStream_t stream);

// The quartets below SPLIT_CUT of one class in pairs of floats (fock_df64.cuh), `items` of its split list.
cudaError_t launch_fock_df64(int bc, int kc, bool uhf, const FockArgs& A, long long items, const NormTable& nt,
                             cudaStream_t stream);
// The same over a fixed grid pulling tiles of `block` quartets (RHF; batches of molecules).
cudaError_t launch_fock_df64_persistent(int bc, int kc, const FockArgs& A, const NormTable& nt, int grid, int block,
                                        cudaStream_t stream);
// `items` of a split list, in FP64 or in pairs of floats, with `lanes` (4 or 32) lanes per quartet.
cudaError_t launch_fock_group(int bc, int kc, bool uhf, const FockArgs& A, long long items, bool pairs_of_floats, int lanes,
                              const NormTable& nt, const double* rys, cudaStream_t stream);
// All for the classes that fock_split_class accepts.  The root tables of the first:
std::vector<float> df_rys_tables();

// The Rys classes that fock_split_class does not accept (la+lb+lc+ld <= 8), one warp per quartet (fock_coop.cuh):
// over A's work list in FP64.  RHF or UHF by A.Pb.
cudaError_t launch_fock_coop(int la, int lb, int lc, int ld, const FockArgs& A, const NormTable& nt, const double* rys,
                             cudaStream_t stream);
// Runtime-L Rys kernel of the same classes' FP32 part, one lane per quartet.
cudaError_t launch_fock_generic32(int la, int lb, int lc, int ld, bool uhf, const FockArgs& A, const NormTable& nt,
                                  const float* rys32, cudaStream_t stream);
// McMurchie-Davidson kernel (la+lb+lc+ld > 8, or every class in the MD mode), FP64.
cudaError_t launch_fock_md(int la, int lb, int lc, int ld, bool uhf, const FockArgs& A, const NormTable& nt,
                           cudaStream_t stream);
// Schwarz diagonal for pairs with la+lb > 2: Rys (la+lb <= 4) into q_out, MD (la+lb > 4) via qbits.
cudaError_t launch_schwarz_high(int la, int lb, const ShellPair* pairs, const PrimPair* prims, int begin, int count,
                                const NormTable& nt, const double* rys, double* q_out, unsigned long long* qbits,
                                cudaStream_t stream);

constexpr int FOCK_THREADS = 128;

}  // namespace ugb
