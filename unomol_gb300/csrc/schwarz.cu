// The Schwarz diagonal of the s, p and d pair classes.
#include "fock_kernels.cuh"
#include "fock_dispatch.cuh"

namespace ugb {

template <int PC>
static cudaError_t schwarz_one(const ShellPair* pairs, const PrimPair* prims, int begin, int count,
                               const NormTable& nt, const double* rys, double* q, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    constexpr int NAB = ncart(pc_la(PC)) * ncart(pc_lb(PC));
    if constexpr (NAB * NAB <= 81)
        schwarz_kernel<pc_la(PC), pc_lb(PC)><<<(unsigned)(((long long)count * 32 + 127) / 128), 128, 0, s>>>(pairs, prims, begin, count, nt, rys, q);
    else
        schwarz_generic<<<(count + 63) / 64, 64, 0, s>>>(pairs, prims, begin, count, nt, rys, q);
    return cudaGetLastError();
}

cudaError_t launch_schwarz(int pc, const ShellPair* pairs, const PrimPair* prims, int begin, int count,
                           const NormTable& nt, const double* rys, double* q_out, cudaStream_t stream) {
    switch (pc) {
        case 0: return schwarz_one<0>(pairs, prims, begin, count, nt, rys, q_out, stream);
        case 1: return schwarz_one<1>(pairs, prims, begin, count, nt, rys, q_out, stream);
        case 2: return schwarz_one<2>(pairs, prims, begin, count, nt, rys, q_out, stream);
#if UGB_MAX_PAIRCLASS > 3
        case 3: return schwarz_one<3>(pairs, prims, begin, count, nt, rys, q_out, stream);
        case 4: return schwarz_one<4>(pairs, prims, begin, count, nt, rys, q_out, stream);
        case 5: return schwarz_one<5>(pairs, prims, begin, count, nt, rys, q_out, stream);
#endif
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ugb
