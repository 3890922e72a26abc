// Index arithmetic that kernels and host code share, free of CUDA types, so
// that a host compiler checks it at the ends of its ranges.
#ifndef SLBC_INDEX_CUH
#define SLBC_INDEX_CUH

#ifdef __CUDACC__
#define SLBC_HD __host__ __device__ __forceinline__
#else
#define SLBC_HD inline
#endif

namespace slbc {

// f(e) for e = first, first + step, ... below count, in 32 bits: a lattice has
// fewer than 2^31 nodes and a grid fewer than 2^31 threads, so the last e +
// step stays below 2^32 and does not wrap (in int it would, to a negative
// element, for counts within one step of 2^31).
template <typename F>
SLBC_HD void grid_turns(unsigned first, unsigned step, unsigned count, F f) {
  for (unsigned e = first; e < count; e += step) f(e);
}

}  // namespace slbc

#endif
