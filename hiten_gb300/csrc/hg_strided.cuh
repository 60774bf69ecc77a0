// Index arithmetic of launches over up to 2^31 - 1 items.  The step that takes
// an index past its count, and a count rounded up to whole blocks, leave 32 bits
// at the upper end, so both are formed in 64.  Compiles as device code and as
// host C++, so that the ends can be tested on the CPU.
#pragma once

#if defined(__CUDACC__)
#define HG_SHD __host__ __device__ __forceinline__
#else
#define HG_SHD inline
#endif

// `for (int i : Strided{first, step, n})`: first, first + step, ... below n.
struct Strided {
  struct At {
    long long i, step;
    HG_SHD int operator*() const { return (int)i; }
    HG_SHD void operator++() { i += step; }
    HG_SHD bool operator!=(const At& end) const { return i < end.i; }
  };
  long long first, step, n;
  HG_SHD At begin() const { return At{first, step}; }
  HG_SHD At end() const { return At{n, step}; }
};

// Blocks of `block` threads for one thread an item.
HG_SHD unsigned blocks_of(long long n, int block) { return (unsigned)((n + block - 1) / block); }

#if defined(__CUDACC__)
__device__ __forceinline__ long long global_thread() { return (long long)blockIdx.x * blockDim.x + threadIdx.x; }
// This thread's items of n: all threads of the grid together take each once.
__device__ __forceinline__ Strided grid_strided(long long n) {
  return Strided{global_thread(), (long long)gridDim.x * blockDim.x, n};
}
#endif
