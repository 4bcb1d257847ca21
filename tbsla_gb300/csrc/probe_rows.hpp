// The row of an element of a probe block (n x P row-major).
#pragma once

#ifdef __CUDACC__
#define TBSLA_HD __host__ __device__ __forceinline__
#else
#define TBSLA_HD inline
#endif

namespace tbsla_gpu {

// t / P by a 32-bit division (a fifth of the instructions of a 64-bit one);
// WIDE, for blocks with an element whose index it cannot hold: a 64-bit one.
inline bool probe_rows_wide(long len) { return len - 1 > 0xffffffffL; }
template <bool WIDE>
TBSLA_HD long probe_row(long t, int P) {
  return WIDE ? t / P : (long)((unsigned)t / (unsigned)P);
}

}  // namespace tbsla_gpu
