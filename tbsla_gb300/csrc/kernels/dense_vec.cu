// DENSE GEMV and the small vector / preparation kernels of the path.
//
// dense_gemv and dense_gemv_df replace tbsla::cpp::MatrixDENSE::Ax
// (src/cpp/matrix/MatrixDENSE.cpp:77-86): r_i += sum_j A_ij v_j on a
// row-major ln_row x ln_col matrix.  FP64 values: a CTA per row for rows of
// at least 2048 columns, a warp per row below; 16-byte loads (pairs of
// doubles) where the row start is 16-byte aligned, x through L1 (every row
// reuses it), one FP64 multiply-add per entry (GB300's FP64 pipe, not HBM,
// bounds an FP64 GEMV), partial sums combined in a fixed order and added to
// r_i.  Values of every precision whose magnitudes lie in [2^-40, 2^40]
// (checked once at upload): double-float arithmetic on the FP32 pipes
// (dense_gemv_df, below); an FP64 value is split on load, on the integer
// pipe, into two floats that hold it to 2^-48.
#include <algorithm>

#include "common.cuh"
#include "df.cuh"
#include "kernels.hpp"

namespace tbsla_gpu {

namespace {

constexpr int NT = 256;
constexpr int kDenseU = 4;  // 16-byte loads in flight per thread, CTA-per-row kernel
__device__ __forceinline__ double2 ld_stream2(const double* p, uint64_t pol) {
  double2 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
               : "=d"(v.x), "=d"(v.y) : "l"(p), "l"(pol));
  return v;
}

template <class V>
__global__ void __launch_bounds__(NT) k_dense(const V* __restrict__ A, int ln_row, int ln_col,
                                             const double* __restrict__ x, double* __restrict__ y) {
  const int lane = threadIdx.x % kWarp;
  const int gw = (blockIdx.x * NT + threadIdx.x) / kWarp;
  const int nw = gridDim.x * NT / kWarp;
  const uint64_t pol = policy_evict_first();
  for (int row = gw; row < ln_row; row += nw) {
    const V* a = A + (size_t)row * ln_col;
    double acc = 0;
    int j = lane;
    for (; j + 3 * kWarp < ln_col; j += 4 * kWarp) {
      double v0 = widen(ld_stream(a + j, pol)), v1 = widen(ld_stream(a + j + kWarp, pol));
      double v2 = widen(ld_stream(a + j + 2 * kWarp, pol)), v3 = widen(ld_stream(a + j + 3 * kWarp, pol));
      acc = fma_rn(v0, __ldg(x + j), acc);
      acc = fma_rn(v1, __ldg(x + j + kWarp), acc);
      acc = fma_rn(v2, __ldg(x + j + 2 * kWarp), acc);
      acc = fma_rn(v3, __ldg(x + j + 3 * kWarp), acc);
    }
    for (; j < ln_col; j += kWarp) acc = fma_rn(widen(ld_stream(a + j, pol)), __ldg(x + j), acc);
    acc = warp_sum(acc);
    if (lane == 0) y[row] = add_rn(y[row], acc);
  }
}

// FP64 rows of at least 2*NT*U columns with 16-byte aligned starts: one CTA
// per row (launched with a CTA per row; the loop also accepts fewer CTAs),
// every thread with U 16-byte loads in flight.
// A warp per row leaves the last round of rows to a fraction of the warps
// (32768 rows over 9728 warps: 4 rounds for some, 3 for the rest); a CTA per
// row spreads each row over the whole CTA and the rows over 8x fewer
// workers, so the last round is a small share of the launch.  Partial sums:
// warp butterfly, then the NT/32 warp sums in a fixed order (a double-
// buffered slot per row parity, one barrier per row).
template <int U>
__global__ void __launch_bounds__(NT) k_dense_rows_f64x2(const double* __restrict__ A, int ln_row,
                                                        int ln_col, const double* __restrict__ x,
                                                        double* __restrict__ y) {
  __shared__ double s_part[2][NT / kWarp];
  const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
  const uint64_t pol = policy_evict_first();
  const int half = ln_col / 2;
  const double2* x2 = reinterpret_cast<const double2*>(x);
  int parity = 0;
  for (int row = blockIdx.x; row < ln_row; row += gridDim.x, parity ^= 1) {
    const double* a = A + (size_t)row * ln_col;
    double acc0 = 0, acc1 = 0;
    int j = threadIdx.x;
    for (; j + (U - 1) * NT < half; j += U * NT) {
      double2 av[U], bv[U];
#pragma unroll
      for (int u = 0; u < U; u++) av[u] = ld_stream2(a + 2 * (j + u * NT), pol);
#pragma unroll
      for (int u = 0; u < U; u++) bv[u] = __ldg(x2 + j + u * NT);
#pragma unroll
      for (int u = 0; u < U; u++) {
        acc0 = fma_rn(av[u].x, bv[u].x, acc0);
        acc1 = fma_rn(av[u].y, bv[u].y, acc1);
      }
    }
    for (; j < half; j += NT) {
      const double2 a0 = ld_stream2(a + 2 * j, pol);
      const double2 b0 = __ldg(x2 + j);
      acc0 = fma_rn(a0.x, b0.x, acc0);
      acc1 = fma_rn(a0.y, b0.y, acc1);
    }
    const double w = warp_sum(add_rn(acc0, acc1));
    if (lane == 0) s_part[parity][warp] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
#pragma unroll
      for (int i = 0; i < NT / kWarp; i++) t = add_rn(t, s_part[parity][i]);
      y[row] = add_rn(y[row], t);
    }
  }
}

// Values in double-float arithmetic.  Widening every value to FP64 for one
// FP64 multiply-add kept the FP64 pipe as busy as the FP64 matrix does (0.99 ms
// for 537 M entries) although the bytes halve.  Here:
//  * x is split once per call into floats xh = fl32(x), xl = fl32(x - xh),
//    which hold x to 2^-48 relative, kept as two arrays;
//  * a warp takes R rows and a part of the columns, 128 (BF16: 256) columns a
//    step: each lane loads 16 bytes of every row (FP64: 32, in one go where the
//    rows are aligned for it) and their xh / xl, which serve all R rows, and
//    adds them with compensated Dot2 steps (the product's and the sum's
//    rounding errors carried exactly into a second float);
//  * the lanes' pairs are summed across the warp in FP64, the R rows at once
//    (each half of the warp goes on with half of the rows), and so are the
//    column parts, in a fixed order.
// Bound: HBM for FP64 and FP32 values (16384 x 8192: 160 and 89 us, 6.7 and
// 6.0 TB/s with the launches), instruction issue (about 15 per entry, 16 to 18
// on short rows, see Sums) for BF16 (24576 x 8192: 103 us).  With a CTA per row,
// one row's x loads, its warp reductions and a barrier came to more
// instructions than the entries themselves: 178, 122 and 164 us, and 65 us for
// 9000 x 600 FP32, now 8.3.
// The float arithmetic is exact only inside the float exponent range, so the
// path needs every nonzero |x| and |a| in [2^-40, 2^40] (products within
// [2^-80, 2^80], sums of up to 2^31 of them finite, error terms normal): the
// values are checked once at upload, x by the split kernel on every call,
// whose CTAs leave a flag each; a launch that reads a set flag runs every row
// in FP64 instead, in the same kernel (no host round trip).  Bound there: the
// FP64 pipe, and HBM for FP64 values.
constexpr float kDfLo = 9.094947017729282e-13f;  // 2^-40
constexpr float kDfHi = 1.099511627776e12f;      // 2^40

__device__ __forceinline__ bool df_in_range(double v) {
  const double a = fabs(v);
  return a == 0.0 || (a >= (double)kDfLo && a <= (double)kDfHi);  // false for NaN
}

// xs[0, n) = xh, xs[n, 2n) = xl: separate arrays, so that the GEMV's lanes
// read consecutive words of each.  bad[CTA]: x leaves the range there.
__global__ void __launch_bounds__(NT) k_df_split_x(const double* x, int n, float* xs, int* bad) {
  wait_for_earlier();
  int any = 0;
  for (int i = blockIdx.x * NT + threadIdx.x; i < n; i += gridDim.x * NT) {
    const double v = x[i];
    const float h = __double2float_rn(v);
    xs[i] = h;
    xs[n + i] = __double2float_rn(v - (double)h);
    any |= !df_in_range(v);
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) bad[blockIdx.x] = any;
}

template <class V>
__global__ void k_df_range_vals(const V* __restrict__ a, size_t n, int* __restrict__ bad) {
  int any = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    any |= !df_in_range(widen(a[i]));
  if (__any_sync(0xffffffffu, any) && threadIdx.x % kWarp == 0) atomicOr(bad, 1);
}

// An FP64 value a = h + l split into two floats on the integer pipe: h is a
// rounded to 24 significand bits (half away from zero; a carry moves into the
// exponent by itself), l the float nearest to the rest a - h (at most 2^28 in
// units of a's last bit, so a is held to 2^-49 relative).  For a == 0 or |a| in
// [2^-60, 2^60]; the values reaching it passed the [2^-40, 2^40] check.  No
// FP64 instruction.
__device__ __forceinline__ void split_f64(double a, float& h, float& l) {
  const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
  // the low 8 bits of the exponent and the leading 23 of the mantissa; a
  // float's exponent is e - 896, whose low 8 bits are e's with the top one
  // flipped
  const unsigned top = __funnelshift_l(lo, hi, 3) ^ 0x40000000u;
  const unsigned t = (hi & 0x80000000u) | (top & 0x7fffffffu);
  h = (hi & 0x7ff00000u) == 0u ? 0.f : __uint_as_float(t + (lo >> 28 & 1u));
  // the last 29 bits as a signed number (0 for a == 0), times +- 2^(e - 1075)
  const float scale = __uint_as_float((t & 0xff800000u) - (52u << 23));
  l = __fmul_rn(__int2float_rn((int)(lo << 3) >> 3), scale);
}

// One term a (xh + xl) of a Dot2 sum: the rounding errors of product and sum are
// carried into c with the small products, all of the term's before they meet c,
// which then is rounded once a term (dot2_step: twice).  L: l * xh too.
template <bool L = false>
__device__ __forceinline__ void dense_step(float& s, float& c, float a, float xh, float xl, float l = 0.f) {
  const float pr = __fmul_rn(a, xh);
  float e = __fmaf_rn(a, xl, __fmaf_rn(a, xh, -pr));
  if constexpr (L) e = __fmaf_rn(l, xh, e);
  const DF t = two_sum(s, pr);
  s = t.h;
  c = __fadd_rn(c, __fadd_rn(e, t.l));
}

// A step is 32 * NV columns; one lane's NV values of a row's step, as loaded:
// 16 bytes (FP64: 32).  VEC: columns c .. c + NV - 1, the row aligned for it;
// else columns c, c + 32, ...  A column past the row's last one (`last`: its
// index, VEC its last vector's) is read at `last` instead and meets a zero of
// x.
template <class V, bool VEC>
struct Step;
template <bool VEC>
struct Step<double, VEC> {
  static constexpr int NV = 4;
  double v[NV];
  __device__ __forceinline__ void load(const double* p, int c, int last, uint64_t pol) {
    if constexpr (VEC) {
      p += min(c, last);
      asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
                   : "=d"(v[0]), "=d"(v[1]) : "l"(p), "l"(pol));
      asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
                   : "=d"(v[2]), "=d"(v[3]) : "l"(p + 2), "l"(pol));
    } else {
#pragma unroll
      for (int k = 0; k < NV; k++) v[k] = ld_stream(p + min(c + 32 * k, last), pol);
    }
  }
  __device__ __forceinline__ double value(int k) const { return v[k]; }
  // a = h + l: Dot2 on h (x as xh + xl), with l * xh among the small terms
  // (l * xl is below 2^-48 of the product)
  __device__ __forceinline__ void add(float& s, float& c, int k, float xh, float xl) const {
    float h, l;
    split_f64(v[k], h, l);
    dense_step<true>(s, c, h, xh, xl, l);
  }
};
template <bool VEC>
struct Step<float, VEC> {
  static constexpr int NV = 4;
  float v[NV];
  __device__ __forceinline__ void load(const float* p, int c, int last, uint64_t pol) {
    if constexpr (VEC) {
      asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                   : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p + min(c, last)), "l"(pol));
    } else {
#pragma unroll
      for (int k = 0; k < NV; k++) v[k] = ld_stream(p + min(c + 32 * k, last), pol);
    }
  }
  __device__ __forceinline__ double value(int k) const { return widen(v[k]); }
  __device__ __forceinline__ void add(float& s, float& c, int k, float xh, float xl) const {
    dense_step(s, c, v[k], xh, xl);
  }
};
template <bool VEC>
struct Step<__nv_bfloat16, VEC> {  // a bfloat16 is the high half of its float; VEC: two values a word
  static constexpr int NV = 8;
  unsigned v[VEC ? NV / 2 : NV];
  __device__ __forceinline__ void load(const __nv_bfloat16* p, int c, int last, uint64_t pol) {
    if constexpr (VEC) {
      asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                   : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p + min(c, last)), "l"(pol));
    } else {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const __nv_bfloat16 b = ld_stream(p + min(c + 32 * k, last), pol);
        v[k] = *reinterpret_cast<const unsigned short*>(&b);
      }
    }
  }
  __device__ __forceinline__ unsigned word(int k) const {
    if constexpr (!VEC) return v[k] << 16;
    return k & 1 ? v[k >> 1] & 0xffff0000u : v[k >> 1] << 16;
  }
  __device__ __forceinline__ double value(int k) const { return widen_bits(word(k)); }
  __device__ __forceinline__ void add(float& s, float& c, int k, float xh, float xl) const {
    dense_step(s, c, __uint_as_float(word(k)), xh, xl);
  }
};

// The warp's sums of R values per lane: the halves of the warp go on with half
// of the values each until one is left, which the remaining lanes add up.  Lanes
// [r * 32 / R, (r + 1) * 32 / R) get value r.  In FP64: a double-float addition
// rounds as much as some columns' terms do, and costs more.  With `brief`, the
// halves in double-float (short rows, which have the error to spare and for
// which the FP64 pipe would be the bound: 40,000 x 200 BF16 15.2 us, not 19.6).
template <int R>
__device__ __forceinline__ double warp_sum_rows(DF (&t)[R], bool brief) {
  constexpr unsigned full = 0xffffffffu;
  double sum;
  if (R > 1 && brief) {
    int o = 16;
#pragma unroll
    for (int n = R; n > 1; n /= 2, o /= 2) {
      const bool up = threadIdx.x & o;
#pragma unroll
      for (int i = 0; i < n / 2; i++) {
        const DF keep = up ? t[i + n / 2] : t[i], give = up ? t[i] : t[i + n / 2];
        t[i] = df_add(keep, DF{__shfl_xor_sync(full, give.h, o), __shfl_xor_sync(full, give.l, o)});
      }
    }
    sum = add_rn(widen(t[0].h), widen(t[0].l));
  } else {
    double d[R];
#pragma unroll
    for (int r = 0; r < R; r++) d[r] = add_rn(widen(t[r].h), widen(t[r].l));
    int o = 16;
#pragma unroll
    for (int n = R; n > 1; n /= 2, o /= 2) {
      const bool up = threadIdx.x & o;
#pragma unroll
      for (int i = 0; i < n / 2; i++) {
        const double keep = up ? d[i + n / 2] : d[i], give = up ? d[i] : d[i + n / 2];
        d[i] = add_rn(keep, __shfl_xor_sync(full, give, o));
      }
    }
    sum = d[0];
  }
#pragma unroll
  for (int o = 16 / R; o > 0; o /= 2) sum = add_rn(sum, __shfl_xor_sync(full, sum, o));
  return sum;
}

// The sum of row lane / (32 / R) of the warp's R rows from row0 on, of this
// warp's columns, into y (y += sum; fresh: y = sum).
template <int R>
__device__ __forceinline__ void store_rows(double mine, long row0, int ln_row, int log2s, double* y, int fresh,
                                           double (*s_part)[R]) {
  constexpr int NW = NT / kWarp;
  const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp, S = 1 << log2s;
  const int r = lane / (kWarp / R);
  const bool head = lane % (kWarp / R) == 0;
  if (S == 1) {
    if (head && row0 + r < ln_row) y[row0 + r] = add_rn(fresh ? 0.0 : y[row0 + r], mine);
    return;
  }
  if (head) s_part[warp][r] = mine;
  __syncthreads();
  if (threadIdx.x < (NW >> log2s) * R) {
    const int g = threadIdx.x / R, q = threadIdx.x % R;
    const long row = ((long)blockIdx.x * (NW >> log2s) + g) * R + q;
    double t = 0;
    for (int k = 0; k < S; k++) t = add_rn(t, s_part[g * S + k][q]);
    if (row < ln_row) y[row] = add_rn(fresh ? 0.0 : y[row], t);
  }
}

// The same rows and columns in FP64 (x out of the range): a row at a time, eight
// sums a lane, as short as those of 256 threads a row, so that the multiply-adds
// do not wait for one another.  A function of its own that nothing comes after,
// so that the double-float loop keeps its registers.
template <class V, int R, bool VEC>
__device__ __noinline__ void rows_f64(const V* a0, int rows, long row0, int ln_row, int ln_col, int log2s,
                                      const double* x, double* y, int fresh, double (*s_part)[R]) {
  constexpr int NV = Step<V, VEC>::NV, SC = 32 * NV;
  const int lane = threadIdx.x % kWarp, S = 1 << log2s, part = threadIdx.x / kWarp & (S - 1);
  const int nsteps = (ln_col + SC - 1) / SC;
  const int last = ln_col - (VEC ? NV : 1), c0 = VEC ? NV * lane : lane;
  const uint64_t pol = policy_evict_first();
  double mine = 0;
  for (int r = 0; r < rows; r++) {
    const V* a = a0 + (size_t)r * ln_col;
    double acc[8];
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] = 0;
    auto add = [&](const Step<V, VEC>& f, int c, int to) {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const int cc = VEC ? c + k : c + 32 * k;
        const double xv = cc < ln_col ? x[cc] : 0.0;
        acc[to + k] = fma_rn(f.value(k), xv, acc[to + k]);
      }
    };
    for (int st = part; st < nsteps; st += 2 * S) {
      Step<V, VEC> f0, f1;
      const bool two = st + S < nsteps;
      f0.load(a, st * SC + c0, last, pol);
      f1.load(a, (two ? st + S : st) * SC + c0, last, pol);
      add(f0, st * SC + c0, 0);
      if (two) add(f1, (st + S) * SC + c0, 8 - NV);
    }
#pragma unroll
    for (int o = 4; o > 0; o /= 2) {
#pragma unroll
      for (int k = 0; k < o; k++) acc[k] = add_rn(acc[k], acc[k + o]);
    }
    const double sum = warp_sum(acc[0]);
    if (lane / (kWarp / R) == r) mine = sum;
  }
  store_rows<R>(mine, row0, ln_row, log2s, y, fresh, s_part);
}

constexpr int kBriefColumns = 512;

// How a lane's Dot2 sums are kept: their error grows with the entries of one sum
// and with the folds of such sums into one pair, and a lane adds up to eight
// times the entries that a thread of a CTA per row (the kernel before this one)
// did.  Each is used where its error against 64 bits is no larger than that
// kernel's, which holds 2.7e-15 of the 2-norm at 513 columns, 3.3e-15 (FP32 and
// BF16) to 5e-15 (FP64) at 600 to 1000, twice that at 4096:
enum Sums {
  kLong,    // a step or two folded into one pair: error 3.4 to 5.2e-15 (FP32, FP64), 6.8e-15 (BF16)
  kFours,   // four entries, two or four pairs: 2.6 to 3.9e-15
  kPairs,   // two entries, four pairs: 2.2 to 3.3e-15; only for unaligned rows, which had the least error
  kEights,  // eight entries, two pairs (BF16): 4.1 to 4.4e-15
};

// y += A x (fresh: y = A x).  The CTA's eight warps are 8 / S groups of R rows
// times S = 1 << log2s parts of the columns (steps part, part + S, ...).  The
// values of two steps are loaded, then used: 32 warps on an SM (64 registers)
// keep as many loads in flight as 24 that load a step ahead (80 registers: BF16
// 117, FP32 98, FP64 193 us where 109, 101 and 185 were taken then).
template <class V, int R, bool VEC, Sums SUMS>
__global__ void __launch_bounds__(NT, 4) k_dense_df(const V* __restrict__ A, int ln_row, int ln_col, int log2s,
                                                   const float* xs, const double* x, const int* bad, int nbad,
                                                   double* y, int fresh) {
  wait_for_earlier();
  constexpr int NV = Step<V, VEC>::NV, SC = 32 * NV, NW = NT / kWarp;
  __shared__ double s_part[NW][R];
  const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
  const int S = 1 << log2s, part = warp & (S - 1);
  const long row0 = (((long)blockIdx.x * NW + warp) >> log2s) * R;
  const uint64_t pol = policy_evict_first();
  const int nsteps = (ln_col + SC - 1) / SC;
  // rows past the last one repeat it; their sums are not stored
  const V* const a0 = A + (size_t)min(row0, (long)ln_row - 1) * ln_col;
  const int rows = (int)min((long)R, max(1L, ln_row - row0));
  auto row_at = [&](int r) { return a0 + (size_t)min(r, rows - 1) * ln_col; };
  const int last = ln_col - (VEC ? NV : 1), c0 = VEC ? NV * lane : lane;
  // the first values on their way to L2 under the flags (24576 x 8192 BF16: 107.9
  // -> 104 us)
#pragma unroll
  for (int r = 0; r < R; r++) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row_at(r) + min(part * SC + c0, last)));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row_at(r) + min((part + S) * SC + c0, last)));
  }
  int out = 0;  // x out of the range somewhere: the same in every CTA
  for (int k = lane; k < nbad; k += kWarp) out |= bad[k];
  if (__any_sync(0xffffffffu, out)) {
    rows_f64<V, R, VEC>(a0, rows, row0, ln_row, ln_col, log2s, x, y, fresh, s_part);
    return;
  }
  // (sh, sc): the Dot2 sum of P entries of a lane (kLong: of one step, FP32, or
  // two), then folded into one of the sums (th, tl) in turn
  constexpr bool LONG = SUMS == kLong;
  constexpr int P = SUMS == kEights ? 8 : SUMS == kPairs ? 2 : 4;
  constexpr int CH = LONG ? 1 : SUMS == kEights || (SUMS == kFours && NV == 4) ? 2 : 4;
  float sh[R], sc[R], th[CH][R], tl[CH][R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    sh[r] = sc[r] = 0.f;
#pragma unroll
    for (int q = 0; q < CH; q++) th[q][r] = tl[q][r] = 0.f;
  }
  auto fold = [&](int q) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const DF t = two_sum(th[q][r], sh[r]);
      th[q][r] = t.h;
      tl[q][r] = __fadd_rn(tl[q][r], __fadd_rn(t.l, sc[r]));
      const DF u = fast_two_sum(th[q][r], tl[q][r]);  // keeps tl small against th
      th[q][r] = u.h;
      tl[q][r] = u.l;
      sh[r] = sc[r] = 0.f;
    }
  };
  auto load = [&](Step<V, VEC>(&f)[R], int st) {
#pragma unroll
    for (int r = 0; r < R; r++) f[r].load(row_at(r), st * SC + c0, last, pol);
  };
  auto add = [&](const Step<V, VEC>(&f)[R], int st, int half) {
    const int c = st * SC + c0;
#pragma unroll
    for (int k0 = 0; k0 < NV; k0 += 4) {
      float xh[4], xl[4];
      if constexpr (VEC) {
        const int cc = min(c, last) + k0;
        const float4 h4 = *reinterpret_cast<const float4*>(xs + cc);
        const float4 l4 = *reinterpret_cast<const float4*>(xs + ln_col + cc);
        xh[0] = h4.x; xh[1] = h4.y; xh[2] = h4.z; xh[3] = h4.w;
        xl[0] = l4.x; xl[1] = l4.y; xl[2] = l4.z; xl[3] = l4.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int cc = min(c + 32 * (k0 + k), last);
          xh[k] = xs[cc];
          xl[k] = xs[ln_col + cc];
        }
      }
      if (st == nsteps - 1) {
#pragma unroll
        for (int k = 0; k < 4; k++)
          if ((VEC ? c : c + 32 * (k0 + k)) > last) xh[k] = xl[k] = 0.f;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int r = 0; r < R; r++) f[r].add(sh[r], sc[r], k0 + k, xh[k], xl[k]);
        if (!LONG && (k0 + k + 1) % P == 0) fold(((k0 + k) / P + half * (NV / P)) % CH);
      }
    }
  };
  int st = part;
  for (; st + S < nsteps; st += 2 * S) {
    Step<V, VEC> f0[R], f1[R];
    load(f0, st);
    load(f1, st + S);
    add(f0, st, 0);
    if constexpr (LONG && sizeof(V) == 4) fold(0);
    add(f1, st + S, 1);
    if constexpr (LONG) fold(0);
  }
  if (st < nsteps) {
    Step<V, VEC> f0[R];
    load(f0, st);
    add(f0, st, 0);
    if constexpr (LONG) fold(0);
  }
  DF t[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    t[r] = DF{th[0][r], tl[0][r]};
#pragma unroll
    for (int q = 1; q < CH; q++) t[r] = df_add(t[r], DF{th[q][r], tl[q][r]});
  }
  store_rows<R>(warp_sum_rows<R>(t, VEC && ln_col <= kBriefColumns), row0, ln_row, log2s, y, fresh, s_part);
}

// FP64 rows with 16-byte aligned starts (ln_col even): 16-byte loads.
__global__ void __launch_bounds__(NT) k_dense_f64x2(const double* __restrict__ A, int ln_row,
                                                   int ln_col, const double* __restrict__ x,
                                                   double* __restrict__ y) {
  const int lane = threadIdx.x % kWarp;
  const int gw = (blockIdx.x * NT + threadIdx.x) / kWarp;
  const int nw = gridDim.x * NT / kWarp;
  const uint64_t pol = policy_evict_first();
  const int half = ln_col / 2;
  const double2* x2 = reinterpret_cast<const double2*>(x);
  for (int row = gw; row < ln_row; row += nw) {
    const double* a = A + (size_t)row * ln_col;
    double acc0 = 0, acc1 = 0;
    int j = lane;
    for (; j + 3 * kWarp < half; j += 4 * kWarp) {
      double2 a0 = ld_stream2(a + 2 * j, pol), a1 = ld_stream2(a + 2 * (j + kWarp), pol);
      double2 a2 = ld_stream2(a + 2 * (j + 2 * kWarp), pol), a3 = ld_stream2(a + 2 * (j + 3 * kWarp), pol);
      double2 b0 = __ldg(x2 + j), b1 = __ldg(x2 + j + kWarp);
      double2 b2 = __ldg(x2 + j + 2 * kWarp), b3 = __ldg(x2 + j + 3 * kWarp);
      acc0 = fma_rn(a0.x, b0.x, acc0); acc1 = fma_rn(a0.y, b0.y, acc1);
      acc0 = fma_rn(a1.x, b1.x, acc0); acc1 = fma_rn(a1.y, b1.y, acc1);
      acc0 = fma_rn(a2.x, b2.x, acc0); acc1 = fma_rn(a2.y, b2.y, acc1);
      acc0 = fma_rn(a3.x, b3.x, acc0); acc1 = fma_rn(a3.y, b3.y, acc1);
    }
    for (; j < half; j += kWarp) {
      double2 a0 = ld_stream2(a + 2 * j, pol);
      double2 b0 = __ldg(x2 + j);
      acc0 = fma_rn(a0.x, b0.x, acc0);
      acc1 = fma_rn(a0.y, b0.y, acc1);
    }
    double acc = warp_sum(add_rn(acc0, acc1));
    if (lane == 0) y[row] = add_rn(y[row], acc);
  }
}

__global__ void k_vec_add(double* __restrict__ y, const double* __restrict__ x, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = add_rn(y[i], x[i]);
}

__global__ void k_vec_fill(double* __restrict__ y, double v, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = v;
}

// Warp per row; each entry's value added to its column's sum.
__global__ void k_col_sums(const double* __restrict__ vals, const int* __restrict__ rowptr,
                           const int* __restrict__ colidx, int n_row, int f_col, double* s) {
  const int lane = threadIdx.x % kWarp;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int nw = gridDim.x * blockDim.x / kWarp;
  for (int row = gw; row < n_row; row += nw)
    for (int j = rowptr[row] + lane; j < rowptr[row + 1]; j += kWarp)
      atomicAdd(s + (colidx[j] - f_col), vals[j]);
}

__global__ void k_normalize_cols(double* __restrict__ vals, const int* __restrict__ rowptr,
                                 const int* __restrict__ colidx, int n_row, int f_col,
                                 const double* __restrict__ s) {
  const int lane = threadIdx.x % kWarp;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int nw = gridDim.x * blockDim.x / kWarp;
  for (int row = gw; row < n_row; row += nw)
    for (int j = rowptr[row] + lane; j < rowptr[row + 1]; j += kWarp) {
      const double sv = s[colidx[j] - f_col];
      if (sv > 0) vals[j] = __ddiv_rn(vals[j], sv);
    }
}

// Pass 1: CTA b sums rows b, b + grid, ... per column into partials[b][k].
// With ncol == 1 all 256 threads stride over the vector.
__global__ void __launch_bounds__(256) k_colsum_pass1(const double* __restrict__ x, long n, int ncol,
                                                     double* __restrict__ partials) {
  __shared__ double s[256];
  double acc = 0;
  if (ncol == 1) {
    for (long i = blockIdx.x * 256L + threadIdx.x; i < n; i += (long)gridDim.x * 256) acc = add_rn(acc, x[i]);
    s[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
      for (int i = 0; i < 256; i++) t = add_rn(t, s[i]);
      partials[(size_t)blockIdx.x * 32] = t;
    }
    return;
  }
  const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
  if (lane < ncol)
    for (long i = (long)blockIdx.x * 8 + warp; i < n; i += (long)gridDim.x * 8) acc = add_rn(acc, x[i * ncol + lane]);
  s[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x < ncol) {
    double t = 0;
    for (int w = 0; w < 8; w++) t = add_rn(t, s[w * kWarp + threadIdx.x]);
    partials[(size_t)blockIdx.x * 32 + threadIdx.x] = t;
  }
}

__global__ void k_colsum_pass2(const double* __restrict__ partials, int nblk, int ncol, double* out) {
  if ((int)threadIdx.x >= ncol) return;
  double t = 0;
  for (int b = 0; b < nblk; b++) t = add_rn(t, partials[(size_t)b * 32 + threadIdx.x]);
  out[threadIdx.x] = t;
}

__global__ void k_scale_cols(double* __restrict__ x, long n, int ncol, const double* __restrict__ d) {
  const long total = n * ncol;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x)
    x[i] = __ddiv_rn(x[i], d[i % ncol]);
}

template <class V>
__global__ void k_convert(const double* __restrict__ src, V* __restrict__ dst, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = narrow<V>(src[i]);
}

inline int grid_for(long n, int per = 256) {
  return (int)std::max<long>(1, std::min<long>((n + per - 1) / per, 152L * 16));
}

}  // namespace

cudaError_t dense_gemv(const void* vals, int prec, int ln_row, int ln_col, const double* x,
                       double* y, cudaStream_t s) {
  if (ln_row == 0 || ln_col == 0) return cudaSuccess;
  const int grid = (int)std::min<long>(((long)ln_row + NT / kWarp - 1) / (NT / kWarp), 152L * 8);
  switch (prec) {
    case kF64:
      if (ln_col % 2 == 0 && ln_col >= 2 * NT * kDenseU && ((uintptr_t)vals % 16) == 0 && ((uintptr_t)x % 16) == 0)
        k_dense_rows_f64x2<kDenseU><<<ln_row, NT, 0, s>>>(  // a CTA per row, scheduled as CTAs retire
            static_cast<const double*>(vals), ln_row, ln_col, x, y);
      else if (ln_col % 2 == 0 && ((uintptr_t)vals % 16) == 0 && ((uintptr_t)x % 16) == 0)
        k_dense_f64x2<<<grid, NT, 0, s>>>(static_cast<const double*>(vals), ln_row, ln_col, x, y);
      else
        k_dense<double><<<grid, NT, 0, s>>>(static_cast<const double*>(vals), ln_row, ln_col, x, y);
      break;
    case kF32: k_dense<float><<<grid, NT, 0, s>>>(static_cast<const float*>(vals), ln_row, ln_col, x, y); break;
    case kBF16: k_dense<__nv_bfloat16><<<grid, NT, 0, s>>>(static_cast<const __nv_bfloat16*>(vals), ln_row, ln_col, x, y); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t dense_values_df_range(const void* vals, int prec, size_t n, int* flag, bool* ok, cudaStream_t s) {
  *ok = false;
  if (n == 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
  if (e) return e;
  const int grid = (int)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, 152 * 16));
  if (prec == kF64) k_df_range_vals<double><<<grid, 256, 0, s>>>(static_cast<const double*>(vals), n, flag);
  else if (prec == kF32) k_df_range_vals<float><<<grid, 256, 0, s>>>(static_cast<const float*>(vals), n, flag);
  else k_df_range_vals<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(vals), n, flag);
  int h = 1;
  if ((e = cudaGetLastError()) || (e = cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, s)) ||
      (e = cudaStreamSynchronize(s)))
    return e;
  *ok = h == 0;
  return cudaSuccess;
}

namespace {
template <class V, int R, bool VEC, Sums SUMS>
cudaError_t launch_dense_df(const V* a, int ln_row, int ln_col, int log2s, const float* xs, const double* x, const int* bad,
                     int nbad, double* y, int fresh, cudaStream_t s) {
  const long warps = (((long)ln_row + R - 1) / R) << log2s;
  const unsigned grid = (unsigned)((warps + NT / kWarp - 1) / (NT / kWarp));
  return launch_early(k_dense_df<V, R, VEC, SUMS>, grid, NT, 0, s, a, ln_row, ln_col, log2s, xs, x, bad, nbad, y, fresh);
}

// Rows per warp: 4 (FP32) or 2 (the others and kPairs, whose rows cost more
// registers a step: with 4, BF16 24576 x 8192 takes 120 us where 2 take 109, FP64
// 20000 x 8192 238 and 204), fewer where the GPU would not get half a warp's work for
// each resident warp.  Column parts: until there are four for each resident
// warp (FP32 16384 x 8192 with 1 / 2 / 4 / 8 parts: 106 / 104 / 102 / 100 us;
// BF16 24576 x 8192: 106 / 105 / 111 / 128), while a part keeps four steps (FP64
// 4000 x 2000, 16 steps: 4 parts 20.6 us, 8 parts 22.6).  Wide aligned FP64 rows
// (5120 columns: where it starts to pay) take four parts at least: a CTA then
// reads long pieces of few rows, and HBM gives more for fewer streams (20000
// rows, 2 / 4 / 8 parts: 5120 columns 133 / 132 / 144 us, 16384 columns 396 /
// 381 / 384).
template <class V, bool VEC, Sums SUMS>
cudaError_t dense_df_shape(const V* a, int ln_row, int ln_col, const float* xs, const double* x, const int* bad, int nbad,
                    double* y, int fresh, cudaStream_t s) {
  constexpr int kMost = sizeof(V) == 4 && SUMS != kPairs ? 4 : 2;
  constexpr long kWarps = 152L * 32;
  constexpr int SC = 32 * Step<V, VEC>::NV;
  const int nsteps = (ln_col + SC - 1) / SC;
  int most = 0;  // log2 of the most parts
  while (most < 3 && (nsteps >> (most + 1)) >= 4) most++;
  int r = kMost;
  while (r > 1 && (((long)ln_row + r - 1) / r << most) < kWarps / 2) r /= 2;
  int log2s = 0;
  while (log2s < most && (((long)ln_row + r - 1) / r << log2s) < 4 * kWarps) log2s++;
  if (sizeof(V) == 8 && VEC && nsteps >= 40) log2s = std::max(log2s, 2);
  if (r == 1) return launch_dense_df<V, 1, VEC, SUMS>(a, ln_row, ln_col, log2s, xs, x, bad, nbad, y, fresh, s);
  if constexpr (kMost >= 4)
    if (r == 4) return launch_dense_df<V, 4, VEC, SUMS>(a, ln_row, ln_col, log2s, xs, x, bad, nbad, y, fresh, s);
  return launch_dense_df<V, 2, VEC, SUMS>(a, ln_row, ln_col, log2s, xs, x, bad, nbad, y, fresh, s);
}

// The sums by the columns (see Sums; us of 24,000 rows, against kLong): BF16
// fours to 1792 columns (1104: 23.5, 19.9), eights to 4608 (1800: 34.6, 32.7;
// 2312: 41.3, 40.9), FP32 fours to 1536 (1104: 28.4, 26.2; 1504: 36.2, 33.2), FP64
// too (1104: 43.1, 42.9; 1504: 53.2, 52.8; HBM bounds it).
template <class V, bool VEC>
cudaError_t dense_df_sums(const V* a, int ln_row, int ln_col, const float* xs, const double* x, const int* bad, int nbad,
                          double* y, int fresh, cudaStream_t s) {
  constexpr int fours = sizeof(V) == 2 ? 1792 : 1536;
  if (ln_col <= fours) return dense_df_shape<V, VEC, kFours>(a, ln_row, ln_col, xs, x, bad, nbad, y, fresh, s);
  if constexpr (sizeof(V) == 2)
    if (ln_col <= 4608) return dense_df_shape<V, VEC, kEights>(a, ln_row, ln_col, xs, x, bad, nbad, y, fresh, s);
  return dense_df_shape<V, VEC, kLong>(a, ln_row, ln_col, xs, x, bad, nbad, y, fresh, s);
}

template <class V>
cudaError_t dense_df_vec(const void* vals, int ln_row, int ln_col, const float* xs, const double* x, const int* bad, int nbad,
                  double* y, int fresh, cudaStream_t s) {
  const V* a = static_cast<const V*>(vals);
  // NV values per lane and load when every row starts on a 16-byte boundary
  // and holds whole vectors (xs from cudaMalloc)
  constexpr int NV = Step<V, true>::NV;
  if ((uintptr_t)vals % 16 == 0 && (uintptr_t)xs % 16 == 0 && ln_col % NV == 0)
    return dense_df_sums<V, true>(a, ln_row, ln_col, xs, x, bad, nbad, y, fresh, s);
  if (ln_col <= (sizeof(V) == 8 ? 512 : 1100)) return dense_df_shape<V, false, kPairs>(a, ln_row, ln_col, xs, x, bad, nbad, y, fresh, s);
  return dense_df_sums<V, false>(a, ln_row, ln_col, xs, x, bad, nbad, y, fresh, s);
}
}  // namespace

cudaError_t dense_gemv_df(const void* vals, int prec, int ln_row, int ln_col, const double* x, float* xs,
                          int* bad, double* y, bool fresh, cudaStream_t s) {
  if (ln_row == 0 || ln_col == 0) return cudaSuccess;
  const int nbad = std::min((ln_col + NT - 1) / NT, kDenseFlags);
  cudaError_t e = launch_early(k_df_split_x, nbad, NT, 0, s, x, ln_col, xs, bad);
  if (e != cudaSuccess) return e;
  const int f = fresh ? 1 : 0;
  if (prec == kF64) return dense_df_vec<double>(vals, ln_row, ln_col, xs, x, bad, nbad, y, f, s);
  if (prec == kF32) return dense_df_vec<float>(vals, ln_row, ln_col, xs, x, bad, nbad, y, f, s);
  return dense_df_vec<__nv_bfloat16>(vals, ln_row, ln_col, xs, x, bad, nbad, y, f, s);
}

cudaError_t vec_add(double* y, const double* x, long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_vec_add<<<grid_for(n), 256, 0, s>>>(y, x, n);
  return cudaGetLastError();
}

cudaError_t vec_fill(double* y, double v, long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_vec_fill<<<grid_for(n), 256, 0, s>>>(y, v, n);
  return cudaGetLastError();
}

cudaError_t mat_colsum(const double* x, long n, int ncol, double* partials, double* out,
                       cudaStream_t s) {
  if (ncol < 1 || ncol > kWarp) return cudaErrorInvalidValue;
  k_colsum_pass1<<<kSumBlocks, 256, 0, s>>>(x, n, ncol, partials);
  k_colsum_pass2<<<1, 32, 0, s>>>(partials, kSumBlocks, ncol, out);
  return cudaGetLastError();
}

cudaError_t mat_scale_cols(double* x, long n, int ncol, const double* denom, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_scale_cols<<<grid_for(n * ncol), 256, 0, s>>>(x, n, ncol, denom);
  return cudaGetLastError();
}

cudaError_t csr_col_sums(const double* vals, const int* rowptr, const int* colidx, int n_row,
                         int f_col, double* s, cudaStream_t st) {
  if (n_row <= 0) return cudaSuccess;
  k_col_sums<<<grid_for((long)n_row * kWarp), 256, 0, st>>>(vals, rowptr, colidx, n_row, f_col, s);
  return cudaGetLastError();
}

cudaError_t csr_normalize_cols(double* vals, const int* rowptr, const int* colidx, int n_row,
                               int f_col, const double* s, cudaStream_t st) {
  if (n_row <= 0) return cudaSuccess;
  k_normalize_cols<<<grid_for((long)n_row * kWarp), 256, 0, st>>>(vals, rowptr, colidx, n_row, f_col, s);
  return cudaGetLastError();
}

cudaError_t convert_values(const double* src, void* dst, int prec, long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  switch (prec) {
    case kF64: return cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDeviceToDevice, s);
    case kF32: k_convert<float><<<grid_for(n), 256, 0, s>>>(src, (float*)dst, n); break;
    case kBF16: k_convert<__nv_bfloat16><<<grid_for(n), 256, 0, s>>>(src, (__nv_bfloat16*)dst, n); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace tbsla_gpu
