// Learned preconditioner for CG: a small message-passing network over the
// pattern of an SPD CSR matrix A that emits a lower-triangular factor L on
// the pattern of tril(A), so that M^-1 = L L^T stays SPD (every L_ii > 0).
// The reference has no preconditioner (src/mpi/matrix/CG.cpp:32-73 is plain
// CG); this is the project's own model, with Jacobi (L = D^-1/2, the
// network's starting point) as its fallback.
//
//   s_i = a_ii^-1/2, e_ij = a_ij s_i s_j on the stored entries (symmetric A),
//   computed in FP32
//   x_i = [1, sum_{j!=i} e_ij, sum_{j!=i} e_ij^2, deg_i / 8]
//   h0  = relu(W0 x + b0)                                  (width H = 32)
//   3 layers: m_i = sum_{j!=i} e_ij h_j;  z = W_l [h; m] + b_l;  h += relu(z)
//   L_ij = s_i (w_e . (h_i * h_j) + c_e e_ij + b_e)   (j < i)
//   L_ii = s_i softplus(w_d . h_i + b_d)
//   training loss over Gaussian probes Z (n x P): sum (L L^T A Z - Z)^2 / (nP)
//
// GPU mapping: one warp per node with the 32 features on the 32 lanes, so
// every gather of a neighbour's features is one 128-byte load.  The graph of a
// system (scaled edge weights, the patterns of L and L^T) is built on the
// device from the CSR arrays of each call.  Forward and backward are
// hand-written kernels in FP32 with the weights rounded to bfloat16 (FP32
// master copy in the Adam state); in the dense layers a lane keeps its
// output's 64 weights (and, backward, its 64 weight gradients) in registers
// and the activations of four nodes are read from shared memory by broadcast,
// so a node costs its 64 (backward 128) multiply-adds and little else;
// parameter gradients are reduced per CTA in shared memory, then added to
// global memory once per CTA.
// 48^3 nodes, 8 probes, loss and gradient from the host arrays: 5.17 -> 0.79 ms
// (the host's graph 3.9 ms of it, a layer backward 268 -> 35 us, forward 57 ->
// 28 us without its gather).
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <vector>

#include "api_guard.hpp"
#include "device.hpp"
#include "host/matrix.hpp"
#include "kernels/common.cuh"
#include "kernels/kernels.hpp"
#include "probe_rows.hpp"
#include "tbsla_gb300.h"

namespace {

using tbsla_gpu::kWarp;

constexpr int H = 32, F0 = 4, NL = 3, NT = 256;
constexpr int LSZ = 2 * H * H + H;  // one message layer: W (H x 2H) then b
constexpr int OFF_W0 = 0, OFF_B0 = H * F0, OFF_L = OFF_B0 + H;
constexpr int OFF_WE = OFF_L + NL * LSZ, OFF_CE = OFF_WE + H, OFF_BE = OFF_CE + 1;
constexpr int OFF_WD = OFF_BE + 1, OFF_BD = OFF_WD + H;
constexpr int NPARAMS = OFF_BD + 1;
static_assert(NPARAMS == 6467, "parameter layout");
constexpr unsigned FULL = 0xffffffffu;

__host__ __device__ inline int off_layer(int l) { return OFF_L + (l - 1) * LSZ; }  // l = 1..NL

// ---- device kernels: one system's graph ------------------------------------------------
// L: per row its strictly lower entries (in A's order), then the diagonal;
// L^T: per column j the L entries of that column, in row order.

// What the host looks at before the lists are built.
struct GraphCheck {
  int bad_col;   // a column outside the matrix
  int bad_diag;  // a row without a positive diagonal entry
  int max_col;   // most L entries in a column
};
constexpr int kShortCol = 32;  // longest column of L that is ordered in place

// s_i = a_ii^-1/2 in FP32 (repeated diagonal entries added in FP64), A's
// values in FP32, and the lengths of L's row and column i.  The FP32
// operations of s, e and x are those of k_dia_features, so that both give the
// same bits.
__global__ void __launch_bounds__(NT) k_graph_rows(int n, int base, const int* __restrict__ rowptr,
                                                  const int* __restrict__ colidx, const double* __restrict__ a64,
                                                  float* __restrict__ aval, float* __restrict__ s,
                                                  unsigned* __restrict__ lcount, unsigned* __restrict__ tcount,
                                                  GraphCheck* __restrict__ check) {
  int most = 0;
  for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) {
    const int k0 = rowptr[i] - base, k1 = rowptr[i + 1] - base;
    double d = 0;
    unsigned nl = 1;
    for (int k = k0; k < k1; k++) {
      const double v = a64[k];
      const int j = colidx[k];
      aval[k] = (float)v;
      if (j < 0 || j >= n) {
        check->bad_col = 1;
        continue;
      }
      if (j == i) d += v;
      if (j < i) {
        nl++;
        most = max(most, (int)atomicAdd(tcount + j, 1u) + 1);
      }
    }
    if (!(d > 0)) check->bad_diag = 1;
    s[i] = 1.0f / sqrtf((float)d);
    lcount[i] = nl;
    most = max(most, (int)atomicAdd(tcount + i, 1u) + 1);
  }
  most = __reduce_max_sync(FULL, most);
  if ((threadIdx.x & 31) == 0) atomicMax(&check->max_col, most);
}

// Edge weights and node inputs; L's entries (lsrc: the entry of A, -1 for the
// diagonal), and into L^T's lists either their places (tnext: the next free
// place of each column, in any order) or, with tnext null, sort keys.
__global__ void __launch_bounds__(NT) k_graph_fill(int n, const int* __restrict__ rowptr,
                                                  const int* __restrict__ colidx, const float* __restrict__ aval,
                                                  const float* __restrict__ s, const int* __restrict__ lrowptr,
                                                  float* __restrict__ e, float* __restrict__ x,
                                                  int* __restrict__ lcol, int* __restrict__ lsrc,
                                                  int* __restrict__ lrow, unsigned* __restrict__ tnext,
                                                  uint64_t* __restrict__ keys, int* __restrict__ tidx) {
  for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) {
    const float si = s[i];
    float se = 0.f, se2 = 0.f;
    int deg = 0, q = lrowptr[i];
    auto entry = [&](int col, int src) {
      lcol[q] = col;
      lsrc[q] = src;
      lrow[q] = (int)i;
      if (tnext) {
        tidx[atomicAdd(tnext + col, 1u)] = q;
      } else {
        keys[q] = (unsigned)col;
        tidx[q] = q;
      }
      q++;
    };
    for (int k = rowptr[i]; k < rowptr[i + 1]; k++) {
      const int j = colidx[k];
      const float ev = __fmul_rn(__fmul_rn(aval[k], si), s[j]);
      e[k] = ev;
      if (j != i) {
        se = __fadd_rn(se, ev);
        se2 = fmaf(ev, ev, se2);
        deg++;
      }
      if (j < i) entry(j, k);
    }
    entry((int)i, -1);
    x[i * F0 + 0] = 1.f;
    x[i * F0 + 1] = se;
    x[i * F0 + 2] = se2;
    x[i * F0 + 3] = deg / 8.f;
  }
}

// L^T's lists into row order (columns of at most kShortCol entries).
__global__ void __launch_bounds__(NT) k_order_columns(int n, const int* __restrict__ trowptr,
                                                     int* __restrict__ tidx) {
  for (long j = blockIdx.x * (long)NT + threadIdx.x; j < n; j += (long)gridDim.x * NT) {
    const int t0 = trowptr[j], t1 = trowptr[j + 1];
    for (int t = t0 + 1; t < t1; t++) {
      const int q = tidx[t];
      int u = t;
      for (; u > t0 && tidx[u - 1] > q; u--) tidx[u] = tidx[u - 1];
      tidx[u] = q;
    }
  }
}

__global__ void k_shift(int n, int base, int* __restrict__ v) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] -= base;
}

__global__ void k_narrow(long len, const double* __restrict__ src, float* __restrict__ dst) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < len; t += (long)gridDim.x * blockDim.x)
    dst[t] = __double2float_rn(src[t]);
}

// ---- device kernels: forward ---------------------------------------------------------

__device__ __forceinline__ float relu(float v) { return v > 0.f ? v : 0.f; }
__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
__device__ __forceinline__ float softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float sigmoid(float v) { return 1.f / (1.f + expf(-v)); }

__device__ __forceinline__ long warp_id() { return ((long)blockIdx.x * NT + threadIdx.x) / kWarp; }
__device__ __forceinline__ long warp_count() { return (long)gridDim.x * NT / kWarp; }

// h0 = relu(W0 x + b0); lane o is feature o.  mask[i] bit o: the
// pre-activation is positive (what the backward pass needs of it).
__global__ void __launch_bounds__(NT) k_layer0(int n, const float* __restrict__ x, const float* __restrict__ w,
                                              unsigned* __restrict__ mask, float* __restrict__ h0) {
  const int o = threadIdx.x & 31;
  float wr[F0];
#pragma unroll
  for (int k = 0; k < F0; k++) wr[k] = w[OFF_W0 + o * F0 + k];
  const float b = w[OFF_B0 + o];
  for (long i = warp_id(); i < n; i += warp_count()) {
    float z = b;
#pragma unroll
    for (int k = 0; k < F0; k++) z += wr[k] * x[i * F0 + k];
    const unsigned pos = __ballot_sync(FULL, z > 0.f);
    if (o == 0) mask[i] = pos;
    h0[i * H + o] = relu(z);
  }
}

constexpr int NB = 4;  // nodes that a warp takes together

// The lists ptr[i] .. ptr[i + 1) of nodes i0 .. i0 + 3 when all of them have
// at most 8 entries (every 7-point stencil): lane 8 u + t holds entry t of node
// i0 + u, so the four lists are read in one go instead of one after another.
struct Quad {
  int k;          // this lane's entry (valid if `live`)
  bool live;
  bool all_short; // same on every lane
  __device__ __forceinline__ Quad(const int* __restrict__ ptr, int drop, long i0, int n) {
    const int lane = threadIdx.x & 31;
    const long i = i0 + (lane >> 3);
    const int b = i < n ? ptr[i] : 0, len = i < n ? ptr[i + 1] - drop - b : 0;
    k = b + (lane & 7);
    live = (lane & 7) < len;
    all_short = !__any_sync(FULL, len > 8);
  }
};

// acc[u] += sum_{j != i} e_ij in_j over A's row i = i0 + u (e symmetric, so
// this is also the transpose product the backward pass needs); lane f is
// feature f, entries in order, 16 neighbours' features in flight.
__device__ __forceinline__ void gather_rows(const int* __restrict__ rowptr, const int* __restrict__ colidx,
                                            const float* __restrict__ e, const float* __restrict__ in, long i0,
                                            int n, int f, float (&acc)[NB]) {
  const Quad qd(rowptr, 0, i0, n);
  if (qd.all_short) {
    const int cl = qd.live ? colidx[qd.k] : 0;
    const float el = qd.live ? e[qd.k] : 0.f;
    const unsigned use = __ballot_sync(FULL, qd.live && cl != i0 + (f >> 3));
#pragma unroll
    for (int u = 0; u < NB; u += 2) {
      float v[16];
#pragma unroll
      for (int t = 0; t < 16; t++) {
        const int c = __shfl_sync(FULL, cl, 8 * u + t);
        v[t] = use >> (8 * u + t) & 1u ? in[(long)c * H + f] : 0.f;
      }
#pragma unroll
      for (int t = 0; t < 16; t++) {
        const float ev = __shfl_sync(FULL, el, 8 * u + t);
        if (use >> (8 * u + t) & 1u) acc[u + (t >> 3)] += ev * v[t];
      }
    }
    return;
  }
#pragma unroll
  for (int u = 0; u < NB; u++) {
    const long i = i0 + u;
    if (i >= n) break;
    const int k1 = rowptr[i + 1];
    for (int k0 = rowptr[i]; k0 < k1; k0 += kWarp) {
      const int m = min(kWarp, k1 - k0);
      const int cl = f < m ? colidx[k0 + f] : (int)i;
      const float el = f < m ? e[k0 + f] : 0.f;
      for (int t = 0; t < m; t += 8) {
        int c[8];
        float v[8];
#pragma unroll
        for (int r = 0; r < 8; r++) {
          c[r] = __shfl_sync(FULL, cl, (t + r) & 31);
          v[r] = t + r < m ? in[(long)c[r] * H + f] : 0.f;
        }
#pragma unroll
        for (int r = 0; r < 8; r++) {
          const float ev = __shfl_sync(FULL, el, (t + r) & 31);
          if (t + r < m && c[r] != i) acc[u] += ev * v[r];
        }
      }
    }
  }
}

// out_i = [out_i +] the gathered neighbours of i.  A kernel of its own: fused
// into the dense layers, whose weights in registers leave 8 to 16 warps on an
// SM, the gathers' latency showed (48^3 nodes, caches cold: 70 us forward and
// 185 us backward per layer, against 24 + 28 and 24 + 35 us).
__global__ void __launch_bounds__(NT) k_gather(int n, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                                              const float* __restrict__ e, const float* __restrict__ in,
                                              float* __restrict__ out, int accumulate) {
  const int f = threadIdx.x & 31;
  for (long i0 = warp_id() * NB; i0 < n; i0 += warp_count() * NB) {
    float old[NB], acc[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      old[u] = accumulate && i0 + u < n ? out[(i0 + u) * H + f] : 0.f;
      acc[u] = 0.f;
    }
    gather_rows(rowptr, colidx, e, in, i0, n, f, acc);
#pragma unroll
    for (int u = 0; u < NB; u++)
      if (i0 + u < n) out[(i0 + u) * H + f] = accumulate ? old[u] + acc[u] : acc[u];
  }
}

// z = W [h; m] + b, h_out = h + relu(z).  Lane o holds row o of W (H x 2H) in
// registers; the next pass's activations are loaded under this one's
// multiply-adds.
__global__ void __launch_bounds__(NT, 2) k_layer(int n, const float* __restrict__ w, const float* __restrict__ h,
                                                 const float* __restrict__ m, unsigned* __restrict__ mask,
                                                 float* __restrict__ hout) {
  __shared__ float ws[H][2 * H + 1];
  __shared__ __align__(16) float in[NT / kWarp][NB][2 * H];
  for (int t = threadIdx.x; t < 2 * H * H; t += NT) ws[t / (2 * H)][t % (2 * H)] = w[t];
  __syncthreads();
  const int o = threadIdx.x & 31;
  float wr[2 * H];
#pragma unroll
  for (int k = 0; k < 2 * H; k++) wr[k] = ws[o][k];
  const float b = w[2 * H * H + o];
  auto& st = in[threadIdx.x / kWarp];
  float hi[NB], mi[NB];
  auto load = [&](long i0) {
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const bool live = i0 + u < n;
      hi[u] = live ? h[(i0 + u) * H + o] : 0.f;
      mi[u] = live ? m[(i0 + u) * H + o] : 0.f;
    }
  };
  const long step = warp_count() * NB;
  long i0 = warp_id() * NB;
  load(i0);
  for (; i0 < n; i0 += step) {
    float hc[NB], acc[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      st[u][o] = hc[u] = hi[u];
      st[u][H + o] = mi[u];
      acc[u] = b;
    }
    __syncwarp();
    load(i0 + step);
#pragma unroll
    for (int k = 0; k < H; k += 4) {
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const float4 hv = *reinterpret_cast<const float4*>(&st[u][k]);
        const float4 mv = *reinterpret_cast<const float4*>(&st[u][H + k]);
        acc[u] += wr[k] * hv.x;
        acc[u] += wr[H + k] * mv.x;
        acc[u] += wr[k + 1] * hv.y;
        acc[u] += wr[H + k + 1] * mv.y;
        acc[u] += wr[k + 2] * hv.z;
        acc[u] += wr[H + k + 2] * mv.z;
        acc[u] += wr[k + 3] * hv.w;
        acc[u] += wr[H + k + 3] * mv.w;
      }
    }
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const unsigned pos = __ballot_sync(FULL, acc[u] > 0.f);
      if (i0 + u < n) {
        if (o == 0) mask[i0 + u] = pos;
        hout[(i0 + u) * H + o] = hc[u] + relu(acc[u]);
      }
    }
    __syncwarp();
  }
}

// The warp sums wsum() of v0 .. v3 -- the same pairs in the same order -- on
// every lane of the quarter q = (lane >> 3) of the warp that belongs to v_q:
// six shuffles instead of twenty.
__device__ __forceinline__ float wsum4(float v0, float v1, float v2, float v3) {
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 16, mid = lane & 8;
  // distance 16: the lower half keeps v0 and v1, the upper one v2 and v3
  const float a = (hi ? v2 : v0) + __shfl_xor_sync(FULL, hi ? v0 : v2, 16);
  const float b = (hi ? v3 : v1) + __shfl_xor_sync(FULL, hi ? v1 : v3, 16);
  float r = (mid ? b : a) + __shfl_xor_sync(FULL, mid ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(FULL, r, o);
  return r;
}

// L values: a warp per four rows; lower entries then the diagonal.  xi (the
// diagonal's pre-activation) is kept for the backward pass.
__global__ void __launch_bounds__(NT) k_head(int n, const int* __restrict__ lrowptr, const int* __restrict__ lcol,
                                            const int* __restrict__ lsrc, const float* __restrict__ e,
                                            const float* __restrict__ s, const float* __restrict__ w,
                                            const float* __restrict__ h, float* __restrict__ lval,
                                            float* __restrict__ xi) {
  const int f = threadIdx.x & 31;
  const float we = w[OFF_WE + f], wd = w[OFF_WD + f];
  const float ce = w[OFF_CE], be = w[OFF_BE], bd = w[OFF_BD];
  for (long i0 = warp_id() * NB; i0 < n; i0 += warp_count() * NB) {
    float hi[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) hi[u] = i0 + u < n ? h[(i0 + u) * H + f] : 0.f;
    const Quad qd(lrowptr, 1, i0, n);  // the strictly lower entries
    if (qd.all_short) {
      const int cl = qd.live ? lcol[qd.k] : 0;
      const float el = qd.live ? e[lsrc[qd.k]] : 0.f;
      const unsigned use = __ballot_sync(FULL, qd.live);
      float dot = 0.f;  // this lane's entry's sum
#pragma unroll
      for (int u = 0; u < NB; u++) {
#pragma unroll
        for (int t = 0; t < 8; t += 4) {
          if ((use >> (8 * u + t) & 0xfu) == 0) continue;
          float v[4];
#pragma unroll
          for (int r = 0; r < 4; r++) {
            const int j = __shfl_sync(FULL, cl, 8 * u + t + r);
            v[r] = use >> (8 * u + t + r) & 1u ? h[(long)j * H + f] : 0.f;
          }
#pragma unroll
          for (int r = 0; r < 4; r++) v[r] = we * hi[u] * v[r];
          // v[r]'s sum from a lane of quarter r to the lane that holds the entry
          const float q = wsum4(v[0], v[1], v[2], v[3]);
          const float d = __shfl_sync(FULL, q, (f & 3) * 8);
          if (f >> 2 == 2 * u + (t >> 2)) dot = d;
        }
      }
      if (qd.live) lval[qd.k] = s[i0 + (f >> 3)] * (dot + ce * el + be);
    } else {
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const long i = i0 + u;
        if (i >= n) break;
        for (int q = lrowptr[i]; q < lrowptr[i + 1] - 1; q++) {
          const float o = wsum(we * hi[u] * h[(long)lcol[q] * H + f]) + ce * e[lsrc[q]] + be;
          if (f == 0) lval[q] = s[i] * o;
        }
      }
    }
    const float x = wsum4(wd * hi[0], wd * hi[1], wd * hi[2], wd * hi[3]) + bd;
    const long i = i0 + (f >> 3);
    if ((f & 7) == 0 && i < n) {
      xi[i] = x;
      lval[lrowptr[i + 1] - 1] = s[i] * softplus(x);
    }
  }
}

// ---- device kernels: loss ------------------------------------------------------------
// Probe blocks are n x P row-major (P <= 16), a thread per row and probe: the
// P threads of a row read consecutive words of every X row.

constexpr int PMAX = 16;

// Y = A X on A's pattern (FP32 values).
template <bool WIDE>
__global__ void k_spmm_a(int n, int P, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                         const float* __restrict__ a, const float* __restrict__ X, float* __restrict__ Y) {
  const long len = (long)n * P;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < len; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)tbsla_gpu::probe_row<WIDE>(t, P), p = (int)(t - (long)i * P);
    float acc = 0.f;
    for (int k = rowptr[i]; k < rowptr[i + 1]; k++) acc += a[k] * X[(long)colidx[k] * P + p];
    Y[t] = acc;
  }
}

// Y = L X (rows of L) or Y = L^T X (columns of L, through the L^T index).
template <bool WIDE>
__global__ void k_spmm_l(int n, int P, const int* __restrict__ ptr, const int* __restrict__ idx,
                         const int* __restrict__ other, const float* __restrict__ lval, int transpose,
                         const float* __restrict__ X, float* __restrict__ Y) {
  const long len = (long)n * P;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < len; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)tbsla_gpu::probe_row<WIDE>(t, P), p = (int)(t - (long)i * P);
    float acc = 0.f;
    for (int k = ptr[i]; k < ptr[i + 1]; k++) {
      const int q = transpose ? idx[k] : k;  // L entry; its column (L) or row (L^T):
      acc += lval[q] * X[(long)other[q] * P + p];
    }
    Y[t] = acc;
  }
}

// G = 2 (W - Z) / (nP) and the loss sum((W - Z)^2) / (nP) (double atomics
// of per-CTA sums).
__global__ void __launch_bounds__(NT) k_residual(long len, float scale, const float* __restrict__ W,
                                                const float* __restrict__ Z, float* __restrict__ G,
                                                double* __restrict__ loss) {
  __shared__ double red[NT / kWarp];
  double acc = 0;
  for (long t = blockIdx.x * (long)NT + threadIdx.x; t < len; t += (long)gridDim.x * NT) {
    const float r = W[t] - Z[t];
    G[t] = 2.f * r * scale;
    acc += (double)r * r;
  }
  acc = tbsla_gpu::block_sum<NT>(acc, red);
  if (threadIdx.x == 0) atomicAdd(loss, acc * scale);
}

// dL_q = sum_p G_ip V_jp + U_ip GV_jp for L entry q = (i, j).
__global__ void k_dl(long nl, int P, const int* __restrict__ lrow, const int* __restrict__ lcol,
                     const float* __restrict__ G, const float* __restrict__ V, const float* __restrict__ U,
                     const float* __restrict__ GV, float* __restrict__ dl) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < nl; q += (long)gridDim.x * blockDim.x) {
    const long i = lrow[q], j = lcol[q];
    float acc = 0.f;
    for (int p = 0; p < P; p++) acc += G[i * P + p] * V[j * P + p] + U[i * P + p] * GV[j * P + p];
    dl[q] = acc;
  }
}

// Gaussian probes (Box-Muller over a counter-based SplitMix64 stream).
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__global__ void k_gauss(long len, unsigned long long seed, float* __restrict__ Z) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < len; t += (long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix64(seed * 0x100000001b3ull + (unsigned long long)t);
    const float u1 = ((r >> 40) + 0.5f) * (1.f / 16777216.f);
    const float u2 = ((r & 0xffffff) + 0.5f) * (1.f / 16777216.f);
    Z[t] = sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
  }
}

// ---- device kernels: backward --------------------------------------------------------

// Head: dL -> parameter gradients of the head, and dh (written, not added: the
// first contribution to it), a warp per four nodes.  Row side: the row's lower
// entries and its diagonal; column side: dh_i += sum over the strictly lower
// entries (r, i) of s_r dL_ri w_e * h_r.
__global__ void __launch_bounds__(NT) k_head_bwd(int n, const int* __restrict__ lrowptr,
                                                const int* __restrict__ lcol, const int* __restrict__ lsrc,
                                                const int* __restrict__ trowptr, const int* __restrict__ tidx,
                                                const int* __restrict__ lrow, const float* __restrict__ e,
                                                const float* __restrict__ s, const float* __restrict__ w,
                                                const float* __restrict__ h, const float* __restrict__ dl,
                                                const float* __restrict__ xi, float* __restrict__ dh,
                                                float* __restrict__ grad) {
  __shared__ float part[NT / kWarp][2 * H + 3];
  const int f = threadIdx.x & 31, wi = threadIdx.x / kWarp;
  const float we = w[OFF_WE + f], wd = w[OFF_WD + f];
  float gwe = 0.f, gwd = 0.f, gce = 0.f, gbe = 0.f, gbd = 0.f;  // gce, gbe, gbd: this lane's entries
  for (long i0 = warp_id() * NB; i0 < n; i0 += warp_count() * NB) {
    float hi[NB], d[NB], dc[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      hi[u] = i0 + u < n ? h[(i0 + u) * H + f] : 0.f;
      d[u] = dc[u] = 0.f;
    }
    const Quad lo(lrowptr, 1, i0, n), up(trowptr, 0, i0, n);
    if (lo.all_short && up.all_short) {
      const long i = i0 + (f >> 3);
      const int cl = lo.live ? lcol[lo.k] : 0, src = lo.live ? lsrc[lo.k] : 0;
      const int q = up.live ? tidx[up.k] : 0;
      const float dO = lo.live ? s[i] * dl[lo.k] : 0.f;
      const int rl = up.live ? lrow[q] : 0;
      const float cf = up.live ? s[rl] * dl[q] : 0.f;
      if (lo.live) {
        gce += dO * e[src];
        gbe += dO;
      }
      const unsigned ul = __ballot_sync(FULL, lo.live), uc = __ballot_sync(FULL, up.live && rl != i);
#pragma unroll
      for (int u = 0; u < NB; u++) {
        float v[8], r[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int j = __shfl_sync(FULL, cl, 8 * u + t), k = __shfl_sync(FULL, rl, 8 * u + t);
          v[t] = ul >> (8 * u + t) & 1u ? h[(long)j * H + f] : 0.f;
          r[t] = uc >> (8 * u + t) & 1u ? h[(long)k * H + f] : 0.f;
        }
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const float g = __shfl_sync(FULL, dO, 8 * u + t), c = __shfl_sync(FULL, cf, 8 * u + t);
          if (ul >> (8 * u + t) & 1u) {
            gwe += g * hi[u] * v[t];
            d[u] += g * we * v[t];
          }
          if (uc >> (8 * u + t) & 1u) dc[u] += c * we * r[t];
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const long i = i0 + u;
        if (i >= n) break;
        for (int q = lrowptr[i]; q < lrowptr[i + 1] - 1; q++) {
          const float g = s[i] * dl[q], hj = h[(long)lcol[q] * H + f];
          gwe += g * hi[u] * hj;
          d[u] += g * we * hj;
          if (f == 0) {
            gce += g * e[lsrc[q]];
            gbe += g;
          }
        }
        for (int t = trowptr[i]; t < trowptr[i + 1]; t++) {
          const int q = tidx[t], r = lrow[q];
          if (r != i) dc[u] += s[r] * dl[q] * we * h[(long)r * H + f];
        }
      }
    }
    // the diagonals, a lane each, then broadcast
    float dxi = 0.f;
    if (f < NB && i0 + f < n) {
      const long i = i0 + f;
      dxi = s[i] * dl[lrowptr[i + 1] - 1] * sigmoid(xi[i]);
    }
    gbd += dxi;
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const float x = __shfl_sync(FULL, dxi, u);
      gwd += x * hi[u];
      if (i0 + u < n) dh[(i0 + u) * H + f] = d[u] + x * wd + dc[u];
    }
  }
  gce = wsum(gce);
  gbe = wsum(gbe);
  gbd = wsum(gbd);
  part[wi][f] = gwe;
  part[wi][H + f] = gwd;
  if (f == 0) {
    part[wi][2 * H] = gce;
    part[wi][2 * H + 1] = gbe;
    part[wi][2 * H + 2] = gbd;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * H + 3; c += NT) {
    float acc = 0.f;
    for (int v = 0; v < NT / kWarp; v++) acc += part[v][c];
    const int dst = c < H ? OFF_WE + c : c < 2 * H ? OFF_WD + c - H : c == 2 * H ? OFF_CE : c == 2 * H + 1 ? OFF_BE : OFF_BD;
    atomicAdd(grad + dst, acc);
  }
}

// Message layer backward for h_out = h + relu(W [h; m] + b):
//   dz = dh_out where z > 0, else 0;  dW += dz [h; m]^T;  db += dz;
//   dh_in = dh_out + (W^T dz)[:H] (in place);  dm = (W^T dz)[H:]
// Lane o holds columns o and H + o of W and row o of dW in registers; the
// next pass's activations are loaded under this one's multiply-adds.
__global__ void __launch_bounds__(NT, 1) k_layer_bwd(int n, const float* __restrict__ w, const float* __restrict__ h,
                                                    const float* __restrict__ m, const unsigned* __restrict__ mask,
                                                    float* __restrict__ dh, float* __restrict__ dm,
                                                    float* __restrict__ grad) {
  constexpr int S = 2 * H + 1;
  __shared__ float ws[H * S];
  __shared__ __align__(16) float in[NT / kWarp][NB][2 * H];
  __shared__ __align__(16) float sdz[NT / kWarp][NB][H];
  for (int t = threadIdx.x; t < 2 * H * H; t += NT) ws[t / (2 * H) * S + t % (2 * H)] = w[t];
  __syncthreads();
  const int o = threadIdx.x & 31, wi = threadIdx.x / kWarp;
  float wh[H], wm[H], gw[2 * H];
#pragma unroll
  for (int k = 0; k < H; k++) {
    wh[k] = ws[k * S + o];
    wm[k] = ws[k * S + H + o];
  }
#pragma unroll
  for (int k = 0; k < 2 * H; k++) gw[k] = 0.f;
  float gb = 0.f;
  float hi[NB], mi[NB], di[NB];
  unsigned mk[NB];
  auto load = [&](long i0) {
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const bool live = i0 + u < n;
      hi[u] = live ? h[(i0 + u) * H + o] : 0.f;
      mi[u] = live ? m[(i0 + u) * H + o] : 0.f;
      di[u] = live ? dh[(i0 + u) * H + o] : 0.f;
      mk[u] = live ? mask[i0 + u] : 0u;
    }
  };
  const long step = warp_count() * NB;
  long i0 = warp_id() * NB;
  load(i0);
  for (; i0 < n; i0 += step) {
    float dhi[NB], dz[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      dhi[u] = di[u];
      dz[u] = mk[u] >> o & 1u ? di[u] : 0.f;
      in[wi][u][o] = hi[u];
      in[wi][u][H + o] = mi[u];
      sdz[wi][u][o] = dz[u];
      gb += dz[u];
    }
    __syncwarp();
    load(i0 + step);
    float a[NB], c[NB];  // W^T dz
#pragma unroll
    for (int u = 0; u < NB; u++) a[u] = c[u] = 0.f;
#pragma unroll
    for (int k = 0; k < H; k += 4) {
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const float4 z = *reinterpret_cast<const float4*>(&sdz[wi][u][k]);
        a[u] += wh[k] * z.x;
        c[u] += wm[k] * z.x;
        a[u] += wh[k + 1] * z.y;
        c[u] += wm[k + 1] * z.y;
        a[u] += wh[k + 2] * z.z;
        c[u] += wm[k + 2] * z.z;
        a[u] += wh[k + 3] * z.w;
        c[u] += wm[k + 3] * z.w;
      }
    }
#pragma unroll
    for (int u = 0; u < NB; u++) {
#pragma unroll
      for (int k = 0; k < 2 * H; k += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&in[wi][u][k]);
        gw[k] += dz[u] * v.x;
        gw[k + 1] += dz[u] * v.y;
        gw[k + 2] += dz[u] * v.z;
        gw[k + 3] += dz[u] * v.w;
      }
    }
#pragma unroll
    for (int u = 0; u < NB; u++)
      if (i0 + u < n) {
        dh[(i0 + u) * H + o] = dhi[u] + a[u];
        dm[(i0 + u) * H + o] = c[u];
      }
    __syncwarp();
  }
  // the warps' gradients, added in warp order (row o of dW at stride S: no
  // bank conflicts), then one addition per CTA
  __syncthreads();
  for (int wv = 0; wv < NT / kWarp; wv++) {
    if (wi == wv) {
#pragma unroll
      for (int k = 0; k < 2 * H; k++) ws[o * S + k] = wv ? ws[o * S + k] + gw[k] : gw[k];
      in[0][0][o] = wv ? in[0][0][o] + gb : gb;
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < 2 * H * H; t += NT) atomicAdd(grad + t, ws[t / (2 * H) * S + t % (2 * H)]);
  if (threadIdx.x < H) atomicAdd(grad + 2 * H * H + threadIdx.x, in[0][0][threadIdx.x]);
}

// Input layer backward: dW0 += dz0 x^T, db0 += dz0.
__global__ void __launch_bounds__(NT) k_layer0_bwd(int n, const float* __restrict__ x,
                                                  const unsigned* __restrict__ mask, const float* __restrict__ dh,
                                                  float* __restrict__ grad) {
  __shared__ float gsum[NT / kWarp][F0 + 1][H];
  const int o = threadIdx.x & 31, wi = threadIdx.x / kWarp;
  float gw[F0] = {}, gb = 0.f;
  for (long i = warp_id(); i < n; i += warp_count()) {
    const float dz = mask[i] >> o & 1u ? dh[i * H + o] : 0.f;
#pragma unroll
    for (int k = 0; k < F0; k++) gw[k] += dz * x[i * F0 + k];
    gb += dz;
  }
#pragma unroll
  for (int k = 0; k < F0; k++) gsum[wi][k][o] = gw[k];
  gsum[wi][F0][o] = gb;
  __syncthreads();
  for (int t = threadIdx.x; t < (F0 + 1) * H; t += NT) {
    const int k = t / H, r = t % H;
    float acc = 0.f;
    for (int v = 0; v < NT / kWarp; v++) acc += gsum[v][k][r];
    atomicAdd(grad + (k < F0 ? OFF_W0 + r * F0 + k : OFF_B0 + r), acc);
  }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters; the forward copy is
// the bfloat16 rounding of the result.
__global__ void k_adam(int np, float* __restrict__ theta, const float* __restrict__ g, float* __restrict__ mo,
                       float* __restrict__ ve, float* __restrict__ wq, float lr, float c1, float c2) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < np; t += gridDim.x * blockDim.x) {
    const float gt = g[t];
    const float m = b1 * mo[t] + (1.f - b1) * gt;
    const float v = b2 * ve[t] + (1.f - b2) * gt * gt;
    mo[t] = m;
    ve[t] = v;
    const float th = theta[t] - lr * (m / c1) / (sqrtf(v / c2) + eps);
    theta[t] = th;
    wq[t] = __bfloat162float(__float2bfloat16_rn(th));
  }
}


// ---- device kernels: inference on a batch's DIA copy ----------------------------------
// The batch keeps A slot-major per diagonal: a64[k * n + i] is the entry of row i
// on diagonal k of its system (delta adelta[sys * 8 + k], ascending, so slot
// order is the CSR order of a sorted row); 0 where the row has none.  Entries
// stored as exact zeros are therefore absent here.  Activations are kept
// feature-major, hT[f * n + i], so that a thread per node reads and writes
// them coalesced across its warp (32 consecutive nodes, 128 bytes per
// feature).  Every kernel does the FP32 operations of the training path's
// kernels (k_layer0, k_gather + k_layer, k_head), so the factor is
// tbsla_mpnn_factor's up to the order of FP32 sums.

constexpr int DMAX = 8;  // diagonal slots per system

// The weights of one kernel, passed by value: every multiply-add takes its
// weight from the constant bank (a compile-time offset), no load at all.
struct InputW {
  float w0[H * F0];
  float b0[H];
};
struct LayerW {
  float w[2 * H * H];  // W (H x 2H) row-major
  float b[H];
};
struct HeadW {
  float we[H], wd[H];
  float ce, be, bd;
};

// s_i = a_ii^-1/2, e_ij = a_ij s_i s_j and the node inputs x_i (FP32, as
// build_graph), then h0 = relu(W0 x + b0) written feature-major; *bad set
// when a diagonal entry is <= 0.
__global__ void __launch_bounds__(NT) k_dia_features(long n, int K, const double* __restrict__ a64,
                                                     const int* __restrict__ adelta, const int* __restrict__ row_sys,
                                                     const __grid_constant__ InputW P, float* __restrict__ e,
                                                     float* __restrict__ s, float* __restrict__ h0,
                                                     int* __restrict__ bad) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int sys = row_sys[i];
    int kd = -1;
    for (int k = 0; k < K && kd < 0; k++)
      if (adelta[sys * DMAX + k] == 0) kd = k;
    const double di = kd >= 0 ? a64[(size_t)kd * n + i] : 0.0;
    if (!(di > 0)) {
      atomicExch(bad, 1);
      for (int k = 0; k < K; k++) e[(size_t)k * n + i] = 0.f;
      s[i] = 0.f;
      for (int o = 0; o < H; o++) h0[(size_t)o * n + i] = 0.f;
      continue;
    }
    const float si = 1.0f / sqrtf((float)di);
    s[i] = si;
    float se = 0.f, se2 = 0.f;
    int deg = 0;
    for (int k = 0; k < K; k++) {
      const double a = a64[(size_t)k * n + i];
      const int dl = adelta[sys * DMAX + k];
      if (a == 0.0) {
        e[(size_t)k * n + i] = 0.f;
        continue;
      }
      const double dj = a64[(size_t)kd * n + i + dl];
      const float sj = dl == 0 ? si : 1.0f / sqrtf((float)dj);
      const float ev = __fmul_rn(__fmul_rn((float)a, si), sj);
      e[(size_t)k * n + i] = ev;
      if (dl != 0) {
        se = __fadd_rn(se, ev);
        se2 = fmaf(ev, ev, se2);
        deg++;
      }
    }
    const float x1 = se, x2 = se2, x3 = deg / 8.f;
#pragma unroll
    for (int o = 0; o < H; o++) {
      float z = P.b0[o];
      z = fmaf(P.w0[o * F0 + 0], 1.f, z);
      z = fmaf(P.w0[o * F0 + 1], x1, z);
      z = fmaf(P.w0[o * F0 + 2], x2, z);
      z = fmaf(P.w0[o * F0 + 3], x3, z);
      h0[(size_t)o * n + i] = relu(z);
    }
  }
}

// One message layer for inference, a thread per node: m_i = sum_{j != i}
// e_ij h_j over the DIA slots, z = b + W [h; m] (per k the h term, then the
// m term, as k_layer), h_out = h + relu(z).  Four outputs at a time give the
// FMA pipe independent chains.
__global__ void __launch_bounds__(NT, 2) k_layer_fm(long n, int K, const int* __restrict__ adelta,
                                                    const int* __restrict__ row_sys, const float* __restrict__ e,
                                                    const __grid_constant__ LayerW P, const float* __restrict__ hT,
                                                    float* __restrict__ outT) {
  for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) {
    const int sys = row_sys[i];
    float h[H], m[H];
#pragma unroll
    for (int f = 0; f < H; f++) {
      h[f] = hT[(size_t)f * n + i];
      m[f] = 0.f;
    }
    for (int k = 0; k < K; k++) {
      const int dl = adelta[sys * DMAX + k];
      const float ev = e[(size_t)k * n + i];
      if (dl == 0 || ev == 0.f) continue;
      const float* hj = hT + i + dl;
#pragma unroll
      for (int f = 0; f < H; f++) m[f] = fmaf(ev, hj[(size_t)f * n], m[f]);
    }
#pragma unroll
    for (int o = 0; o < H; o += 4) {
      float a0 = P.b[o], a1 = P.b[o + 1], a2 = P.b[o + 2], a3 = P.b[o + 3];
#pragma unroll
      for (int k = 0; k < H; k++) {
        a0 = fmaf(P.w[(o + 0) * 2 * H + k], h[k], a0);
        a1 = fmaf(P.w[(o + 1) * 2 * H + k], h[k], a1);
        a2 = fmaf(P.w[(o + 2) * 2 * H + k], h[k], a2);
        a3 = fmaf(P.w[(o + 3) * 2 * H + k], h[k], a3);
        a0 = fmaf(P.w[(o + 0) * 2 * H + H + k], m[k], a0);
        a1 = fmaf(P.w[(o + 1) * 2 * H + H + k], m[k], a1);
        a2 = fmaf(P.w[(o + 2) * 2 * H + H + k], m[k], a2);
        a3 = fmaf(P.w[(o + 3) * 2 * H + H + k], m[k], a3);
      }
      outT[(size_t)(o + 0) * n + i] = h[o + 0] + relu(a0);
      outT[(size_t)(o + 1) * n + i] = h[o + 1] + relu(a1);
      outT[(size_t)(o + 2) * n + i] = h[o + 2] + relu(a2);
      outT[(size_t)(o + 3) * n + i] = h[o + 3] + relu(a3);
    }
  }
}

__device__ __forceinline__ void store_l(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_l(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// The warp butterfly of wsum() restated over 32 values held by one thread:
// the same pairs in the same order, so the same sum.
__device__ __forceinline__ float tree_sum(float (&p)[H]) {
#pragma unroll
  for (int f = 0; f < 16; f++) p[f] = p[f] + p[f + 16];
#pragma unroll
  for (int f = 0; f < 8; f++) p[f] = p[f] + p[f + 8];
#pragma unroll
  for (int f = 0; f < 4; f++) p[f] = p[f] + p[f + 4];
#pragma unroll
  for (int f = 0; f < 2; f++) p[f] = p[f] + p[f + 2];
  return p[0] + p[1];
}

// L into the batch's DIA factor, a thread per node: slot 0 the diagonal s_i
// softplus(w_d . h_i + b_d); slot q > 0 (delta ldelta[q] < 0, 0 = padding)
// s_i (w_e . (h_i * h_j) + c_e e_ij + b_e) where A has the entry, else 0.
template <class LV>
__global__ void __launch_bounds__(NT, 2) k_head_fm(long n, int K, const int* __restrict__ adelta, int KL,
                                                   const int* __restrict__ ldelta, const int* __restrict__ row_sys,
                                                   const float* __restrict__ e, const float* __restrict__ s,
                                                   const __grid_constant__ HeadW P, const float* __restrict__ hT,
                                                   LV* __restrict__ lv) {
  for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) {
    const int sys = row_sys[i];
    const float si = s[i];
    float h[H], p[H];
#pragma unroll
    for (int f = 0; f < H; f++) h[f] = hT[(size_t)f * n + i];
    for (int q = 1; q < KL; q++) {
      const int dl = ldelta[sys * DMAX + q];
      float ev = 0.f;
      if (dl != 0)
        for (int k = 0; k < K; k++)
          if (adelta[sys * DMAX + k] == dl) ev = e[(size_t)k * n + i];
      float out = 0.f;
      if (ev != 0.f) {
        const float* hj = hT + i + dl;
#pragma unroll
        for (int f = 0; f < H; f++) p[f] = P.we[f] * h[f] * hj[(size_t)f * n];
        const float o = tree_sum(p) + P.ce * ev + P.be;
        out = si * o;
      }
      store_l(lv + (size_t)q * n + i, out);
    }
#pragma unroll
    for (int f = 0; f < H; f++) p[f] = P.wd[f] * h[f];
    const float xd = tree_sum(p) + P.bd;
    store_l(lv + i, si * softplus(xd));
  }
}

// ---- host orchestration --------------------------------------------------------------

#define MCK(call)                                               \
  do {                                                          \
    cudaError_t e_ = (call);                                    \
    if (e_ != cudaSuccess) {                                    \
      cudaGetLastError();                                       \
      return e_ == cudaErrorMemoryAllocation ? TBSLA_ERR_ALLOC  \
                                             : TBSLA_ERR_CUDA;  \
    }                                                           \
  } while (0)

// A device buffer that grows on demand.
template <class T>
struct Grow {
  T* p = nullptr;
  size_t cap = 0;
  int need(size_t n) {
    if (n <= cap && p) return TBSLA_OK;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    MCK(cudaMalloc((void**)&p, std::max<size_t>(n, 1) * sizeof(T)));
    cap = n;
    return TBSLA_OK;
  }
  template <class V>
  int put(const std::vector<V>& v, cudaStream_t s) {
    int st = need(v.size());
    if (st) return st;
    if (!v.empty()) MCK(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    return TBSLA_OK;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
};

// One system's graph plus the activations and probe blocks of one pass.
struct Work {
  int n = 0, P = 0;
  long nnz = 0, nl = 0;
  Grow<int> rowptr, colidx, lrowptr, lcol, lsrc, lrow, trowptr, tidx, tidx2;
  Grow<GraphCheck> check;
  Grow<uint64_t> keys, keys2;
  Grow<unsigned> scratch, tnext, mask[NL + 1];
  Grow<double> a64;
  Grow<float> aval, e, s, x, lval, xi, dl;
  Grow<float> h[NL + 1], m[NL + 1], dh, dm;
  Grow<float> Z, U, V, W, G, GV;
  void release() {
    for (auto* g : {&rowptr, &colidx, &lrowptr, &lcol, &lsrc, &lrow, &trowptr, &tidx, &tidx2}) g->release();
    for (auto* g : {&keys, &keys2}) g->release();
    for (auto* g : {&aval, &e, &s, &x, &lval, &xi, &dl, &dh, &dm, &Z, &U, &V, &W, &G, &GV}) g->release();
    check.release();
    tnext.release();
    scratch.release();
    a64.release();
    for (int l = 0; l <= NL; l++) {
      h[l].release();
      m[l].release();
      mask[l].release();
    }
  }
};

int warp_grid(long n) { return (int)std::max<long>(1, std::min<long>((n + NT / kWarp - 1) / (NT / kWarp), 152L * 8)); }
int row_grid(long n) { return (int)std::max<long>(1, std::min<long>((n + NT - 1) / NT, 152L * 16)); }
// CTAs of the dense-layer kernels: a pass of NB nodes per warp, at most `per`
// CTAs per SM, which share the loading of the weights among many passes
int layer_grid(long n, int per) {
  return (int)std::max<long>(1, std::min<long>((n + NB * (NT / kWarp) - 1) / (NB * (NT / kWarp)), 152L * per));
}

// The graph of a square CSR handle, built on the device from its arrays, and
// the buffers of a pass with P probes; TBSLA_ERR_BAD_MATRIX unless every row
// holds a positive diagonal entry.  Synchronises once (the length of L and
// the check of the diagonal).
int build_graph(const tbsla_matrix* mat, int P, Work* w, cudaStream_t st) {
  const tbsla_info& I = mat->info;
  if (mat->format != TBSLA_CSR || I.ln_row != I.ln_col || I.f_col != 0) return TBSLA_ERR_INVALID_ARG;
  const int n = I.ln_row;
  if (n > 0 && I.nnz == 0) return TBSLA_ERR_BAD_MATRIX;
  // the row pointer here (as tbsla_impl::validate does), the columns on the device
  if (n > 0 && mat->idx0.size() != (size_t)n + 1) return TBSLA_ERR_BAD_MATRIX;
  const int* rp = mat->idx0.data();
  const int base = n > 0 ? rp[0] : 0;
  int falls = base < 0;
  for (int i = 0; i < n; i++) falls |= rp[i + 1] < rp[i];
  if (falls) return TBSLA_ERR_BAD_MATRIX;
  const long end = n > 0 ? rp[n] : 0, nnz = end - base;
  if ((size_t)end > mat->idx1.size() || (size_t)end > mat->values.size()) return TBSLA_ERR_BAD_MATRIX;
  w->n = n;
  w->P = P;
  w->nnz = nnz;
  w->nl = 0;
  int r;
  const size_t nh = (size_t)n * H, np = (size_t)n * std::max(P, 1), n1 = (size_t)n + 1;
  if ((r = w->rowptr.need(n1)) || (r = w->colidx.need(nnz)) || (r = w->a64.need(nnz)) || (r = w->aval.need(nnz)) ||
      (r = w->e.need(nnz)) || (r = w->s.need(n)) || (r = w->x.need((size_t)n * F0)) || (r = w->lrowptr.need(n1)) ||
      (r = w->trowptr.need(n1)) || (r = w->tnext.need(n1)) || (r = w->check.need(1)) ||
      (r = w->scratch.need(tbsla_gpu::scan_scratch((long)n1))) || (r = w->dh.need(nh)) || (r = w->dm.need(nh)) ||
      (r = w->xi.need(n)))
    return r;
  for (int l = 0; l <= NL; l++)
    if ((r = w->h[l].need(nh)) || (r = w->m[l].need(nh)) || (r = w->mask[l].need(n))) return r;
  for (auto* b : {&w->Z, &w->U, &w->V, &w->W, &w->G, &w->GV})
    if ((r = b->need(np))) return r;
  if (n == 0) return TBSLA_OK;
  MCK(cudaMemcpyAsync(w->rowptr.p, rp, n1 * 4, cudaMemcpyHostToDevice, st));
  MCK(cudaMemcpyAsync(w->colidx.p, mat->idx1.data() + base, nnz * 4, cudaMemcpyHostToDevice, st));
  MCK(cudaMemcpyAsync(w->a64.p, mat->values.data() + base, nnz * 8, cudaMemcpyHostToDevice, st));
  const int gr = row_grid(n);
  unsigned* lcount = reinterpret_cast<unsigned*>(w->lrowptr.p);
  unsigned* tcount = reinterpret_cast<unsigned*>(w->trowptr.p);
  MCK(cudaMemsetAsync(w->check.p, 0, sizeof(GraphCheck), st));
  MCK(cudaMemsetAsync(tcount, 0, n1 * sizeof(unsigned), st));
  MCK(cudaMemsetAsync(lcount + n, 0, sizeof(unsigned), st));
  k_graph_rows<<<gr, NT, 0, st>>>(n, base, w->rowptr.p, w->colidx.p, w->a64.p, w->aval.p, w->s.p, lcount, tcount,
                                  w->check.p);
  MCK(cudaGetLastError());
  if (base) k_shift<<<gr, NT, 0, st>>>(n + 1, base, w->rowptr.p);
  MCK(tbsla_gpu::exclusive_scan(lcount, (long)n1, w->scratch.p, st));
  MCK(tbsla_gpu::exclusive_scan(tcount, (long)n1, w->scratch.p, st));
  GraphCheck check{};
  int nl = 0;
  MCK(cudaMemcpyAsync(&check, w->check.p, sizeof check, cudaMemcpyDeviceToHost, st));
  MCK(cudaMemcpyAsync(&nl, w->lrowptr.p + n, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  if (check.bad_col || check.bad_diag) return TBSLA_ERR_BAD_MATRIX;
  w->nl = nl;
  // L^T's lists, each in L's order: put in place in any order and ordered
  // there when every column is short (48^3 nodes: 21 us with the fill, against
  // about 150 us for the stable sort by column that the others take)
  const bool in_place = check.max_col <= kShortCol;
  if ((r = w->lcol.need(nl)) || (r = w->lsrc.need(nl)) || (r = w->lrow.need(nl)) || (r = w->tidx.need(nl)) ||
      (r = w->lval.need(nl)) || (r = w->dl.need(nl)))
    return r;
  if (!in_place && ((r = w->tidx2.need(nl)) || (r = w->keys.need(nl)) || (r = w->keys2.need(nl)) ||
                    (r = w->scratch.need(tbsla_gpu::radix_scratch(nl)))))
    return r;
  if (in_place) MCK(cudaMemcpyAsync(w->tnext.p, tcount, n1 * sizeof(unsigned), cudaMemcpyDeviceToDevice, st));
  k_graph_fill<<<gr, NT, 0, st>>>(n, w->rowptr.p, w->colidx.p, w->aval.p, w->s.p, w->lrowptr.p, w->e.p, w->x.p,
                                  w->lcol.p, w->lsrc.p, w->lrow.p, in_place ? w->tnext.p : nullptr, w->keys.p,
                                  w->tidx.p);
  if (in_place) {
    k_order_columns<<<gr, NT, 0, st>>>(n, w->trowptr.p, w->tidx.p);
    MCK(cudaGetLastError());
    return TBSLA_OK;
  }
  MCK(cudaGetLastError());
  int bits = 1, alt = 0;
  while (bits < 31 && (1L << bits) < (long)n) bits++;
  MCK(tbsla_gpu::radix_sort_pairs(w->keys.p, w->keys2.p, w->tidx.p, w->tidx2.p, nl, bits, w->scratch.p, &alt, st));
  if (alt) std::swap(w->tidx, w->tidx2);
  return TBSLA_OK;
}
// Forward pass: activations and L values.
int forward(const float* wq, Work& w, cudaStream_t s) {
  const int n = w.n, gw = warp_grid(n), gq = warp_grid(((long)n + NB - 1) / NB);
  k_layer0<<<gw, NT, 0, s>>>(n, w.x.p, wq, w.mask[0].p, w.h[0].p);
  for (int l = 1; l <= NL; l++) {
    k_gather<<<gq, NT, 0, s>>>(n, w.rowptr.p, w.colidx.p, w.e.p, w.h[l - 1].p, w.m[l].p, 0);
    k_layer<<<layer_grid(n, 2), NT, 0, s>>>(n, wq + off_layer(l), w.h[l - 1].p, w.m[l].p, w.mask[l].p, w.h[l].p);
  }
  k_head<<<gq, NT, 0, s>>>(n, w.lrowptr.p, w.lcol.p, w.lsrc.p, w.e.p, w.s.p, wq, w.h[NL].p, w.lval.p, w.xi.p);
  MCK(cudaGetLastError());
  return TBSLA_OK;
}

// Loss on the probes in w.Z and the gradient into grad (zeroed here).
int backward(const float* wq, Work& w, double* dloss, float* grad, cudaStream_t s) {
  const int n = w.n, P = w.P, gw = warp_grid(n), gq = warp_grid(((long)n + NB - 1) / NB);
  const long len = (long)n * P;
  const int gp = row_grid(len);
  const bool wide = tbsla_gpu::probe_rows_wide(len);
  const auto spmm_a = wide ? k_spmm_a<true> : k_spmm_a<false>;
  const auto spmm_l = wide ? k_spmm_l<true> : k_spmm_l<false>;
  spmm_a<<<gp, NT, 0, s>>>(n, P, w.rowptr.p, w.colidx.p, w.aval.p, w.Z.p, w.U.p);
  spmm_l<<<gp, NT, 0, s>>>(n, P, w.trowptr.p, w.tidx.p, w.lrow.p, w.lval.p, 1, w.U.p, w.V.p);
  spmm_l<<<gp, NT, 0, s>>>(n, P, w.lrowptr.p, nullptr, w.lcol.p, w.lval.p, 0, w.V.p, w.W.p);
  MCK(cudaMemsetAsync(dloss, 0, sizeof(double), s));
  k_residual<<<std::min(gp, 152 * 2), NT, 0, s>>>(len, 1.f / (float)len, w.W.p, w.Z.p, w.G.p, dloss);
  spmm_l<<<gp, NT, 0, s>>>(n, P, w.trowptr.p, w.tidx.p, w.lrow.p, w.lval.p, 1, w.G.p, w.GV.p);
  k_dl<<<row_grid(w.nl), NT, 0, s>>>(w.nl, P, w.lrow.p, w.lcol.p, w.G.p, w.V.p, w.U.p, w.GV.p, w.dl.p);
  MCK(cudaMemsetAsync(grad, 0, NPARAMS * sizeof(float), s));
  k_head_bwd<<<std::min(gq, 152 * 6), NT, 0, s>>>(n, w.lrowptr.p, w.lcol.p, w.lsrc.p, w.trowptr.p, w.tidx.p,
                                                  w.lrow.p, w.e.p, w.s.p, wq, w.h[NL].p, w.dl.p, w.xi.p, w.dh.p,
                                                  grad);
  for (int l = NL; l >= 1; l--) {
    k_layer_bwd<<<layer_grid(n, 1), NT, 0, s>>>(n, wq + off_layer(l), w.h[l - 1].p, w.m[l].p, w.mask[l].p, w.dh.p,
                                                w.dm.p, grad + off_layer(l));
    k_gather<<<gq, NT, 0, s>>>(n, w.rowptr.p, w.colidx.p, w.e.p, w.dm.p, w.dh.p, 1);
  }
  k_layer0_bwd<<<std::min(gw, 152 * 4), NT, 0, s>>>(n, w.x.p, w.mask[0].p, w.dh.p, grad);
  MCK(cudaGetLastError());
  return TBSLA_OK;
}

float bf16_round(float v) {
  uint32_t u;
  std::memcpy(&u, &v, 4);
  if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x7fffu + ((u >> 16) & 1u)) & 0xffff0000u;
  float r;
  std::memcpy(&r, &u, 4);
  return r;
}

}  // namespace

struct tbsla_mpnn {
  int device = 0;
  cudaStream_t stream = nullptr;
  float *theta = nullptr, *wq = nullptr, *grad = nullptr, *mo = nullptr, *ve = nullptr;
  double* dloss = nullptr;
  long step = 0;
  Work work;
  ~tbsla_mpnn() {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    work.release();
    for (void* p : {(void*)theta, (void*)wq, (void*)grad, (void*)mo, (void*)ve, (void*)dloss})
      if (p) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
  }
  int set(const std::vector<float>& th) {
    std::vector<float> q(th.size());
    for (size_t k = 0; k < th.size(); k++) q[k] = bf16_round(th[k]);
    MCK(cudaMemcpyAsync(theta, th.data(), NPARAMS * 4, cudaMemcpyHostToDevice, stream));
    MCK(cudaMemcpyAsync(wq, q.data(), NPARAMS * 4, cudaMemcpyHostToDevice, stream));
    MCK(cudaMemsetAsync(mo, 0, NPARAMS * 4, stream));
    MCK(cudaMemsetAsync(ve, 0, NPARAMS * 4, stream));
    MCK(cudaStreamSynchronize(stream));
    step = 0;
    return TBSLA_OK;
  }
};


namespace tbsla_impl {

int mpnn_factor_dia(tbsla_mpnn* net, long n, int K, const double* a64, const int* adelta, const int* row_sys,
                    int KL, const int* ldelta, void* lvals, int lprec, void* stream) {
  if (!net || n <= 0 || K <= 0 || K > DMAX || KL <= 0 || KL > DMAX || !a64 || !adelta || !row_sys || !ldelta ||
      !lvals || (lprec != TBSLA_F32 && lprec != TBSLA_BF16))
    return TBSLA_ERR_INVALID_ARG;
  cudaSetDevice(net->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Work& w = net->work;
  int st;
  // scratch kept with the network and grown on demand: e [K][n], s, two
  // feature-major activation buffers and the error flag
  if ((st = w.e.need((size_t)K * n)) || (st = w.s.need(n)) || (st = w.h[0].need((size_t)n * H)) ||
      (st = w.h[1].need((size_t)n * H)) || (st = w.xi.need(1)))
    return st;
  int* bad = reinterpret_cast<int*>(w.xi.p);
  MCK(cudaMemsetAsync(bad, 0, sizeof(int), s));
  // the bfloat16-rounded forward weights, by value into each kernel
  std::vector<float> wh(NPARAMS);
  MCK(cudaMemcpyAsync(wh.data(), net->wq, NPARAMS * 4, cudaMemcpyDeviceToHost, s));
  MCK(cudaStreamSynchronize(s));
  InputW pin;
  std::memcpy(pin.w0, wh.data() + OFF_W0, sizeof pin.w0);
  std::memcpy(pin.b0, wh.data() + OFF_B0, sizeof pin.b0);
  HeadW phd;
  std::memcpy(phd.we, wh.data() + OFF_WE, sizeof phd.we);
  std::memcpy(phd.wd, wh.data() + OFF_WD, sizeof phd.wd);
  phd.ce = wh[OFF_CE];
  phd.be = wh[OFF_BE];
  phd.bd = wh[OFF_BD];
  const int grow = row_grid(n);
  float* cur = w.h[0].p;  // feature-major activations [H][n]
  float* nxt = w.h[1].p;
  k_dia_features<<<grow, NT, 0, s>>>(n, K, a64, adelta, row_sys, pin, w.e.p, w.s.p, cur, bad);
  for (int l = 1; l <= NL; l++) {
    LayerW pl;
    std::memcpy(pl.w, wh.data() + off_layer(l), sizeof pl.w);
    std::memcpy(pl.b, wh.data() + off_layer(l) + 2 * H * H, sizeof pl.b);
    k_layer_fm<<<grow, NT, 0, s>>>(n, K, adelta, row_sys, w.e.p, pl, cur, nxt);
    std::swap(cur, nxt);
  }
  if (lprec == TBSLA_BF16)
    k_head_fm<__nv_bfloat16><<<grow, NT, 0, s>>>(n, K, adelta, KL, ldelta, row_sys, w.e.p, w.s.p, phd, cur,
                                                 static_cast<__nv_bfloat16*>(lvals));
  else
    k_head_fm<float><<<grow, NT, 0, s>>>(n, K, adelta, KL, ldelta, row_sys, w.e.p, w.s.p, phd, cur,
                                         static_cast<float*>(lvals));
  MCK(cudaGetLastError());
  int hbad = 0;
  MCK(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  MCK(cudaStreamSynchronize(s));
  return hbad ? TBSLA_ERR_BAD_MATRIX : TBSLA_OK;
}

}  // namespace tbsla_impl

// ---- C ABI ---------------------------------------------------------------------------

extern "C" {

int tbsla_mpnn_create(tbsla_mpnn** out, unsigned long long seed) try {
  if (!out) return TBSLA_ERR_INVALID_ARG;
  *out = nullptr;
  int dev = 0;
  int st = tbsla_impl::dev_ready(&dev);
  if (st) return st;
  std::unique_ptr<tbsla_mpnn> net(new (std::nothrow) tbsla_mpnn());  // freed on every failure path
  if (!net) return TBSLA_ERR_ALLOC;
  net->device = dev;
  cudaSetDevice(dev);
  if (cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&net->theta, NPARAMS * 4) != cudaSuccess || cudaMalloc(&net->wq, NPARAMS * 4) != cudaSuccess ||
      cudaMalloc(&net->grad, NPARAMS * 4) != cudaSuccess || cudaMalloc(&net->mo, NPARAMS * 4) != cudaSuccess ||
      cudaMalloc(&net->ve, NPARAMS * 4) != cudaSuccess || cudaMalloc(&net->dloss, 8) != cudaSuccess) {
    cudaGetLastError();
    return TBSLA_ERR_ALLOC;
  }
  // He-scaled message layers, zero biases; the head starts at L = D^-1/2
  // (Jacobi): w_e = c_e = b_e = w_d = 0 and softplus(b_d) = 1.
  std::vector<float> th(NPARAMS, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> n0(0.f, std::sqrt(2.f / F0)), nl(0.f, 0.5f * std::sqrt(2.f / (2 * H)));
  for (int k = 0; k < H * F0; k++) th[OFF_W0 + k] = n0(rng);
  for (int l = 1; l <= NL; l++)
    for (int k = 0; k < 2 * H * H; k++) th[off_layer(l) + k] = nl(rng);
  th[OFF_BD] = std::log(std::exp(1.f) - 1.f);
  st = net->set(th);
  if (st) return st;
  *out = net.release();
  return TBSLA_OK;
} TBSLA_API_CATCH

int tbsla_mpnn_destroy(tbsla_mpnn* net) try {
  delete net;
  return TBSLA_OK;
} TBSLA_API_CATCH

int tbsla_mpnn_params(const tbsla_mpnn* net, float* theta, int* nparams) try {
  if (!net) return TBSLA_ERR_INVALID_ARG;
  if (nparams) *nparams = NPARAMS;
  if (theta) {
    cudaSetDevice(net->device);
    MCK(cudaMemcpyAsync(theta, net->theta, NPARAMS * 4, cudaMemcpyDeviceToHost, net->stream));
    MCK(cudaStreamSynchronize(net->stream));
  }
  return TBSLA_OK;
} TBSLA_API_CATCH

int tbsla_mpnn_set_params(tbsla_mpnn* net, const float* theta, int nparams) try {
  if (!net || !theta || nparams != NPARAMS) return TBSLA_ERR_INVALID_ARG;
  cudaSetDevice(net->device);
  return net->set(std::vector<float>(theta, theta + NPARAMS));
} TBSLA_API_CATCH

int tbsla_mpnn_loss_grad(tbsla_mpnn* net, const tbsla_matrix* A, int nprobes, const double* Z, double* loss,
                         float* grad) try {
  if (!net || !A || nprobes < 1 || nprobes > PMAX || !Z) return TBSLA_ERR_INVALID_ARG;
  cudaSetDevice(net->device);
  cudaStream_t s = net->stream;
  Work& w = net->work;
  int st = build_graph(A, nprobes, &w, s);
  if (st) return st;
  const long len = (long)w.n * nprobes;
  if (len > 0) {  // the probes in FP32
    if ((st = w.a64.need(len))) return st;
    MCK(cudaMemcpyAsync(w.a64.p, Z, len * 8, cudaMemcpyHostToDevice, s));
    k_narrow<<<row_grid(len), NT, 0, s>>>(len, w.a64.p, w.Z.p);
  }
  if ((st = forward(net->wq, w, s)) || (st = backward(net->wq, w, net->dloss, net->grad, s))) return st;
  double l = 0;
  MCK(cudaMemcpyAsync(&l, net->dloss, 8, cudaMemcpyDeviceToHost, s));
  if (grad) MCK(cudaMemcpyAsync(grad, net->grad, NPARAMS * 4, cudaMemcpyDeviceToHost, s));
  MCK(cudaStreamSynchronize(s));
  if (loss) *loss = l;
  return TBSLA_OK;
} TBSLA_API_CATCH

int tbsla_mpnn_train_step(tbsla_mpnn* net, const tbsla_matrix* A, int nprobes, unsigned long long seed, float lr,
                          double* loss) try {
  if (!net || !A || nprobes < 1 || nprobes > PMAX || !(lr > 0)) return TBSLA_ERR_INVALID_ARG;
  cudaSetDevice(net->device);
  cudaStream_t s = net->stream;
  Work& w = net->work;
  int st = build_graph(A, nprobes, &w, s);
  if (st) return st;
  const long len = (long)w.n * nprobes;
  k_gauss<<<row_grid(len), NT, 0, s>>>(len, seed, w.Z.p);
  if ((st = forward(net->wq, w, s)) || (st = backward(net->wq, w, net->dloss, net->grad, s))) return st;
  net->step++;
  const float c1 = 1.f - std::pow(0.9f, (float)net->step), c2 = 1.f - std::pow(0.999f, (float)net->step);
  k_adam<<<(NPARAMS + NT - 1) / NT, NT, 0, s>>>(NPARAMS, net->theta, net->grad, net->mo, net->ve, net->wq, lr, c1,
                                               c2);
  MCK(cudaGetLastError());
  double l = 0;
  MCK(cudaMemcpyAsync(&l, net->dloss, 8, cudaMemcpyDeviceToHost, s));
  MCK(cudaStreamSynchronize(s));
  if (loss) *loss = l;
  return TBSLA_OK;
} TBSLA_API_CATCH

int tbsla_mpnn_factor(tbsla_mpnn* net, const tbsla_matrix* A, tbsla_matrix* L) try {
  if (!net || !A || !L || L->format != TBSLA_CSR) return TBSLA_ERR_INVALID_ARG;
  cudaSetDevice(net->device);
  cudaStream_t s = net->stream;
  Work& w = net->work;
  int st = build_graph(A, 1, &w, s);
  if (st || (st = forward(net->wq, w, s))) return st;
  std::vector<float> lv(w.nl);
  std::vector<int> lrp(w.n + 1, 0), lci(w.nl);
  if (w.n > 0) {
    MCK(cudaMemcpyAsync(lv.data(), w.lval.p, w.nl * 4, cudaMemcpyDeviceToHost, s));
    MCK(cudaMemcpyAsync(lrp.data(), w.lrowptr.p, lrp.size() * 4, cudaMemcpyDeviceToHost, s));
    MCK(cudaMemcpyAsync(lci.data(), w.lcol.p, w.nl * 4, cudaMemcpyDeviceToHost, s));
  }
  MCK(cudaStreamSynchronize(s));
  std::vector<double> vals(lv.begin(), lv.end());
  tbsla_info I{};
  I.n_row = I.n_col = I.ln_row = I.ln_col = w.n;
  I.nnz = w.nl;
  I.NR = I.NC = 1;
  return tbsla_matrix_set_csr(L, &I, vals.data(), lrp.data(), lci.data());
} TBSLA_API_CATCH

}  // extern "C"
