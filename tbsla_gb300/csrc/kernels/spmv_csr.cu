// CSR SpMV, row-block adaptive (the CSR-Stream / CSR-Vector scheme of
// Greathouse & Daga, SC'14, built here for sm_103a), and the PageRank steps
// that reuse its traversal with a fused epilogue.
//
// Replaces tbsla::cpp::MatrixCSR::Ax (src/cpp/matrix/MatrixCSR.cpp:209-233):
// y_i = sum_j values_j * v[colidx_j - f_col], overwriting y.
//
// Layout: the reference CSR arrays as they are (int32 rowptr / colidx, values
// in the storage precision) plus a row-block partition built once per
// matrix (csr_partition).  A block is either
//  - a run of <= 256 consecutive rows holding <= 256*ITEMS entries
//    ("stream" block): the CTA reads the block's values and column indices
//    with coalesced loads, gathers x, stages (value, x) pairs in shared
//    memory, then sums each row with a group of G lanes, G = the largest
//    power of two with G * rows <= 256 (capped at 32), one fused
//    multiply-add per entry in entry order;
//  - one row longer than 256*ITEMS, or longer than its G lanes would walk in
//    kCsrMaxSteps steps ("vector" block): the whole CTA strides over it and
//    reduces.  One row of 1024 entries among rows of 10 kept its block's other
//    255 threads waiting for one (G = 1): 27 us where now 8 (10,000 rows);
//    3000 rows of a power law, 24 entries a row: 39 -> 8.4 us.
// GB300's FP64 pipe is narrow, so the kernel spends exactly one FP64
// instruction (DFMA) per entry, widens FP32 / BF16 values on the integer
// pipes, and keeps reductions to one add per row-group lane.
// Matrix values, indices and row pointers are read once, through the
// non-allocating read-only path with an L2 evict-first policy; x is gathered
// through L1 so that it owns L2.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "df.cuh"
#include "csr_block.cuh"
#include "kernels.hpp"

namespace tbsla_gpu {

namespace {

using namespace csr;

// y = A x; add: y += A x, a row without entries not touched.
struct EpiStore {
  double* y;
  int add;
  __device__ __forceinline__ void emit(int row, double s, double*) const {
    if (!add) y[row] = s;
    else if (s != 0.0) y[row] = add_rn(y[row], s);
  }
};

template <class V, int ITEMS>
__global__ void __launch_bounds__(NT) k_csr_spmv(CsrArgs a, const double* x, double* y, int add) {
  extern __shared__ __align__(16) unsigned char stage[];
  __shared__ Smem sm;
  wait_for_earlier();
  const uint64_t pol = policy_evict_first();
  EpiStore epi{y, add};
  csr_block<V, ITEMS, EpiStore, true>(a, blockIdx.x, x, epi, nullptr, stage, sm, pol);
}

template <class V, int ITEMS>
__global__ void __launch_bounds__(NT) k_csr_pagerank(CsrArgs a, const double* __restrict__ x,
                                                    double* __restrict__ y, PageRankArgs p,
                                                    Ctl ctl) {
  extern __shared__ __align__(16) unsigned char stage[];
  __shared__ Smem sm;
  if (*(volatile int*)p.done) return;  // converged in an earlier launch: no-op
  const uint64_t pol = policy_evict_first();
  const double s = p.coef_in[0], t = p.coef_in[1];
  EpiPageRank epi{y, x, p.colw, p.tele, mul_rn(p.beta, s), s, t, t / p.n_nodes};
  double red[3] = {0, 0, 0};
  for (int b = next_block(ctl, sm); b < a.nblocks; b = next_block(ctl, sm))
    csr_block<V, ITEMS>(a, b, x, epi, red, stage, sm, pol);
  reduce_and_finish<3>(ctl, red, sm, PageRankFinish::of(p));
}

// PageRank epilogue over a separately computed t = A x: the EpiPageRank
// step of every row (grid-stride, fixed grid, so the reduction order is
// fixed), then the deterministic CTA reduction and the next coefficients.
__global__ void __launch_bounds__(NT) k_pagerank_epilogue(const double* __restrict__ t,
                                                         const double* __restrict__ x, double* __restrict__ y,
                                                         long n, PageRankArgs p, Ctl ctl) {
  __shared__ Smem sm;
  if (*(volatile int*)p.done) return;
  const double s = p.coef_in[0], tw = p.coef_in[1];
  EpiPageRank epi{y, x, p.colw, p.tele, mul_rn(p.beta, s), s, tw, tw / p.n_nodes};
  double red[3] = {0, 0, 0};
  for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT)
    epi.emit((int)i, t[i], red);
  reduce_and_finish<3>(ctl, red, sm, PageRankFinish::of(p));
}

// The end of a batched PageRank step: per-column CTA sums over warps (in
// warp order), per-CTA partials, and the last CTA's sums in CTA order
// (deterministic), coefficients of the next step and the done flag.
__device__ __forceinline__ void batched_finish(double err, double sum, double dsum, int nvec,
                                               double (*s_red)[3 * kWarp], Smem& sm, const PageRankArgs& p,
                                               Ctl ctl) {
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  s_red[warp][lane] = err;
  s_red[warp][kWarp + lane] = sum;
  s_red[warp][2 * kWarp + lane] = dsum;
  __syncthreads();
  if (threadIdx.x < 3 * kWarp) {
    double acc = 0;
    for (int w = 0; w < NT / kWarp; w++) acc = add_rn(acc, s_red[w][threadIdx.x]);
    ctl.partials[(size_t)blockIdx.x * 3 * kWarp + threadIdx.x] = acc;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = atomicAdd(ctl.counter + 1, 1u);
    sm.flag = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!sm.flag) return;
  __threadfence();
  // warp w adds the partials of CTAs w, w + 8, ... (coalesced over the
  // columns), then the eight sums are added in warp order; one thread per
  // column finishes it
  double acc[3] = {0, 0, 0};
#pragma unroll 4
  for (int i = warp; i < (int)gridDim.x; i += NT / kWarp) {
    const double* q = ctl.partials + (size_t)i * 3 * kWarp + lane;
#pragma unroll
    for (int k = 0; k < 3; k++) acc[k] = add_rn(acc[k], __ldcg(q + k * kWarp));
  }
#pragma unroll
  for (int k = 0; k < 3; k++) s_red[warp][k * kWarp + lane] = acc[k];
  __syncthreads();
  if (warp == 0) {
    double v[3] = {0, 0, 0};
    for (int w = 0; w < NT / kWarp; w++)
      for (int k = 0; k < 3; k++) v[k] = add_rn(v[k], s_red[w][k * kWarp + lane]);
    bool ok = true;
    if (lane < nvec) {
      ctl.result[lane] = v[0];
      ctl.result[nvec + lane] = v[1];
      ctl.result[2 * nvec + lane] = v[2];
      const double s1 = 1.0 / v[1];
      p.coef_out[lane] = s1;
      p.coef_out[kWarp + lane] = teleport_weight(p.beta, s1, v[2]);
      ok = v[0] < p.eps;
    }
    const bool all = __all_sync(0xffffffffu, ok);
    if (lane == 0) {
      *p.iters += 1;
      if (all) *p.done = 1;
      ctl.counter[0] = 0;
      ctl.counter[1] = 0;
    }
    __threadfence();
  }
}


__device__ __forceinline__ DF df_ld(const float2* p) {
  const float2 v = *p;
  return {v.x, v.y};
}
__device__ __forceinline__ float as_f32(float v) { return v; }
__device__ __forceinline__ float as_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

// The batched step in double-float, for FP32 / BF16 values (exact in one
// float): X, Y, T and the column sums w are stored as float pairs; each
// lane sums its row's products a_ij X[j, k] in entry order as a compensated
// dot product (Dot2: about twice FP32 precision), and the epilogue forms the
// single-vector epilogue's quantities (y = beta s acc + t T, |y - x s|, y,
// w y) in the same arithmetic: the difference y - x s, which cancels as the
// iteration converges, with the full double-float addition, the sums of
// terms of one sign (y's two terms, the three running sums) with the
// same-sign one.  The CTA and grid reductions run in FP64 (batched_finish).
template <class V, int GB>
__global__ void __launch_bounds__(NT) k_csr_pagerank_batched_df(CsrArgs a, int nvec, const float2* __restrict__ X,
                                                               float2* __restrict__ Y, const float2* __restrict__ T,
                                                               const float2* __restrict__ W, PageRankArgs p,
                                                               Ctl ctl) {
  __shared__ Smem sm;
  __shared__ double s_red[NT / kWarp][3 * kWarp];
  __shared__ double s_long[NT / kWarp][kWarp];
  if (*(volatile int*)p.done) return;
  const uint64_t pol = policy_evict_first();
  const V* vals = static_cast<const V*>(a.vals);
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const bool active = lane < nvec;
  const double scd = active ? p.coef_in[lane] : 0.0;
  const DF sc = df_of(scd), tc = df_of(active ? p.coef_in[kWarp + lane] : 0.0), bsc = df_of(mul_rn(p.beta, scd));
  DF err{0.f, 0.f}, sum{0.f, 0.f}, dsum{0.f, 0.f};
  // the row's value a (this lane's column) through the epilogue
  auto emit = [&](int row, DF acc) {
    const size_t o = (size_t)row * nvec + lane;
    const DF yn = df_add_same_sign(df_mul(bsc, acc), df_mul(tc, df_ld(T + o)));
    DF dx = df_add(yn, df_neg(df_mul(df_ld(X + o), sc)));
    if (dx.h < 0) dx = df_neg(dx);
    err = df_add_same_sign(err, dx);
    sum = df_add_same_sign(sum, yn);
    dsum = df_add_same_sign(dsum, df_mul(df_ld(W + row), yn));
    Y[o] = make_float2(yn.h, yn.l);
  };
  // adds the products of 32 entries (fewer at the end) to (as, ac)
  auto chunk = [&](int base, int e, float& as, float& ac) {
    const int j = base + lane;
    int c = 0;
    float v = 0.f;
    if (j < e) {
      c = ld_stream(a.colidx + j, pol);
      v = as_f32(ld_stream(vals + j, pol));
    }
    const int m = min(kWarp, e - base);
    // GB entries' gathers of X in flight (8 or 16, a tuning choice),
    // then their products added in entry order; a short tail runs as a
    // masked batch (a dead slot adds 0 * 0, which leaves s and c as they
    // are), so a row of a few entries waits for one gather latency, not
    // one per entry
    for (int t = 0; t < m; t += GB) {
      DF xv[GB];
      float vv[GB];
#pragma unroll
      for (int u = 0; u < GB; u++) {
        const bool live = t + u < m;
        const int ct = __shfl_sync(0xffffffffu, c, (t + u) & (kWarp - 1));
        const float vu = __shfl_sync(0xffffffffu, v, (t + u) & (kWarp - 1));
        vv[u] = live ? vu : 0.f;
        xv[u] = (active && live) ? df_ld(X + (size_t)(ct - a.f_col) * nvec + lane) : DF{0.f, 0.f};
      }
#pragma unroll
      for (int u = 0; u < GB; u++) dot2_step(as, ac, vv[u], xv[u]);
    }
  };
  for (int b = next_block(ctl, sm); b < a.nblocks; b = next_block(ctl, sm)) {
    const int r0 = a.blocks[b], r1 = a.blocks[b + 1];
    if (r1 - r0 == 1) {
      // a long row (more entries than a block holds): the CTA's warps take
      // a run of chunks each, every chunk summed from zero and added in
      // FP64, since the rounding of the carried errors grows with the
      // entries summed (20,000 entries in one Dot2 sum: 1e-11 of the row's
      // value), then warp 0 adds the runs in order
      const int s = a.rowptr[r0], e = a.rowptr[r0 + 1];
      const int run = (((e - s + kWarp - 1) / kWarp + NT / kWarp - 1) / (NT / kWarp)) * kWarp;
      double part = 0;
      const int lo = s + warp * run, hi = min(e, lo + run);
      for (int base = lo; base < hi; base += kWarp) {
        float as = 0.f, ac = 0.f;
        chunk(base, hi, as, ac);
        part = add_rn(part, df_val(fast_two_sum(as, ac)));
      }
      s_long[warp][lane] = part;
      __syncthreads();
      if (warp == 0 && active) {
        double acc = 0;
        for (int w = 0; w < NT / kWarp; w++) acc = add_rn(acc, s_long[w][lane]);
        emit(r0, df_of(acc));
      }
      continue;  // next_block's barrier keeps s_long until warp 0 has read it
    }
    for (int row = r0 + warp; row < r1; row += NT / kWarp) {
      const int s = a.rowptr[row], e = a.rowptr[row + 1];
      float as = 0.f, ac = 0.f;  // compensated sum of the row's products
      for (int base = s; base < e; base += kWarp) chunk(base, e, as, ac);
      if (active) emit(row, fast_two_sum(as, ac));
    }
  }
  batched_finish(df_val(err), df_val(sum), df_val(dsum), nvec, s_red, sm, p, ctl);
}

// Arithmetic of the entry-stream form: elements of X / Y / T / W, a value of
// A, a row's running sum, and the terms of the norms.
// Double-float, for FP32 / BF16 values: the steps of the form above.
struct StreamDF {
  using Elem = float2;
  using Val = float;
  struct Ent {
    int off;
    float v;
  };
  struct Sum {
    float s = 0.f, c = 0.f;
  };
  DF sc, tc, bsc;
  DF err{0.f, 0.f}, sum{0.f, 0.f}, dsum{0.f, 0.f};
  __device__ __forceinline__ void init(double scale, double tele, double beta) {
    sc = df_of(scale);
    tc = df_of(tele);
    bsc = df_of(mul_rn(beta, scale));
  }
  template <class V>
  static __device__ __forceinline__ float value(V v) { return as_f32(v); }
  static __device__ __forceinline__ Elem zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ void step(Sum& a, float v, float2 x) { dot2_step(a.s, a.c, v, DF{x.x, x.y}); }
  static __device__ __forceinline__ Elem pack(const Sum& a) {
    const DF t = fast_two_sum(a.s, a.c);
    return make_float2(t.h, t.l);
  }
  // a piece's sum, and the element of a total of such sums
  static __device__ __forceinline__ double wide(const Sum& a) { return df_val(fast_two_sum(a.s, a.c)); }
  static __device__ __forceinline__ Elem narrow(double v) {
    const DF t = df_of(v);
    return make_float2(t.h, t.l);
  }
  __device__ __forceinline__ Elem row(Elem a, Elem t, Elem x, Elem w) {
    const DF yn = df_add_same_sign(df_mul(bsc, DF{a.x, a.y}), df_mul(tc, DF{t.x, t.y}));
    DF dx = df_add(yn, df_neg(df_mul(DF{x.x, x.y}, sc)));
    if (dx.h < 0) dx = df_neg(dx);
    err = df_add_same_sign(err, dx);
    sum = df_add_same_sign(sum, yn);
    dsum = df_add_same_sign(dsum, df_mul(DF{w.x, w.y}, yn));
    return make_float2(yn.h, yn.l);
  }
  __device__ __forceinline__ double e() const { return df_val(err); }
  __device__ __forceinline__ double m() const { return df_val(sum); }
  __device__ __forceinline__ double d() const { return df_val(dsum); }
};
// FP64, for FP64 values: one multiply-add per entry and the single-vector
// epilogue's operations (EpiPageRank), per column.
struct StreamF64 {
  using Elem = double;
  using Val = double;
  struct Ent {
    long off;
    double v;
  };
  struct Sum {
    double s = 0;
  };
  double sc, tc, bsc;
  double err = 0, sum = 0, dsum = 0;
  __device__ __forceinline__ void init(double scale, double tele, double beta) {
    sc = scale;
    tc = tele;
    bsc = mul_rn(beta, scale);
  }
  static __device__ __forceinline__ double value(double v) { return v; }
  static __device__ __forceinline__ Elem zero() { return 0.0; }
  static __device__ __forceinline__ void step(Sum& a, double v, double x) { a.s = fma_rn(v, x, a.s); }
  static __device__ __forceinline__ Elem pack(const Sum& a) { return a.s; }
  static __device__ __forceinline__ double wide(const Sum& a) { return a.s; }
  static __device__ __forceinline__ Elem narrow(double v) { return v; }
  __device__ __forceinline__ Elem row(Elem a, Elem t, Elem x, Elem w) {
    const double yn = fma_rn(bsc, a, mul_rn(tc, t));
    err = add_rn(err, fabs(fma_rn(-x, sc, yn)));
    sum = add_rn(sum, yn);
    dsum = fma_rn(w, yn, dsum);
    return yn;
  }
  __device__ __forceinline__ double e() const { return err; }
  __device__ __forceinline__ double m() const { return sum; }
  __device__ __forceinline__ double d() const { return dsum; }
};

// The same step in an entry-stream form: each warp claims items of the plan
// (runs of rows of about equal work) and walks an item's entries as one
// stream, GB X-row gathers in flight whatever the row boundaries, finishing
// each row (the same epilogue) where its last entry is added.  Each row's
// products are added in entry order with the same steps, so Y is the same
// bit for bit as with a warp per row, cut rows apart (below), and the order in
// which rows enter the norms' partial sums differs.  Rows of a few entries (most rows of a
// power-law graph) then share one gather latency instead of paying one each,
// and a row's epilogue operands (T, X, w) are loaded when the previous row
// finishes.
//
// A row longer than an item is cut into pieces, an item each and the first
// ones claimed: one warp walking a hub row was the critical path of the step
// (2^20 nodes, 14.8 M entries, the longest row 35,187, 32 vectors, FP32 values:
// 3.95 -> 0.72 ms a step; FP64 values 6.2 -> 1.4 ms).  The warp that finishes a
// row's last piece adds the pieces' sums in entry order, in FP64, and runs the
// row's epilogue.
//
// The kernel is bound by instruction issue and by how many warps hide the
// gathers (FP64 values: by the FP64 pipe), so the per-entry work is kept
// small: each lane turns its entry of a 32-entry chunk into (X row offset,
// value) once and leaves it in shared memory, where every lane reads it back
// with one broadcast load (in double-float the offset is 32-bit: the host
// takes this form only when n_col * nvec < 2^31); a batch of GB whole entries
// that no row ends inside runs without the per-entry row-end test; and the
// register cap keeps four CTAs (32 warps) on an SM for GB = 8 in double-float
// (three in FP64, two for GB = 16).
template <class V, int GB, class AR>
__global__ void __launch_bounds__(NT, GB > 8 ? 2 : sizeof(V) == 8 ? 3 : 4)
    k_csr_pagerank_batched_stream(CsrArgs a, BatchPlan plan, int nvec, const typename AR::Elem* __restrict__ X,
                                  typename AR::Elem* __restrict__ Y, const typename AR::Elem* __restrict__ T,
                                  const typename AR::Elem* __restrict__ W, PageRankArgs p, Ctl ctl) {
  using Elem = typename AR::Elem;
  using Val = typename AR::Val;
  using Ent = typename AR::Ent;
  __shared__ Smem sm;
  __shared__ double s_red[NT / kWarp][3 * kWarp];
  __shared__ Ent s_ent[NT / kWarp][kWarp];     // per warp: its chunk's (X row offset, value)
  __shared__ double s_piece[NT / kWarp][kWarp];  // a piece's running sums
  if (*(volatile int*)p.done) return;
  constexpr unsigned full = 0xffffffffu;
  const uint64_t pol = policy_evict_first();
  const V* vals = static_cast<const V*>(a.vals);
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const bool active = lane < nvec;
  const Elem* __restrict__ Xl = X + lane;
  Ent* const ent = s_ent[warp];
  AR ar;
  ar.init(active ? p.coef_in[lane] : 0.0, active ? p.coef_in[kWarp + lane] : 0.0, p.beta);
  int b = 0;
  if (lane == 0) b = (int)atomicAdd(ctl.counter, 1u);
  b = __shfl_sync(full, b, 0);
  while (b < plan.nitems) {
    int nb = 0;  // the next item, claimed under this one
    if (lane == 0) nb = (int)atomicAdd(ctl.counter, 1u);
    const int4 item = __ldg(plan.item + b);
    const int r0 = item.x, r1 = item.y, s0 = item.z, e0 = item.w;
    const bool piece = b < plan.npieces;
    // ends of rows [rw, rw + 32): lane k holds rowptr[rw + k + 1]
    int rw = r0;
    int rpw = rw + 1 + lane <= r1 ? a.rowptr[rw + 1 + lane] : 0;
    int row = r0;
    int row_end = piece ? 0x7fffffff : __shfl_sync(full, rpw, 0);
    Elem tn = AR::zero(), xn = AR::zero(), wn;
    auto load_ops = [&](int r) {
      if (active) {
        const size_t o = (size_t)r * nvec + lane;
        tn = T[o];
        xn = X[o];
      }
      wn = W[r];
    };
    load_ops(row);
    typename AR::Sum acc;
    if (piece) s_piece[warp][lane] = 0;
    // the epilogue of `row`, then the next row's end and operands
    auto finish = [&]() {
      if (active) Y[(size_t)row * nvec + lane] = ar.row(AR::pack(acc), tn, xn, wn);
      acc = typename AR::Sum{};
      row++;
      if (row < r1) {
        if (row - rw >= kWarp) {
          rw += kWarp;
          rpw = rw + 1 + lane <= r1 ? a.rowptr[rw + 1 + lane] : 0;
        }
        row_end = __shfl_sync(full, rpw, row - rw);
        load_ops(row);
      }
    };
    for (int base = s0; base < e0; base += kWarp) {
      const int j = base + lane;
      Ent en{};
      if (j < e0) {
        en.off = (ld_stream(a.colidx + j, pol) - a.f_col) * (decltype(en.off))nvec;
        en.v = AR::value(ld_stream(vals + j, pol));
      }
      __syncwarp();
      ent[lane] = en;
      __syncwarp();
      const int m = min(kWarp, e0 - base);
      int t = 0;
      for (; t + GB <= m; t += GB) {
        Elem xv[GB];
        Val vv[GB];
#pragma unroll
        for (int u = 0; u < GB; u++) {
          const Ent ev = ent[t + u];
          vv[u] = ev.v;
          xv[u] = active ? Xl[ev.off] : AR::zero();
        }
        if (base + t + GB <= row_end) {  // no row ends inside the batch
#pragma unroll
          for (int u = 0; u < GB; u++) AR::step(acc, vv[u], xv[u]);
        } else {
#pragma unroll
          for (int u = 0; u < GB; u++) {
            while (base + t + u >= row_end) finish();  // rows ending before this entry (empty ones too)
            AR::step(acc, vv[u], xv[u]);
          }
        }
      }
      if (t < m) {  // the item's last, partial batch (its dead slots neither load nor add)
        Elem xv[GB];
        Val vv[GB];
#pragma unroll
        for (int u = 0; u < GB; u++) {
          const bool live = t + u < m;
          const Ent ev = ent[(t + u) & (kWarp - 1)];
          vv[u] = live ? ev.v : (Val)0;
          xv[u] = (active && live) ? Xl[ev.off] : AR::zero();
        }
#pragma unroll
        for (int u = 0; u < GB; u++) {
          if (t + u < m) {
            while (base + t + u >= row_end) finish();
            AR::step(acc, vv[u], xv[u]);
          }
        }
      }
      if (piece) {  // every chunk summed from zero, as in a long row of the form above
        s_piece[warp][lane] = add_rn(s_piece[warp][lane], AR::wide(acc));
        acc = typename AR::Sum{};
      }
    }
    if (piece) {
      const int c = __ldg(plan.piece_cut + b);
      const int first = __ldg(plan.cut_first + c), n = __ldg(plan.cut_first + c + 1) - first;
      double* ps = plan.piece_sum;
      if (active) ps[(size_t)b * kWarp + lane] = s_piece[warp][lane];
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(plan.cut_done + c, 1u) == (unsigned)n - 1;
      if (__shfl_sync(full, last, 0)) {
        __threadfence();
        if (active) {
          double tot = 0;
#pragma unroll 4
          for (int k = 0; k < n; k++) tot = add_rn(tot, __ldcg(ps + (size_t)(first + k) * kWarp + lane));
          Y[(size_t)row * nvec + lane] = ar.row(AR::narrow(tot), tn, xn, wn);
        }
        if (lane == 0) plan.cut_done[c] = 0;  // for the next launch
      }
    } else {
      while (row < r1) finish();  // the last row with entries and the empty rows after it
    }
    b = __shfl_sync(full, nb, 0);
  }
  batched_finish(ar.e(), ar.m(), ar.d(), nvec, s_red, sm, p, ctl);
}

__global__ void k_f64_to_df(const double* src, float2* dst, long n) {  // may run in place
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const DF v = df_of(src[i]);
    dst[i] = make_float2(v.h, v.l);
  }
}

__global__ void k_df_to_f64(const float2* src, double* dst, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float2 v = src[i];
    dst[i] = (double)v.x + (double)v.y;
  }
}

template <class V, int ITEMS>
cudaError_t launch_spmv(const CsrArgs& a, const double* x, double* y, bool add, cudaStream_t s) {
  constexpr size_t smem = stage_bytes<V, ITEMS>();
  cudaError_t ready = smem_opt_in<k_csr_spmv<V, ITEMS>>(smem);
  if (ready != cudaSuccess) return ready;
  return launch_early(k_csr_spmv<V, ITEMS>, a.nblocks, NT, smem, s, a, x, y, add ? 1 : 0);
}

template <class V>
cudaError_t spmv_items(const CsrArgs& a, const double* x, double* y, bool add, cudaStream_t s) {
  switch (a.items) {
    case 4: return launch_spmv<V, 4>(a, x, y, add, s);
    case 8: return launch_spmv<V, 8>(a, x, y, add, s);
    case 16: return launch_spmv<V, 16>(a, x, y, add, s);
  }
  return cudaErrorInvalidValue;
}

template <class V, int ITEMS>
cudaError_t launch_pr(const CsrArgs& a, const double* x, double* y, const PageRankArgs& p, Ctl c,
                      int grid, cudaStream_t s) {
  constexpr size_t smem = stage_bytes<V, ITEMS>();
  cudaError_t ready = smem_opt_in<k_csr_pagerank<V, ITEMS>>(smem);
  if (ready != cudaSuccess) return ready;
  k_csr_pagerank<V, ITEMS><<<grid, NT, smem, s>>>(a, x, y, p, c);
  return cudaGetLastError();
}

template <class V>
cudaError_t pr_items(const CsrArgs& a, const double* x, double* y, const PageRankArgs& p, Ctl c,
                     int grid, cudaStream_t s) {
  switch (a.items) {
    case 4: return launch_pr<V, 4>(a, x, y, p, c, grid, s);
    case 8: return launch_pr<V, 8>(a, x, y, p, c, grid, s);
    case 16: return launch_pr<V, 16>(a, x, y, p, c, grid, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

void csr_partition(const int* rowptr, int n_row, int tile, int max_steps, int** out, int* nblocks) {
  std::vector<int> b;
  b.reserve((size_t)n_row / 64 + 16);
  b.push_back(0);
  int r = 0;
  while (r < n_row) {
    const long len = (long)rowptr[r + 1] - rowptr[r];
    if (len > tile) {
      r++;
      b.push_back(r);
      continue;
    }
    const int start = r;
    const long base = rowptr[r];
    while (r < n_row && r - start < NT && (long)rowptr[r + 1] - base <= tile) r++;
    if (max_steps > 0 && r - start > 1) {
      const long most = (long)max_steps * csr::row_lanes(r - start);
      int q = start;
      while (q < r && (long)rowptr[q + 1] - rowptr[q] <= most) q++;
      r = q == start ? start + 1 : q;  // (fewer rows: more lanes each, so those before q stay within it)
    }
    b.push_back(r);
  }
  *nblocks = (int)b.size() - 1;
  *out = new int[b.size()];
  std::copy(b.begin(), b.end(), *out);
}

namespace {
template <auto Kernel>
int resident_grid(size_t smem = 0) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (smem) smem_opt_in<Kernel>(smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, Kernel, NT, smem);
  return std::max(1, sms * std::max(1, per));
}
}  // namespace

int csr_pagerank_grid(int items, int prec) {
  switch (prec * 100 + items) {
    case kF64 * 100 + 4: return resident_grid<k_csr_pagerank<double, 4>>(stage_bytes<double, 4>());
    case kF64 * 100 + 8: return resident_grid<k_csr_pagerank<double, 8>>(stage_bytes<double, 8>());
    case kF64 * 100 + 16: return resident_grid<k_csr_pagerank<double, 16>>(stage_bytes<double, 16>());
    case kF32 * 100 + 4: return resident_grid<k_csr_pagerank<float, 4>>(stage_bytes<float, 4>());
    case kF32 * 100 + 8: return resident_grid<k_csr_pagerank<float, 8>>(stage_bytes<float, 8>());
    case kF32 * 100 + 16: return resident_grid<k_csr_pagerank<float, 16>>(stage_bytes<float, 16>());
    case kBF16 * 100 + 4: return resident_grid<k_csr_pagerank<__nv_bfloat16, 4>>(stage_bytes<__nv_bfloat16, 4>());
    case kBF16 * 100 + 8: return resident_grid<k_csr_pagerank<__nv_bfloat16, 8>>(stage_bytes<__nv_bfloat16, 8>());
    case kBF16 * 100 + 16: return resident_grid<k_csr_pagerank<__nv_bfloat16, 16>>(stage_bytes<__nv_bfloat16, 16>());
  }
  return 152;
}

namespace {
template <class V, int GB>
using StreamOf = std::conditional_t<sizeof(V) == 8, StreamF64, StreamDF>;

// f(kernel) for the batched PageRank kernel of (precision, gathers in flight, form)
template <class F>
auto with_batched(int prec, int gather, int stream, F f) {
  const bool wide = gather == 16;
  if (prec == kF64) return f.template stream<double, 8>();
  if (prec == kF32) {
    if (stream) return wide ? f.template stream<float, 16>() : f.template stream<float, 8>();
    return wide ? f.template rows<float, 16>() : f.template rows<float, 8>();
  }
  if (stream) return wide ? f.template stream<__nv_bfloat16, 16>() : f.template stream<__nv_bfloat16, 8>();
  return wide ? f.template rows<__nv_bfloat16, 16>() : f.template rows<__nv_bfloat16, 8>();
}

struct BatchedGrid {
  template <class V, int GB>
  int stream() { return resident_grid<k_csr_pagerank_batched_stream<V, GB, StreamOf<V, GB>>>(); }
  template <class V, int GB>
  int rows() { return resident_grid<k_csr_pagerank_batched_df<V, GB>>(); }
};

struct BatchedStep {
  const CsrArgs& a;
  const BatchPlan& plan;
  int nvec;
  const void *X, *T, *W;
  void* Y;
  const PageRankArgs& p;
  Ctl ctl;
  int grid;
  cudaStream_t s;
  template <class V, int GB>
  cudaError_t stream() {
    using AR = StreamOf<V, GB>;
    using E = typename AR::Elem;
    const int g = std::max(1, std::min(grid, (plan.nitems + NT / kWarp - 1) / (NT / kWarp)));
    k_csr_pagerank_batched_stream<V, GB, AR>
        <<<g, NT, 0, s>>>(a, plan, nvec, static_cast<const E*>(X), static_cast<E*>(Y), static_cast<const E*>(T),
                          static_cast<const E*>(W), p, ctl);
    return cudaGetLastError();
  }
  template <class V, int GB>
  cudaError_t rows() {
    k_csr_pagerank_batched_df<V, GB>
        <<<grid, NT, 0, s>>>(a, nvec, static_cast<const float2*>(X), static_cast<float2*>(Y),
                             static_cast<const float2*>(T), static_cast<const float2*>(W), p, ctl);
    return cudaGetLastError();
  }
};
}  // namespace

int csr_pagerank_batched_grid(int prec, int gather, int stream) {
  return with_batched(prec, gather, stream, BatchedGrid{});
}

cudaError_t csr_pagerank_batched_step(const CsrArgs& a, const BatchPlan& plan, int nvec, const void* X, void* Y,
                                      const void* T, const void* W, const PageRankArgs& p, Ctl ctl, int grid,
                                      int gather, int stream, cudaStream_t s) {
  if (nvec < 1 || nvec > kWarp) return cudaErrorInvalidValue;
  return with_batched(a.prec, gather, stream, BatchedStep{a, plan, nvec, X, T, W, Y, p, ctl, grid, s});
}

int batch_plan_budget(long nnz, int n, int warps) {
  return (int)std::max(64L, std::min(1024L, (nnz + 4L * n) / (6L * std::max(warps, 1))));
}

void batch_plan_build(const int* rowptr, int n, int budget, std::vector<int4>* items, std::vector<int>* piece_cut,
                      std::vector<int>* cut_first) {
  items->clear();
  piece_cut->clear();
  cut_first->clear();
  for (int i = 0; i < n; i++) {
    const long len = (long)rowptr[i + 1] - rowptr[i];
    if (len <= budget) continue;
    const long np = (len + budget - 1) / budget, size = ((len + np - 1) / np + kWarp - 1) / kWarp * kWarp;
    cut_first->push_back((int)piece_cut->size());
    for (long at = 0; at < len; at += size) {
      piece_cut->push_back((int)cut_first->size() - 1);
      items->push_back(make_int4(i, i + 1, (int)(rowptr[i] + at), (int)(rowptr[i] + std::min(len, at + size))));
    }
  }
  cut_first->push_back((int)piece_cut->size());
  int r = 0;
  while (r < n) {
    const int start = r;
    long cost = 0;
    while (r < n) {
      const long len = (long)rowptr[r + 1] - rowptr[r];
      if (len > budget || (r > start && cost + len + 4 > budget)) break;
      cost += len + 4;
      r++;
    }
    if (r > start) items->push_back(make_int4(start, r, rowptr[start], rowptr[r]));
    if (r < n && (long)rowptr[r + 1] - rowptr[r] > budget) r++;  // a cut row
  }
}

cudaError_t f64_to_df(const double* src, void* dst, long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_f64_to_df<<<(int)std::min<long>((n + 255) / 256, 152L * 16), 256, 0, s>>>(src, static_cast<float2*>(dst), n);
  return cudaGetLastError();
}

cudaError_t df_to_f64(const void* src, double* dst, long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_df_to_f64<<<(int)std::min<long>((n + 255) / 256, 152L * 16), 256, 0, s>>>(static_cast<const float2*>(src), dst,
                                                                           n);
  return cudaGetLastError();
}

cudaError_t csr_spmv(const CsrArgs& a, const double* x, double* y, bool add, cudaStream_t s) {
  if (a.nblocks == 0) return cudaSuccess;
  switch (a.prec) {
    case kF64: return spmv_items<double>(a, x, y, add, s);
    case kF32: return spmv_items<float>(a, x, y, add, s);
    case kBF16: return spmv_items<__nv_bfloat16>(a, x, y, add, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t csr_pagerank_step(const CsrArgs& a, const double* x, double* y,
                              const PageRankArgs& p, Ctl ctl, int grid, cudaStream_t s) {
  switch (a.prec) {
    case kF64: return pr_items<double>(a, x, y, p, ctl, grid, s);
    case kF32: return pr_items<float>(a, x, y, p, ctl, grid, s);
    case kBF16: return pr_items<__nv_bfloat16>(a, x, y, p, ctl, grid, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t pagerank_epilogue(const double* t, const double* x, double* y, long n, const PageRankArgs& p,
                              Ctl ctl, int grid, cudaStream_t s) {
  k_pagerank_epilogue<<<grid, NT, 0, s>>>(t, x, y, n, p, ctl);
  return cudaGetLastError();
}

}  // namespace tbsla_gpu
