// Device helpers shared by the kernels: tile ranges, block reductions, the
// last-tile ticket, index arithmetic for one- and two-qubit gates, and the
// per-step gate selection.
#pragma once

#include "internal.h"
#include "launch.cuh"
#include "small_linalg.h"

__device__ __forceinline__ void tile_range(int64_t total, int idx, int nt, int64_t* lo, int64_t* hi) {
  int64_t per = (total + nt - 1) / nt;
  int64_t a = per * idx;
  int64_t b = a + per;
  if (a > total) a = total;
  if (b > total) b = total;
  *lo = a;
  *hi = b;
}

// Sum K doubles over the block; result valid in thread 0 (vals of thread 0).
template <int K>
__device__ __forceinline__ void block_sum(double (&vals)[K]) {
  __shared__ double red[BLOCK_THREADS / 32][K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double v = vals[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    vals[k] = v;
  }
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) red[warp][k] = vals[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double v = 0.0;
      for (int w = 0; w < BLOCK_THREADS / 32; ++w) v += red[w][k];
      vals[k] = v;
    }
  }
  __syncthreads();
}

#define WARPS WARPS_PER_BLOCK
static_assert(WARPS_PER_BLOCK * 32 == BLOCK_THREADS, "per-warp partials assume BLOCK_THREADS / 32 warps");

// Thread 0 publishes its partial (already written) and takes a ticket.
// Returns true in every thread of the block that finishes state b last.
__device__ __forceinline__ bool last_tile_ticket(int* ticket, int b, int nt) {
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    __threadfence();
    int t = atomicAdd(&ticket[b], 1);
    s_last = (t == nt - 1);
  }
  __syncthreads();
  bool last = s_last != 0;
  if (last) __threadfence();
  return last;
}

// Index of amplitude for quad r on bits (hi, lo = hi - 1), with values (bh, bl).
__device__ __forceinline__ int64_t quad_base(int64_t r, int lo) {
  return ((r >> lo) << (lo + 2)) | (r & ((((int64_t)1) << lo) - 1));
}
__device__ __forceinline__ int64_t pair_base(int64_t r, int bit) {
  return ((r >> bit) << (bit + 1)) | (r & ((((int64_t)1) << bit) - 1));
}

// Which gate state b applies at this step (all threads of a block agree).
__device__ __forceinline__ bool select_gate(const GateSel& sel, const BatchDev& bd, int b, int n,
                                            int64_t* slot, int* q, int* k) {
  if (sel.active && !sel.active[b]) return false;
  int l, s;
  if (sel.mode == SEL_INVERSE || sel.mode == SEL_LAYER_FWD) {
    if (sel.step >= n) return false;
    l = sel.layer;
    s = sel.mode == SEL_INVERSE ? n - 1 - sel.step : sel.step;
  } else {
    int L = sel.nlayers[b];
    if (sel.step >= L * n) return false;
    if (sel.mode == SEL_REBUILD) {
      l = L - 1 - sel.step / n;
      s = sel.step % n;
    } else {
      l = sel.step / n;
      s = n - 1 - sel.step % n;
    }
  }
  *slot = (int64_t)l * n + s;
  *q = s;
  *k = sel.arity[bd.gate_off[b] / 16 + *slot];
  if (!((*k == 1) || (*k == 2 && s <= n - 2))) {   // never index with a bad slot
    if (threadIdx.x == 0) atomicOr(bd.err, KERR_BAD_GATE);
    return false;
  }
  return true;
}

// Load an M x M gate into fp32 registers, optionally as its adjoint.  M is a
// compile-time constant so every index is static and `out` stays in
// registers.
template <int M>
__device__ __forceinline__ void load_gate_m(const double2* g, int adjoint, float2 (&out)[16]) {
#pragma unroll
  for (int r = 0; r < M; ++r)
#pragma unroll
    for (int c = 0; c < M; ++c) {
      const double2 v = adjoint ? cconj(g[c * M + r]) : g[r * M + c];
      out[r * M + c] = cf((float)v.x, (float)v.y);
    }
}

__device__ __forceinline__ void load_gate(const double2* g, int m, int adjoint, float2 (&out)[16]) {
  if (m == 4) load_gate_m<4>(g, adjoint, out);
  else load_gate_m<2>(g, adjoint, out);
}

__device__ __forceinline__ float2 fmac(float2 acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x));
  acc.y = fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y));
  return acc;
}

// Compensated accumulation of exact products (double-float): p = u v is
// split exactly into ph + pl (fma), ph enters (hi, lo) through a TwoSum and
// pl and the TwoSum error land in lo, whose own roundings grow with the run.
// A run of TT_FLUSH = 32 squares is off by 2^-47 of its sum (root mean square;
// 2^-44 the largest of 2000), 256 of them by 2^-44 (2^-42), 4096 by 2^-40, so
// runs end after TT_FLUSH rows: in FP64, or in stage (a)'s fast Gram in
// another double-float sum (16 runs 2^-47, 256 runs 2^-44).  The 1e-10 cutoff
// that the eigenvalues decide is 2^-33.
struct DF {
  float hi, lo;
};

// Every operation is an explicitly rounded intrinsic, so the compiler never
// contracts the product into the sum (which would break the error terms).
__device__ __forceinline__ void df_add_prod(DF& s, float u, float v) {
  const float ph = __fmul_rn(u, v);
  const float pl = __fmaf_rn(u, v, -ph);
  const float t = __fadd_rn(s.hi, ph);
  const float bv = __fsub_rn(t, s.hi);
  const float err = __fadd_rn(__fsub_rn(s.hi, __fsub_rn(t, bv)), __fsub_rn(ph, bv));
  s.lo = __fadd_rn(s.lo, __fadd_rn(err, pl));
  s.hi = t;
}

// rows summed in double-float before their sum is passed on
#define TT_FLUSH 32
