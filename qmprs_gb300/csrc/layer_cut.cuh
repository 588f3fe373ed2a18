// One cut of the layer stage's bond-2 truncated SVD in one launch, shared by
// the fast mode (complex64, layers.cu) and the exact mode (double-float,
// exact.cu).
//
// Step j of a state works at cut c = n - 1 - j.  A block takes a unit of
// CUT_ROWS rows of the remainder M_c (2^c x 2 r): it forms them from two rows
// each of M_{c+1} times the kept vectors of the previous cut (step 0 reads
// the working state as it is), stores them, and sums their Gram matrix; the
// state's last block diagonalises it and stores the vectors, the bond and
// the site tensor.  In the last launch, the first in which every state has
// one unit, a block does all the cuts that are left: a launch each, with its
// start and the reload of the state's tables, took as long as the cut (20
// qubits: 19 launches, now 8; a state whose tail started in an earlier launch
// would hold up the larger ones').  A separate projection read and a separate eigenvalue
// launch are gone: a cut of a 20-qubit state took 215 us (Gram 24, FP64
// Jacobi of one thread 187, projection 4.7) and takes 22 us now.
//
// The Gram's sums are exact FP32 products in double-float over a thread's
// at most 16 rows and over the warp's lanes (in three parts there for the
// exact mode, whose rows carry 48 bits), FP64 across the warps (fixed order)
// and the units; the eigensolver takes the FP64 sums.  4096 rows a unit keep the
// double-float runs short and give a 20-qubit state 128 blocks; the table
// of units is sorted by the last step that needs them, so a step's launch
// holds only blocks with work.
#pragma once

#include "warp_polar.cuh"

#define CUT_ROWS (1 << CUT_ROW_BITS)

struct CutFast {
  typedef float2 T;
  static __device__ __forceinline__ double lane_sums(DF (&s)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 16; ++k) df_shfl_add(s[k], s[k], 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < o; ++k) {
        const DF give = up ? s[k] : s[k + o];
        if (up) s[k] = s[k + o];
        df_shfl_add(s[k], give, o);
      }
    }
    return (double)s[0].hi + (double)s[0].lo;
  }
  static __device__ __forceinline__ T load_v(double2 v) { return cf((float)v.x, (float)v.y); }
  static __device__ __forceinline__ double2 to_d(T v) { return f2d(v); }
  template <int N>
  static __device__ __forceinline__ void load(const T* p, T (&x)[N]) {   // N even, 16-byte aligned
    const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const float4 v = q[i];
      x[2 * i] = cf(v.x, v.y);
      x[2 * i + 1] = cf(v.z, v.w);
    }
  }
  template <int N>
  static __device__ __forceinline__ void store(T* p, const T (&x)[N]) {
    float4* q = reinterpret_cast<float4*>(p);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) q[i] = make_float4(x[2 * i].x, x[2 * i].y, x[2 * i + 1].x, x[2 * i + 1].y);
  }
  template <int W>
  static __device__ __forceinline__ T project(const T* x, const T* vm, int col) {
    T acc = cf(0.f, 0.f);
#pragma unroll
    for (int a = 0; a < W; ++a) acc = fmac(acc, x[a], vm[a * 4 + col]);
    return acc;
  }
  static __device__ __forceinline__ void norm2(DF& s, T x) {
    df_add_prod(s, x.x, x.x);
    df_add_prod(s, x.y, x.y);
  }
  static __device__ __forceinline__ void dot(DF& re, DF& im, T x, T y) {   // conj(x) y
    df_add_prod(re, x.x, y.x);
    df_add_prod(re, x.y, y.y);
    df_add_prod(im, x.x, y.y);
    df_add_prod(im, -x.y, y.x);
  }
};

struct CutExact {
  typedef xc T;
  static __device__ __forceinline__ double lane_sums(DF (&s)[16]) {
    TF t[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      t[k] = tf_from(s[k]);
      tf_shfl_add(t[k], t[k], 16);
    }
    return tf_to_d(warp_fold_tf(t));
  }
  static __device__ __forceinline__ T load_v(double2 v) { return xc_from_d(v); }
  static __device__ __forceinline__ double2 to_d(T v) { return xc_to_d(v); }
  template <int N>
  static __device__ __forceinline__ void load(const T* p, T (&x)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = p[i];
  }
  template <int N>
  static __device__ __forceinline__ void store(T* p, const T (&x)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = x[i];
  }
  template <int W>
  static __device__ __forceinline__ T project(const T* x, const T* vm, int col) {
    XA s = xa_zero();
#pragma unroll
    for (int a = 0; a < W; ++a) xa_mac(s, vm[a * 4 + col], x[a]);
    return xa_round(s);
  }
  static __device__ __forceinline__ void norm2(DF& s, T x) {
    df_mac(s, x.x, x.z, x.x, x.z);
    df_mac(s, x.y, x.w, x.y, x.w);
  }
  static __device__ __forceinline__ void dot(DF& re, DF& im, T x, T y) {
    df_mac(re, x.x, x.z, y.x, y.z);
    df_mac(re, x.y, x.w, y.y, y.w);
    df_mac(im, x.x, x.z, y.y, y.w);
    df_mac(im, -x.y, -x.w, y.x, y.z);
  }
};

// Sums of a Gram of width 4: values 0-3 the diagonal, then real and
// imaginary part of (0,1), (0,2), (0,3), (1,2), (1,3), (2,3).
__device__ __forceinline__ int cut_pair(int a, int e) { return a == 0 ? e - 1 : a + e; }   // a < e

template <class P, int N>
__device__ __forceinline__ void cut_gram(DF (&s)[16], const typename P::T (&y)[N]) {
#pragma unroll
  for (int a = 0; a < N; ++a) {
    P::norm2(s[a], y[a]);
#pragma unroll
    for (int e = a + 1; e < N; ++e) {
      const int k = 4 + 2 * (a == 0 ? e - 1 : a + e);
      P::dot(s[k], s[k + 1], y[a], y[e]);
    }
  }
}

// Rows lo .. hi of M_c from M_{c+1} (rows of W, K kept columns).
template <class P, int W, int K>
__device__ __forceinline__ void cut_rows(const typename P::T* src, typename P::T* dst, const typename P::T* vm, int lo,
                                         int hi, DF (&s)[16]) {
  for (int row = lo + threadIdx.x; row < hi; row += BLOCK_THREADS) {
    typename P::T x[2 * W], y[2 * K];
    P::template load<2 * W>(src + (int64_t)row * 2 * W, x);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int col = 0; col < K; ++col) y[h * K + col] = P::template project<W>(x + h * W, vm, col);
    P::template store<2 * K>(dst + (int64_t)row * 2 * K, y);
    cut_gram<P, 2 * K>(s, y);
  }
}

// Eigenvectors of the Gram g (warp_gram_vectors) by one warp, in descending
// order of the eigenvalues (ties in index order): ws.B's columns, lam[0..3]
// the eigenvalues times a power of two.
__device__ __forceinline__ void warp_gram_eig(WarpPolar& ws, double2 g, double* lam) {
  const int lane = threadIdx.x & 31;
  double p[4], l[4];
  int odd;
  warp_gram_vectors(ws, g, p, &odd);
#pragma unroll
  for (int c = 0; c < 4; ++c) l[c] = p[c >= 2 && odd ? 5 - c : c];   // by original index
  // ranks by the order of the bits (the values are not negative): an FP64
  // comparison takes 64 cycles
  int rk[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    rk[a] = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const long long x = __double_as_longlong(l[b]), y = __double_as_longlong(l[a]);
      rk[a] += x > y || (x == y && b < a);
    }
    if (lane == 0) lam[rk[a]] = l[a];
  }
  double2 v = ws.B[lane & 15];
  const int pos = lane & 3, idx = pos >= 2 && odd ? 5 - pos : pos;
  __syncwarp();
  if (lane < 16) ws.B[(lane & 12) + (idx == 0 ? rk[0] : idx == 1 ? rk[1] : idx == 2 ? rk[2] : rk[3])] = v;
  __syncwarp();
}

// Make column `lane` (< keep) of the row-major 4 x 4 v's pivot entry real
// and positive (the rule of phase_fix_column).
__device__ __forceinline__ void warp_phase_fix(double2* v, int keep) {
  const int lane = threadIdx.x & 31;
  if (lane < keep) {
    double m2 = 0.0;
    double a2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a2[i] = cnorm2(v[i * 4 + lane]);
      m2 = fmax(m2, a2[i]);
    }
    const double lim = (1.0 - QM_PIVOT_TOL) * (1.0 - QM_PIVOT_TOL) * m2;
    int piv = 3;
#pragma unroll
    for (int i = 3; i >= 0; --i)
      if (a2[i] >= lim) piv = i;
    const double2 z = v[piv * 4 + lane];
    const double inv = wp_rsqrt(cnorm2(z));   // the pivot of a unit column is at least 1/2
    const double2 ph = cd(z.x * inv, -z.y * inv);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i * 4 + lane] = cmul(v[i * 4 + lane], ph);
  }
  __syncwarp();
}

template <class P>
__global__ void __launch_bounds__(BLOCK_THREADS) k_layer_cut(BatchDev bd, int step, int last, const typename P::T* work,
                                                             int* bonds, double2* vsel, double2* site_t,
                                                             double* partials, typename P::T* rem0,
                                                             typename P::T* rem1, const int* active) {
  grid_wait();
  typedef typename P::T T;
  __shared__ T vm[16];
  __shared__ double wred[WARPS][16];
  __shared__ double lam[4];
  __shared__ WarpPolar ws;
  __shared__ int s_keep;
  const int unit = blockIdx.x, b = bd.cut_state[unit], idx = bd.cut_idx[unit];
  const int n = bd.n[b];
  int c = n - 1 - step;
  if (c < 1 || (active && !active[b])) return;
  int* bond = bonds + (int64_t)b * (bd.max_n + 1);
  int r = bond[c + 1], rp = step > 0 ? bond[c + 2] : 0;
  if (r != 1 && r != 2) return;
  const int units = c > CUT_ROW_BITS ? 1 << (c - CUT_ROW_BITS) : 1;
  if (idx >= units) return;
  const int tid = threadIdx.x, lane = tid & 31;
  double2* vs = vsel + (int64_t)b * 16;
  if (step > 0 && tid < 16) vm[tid] = P::load_v(vs[tid]);
  for (;; ++step, --c) {
    const int lo = idx * CUT_ROWS, hi = min(lo + CUT_ROWS, 1 << c);
    DF s[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) s[k] = DF{0.f, 0.f};
    const T* m = work + bd.vec_off[b];   // this step's remainder (rows of 2 r)
    if (step == 0) {
      for (int row = lo + tid; row < hi; row += BLOCK_THREADS) {
        T x[2];
        P::template load<2>(m + (int64_t)row * 2, x);
        cut_gram<P, 2>(s, x);
      }
    } else {
      __syncthreads();
      // step j reads the remainder of step j - 1 and writes its own to the other buffer
      const T* src = (step == 1 ? work : (step & 1) ? rem1 : rem0) + bd.vec_off[b];
      T* o = ((step & 1) ? rem0 : rem1) + bd.vec_off[b];
      m = o;
      if (rp == 1) {
        if (r == 1) cut_rows<P, 2, 1>(src, o, vm, lo, hi, s);
        else cut_rows<P, 2, 2>(src, o, vm, lo, hi, s);
      } else {
        if (r == 1) cut_rows<P, 4, 1>(src, o, vm, lo, hi, s);
        else cut_rows<P, 4, 2>(src, o, vm, lo, hi, s);
      }
    }
    // 16 sums over the lanes (lane l holds value l mod 16), then the warps
    const double sum = P::lane_sums(s);
    if (lane < 16) wred[tid >> 5][lane] = sum;
    __syncthreads();
    double* part = partials + (int64_t)bd.state_tile0[b] * WARPS * 32;   // 16 doubles per unit
    if (tid < 16) {
      double v[WARPS];
#pragma unroll
      for (int w = 0; w < WARPS; ++w) v[w] = wred[w][tid];
      part[idx * 16 + tid] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    }
    __syncthreads();
    if (units > 1 && !last_tile_ticket(bd.ticket, b, units)) return;
    // the state's last block: Gram, eigenvectors, truncation
    {
      const int val = tid >> 4, l16 = tid & 15;
      double v = 0.0;
      for (int u = l16; u < units; u += 16) v += __ldcg(part + u * 16 + val);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o, 16);
      __syncthreads();
      if (l16 == 0) wred[0][val] = v;
    }
    __syncthreads();
    const int w = 2 * r;
    if (tid < 32) {
      double2 g = czero();
      {
        const int a = (tid >> 2) & 3, e = tid & 3;
        if (a < w && e < w) {
          if (a == e) {
            g = cd(wred[0][a], 0.0);
          } else {
            const int k = 4 + 2 * cut_pair(min(a, e), max(a, e));
            g = cd(wred[0][k], a < e ? wred[0][k + 1] : -wred[0][k + 1]);
          }
        }
      }
      warp_gram_eig(ws, g, lam);
      if (lane == 0) {
        s_keep = rank_by_cutoff(lam, w, QM_CUTOFF, 2);
        bond[c] = s_keep;
        if (units > 1) bd.ticket[b] = 0;
      }
      __syncwarp();
      const int keep = s_keep;
      warp_phase_fix(ws.B, keep);
      if (lane < 16) {
        const int a = lane >> 2, col = lane & 3;
        const double2 v = a < w && col < keep ? ws.B[lane] : czero();
        vs[lane] = v;
        vm[lane] = P::load_v(v);
        if (a < w && col < keep) site_t[((int64_t)b * bd.max_n + c) * 8 + col * w + a] = cconj(v);
      }
    }
    if (c > 1) {
      if (!last) return;
      __syncthreads();
      rp = r;
      r = s_keep;
      if (r != 1 && r != 2) return;
      continue;
    }
    // the last remainder (2 rows) for site 0
    __syncthreads();
    if (tid < 2 * s_keep) {
      const int row = tid / s_keep, col = tid % s_keep;
      const T* x = m + row * w;
      T xr[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) xr[a] = x[a < w ? a : 0];
      const T y = w == 2 ? P::template project<2>(xr, vm, col) : P::template project<4>(xr, vm, col);
      ((n & 1) ? rem1 : rem0)[bd.vec_off[b] + tid] = y;
    }
    return;
  }
}

// Site 0 from the last remainder, then the n gates of the layer.  One block
// per state: a warp per kind of site, so that its lanes run one code path:
// warp 0 the middle sites, warp 1 the first sites of blocks, warp 2 last and
// single sites; lane s takes site s.  The gates' unitarity is checked by
// all threads.  One thread per state took 43 us a site (FP64 chains).
// Measured (20 qubits, one layer): 861 us, 32 us now.
#define BUILD_THREADS 96
static_assert(MAX_QUBITS <= 32, "a lane per site");
template <class P>
__global__ void __launch_bounds__(BUILD_THREADS) k_layer_build(BatchDev bd, int layer, const typename P::T* rem0,
                                                               const typename P::T* rem1, const int* bonds,
                                                               double2* site_t, double2* gates, signed char* arity,
                                                               const int* active) {
  grid_wait();
  __shared__ double2 g_s[MAX_QUBITS][16];
  __shared__ double2 st0[4];
  __shared__ signed char ks[MAX_QUBITS];
  const int b = blockIdx.x;
  if (active && !active[b]) return;
  const int n = bd.n[b], warp = threadIdx.x >> 5, s = threadIdx.x & 31;
  const int* bond = bonds + (int64_t)b * (bd.max_n + 1);
  const double2* st = site_t + (int64_t)b * bd.max_n * 8;
  if (threadIdx.x == 0) {
    const typename P::T* rem = (((n - 2) & 1) ? rem1 : rem0) + bd.vec_off[b];
    const int r1 = bond[1];
    double nrm = 0.0;
    for (int i = 0; i < 2 * r1; ++i) nrm += cnorm2(P::to_d(rem[i]));
    const double f = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    for (int i = 0; i < 2 * r1; ++i) st0[i] = cscale(P::to_d(rem[i]), f);
  }
  __syncthreads();
  if (s < n) {
    const bool is_end = (s == n - 1) || bond[s + 1] == 1;
    const bool is_start = (s == 0) || bond[s] == 1;
    if (warp == (is_end ? 2 : is_start ? 1 : 0)) {
      const double2* d = s == 0 ? st0 : st + s * 8;
      double2 g[16];
      for (int i = 0; i < 16; ++i) g[i] = czero();
      if (warp == 2) {
        if (is_start) ran_gate_single(d, g);
        else ran_gate_last(d, g);
      } else {
        if (is_start) ran_gate_first(d, g);
        else ran_gate_middle(d, g);
      }
      for (int i = 0; i < 16; ++i) g_s[s][i] = g[i];
      ks[s] = (signed char)(is_end ? 1 : 2);
      arity[bd.gate_off[b] / 16 + (int64_t)layer * n + s] = ks[s];
    }
  }
  __syncthreads();
  // max |G G^H - I| over entries at most 1e-6 (a NaN fails)
  bool good = true;
  for (int e = threadIdx.x; e < 16 * n; e += BUILD_THREADS) {
    const double2* g = g_s[e >> 4];
    const int m = 1 << ks[e >> 4], i = (e & 15) / m, j = (e & 15) % m;
    gates[bd.gate_off[b] + (int64_t)layer * n * 16 + e] = g[e & 15];
    if (i >= m) continue;
    double2 acc = czero();
    for (int k = 0; k < m; ++k) acc = cadd(acc, cmul(g[i * m + k], cconj(g[j * m + k])));
    if (i == j) acc.x -= 1.0;
    good = good && cnorm2(acc) <= 1e-12;
  }
  if (!good) atomicOr(bd.err, KERR_NONUNITARY);
}
