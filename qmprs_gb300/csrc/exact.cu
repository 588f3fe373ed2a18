// Exact precision mode: the encoding path with double-float working states.
//
// The bond-2 truncations of the layer stage amplify a perturbation of the
// working state by about 3-5x per layer, so a complex64 working state
// (relative rounding 6e-8) drifts from an FP64 run by 1e-4..1e-3 after
// 10-15 layers (10 qubits, 15 layers; 14 qubits, 10 layers), and the
// sweeps inherit it.  GB300 issues FP64 at 1/64 of the FP32 rate with a
// 64-cycle dependent latency, so this mode keeps every large vector in
// double-float instead: each complex amplitude is a float4 (re hi, im hi,
// re lo, im lo) with value hi + lo, 16 bytes like complex128, and all
// arithmetic on the vectors is FP32 with error-free transformations:
//   products     a*b = ph + pl exactly (ph = fl(a*b), pl = fma(a, b, -ph));
//   sums         TwoSum of the high parts, low parts and the cross terms
//                a_hi*b_lo + a_lo*b_hi accumulated in FP32;
// which keeps about 2^-46 of relative precision on the FP32 pipes.  Sums
// that end in a small matrix keep what FP64 would (Grams of stage (a) and of
// the layer cuts, environments), and the small algebra ends in FP64: the
// eigenvectors of stage (a) up to width 64 come from FP32 sweeps and
// double-float products, those of a layer cut from FP32 and double-float
// one-sided sweeps, the sweep's polar factor (one warp) from the same, each
// with a first-order correction from FP64 products, or FP64 sweeps where that
// does not do; the closed-form gate construction is FP64 throughout.  The
// fast mode's polar factor is accurate to ~1e-7, which rank-deficient
// environments carry into later steps at first order.
//
// Caller-facing statevector buffers of this mode are complex128; the plan
// converts them to double-float scratch on entry and back on exit.
//
// Kernels (all deterministic: fixed-order reductions):
//   k_x_from_d / k_x_to_d / k_x_copy / k_x_zero / k_x_scale   conversions
//   k_x_dot, k_d_dot          per-state <a|b> partials (double-float / FP64)
//   k_x_gram_tile / k_x_gram_reduce   stage (a): Gram M^H M of one state's
//                             remainder, upper-triangle tiles x row splits
//   k_x_gemm                  C = A B, A double-float, B complex128 (the
//                             projection M V and the target contraction)
//   k_x_site0                 site 0 from the last remainder
//   k_layer_cut, k_layer_build, k_x_layer_fidelity   the layer stage's
//                             bond-2 cuts (layer_cut.cuh, shared with the
//                             fast mode)
//   k_x_apply_gate            one gate per state
//   k_x_sweep_step            a backward sweep step: peel the step's gate
//                             from the circuit state, reduce the gate's
//                             environment, and (last tile of the state)
//                             replace the gate by the conjugate of the
//                             environment's polar factor (one warp,
//                             warp_polar.cuh)
#include "dfloat.cuh"
#include "layer_cut.cuh"

static int grid_for(const BatchDev& bd) {
  const int cap = 152 * 8;
  return bd.ntiles < cap ? bd.ntiles : cap;
}

// ---- conversions -------------------------------------------------------------------

__global__ void k_x_from_d(BatchDev bd, const double2* src, xc* dst) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    const double2* s = src + bd.vec_off[b];
    xc* d = dst + bd.vec_off[b];
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) d[i] = xc_from_d(s[i]);
  }
}

__global__ void k_x_to_d(BatchDev bd, const xc* src, double2* dst) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    const xc* s = src + bd.vec_off[b];
    double2* d = dst + bd.vec_off[b];
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) d[i] = xc_to_d(s[i]);
  }
}

__global__ void k_x_copy(BatchDev bd, const xc* src, xc* dst, const int* active) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    if (active && !active[b]) continue;
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    const xc* s = src + bd.vec_off[b];
    xc* d = dst + bd.vec_off[b];
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) d[i] = s[i];
  }
}

__global__ void k_x_zero(BatchDev bd, xc* vec, const int* active) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    if (active && !active[b]) continue;
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    xc* v = vec + bd.vec_off[b];
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) v[i] = make_float4(i == 0 ? 1.f : 0.f, 0.f, 0.f, 0.f);
  }
}

// dst = src / sqrt(sq[b].x) in double-float (the factor split once per tile).
__global__ void k_x_scale(BatchDev bd, const xc* src, xc* dst, const double2* sq) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    const double f = sq[b].x > 0.0 ? 1.0 / sqrt(sq[b].x) : 0.0;
    const float fh = __double2float_rn(f), fl = __double2float_rn(f - (double)fh);
    const xc* s = src + bd.vec_off[b];
    xc* d = dst + bd.vec_off[b];
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      const xc x = s[i];
      DF re = {0.f, 0.f}, im = {0.f, 0.f};
      df_mac(re, x.x, x.z, fh, fl);
      df_mac(im, x.y, x.w, fh, fl);
      const float2 r = df_norm(re), m = df_norm(im);
      d[i] = make_float4(r.x, m.x, r.y, m.y);
    }
  }
}

// <a|b> per tile: double-float accumulation flushed to fp64, block sum in
// fixed order; k_reduce_tiles (dense.cu) sums the tiles of each state.
__global__ void __launch_bounds__(BLOCK_THREADS) k_x_dot(BatchDev bd, const xc* a, const xc* bv, double2* partials) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    const xc* pa = a + bd.vec_off[b];
    const xc* pb = bv + bd.vec_off[b];
    double acc[2] = {0.0, 0.0};
    int64_t i = lo + threadIdx.x;
    while (i < hi) {
      XA s = xa_zero();
      for (int f = 0; f < TT_FLUSH && i < hi; ++f, i += blockDim.x) xa_macc(s, pa[i], pb[i]);
      const double2 d = xa_to_d(s);
      acc[0] += d.x;
      acc[1] += d.y;
    }
    block_sum<2>(acc);
    if (threadIdx.x == 0) partials[tile] = cd(acc[0], acc[1]);
  }
}

// <a|b> per tile of two complex128 vectors, in FP64 (one pass; used for the
// caller-facing overlaps of this mode).
__global__ void __launch_bounds__(BLOCK_THREADS) k_d_dot(BatchDev bd, const double2* a, const double2* bv,
                                                         double2* partials) {
  grid_wait();
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    int64_t lo, hi;
    tile_range(ipow2(bd.n[b]), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    const double2* pa = a + bd.vec_off[b];
    const double2* pb = bv + bd.vec_off[b];
    double acc[2] = {0.0, 0.0};
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      const double2 p = cmulc(pa[i], pb[i]);
      acc[0] += p.x;
      acc[1] += p.y;
    }
    block_sum<2>(acc);
    if (threadIdx.x == 0) partials[tile] = cd(acc[0], acc[1]);
  }
}

// ---- stage (a): Gram, projection, contraction -----------------------------------------

// Tile geometry of a w x w Gram: tiles of TI x TI entries (TI = min(w, 32),
// w even), each thread a 2 x 2 entry block; the tiles of the upper triangle
// are numbered column block by column block.
__host__ __device__ inline int x_gram_ti(int w) { return w < 32 ? w : 32; }
__host__ __device__ inline int x_gram_nt(int w) { const int ti = x_gram_ti(w); return (w + ti - 1) / ti; }

template <class J>
struct XJobs {
  J job[X_JOBS];
  int count;
};
// The job of block `block` (uniform): the last whose first block is at most that.
template <class J>
__device__ __forceinline__ const J& x_job(const XJobs<J>& jobs, int J::*first, int block) {
  int k = 0;
  while (k + 1 < jobs.count && jobs.job[k + 1].*first <= block) ++k;
  return jobs.job[k];
}

// Partial Gram sums of one tile over one split of the rows:
// part[split * WW + a * w + c] for the tile's entries with a <= c.
// The states of a batch run side by side: one after another, every launch of
// a few dozen blocks waited on its own rows (14 states of 8-14 qubits: 145
// launches of 18.4 us, and 145 of 2 us to sum them).
__global__ void __launch_bounds__(BLOCK_THREADS) k_x_gram_tile(const __grid_constant__ XJobs<XGramJob> jobs,
                                                               int64_t WW) {
  grid_wait();
  __shared__ double2 red[BLOCK_THREADS * 4];
  const XGramJob& jb = x_job(jobs, &XGramJob::block0, blockIdx.x);
  const xc* m = jb.m;
  const int64_t rows = jb.rows;
  const int w = jb.w, nt = x_gram_nt(w), ntri = nt * (nt + 1) / 2;
  const int tile = (blockIdx.x - jb.block0) % ntri, split = (blockIdx.x - jb.block0) / ntri;
  double2* part = jb.part + (int64_t)split * WW;
  const int TI = x_gram_ti(w), G = TI / 2, EG = G * G;
  const int RL = BLOCK_THREADS / EG;
  int ti = 0, tj = 0;
  {
    int t = tile, j = 0;
    while (t > j) {
      t -= j + 1;
      ++j;
    }
    ti = t;
    tj = j;
  }
  const int e = threadIdx.x % EG, rl = threadIdx.x / EG;
  const int a0 = ti * TI + 2 * (e / G), c0 = tj * TI + 2 * (e % G);
  int64_t lo, hi;
  tile_range(rows, split, jb.nsplit, &lo, &hi);
  double2 acc[4] = {czero(), czero(), czero(), czero()};
  if (rl < RL && a0 < w && c0 < w) {
    int64_t r = lo + rl;
    while (r < hi) {
      XA s[4] = {xa_zero(), xa_zero(), xa_zero(), xa_zero()};
      for (int f = 0; f < TT_FLUSH && r < hi; ++f, r += RL) {
        const xc* x = m + r * w;
        const xc u0 = x[a0], u1 = x[a0 + 1], v0 = x[c0], v1 = x[c0 + 1];
        xa_macc(s[0], u0, v0);
        xa_macc(s[1], u0, v1);
        xa_macc(s[2], u1, v0);
        xa_macc(s[3], u1, v1);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = cadd(acc[k], xa_to_d(s[k]));
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) red[threadIdx.x * 4 + k] = acc[k];
  __syncthreads();
  for (int o = threadIdx.x; o < EG * 4; o += blockDim.x) {
    const int eo = o / 4, k = o % 4;
    double2 s = czero();
    for (int l = 0; l < RL; ++l) s = cadd(s, red[(l * EG + eo) * 4 + k]);
    const int a = ti * TI + 2 * (eo / G) + k / 2, c = tj * TI + 2 * (eo % G) + k % 2;
    if (a < w && c < w && a <= c) part[(int64_t)a * w + c] = s;
  }
}

// gram[a * w + c] = sum over splits (in order), mirrored to the lower triangle.
__global__ void __launch_bounds__(BLOCK_THREADS) k_x_gram_reduce(const __grid_constant__ XJobs<XGramJob> jobs,
                                                                 int64_t WW) {
  grid_wait();
  const XGramJob& jb = x_job(jobs, &XGramJob::rblock0, blockIdx.x);
  const int w = jb.w, nsplit = jb.nsplit;
  const double2* part = jb.part;
  double2* gram = jb.gram;
  const int64_t e = (int64_t)(blockIdx.x - jb.rblock0) * BLOCK_THREADS + threadIdx.x;
  if (e < (int64_t)w * w) {
    const int a = (int)(e / w), c = (int)(e % w);
    if (a > c) return;
    double2 s = czero();
    for (int t = 0; t < nsplit; ++t) s = cadd(s, part[(int64_t)t * WW + e]);
    if (a == c) {
      gram[e] = cd(s.x, 0.0);
    } else {
      gram[e] = s;
      gram[(int64_t)c * w + a] = cconj(s);
    }
  }
}

#define XG_KC 32   // K chunk of k_x_gemm

// C (M x N, double-float, ldc) = A (M x K, double-float, lda) * B (K x N,
// complex128, ldb), the states of a batch side by side.  Block tile: tn =
// min(N, 32) columns (a power of two) x 256 / tn rows, one output per thread;
// B is split into double-float in shared memory one K chunk at a time; sums
// flushed to fp64 per chunk.
__global__ void __launch_bounds__(BLOCK_THREADS) k_x_gemm(const __grid_constant__ XJobs<XGemmJob> jobs) {
  grid_wait();
  __shared__ xc Bs[XG_KC][32];
  const XGemmJob& jb = x_job(jobs, &XGemmJob::block0, blockIdx.x);
  const xc* A = jb.A;
  const double2* B = jb.B;
  const int64_t lda = jb.lda, ldb = jb.ldb, M = jb.M;
  const int N = jb.N, K = jb.K, TN = jb.tn, TM = BLOCK_THREADS / TN;
  const int gm = (int)((M + TM - 1) / TM), bx = (blockIdx.x - jb.block0) % gm, by = (blockIdx.x - jb.block0) / gm;
  const int64_t row = (int64_t)bx * TM + threadIdx.x / TN;
  const int col = by * TN + threadIdx.x % TN;
  const bool act = row < M && col < N;
  double2 acc = czero();
  for (int k0 = 0; k0 < K; k0 += XG_KC) {
    __syncthreads();
    for (int e = threadIdx.x; e < XG_KC * TN; e += blockDim.x) {
      const int kk = e / TN, nn = e % TN;
      const int gk = k0 + kk, gn = by * TN + nn;
      Bs[kk][nn] = (gk < K && gn < N) ? xc_from_d(B[(int64_t)gk * ldb + gn]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    if (act) {
      XA s = xa_zero();
      const int kn = K - k0 < XG_KC ? K - k0 : XG_KC;
      const xc* ar = A + row * lda + k0;
      for (int kk = 0; kk < kn; ++kk) xa_mac(s, Bs[kk][threadIdx.x % TN], ar[kk]);
      acc = cadd(acc, xa_to_d(s));
    }
  }
  if (act) {
    const xc v = xc_from_d(acc);
    jb.C[row * jb.ldc + col] = v;
    if (jb.C2) jb.C2[row * jb.ldc + col] = v;
  }
}

// Site 0 of state b: the last remainder (2 x r1) rescaled to the input norm
// (quimb's rsum2 renormalisation), in FP64; the factor goes to *f_out.
// One block.
__global__ void k_x_site0(const xc* rem, int r1, double in_sq, double2* t0, double* f_out) {
  grid_wait();
  __shared__ double s_nrm;
  if (threadIdx.x == 0) {
    double nrm = 0.0;
    for (int i = 0; i < 2 * r1; ++i) nrm += cnorm2(xc_to_d(rem[i]));
    s_nrm = sqrt(nrm);
  }
  __syncthreads();
  const double f = s_nrm > 0.0 ? sqrt(in_sq) / s_nrm : 0.0;
  if (threadIdx.x == 0) *f_out = f;
  for (int i = threadIdx.x; i < 2 * r1; i += blockDim.x) t0[i] = cscale(xc_to_d(rem[i]), f);
}

// dst[i] = f * src[i] for count entries, f = *f_ptr (double-float product).
__global__ void k_x_scale_flat(const xc* src, xc* dst, int64_t count, const double* f_ptr) {
  grid_wait();
  const double f = *f_ptr;
  const float fh = __double2float_rn(f), fl = __double2float_rn(f - (double)fh);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
    const xc x = src[i];
    DF re = {0.f, 0.f}, im = {0.f, 0.f};
    df_mac(re, x.x, x.z, fh, fl);
    df_mac(im, x.y, x.w, fh, fl);
    const float2 r = df_norm(re), m = df_norm(im);
    dst[i] = make_float4(r.x, m.x, r.y, m.y);
  }
}

// Row-major complex128 -> double-float copy of count entries.
__global__ void k_x_from_d_flat(const double2* src, xc* dst, int64_t count) {
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = xc_from_d(src[i]);
}

// ---- (b) layer stage -----------------------------------------------------------------

// The cuts and the gates are layer_cut.cuh's kernels on double-float rows.

__global__ void k_x_layer_fidelity(BatchDev bd, int layer, const xc* work, int num_layers, double atol,
                                   double2* layer_fid, int* nlayers, int* active) {
  grid_wait();
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < bd.B; b += gridDim.x * blockDim.x) {
    if (!active[b]) continue;
    const double2 f = cconj(xc_to_d(work[bd.vec_off[b]]));
    layer_fid[(int64_t)b * num_layers + layer] = f;
    nlayers[b] = layer + 1;
    const double d = cabs_(csub(f, cd(1.0, 0.0)));
    if (d <= atol + 1e-5) active[b] = 0;
  }
}

// ---- gates and sweeps ------------------------------------------------------------------

// The selected gate (or its adjoint) of state b as double-float, in shared memory.
__device__ __forceinline__ void x_load_gate(const double2* g, int m, int adjoint, xc* gs) {
  if (threadIdx.x < m * m) {
    const int r = threadIdx.x / m, c = threadIdx.x % m;
    gs[threadIdx.x] = xc_from_d(adjoint ? cconj(g[c * m + r]) : g[r * m + c]);
  }
}

__global__ void __launch_bounds__(BLOCK_THREADS) k_x_apply_gate(BatchDev bd, xc* vec, GateSel sel) {
  grid_wait();
  __shared__ xc gs[16];
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    const int n = bd.n[b];
    int64_t slot;
    int q, k;
    if (!select_gate(sel, bd, b, n, &slot, &q, &k)) continue;
    __syncthreads();
    x_load_gate(sel.gates + bd.gate_off[b] + slot * 16, 1 << k, sel.adjoint, gs);
    __syncthreads();
    xc* v = vec + bd.vec_off[b];
    int64_t lo, hi;
    tile_range(ipow2(n - k), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    if (k == 2) {
      const int slo = n - 2 - q;
      const int64_t dlo = (int64_t)1 << slo, dhi = dlo << 1;
      for (int64_t r = lo + threadIdx.x; r < hi; r += blockDim.x) {
        const int64_t i0 = quad_base(r, slo);
        const int64_t idx[4] = {i0, i0 + dlo, i0 + dhi, i0 + dhi + dlo};
        xc x[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = v[idx[a]];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          XA s = xa_zero();
#pragma unroll
          for (int c = 0; c < 4; ++c) xa_mac(s, gs[a * 4 + c], x[c]);
          v[idx[a]] = xa_round(s);
        }
      }
    } else {
      const int bit = n - 1 - q;
      const int64_t d = (int64_t)1 << bit;
      for (int64_t r = lo + threadIdx.x; r < hi; r += blockDim.x) {
        const int64_t i0 = pair_base(r, bit);
        const xc x0 = v[i0], x1 = v[i0 + d];
        XA s0 = xa_zero(), s1 = xa_zero();
        xa_mac(s0, gs[0], x0);
        xa_mac(s0, gs[1], x1);
        xa_mac(s1, gs[2], x0);
        xa_mac(s1, gs[3], x1);
        v[i0] = xa_round(s0);
        v[i0 + d] = xa_round(s1);
      }
    }
  }
}

// e[2 i], e[2 i + 1] += real and imaginary part of conj(u) v
__device__ __forceinline__ void x_env_mac(DF (&e)[32], int i, xc u, xc v) {
  df_mac(e[2 * i], u.x, u.z, v.x, v.z);
  df_mac(e[2 * i], u.y, u.w, v.y, v.w);
  df_mac(e[2 * i + 1], u.x, u.z, v.y, v.w);
  df_mac(e[2 * i + 1], -u.y, -u.w, v.x, v.z);
}

// Backward sweep step `step` of every active state (the reference's
// per-gate update, qmprs/synthesis/mps_encoding/sequential.py:452-505):
//   psi <- G^H psi                      (peel the gate from the circuit state)
//   E[a][b] = sum_rest conj(t[a, rest]) psi[b, rest]
//   W = polar(E) (null directions towards conj(G)), G <- conj(W)
// The environment is reduced per tile in fixed order (warps, then tiles);
// the last tile of a state (ticket) computes the polar factor.  The target
// update t <- G_new^H t is the next launch (k_x_apply_gate).
__global__ void __launch_bounds__(BLOCK_THREADS) k_x_sweep_step(BatchDev bd, int step, xc* psi, const xc* t,
                                                                double2* gates, const signed char* arity,
                                                                const int* nlayers, const int* active,
                                                                double2* partials, double* nuc) {
  grid_wait();
  __shared__ xc gs[16];
  __shared__ TF wred[WARPS][32];
  __shared__ double2 env[16];
  __shared__ double2 gd[16];
  __shared__ WarpPolar wp;
  GateSel sel;
  sel.mode = SEL_SWEEP;
  sel.step = step;
  sel.layer = 0;
  sel.adjoint = 1;
  sel.gates = gates;
  sel.arity = arity;
  sel.nlayers = nlayers;
  sel.active = active;
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    const int n = bd.n[b];
    int64_t slot;
    int q, k;
    if (!select_gate(sel, bd, b, n, &slot, &q, &k)) continue;
    const int m = 1 << k;
    double2* gptr = gates + bd.gate_off[b] + slot * 16;
    __syncthreads();
    x_load_gate(gptr, m, 1, gs);
    __syncthreads();
    xc* v = psi + bd.vec_off[b];
    const xc* tv = t + bd.vec_off[b];
    const int nt = bd.state_ntiles[b];
    int64_t lo, hi;
    tile_range(ipow2(n - k), bd.tile_idx[tile], nt, &lo, &hi);
    DF e[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) e[i] = DF{0.f, 0.f};
    if (k == 2) {
      const int slo = n - 2 - q;
      const int64_t dlo = (int64_t)1 << slo, dhi = dlo << 1;
      for (int64_t r = lo + threadIdx.x; r < hi; r += blockDim.x) {
        const int64_t i0 = quad_base(r, slo);
        const int64_t idx[4] = {i0, i0 + dlo, i0 + dhi, i0 + dhi + dlo};
        xc x[4], y[4], tt[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = v[idx[a]];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          XA s = xa_zero();
#pragma unroll
          for (int c = 0; c < 4; ++c) xa_mac(s, gs[a * 4 + c], x[c]);
          y[a] = xa_round(s);
          v[idx[a]] = y[a];
          tt[a] = tv[idx[a]];
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int c = 0; c < 4; ++c) x_env_mac(e, a * 4 + c, tt[a], y[c]);
      }
    } else {
      const int bit = n - 1 - q;
      const int64_t d = (int64_t)1 << bit;
      for (int64_t r = lo + threadIdx.x; r < hi; r += blockDim.x) {
        const int64_t i0 = pair_base(r, bit);
        const xc x0 = v[i0], x1 = v[i0 + d];
        XA s0 = xa_zero(), s1 = xa_zero();
        xa_mac(s0, gs[0], x0);
        xa_mac(s0, gs[1], x1);
        xa_mac(s1, gs[2], x0);
        xa_mac(s1, gs[3], x1);
        const xc y0 = xa_round(s0), y1 = xa_round(s1);
        v[i0] = y0;
        v[i0 + d] = y1;
        const xc t0 = tv[i0], t1 = tv[i0 + d];
        x_env_mac(e, 0, t0, y0);
        x_env_mac(e, 1, t0, y1);
        x_env_mac(e, 2, t1, y0);
        x_env_mac(e, 3, t1, y1);
      }
    }
    // per warp (fixed exchange), then the block's warps in a fixed order
    wred[warp][tid & 31] = warp_sum32_tf(e);
    __syncthreads();
    if (tid < 32) env_sum_warps(wred, partials + (int64_t)tile * 16, tid);
    __syncthreads();
    if (last_tile_ticket(bd.ticket, b, nt)) {
      const int entry = tid >> 4, l16 = tid & 15;
      const int t0 = bd.state_tile0[b];
      double2 s = czero();
      for (int tt = l16; tt < nt; tt += 16) s = cadd(s, __ldcg(&partials[(int64_t)(t0 + tt) * 16 + entry]));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s.x += __shfl_down_sync(0xffffffffu, s.x, o, 16);
        s.y += __shfl_down_sync(0xffffffffu, s.y, o, 16);
      }
      if (l16 == 0) env[entry] = s;
      if (tid < m * m) gd[tid] = gptr[tid];
      __syncthreads();
      if (tid < 32) {
        // to FP64: rank-deficient environments leave null directions that
        // follow the current gate, and an FP32 completion of them would
        // enter the later steps at first order
        bool finite;
        const bool last = step == nlayers[b] * n - 1;
        const double nn = warp_polar_exact(wp, env, gd, m, last, &finite);
        if (finite && tid < m * m) gptr[tid] = gd[tid];
        if (tid == 0) {
          if (finite && last) nuc[b] = nn;
          if (!finite) atomicOr(bd.err, KERR_NONFINITE);
          bd.ticket[b] = 0;
        }
      }
      __syncthreads();
    }
  }
}

// Every sweep of a state in one block (states of at most X_FUSED_MAXN
// qubits): psi and t as double-float in shared memory, the same steps as
// the launch-per-step path (k_x_apply_gate / k_x_sweep_step /
// k_sweep_finish): C|0> rebuilt gate by gate, t from the target, then per
// gate (backward order) psi <- G^H psi, E = sum conj(t) psi, the FP64
// polar factor by warp 0 (G <- conj(W)), t <- G^H t; after the sweep
// the fidelity nuc / ||target||, the sweep count and the stop at
// stop_fidelity.  The environment is reduced per warp (fixed exchange)
// and over the warps in order.  As in k_sweep_fused the polar factor bounds
// a step, and the other warps peel the next gate from psi meanwhile.
// Measured (10 qubits, 15 layers, 2 sweeps, 300 steps): 51.2 ms with a
// single-thread factor, 4.7 ms now (16 us a step; environments summed and
// handed on in double-float took 0.5 us less and up to doubled the gates'
// error, their last sums in FP64 half a microsecond more).
__device__ __forceinline__ void x_fused_apply(xc* v, int n, int q, int k, const xc* gs, int tid, int step) {
  if (k == 2) {
    const int slo = n - 2 - q, dlo = 1 << slo, dhi = dlo << 1;
    for (int r = tid; r < (1 << (n - 2)); r += step) {
      const int i0 = (int)quad_base(r, slo);
      const int idx[4] = {i0, i0 + dlo, i0 + dhi, i0 + dhi + dlo};
      xc x[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) x[a] = v[idx[a]];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        XA acc = xa_zero();
#pragma unroll
        for (int c = 0; c < 4; ++c) xa_mac(acc, gs[a * 4 + c], x[c]);
        v[idx[a]] = xa_round(acc);
      }
    }
  } else {
    const int bit = n - 1 - q, d = 1 << bit;
    for (int r = tid; r < (1 << (n - 1)); r += step) {
      const int i0 = (int)pair_base(r, bit);
      const xc x0 = v[i0], x1 = v[i0 + d];
      XA s0 = xa_zero(), s1 = xa_zero();
      xa_mac(s0, gs[0], x0);
      xa_mac(s0, gs[1], x1);
      xa_mac(s1, gs[2], x0);
      xa_mac(s1, gs[3], x1);
      v[i0] = xa_round(s0);
      v[i0 + d] = xa_round(s1);
    }
  }
}

__global__ void __launch_bounds__(BLOCK_THREADS) k_x_sweep_fused(BatchDev bd, const xc* target, double2* gates,
                                                                 const signed char* arity, const int* nlayers,
                                                                 int* active, const double2* tnorm2, int num_sweeps,
                                                                 double stop_fid, double* sweep_fid,
                                                                 int* sweeps_done) {
  grid_wait();
  extern __shared__ xc xsm[];
  __shared__ xc gs[2][16];           // the gate to apply (rebuild), or to peel
  __shared__ xc gt[16];              // the new gate's adjoint
  __shared__ double2 gd[2][16];      // the step's gate and the next step's
  __shared__ TF wred[WARPS][32];
  __shared__ double2 env[16];
  __shared__ WarpPolar wp;
  const int b = blockIdx.x;
  if (b >= bd.B) return;
  const int n = bd.n[b];
  const int N = 1 << n;
  xc* psi = xsm;
  xc* tt = xsm + N;
  const int L = nlayers[b];
  const int G = L * n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const signed char* ar = arity + bd.gate_off[b] / 16;
  double2* gb = gates + bd.gate_off[b];
  double nuc = 0.0;   // warp 0
  // the first step at or after j whose gate is valid (G if none); invalid
  // slots raise the error flag and are skipped
  auto next_step = [&](int j, bool forward, int& slot, int& site, int& k) {
    for (; j < G; ++j) {
      const int l = forward ? L - 1 - j / n : j / n;
      site = forward ? j % n : n - 1 - j % n;
      slot = l * n + site;
      k = ar[slot];
      if (k == 1 || (k == 2 && site <= n - 2)) break;
      if (tid == 0) atomicOr(bd.err, KERR_BAD_GATE);
    }
    return j;
  };
  for (int sw = 0; sw < num_sweeps; ++sw) {
    __syncthreads();
    if (!active[b]) break;
    for (int i = tid; i < N; i += BLOCK_THREADS) {
      psi[i] = make_float4(i == 0 ? 1.f : 0.f, 0.f, 0.f, 0.f);
      tt[i] = target[bd.vec_off[b] + i];
    }
    // C|0>; the next gate is fetched while one is applied
    int slot, site, k;
    int j = next_step(0, true, slot, site, k);
    if (j < G && tid < (1 << (2 * k))) gs[0][tid] = xc_from_d(gb[(int64_t)slot * 16 + tid]);
    for (int buf = 0; j < G; buf ^= 1) {
      __syncthreads();
      int slot2 = 0, site2 = 0, k2 = 0;
      const int j2 = next_step(j + 1, true, slot2, site2, k2);
      double2 pre = czero();
      const bool fetch = j2 < G && tid < (1 << (2 * k2));
      if (fetch) pre = gb[(int64_t)slot2 * 16 + tid];
      x_fused_apply(psi, n, site, k, gs[buf], tid, BLOCK_THREADS);
      if (fetch) gs[buf ^ 1][tid] = xc_from_d(pre);
      j = j2;
      slot = slot2;
      site = site2;
      k = k2;
    }
    __syncthreads();
    // backward sweep: the first gate is peeled here, every later one while
    // its predecessor's polar factor is computed
    j = next_step(0, false, slot, site, k);
    if (j < G) {
      if (tid < (1 << (2 * k))) {
        const double2 v = gb[(int64_t)slot * 16 + tid];
        gd[0][tid] = v;
        gs[0][(tid % (1 << k)) * (1 << k) + tid / (1 << k)] = xc_from_d(cconj(v));
      }
      __syncthreads();
      x_fused_apply(psi, n, site, k, gs[0], tid, BLOCK_THREADS);
    }
    for (int buf = 0; j < G; buf ^= 1) {
      __syncthreads();
      const int m = 1 << k;
      int slot2 = 0, site2 = 0, k2 = 0;
      const int j2 = next_step(j + 1, false, slot2, site2, k2);
      double2 pre = czero();
      const bool fetch = j2 < G && tid < (1 << (2 * k2));
      if (fetch) pre = gb[(int64_t)slot2 * 16 + tid];
      DF e[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) e[i] = DF{0.f, 0.f};
      if (k == 2) {
        const int slo = n - 2 - site, dlo = 1 << slo, dhi = dlo << 1;
        for (int r = tid; r < (N >> 2); r += BLOCK_THREADS) {
          const int i0 = (int)quad_base(r, slo);
          const int idx[4] = {i0, i0 + dlo, i0 + dhi, i0 + dhi + dlo};
          xc y[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) y[a] = psi[idx[a]];
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const xc tv = tt[idx[a]];
#pragma unroll
            for (int c = 0; c < 4; ++c) x_env_mac(e, a * 4 + c, tv, y[c]);
          }
        }
      } else {
        const int bit = n - 1 - site, d = 1 << bit;
        for (int r = tid; r < (N >> 1); r += BLOCK_THREADS) {
          const int i0 = (int)pair_base(r, bit);
          const xc y0 = psi[i0], y1 = psi[i0 + d], t0 = tt[i0], t1 = tt[i0 + d];
          x_env_mac(e, 0, t0, y0);
          x_env_mac(e, 1, t0, y1);
          x_env_mac(e, 2, t1, y0);
          x_env_mac(e, 3, t1, y1);
        }
      }
      wred[warp][lane] = warp_sum32_tf(e);
      if (fetch) {
        gd[buf ^ 1][tid] = pre;
        gs[buf ^ 1][(tid % (1 << k2)) * (1 << k2) + tid / (1 << k2)] = xc_from_d(cconj(pre));
      }
      __syncthreads();
      if (warp == 0) {
        env_sum_warps(wred, env, lane);
        __syncwarp();
        bool finite;
        double2* g = gd[buf];
        const double nn = warp_polar_exact(wp, env, g, m, j2 >= G, &finite);
        if (finite && j2 >= G) nuc = nn;
        if (finite && lane < m * m) gb[(int64_t)slot * 16 + lane] = g[lane];
        if (!finite && lane == 0) atomicOr(bd.err, KERR_NONFINITE);
        if (lane < m * m) gt[(lane % m) * m + lane / m] = xc_from_d(cconj(g[lane]));
      } else if (j2 < G) {
        x_fused_apply(psi, n, site2, k2, gs[buf ^ 1], tid - 32, BLOCK_THREADS - 32);
      }
      __syncthreads();
      if (j2 < G) x_fused_apply(tt, n, site, k, gt, tid, BLOCK_THREADS);   // t <- G_new^H t
      j = j2;
      slot = slot2;
      site = site2;
      k = k2;
    }
    if (tid == 0) {
      const double f = nuc / sqrt(tnorm2[b].x);
      sweep_fid[(int64_t)b * num_sweeps + sw] = f;
      sweeps_done[b] = sw + 1;
      if (stop_fid > 0.0 && f >= stop_fid) active[b] = 0;
    }
  }
}

// ---- launches ---------------------------------------------------------------------------

void launch_x_from_d(const BatchDev& bd, const double2* src, xc* dst, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_from_d, grid_for(bd), BLOCK_THREADS, 0, s, bd, src, dst);
}

void launch_x_to_d(const BatchDev& bd, const xc* src, double2* dst, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_to_d, grid_for(bd), BLOCK_THREADS, 0, s, bd, src, dst);
}

void launch_x_copy(const BatchDev& bd, const xc* src, xc* dst, const int* active, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_copy, grid_for(bd), BLOCK_THREADS, 0, s, bd, src, dst, active);
}

void launch_x_zero(const BatchDev& bd, xc* vec, const int* active, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_zero, grid_for(bd), BLOCK_THREADS, 0, s, bd, vec, active);
}

void launch_x_dot(const BatchDev& bd, const xc* a, const xc* b, double2* partials, double2* out, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_dot, grid_for(bd), BLOCK_THREADS, 0, s, bd, a, b, partials);
  launch_reduce_tiles(bd, partials, out, s);
}

void launch_d_dot(const BatchDev& bd, const double2* a, const double2* b, double2* partials, double2* out,
                  cudaStream_t s) {
  qm_note_launch();
  launch_after(k_d_dot, grid_for(bd), BLOCK_THREADS, 0, s, bd, a, b, partials);
  launch_reduce_tiles(bd, partials, out, s);
}

void launch_x_normalize(const BatchDev& bd, const xc* src, xc* dst, double2* partials, double2* sq, cudaStream_t s) {
  launch_x_dot(bd, src, src, partials, sq, s);
  qm_note_launch();
  launch_after(k_x_scale, grid_for(bd), BLOCK_THREADS, 0, s, bd, src, dst, sq);
}

void launch_x_grams(XGramJob* jobs, int count, int64_t WW, cudaStream_t s) {
  for (int j0 = 0; j0 < count; j0 += X_JOBS) {
    XJobs<XGramJob> js;
    js.count = std::min(X_JOBS, count - j0);
    int blocks = 0, rblocks = 0;
    for (int k = 0; k < js.count; ++k) {
      XGramJob& jb = js.job[k];
      jb = jobs[j0 + k];
      jb.nsplit = (int)std::min<int64_t>(TT_SPLIT, std::max<int64_t>(1, jb.rows / 1024));
      jb.block0 = blocks;
      jb.rblock0 = rblocks;
      const int nt = x_gram_nt(jb.w);
      blocks += nt * (nt + 1) / 2 * jb.nsplit;
      rblocks += (int)(((int64_t)jb.w * jb.w + BLOCK_THREADS - 1) / BLOCK_THREADS);
    }
    qm_note_launch();
    launch_after(k_x_gram_tile, blocks, BLOCK_THREADS, 0, s, js, WW);
    qm_note_launch();
    launch_after(k_x_gram_reduce, rblocks, BLOCK_THREADS, 0, s, js, WW);
  }
}

void launch_x_gemms(XGemmJob* jobs, int count, cudaStream_t s) {
  for (int j0 = 0; j0 < count; j0 += X_JOBS) {
    XJobs<XGemmJob> js;
    js.count = std::min(X_JOBS, count - j0);
    int64_t blocks = 0;
    for (int k = 0; k < js.count; ++k) {
      XGemmJob& jb = js.job[k];
      jb = jobs[j0 + k];
      jb.tn = 1;
      while (jb.tn < jb.N && jb.tn < 32) jb.tn <<= 1;
      const int tm = BLOCK_THREADS / jb.tn;
      jb.block0 = (int)blocks;
      blocks += (jb.M + tm - 1) / tm * ((jb.N + jb.tn - 1) / jb.tn);
    }
    qm_note_launch();
    launch_after(k_x_gemm, (unsigned)blocks, BLOCK_THREADS, 0, s, js);
  }
}

void launch_x_site0(const xc* rem, int r1, double in_sq, double2* t0, double* f_out, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_site0, 1, 64, 0, s, rem, r1, in_sq, t0, f_out);
}

void launch_x_scale_flat(const xc* src, xc* dst, int64_t count, const double* f, cudaStream_t s) {
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, 1024));
  qm_note_launch();
  launch_after(k_x_scale_flat, blocks, 256, 0, s, src, dst, count, f);
}

void launch_x_from_d_flat(const double2* src, xc* dst, int64_t count, cudaStream_t s) {
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, 1024));
  qm_note_launch();
  launch_after(k_x_from_d_flat, blocks, 256, 0, s, src, dst, count);
}

void launch_x_layer_cut(const BatchDev& bd, int units, int step, int last, const xc* work, xc* buf0, xc* buf1, int* bonds,
                        double2* vsel, double2* site_t, double2* partials, const int* active, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_layer_cut<CutExact>, units, BLOCK_THREADS, 0, s, bd, step, last, work, bonds, vsel, site_t,
               reinterpret_cast<double*>(partials), buf0, buf1, active);
}

void launch_x_layer_build(const BatchDev& bd, int layer, const xc* rem0, const xc* rem1, const int* bonds,
                          double2* site_t, double2* gates, signed char* arity, const int* active, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_layer_build<CutExact>, bd.B, BUILD_THREADS, 0, s, bd, layer, rem0, rem1, bonds, site_t, gates, arity,
               active);
}

void launch_x_layer_fidelity(const BatchDev& bd, int layer, const xc* work, int num_layers, double atol,
                             double2* layer_fid, int* nlayers, int* active, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_layer_fidelity, (bd.B + 127) / 128, 128, 0, s, bd, layer, work, num_layers, atol, layer_fid,
               nlayers, active);
}

void launch_x_apply_gate(const BatchDev& bd, xc* vec, const GateSel& sel, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_apply_gate, grid_for(bd), BLOCK_THREADS, 0, s, bd, vec, sel);
}

void launch_x_sweep_step(const BatchDev& bd, int step, xc* psi, const xc* t, double2* gates, const signed char* arity,
                         const int* nlayers, const int* active, double2* partials, double* nuc, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_x_sweep_step, grid_for(bd), BLOCK_THREADS, 0, s, bd, step, psi, t, gates, arity, nlayers, active,
               partials, nuc);
}

int launch_x_sweep_fused(const BatchDev& bd, int max_n, const xc* target, double2* gates, const signed char* arity,
                         const int* nlayers, int* active, const double2* tnorm2, int num_sweeps, double stop_fid,
                         double* sweep_fid, int* sweeps_done, cudaStream_t s) {
  const size_t smem = 2 * sizeof(xc) * (size_t)ipow2(max_n);
  cudaError_t e = cudaFuncSetAttribute(k_x_sweep_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  qm_note_launch();
  launch_after(k_x_sweep_fused, bd.B, BLOCK_THREADS, smem, s, bd, target, gates, arity, nlayers, active, tnorm2,
               num_sweeps, stop_fid, sweep_fid, sweeps_done);
  return (int)cudaGetLastError();
}
