// Fast mode: every sweep of a batch of small states in one launch.
//
// For batches whose states all have at most SWEEP_FUSED_MAXN qubits, one
// block per state keeps psi and t (complex64) in shared memory and runs the
// reference's per-gate sweep (qmprs/synthesis/mps_encoding/sequential.py:
// 452-505) for every sweep:
//   C|0>               rebuilt gate by gate (forward circuit order);
//   t                  the target;
//   per gate (backward circuit order)
//     psi <- G^H psi   peel the gate from the circuit state,
//     E = sum_rest conj(t[a, rest]) psi[c, rest]   (FP32 per thread and
//                      across a warp's lanes, double-float across the warps,
//                      in fixed order),
//     W = polar(E)     warp 0 (warp_polar.cuh; null directions towards the
//                      current gate), G <- conj(W),
//     t <- G^H t;
//   the sweep fidelity nuc / ||target||, the sweep count, the stop at
//   stop_fidelity.
// With env_out set, one pass computes every gate's environment at the fixed
// circuit instead: E is written to the gate's slot of env_out (the gate
// store's layout, <target|C|0> = sum_ac G[a, c] E[a, c] for every gate),
// the gates stay as they are and no fidelity is written.
// On a 1024-amplitude state the grouped sweep is bound by launches and its
// window algebra (about 130 launches per sweep); here a step is a few
// block-wide passes over shared memory and one warp's polar factor, which
// bounds it: peeling the next gate from psi does not depend on the new
// gate, so the other warps do it meanwhile.
// Measured (10 qubits, 15 layers, 4 sweeps, 600 steps): 29.1 ms with
// a single-thread factor and the peel on the chain, 4.2 ms now (6 us a step).
#include "warp_polar.cuh"

__device__ __forceinline__ bool fused_valid(int k, int site, int n) { return k == 1 || (k == 2 && site <= n - 2); }

// v <- g v (row-major, complex64 in shared memory) on qubit q (and q + 1)
// by threads tid, tid + step, ... of the block.
__device__ __forceinline__ void fused_apply(float2* v, int n, int q, int k, const float2* gs, int tid, int step) {
  if (k == 2) {
    const int slo = n - 2 - q, dlo = 1 << slo, dhi = dlo << 1;
    for (int r = tid; r < (1 << (n - 2)); r += step) {
      const int i0 = (int)quad_base(r, slo);
      const int idx[4] = {i0, i0 + dlo, i0 + dhi, i0 + dhi + dlo};
      float2 x[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) x[a] = v[idx[a]];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        float2 acc = cf(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc = fmac(acc, gs[a * 4 + c], x[c]);
        v[idx[a]] = acc;
      }
    }
  } else {
    const int bit = n - 1 - q, d = 1 << bit;
    for (int r = tid; r < (1 << (n - 1)); r += step) {
      const int i0 = (int)pair_base(r, bit);
      const float2 x0 = v[i0], x1 = v[i0 + d];
      v[i0] = fmac(fmac(cf(0.f, 0.f), gs[0], x0), gs[1], x1);
      v[i0 + d] = fmac(fmac(cf(0.f, 0.f), gs[2], x0), gs[3], x1);
    }
  }
}

// acc += conj(a) b, real and imaginary part separately
__device__ __forceinline__ void conj_mac(float& re, float& im, float2 a, float2 b) {
  re = fmaf(a.x, b.x, fmaf(a.y, b.y, re));
  im = fmaf(a.x, b.y, fmaf(-a.y, b.x, im));
}

// entry e of an m x m gate (or its adjoint) as complex64
__device__ __forceinline__ float2 fused_entry(const double2* g, int m, int adjoint, int e) {
  const double2 v = adjoint ? cconj(g[(e % m) * m + e / m]) : g[e];
  return cf((float)v.x, (float)v.y);
}

__global__ void __launch_bounds__(BLOCK_THREADS) k_sweep_fused(BatchDev bd, const float2* target, double2* gates,
                                                               const signed char* arity, const int* nlayers,
                                                               int* active, const double2* tnorm2, int num_sweeps,
                                                               double stop_fid, double* sweep_fid,
                                                               int* sweeps_done, double2* env_out) {
  grid_wait();
  extern __shared__ float2 fsm[];
  __shared__ float2 gs[2][16];       // the gate to apply (rebuild), or to peel
  __shared__ float2 gt[16];          // the new gate's adjoint
  __shared__ double2 gd[2][16];      // the step's gate and the next step's
  __shared__ float2 wred[WARPS][32];
  __shared__ xc env[16];
  __shared__ WarpPolar wp;
  const int b = blockIdx.x;
  if (b >= bd.B) return;
  const int n = bd.n[b];
  const int N = 1 << n;
  float2* psi = fsm;
  float2* tt = fsm + N;
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
      if (fused_valid(k, site, n)) break;
      if (tid == 0) atomicOr(bd.err, KERR_BAD_GATE);
    }
    return j;
  };
  for (int sw = 0; sw < num_sweeps; ++sw) {
    __syncthreads();
    if (!active[b]) break;
    for (int i = tid; i < N; i += BLOCK_THREADS) {
      psi[i] = cf(i == 0 ? 1.f : 0.f, 0.f);
      tt[i] = target[bd.vec_off[b] + i];
    }
    // C|0>; the next gate is fetched while one is applied
    int slot, site, k;
    int j = next_step(0, true, slot, site, k);
    if (j < G && tid < (1 << (2 * k))) gs[0][tid] = fused_entry(gb + (int64_t)slot * 16, 1 << k, 0, tid);
    for (int buf = 0; j < G; buf ^= 1) {
      __syncthreads();
      int slot2 = 0, site2 = 0, k2 = 0;
      const int j2 = next_step(j + 1, true, slot2, site2, k2);
      float2 pre = cf(0.f, 0.f);
      const bool fetch = j2 < G && tid < (1 << (2 * k2));
      if (fetch) pre = fused_entry(gb + (int64_t)slot2 * 16, 1 << k2, 0, tid);
      fused_apply(psi, n, site, k, gs[buf], tid, BLOCK_THREADS);
      if (fetch) gs[buf ^ 1][tid] = pre;
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
        gd[0][tid] = gb[(int64_t)slot * 16 + tid];
        gs[0][tid] = fused_entry(gb + (int64_t)slot * 16, 1 << k, 1, tid);
      }
      __syncthreads();
      fused_apply(psi, n, site, k, gs[0], tid, BLOCK_THREADS);
    }
    for (int buf = 0; j < G; buf ^= 1) {
      __syncthreads();
      const int m = 1 << k;
      int slot2 = 0, site2 = 0, k2 = 0;
      const int j2 = next_step(j + 1, false, slot2, site2, k2);
      double2 pre = czero();
      const bool fetch = j2 < G && tid < (1 << (2 * k2));
      if (fetch) pre = gb[(int64_t)slot2 * 16 + tid];
      // environment: value 2 i is Re E_i, 2 i + 1 Im E_i
      float e[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) e[i] = 0.f;
      if (k == 2) {
        const int slo = n - 2 - site, dlo = 1 << slo, dhi = dlo << 1;
        for (int r = tid; r < (N >> 2); r += BLOCK_THREADS) {
          const int i0 = (int)quad_base(r, slo);
          const int idx[4] = {i0, i0 + dlo, i0 + dhi, i0 + dhi + dlo};
          float2 y[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) y[a] = psi[idx[a]];
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const float2 tv = tt[idx[a]];
#pragma unroll
            for (int c = 0; c < 4; ++c) conj_mac(e[2 * (a * 4 + c)], e[2 * (a * 4 + c) + 1], tv, y[c]);
          }
        }
      } else {
        const int bit = n - 1 - site, d = 1 << bit;
        for (int r = tid; r < (N >> 1); r += BLOCK_THREADS) {
          const int i0 = (int)pair_base(r, bit);
          const float2 y0 = psi[i0], y1 = psi[i0 + d], t0 = tt[i0], t1 = tt[i0 + d];
          conj_mac(e[0], e[1], t0, y0);
          conj_mac(e[2], e[3], t0, y1);
          conj_mac(e[4], e[5], t1, y0);
          conj_mac(e[6], e[7], t1, y1);
        }
      }
      // over a warp's lanes in FP32 (a lane holds one to eight quads), over
      // the warps in double-float
      wred[warp][lane] = make_float2(warp_sum32(e), 0.f);
      if (fetch) {
        gd[buf ^ 1][tid] = pre;
        gs[buf ^ 1][(tid % (1 << k2)) * (1 << k2) + tid / (1 << k2)] = cf((float)pre.x, -(float)pre.y);
      }
      __syncthreads();
      if (warp == 0) {
        env_sum_warps(wred, env, lane);
        __syncwarp();
        bool finite = true;
        double2* g = gd[buf];
        if (env_out) {
          const bool mine = lane < m * m;
          const double2 ev = mine ? xc_to_d(env[lane]) : czero();
          finite = __all_sync(0xffffffffu, isfinite(ev.x) && isfinite(ev.y));
          if (mine && finite) env_out[bd.gate_off[b] + (int64_t)slot * 16 + lane] = ev;
        } else {
          const double nn = warp_polar(wp, env, g, m, j2 >= G, &finite);
          if (finite && j2 >= G) nuc = nn;
          if (finite && lane < m * m) gb[(int64_t)slot * 16 + lane] = g[lane];
        }
        if (!finite && lane == 0) atomicOr(bd.err, KERR_NONFINITE);
        if (lane < m * m) gt[lane] = fused_entry(g, m, 1, lane);
      } else if (j2 < G) {
        fused_apply(psi, n, site2, k2, gs[buf ^ 1], tid - 32, BLOCK_THREADS - 32);
      }
      __syncthreads();
      if (j2 < G) fused_apply(tt, n, site, k, gt, tid, BLOCK_THREADS);   // t <- G_new^H t
      j = j2;
      slot = slot2;
      site = site2;
      k = k2;
    }
    if (tid == 0 && !env_out) {
      const double f = nuc / sqrt(tnorm2[b].x);
      sweep_fid[(int64_t)b * num_sweeps + sw] = f;
      sweeps_done[b] = sw + 1;
      if (stop_fid > 0.0 && f >= stop_fid) active[b] = 0;
    }
  }
}
int launch_sweep_fused(const BatchDev& bd, int max_n, const float2* target, double2* gates, const signed char* arity,
                       const int* nlayers, int* active, const double2* tnorm2, int num_sweeps, double stop_fid,
                       double* sweep_fid, int* sweeps_done, cudaStream_t s, double2* env_out) {
  const size_t smem = 2 * sizeof(float2) * (size_t)ipow2(max_n);
  cudaError_t e = cudaFuncSetAttribute(k_sweep_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  qm_note_launch();
  launch_after(k_sweep_fused, bd.B, BLOCK_THREADS, smem, s, bd, target, gates, arity, nlayers, active, tnorm2,
               num_sweeps, stop_fid, sweep_fid, sweeps_done, env_out);
  return (int)cudaGetLastError();
}
