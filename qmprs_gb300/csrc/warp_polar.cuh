// Unitary polar factor of a 4 x 4 (or 2 x 2) environment by one warp:
// warp_polar for the fast mode, warp_polar_exact for the exact mode.
//
// The same definition as polar_sweep in small_linalg.h: W maximises
// Re Tr(W^H E), singular values up to QM_POLAR_NULL_TOL of the largest
// count as zero, and on that null space W is the completion nearest to the
// current gate's.  One thread's chain of dependent FP32 and FP64 operations
// is what bounded every sweep step (GB300: 31 ns per dependent FP64
// operation, and an FP64 warp instruction holds the SM's two FP64 units for
// 16 cycles whatever its active lanes), so the algebra is spread over the
// lanes instead:
//   * one-sided (Hestenes) Jacobi in FP32: lane (pair, row) of a group of
//     eight holds one row of two columns; the two pairs of a round rotate
//     at once and a swap of columns between the pairs gives the next round,
//     so a cyclic sweep is three rounds instead of six rotations;
//   * FP64 4 x 4 products, one real or imaginary part of an entry per lane
//     (eight multiply-adds in chains of two), which turn the FP32 basis
//     into an FP64-orthonormal W: V is re-orthonormalised by one
//     Newton-Schulz step, B = E V, U the first-order polar factor of B's
//     normalised columns, W = U V^H and one more Newton-Schulz step.
// The error left is second order in the FP32 one (about 1e-7), where the
// single-thread factor kept the FP32 error itself.  A null space on which
// the current gate has no component either (rare) takes the single-thread
// code.
// The exact mode's factor (the definition of polar_jacobi_pre) starts the
// same way, then finishes with Hestenes sweeps on FP64 columns.  Their
// rotations take the angle from FP32 (FP64 square roots and divisions are
// chains of about ten dependent operations each) as a complex tangent w, and
// only c = 1 / sqrt(1 + |w|^2) in FP64, so every rotation is unitary to FP64
// rounding and an inexact angle costs at most one more sweep.
// Measured on a 10-qubit state (15 layers, one block): 48.5 us per sweep
// step with the single-thread factor, 11.2 us with this one.
#pragma once

#include "dfloat.cuh"

struct WarpPolar {
  double2 E[16];          // the environment, scaled by a power of two, padded to 4 x 4
  double2 Wp[16];         // the current gate's conjugate, padded with the identity
  double2 V[16], U[16], T[16], C[16];
  float sig[4], rsig[4];  // column norms of E V and their reciprocals; 0 for null columns
  int null_mask;
};

// One part (0 real, 1 imaginary) of entry (i, j) of op(A) op(B), 4 x 4
// row-major in shared memory; op is the adjoint where ADJ.
template <bool ADJ_A, bool ADJ_B>
__device__ __forceinline__ double wmm_part(const double2* A, const double2* B, int i, int j, int part) {
  double acc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double2 a = ADJ_A ? cconj(A[k * 4 + i]) : A[i * 4 + k];
    const double2 b = ADJ_B ? cconj(B[j * 4 + k]) : B[k * 4 + j];
    acc[k] = fma(a.y, part ? b.x : -b.y, a.x * (part ? b.y : b.x));
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

__device__ __forceinline__ void wmm_store(double2* C, int lane, double v) {
  reinterpret_cast<double*>(C)[lane] = v;   // lane = 2 * entry + part
}

__device__ __forceinline__ float quad_sum(float v) {   // over the four rows of a column
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}

__device__ __forceinline__ float2 shfl_xor2(float2 v, int o) {
  return cf(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// The FP32 rotation of columns p, q with norms^2 al, be and inner product
// (gx, gy): c and s e, the identity unless |g|^2 > 1e-12 al be (as
// jacobi_pair_f).  Approximate reciprocals and square roots: an inexact
// angle only leaves a little for the next sweep.
__device__ __forceinline__ bool wh_rotation(float al, float be, float gx, float gy, bool allowed, float& c, float& sx,
                                            float& sy) {
  const float ag2 = fmaf(gx, gx, gy * gy);
  const bool go = allowed && ag2 > 1e-12f * al * be;
  const float ri = rsqrtf(go ? ag2 : 1.f);
  const float zeta = 0.5f * (be - al) * ri, az = fabsf(zeta);
  const float s1 = fmaf(az, az, 1.f);
  float t = az > 1e4f ? __fdividef(0.5f, az) : __fdividef(1.f, az + s1 * rsqrtf(s1));
  t = go ? copysignf(t, zeta) : 0.f;
  c = rsqrtf(fmaf(t, t, 1.f));
  const float s = c * t * ri;
  sx = gx * s;
  sy = gy * s;
  return t != 0.f;
}

__device__ __forceinline__ void wh_apply(float2& p, float2& q, float c, float sx, float sy) {
  // p <- c p - s conj(e) q ; q <- s e p + c q
  const float2 np = cf(c * p.x - fmaf(sx, q.x, sy * q.y), c * p.y - fmaf(sx, q.y, -sy * q.x));
  const float2 nq = cf(fmaf(c, q.x, fmaf(sx, p.x, -sy * p.y)), fmaf(c, q.y, fmaf(sx, p.y, sy * p.x)));
  p = np;
  q = nq;
}

// FP32 Hestenes sweeps of the four columns (lane l & 7 = 4 pair + row holds
// rows of columns p and q of A and V); with `masked` only pairs of flagged
// columns rotate.  Flags move with their columns.  Returns 1 after an odd
// number of sweeps, which leaves columns 2 and 3 exchanged.
__device__ __forceinline__ int wh_sweeps(float2& ap, float2& aq, float2& vp, float2& vq, int& fp, int& fq,
                                          bool masked) {
  const bool hi = (threadIdx.x & 4) != 0;   // the second pair's lanes
  int odd = 0;
  for (int sweep = 0; sweep < 30; ++sweep) {
    odd ^= 1;
    bool rot = false;
#pragma unroll
    for (int rd = 0; rd < 3; ++rd) {
      const float al = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y)), be = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
      const float gx = quad_sum(fmaf(ap.x, aq.x, ap.y * aq.y)), gy = quad_sum(fmaf(ap.x, aq.y, -ap.y * aq.x));
      float c, sx, sy;
      rot |= wh_rotation(al, be, gx, gy, !masked || (fp && fq), c, sx, sy);
      wh_apply(ap, aq, c, sx, sy);
      wh_apply(vp, vq, c, sx, sy);
      // next pairing: rounds 0 and 2 swap q of pair 0 with p of pair 1,
      // round 1 swaps the two q; three rounds meet all six pairs
      const bool give_p = rd != 1 && hi;
      const float2 ao = shfl_xor2(give_p ? ap : aq, 4), vo = shfl_xor2(give_p ? vp : vq, 4);
      const int fo = masked ? __shfl_xor_sync(0xffffffffu, give_p ? fp : fq, 4) : 0;
      if (give_p) {
        ap = ao;
        vp = vo;
        fp = fo;
      } else {
        aq = ao;
        vq = vo;
        fq = fo;
      }
    }
    if (!__any_sync(0xffffffffu, rot)) break;
  }
  return odd;
}

// Scale ws.E (m x m, stride m, unscaled in `env`) into the 4 x 4 workspace:
// multiplied by a power of two that brings the largest part into [1/2, 1);
// a 2 x 2 environment is padded with its largest part on the diagonal
// (neither null nor larger than its norm), its gate with the identity.
// Returns the exponent; *finite is false if any entry is not.
__device__ __forceinline__ int wp_load(WarpPolar& ws, const double2* env, const double2* gate, int m, int lane,
                                       bool* finite) {
  const int r = (lane >> 2) & 3, c = lane & 3;
  const bool in = r < m && c < m;
  const double2 e = in ? env[r * m + c] : czero();
  *finite = __all_sync(0xffffffffu, isfinite(e.x) && isfinite(e.y));
  const float mag = fmaxf(fabsf((float)e.x), fabsf((float)e.y));
  const int mbits = __reduce_max_sync(0xffffffffu, __float_as_int(mag));
  int ex = (mbits >> 23) - 126;
  if (mbits == 0) ex = 0;
  const double sc = __hiloint2double((1023 - ex) << 20, 0);
  if (lane < 16) {
    const double pad = r == c ? (double)__int_as_float(mbits) * sc : 0.0;
    ws.E[lane] = in ? cd(e.x * sc, e.y * sc) : cd(pad, 0.0);
    ws.Wp[lane] = in ? cconj(gate[r * m + c]) : cd(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncwarp();
  return ex;
}

// Null columns (f set) of the orthogonalised A become X = (I - U_s U_s^H)
// Wp V_N, rotated among themselves to orthogonal columns; false if one of
// them vanishes (the caller takes the single-thread code).
__device__ __forceinline__ bool wp_null_columns(const WarpPolar& ws, float2& ap, float2& aq, float2& vp, float2& vq,
                                                int& fp, int& fq, float al, float be, int lane) {
  const int row = lane & 3;
  float2 xp = cf(0.f, 0.f), xq = cf(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int src = (lane & ~3) | k;
    const float2 w = cf((float)ws.Wp[row * 4 + k].x, (float)ws.Wp[row * 4 + k].y);
    xp = fmac(xp, w, cf(__shfl_sync(0xffffffffu, vp.x, src), __shfl_sync(0xffffffffu, vp.y, src)));
    xq = fmac(xq, w, cf(__shfl_sync(0xffffffffu, vq.x, src), __shfl_sync(0xffffffffu, vq.y, src)));
  }
  const float rp = fp ? 0.f : rsqrtf(al), rq = fq ? 0.f : rsqrtf(be);
  float2 u[4];
  u[0] = cf(ap.x * rp, ap.y * rp);
  u[1] = cf(aq.x * rq, aq.y * rq);
  u[2] = shfl_xor2(u[0], 4);
  u[3] = shfl_xor2(u[1], 4);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float px = quad_sum(fmaf(u[i].x, xp.x, u[i].y * xp.y)), py = quad_sum(fmaf(u[i].x, xp.y, -u[i].y * xp.x));
    const float qx = quad_sum(fmaf(u[i].x, xq.x, u[i].y * xq.y)), qy = quad_sum(fmaf(u[i].x, xq.y, -u[i].y * xq.x));
    xp = fmac(xp, cf(-u[i].x, -u[i].y), cf(px, py));
    xq = fmac(xq, cf(-u[i].x, -u[i].y), cf(qx, qy));
  }
  if (fp) ap = xp;
  if (fq) aq = xq;
  wh_sweeps(ap, aq, vp, vq, fp, fq, true);
  const float np = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y)), nq = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
  return __all_sync(0xffffffffu, (!fp || np > 1e-8f) && (!fq || nq > 1e-8f));
}

// The single-thread factor of the workspace's m x m block, for one lane:
// writes the gate, returns Re Tr(W^H E) of the scaled environment.
static __device__ __noinline__ double wp_single_thread(const WarpPolar& ws, double2* gate, int m) {
  double2 e[16], w[16], wprev[16];
  for (int i = 0; i < m * m; ++i) {
    e[i] = ws.E[(i / m) * 4 + i % m];
    wprev[i] = ws.Wp[(i / m) * 4 + i % m];
  }
  const double nn = polar_sweep(e, m, w, wprev);
  for (int i = 0; i < m * m; ++i) gate[i] = cconj(w[i]);
  return nn;
}

// Polar factor of the m x m environment `env` (row-major) by the 32 lanes
// of a warp; `gate` (m x m, shared memory) holds the current gate G and
// receives conj(W).  Returns Re Tr(W^H E) in every lane when `want_trace`.
// *finite is false (and nothing else is done) if env is not finite.
static __device__ __noinline__ double warp_polar(WarpPolar& ws, const double2* env, double2* gate, int m, bool want_trace,
                                          bool* finite) {
  const int lane = threadIdx.x & 31;
  const int ex = wp_load(ws, env, gate, m, lane, finite);
  if (!*finite) return 0.0;
  const double unscale = __hiloint2double((1023 + ex) << 20, 0);
  const int row = lane & 3, pr = (lane >> 2) & 1;
  float2 ap = cf((float)ws.E[row * 4 + 2 * pr].x, (float)ws.E[row * 4 + 2 * pr].y);
  float2 aq = cf((float)ws.E[row * 4 + 2 * pr + 1].x, (float)ws.E[row * 4 + 2 * pr + 1].y);
  float2 vp = cf(row == 2 * pr ? 1.f : 0.f, 0.f), vq = cf(row == 2 * pr + 1 ? 1.f : 0.f, 0.f);
  int fp = 0, fq = 0;
  wh_sweeps(ap, aq, vp, vq, fp, fq, false);
  float al = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y)), be = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
  const float m2 = fmaxf(fmaxf(al, be), __shfl_xor_sync(0xffffffffu, fmaxf(al, be), 4));
  const float thr = (float)(QM_POLAR_NULL_TOL * QM_POLAR_NULL_TOL) * m2;
  fp = !(al > thr && al > 0.f);
  fq = !(be > thr && be > 0.f);
  bool ok = true;
  if (__any_sync(0xffffffffu, fp || fq)) {
    ok = wp_null_columns(ws, ap, aq, vp, vq, fp, fq, al, be, lane);
    al = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y));
    be = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
  }
  if (!ok) {
    const double nn = lane == 0 ? wp_single_thread(ws, gate, m) * unscale : 0.0;
    __syncwarp();
    return __shfl_sync(0xffffffffu, nn, 0);
  }
  // V and the null columns of U to shared memory, column order as it fell
  const unsigned nb_p = __ballot_sync(0xffffffffu, fp), nb_q = __ballot_sync(0xffffffffu, fq);
  const int nmask = (nb_p & 1) | ((nb_q & 1) << 1) | (((nb_p >> 4) & 1) << 2) | (((nb_q >> 4) & 1) << 3);
  if (lane < 8) {
    const float rp = rsqrtf(al), rq = rsqrtf(be);
    ws.V[row * 4 + 2 * pr] = f2d(vp);
    ws.V[row * 4 + 2 * pr + 1] = f2d(vq);
    if (fp) ws.U[row * 4 + 2 * pr] = f2d(cf(ap.x * rp, ap.y * rp));
    if (fq) ws.U[row * 4 + 2 * pr + 1] = f2d(cf(aq.x * rq, aq.y * rq));
    if (row == 0) {
      ws.sig[2 * pr] = al * rp;
      ws.sig[2 * pr + 1] = be * rq;
      ws.rsig[2 * pr] = rp;
      ws.rsig[2 * pr + 1] = rq;
    }
  }
  __syncwarp();
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  const double eye = i == j && part == 0 ? 1.0 : 0.0;
  // V <- V (3I - V^H V) / 2
  double v = wmm_part<true, false>(ws.V, ws.V, i, j, part);
  wmm_store(ws.T, lane, 1.5 * eye - 0.5 * v);
  __syncwarp();
  v = wmm_part<false, false>(ws.V, ws.T, i, j, part);
  __syncwarp();
  wmm_store(ws.V, lane, v);
  __syncwarp();
  // U: the columns of E V over their norms (null columns are already there)
  v = wmm_part<false, false>(ws.E, ws.V, i, j, part);
  if (!((nmask >> j) & 1)) wmm_store(ws.U, lane, v * (double)ws.rsig[j]);
  __syncwarp();
  // polar factor of U Sigma to first order in D = U^H U - I:
  // U - U Z, Z_ij = s_i D_ij / (s_i + s_j); a null column yields to the others
  v = wmm_part<true, false>(ws.U, ws.U, i, j, part) - eye;
  {
    const bool ni = (nmask >> i) & 1, nj = (nmask >> j) & 1;
    const float si = ws.sig[i], sj = ws.sig[j];
    const float wgt = ni == nj ? (ni || i == j ? 0.5f : __fdividef(si, si + sj)) : (nj ? 1.f : 0.f);
    wmm_store(ws.T, lane, eye - (double)wgt * v);
  }
  __syncwarp();
  v = wmm_part<false, false>(ws.U, ws.T, i, j, part);
  __syncwarp();
  wmm_store(ws.U, lane, v);
  __syncwarp();
  // W = U V^H, then W <- W (3I - W^H W) / 2
  v = wmm_part<false, true>(ws.U, ws.V, i, j, part);
  __syncwarp();
  wmm_store(ws.U, lane, v);
  __syncwarp();
  v = wmm_part<true, false>(ws.U, ws.U, i, j, part);
  wmm_store(ws.T, lane, 1.5 * eye - 0.5 * v);
  __syncwarp();
  v = wmm_part<false, false>(ws.U, ws.T, i, j, part);
  const bool in = i < m && j < m;
  if (in) reinterpret_cast<double*>(gate)[2 * (i * m + j) + part] = part ? -v : v;
  double tr = 0.0;
  if (want_trace) {
    const double2 e = ws.E[ent];
    tr = in ? v * (part ? e.y : e.x) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    tr *= unscale;
  }
  __syncwarp();
  return tr;
}

__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}

__device__ __forceinline__ double2 shfl_xor2(double2 v, int o) {
  return cd(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// 1 / sqrt(x) in FP64 for x in FP32's normal range: an FP32 seed and one
// third-order step (relative error about 1e-20 before rounding).
__device__ __forceinline__ double wp_rsqrt(double x) {
  const double r = (double)rsqrtf((float)x), h = fma(-x * r, r, 1.0);
  return fma(r * h, fma(0.375, h, 0.5), r);
}

#define WPX_TINY 1e-36f   // column norms^2 (of entries at most 1) below this are zero

// Hestenes sweeps on FP64 columns: lane bits 0-1 row, 2 pair, 3 matrix (A or
// V); the upper half warp repeats the lower one.  A pair rotates while the
// cosine of its columns is above 1e-15 (as jacobi_pair).  Returns 1 after an
// odd number of sweeps.
__device__ __forceinline__ int wx_sweeps(double2& xp, double2& xq, int& fp, int& fq, bool masked) {
  const int lane = threadIdx.x & 31;
  const bool hi = (lane & 4) != 0;
  int odd = 0;
  for (int sweep = 0; sweep < 60; ++sweep) {
    odd ^= 1;
    bool rot = false;
#pragma unroll
    for (int rd = 0; rd < 3; ++rd) {
      const double al = quad_sum(fma(xp.x, xp.x, xp.y * xp.y)), be = quad_sum(fma(xq.x, xq.x, xq.y * xq.y));
      const double gx = quad_sum(fma(xp.x, xq.x, xp.y * xq.y)), gy = quad_sum(fma(xp.x, xq.y, -xp.y * xq.x));
      const float fa = (float)al, fb = (float)be;
      const bool live = fa > WPX_TINY && fb > WPX_TINY && (!masked || (fp && fq));
      const float rr = rsqrtf(live ? fa : 1.f) * rsqrtf(live ? fb : 1.f);
      const float cx = (float)gx * rr, cy = (float)gy * rr, c2 = fmaf(cx, cx, cy * cy);
      const bool go = live && c2 > 1e-30f && !(lane & 8);
      const float ri = rsqrtf(go ? c2 : 1.f);
      const float zeta = 0.5f * (float)(be - al) * rr * ri, az = fabsf(zeta);
      const float s1 = fmaf(az, az, 1.f);
      float t = az > 1e4f ? __fdividef(0.5f, az) : __fdividef(1.f, az + s1 * rsqrtf(s1));
      t = go ? copysignf(t, zeta) * ri : 0.f;
      // the columns of V follow those of A
      const double wx = (double)__shfl_sync(0xffffffffu, cx * t, lane & 7);
      const double wy = (double)__shfl_sync(0xffffffffu, cy * t, lane & 7);
      rot |= go && t != 0.f;
      if (__any_sync(0xffffffffu, go)) {
        const double c = wp_rsqrt(fma(wx, wx, fma(wy, wy, 1.0))), sx = c * wx, sy = c * wy;
        const double2 np = cd(fma(c, xp.x, -fma(sx, xq.x, sy * xq.y)), fma(c, xp.y, -fma(sx, xq.y, -sy * xq.x)));
        const double2 nq = cd(fma(c, xq.x, fma(sx, xp.x, -sy * xp.y)), fma(c, xq.y, fma(sx, xp.y, sy * xp.x)));
        xp = np;
        xq = nq;
      }
      const bool give_p = rd != 1 && hi;   // next pairing, as in wh_sweeps
      const double2 o = shfl_xor2(give_p ? xp : xq, 4);
      const int fo = masked ? __shfl_xor_sync(0xffffffffu, give_p ? fp : fq, 4) : 0;
      if (give_p) {
        xp = o;
        fp = fo;
      } else {
        xq = o;
        fq = fo;
      }
    }
    if (!__any_sync(0xffffffffu, rot)) break;
  }
  return odd;
}

static __device__ __noinline__ double wp_single_thread_exact(const WarpPolar& ws, double2* gate, int m) {
  double2 e[16], w[16], wprev[16];
  for (int i = 0; i < m * m; ++i) {
    e[i] = ws.E[(i / m) * 4 + i % m];
    wprev[i] = ws.Wp[(i / m) * 4 + i % m];
  }
  const double nn = polar_jacobi_pre(e, m, w, wprev);
  for (int i = 0; i < m * m; ++i) gate[i] = cconj(w[i]);
  return nn;
}

// As warp_polar, to FP64 accuracy; returns the nuclear norm of env.
static __device__ __noinline__ double warp_polar_exact(WarpPolar& ws, const double2* env, double2* gate, int m,
                                                       bool* finite) {
  const int lane = threadIdx.x & 31;
  const int ex = wp_load(ws, env, gate, m, lane, finite);
  if (!*finite) return 0.0;
  const double unscale = __hiloint2double((1023 + ex) << 20, 0);
  const int row = lane & 3, pr = (lane >> 2) & 1, ip = row * 4 + 2 * pr, iq = ip + 1;
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  const double eye = i == j && part == 0 ? 1.0 : 0.0;
  int fp = 0, fq = 0;
  {
    float2 ap = cf((float)ws.E[ip].x, (float)ws.E[ip].y), aq = cf((float)ws.E[iq].x, (float)ws.E[iq].y);
    float2 vp = cf(row == 2 * pr ? 1.f : 0.f, 0.f), vq = cf(row == 2 * pr + 1 ? 1.f : 0.f, 0.f);
    wh_sweeps(ap, aq, vp, vq, fp, fq, false);
    if (lane < 8) {
      ws.V[ip] = f2d(vp);
      ws.V[iq] = f2d(vq);
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int step = 0; step < 2; ++step) {   // V <- V (3I - V^H V) / 2: 1e-6, 1e-12, rounding
    double v = wmm_part<true, false>(ws.V, ws.V, i, j, part);
    wmm_store(ws.T, lane, 1.5 * eye - 0.5 * v);
    __syncwarp();
    v = wmm_part<false, false>(ws.V, ws.T, i, j, part);
    __syncwarp();
    wmm_store(ws.V, lane, v);
    __syncwarp();
  }
  wmm_store(ws.U, lane, wmm_part<false, false>(ws.E, ws.V, i, j, part));
  __syncwarp();
  double2* mine = (lane & 8) ? ws.V : ws.U;
  double2 xp = mine[ip], xq = mine[iq];
  wx_sweeps(xp, xq, fp, fq, false);
  // norms of A's columns, in every lane of their pair
  double al = quad_sum(cnorm2(xp)), be = quad_sum(cnorm2(xq));
  al = __shfl_sync(0xffffffffu, al, lane & 7);
  be = __shfl_sync(0xffffffffu, be, lane & 7);
  double m2 = fmax(al, be);
  m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, 4));
  const double thr = fmax(QM_POLAR_NULL_TOL * QM_POLAR_NULL_TOL * m2, (double)WPX_TINY);
  fp = !(al > thr);
  fq = !(be > thr);
  const double ra = wp_rsqrt(al > WPX_TINY ? al : 1.0), rb = wp_rsqrt(be > WPX_TINY ? be : 1.0);
  double nuc = (al > WPX_TINY ? al * ra : 0.0) + (be > WPX_TINY ? be * rb : 0.0);
  nuc += __shfl_xor_sync(0xffffffffu, nuc, 4);
  if (m == 2) nuc -= 2.0 * ws.E[10].x;   // the padding's two singular values
  const bool any_null = __any_sync(0xffffffffu, fp || fq);
  if (lane < 16) {
    const bool a = lane < 8;
    mine[ip] = a ? (fp ? czero() : cscale(xp, ra)) : xp;
    mine[iq] = a ? (fq ? czero() : cscale(xq, rb)) : xq;
  }
  __syncwarp();
  if (any_null) {
    // null columns of U: X = (I - U_s U_s^H) Wp V_N rotated to orthogonal columns
    wmm_store(ws.T, lane, wmm_part<false, false>(ws.Wp, ws.V, i, j, part));
    __syncwarp();
    wmm_store(ws.C, lane, wmm_part<true, false>(ws.U, ws.T, i, j, part));
    __syncwarp();
    const double x = reinterpret_cast<double*>(ws.T)[lane] - wmm_part<false, false>(ws.U, ws.C, i, j, part);
    __syncwarp();
    wmm_store(ws.T, lane, x);
    __syncwarp();
    if (!(lane & 8)) {
      xp = fp ? ws.T[ip] : ws.U[ip];
      xq = fq ? ws.T[iq] : ws.U[iq];
    }
    wx_sweeps(xp, xq, fp, fq, true);
    al = quad_sum(cnorm2(xp));
    be = quad_sum(cnorm2(xq));
    if (!__all_sync(0xffffffffu, (lane & 8) || ((!fp || al > 1e-16) && (!fq || be > 1e-16)))) {
      const double nn = lane == 0 ? wp_single_thread_exact(ws, gate, m) : 0.0;
      __syncwarp();
      return __shfl_sync(0xffffffffu, nn, 0) * unscale;
    }
    if (lane < 16) {
      const bool a = lane < 8;
      mine[ip] = a && fp ? cscale(xp, wp_rsqrt(al)) : xp;
      mine[iq] = a && fq ? cscale(xq, wp_rsqrt(be)) : xq;
    }
    __syncwarp();
  }
  const double v = wmm_part<false, true>(ws.U, ws.V, i, j, part);
  if (i < m && j < m) reinterpret_cast<double*>(gate)[2 * (i * m + j) + part] = part ? -v : v;
  __syncwarp();
  return nuc * unscale;
}

// s += the partner lane's `give` (lane ^ o), double-float
__device__ __forceinline__ void df_shfl_add(DF& s, const DF& give, int o) {
  df_add(s, __shfl_xor_sync(0xffffffffu, give.hi, o), __shfl_xor_sync(0xffffffffu, give.lo, o));
}

// Sum of 32 double-float values per lane over the warp: lane l returns the
// total of value l (exchange as warp_sum32).
__device__ __forceinline__ double warp_sum32_df(DF (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const DF give = up ? v[i] : v[i + o];
      if (up) v[i] = v[i + o];
      df_shfl_add(v[i], give, o);
    }
  }
  return (double)v[0].hi + (double)v[0].lo;
}

// Sum of 32 values per lane over the warp: lane l returns the total of
// value l.  Halving exchange (31 shuffles; the same pairwise order as a
// butterfly per value, which takes 160).
__device__ __forceinline__ float warp_sum32(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float give = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0];
}
