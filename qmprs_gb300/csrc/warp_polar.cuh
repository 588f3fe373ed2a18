// Unitary polar factor of a 4 x 4 (or 2 x 2) environment by one warp
// (warp_polar for the fast mode, warp_polar_exact for the exact mode), and
// the eigenvectors of the layer stage's 4 x 4 Grams (warp_gram_vectors).
//
// The definition is that of polar_sweep / polar_jacobi_pre in
// small_linalg.h: W maximises Re Tr(W^H E), singular values up to
// QM_POLAR_NULL_TOL of the largest count as zero, and on that null space W is
// the completion nearest to the current gate's.  One thread's chain of
// dependent FP32 and FP64 operations bounded every sweep step, so the algebra
// is spread over the lanes and kept off the FP64 units: GB300 issues an FP64
// warp instruction every 64 cycles whatever its active lanes, an FP32 one
// every cycle, and a double-float multiply-add (2^-46) is 12 FP32 ones.
//   * One-sided (Hestenes) Jacobi: lane (pair, row) holds one row of two
//     columns; the two pairs of a round rotate at once and a swap of columns
//     between the pairs gives the next round, so a cyclic sweep is three
//     rounds.  A rotation's angle comes from FP32 as a complex tangent w =
//     g / (|d| + sqrt(d^2 + |g|^2)), d half the difference of the norms^2, and
//     only c = 1 / sqrt(1 + |w|^2) in the columns' precision: every rotation
//     is unitary to that precision, and an inexact angle only leaves a little
//     for the next sweep.  Convergence is quadratic, so a precision's sweeps
//     end with the one whose tangents were all below the square root of what
//     is wanted.
//   * 4 x 4 products with one real or imaginary part of an entry per lane.
// The fast mode takes FP32 sweeps, then double-float products: V is made
// orthonormal, U is the first-order polar factor of E V's normalised columns,
// W = U V^H, and one FP64 Gram makes W unitary to rounding.  The error left
// is second order in the FP32 one.  The exact mode goes on with double-float
// sweeps and a first-order correction from FP64 Grams.
// A null space on which the current gate has no component either (rare)
// takes the single-thread code.
// Measured (cycles at full rank / rank 2): single-thread fast factor about
// 80000; the same sweeps spread over the lanes, in FP64, 16500 / 18500, exact
// 45900 / 66500; with the double-float sweeps fast 7400 / 9900, exact 15700 /
// 31500, Gram eigenvectors 17000 (45000 in FP64).
#pragma once

#include "dfloat.cuh"

struct WarpPolar {
  xc E[16];               // the matrix, scaled by a power of two, padded to 4 x 4
  xc V[16], U[16];
  double2 D[16];          // the matrix in FP64 (exact mode, Grams)
  double2 A[16], B[16], C[16];
  float2 T[16];
  float sig[4], rsig[4];  // column norms of E V and their reciprocals; 0 for null columns
  DF sq[4], rs[4];        // norms^2 and reciprocal norms in double-float (exact mode, Grams)
};

// ---- 4 x 4 products, one part (0 real, 1 imaginary) of entry (i, j) per lane ----------

// op(A) op(B) in FP64, row-major in shared memory; op is the adjoint where ADJ.
template <bool ADJ_A, bool ADJ_B>
__device__ __forceinline__ double wmm_part(const double2* A, const double2* B, int i, int j, int part) {
  double acc[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double s = 0.0;
#pragma unroll
    for (int k = 2 * h; k < 2 * h + 2; ++k) {
      const double2 a = ADJ_A ? cconj(A[k * 4 + i]) : A[i * 4 + k];
      const double2 b = ADJ_B ? cconj(B[j * 4 + k]) : B[k * 4 + j];
      const double b0 = part ? b.y : b.x, b1 = part ? b.x : -b.y;
      s = k == 2 * h ? a.x * b0 : fma(a.x, b0, s);
      s = fma(a.y, b1, s);
    }
    acc[h] = s;
  }
  return acc[0] + acc[1];
}

__device__ __forceinline__ void wmm_store(double2* C, int lane, double v) {
  reinterpret_cast<double*>(C)[lane] = v;   // lane = 2 * entry + part
}

// The same in double-float.
template <bool ADJ_A, bool ADJ_B>
__device__ __forceinline__ DF wdf_part(const xc* A, const xc* B, int i, int j, int part) {
  DF s = {0.f, 0.f};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const xc a = ADJ_A ? xc_conj(A[k * 4 + i]) : A[i * 4 + k];
    const xc b = ADJ_B ? xc_conj(B[j * 4 + k]) : B[k * 4 + j];
    df_mac(s, a.x, a.z, part ? b.y : b.x, part ? b.w : b.z);
    df_mac(s, a.y, a.w, part ? b.x : -b.y, part ? b.z : -b.w);
  }
  return s;
}

__device__ __forceinline__ void wdf_store(xc* M, int lane, DF s) {
  const float2 v = df_norm(s);
  float* e = reinterpret_cast<float*>(M + (lane >> 1));
  e[lane & 1] = v.x;
  e[(lane & 1) + 2] = v.y;
}

__device__ __forceinline__ DF wdf_load(const xc* M, int lane) {
  const float* e = reinterpret_cast<const float*>(M + (lane >> 1));
  return DF{e[lane & 1], e[(lane & 1) + 2]};
}

// A T in FP32, A the rounding of a double-float or FP64 matrix.
__device__ __forceinline__ float2 wf_entry(const xc& a) { return cf(a.x, a.y); }
__device__ __forceinline__ float2 wf_entry(const double2& a) { return cf((float)a.x, (float)a.y); }
__device__ __forceinline__ float2 wf_entry(const float2& a) { return a; }
template <class M>
__device__ __forceinline__ float wf_part(const M* A, const float2* T, int i, int j, int part) {
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 a = wf_entry(A[i * 4 + k]), b = T[k * 4 + j];
    s = fmaf(a.x, part ? b.y : b.x, s);
    s = fmaf(a.y, part ? b.x : -b.y, s);
  }
  return s;
}

__device__ __forceinline__ void wf_store(float2* T, int lane, float v) { reinterpret_cast<float*>(T)[lane] = v; }

// M <- M + M T for a small T (double-float M, FP32 product); M T's rounding
// is 2^-24 of it.
__device__ __forceinline__ void wdf_correct(xc* M, const float2* T, int lane) {
  const int ent = lane >> 1;
  DF s = wdf_load(M, lane);
  df_add(s, wf_part(M, T, ent >> 2, ent & 3, lane & 1), 0.f);
  __syncwarp();
  wdf_store(M, lane, s);
  __syncwarp();
}

// T <- (I - M^H M) / 2 in FP32 of a nearly orthonormal FP64 M (16 real
// values, two lanes each: five FP64 operations instead of eleven).
__device__ __forceinline__ void wp_gram_defect(const double2* M, float2* T, int lane) {
  const int v = lane >> 1, h = lane & 1;
  // values 0-3: diagonal; then real and imaginary parts of (0,1), (0,2), (0,3), (1,2), (1,3), (2,3)
  const int p = (v - 4) >> 1;
  const int a = v < 4 ? v : p < 3 ? 0 : p < 5 ? 1 : 2, e = v < 4 ? v : p < 3 ? p + 1 : p < 5 ? p - 1 : 3;
  const bool im = v >= 4 && (v & 1);
  const double2 a0 = M[(2 * h) * 4 + a], e0 = M[(2 * h) * 4 + e], a1 = M[(2 * h + 1) * 4 + a],
                e1 = M[(2 * h + 1) * 4 + e];
  // conj(a) e
  double s = a0.x * (im ? e0.y : e0.x);
  s = fma(im ? -a0.y : a0.y, im ? e0.x : e0.y, s);
  s = fma(a1.x, im ? e1.y : e1.x, s);
  s = fma(im ? -a1.y : a1.y, im ? e1.x : e1.y, s);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if (h == 0) {
    float* t = reinterpret_cast<float*>(T);
    if (v < 4) {
      t[2 * (a * 4 + a)] = (float)(0.5 - 0.5 * s);
      t[2 * (a * 4 + a) + 1] = 0.f;
    } else {
      const float d = -0.5f * (float)s;
      t[2 * (a * 4 + e) + (im ? 1 : 0)] = d;
      t[2 * (e * 4 + a) + (im ? 1 : 0)] = im ? -d : d;
    }
  }
  __syncwarp();
}

// ---- Hestenes sweeps -------------------------------------------------------------------

__device__ __forceinline__ float quad_sum(float v) {   // over the four rows of a column
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}
// s += the partner lane's `give` (lane ^ o), double-float
__device__ __forceinline__ void df_shfl_add(DF& s, const DF& give, int o) {
  df_add(s, __shfl_xor_sync(0xffffffffu, give.hi, o), __shfl_xor_sync(0xffffffffu, give.lo, o));
}
__device__ __forceinline__ DF quad_sum(DF v) {
  df_shfl_add(v, v, 1);
  df_shfl_add(v, v, 2);
  return v;
}

__device__ __forceinline__ float2 shfl_xor2(float2 v, int o) {
  return cf(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ double2 shfl_xor2(double2 v, int o) {
  return cd(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ xc shfl_xor2(xc v, int o) {
  return make_float4(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o),
                     __shfl_xor_sync(0xffffffffu, v.z, o), __shfl_xor_sync(0xffffffffu, v.w, o));
}

// Next pairing of columns: rounds 0 and 2 swap q of pair 0 with p of pair 1,
// round 1 swaps the two q; three rounds meet all six pairs and leave columns
// 2 and 3 exchanged.  Flags move with their columns.
template <class T>
__device__ __forceinline__ void wh_swap(T& p, T& q, bool give_p) {
  const T o = shfl_xor2(give_p ? p : q, 4);
  if (give_p) p = o;
  else q = o;
}
__device__ __forceinline__ void wh_swap_flags(int& fp, int& fq, bool give_p) {
  const int o = __shfl_xor_sync(0xffffffffu, give_p ? fp : fq, 4);
  if (give_p) fp = o;
  else fq = o;
}

// Which pairs rotate: all, only pairs of flagged columns, or all but those.
enum { WH_ALL = 0, WH_FLAGGED = 1, WH_OTHERS = 2 };
__device__ __forceinline__ bool wh_allowed(int which, int fp, int fq) {
  return which == WH_ALL || (which == WH_FLAGGED) == (fp && fq);
}

// The complex tangent of a pair: d half the difference of the norms^2, g
// the inner product, both over any common scale.
__device__ __forceinline__ float2 wh_tangent(float d, float gx, float gy, bool go) {
  const float h = fmaf(d, d, fmaf(gx, gx, gy * gy));
  go = go && h > 1e-36f;
  const float hh = go ? h : 1.f;
  const float f = copysignf(__fdividef(1.f, fabsf(d) + hh * rsqrtf(hh)), d);
  return go ? cf(gx * f, gy * f) : cf(0.f, 0.f);
}

__device__ __forceinline__ void wh_apply(float2& p, float2& q, float c, float sx, float sy) {
  // p <- c p - s conj(e) q ; q <- s e p + c q
  const float2 np = cf(c * p.x - fmaf(sx, q.x, sy * q.y), c * p.y - fmaf(sx, q.y, -sy * q.x));
  const float2 nq = cf(fmaf(c, q.x, fmaf(sx, p.x, -sy * p.y)), fmaf(c, q.y, fmaf(sx, p.y, sy * p.x)));
  p = np;
  q = nq;
}

// FP32 sweeps of the four columns: lane l & 7 = 4 pair + row holds rows of
// columns p and q of A and V.  A pair rotates while |g|^2 > 1e-12 al be (as
// jacobi_pair_f); the last sweep is the one whose tangents were all below
// 3e-4.  Returns 1 after an odd number of sweeps, which leaves columns 2 and
// 3 exchanged.
__device__ __forceinline__ int wh_sweeps(float2& ap, float2& aq, float2& vp, float2& vq, int& fp, int& fq, int which) {
  const bool hi = (threadIdx.x & 4) != 0;   // the second pair's lanes
  int odd = 0;
  for (int sweep = 0; sweep < 30; ++sweep) {
    odd ^= 1;
    bool more = false;
#pragma unroll
    for (int rd = 0; rd < 3; ++rd) {
      const float al = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y)), be = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
      const float gx = quad_sum(fmaf(ap.x, aq.x, ap.y * aq.y)), gy = quad_sum(fmaf(ap.x, aq.y, -ap.y * aq.x));
      const bool go = wh_allowed(which, fp, fq) && fmaf(gx, gx, gy * gy) > 1e-12f * al * be;
      const float2 w = wh_tangent(0.5f * (be - al), gx, gy, go);
      const float w2 = fmaf(w.x, w.x, w.y * w.y), c = rsqrtf(1.f + w2);
      more |= w2 > 1e-7f;
      wh_apply(ap, aq, c, c * w.x, c * w.y);
      wh_apply(vp, vq, c, c * w.x, c * w.y);
      const bool give_p = rd != 1 && hi;
      wh_swap(ap, aq, give_p);
      wh_swap(vp, vq, give_p);
      if (which != WH_ALL) wh_swap_flags(fp, fq, give_p);
    }
    if (!__any_sync(0xffffffffu, more)) break;
  }
  return odd;
}

#define WPX_TINY 1e-36f   // column norms^2 (of entries at most 1) below this are zero

// c = 1 / sqrt(1 + |w|^2) in double-float: an FP32 seed and one third-order
// step with the residual from exact products.
__device__ __forceinline__ DF wd_cosine(float2 w) {
  DF q = {0.f, 0.f};
  df_add_prod(q, w.x, w.x);
  df_add_prod(q, w.y, w.y);
  const float r = rsqrtf(1.f + q.hi);
  const float ph = __fmul_rn(r, r), pl = __fmaf_rn(r, r, -ph);
  const float m = __fmul_rn(q.hi, ph), ml = __fmaf_rn(q.hi, ph, -m);
  const float h = __fsub_rn(__fsub_rn(__fsub_rn(1.f, ph), m), pl + ml + fmaf(q.lo, ph, q.hi * pl));
  DF c = {r, r * h * fmaf(0.375f, h, 0.5f)};
  const float2 n = df_norm(c);
  return DF{n.x, n.y};
}

// Sweeps on double-float columns: lane bits 0-1 row, 2 pair, 3 matrix (A or
// V, which follows A's rotations); the upper half warp repeats the lower
// one.  A pair rotates while its columns' cosine is above 1e-13; the last
// sweep is the one whose tangents were all below 1e-6.
__device__ __forceinline__ int wd_sweeps(xc& xp, xc& xq, int& fp, int& fq, int which) {
  const int lane = threadIdx.x & 31;
  const bool hi = (lane & 4) != 0;
  int odd = 0;
#pragma unroll 1
  for (int sweep = 0; sweep < 30; ++sweep) {
    odd ^= 1;
    bool more = false;
#pragma unroll 1
    for (int rd = 0; rd < 3; ++rd) {
      const float al = quad_sum(fmaf(xp.x, xp.x, xp.y * xp.y)), be = quad_sum(fmaf(xq.x, xq.x, xq.y * xq.y));
      DF d = {0.f, 0.f}, gx = {0.f, 0.f}, gy = {0.f, 0.f};
      df_mac(d, xq.x, xq.z, xq.x, xq.z);
      df_mac(d, xq.y, xq.w, xq.y, xq.w);
      df_mac(d, -xp.x, -xp.z, xp.x, xp.z);
      df_mac(d, -xp.y, -xp.w, xp.y, xp.w);
      df_mac(gx, xp.x, xp.z, xq.x, xq.z);
      df_mac(gx, xp.y, xp.w, xq.y, xq.w);
      df_mac(gy, xp.x, xp.z, xq.y, xq.w);
      df_mac(gy, -xp.y, -xp.w, xq.x, xq.z);
      d = quad_sum(d);
      gx = quad_sum(gx);
      gy = quad_sum(gy);
      const bool live = al > WPX_TINY && be > WPX_TINY;
      const float rr = rsqrtf(live ? al : 1.f) * rsqrtf(live ? be : 1.f);
      const float cx = (gx.hi + gx.lo) * rr, cy = (gy.hi + gy.lo) * rr;
      const bool go = live && wh_allowed(which, fp, fq) && fmaf(cx, cx, cy * cy) > 1e-26f;
      float2 w = wh_tangent(0.5f * (d.hi + d.lo) * rr, cx, cy, go);
      w = cf(__shfl_sync(0xffffffffu, w.x, lane & 7), __shfl_sync(0xffffffffu, w.y, lane & 7));
      more |= fmaf(w.x, w.x, w.y * w.y) > 1e-12f;
      const DF c = wd_cosine(w);
      const float sxh = __fmul_rn(c.hi, w.x), sxl = __fmaf_rn(c.hi, w.x, -sxh) + c.lo * w.x;
      const float syh = __fmul_rn(c.hi, w.y), syl = __fmaf_rn(c.hi, w.y, -syh) + c.lo * w.y;
      XA np = xa_zero(), nq = xa_zero();
      df_mac(np.re, c.hi, c.lo, xp.x, xp.z);
      df_mac(np.re, -sxh, -sxl, xq.x, xq.z);
      df_mac(np.re, -syh, -syl, xq.y, xq.w);
      df_mac(np.im, c.hi, c.lo, xp.y, xp.w);
      df_mac(np.im, -sxh, -sxl, xq.y, xq.w);
      df_mac(np.im, syh, syl, xq.x, xq.z);
      df_mac(nq.re, c.hi, c.lo, xq.x, xq.z);
      df_mac(nq.re, sxh, sxl, xp.x, xp.z);
      df_mac(nq.re, -syh, -syl, xp.y, xp.w);
      df_mac(nq.im, c.hi, c.lo, xq.y, xq.w);
      df_mac(nq.im, sxh, sxl, xp.y, xp.w);
      df_mac(nq.im, syh, syl, xp.x, xp.z);
      xp = xa_round(np);
      xq = xa_round(nq);
      const bool give_p = rd != 1 && hi;
      wh_swap(xp, xq, give_p);
      wh_swap_flags(fp, fq, give_p);
    }
    if (!__any_sync(0xffffffffu, more)) break;
  }
  return odd;
}

// 1 / sqrt(x) in FP64 for x in FP32's normal range: an FP32 seed and one
// third-order step (relative error about 1e-20 before rounding).
__device__ __forceinline__ double wp_rsqrt(double x) {
  const double r = (double)rsqrtf((float)x), h = fma(-x * r, r, 1.0);
  return fma(r * h, fma(0.375, h, 0.5), r);
}

// Sweeps on FP64 columns (lanes as wd_sweeps): the polish of columns that
// are orthogonal to double-float.  A pair rotates while its columns' cosine
// is above 1e-15 (as jacobi_pair); tangents up to 3e-9 have c = 1 to
// rounding; the last sweep is the one whose tangents were all below 1e-8.
__device__ __forceinline__ int wx_sweeps(double2& xp, double2& xq, int& fp, int& fq, int which) {
  const int lane = threadIdx.x & 31;
  const bool hi = (lane & 4) != 0;
  int odd = 0;
#pragma unroll 1
  for (int sweep = 0; sweep < 60; ++sweep) {
    odd ^= 1;
    bool more = false;
#pragma unroll 1
    for (int rd = 0; rd < 3; ++rd) {
      const float2 p32 = cf((float)xp.x, (float)xp.y), q32 = cf((float)xq.x, (float)xq.y);
      const float al = quad_sum(fmaf(p32.x, p32.x, p32.y * p32.y)), be = quad_sum(fmaf(q32.x, q32.x, q32.y * q32.y));
      const double gx = quad_sum(fma(xp.x, xq.x, xp.y * xq.y)), gy = quad_sum(fma(xp.x, xq.y, -xp.y * xq.x));
      const double d = quad_sum(fma(xq.x, xq.x, fma(xq.y, xq.y, fma(-xp.x, xp.x, -xp.y * xp.y))));
      const bool live = al > WPX_TINY && be > WPX_TINY;
      const float rr = rsqrtf(live ? al : 1.f) * rsqrtf(live ? be : 1.f);
      const float cx = (float)gx * rr, cy = (float)gy * rr;
      const bool go = live && wh_allowed(which, fp, fq) && fmaf(cx, cx, cy * cy) > 1e-30f;
      float2 w = wh_tangent(0.5f * (float)d * rr, cx, cy, go);
      w = cf(__shfl_sync(0xffffffffu, w.x, lane & 7), __shfl_sync(0xffffffffu, w.y, lane & 7));
      const float w2 = fmaf(w.x, w.x, w.y * w.y);
      more |= w2 > 1e-16f;
      const double wx = (double)w.x, wy = (double)w.y;
      if (__any_sync(0xffffffffu, w2 > 1e-17f)) {
        const double c = wp_rsqrt(fma(wx, wx, fma(wy, wy, 1.0))), sx = c * wx, sy = c * wy;
        const double2 np = cd(fma(c, xp.x, -fma(sx, xq.x, sy * xq.y)), fma(c, xp.y, -fma(sx, xq.y, -sy * xq.x)));
        const double2 nq = cd(fma(c, xq.x, fma(sx, xp.x, -sy * xp.y)), fma(c, xq.y, fma(sx, xp.y, sy * xp.x)));
        xp = np;
        xq = nq;
      } else if (__any_sync(0xffffffffu, w2 > 0.f)) {
        const double2 np = cd(fma(-wx, xq.x, fma(-wy, xq.y, xp.x)), fma(-wx, xq.y, fma(wy, xq.x, xp.y)));
        const double2 nq = cd(fma(wx, xp.x, fma(-wy, xp.y, xq.x)), fma(wx, xp.y, fma(wy, xp.x, xq.y)));
        xp = np;
        xq = nq;
      }
      const bool give_p = rd != 1 && hi;
      wh_swap(xp, xq, give_p);
      wh_swap_flags(fp, fq, give_p);
    }
    if (!__any_sync(0xffffffffu, more)) break;
  }
  return odd;
}

// ---- the matrix -------------------------------------------------------------------------

// Scale the m x m environment (row-major, double-float) into ws.E: times a
// power of two that brings the largest part into [1/2, 1); a 2 x 2 one is
// padded with its largest part on the diagonal (neither null nor larger than
// its norm).  Returns the exponent; *finite is false if any entry is not.
__device__ __forceinline__ int wp_load(WarpPolar& ws, const xc* env, int m, int lane, bool* finite) {
  const int r = (lane >> 2) & 3, c = lane & 3;
  const bool in = r < m && c < m;
  const xc e = in ? env[r * m + c] : make_float4(0.f, 0.f, 0.f, 0.f);
  *finite = __all_sync(0xffffffffu, isfinite(e.x) && isfinite(e.y) && isfinite(e.z) && isfinite(e.w));
  const int mbits = __reduce_max_sync(0xffffffffu, __float_as_int(fmaxf(fabsf(e.x), fabsf(e.y))));
  const int ex = mbits == 0 ? 0 : min(max((mbits >> 23) - 126, -125), 126);
  const float sc = __int_as_float((127 - ex) << 23);
  const float pad = r == c && m < 4 ? __int_as_float(mbits) * sc : 0.f;
  if (lane < 16) ws.E[lane] = in ? make_float4(e.x * sc, e.y * sc, e.z * sc, e.w * sc) : make_float4(pad, 0.f, 0.f, 0.f);
  __syncwarp();
  return ex;
}

// The same of an FP64 environment: ws.D, and its double-float rounding in
// ws.E.
__device__ __forceinline__ int wp_load(WarpPolar& ws, const double2* env, int m, int lane, bool* finite) {
  const int r = (lane >> 2) & 3, c = lane & 3;
  const bool in = r < m && c < m;
  const double2 e = in ? env[r * m + c] : czero();
  *finite = __all_sync(0xffffffffu, isfinite(e.x) && isfinite(e.y));
  const int hx = __double2hiint(e.x) & 0x7fffffff, hy = __double2hiint(e.y) & 0x7fffffff;
  const int mbits = __reduce_max_sync(0xffffffffu, max(hx, hy));
  const int ex = mbits == 0 ? 0 : min(max((mbits >> 20) - 1022, -1000), 1000);
  // times 2^-ex by the exponents (an FP64 product takes 64 cycles); what would
  // leave the normal range is far below the others' rounding, and what is not
  // finite stays so
  auto scaled = [ex](double v) {
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    if (e == 0x7ff) return v;
    return e > 0 && e > ex ? __hiloint2double(__double2hiint(v) - ex * (1 << 20), __double2loint(v)) : 0.0;
  };
  const double pad = r == c && m < 4 ? scaled(__hiloint2double(mbits, 0)) : 0.0;
  const double2 d = in ? cd(scaled(e.x), scaled(e.y)) : cd(pad, 0.0);
  if (lane < 16) {
    ws.D[lane] = d;
    ws.E[lane] = xc_split(d);
  }
  __syncwarp();
  return ex;
}

__device__ __forceinline__ double wp_unscale(int ex) { return __hiloint2double((1023 + ex) << 20, 0); }

// Entry (r, c) of the current gate's conjugate, padded with the identity.
__device__ __forceinline__ double2 wp_gate(const double2* gate, int m, int r, int c) {
  return r < m && c < m ? cconj(gate[r * m + c]) : cd(r == c ? 1.0 : 0.0, 0.0);
}

// FP32 columns of ws.E and V = I in their lanes.
__device__ __forceinline__ void wp_columns(const WarpPolar& ws, int lane, float2& ap, float2& aq, float2& vp, float2& vq) {
  const int row = lane & 3, ip = row * 4 + 2 * ((lane >> 2) & 1);
  ap = cf(ws.E[ip].x, ws.E[ip].y);
  aq = cf(ws.E[ip + 1].x, ws.E[ip + 1].y);
  vp = cf(ip % 4 == row ? 1.f : 0.f, 0.f);
  vq = cf(ip % 4 + 1 == row ? 1.f : 0.f, 0.f);
}

// T <- (I - V^H V) / 2 in FP32 of a double-float V; with `second` plus 3/2 of
// its square, so that V + V T is orthonormal to third order.
__device__ __forceinline__ void wp_defect(WarpPolar& ws, int lane, bool second) {
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  const float eye = i == j && part == 0 ? 1.f : 0.f;
  const DF s = wdf_part<true, false>(ws.V, ws.V, i, j, part);
  const float d = 0.5f * ((eye - s.hi) - s.lo);
  wf_store(ws.T, lane, d);
  __syncwarp();
  if (second) {
    const float d2 = wf_part(ws.T, ws.T, i, j, part);
    __syncwarp();
    wf_store(ws.T, lane, fmaf(1.5f, d2, d));
    __syncwarp();
  }
}

// ---- fast mode -----------------------------------------------------------------------------

// Null columns (f set) of the orthogonalised A become X = (I - U_s U_s^H)
// Wp V_N, rotated among themselves to orthogonal columns; false if one of
// them vanishes (the caller takes the single-thread code).
__device__ __forceinline__ bool wp_null_columns(const double2* gate, int m, float2& ap, float2& aq, float2& vp,
                                                float2& vq, int& fp, int& fq, float al, float be, int lane) {
  const int row = lane & 3;
  float2 xp = cf(0.f, 0.f), xq = cf(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int src = (lane & ~3) | k;
    const double2 g = wp_gate(gate, m, row, k);
    const float2 w = cf((float)g.x, (float)g.y);
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
  wh_sweeps(ap, aq, vp, vq, fp, fq, WH_FLAGGED);
  const float np = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y)), nq = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
  return __all_sync(0xffffffffu, (!fp || np > 1e-8f) && (!fq || nq > 1e-8f));
}

// The single-thread factor of the workspace's m x m block, for one lane:
// writes the gate, returns Re Tr(W^H E) (fast) or the nuclear norm (exact) of
// the scaled environment.
template <bool EXACT>
__device__ __noinline__ double wp_single_thread(const WarpPolar& ws, double2* gate, int m) {
  double2 e[16], w[16], wprev[16];
  for (int i = 0; i < m * m; ++i) {
    e[i] = EXACT ? ws.D[(i / m) * 4 + i % m] : xc_to_d(ws.E[(i / m) * 4 + i % m]);
    wprev[i] = cconj(gate[i]);
  }
  const double nn = EXACT ? polar_jacobi_pre(e, m, w, wprev) : polar_sweep(e, m, w, wprev);
  for (int i = 0; i < m * m; ++i) gate[i] = cconj(w[i]);
  return nn;
}

// Polar factor of the m x m environment `env` (row-major, double-float) by
// the 32 lanes of a warp; `gate` (m x m, shared memory) holds the current
// gate G and receives conj(W).  Returns Re Tr(W^H E) in every lane when
// `want_trace`.  *finite is false (and nothing else is done) if env is not
// finite.
static __device__ __noinline__ double warp_polar(WarpPolar& ws, const xc* env, double2* gate, int m, bool want_trace,
                                                 bool* finite) {
  const int lane = threadIdx.x & 31;
  const int ex = wp_load(ws, env, m, lane, finite);
  if (!*finite) return 0.0;
  const int row = lane & 3, pr = (lane >> 2) & 1, ip = row * 4 + 2 * pr;
  float2 ap, aq, vp, vq;
  int fp = 0, fq = 0;
  wp_columns(ws, lane, ap, aq, vp, vq);
  wh_sweeps(ap, aq, vp, vq, fp, fq, WH_ALL);
  float al = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y)), be = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
  const float m2 = fmaxf(fmaxf(al, be), __shfl_xor_sync(0xffffffffu, fmaxf(al, be), 4));
  const float thr = (float)(QM_POLAR_NULL_TOL * QM_POLAR_NULL_TOL) * m2;
  fp = !(al > thr && al > 0.f);
  fq = !(be > thr && be > 0.f);
  if (__any_sync(0xffffffffu, fp || fq)) {
    if (!wp_null_columns(gate, m, ap, aq, vp, vq, fp, fq, al, be, lane)) {
      const double nn = lane == 0 ? wp_single_thread<false>(ws, gate, m) : 0.0;
      __syncwarp();
      return __shfl_sync(0xffffffffu, nn, 0) * wp_unscale(ex);
    }
    al = quad_sum(fmaf(ap.x, ap.x, ap.y * ap.y));
    be = quad_sum(fmaf(aq.x, aq.x, aq.y * aq.y));
  }
  // V and the null columns of U to shared memory, column order as it fell
  const unsigned nb_p = __ballot_sync(0xffffffffu, fp), nb_q = __ballot_sync(0xffffffffu, fq);
  const int nmask = (nb_p & 1) | ((nb_q & 1) << 1) | (((nb_p >> 4) & 1) << 2) | (((nb_q >> 4) & 1) << 3);
  if (lane < 8) {
    const float rp = rsqrtf(al), rq = rsqrtf(be);
    ws.V[ip] = make_float4(vp.x, vp.y, 0.f, 0.f);
    ws.V[ip + 1] = make_float4(vq.x, vq.y, 0.f, 0.f);
    if (fp) ws.U[ip] = make_float4(ap.x * rp, ap.y * rp, 0.f, 0.f);
    if (fq) ws.U[ip + 1] = make_float4(aq.x * rq, aq.y * rq, 0.f, 0.f);
    if (row == 0) {
      ws.sig[2 * pr] = al * rp;
      ws.sig[2 * pr + 1] = be * rq;
      ws.rsig[2 * pr] = rp;
      ws.rsig[2 * pr + 1] = rq;
    }
  }
  __syncwarp();
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  const float eye = i == j && part == 0 ? 1.f : 0.f;
  wp_defect(ws, lane, false);
  wdf_correct(ws.V, ws.T, lane);
  // U: the columns of E V over their norms (null columns are already there)
  {
    const DF b = wdf_part<false, false>(ws.E, ws.V, i, j, part);
    DF s = {0.f, 0.f};
    df_mac(s, b.hi, b.lo, ws.rsig[j], 0.f);
    if (!((nmask >> j) & 1)) wdf_store(ws.U, lane, s);
  }
  __syncwarp();
  // polar factor of U Sigma to first order in D = U^H U - I:
  // U - U Z, Z_ij = s_i D_ij / (s_i + s_j); a null column yields to the others
  {
    const DF s = wdf_part<true, false>(ws.U, ws.U, i, j, part);
    const float d = (s.hi - eye) + s.lo;
    const bool ni = (nmask >> i) & 1, nj = (nmask >> j) & 1;
    const float si = ws.sig[i], sj = ws.sig[j];
    const float wgt = ni == nj ? (ni || i == j ? 0.5f : __fdividef(si, si + sj)) : (nj ? 1.f : 0.f);
    wf_store(ws.T, lane, -wgt * d);
  }
  __syncwarp();
  wdf_correct(ws.U, ws.T, lane);
  // W = U V^H, then W + W (I - W^H W) / 2 with the defect from FP64
  const DF w0 = wdf_part<false, true>(ws.U, ws.V, i, j, part);
  const double wd = (double)w0.hi + (double)w0.lo;
  wmm_store(ws.A, lane, wd);
  __syncwarp();
  wp_gram_defect(ws.A, ws.T, lane);
  const double v = wd + (double)wf_part(ws.A, ws.T, i, j, part);
  const bool in = i < m && j < m;
  if (in) reinterpret_cast<double*>(gate)[2 * (i * m + j) + part] = part ? -v : v;
  double tr = 0.0;
  if (want_trace) {
    const DF e = wdf_load(ws.E, lane);
    tr = in ? v * ((double)e.hi + (double)e.lo) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    tr *= wp_unscale(ex);
  }
  __syncwarp();
  return tr;
}

// ---- exact mode and Grams --------------------------------------------------------------------

// Orthogonalise the columns of ws.E: FP32 sweeps, then double-float ones.
// xp, xq: the columns of A = E V and V in their lanes (wd_sweeps).  Returns
// the parity of the sweeps.
__device__ __forceinline__ int wp_df_columns(WarpPolar& ws, int lane, xc& xp, xc& xq) {
  const int ip = (lane & 3) * 4 + 2 * ((lane >> 2) & 1);
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  int fp = 0, fq = 0;
  float2 ap, aq, vp, vq;
  wp_columns(ws, lane, ap, aq, vp, vq);
  int odd = wh_sweeps(ap, aq, vp, vq, fp, fq, WH_ALL);
  if (lane < 8) {
    ws.V[ip] = make_float4(vp.x, vp.y, 0.f, 0.f);
    ws.V[ip + 1] = make_float4(vq.x, vq.y, 0.f, 0.f);
  }
  __syncwarp();
  wp_defect(ws, lane, true);
  wdf_correct(ws.V, ws.T, lane);
  const DF a = wdf_part<false, false>(ws.E, ws.V, i, j, part);
  wdf_store(ws.U, lane, a);
  __syncwarp();
  const xc* mine = (lane & 8) ? ws.V : ws.U;
  xp = mine[ip];
  xq = mine[ip + 1];
  odd ^= wd_sweeps(xp, xq, fp, fq, WH_ALL);
  return odd;
}

// Norms^2 and reciprocal norms (0 for flagged and for zero columns) of the
// double-float columns in lanes 0-7, to ws.sq and ws.rs.
__device__ __forceinline__ void wp_norms(WarpPolar& ws, int lane, xc xp, xc xq, int fp, int fq) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const xc x = k ? xq : xp;
    DF al = {0.f, 0.f};
    df_mac(al, x.x, x.z, x.x, x.z);
    df_mac(al, x.y, x.w, x.y, x.w);
    al = quad_sum(al);
    const bool live = al.hi > WPX_TINY && !(k ? fq : fp);
    const float r = rsqrtf(live ? al.hi : 1.f);
    const float ph = __fmul_rn(r, r), pl = __fmaf_rn(r, r, -ph);
    const float m = __fmul_rn(al.hi, ph), ml = __fmaf_rn(al.hi, ph, -m);
    const float h = __fsub_rn(1.f, m) - (ml + fmaf(al.lo, ph, al.hi * pl));
    if (lane < 8 && (lane & 3) == 0) {
      const int col = 2 * (lane >> 2) + k;
      ws.sq[col] = al;
      ws.rs[col] = live ? DF{r, r * h * fmaf(0.375f, h, 0.5f)} : DF{0.f, 0.f};
      ws.sig[col] = live ? al.hi * r : 0.f;
    }
  }
}

// FP64 from double-float: V (lanes 8-15 of vp, vq) orthonormal to rounding
// in ws.B, D V in ws.A, its columns over their norms (ws.rs) in ws.C, and
// T = (I - C^H C) / 2.
__device__ __forceinline__ void wp_to_fp64(WarpPolar& ws, int lane, xc vp, xc vq) {
  const int ip = (lane & 3) * 4 + 2 * ((lane >> 2) & 1);
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  if (lane >= 8 && lane < 16) {
    ws.B[ip] = xc_to_d(vp);
    ws.B[ip + 1] = xc_to_d(vq);
  }
  __syncwarp();
  wp_gram_defect(ws.B, ws.T, lane);
  const double v = reinterpret_cast<const double*>(ws.B)[lane] + (double)wf_part(ws.B, ws.T, i, j, part);
  __syncwarp();
  wmm_store(ws.B, lane, v);
  __syncwarp();
  const double a = wmm_part<false, false>(ws.D, ws.B, i, j, part);
  wmm_store(ws.A, lane, a);
  const DF r = ws.rs[j];
  wmm_store(ws.C, lane, a * ((double)r.hi + (double)r.lo));
  __syncwarp();
  wp_gram_defect(ws.C, ws.T, lane);
}

// M <- M + M T, FP64 with an FP32 product.
__device__ __forceinline__ void wmm_correct(double2* M, const float2* T, int lane) {
  const int ent = lane >> 1;
  const double v = reinterpret_cast<const double*>(M)[lane] + (double)wf_part(M, T, ent >> 2, ent & 3, lane & 1);
  __syncwarp();
  wmm_store(M, lane, v);
  __syncwarp();
}

// T (from wp_gram_defect of C) to the first-order polar correction of C
// Sigma: 2 w_ij T_ij, w_ij = s_i / (s_i + s_j); between a significant and a
// null column the null one yields, two null ones share.
__device__ __forceinline__ void wp_polar_weights(WarpPolar& ws, int lane, int nmask) {
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3;
  const bool ni = (nmask >> i) & 1, nj = (nmask >> j) & 1;
  const float si = ws.sig[i], sj = ws.sig[j];
  const float w = ni == nj ? (ni || i == j ? 1.f : __fdividef(2.f * si, si + sj)) : (nj ? 2.f : 0.f);
  const float t = w * reinterpret_cast<const float*>(ws.T)[lane];
  __syncwarp();
  wf_store(ws.T, lane, t);
  __syncwarp();
}

// As warp_polar, to FP64 accuracy and of an FP64 environment: with the columns
// orthogonal to double-float, one first-order correction (defects of about
// 1e-13 from FP64 Grams, products with them in FP32) reaches FP64 rounding.  Returns the
// nuclear norm of env when `want_norm`.
static __device__ __noinline__ double warp_polar_exact(WarpPolar& ws, const double2* env, double2* gate, int m,
                                                       bool want_norm, bool* finite) {
  const int lane = threadIdx.x & 31;
  const int ex = wp_load(ws, env, m, lane, finite);
  if (!*finite) return 0.0;
  const int row = lane & 3, pr = (lane >> 2) & 1, ip = row * 4 + 2 * pr, iq = ip + 1;
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3, part = lane & 1;
  xc yp, yq;
  wp_df_columns(ws, lane, yp, yq);
  // null columns, known to every lane of their pair
  float al32 = quad_sum(fmaf(yp.x, yp.x, yp.y * yp.y)), be32 = quad_sum(fmaf(yq.x, yq.x, yq.y * yq.y));
  al32 = __shfl_sync(0xffffffffu, al32, lane & 7);
  be32 = __shfl_sync(0xffffffffu, be32, lane & 7);
  float m2 = fmaxf(al32, be32);
  m2 = fmaxf(m2, __shfl_xor_sync(0xffffffffu, m2, 4));
  const float thr = fmaxf((float)(QM_POLAR_NULL_TOL * QM_POLAR_NULL_TOL) * m2, WPX_TINY);
  int fp = !(al32 > thr), fq = !(be32 > thr);
  const bool any_null = __any_sync(0xffffffffu, fp || fq);
  if (any_null) {
    // X = (I - U_s U_s^H) Wp V_N in double-float, to turn V_N so that X's
    // columns are orthogonal (X itself is formed again in FP64)
    wp_norms(ws, lane, yp, yq, fp, fq);
    __syncwarp();
    xc* mine = (lane & 8) ? ws.V : ws.U;
    if (lane < 16) {
      XA u = xa_zero(), v = xa_zero();
      const DF a = lane < 8 ? ws.rs[2 * pr] : DF{1.f, 0.f}, b = lane < 8 ? ws.rs[2 * pr + 1] : DF{1.f, 0.f};
      df_mac(u.re, yp.x, yp.z, a.hi, a.lo);
      df_mac(u.im, yp.y, yp.w, a.hi, a.lo);
      df_mac(v.re, yq.x, yq.z, b.hi, b.lo);
      df_mac(v.im, yq.y, yq.w, b.hi, b.lo);
      mine[ip] = xa_round(u);
      mine[iq] = xa_round(v);
    }
    xc* const G = reinterpret_cast<xc*>(ws.C);
    xc* const X = reinterpret_cast<xc*>(ws.A);
    xc* const Cx = reinterpret_cast<xc*>(ws.B);
    if (lane < 16) G[lane] = xc_from_d(wp_gate(gate, m, lane >> 2, lane & 3));
    __syncwarp();
    const DF y = wdf_part<false, false>(G, ws.V, i, j, part);   // Wp V
    wdf_store(X, lane, y);
    __syncwarp();
    wdf_store(Cx, lane, wdf_part<true, false>(ws.U, X, i, j, part));
    __syncwarp();
    DF x = wdf_part<false, false>(ws.U, Cx, i, j, part);
    x = DF{-x.hi, -x.lo};
    df_add(x, y.hi, y.lo);
    __syncwarp();
    wdf_store(X, lane, x);
    __syncwarp();
    if (!(lane & 8)) {
      if (fp) yp = X[ip];
      if (fq) yq = X[iq];
    }
    wd_sweeps(yp, yq, fp, fq, WH_FLAGGED);
    __syncwarp();
  }
  const unsigned nb_p = __ballot_sync(0xffffffffu, fp), nb_q = __ballot_sync(0xffffffffu, fq);
  const int nmask = (nb_p & 1) | ((nb_q & 1) << 1) | (((nb_p >> 4) & 1) << 2) | (((nb_q >> 4) & 1) << 3);
  wp_norms(ws, lane, yp, yq, fp, fq);
  __syncwarp();
  wp_to_fp64(ws, lane, yp, yq);
  double nuc = 0.0;
  if (want_norm) {   // sum of the norms of E V's columns but the padding's
    const double a = reinterpret_cast<const double*>(ws.A)[lane];
    double q = a * a;
    q += __shfl_xor_sync(0xffffffffu, q, 1);
    q += __shfl_xor_sync(0xffffffffu, q, 8);
    q += __shfl_xor_sync(0xffffffffu, q, 16);
    nuc = q > WPX_TINY ? q * wp_rsqrt(q) : 0.0;
    nuc += __shfl_xor_sync(0xffffffffu, nuc, 2);
    nuc += __shfl_xor_sync(0xffffffffu, nuc, 4);
    if (m == 2) nuc -= 2.0 * (double)ws.E[10].x;
  }
  {   // null columns of C are zero here: nothing between them and the others
    const bool skip = ((nmask >> i) & 1) || ((nmask >> j) & 1);
    wp_polar_weights(ws, lane, 0);
    if (skip) wf_store(ws.T, lane, 0.f);
    __syncwarp();
  }
  wmm_correct(ws.C, ws.T, lane);
  if (any_null) {
    // V_N off E's row space: rotate by -C_s^H (E v_n) / s_s
    {
      float c = 0.f;
      const bool sn = !((nmask >> i) & 1) && ((nmask >> j) & 1), ns = ((nmask >> i) & 1) && !((nmask >> j) & 1);
      const int u = sn ? i : j, x = sn ? j : i;   // significant, null
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 a = wf_entry(ws.C[k * 4 + u]), b = wf_entry(ws.A[k * 4 + x]);
        c += part ? a.x * b.y - a.y * b.x : a.x * b.x + a.y * b.y;   // conj(a) b
      }
      c *= ws.rs[u].hi;
      wf_store(ws.T, lane, sn ? -c : ns ? (part ? -c : c) : 0.f);
      __syncwarp();
    }
    wmm_correct(ws.B, ws.T, lane);
    // null columns of C: X in FP64, its columns orthogonal
    double2* const Wp = ws.A;
    double2* const Y = reinterpret_cast<double2*>(ws.V);
    double2* const Cm = reinterpret_cast<double2*>(ws.U);
    if (lane < 16) Wp[lane] = wp_gate(gate, m, lane >> 2, lane & 3);
    __syncwarp();
    const double y = wmm_part<false, false>(Wp, ws.B, i, j, part);
    wmm_store(Y, lane, y);
    __syncwarp();
    wmm_store(Cm, lane, wmm_part<true, false>(ws.C, Y, i, j, part));
    __syncwarp();
    const double x = y - wmm_part<false, false>(ws.C, Cm, i, j, part);
    __syncwarp();
    wmm_store(Y, lane, x);
    __syncwarp();
    const xc xp = xc_from_d(Y[ip]), xq = xc_from_d(Y[iq]);
    const float np = quad_sum(fmaf(xp.x, xp.x, xp.y * xp.y)), nq = quad_sum(fmaf(xq.x, xq.x, xq.y * xq.y));
    if (!__all_sync(0xffffffffu, (!fp || np > 1e-16f) && (!fq || nq > 1e-16f))) {
      const double nn = lane == 0 ? wp_single_thread<true>(ws, gate, m) : 0.0;
      __syncwarp();
      return __shfl_sync(0xffffffffu, nn, 0) * wp_unscale(ex);
    }
    wp_norms(ws, lane, xp, xq, !fp, !fq);
    __syncwarp();
    if ((nmask >> j) & 1) wmm_store(ws.C, lane, x * ((double)ws.rs[j].hi + (double)ws.rs[j].lo));
    __syncwarp();
    wp_gram_defect(ws.C, ws.T, lane);
    // sig is now the null columns': only the null yield (a significant
    // column's own defect was corrected above and halves are exact)
    {
      const bool ni = (nmask >> i) & 1, nj = (nmask >> j) & 1;
      const float t = (nj ? (ni ? 1.f : 2.f) : 0.f) * reinterpret_cast<const float*>(ws.T)[lane];
      __syncwarp();
      wf_store(ws.T, lane, t);
      __syncwarp();
    }
    wmm_correct(ws.C, ws.T, lane);
  }
  const double v = wmm_part<false, true>(ws.C, ws.B, i, j, part);
  if (i < m && j < m) reinterpret_cast<double*>(gate)[2 * (i * m + j) + part] = part ? -v : v;
  __syncwarp();
  return nuc * wp_unscale(ex);
}

// Eigenvectors of the Hermitian positive semidefinite Gram g (lane's entry
// of the 4 x 4 matrix, zero padded; lanes 16-31 repeat): one-sided Jacobi on
// its columns, G V = U Lambda.  ws.B receives the vectors as columns,
// l[0..3] (every lane) the eigenvalue of each times a power of two; *odd is
// 1 where columns 2 and 3 stand exchanged.
// The columns are orthogonal to double-float; what is left is one
// first-order rotation v_j += v_i g_ij / (l_j^2 - l_i^2) where that is below
// 1e-8, else FP64 sweeps (eigenvalues that agree to about 1e-6, and those
// below 2e-7 of the largest, which the rounding of g to double-float for the
// sweeps before turns by more; a cut of them takes no longer than when their
// vectors stayed so).  Vectors of eigenvalues below 1e-11 of the largest keep
// any rotation among themselves.
__device__ __forceinline__ void warp_gram_vectors(WarpPolar& ws, double2 g, double (&l)[4], int* odd) {
  const int lane = threadIdx.x & 31;
  const int ip = (lane & 3) * 4 + 2 * ((lane >> 2) & 1);
  const int ent = lane >> 1, i = ent >> 2, j = ent & 3;
  bool finite;
  if (lane < 16) ws.A[lane] = g;
  __syncwarp();
  wp_load(ws, ws.A, 4, lane, &finite);
  xc yp, yq;
  int fp = 0, fq = 0;
  *odd = wp_df_columns(ws, lane, yp, yq);
  wp_norms(ws, lane, yp, yq, 0, 0);
  __syncwarp();
  wp_to_fp64(ws, lane, yp, yq);
  // T holds -cos / 2 of every pair: the rotation's tangent
  float t = 0.f;
  if (i != j) {
    const float top = fmaxf(fmaxf(ws.sq[0].hi, ws.sq[1].hi), fmaxf(ws.sq[2].hi, ws.sq[3].hi));
    const bool noise = ws.sq[i].hi <= 1e-22f * top && ws.sq[j].hi <= 1e-22f * top;
    DF d = ws.sq[j];
    df_add(d, -ws.sq[i].hi, -ws.sq[i].lo);
    const float gij = -2.f * reinterpret_cast<const float*>(ws.T)[lane] * ws.sig[i] * ws.sig[j];
    if (!noise && gij != 0.f) t = __fdividef(gij, d.hi + d.lo);   // d = 0: not finite, the sweeps take it
  }
  const bool small = __all_sync(0xffffffffu, fabsf(t) < 1e-8f);
  if (small) {
    wf_store(ws.T, lane, t);
    __syncwarp();
    wmm_correct(ws.B, ws.T, lane);
#pragma unroll
    for (int c = 0; c < 4; ++c) l[c] = (double)ws.sig[c];
    // to FP64: l^2 = sq, one Newton step from the FP32 root
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const double q = (double)ws.sq[c].hi + (double)ws.sq[c].lo;
      l[c] = l[c] > 0.0 ? fma(0.5 * (double)ws.rs[c].hi, fma(-l[c], l[c], q), l[c]) : 0.0;
    }
    return;
  }
  double2* mine = (lane & 8) ? ws.B : ws.A;
  double2 xp = mine[ip], xq = mine[ip + 1];
  *odd ^= wx_sweeps(xp, xq, fp, fq, WH_ALL);
  const double al = quad_sum(cnorm2(xp)), be = quad_sum(cnorm2(xq));
  const double lp = al > WPX_TINY ? al * wp_rsqrt(al) : 0.0, lq = be > WPX_TINY ? be * wp_rsqrt(be) : 0.0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const double a = __shfl_sync(0xffffffffu, lp, (c >> 1) * 4), b = __shfl_sync(0xffffffffu, lq, (c >> 1) * 4);
    l[c] = (c & 1) ? b : a;
  }
  __syncwarp();
  if (lane >= 8 && lane < 16) {
    ws.B[ip] = xp;
    ws.B[ip + 1] = xq;
  }
  __syncwarp();
}

// ---- sums over a warp --------------------------------------------------------------------------

// s += the partner lane's `give` (lane ^ o)
__device__ __forceinline__ void tf_shfl_add(TF& s, const TF& give, int o) {
  tf_add(s, TF{__shfl_xor_sync(0xffffffffu, give.h, o), __shfl_xor_sync(0xffffffffu, give.m, o),
               __shfl_xor_sync(0xffffffffu, give.l, o)});
}

// Halving exchange over lanes N / 2, N / 4 .. 1: lane l returns the sum over
// them of value l mod N.
template <int N>
__device__ __forceinline__ TF warp_fold_tf(TF (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const TF give = up ? v[i] : v[i + o];
      if (up) v[i] = v[i + o];
      tf_shfl_add(v[i], give, o);
    }
  }
  return v[0];
}

// Sum of 32 double-float values per lane over the warp: lane l returns the
// total of value l (exchange as warp_sum32), as exact as FP64 sums but for the
// first of five steps, whose roundings average out as those of the lanes' own
// sums do.
__device__ __forceinline__ TF warp_sum32_tf(DF (&v)[32]) {
  TF t[16];
  const bool up = (threadIdx.x & 16) != 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const DF give = up ? v[i] : v[i + 16];
    if (up) v[i] = v[i + 16];
    df_shfl_add(v[i], give, 16);
    t[i] = tf_from(v[i]);
  }
  return warp_fold_tf(t);
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

// Sum over the block's eight warps of part `lane` of an environment, in
// fixed order, as one part of a double-float entry.
__device__ __forceinline__ void env_sum_warps(const float2 (*wred)[32], xc* env, int lane) {
  DF s = {0.f, 0.f};
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const float2 v = wred[w][lane];
    df_add(s, v.x, v.y);
  }
  wdf_store(env, lane, s);
}
// The same of three-part sums, as one part of an FP64 entry.
__device__ __forceinline__ void env_sum_warps(const TF (*wred)[32], double2* env, int lane) {
  TF v[WARPS];
#pragma unroll
  for (int w = 0; w < WARPS; ++w) v[w] = wred[w][lane];
#pragma unroll
  for (int o = WARPS / 2; o > 0; o >>= 1)
#pragma unroll
    for (int w = 0; w < o; ++w) tf_add(v[w], v[w + o]);
  wmm_store(env, lane, tf_to_d(v[0]));
}
static_assert(sizeof(xc) == sizeof(double2), "work matrices are shared between the precisions");
