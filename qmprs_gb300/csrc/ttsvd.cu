// (a) statevector -> MPS: right-to-left sequential truncated SVD to bond chi.
//
// Restates MPS.from_statevector (reference qmprs/primitives/mps.py:219-249):
// quimb's from_dense followed by tensor_network_1d_compress(max_bond=chi),
// whose density-matrix method truncates from the right and leaves a
// right-canonical MPS.  Cut c (c = n-1 .. 1) of state b holds the remainder
// M (2^c x w, w = 2 r, r = bond c+1).  Per cut:
//   k_tt_gram     Gram matrix M^H M in double-float, split over row ranges;
//   k_tt_gram_sum the ranges' partials summed in order, in fp64;
//   k_tt_eig      one CTA per state: parallel cyclic Jacobi (round-robin
//                 pairs) on the w x w Gram, fp32 passes with double-float
//                 products (w <= 64) or fp32 and fp64 sweeps; sort, rsum2
//                 cutoff + max_bond, canonical phases; site tensor c;
//   k_tt_project  next remainder M V (fp32).
// k_tt_site0 stores site 0 (the last remainder, rescaled to the input norm,
// as quimb's rsum2 renormalisation does) and k_mps_contract rebuilds the
// truncated dense target, left to right.
//
// Widths: the one-block kernels take Grams up to bd.eig_wmax (128, or 64 in
// batches of at most BJ_SMALL_BATCH states); wider ones are diagonalised by
// the blocked solver (ttsvd_wide.cu).  A state whose bond exceeds the plan's
// capacity raises KERR_EIG_WIDTH and has its bond poisoned (-1); every
// later kernel of the stage skips a state whose bonds are out of range, so
// no access ever depends on an unset bond.
#include "dfloat.cuh"

#define TT_CH 32
#define TT_EIG_THREADS 512
#define TT_EIG_PAD 2

__host__ __device__ inline int chi_eff(int chi, int n) {
  const int cap = 1 << (n / 2);
  return chi < cap ? chi : cap;
}

__device__ __forceinline__ bool bond_ok(int r, int lim) { return r >= 1 && r <= lim; }

#define TT_EPB 8   // entries per thread: a 2 x 4 block (a in {2i, 2i+1}, cc in {4j .. 4j+3})

// Entry block e of the upper triangle of a w x w Gram, ordered by column
// block j (2j + 2 blocks in column block j, capped at w / 2 rows).
__device__ __forceinline__ void gram_block(int e, int w, int* i0, int* j0) {
  const int half = w >> 1;
  int j = 0, base = 0;
  for (;; ++j) {
    const int cnt = min(half, 2 * j + 2);
    if (e < base + cnt) break;
    base += cnt;
  }
  *i0 = e - base;
  *j0 = j;
}

__device__ __forceinline__ int gram_nblocks(int w) {
  const int half = w >> 1, nj = (w + 3) / 4;
  int t = 0;
  for (int j = 0; j < nj; ++j) t += min(half, 2 * j + 2);
  return t;
}

// Row splits of a state's Gram: as many as it has tiles, at most
// TT_SPLIT_MAX, at least 32 rows each, and as many w x w partials as its
// slot holds.  A 20-qubit state's 64-wide Gram has 16384 rows and one chunk
// of entry blocks, so eight splits kept 16 SMs busy.
__device__ __forceinline__ int tt_splits(const BatchDev& bd, int b, int c, int w) {
  const int n = min(min(bd.state_ntiles[b], TT_SPLIT_MAX), c > 5 ? 1 << min(c - 5, 8) : 1);
  return n > 1 ? min(n, (int)(bd.tt_off[b + 1] - bd.tt_off[b]) / (w * w)) : 1;   // a slot holds at least eight
}

// The sums over a state's rows are scaled where its norm^2 is near the end of
// FP32's range, which holds a TT_FLUSH run of products but not their sum.
#define TT_GRAM_DOWN 0x1p-40f
__device__ __forceinline__ bool tt_gram_large(double2 sq) { return sq.x > 0x1p120; }

__device__ __forceinline__ bool tt_gram_here(const BatchDev& bd, const int* bond, int c, int* w) {
  if (c < 1 || !bond_ok(bond[c + 1], bd.tt_b)) return false;
  *w = 2 * bond[c + 1];
  return !(*w > bd.eig_wmax && ipow2(c) < (int64_t)*w);   // else the row Gram (ttsvd_wide.cu)
}

// Upper triangle of M^H M (M = the 2^c x w remainder) per state, row split
// by row split; in a block, thread t takes the entry block (t mod nb) and
// every (256 / nb)-th row of the split, sums exact fp32 products in
// double-float over TT_FLUSH rows, those sums in double-float too, and the
// rest groups are then summed in fixed order through shared memory
// (k_tt_gram_sum adds the splits in order).
// Measured (20 qubits, 64 wide): 1380 us with eight splits and FP64 sums,
// 86 us now (512 wide, FP32 bound: 1630 -> 520 us).
__global__ void __launch_bounds__(BLOCK_THREADS) k_tt_gram(BatchDev bd, int step, const float2* sv,
                                                           const float2* src, const int* bonds, const double2* sq,
                                                           xc* partials) {
  grid_wait();
  __shared__ xc red[BLOCK_THREADS * TT_EPB];   // 32 KB
  __shared__ volatile int large;               // not a register over the rows
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    const int n = bd.n[b];
    const int c = n - 1 - step;
    if (c < 1) continue;
    const int* bond = bonds + (int64_t)b * (bd.max_n + 1);
    const int idx = bd.tile_idx[tile];
    if (bond[c + 1] > bd.tt_b && idx == 0 && threadIdx.x == 0) atomicOr(bd.err, KERR_EIG_WIDTH);
    int w;
    if (!tt_gram_here(bd, bond, c, &w)) continue;
    if (threadIdx.x == 0) large = tt_gram_large(sq[b]);
    __syncthreads();
    const int nt = bd.state_ntiles[b], nsplit = tt_splits(bd, b, c, w);
    const float2* m = (step == 0 ? sv : src) + bd.vec_off[b];
    const int nb = gram_nblocks(w);
    // work units: (row split, chunk of BLOCK_THREADS entry blocks), taken by
    // the state's tiles in turn, so wide Grams spread over many blocks
    const int nech = (nb + BLOCK_THREADS - 1) / BLOCK_THREADS;
    const int units = nsplit * nech;
    for (int unit = idx; unit < units; unit += nt) {
      const int split = unit % nsplit;
      int64_t lo, hi;
      tile_range(ipow2(c), split, nsplit, &lo, &hi);
      xc* part = partials + bd.tt_off[b] + (int64_t)split * w * w;
      const int e0 = (unit / nsplit) * BLOCK_THREADS;
      const int nbp = nb - e0 < BLOCK_THREADS ? nb - e0 : BLOCK_THREADS;
      const int nsub = BLOCK_THREADS / nbp;
      const int eb = threadIdx.x % nbp, sub = threadIdx.x / nbp;
      const bool act = sub < nsub;
      int bi = 0, bj = 0;
      if (act) gram_block(e0 + eb, w, &bi, &bj);
      const int a0 = 2 * bi, c0 = 4 * bj;
      XA acc[TT_EPB];
#pragma unroll
      for (int k = 0; k < TT_EPB; ++k) acc[k] = xa_zero();
      if (act) {
        int64_t row = lo + sub;
        while (row < hi) {
          XA s[TT_EPB];
#pragma unroll
          for (int k = 0; k < TT_EPB; ++k) s[k] = xa_zero();
          for (int f = 0; f < TT_FLUSH && row < hi; ++f, row += nsub) {
            const float2* x = m + row * w;
            float2 xa[2], xv[4];
#pragma unroll
            for (int u = 0; u < 2; ++u) xa[u] = x[a0 + u];
#pragma unroll
            for (int v = 0; v < 4; ++v) xv[v] = c0 + v < w ? x[c0 + v] : cf(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                // conj(xa) * xv
                XA& o = s[u * 4 + v];
                df_add_prod(o.re, xa[u].x, xv[v].x);
                df_add_prod(o.re, xa[u].y, xv[v].y);
                df_add_prod(o.im, xa[u].x, xv[v].y);
                df_add_prod(o.im, -xa[u].y, xv[v].x);
              }
          }
          if (large) {
#pragma unroll
            for (int k = 0; k < TT_EPB; ++k) {
              s[k].re = DF{s[k].re.hi * TT_GRAM_DOWN, s[k].re.lo * TT_GRAM_DOWN};
              s[k].im = DF{s[k].im.hi * TT_GRAM_DOWN, s[k].im.lo * TT_GRAM_DOWN};
            }
          }
#pragma unroll
          for (int k = 0; k < TT_EPB; ++k) {
            df_add(acc[k].re, s[k].re.hi, s[k].re.lo);
            df_add(acc[k].im, s[k].im.hi, s[k].im.lo);
          }
        }
      }
      // sum the row groups of each entry block in fixed order
      __syncthreads();
#pragma unroll
      for (int k = 0; k < TT_EPB; ++k) red[threadIdx.x * TT_EPB + k] = xa_round(acc[k]);
      __syncthreads();
      for (int o = threadIdx.x; o < nbp * TT_EPB; o += BLOCK_THREADS) {
        const int ebo = o / TT_EPB, k = o % TT_EPB;
        XA sacc = xa_zero();
        for (int sb = 0; sb < nsub; ++sb) {
          const xc v = red[(sb * nbp + ebo) * TT_EPB + k];
          df_add(sacc.re, v.x, v.z);
          df_add(sacc.im, v.y, v.w);
        }
        int gi, gj;
        gram_block(e0 + ebo, w, &gi, &gj);
        const int a = 2 * gi + k / 4, cc = 4 * gj + k % 4;
        if (a <= cc && cc < w) part[(int64_t)a * w + cc] = xa_round(sacc);
      }
    }
  }
}

// The Gram of every state: the splits' partials summed in a fixed order
// (eight lanes per entry, each every eighth split, then the lanes), the lower
// triangle mirrored.  Block x takes 32 entries at a time, block y a state.
// Latency bounds it, so six blocks an SM (48 registers took 5.9 ms where 40
// take 4.7, 2000 states of 11 qubits at bond 16).
__global__ void __launch_bounds__(BLOCK_THREADS, 6) k_tt_gram_sum(BatchDev bd, int step, const int* bonds,
                                                               const double2* sq, const xc* partials,
                                                               double2* gram) {
  grid_wait();
  const int l8 = threadIdx.x & 7;
  for (int b = blockIdx.y; b < bd.B; b += gridDim.y) {
    const int c = bd.n[b] - 1 - step;
    int w;
    if (!tt_gram_here(bd, bonds + (int64_t)b * (bd.max_n + 1), c, &w)) continue;
    const int nsplit = tt_splits(bd, b, c, w), ww = w * w;
    const xc* part = partials + bd.tt_off[b];
    double2* g = gram + (int64_t)b * bd.tt_w * bd.tt_w;
    const bool large = tt_gram_large(sq[b]);
    for (int e0 = blockIdx.x * (BLOCK_THREADS / 8); e0 < ww; e0 += gridDim.x * (BLOCK_THREADS / 8)) {
      const int e = e0 + (threadIdx.x >> 3), a = e / w, cc = e % w;
      XA s = xa_zero();
      if (e < ww && a <= cc) {
#pragma unroll 4
        for (int t = l8; t < nsplit; t += 8) {
          const xc v = part[(int64_t)t * ww + e];
          df_add(s.re, v.x, v.z);
          df_add(s.im, v.y, v.w);
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        df_add(s.re, __shfl_xor_sync(0xffffffffu, s.re.hi, o), __shfl_xor_sync(0xffffffffu, s.re.lo, o));
        df_add(s.im, __shfl_xor_sync(0xffffffffu, s.im.hi, o), __shfl_xor_sync(0xffffffffu, s.im.lo, o));
      }
      if (l8 == 0 && e < ww && a <= cc) {
        double2 r = xa_to_d(s);
        if (large) r = cscale(r, 1.0 / TT_GRAM_DOWN);
        g[e] = a == cc ? cd(r.x, 0.0) : r;
        if (a != cc) g[(int64_t)cc * w + a] = cconj(r);
      }
    }
  }
}

// ---- Jacobi rounds in either precision -----------------------------------------

__device__ __forceinline__ float2 jmk(float re, float im) { return cf(re, im); }
__device__ __forceinline__ double2 jmk(double re, double im) { return cd(re, im); }
template <class C, class R>
__device__ __forceinline__ C jscale(C a, R t) { return jmk(a.x * t, a.y * t); }
template <class C>
__device__ __forceinline__ C jmul(C a, C b) { return jmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <class C>
__device__ __forceinline__ C jadd(C a, C b) { return jmk(a.x + b.x, a.y + b.y); }
template <class C>
__device__ __forceinline__ C jsub(C a, C b) { return jmk(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float jsqrt(float v) { return sqrtf(v); }
__device__ __forceinline__ double jsqrt(double v) { return sqrt(v); }
__device__ __forceinline__ float jabs(float2 a) { return hypotf(a.x, a.y); }
__device__ __forceinline__ double jabs(double2 a) { return hypot(a.x, a.y); }

template <class C, class R>
struct JacobiShared {
  R c[TT_MAXW / 2];
  C se[TT_MAXW / 2], sce[TT_MAXW / 2];
  int p[TT_MAXW / 2], q[TT_MAXW / 2], flag[TT_MAXW / 2];
  int rot;
};

// Parallel cyclic Jacobi (round-robin pairing, w / 2 disjoint rotations per
// round) on the Hermitian G (row-major, stride ld), accumulating V <- V R.
// A pair rotates unless |g_pq| <= rel sqrt(|g_pp g_qq|) or |g_pq| <=
// floor_abs.  Runs whole sweeps until one makes no rotation (at most
// max_sweeps).  The block must call it uniformly.
template <class C, class R>
__device__ void jacobi_run(C* G, C* V, int w, int ld, R rel, R floor_abs, int max_sweeps, JacobiShared<C, R>& js) {
  const int half = w / 2;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) js.rot = 0;
    __syncthreads();
    for (int k = 0; k < w - 1; ++k) {
      if (threadIdx.x < half) {
        const int i = threadIdx.x;
        const int t1 = i, t2 = w - 1 - i;
        int p = t1 == 0 ? 0 : 1 + ((t1 - 1 + k) % (w - 1));
        int q = 1 + ((t2 - 1 + k) % (w - 1));
        if (p > q) {
          const int tmp = p;
          p = q;
          q = tmp;
        }
        const C g = G[p * ld + q];
        const R ag = jabs(g);
        const R app = G[p * ld + p].x, aqq = G[q * ld + q].x;
        const int rot = !(ag == R(0) || ag <= rel * jsqrt(fabs(app * aqq)) || ag <= floor_abs);
        js.p[i] = p;
        js.q[i] = q;
        js.flag[i] = rot;
        if (rot) {
          const R zeta = (aqq - app) / (R(2) * ag);
          const R t = (zeta >= R(0) ? R(1) : R(-1)) / (fabs(zeta) + jsqrt(R(1) + zeta * zeta));
          const R cc = R(1) / jsqrt(R(1) + t * t);
          const R ss = cc * t;
          const C e = jscale(g, R(1) / ag);
          js.c[i] = cc;
          js.se[i] = jscale(e, ss);
          js.sce[i] = jscale(jmk(e.x, -e.y), ss);
          js.rot = 1;
        }
      }
      __syncthreads();
      for (int idx = threadIdx.x; idx < half * w; idx += blockDim.x) {
        const int i = idx / w, row = idx % w;
        if (!js.flag[i]) continue;
        const int p = js.p[i], q = js.q[i];
        const R cc = js.c[i];
        const C se = js.se[i], sce = js.sce[i];
        const C xp = G[row * ld + p], xq = G[row * ld + q];
        G[row * ld + p] = jsub(jscale(xp, cc), jmul(sce, xq));
        G[row * ld + q] = jadd(jmul(se, xp), jscale(xq, cc));
        const C vp = V[row * ld + p], vq = V[row * ld + q];
        V[row * ld + p] = jsub(jscale(vp, cc), jmul(sce, vq));
        V[row * ld + q] = jadd(jmul(se, vp), jscale(vq, cc));
      }
      __syncthreads();
      for (int idx = threadIdx.x; idx < half * w; idx += blockDim.x) {
        const int i = idx / w, col = idx % w;
        if (!js.flag[i]) continue;
        const int p = js.p[i], q = js.q[i];
        const R cc = js.c[i];
        const C se = js.se[i], sce = js.sce[i];
        const C xp = G[p * ld + col], xq = G[q * ld + col];
        G[p * ld + col] = jsub(jscale(xp, cc), jmul(se, xq));
        G[q * ld + col] = jadd(jmul(sce, xp), jscale(xq, cc));
      }
      __syncthreads();
      if (threadIdx.x < half && js.flag[threadIdx.x]) {
        const int p = js.p[threadIdx.x], q = js.q[threadIdx.x];
        G[p * ld + q] = jmk(R(0), R(0));
        G[q * ld + p] = jmk(R(0), R(0));
        G[p * ld + p].y = R(0);
        G[q * ld + q].y = R(0);
      }
      __syncthreads();
    }
    if (!js.rot) break;
    __syncthreads();
  }
}

// C = A^H B (adj = true) or A B, w x w row-major matrices of stride ld in
// shared memory; C is neither A nor B.
__device__ void smem_matmul(const double2* A, const double2* B, double2* Cm, int w, int ld, bool adj) {
  for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
    const int i = e / w, j = e % w;
    double2 acc = czero();
    if (adj)
      for (int k = 0; k < w; ++k) acc = cadd(acc, cmulc(A[k * ld + i], B[k * ld + j]));
    else
      for (int k = 0; k < w; ++k) acc = cadd(acc, cmul(A[i * ld + k], B[k * ld + j]));
    Cm[i * ld + j] = acc;
  }
}

// ---- eigenvectors of a Gram in shared memory (w <= 64) -------------------------------
//
// GB300 runs an FP64 warp instruction in 64 cycles per SM quarter, so both
// FP64 Jacobi sweeps and FP64 matrix products of a 64 x 64 Gram cost about a
// millisecond each.  The vectors are found by passes instead: FP32 Jacobi
// sweeps on the FP32 rounding of G give V_k, which is made orthonormal, and
//   G <- V_k^H G V_k,  V <- V V_k
// are double-float products on the FP32 pipes (2^-46).  G is then graded and
// nearly diagonal, its small entries known to their own FP32 precision, so
// the next pass resolves what FP32 could not see at G's scale (each pass
// gains about seven digits), down to a rotation floor of 1e-13 of the trace
// (ten times the products' rounding; the truncation decides at 1e-10).
// Three or four passes; a pass at that floor whose rotations were all below
// 3e-7 is the last.  Measured (48 states, w = 64): about 6 ms per cut with FP64 products
// and FP64 finishing sweeps, 1.4 ms now, half of it the FP32 sweeps and half
// the double-float products (three quarters of the FP32 pipes' rate).

extern __shared__ double2 eig_sm[];
__device__ __forceinline__ float2* tt_smf() { return reinterpret_cast<float2*>(eig_sm); }
__device__ __forceinline__ xc* tt_smx() { return reinterpret_cast<xc*>(eig_sm); }

#define JW (TT_EIG_THREADS / 32)
static_assert(JW == 16, "the Jacobi sweeps' warp roles");

// p <- c p - conj(s) q, q <- s p + c q
__device__ __forceinline__ void jacobi32_cols(float2& p, float2& q, float c, float sx, float sy) {
  const float2 a = cf(c * p.x - fmaf(sx, q.x, sy * q.y), c * p.y - fmaf(sx, q.y, -sy * q.x));
  const float2 b = cf(fmaf(c, q.x, fmaf(sx, p.x, -sy * p.y)), fmaf(c, q.y, fmaf(sx, p.y, sy * p.x)));
  p = a;
  q = b;
}

// ---- FP32 Jacobi sweeps in one block (w <= 64) ----
//
// Round-robin pairing by position: a round pairs position x with pw - 1 - x
// (pair l: p = l, q = pw - 1 - l), and every column then moves to next(x),
// so a sweep of pw - 1 rounds brings each one home.  pw is w rounded
// up; the padding is zero and never rotates.  The block's warps take roles:
//   warp 0        the rotations, one round ahead: lane l keeps pair l's
//                 diagonal in registers and rotates the one entry the next
//                 round's pair needs by itself, so that the angles of round
//                 k + 1 are ready when the others finish round k;
//   warps 1 - 8   v <- v R in registers: a lane holds a quarter of a row (a
//                 warp one quarter of 32 rows, so that every angle is one
//                 broadcast), whose columns change place by register, and
//                 from quarter to quarter through shared memory;
//   the others    G <- R^H G R on the 2 x 2 blocks of pairs R < C (G is
//                 Hermitian; an entry is kept in the row of the smaller
//                 pair), double-buffered in shared memory, the blocks of
//                 pair rows P and half - 1 - P sharing a warp's lanes.
// One barrier a round.  A pair rotates when |g_pq| is above rel sqrt(|g_pp
// g_qq|) and floor_abs, and its entry counts as zero from then on; sweeps
// repeat while a rotation was above 1e-4 of sqrt(|g_pp g_qq|) (convergence
// is quadratic).  *moved: a rotation of tangent above 3e-7 was made.
// With v in shared memory, both halves of G and the angles on the chain, a
// round at w = 64 took 2800 cycles (128 KB of shared-memory traffic, 920 of
// issue), 1050 now; the chain through warp 0 is about 500, which narrow
// Grams take.
#define JAC_G(buf) ((4 + (buf)) * TT_EIG_SMEM_W * (TT_EIG_SMEM_W + TT_EIG_PAD))
#define JAC_SHARED (3 * TT_EIG_SMEM_W * (TT_EIG_SMEM_W + TT_EIG_PAD))
struct JacShared {
  float4 rot[2][TT_EIG_SMEM_W / 2];   // (c, Re s, Im s, 0) per pair
  float2 edge[2][2][TT_EIG_SMEM_W / 16][TT_EIG_SMEM_W];   // columns between quarters: to the lower, to the upper
  int again;
};

__device__ __forceinline__ int jac_next(int x, int pw) { return x == 0 ? 0 : x == 1 ? pw - 1 : x - 1; }

static_assert(sizeof(JacShared) <= TT_EIG_SMEM_W * (TT_EIG_SMEM_W + TT_EIG_PAD) * sizeof(float2), "below JAC_G(0)");

// Rotation of a pair with diagonal app, aqq and entry g: (c, Re s, Im s) and
// the diagonal's shift.
struct JacRot {
  float c, sx, sy, shift;
  bool again, moved;
};
__device__ __forceinline__ JacRot jac_rotation(float app, float aqq, float2 g, float rel, float floor_abs) {
  JacRot o = {1.f, 0.f, 0.f, 0.f, false, false};
  const float g2n = fmaf(g.x, g.x, g.y * g.y), sc = fabsf(app) * fabsf(aqq);
  if (g2n > rel * rel * sc && g2n > floor_abs * floor_abs) {
    const float d = 0.5f * (aqq - app);
    const float ri = rsqrtf(fmaf(d, d, g2n));
    const float c2 = fmaf(0.5f * fabsf(d), ri, 0.5f), ci = rsqrtf(c2);
    const float h = copysignf(0.5f * ri * ci, d);
    const float c = c2 * ci, sx = g.x * h, sy = g.y * h;
    // unitary to rounding: rsqrtf's own errors would add up over the sweeps
    const float e = 0.5f * fmaf(-sy, sy, fmaf(-sx, sx, fmaf(-c, c, 1.f)));
    o.c = fmaf(c, e, c);
    o.sx = fmaf(sx, e, sx);
    o.sy = fmaf(sy, e, sy);
    o.shift = h * ci * g2n;
    o.again = g2n > 1e-8f * sc;
    o.moved = fmaf(o.sx, o.sx, o.sy * o.sy) > 9e-14f * c2;
  }
  return o;
}

// NG groups of NP pairs to a row of v
// (not inlined: the caller's values would leave the roles too few registers)
template <int NP, int NG>
__device__ __noinline__ bool jacobi32_sweeps(int vout, int w, int ld, float rel, float floor_abs) {
  constexpr int PW = 2 * NP * NG, HALF = NP * NG, LJ = PW + 1, SPARE = PW * LJ;
  constexpr int GWARP = 9, GWARPS = JW - GWARP, GIT = (HALF / 2 + GWARPS - 1) / GWARPS;
  static_assert(SPARE + 32 <= TT_EIG_SMEM_W * (TT_EIG_SMEM_W + TT_EIG_PAD), "spare slots behind the matrix");
  float2* S = tt_smf();
  JacShared& js = *reinterpret_cast<JacShared*>(S + JAC_SHARED);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int buf = 0;
  bool mv = false;
  if (warp == 0) {
    const bool act = lane < HALF;
    const int l = act ? lane : HALF - 1;
    const int R = l == 0 ? 0 : l == HALF - 1 ? HALF - 2 : l - 1, C = l == 0 ? 1 : l == HALF - 1 ? HALF - 1 : l + 1;
    const int o00 = R * LJ + C, o01 = R * LJ + PW - 1 - C, o10 = (PW - 1 - R) * LJ + C,
              o11 = (PW - 1 - R) * LJ + PW - 1 - C;
    const bool rowq = l != 0, colq = l == HALF - 1;
    // where the pair's own entry, now zero, goes
    const int zero = jac_next(l, PW) * LJ + jac_next(PW - 1 - l, PW);
    float app = S[JAC_G(0) + l * LJ + l].x, aqq = S[JAC_G(0) + (PW - 1 - l) * (LJ + 1)].x;
    JacRot r = jac_rotation(app, aqq, S[JAC_G(0) + l * LJ + PW - 1 - l], rel, floor_abs);
    if (act) js.rot[0][l] = make_float4(r.c, r.sx, r.sy, 0.f);
    bool again = act && r.again, pend = act && r.moved;
    __syncthreads();
    for (int sweep = 0; sweep < 30; ++sweep) {
      mv |= pend;
      for (int k = 0; k < PW - 1; ++k) {
        if (k == PW - 2) {
          const bool any = __any_sync(0xffffffffu, again);
          if (lane == 0) js.again = any;
          again = false;
        }
        const float2* g = S + JAC_G(buf);
        const float2 x00 = g[o00], x01 = g[o01], x10 = g[o10], x11 = g[o11];
        const float4 rr = js.rot[buf][R], rc = js.rot[buf][C];
        // the diagonals after this round, at their new pairs
        const float np = app - r.shift, nq = aqq + r.shift;
        const float dn = __shfl_down_sync(0xffffffffu, np, 1), up = __shfl_up_sync(0xffffffffu, nq, 1);
        app = l == 0 ? np : l == HALF - 1 ? nq : dn;
        aqq = l == 0 ? dn : up;
        // columns (c, -conj(s)) or (s, c), rows (c, -s) or (conj(s), c)
        const float2 ca = colq ? cf(rc.y, rc.z) : cf(rc.x, 0.f), cb = colq ? cf(rc.x, 0.f) : cf(-rc.y, rc.z);
        const float2 ra = rowq ? cf(rr.y, -rr.z) : cf(rr.x, 0.f), rb = rowq ? cf(rr.x, 0.f) : cf(-rr.y, -rr.z);
        float2 top = fmac(fmac(cf(0.f, 0.f), ca, x00), cb, x01);
        float2 bot = fmac(fmac(cf(0.f, 0.f), ca, x10), cb, x11);
        float2 e = fmac(fmac(cf(0.f, 0.f), ra, top), rb, bot);
        if (l != 0) e.y = -e.y;
        r = jac_rotation(app, aqq, e, rel, floor_abs);
        if (act) {
          js.rot[buf ^ 1][l] = make_float4(r.c, r.sx, r.sy, 0.f);
          S[JAC_G(buf ^ 1) + zero] = cf(0.f, 0.f);
        }
        again |= act && r.again;
        pend = act && r.moved;
        if (k < PW - 2) mv |= pend;
        __syncthreads();
        buf ^= 1;
      }
      if (!js.again) break;
    }
  } else if (warp < GWARP) {
    const int h = (warp - 1) & 3, row = ((warp - 1) >> 2) * 32 + lane;
    const bool idle = h >= NG || row - lane >= w;
    float2 p[NP], q[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int l = h * NP + i;
      p[i] = cf(row == l ? 1.f : 0.f, 0.f);
      q[i] = cf(row == PW - 1 - l ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    for (int sweep = 0; sweep < 30; ++sweep) {
      for (int k = 0; k < PW - 1; ++k) {
        if (!idle) {
          if (k + sweep > 0) {
            if (h > 0) q[0] = js.edge[buf ^ 1][1][h - 1][row];
            if (h < NG - 1) (NP == 1 && h == 0 ? q[0] : p[NP - 1]) = js.edge[buf ^ 1][0][h + 1][row];
          }
          const float4* rot = js.rot[buf] + h * NP;
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            const float4 r = rot[i];
            jacobi32_cols(p[i], q[i], r.x, r.y, r.z);
          }
          // every column one position on; the ends go by shared memory
          const float2 p0 = p[0], p1 = p[NP > 1 ? 1 : 0], q0 = q[NP - 1];
          if (h > 0) js.edge[buf][0][h][row] = p0;
          if (h < NG - 1) js.edge[buf][1][h][row] = q0;
#pragma unroll
          for (int i = NP - 1; i > 0; --i) q[i] = q[i - 1];
#pragma unroll
          for (int i = 0; i < NP - 1; ++i) p[i] = p[i + 1];
          if (h == 0) p[0] = p0, q[0] = p1;
          if (h == NG - 1) p[NP - 1] = q0;
        }
        __syncthreads();
        buf ^= 1;
      }
      if (!js.again) break;
    }
    if (!idle) {   // the last round's exchange
      if (h > 0) q[0] = js.edge[buf ^ 1][1][h - 1][row];
      if (h < NG - 1) (NP == 1 && h == 0 ? q[0] : p[NP - 1]) = js.edge[buf ^ 1][0][h + 1][row];
    }
    if (!idle && row < w)
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const int l = h * NP + i;
        if (l < w) S[vout + row * ld + l] = p[i];
        if (PW - 1 - l < w) S[vout + row * ld + PW - 1 - l] = q[i];
      }
  } else {
    int R[GIT], C[GIT], st[GIT][4];
    bool act[GIT], flip[GIT];
#pragma unroll
    for (int u = 0; u < GIT; ++u) {
      const int P = warp - GWARP + u * GWARPS;
      act[u] = P < HALF / 2 && lane < HALF && lane != P;
      R[u] = lane > P ? P : HALF - 1 - P;
      C[u] = lane > P ? lane : HALF - 1 - lane;
      if (!act[u]) R[u] = 0, C[u] = 1;
      flip[u] = false;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int x = jac_next(e & 2 ? PW - 1 - R[u] : R[u], PW), y = jac_next(e & 1 ? PW - 1 - C[u] : C[u], PW);
        const int px = min(x, PW - 1 - x), py = min(y, PW - 1 - y);
        st[u][e] = px < py ? x * LJ + y : px > py ? y * LJ + x : SPARE + lane;   // the next pair's own: warp 0 has it
        if (e == 2) flip[u] = px > py;
      }
    }
    __syncthreads();
    for (int sweep = 0; sweep < 30; ++sweep) {
      for (int k = 0; k < PW - 1; ++k) {
        const float2* g = S + JAC_G(buf);
        float2* o = S + JAC_G(buf ^ 1);
#pragma unroll
        for (int u = 0; u < GIT; ++u) {
          if (!act[u]) continue;
          const float4 rc = js.rot[buf][C[u]], rr = js.rot[buf][R[u]];
          const float2 *g0 = g + R[u] * LJ, *g1 = g + (PW - 1 - R[u]) * LJ;
          float2 x00 = g0[C[u]], x01 = g0[PW - 1 - C[u]], x10 = g1[C[u]], x11 = g1[PW - 1 - C[u]];
          // columns: col_p <- c col_p - conj(s) col_q ; col_q <- s col_p + c col_q
          jacobi32_cols(x00, x01, rc.x, rc.y, rc.z);
          jacobi32_cols(x10, x11, rc.x, rc.y, rc.z);
          // rows: row_p <- c row_p - s row_q ; row_q <- conj(s) row_p + c row_q
          jacobi32_cols(x00, x10, rr.x, rr.y, -rr.z);
          jacobi32_cols(x01, x11, rr.x, rr.y, -rr.z);
          if (flip[u]) x10.y = -x10.y;
          o[st[u][0]] = x00;
          o[st[u][1]] = x01;
          o[st[u][2]] = x10;
          o[st[u][3]] = x11;
        }
        __syncthreads();
        buf ^= 1;
      }
      if (!js.again) break;
    }
  }
  return __syncthreads_or(mv);
}

// V (stride ld, at offset vout of the shared memory) of the Hermitian w x w
// matrix g(i, j).
template <class F>
__device__ bool jacobi32_run(F g, int vout, int w, int ld, float rel, float floor_abs) {
  // pw: 4, 8, 16, 24, 32, 48 or 64
  const int pw = w <= 4 ? 4 : w <= 8 ? 8 : w <= 32 ? (w + 7) / 8 * 8 : (w + 15) / 16 * 16;
  float2* S = tt_smf() + JAC_G(0);
  for (int e = threadIdx.x; e < pw * pw; e += blockDim.x) {
    const int i = e / pw, j = e % pw;
    S[i * (pw + 1) + j] = i < w && j < w ? g(i, j) : cf(0.f, 0.f);
  }
  __syncthreads();
  switch (pw) {
    case 4: return jacobi32_sweeps<1, 2>(vout, w, ld, rel, floor_abs);
    case 8: return jacobi32_sweeps<1, 4>(vout, w, ld, rel, floor_abs);
    case 16: return jacobi32_sweeps<2, 4>(vout, w, ld, rel, floor_abs);
    case 24: return jacobi32_sweeps<3, 4>(vout, w, ld, rel, floor_abs);
    case 32: return jacobi32_sweeps<4, 4>(vout, w, ld, rel, floor_abs);
    case 48: return jacobi32_sweeps<6, 4>(vout, w, ld, rel, floor_abs);
    default: return jacobi32_sweeps<8, 4>(vout, w, ld, rel, floor_abs);
  }
}

// A 4 x 2 block of outputs of a w x w product: rows r0 .. (rows past w - 1
// repeat the last one and are not used), columns c0, c0 + 1.  Block t of all
// of them, or with `upper` of those that touch the upper triangle; false
// past the last one.
struct TTBlock {
  int r0, c0, nr;
  int rr[4];
};
__device__ __forceinline__ bool tt_block(int w, int t, bool upper, TTBlock& o) {
  const int cp = w / 2, rq = (w + 3) / 4;
  int i = 0, j = t;
  if (upper) {
    while (i < rq && j >= cp - 2 * i) {
      j -= cp - 2 * i;
      ++i;
    }
    j += 2 * i;
  } else {
    i = t / cp;
    j = t % cp;
  }
  o.r0 = 4 * i;
  o.c0 = 2 * j;
  o.nr = min(4, w - o.r0);
#pragma unroll
  for (int k = 0; k < 4; ++k) o.rr[k] = min(o.r0 + k, w - 1);
  return i < rq;
}

// out = op(A) B in double-float, op the adjoint with ADJ.
template <bool ADJ>
__device__ __forceinline__ void tt_df_block(const xc* A, const xc* B, int w, int ld, const TTBlock& o, XA (&acc)[4][2]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = xa_zero();
  for (int k = 0; k < w; ++k) {
    const xc b0 = B[k * ld + o.c0], b1 = B[k * ld + o.c0 + 1];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const xc a = ADJ ? A[k * ld + o.rr[i]] : A[o.rr[i] * ld + k];
      if (ADJ) {
        xa_macc(acc[i][0], a, b0);
        xa_macc(acc[i][1], a, b1);
      } else {
        xa_mac(acc[i][0], a, b0);
        xa_mac(acc[i][1], a, b1);
      }
    }
  }
}

// out = op(A) B in FP32.
template <bool ADJ>
__device__ __forceinline__ void tt_f_block(const float2* A, const float2* B, int w, int ld, const TTBlock& o,
                                           float2 (&acc)[4][2]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = cf(0.f, 0.f);
  for (int k = 0; k < w; ++k) {
    const float2 b0 = B[k * ld + o.c0], b1 = B[k * ld + o.c0 + 1];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 a = ADJ ? A[k * ld + o.rr[i]] : A[o.rr[i] * ld + k];
      if (ADJ) a.y = -a.y;
      acc[i][0] = fmac(acc[i][0], a, b0);
      acc[i][1] = fmac(acc[i][1], a, b1);
    }
  }
}

// v + x in double-float
__device__ __forceinline__ xc tt_plus(xc v, float2 x) {
  DF re = {v.x, v.z}, im = {v.y, v.w};
  df_add(re, x.x, 0.f);
  df_add(im, x.y, 0.f);
  const float2 r = df_norm(re), i = df_norm(im);
  return make_float4(r.x, i.x, r.y, i.y);
}
static_assert(TT_EIG_SMEM_W / 2 * (TT_EIG_SMEM_W / 4) <= TT_EIG_THREADS, "one block of outputs per thread");

// Diagonalise the w x w Gram G (double-float, shared memory, scaled to a
// trace in [1/2, 1)): G's diagonal becomes the eigenvalues, Vg (double-float,
// global memory, stride w) the vectors.  Shared memory holds G, V_k and a
// work matrix, the FP32 copies in the last two.
__device__ void tt_df_eig(xc* Vg, int w, int ld) {
  xc *G = tt_smx(), *vk = tt_smx() + w * ld, *t = tt_smx() + 2 * w * ld;
  float2* t32 = tt_smf() + 4 * w * ld;
  bool first = true;   // V is still I
  float floor_abs = 1e-7f;
  for (int pass = 0; pass < 7; ++pass) {
    const bool moved = jacobi32_run(
        [&](int i, int j) {
          const xc g = G[i * ld + j];
          return cf(g.x, i == j ? 0.f : g.y);
        },
        2 * w * ld, w, ld, 1e-7f, floor_abs);
    // nothing above FP32's noise at G's scale: G is graded as it is, and the
    // couplings among its small entries are resolved from it at once
    const bool coarse = floor_abs > 1e-13f;
    floor_abs = 1e-13f;
    if (!moved && coarse) continue;
    const float2* vr = tt_smf() + 2 * w * ld;
    // the thread's blocks, computed anew in every pass: kept over the sweeps
    // they would be spilled
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    TTBlock o, u;
    const bool mine = tt_block(w, tid, false, o), uppr = tt_block(w, tid, true, u);
    if (!moved) {
      // V_k = I + X with X below 3e-7: D = -(X + X^H + X^H X) / 2 and the
      // products with X or D are FP32, and G's diagonal stands: a tangent x
      // moves its pair's eigenvalues by x^2 of their difference, together
      // less than 1e-13 of the trace, the rotations' floor
      for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
        const int i = e / w, j = e % w;
        const float2 x = vr[i * ld + j];
        t32[i * ld + j] = cf(i == j ? x.x - 1.f : x.x, x.y);
      }
      __syncthreads();
      float2 acc[4][2];
      if (mine) {
        tt_f_block<true>(t32, t32, w, ld, o, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float2 x = t32[o.rr[i] * ld + o.c0 + j], y = t32[(o.c0 + j) * ld + o.rr[i]];
            // X + D
            acc[i][j] = cf(x.x - 0.5f * (x.x + y.x + acc[i][j].x), x.y - 0.5f * (x.y - y.y + acc[i][j].y));
          }
      }
      __syncthreads();
      float2* z = t32 + w * ld;
      if (mine)
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i >= o.nr) continue;
          z[(o.r0 + i) * ld + o.c0] = acc[i][0];
          z[(o.r0 + i) * ld + o.c0 + 1] = acc[i][1];
        }
      for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
        const xc v = first ? make_float4(e / w == e % w ? 1.f : 0.f, 0.f, 0.f, 0.f) : Vg[e];
        t32[(e / w) * ld + e % w] = cf(v.x, v.y);
      }
      __syncthreads();
      if (mine) {
        tt_f_block<false>(t32, z, w, ld, o, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (i >= o.nr) continue;
            const int e = (o.r0 + i) * w + o.c0 + j;
            const xc v = first ? make_float4(o.r0 + i == o.c0 + j ? 1.f : 0.f, 0.f, 0.f, 0.f) : Vg[e];
            Vg[e] = tt_plus(v, acc[i][j]);
          }
      }
      __syncthreads();
      return;
    }
    // D = (I - V_k^H V_k) / 2 (Hermitian)
    float2* d32 = t32;
    if (uppr) {
      DF acc[4][2][2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = DF{0.f, 0.f};
      for (int k = 0; k < w; ++k) {
        const float2 b[2] = {vr[k * ld + u.c0], vr[k * ld + u.c0 + 1]};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = vr[k * ld + u.rr[i]];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            df_add_prod(acc[i][j][0], a.x, b[j].x);
            df_add_prod(acc[i][j][0], a.y, b[j].y);
            df_add_prod(acc[i][j][1], a.x, b[j].y);
            df_add_prod(acc[i][j][1], -a.y, b[j].x);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (i >= u.nr) continue;
          const int r = u.r0 + i, c = u.c0 + j;
          const float one = r == c ? 1.f : 0.f;
          const float2 d = cf(0.5f * ((one - acc[i][j][0].hi) - acc[i][j][0].lo),
                              -0.5f * (acc[i][j][1].hi + acc[i][j][1].lo));
          if (r <= c) d32[r * ld + c] = d;
          if (r < c) d32[c * ld + r] = cf(d.x, -d.y);
        }
    }
    __syncthreads();
    // V_k (I - 2D)^(-1/2) = V_k (I + D + 3/2 D^2 + ...): after many FP32 rotations D is a few
    // 1e-6, whose square shows at 1e-12
    float2* z32 = t32 + w * ld;
    if (mine) {
      float2 acc[4][2];
      tt_f_block<false>(d32, d32, w, ld, o, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (i >= o.nr) continue;
          const float2 d = d32[(o.r0 + i) * ld + o.c0 + j];
          z32[(o.r0 + i) * ld + o.c0 + j] = cf(fmaf(1.5f, acc[i][j].x, d.x), fmaf(1.5f, acc[i][j].y, d.y));
        }
    }
    __syncthreads();
    xc nv[4][2];
    if (mine) {
      float2 acc[4][2];
      tt_f_block<false>(vr, z32, w, ld, o, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 v = vr[o.rr[i] * ld + o.c0 + j];
          nv[i][j] = tt_plus(make_float4(v.x, v.y, 0.f, 0.f), acc[i][j]);
        }
    }
    __syncthreads();
    if (mine)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i >= o.nr) continue;
        vk[(o.r0 + i) * ld + o.c0] = nv[i][0];
        vk[(o.r0 + i) * ld + o.c0 + 1] = nv[i][1];
      }
    __syncthreads();
    // G <- V_k^H (G V_k), Hermitian
    if (mine) {
      XA acc[4][2];
      tt_df_block<false>(G, vk, w, ld, o, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i >= o.nr) continue;
        t[(o.r0 + i) * ld + o.c0] = xa_round(acc[i][0]);
        t[(o.r0 + i) * ld + o.c0 + 1] = xa_round(acc[i][1]);
      }
    }
    __syncthreads();
    if (uppr) {
      XA acc[4][2];
      tt_df_block<true>(vk, t, w, ld, u, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (i >= u.nr) continue;
          const int r = u.r0 + i, c = u.c0 + j;
          const xc g = xa_round(acc[i][j]);
          if (r <= c) G[r * ld + c] = r == c ? make_float4(g.x, 0.f, g.z, 0.f) : g;
          if (r < c) G[c * ld + r] = xc_conj(g);
        }
    }
    __syncthreads();
    // V <- V V_k
    if (first) {
      first = false;
      for (int e = threadIdx.x; e < w * w; e += blockDim.x) Vg[e] = vk[(e / w) * ld + e % w];
    } else {
      for (int e = threadIdx.x; e < w * w; e += blockDim.x) t[(e / w) * ld + e % w] = Vg[e];
      __syncthreads();
      if (mine) {
        XA acc[4][2];
        tt_df_block<false>(t, vk, w, ld, o, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i >= o.nr) continue;
          Vg[(o.r0 + i) * w + o.c0] = xa_round(acc[i][0]);
          Vg[(o.r0 + i) * w + o.c0 + 1] = xa_round(acc[i][1]);
        }
      }
    }
    __syncthreads();
  }
}

// Entry t of the upper triangle, column by column: (i, j), i <= j.
__device__ __forceinline__ void tt_upper(int t, int* i, int* j) {
  int c = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while (c * (c + 1) / 2 > t) --c;
  while ((c + 1) * (c + 2) / 2 <= t) ++c;
  *j = c;
  *i = t - c * (c + 1) / 2;
}

// FP64 finish of nearly exact vectors V of G (both w x w, stride ld, shared
// memory), by one first-order step (Ogita & Aishima, as in ttsvd_wide.cu):
// S = V^H G V and R = I - V^H V in FP64, l_j = S_jj / (1 - R_jj), E_ij =
// (S_ij + l_j R_ij) / (l_j - l_i), E_jj = R_jj / 2, V <- V (I + E + E^2 / 2)
// with FP32 products.  Pairs coupled by at most floor_abs only share their
// defect, E_ij = R_ij / 2.  False, with G and V unchanged, if an entry of E is
// above 2e-6 (its cube, or FP32's rounding of it, would show): FP64 sweeps
// take it.  T is scratch.
// FP64 instructions bound it (64 cycles each per SM quarter): two products
// instead of the four, and the sweeps, that a Newton-Schulz step, the
// similar matrix and Jacobi rotations took.  Measured over the 15 launches
// of a batch of exact encodes (Grams up to 16 wide): 3.6 -> 1.5 ms with the passes before it.
__device__ bool tt_refine(const double2* G, double2* V, double2* T, double* lam, int w, int ld, double floor_abs) {
  const int nu = w * (w + 1) / 2;
  float2* E = reinterpret_cast<float2*>(T);   // after its last use
  float2* V32 = E + w * ld;   // E + E^2 / 2, then V
  // upper triangles of S and R, two entries each per thread (w <= 64: up to five)
  constexpr int PER = (TT_EIG_SMEM_W * (TT_EIG_SMEM_W + 1) / 2 + TT_EIG_THREADS - 1) / TT_EIG_THREADS;
  for (int e = threadIdx.x; e < w * w; e += TT_EIG_THREADS) {   // T = G V
    const int i = e / w, j = e % w;
    double2 a = czero();
    for (int k = 0; k < w; ++k) {
      const double2 x = G[i * ld + k], y = V[k * ld + j];
      a.x = fma(x.x, y.x, a.x);
      a.y = fma(x.x, y.y, a.y);
      a.x = fma(-x.y, y.y, a.x);
      a.y = fma(x.y, y.x, a.y);
    }
    T[i * ld + j] = a;
  }
  __syncthreads();
  double2 S[PER], R[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int t = threadIdx.x + u * TT_EIG_THREADS;
    S[u] = R[u] = czero();
    if (t >= nu) continue;
    int i, j;
    tt_upper(t, &i, &j);
    double2 a = czero(), b = cd(i == j ? 1.0 : 0.0, 0.0);
    for (int k = 0; k < w; ++k) {   // conj(v) (G V), - conj(v) v
      const double2 v = V[k * ld + i], x = T[k * ld + j], y = V[k * ld + j];
      a.x = fma(v.x, x.x, a.x);
      a.y = fma(v.x, x.y, a.y);
      b.x = fma(-v.x, y.x, b.x);
      b.y = fma(-v.x, y.y, b.y);
      a.x = fma(v.y, x.y, a.x);
      a.y = fma(-v.y, x.x, a.y);
      b.x = fma(-v.y, y.y, b.x);
      b.y = fma(v.y, y.x, b.y);
    }
    S[u] = a;
    R[u] = b;
    if (i == j) lam[i] = a.x / (1.0 - b.x);
  }
  __syncthreads();   // lam; T is read
  bool ok = true;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int t = threadIdx.x + u * TT_EIG_THREADS;
    if (t >= nu) continue;
    int i, j;
    tt_upper(t, &i, &j);
    const float2 r = cf((float)R[u].x, (float)R[u].y);
    float2 up = cf(0.5f * r.x, i == j ? 0.f : 0.5f * r.y), lo = cf(up.x, -up.y);
    if (i != j) {
      const float2 b = cf((float)fma(lam[j], R[u].x, S[u].x), (float)fma(lam[j], R[u].y, S[u].y));
      if (fmaf(b.x, b.x, b.y * b.y) > (float)floor_abs * (float)floor_abs) {
        const float d = (float)(lam[j] - lam[i]);
        up = cf(__fdividef(b.x, d), __fdividef(b.y, d));
        lo = cf(r.x - up.x, -(r.y - up.y));   // E + E^H = R
      }
      E[j * ld + i] = lo;
    }
    E[i * ld + j] = up;
    ok = ok && fabsf(up.x) < 2e-6f && fabsf(up.y) < 2e-6f && fabsf(lo.x) < 2e-6f && fabsf(lo.y) < 2e-6f;
  }
  if (!__syncthreads_and(ok)) return false;
  for (int e = threadIdx.x; e < w * w; e += TT_EIG_THREADS) {
    const int i = e / w, j = e % w;
    float2 a = cf(0.f, 0.f);
    for (int k = 0; k < w; ++k) a = fmac(a, E[i * ld + k], E[k * ld + j]);
    V32[i * ld + j] = cf(fmaf(0.5f, a.x, E[i * ld + j].x), fmaf(0.5f, a.y, E[i * ld + j].y));
  }
  __syncthreads();
  {
    float2* t = E;
    E = V32;
    V32 = t;
  }
  for (int e = threadIdx.x; e < w * w; e += TT_EIG_THREADS) {
    const double2 v = V[e / w * ld + e % w];
    V32[e / w * ld + e % w] = cf((float)v.x, (float)v.y);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < w * w; e += TT_EIG_THREADS) {
    const int i = e / w, j = e % w;
    float2 a = cf(0.f, 0.f);
    for (int k = 0; k < w; ++k) a = fmac(a, V32[i * ld + k], E[k * ld + j]);
    const double2 v = V[i * ld + j];
    V[i * ld + j] = cd(v.x + (double)a.x, v.y + (double)a.y);
  }
  __syncthreads();
  return true;
}

// an eigenvalue for sorting: NaN counts as negative, so that ranks stay a permutation
__device__ __forceinline__ double tt_number(double v) { return v == v ? v : -1.0; }

// One CTA per state; G and V are row-major w x w.  For w <= TT_EIG_SMEM_W
// they are diagonalised in shared memory by the double-float passes above;
// the exact mode (fine = 1e-15 of the trace) continues from those vectors
// with one FP64 step (tt_refine), or where that does not do with a
// Newton-Schulz step and FP64 sweeps.  For 64 < w <= 128 the
// vectors are found in global memory (L2 resident) in two precisions: FP32
// Jacobi sweeps on a float copy of G in `scratch32` (the Gram partials,
// already reduced), one Newton-Schulz step V <- V (3I - V^H V) / 2 in FP64
// (its FP32 error of about 1e-7 leaves about 1e-14), G replaced by the
// similar, nearly diagonal V^H G V, and FP64 sweeps down to `fine` of the
// trace, with the FP64 scratch in the state's slot of `vsel` (written only
// at the end).
__global__ void __launch_bounds__(TT_EIG_THREADS) k_tt_eig(BatchDev bd, int step, int* bonds, double2* gram,
                                                          double2* vwork, int max_bond, double cutoff,
                                                          double2* vsel, double2* tensors, int chi,
                                                          float2* scratch32, double fine) {
  grid_wait();
  __shared__ JacobiShared<double2, double> js64;
  __shared__ JacobiShared<float2, float> js32;
  __shared__ double s_floor;
  __shared__ double s_lam[TT_MAXW], s_sorted[TT_MAXW];
  __shared__ int s_perm[TT_MAXW];
  __shared__ int s_keep;
  const int64_t WW = (int64_t)bd.tt_w * bd.tt_w;
  const int b = blockIdx.x;
  if (b >= bd.B) return;
  const int n = bd.n[b];
  const int c = n - 1 - step;
  if (c < 1) return;
  int* bond = bonds + (int64_t)b * (bd.max_n + 1);
  const int r = bond[c + 1];
  if (!bond_ok(r, bd.tt_b)) {
    if (threadIdx.x == 0) bond[c] = -1;   // poison: every later step skips this state
    return;
  }
  const int w = 2 * r;
  if (w > bd.eig_wmax) return;   // diagonalised by the blocked solver (ttsvd_wide.cu)
  double2* Gg = gram + (int64_t)b * WW;
  double2* Vg = vwork + (int64_t)b * WW;
  const bool in_smem = w <= TT_EIG_SMEM_W;
  const int ld = in_smem ? w + TT_EIG_PAD : w;   // padded rows: both diagonals hit distinct banks
  double2* G = in_smem ? eig_sm : Gg;
  double2* V = in_smem ? eig_sm + w * ld : Vg;
  double2* Sc = in_smem ? eig_sm + 2 * w * ld : vsel + (int64_t)b * WW;   // FP64 scratch
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  if (warp == 0) {   // the trace (a positive semidefinite G: its scale)
    double tr = 0.0;
    for (int i = lane; i < w; i += 32) tr += fabs(Gg[i * w + i].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    if (lane == 0) s_floor = tr;
  }
  __syncthreads();
  const double tr = s_floor;
  bool fp64 = !in_smem;   // FP64 sweeps to `fine`
  double trg = tr;        // of the scaled G
  if (in_smem) {
    int ex = 0;
    if (tr > 0.0 && isfinite(tr)) frexp(tr, &ex);
    const double sc = ldexp(1.0, -ex);
    trg = tr * sc;
    xc* Gx = reinterpret_cast<xc*>(G);
    xc* Vx = reinterpret_cast<xc*>(Vg);
    for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
      const double2 g = Gg[e];
      Gx[(e / w) * ld + e % w] = xc_from_d(cd(g.x * sc, g.y * sc));
    }
    __syncthreads();
    tt_df_eig(Vx, w, ld);
    for (int i = threadIdx.x; i < w; i += blockDim.x) s_lam[i] = tt_number(xc_to_d(Gx[i * ld + i]).x);
    for (int e = threadIdx.x; e < w * w; e += blockDim.x) V[(e / w) * ld + e % w] = xc_to_d(Vx[e]);
    __syncthreads();
    if (fine < 1e-14) {
      for (int e = threadIdx.x; e < w * w; e += blockDim.x) G[(e / w) * ld + e % w] = cscale(Gg[e], sc);
      __syncthreads();
      fp64 = !tt_refine(G, V, Sc, s_lam, w, ld, fine * trg);
      if (!fp64) {
        for (int i = threadIdx.x; i < w; i += blockDim.x) s_lam[i] = tt_number(s_lam[i]);
        __syncthreads();
      }
    }
  } else {
    float2* G32 = scratch32 + 2 * bd.tt_off[b];
    float2* V32 = G32 + w * ld;
    for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
      const int i = e / w, j = e % w;
      const double2 g = G[i * ld + j];
      G32[i * ld + j] = cf((float)g.x, (float)g.y);
      V32[i * ld + j] = cf(i == j ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    jacobi_run<float2, float>(G32, V32, w, ld, 1e-7f, (float)(1e-7 * tr), 40, js32);
    for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
      const int i = e / w, j = e % w;
      V[i * ld + j] = f2d(V32[i * ld + j]);
    }
    __syncthreads();
  }
  if (fp64) {
    // Newton-Schulz: Sc = (3I - V^H V) / 2, then V <- V Sc row by row (a
    // warp per row, each lane up to four columns, written after the warp's reads)
    smem_matmul(V, V, Sc, w, ld, true);
    __syncthreads();
    for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
      const int i = e / w, j = e % w;
      const double2 v = Sc[i * ld + j];
      Sc[i * ld + j] = cd((i == j ? 1.5 : 0.0) - 0.5 * v.x, -0.5 * v.y);
    }
    __syncthreads();
    for (int row = warp; row < w; row += nwarps) {
      double2 o[TT_MAXW / 32];
#pragma unroll
      for (int q = 0; q < TT_MAXW / 32; ++q) o[q] = czero();
      for (int k = 0; k < w; ++k) {
        const double2 v = V[row * ld + k];
#pragma unroll
        for (int q = 0; q < TT_MAXW / 32; ++q)
          if (lane + 32 * q < w) o[q] = cadd(o[q], cmul(v, Sc[k * ld + lane + 32 * q]));
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < TT_MAXW / 32; ++q)
        if (lane + 32 * q < w) V[row * ld + lane + 32 * q] = o[q];
    }
    __syncthreads();
    // G <- V^H (G V)
    smem_matmul(G, V, Sc, w, ld, false);
    __syncthreads();
    smem_matmul(V, Sc, G, w, ld, true);
    __syncthreads();
    for (int i = threadIdx.x; i < w; i += blockDim.x) G[i * ld + i].y = 0.0;
    __syncthreads();
    // Absolute rotation floor: off-diagonals at most `fine` of the trace move
    // no eigenvalue by more than that (three to five orders below the 1e-10
    // truncation cutoff).  Without it the rounding-level null-space block of
    // a rank-deficient Gram keeps rotating until the sweep limit.
    jacobi_run<double2, double>(G, V, w, ld, 1e-15, fine * trg, 40, js64);
    for (int i = threadIdx.x; i < w; i += blockDim.x) s_lam[i] = tt_number(G[i * ld + i].x);
    __syncthreads();
  }
  // descending order (ties by index)
  for (int i = threadIdx.x; i < w; i += blockDim.x) {
    const double li = s_lam[i];
    int rank = 0;
    for (int j = 0; j < w; ++j) rank += s_lam[j] > li || (s_lam[j] == li && j < i);
    s_perm[rank] = i;
    s_sorted[rank] = li;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int keep = rank_by_cutoff(s_sorted, w, cutoff, max_bond);
    if (keep > bd.tt_b) keep = bd.tt_b;
    if (c < 30 && keep > (1 << c)) keep = 1 << c;   // M has 2^c rows: rank <= 2^c
    s_keep = keep;
    bond[c] = keep;
  }
  __syncthreads();
  const int keep = s_keep;
  // canonical phases (the rule of phase_fix_column), a warp per kept column
  for (int k = warp; k < keep; k += nwarps) {
    const int col = s_perm[k];
    double mag[TT_MAXW / 32], m2 = -1.0;
#pragma unroll
    for (int q = 0; q < TT_MAXW / 32; ++q) {
      const int i = lane + 32 * q;
      mag[q] = i < w ? cnorm2(V[i * ld + col]) : -1.0;
      m2 = fmax(m2, mag[q]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    const double lim = (1.0 - QM_PIVOT_TOL) * (1.0 - QM_PIVOT_TOL) * m2;
    int piv = w;
#pragma unroll
    for (int q = TT_MAXW / 32 - 1; q >= 0; --q)
      if (lane + 32 * q < w && mag[q] >= lim) piv = lane + 32 * q;
    piv = __reduce_min_sync(0xffffffffu, piv);
    const double2 z = piv < w ? V[piv * ld + col] : czero();
    const double az = sqrt(cnorm2(z));
    __syncwarp();
    if (az > 0.0) {
      const double2 ph = cscale(cconj(z), 1.0 / az);
      for (int i = lane; i < w; i += 32) V[i * ld + col] = cmul(V[i * ld + col], ph);
    }
  }
  __syncthreads();
  double2* vs = vsel + (int64_t)b * WW;
  for (int e = threadIdx.x; e < w * keep; e += blockDim.x) {
    const int a = e / keep, col = e % keep;
    vs[(int64_t)a * bd.tt_b + col] = V[a * ld + s_perm[col]];
  }
  const int ce = chi_eff(chi, n);
  double2* ts = tensors + bd.tensor_off[b] + (int64_t)c * 2 * ce * ce;
  for (int e = threadIdx.x; e < keep * 2 * r; e += blockDim.x) {
    const int l = e / (2 * r), pr = e % (2 * r);   // e = l * 2r + (p * r + rr)
    ts[e] = cconj(V[pr * ld + s_perm[l]]);
  }
}

// Dynamic shared memory: V (TT_MAXW x TT_MAXB float2) then TT_CH rows.
// Sum of `count` complex FP32 products x(k) v(k) in double-float, rounded once.
// States of up to TT_DOT_QUBITS qubits take it in the projections and the
// target's contraction: FP32 chains were most of the target's rounding there
// (8 qubits: 3.3e-7 of its norm, 1.4e-7 so), which the layers multiply (the
// prepared state of two layers and a sweep: error 0.60 times, 160 states).
// A larger state's one block would show the ten times as many operations (12
// qubits at bond 64: 3.7 -> 3.9 ms; 10 qubits at bond 32: within the spread).
#define TT_DOT_QUBITS 10
#define TT_DOT_BOND (1 << (TT_DOT_QUBITS / 2))   // their largest bond
__device__ __forceinline__ void tt_dot_mac(DF& re, DF& im, float2 a, float2 b) {
  df_add_prod(re, a.x, b.x);
  df_add_prod(re, -a.y, b.y);
  df_add_prod(im, a.x, b.y);
  df_add_prod(im, a.y, b.x);
}

// o[row][col] = sum_a x[row][a] v[a][col] for nr x nc outputs (rows of x
// ldx apart; not inlined: the larger states' loops keep their registers)
__device__ __noinline__ void tt_small_product(const float2* x, int ldx, const float2* v, int w, int nr, int nc,
                                              float2* o) {
  for (int e = threadIdx.x; e < nr * nc; e += blockDim.x) {
    const int row = e / nc, col = e % nc;
    DF re = {0.f, 0.f}, im = {0.f, 0.f};
    for (int k = 0; k < w; ++k) tt_dot_mac(re, im, x[row * ldx + k], v[k * nc + col]);
    o[e] = cf(re.hi + re.lo, im.hi + im.lo);
  }
}

__global__ void __launch_bounds__(BLOCK_THREADS) k_tt_project(BatchDev bd, int step, const float2* sv,
                                                              const float2* src, float2* dst,
                                                              const int* bonds, const double2* vsel) {
  grid_wait();
  extern __shared__ float2 sh[];
  float2* vs = sh;
  float2* xs = sh + TT_MAXW * TT_MAXB;
  const int64_t WW = (int64_t)bd.tt_w * bd.tt_w;
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    const int n = bd.n[b];
    const int c = n - 1 - step;
    if (c < 1) continue;
    const int* bond = bonds + (int64_t)b * (bd.max_n + 1);
    const int r = bond[c + 1];
    const int keep = bond[c];
    if (!bond_ok(r, bd.tt_b) || !bond_ok(keep, bd.tt_b)) continue;
    const int w = 2 * r;
    if (w > bd.eig_wmax || keep > TT_MAXB) continue;   // projected by k_cgemm
    __syncthreads();
    for (int e = threadIdx.x; e < w * keep; e += blockDim.x) {
      const double2 v = vsel[(int64_t)b * WW + (int64_t)(e / keep) * bd.tt_b + (e % keep)];
      vs[e] = cf((float)v.x, (float)v.y);
    }
    const float2* m = (step == 0 ? sv : src) + bd.vec_off[b];
    float2* o = dst + bd.vec_off[b];
    int64_t lo, hi;
    tile_range(ipow2(c), bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    for (int64_t r0 = lo; r0 < hi; r0 += TT_CH) {
      const int nr = (int)((hi - r0) < TT_CH ? (hi - r0) : TT_CH);
      __syncthreads();
      for (int e = threadIdx.x; e < nr * w; e += blockDim.x) xs[(e / w) * TT_MAXW + e % w] = m[(r0 + e / w) * w + e % w];
      __syncthreads();
      if (n <= TT_DOT_QUBITS) {
        tt_small_product(xs, TT_MAXW, vs, w, nr, keep, o + r0 * keep);
        continue;
      }
      for (int e = threadIdx.x; e < nr * keep; e += blockDim.x) {
        const int rr = e / keep, col = e % keep;
        float2 acc = cf(0.f, 0.f);
        for (int a = 0; a < w; ++a) acc = fmac(acc, xs[rr * TT_MAXW + a], vs[a * keep + col]);
        o[(r0 + rr) * keep + col] = acc;
      }
    }
    __syncthreads();
  }
}

__global__ void k_tt_site0(BatchDev bd, const float2* rem0, const float2* rem1, const int* bonds,
                           double2* tensors, int chi, const double2* in_sq) {
  grid_wait();
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < bd.B; b += gridDim.x * blockDim.x) {
    const int n = bd.n[b];
    const int* bond = bonds + (int64_t)b * (bd.max_n + 1);
    const int r1 = bond[1];
    if (!bond_ok(r1, bd.tt_b)) continue;
    const float2* rem = (((n - 2) & 1) ? rem1 : rem0) + bd.vec_off[b];
    double nrm = 0.0;
    for (int i = 0; i < 2 * r1; ++i) nrm += cnorm2(f2d(rem[i]));
    nrm = sqrt(nrm);
    const double f = nrm > 0.0 ? sqrt(in_sq[b].x) / nrm : 0.0;
    double2* ts = tensors + bd.tensor_off[b];
    for (int i = 0; i < 2 * r1; ++i) ts[i] = cscale(f2d(rem[i]), f);
  }
}

// v_{c+1}[(x, p), r'] = sum_r v_c[x, r] A_c[r, p, r'], c = step + 1.
// Dynamic shared memory: A_c as float2, at most TT_MAXB x 2 x TT_MAXB.
__global__ void __launch_bounds__(BLOCK_THREADS) k_mps_contract(BatchDev bd, int step, const double2* tensors,
                                                                const int* bonds, int chi,
                                                                const float2* src, float2* dst_buf,
                                                                float2* target) {
  grid_wait();
  extern __shared__ float2 as[];
  for (int tile = blockIdx.x; tile < bd.ntiles; tile += gridDim.x) {
    const int b = bd.tile_state[tile];
    const int n = bd.n[b];
    const int c = step + 1;
    if (c > n - 1) continue;
    const int* bond = bonds + (int64_t)b * (bd.max_n + 1);
    const int rc = bond[c], rn = bond[c + 1];
    if (!bond_ok(rc, bd.tt_b) || !bond_ok(rn, bd.tt_b)) continue;
    if (rc > TT_MAXB || rn > TT_MAXB) continue;   // contracted by k_cgemm
    const int ce = chi_eff(chi, n);
    const double2* a = tensors + bd.tensor_off[b] + (int64_t)c * 2 * ce * ce;
    __syncthreads();
    for (int e = threadIdx.x; e < rc * 2 * rn; e += blockDim.x) as[e] = cf((float)a[e].x, (float)a[e].y);
    __syncthreads();
    const double2* t0 = tensors + bd.tensor_off[b];
    const float2* s = src + bd.vec_off[b];
    float2* o = (c == n - 1 ? target : dst_buf) + bd.vec_off[b];
    static_assert(TT_DOT_BOND * 2 * (TT_DOT_BOND + 1) <= TT_MAXB * 2 * TT_MAXB, "a site's entries and site 0");
    if (n <= TT_DOT_QUBITS && rc <= TT_DOT_BOND && rn <= TT_DOT_BOND) {   // one tile; bonds are the caller's
      const float2* x = s;
      if (step == 0) {   // site 0 (two rows), behind the site's entries
        x = as + rc * 2 * rn;
        __syncthreads();
        for (int e = threadIdx.x; e < 2 * rc; e += blockDim.x) as[rc * 2 * rn + e] = cf((float)t0[e].x, (float)t0[e].y);
        __syncthreads();
      }
      tt_small_product(x, rc, as, rc, (int)ipow2(c), 2 * rn, o);
      continue;
    }
    const int64_t total = ipow2(c + 1) * rn;
    int64_t lo, hi;
    tile_range(total, bd.tile_idx[tile], bd.state_ntiles[b], &lo, &hi);
    for (int64_t e = lo + threadIdx.x; e < hi; e += blockDim.x) {
      const int64_t x = e / (2 * rn);
      const int pr = (int)(e % (2 * rn));
      float2 acc = cf(0.f, 0.f);
      for (int rr = 0; rr < rc; ++rr) {
        float2 sv;
        if (step == 0) { const double2 d = t0[x * rc + rr]; sv = cf((float)d.x, (float)d.y); }
        else sv = s[x * rc + rr];
        acc = fmac(acc, sv, as[rr * 2 * rn + pr]);
      }
      o[e] = acc;
    }
  }
}

#define TT_EIG_SMEM ((size_t)3 * TT_EIG_SMEM_W * (TT_EIG_SMEM_W + TT_EIG_PAD) * sizeof(double2))   // G, V, scratch

static int grid_for(const BatchDev& bd) {
  int g = bd.ntiles;
  const int cap = 152 * 8;
  return g < cap ? g : cap;
}

void launch_tt_gram(const BatchDev& bd, int step, const float2* sv, const float2* src, const int* bonds,
                    const double2* sq, double2* partials, double2* gram, cudaStream_t s) {
  xc* part = reinterpret_cast<xc*>(partials);
  qm_note_launch();
  launch_after(k_tt_gram, grid_for(bd), BLOCK_THREADS, 0, s, bd, step, sv, src, bonds, sq, part);
  // the widest Gram a state can have at this step
  const int64_t wmax = step < 12 ? std::min<int64_t>(ipow2(step + 1), 2 * bd.tt_b) : 2 * bd.tt_b;
  const int64_t gx = std::min<int64_t>((wmax * wmax + BLOCK_THREADS / 8 - 1) / (BLOCK_THREADS / 8), 2048);
  qm_note_launch();
  launch_after(k_tt_gram_sum, dim3((unsigned)gx, (unsigned)std::min(bd.B, 65535)), BLOCK_THREADS, 0, s, bd, step,
               bonds, sq, part, gram);
}

void launch_tt_eig(const BatchDev& bd, int step, int* bonds, double2* gram, double2* vwork, int max_bond,
                   double cutoff, double2* vsel, double2* tensors, int chi, double2* scratch, double fine,
                   cudaStream_t s) {
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_tt_eig, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT_EIG_SMEM);
    attr = true;
  }
  qm_note_launch();
  launch_after(k_tt_eig, bd.B, TT_EIG_THREADS, TT_EIG_SMEM, s, bd, step, bonds, gram, vwork, max_bond, cutoff, vsel,
               tensors, chi, reinterpret_cast<float2*>(scratch), fine);
}

void launch_tt_project(const BatchDev& bd, int step, const float2* sv, const float2* src, float2* dst,
                       const int* bonds, const double2* vsel, cudaStream_t s) {
  const size_t smem = sizeof(float2) * (TT_MAXW * TT_MAXB + TT_CH * TT_MAXW);
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(k_tt_project, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    configured = true;
  }
  qm_note_launch();
  launch_after(k_tt_project, grid_for(bd), BLOCK_THREADS, smem, s, bd, step, sv, src, dst, bonds, vsel);
}

void launch_tt_site0(const BatchDev& bd, const float2* rem0, const float2* rem1, const int* bonds,
                     double2* tensors, int chi, const double2* in_sq, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_tt_site0, (bd.B + 127) / 128, 128, 0, s, bd, rem0, rem1, bonds, tensors, chi, in_sq);
}

void launch_mps_contract(const BatchDev& bd, int step, const double2* tensors, const int* bonds, int chi,
                         const float2* src, float2* dst_buf, float2* target, cudaStream_t s) {
  const size_t smem = sizeof(float2) * TT_MAXB * 2 * TT_MAXB;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(k_mps_contract, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    configured = true;
  }
  qm_note_launch();
  launch_after(k_mps_contract, grid_for(bd), BLOCK_THREADS, smem, s, bd, step, tensors, bonds, chi, src, dst_buf,
               target);
}
