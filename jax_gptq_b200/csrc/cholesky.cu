// Damping + lower Cholesky factor of the inverse Hessian
// (reference gptq.py:155-168 and :44-48).
//
// The reference forms H^-1 explicitly (potrf + potrs against I) and then
// factors it again.  Here the same L (lower, L L^T = H^-1) is obtained with one
// factorization and one triangular inverse: with J the index reversal and
// C = chol_lower(J H J), L = J C^-T J, i.e. L[i][j] = (C^-1)[K-1-j][K-1-i].
// Both C and X = C^-1 are produced in ONE blocked sweep over 64-wide panels:
//
//   step k:  (1) factor diagonal block, invert it            (1 CTA)
//            (2) panel below it  A[i,k] <- A[i,k] * inv_k^T   (row tiles)
//            (3) X[k, <k]  <- -inv_k * S[k, <k]               (column tiles)
//   trailing (4) A[i,j] -= A[i,k] A[j,k]^T                    (lower tiles)
//            (5) S[i>k, <=k] += A[i,k] X[k, <=k]
//
// (4) and (5) run once per outer block of four panels, with depth 256; inside an outer block
// (2) and (3) apply the block's earlier panels to their tiles themselves.  S lives in the
// not-yet-final part of X.  Everything is fp32; roots and quotients are rounded as IEEE's are.
#include "common.cuh"
#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace jgq {

constexpr int CB = 64;          // panel width
constexpr int COB = 4;          // panels per outer block (deferred updates of depth 256)

// ---- (0) diagonal statistics: dead features, damping increment ----------------
__global__ void __launch_bounds__(1024)
diag_stats_kernel(const float* __restrict__ H, int K, float damping,
                  uint8_t* __restrict__ dead, float* __restrict__ damp_add) {
  __shared__ double part[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < K; i += blockDim.x) {
    float d = H[(int64_t)i * K + i];
    const bool is_dead = (d == 0.f);
    dead[i] = is_dead ? 1 : 0;
    if (is_dead) d = 1.f;
    s += (double)d;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += part[w];
    const float mean = (float)(t / (double)K);
    *damp_add = __fmul_rn(mean, damping);
  }
}

// ---- (0b) A = J * (H with dead/damping fix-ups) * J ---------------------------
__global__ void build_reversed_kernel(const float* __restrict__ H, int K,
                                      const uint8_t* __restrict__ dead,
                                      const float* __restrict__ damp_add, float* __restrict__ A) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= K || j >= K) return;
  const int si = K - 1 - i, sj = K - 1 - j;
  float v = H[(int64_t)si * K + sj];
  if (i == j) {
    if (dead[si]) v = 1.f;
    v = __fadd_rn(v, *damp_add);
  }
  A[(int64_t)i * K + j] = v;
}

__global__ void zero_dead_rows_kernel(float* __restrict__ W, int K, int64_t N,
                                      const uint8_t* __restrict__ dead) {
  const int r = blockIdx.y;
  if (!dead[r]) return;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N;
       c += (int64_t)gridDim.x * blockDim.x)
    W[(int64_t)r * N + c] = 0.f;
}

// ---- one panel step: two launches, chained with programmatic stream serialization ----------------
// What bounds the sweep below K of a few thousand is the latency of this chain, K / 64 times in a row, so
// both kernels are built for it: one pass over the pivots of a diagonal block gives the factor and its inverse,
// and everything of the tile kernel that does not need the diagonal block - the updates with the outer
// block's earlier panels - runs beside the diagonal kernel.  Every element's products are summed in the same
// order as in a plain blocked sweep (increasing contraction index inside a panel, panel by panel), so that
// neither the tiling nor the fusion shows in the result.  Measured
// per panel at K = 768 (serialised): diagonal 38 -> 13.4 us, tiles 19.4 -> 16.5 us with the rank-64 updates in them,
// whose own launch (24 us) is gone; the whole stage 757 -> 315 us at K = 768, 3407 -> 1690 at 3072, 5190 -> 2917 at 4096.

constexpr int CS = CB + 4;      // row stride of the shared 64 x 64 tiles: 16-byte rows, eight rows on 32 banks

// d = sqrt(a) and y = 1 / d, both rounded to nearest, for a in [2^-96, 2^96]: Goldschmidt iterations on the
// hardware's reciprocal root with the residual corrections of Markstein (IBM J. R&D 34, 1990).  Equal to the IEEE
// operations for every mantissa and both exponent parities, d always, y but for d's largest mantissa, which leaf16 gives to
// the plain operations (compared through the factorization of diagonal matrices; the tests repeat every 32nd mantissa).  About 70 cycles for the
// pair; an IEEE root takes 55, and each division by it 50 more where divide_by takes 20.
__device__ __forceinline__ void root_and_reciprocal(float a, float& d, float& y) {
  float h, g, e;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
  g = a * y;
  h = 0.5f * y;
  e = fmaf(-h, g, 0.5f);
  g = fmaf(g, e, g);
  h = fmaf(h, e, h);
  e = fmaf(-g, g, a);
  d = fmaf(e, h, g);
  y = h + h;
  e = fmaf(-d, y, 1.f);
  y = fmaf(y, e, y);
  e = fmaf(-d, y, 1.f);
  y = fmaf(y, e, y);
}
// num / d rounded to nearest, given y = 1 / d rounded to nearest (Markstein's theorem: a quotient within one unit
// in the last place, corrected once more with the exact residual).  The residual must stay above the subnormals:
// `ok` is cleared unless |num| is zero or in [2^-90, 2^90].
__device__ __forceinline__ float divide_by(float num, float d, float y, bool& ok) {
  float q = num * y;
  float e = fmaf(-d, q, num);
  q = fmaf(e, y, q);
  e = fmaf(-d, q, num);
  q = fmaf(e, y, q);
  const float m = fabsf(num);
  ok &= (m >= 8.0779356694631609e-28f && m <= 1.2379400392853803e27f) || m == 0.f;
  return m == 0.f ? num : q;
}

// Cholesky factor of the 16 x 16 block at (c0, c0) of `a` (lower triangle significant) and its inverse, one
// warp, one pass.  Lane r < 16 holds row r of the block, lane 16 + c the running sums of column c of the
// forward substitution L X = I.  Pivot k: everybody divides its element k by the pivot's root (column k of L in
// the one half, row k of the inverse in the other), and the products with column k of L go to both the block and
// the sums.  The chain from pivot to pivot is root, quotient, one shuffle and one multiply-add: every lane follows
// the whole diagonal (dg), element k + 1 of column k comes by shuffle, the others (needed a pivot later) through
// shared memory; their products are put off until the next pivot's root is under way.  A warp is alone with this
// chain, so the loop has no branch that would keep its instructions from overlapping: kFast = false is the same
// elimination with the IEEE operations, for the blocks whose values leave the range of the fast ones (returns
// false then; `iv` is written only on success).
template <bool kFast>
__device__ __forceinline__ bool leaf16(const float (*a)[CS], float (*iv)[20], float* col, const int c0, bool& notpd) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, r = lane & 15;
  const bool upper = lane >= 16;                  // the half that builds the inverse
  float v[16], dg[16], l[16], tp = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    v[j] = (!upper && j <= r) ? a[c0 + r][c0 + j] : 0.f;
    dg[j] = a[c0 + j][c0 + j];
    l[j] = 0.f;
  }
  bool ok = true;
  notpd = false;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float akk = dg[k];
    float d, y = 0.f;
    if (kFast) {
      root_and_reciprocal(akk, d, y);
      ok &= akk >= 1.2621774483536189e-29f && akk <= 7.9228162514264338e28f &&
            (__float_as_uint(d) & 0x7fffffu) != 0x7fffffu;      // the one mantissa whose reciprocal the iteration misses
    } else {
      d = __fsqrt_rn(akk);
    }
    notpd |= !(akk > 0.f);
    // products with column k - 1, from row k + 1 on
    if (k > 0) {
#pragma unroll
      for (int j = k + 1; j < 16; ++j) {
        dg[j] = fmaf(l[j], -l[j], dg[j]);
        v[j] = fmaf(l[j], tp, v[j]);
      }
    }
    const float num = upper ? (r == k ? 1.f : -v[k]) : v[k];
    float q = kFast ? divide_by(num, d, y, ok) : __fdiv_rn(num, d);
    if (!upper && r == k) q = d;
    if (upper && r > k) q = 0.f;
    const float t = upper ? q : -q;
    v[k] = q;
    tp = t;
    if (k < 15) {
      const float lnext = __shfl_sync(full, q, k + 1);
      float* cb = col + 16 * (k & 1);
      if (!upper) cb[r] = q;
      dg[k + 1] = fmaf(lnext, -lnext, dg[k + 1]);
      v[k + 1] = fmaf(lnext, t, v[k + 1]);
      __syncwarp();
#pragma unroll
      for (int j4 = 0; j4 < 16; j4 += 4)
        if (j4 + 3 >= k + 2) {
          const float4 l4 = *reinterpret_cast<const float4*>(cb + j4);
          l[j4] = l4.x; l[j4 + 1] = l4.y; l[j4 + 2] = l4.z; l[j4 + 3] = l4.w;
        }
    }
  }
  if (kFast && !__all_sync(full, ok)) return false;
  if (upper) {
#pragma unroll
    for (int i = 0; i < 16; ++i) iv[i][r] = v[i];
  }
  return true;
}

// 64 x 64 tile at (row, col) of a K-stride matrix into registers: thread t holds four consecutive columns
// 4 (t % 16) of rows t / 16 + 16 q; zeros from row_lim / col_lim on.  `vec`: 16-byte loads are legal.
__device__ __forceinline__ void tile_fetch(float4 (&v)[4], const float* P, int K, int row, int col,
                                           int row_lim, int col_lim, bool vec) {
  const int t = threadIdx.x, j = col + 4 * (t & 15);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = row + (t >> 4) + 16 * q;
    const float* src = P + (int64_t)i * K + j;
    v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < row_lim) {
      if (vec && j + 3 < col_lim) v[q] = *reinterpret_cast<const float4*>(src);
      else {
        if (j < col_lim) v[q].x = src[0];
        if (j + 1 < col_lim) v[q].y = src[1];
        if (j + 2 < col_lim) v[q].z = src[2];
        if (j + 3 < col_lim) v[q].w = src[3];
      }
    }
  }
}
__device__ __forceinline__ void tile_put(float (*S)[CS], const float4 (&v)[4]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < 4; ++q) *reinterpret_cast<float4*>(&S[(t >> 4) + 16 * q][4 * (t & 15)]) = v[q];
}

// Inverse of the Cholesky factor of diagonal block kb, written to X; the factor itself is not needed again.
// Sixteen columns at a time: leaf16 inverts the pivot block (iv); the rows below become P = A iv^T and the
// pivot rows of the inverse X = -iv T, T being the sums P X of the earlier steps; then the rows below take
// A -= P P^T and T += P X.  R holds the right factors of both updates side by side (P^T, then the pivot rows
// of X), so that they are one loop.  Warp 0 brings the next pivot block up to date and goes on with it while
// the other warps finish the update.  (A is not __restrict__: the tile kernel in front may still be writing it when this
// one starts, which the read-only path that a const __restrict__ pointer allows does not permit.)
__global__ void __launch_bounds__(256)
chol_diag_kernel(const float* A, float* X, int K, int kb, int vec,
                 int32_t* __restrict__ status) {
  __shared__ __align__(16) float a[CB][CS];
  __shared__ __align__(16) float x[CB][CS];        // T
  __shared__ __align__(16) float R[16][2 * CB + 4];
  __shared__ __align__(16) float P[CB - 16][20];   // from row 16 on
  __shared__ __align__(16) float iv[16][20];
  __shared__ __align__(16) float col[32];
  const int r0 = kb * CB;
  const int nb = min(CB, K - r0);
  const int tid = threadIdx.x, warp = tid >> 5;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // The tile kernel of this step may be scheduled from here on: all it reads before its own wait was
  // complete when this wait returned.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  {
    float4 v[4];
    tile_fetch(v, A, K, r0, r0, K, K, vec != 0);
    tile_put(a, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    tile_put(x, v);
  }
  __syncthreads();
  if (nb < CB) {
    if (tid >= nb && tid < CB) a[tid][tid] = 1.f;   // identity padding of a partial last block
    __syncthreads();
  }

  // one item = 4 columns of one row of the update of step c0 / 16: rows / 4 items per row for A, (c0 + 16) / 4 for T
  auto update = [&](int c0, int i, int qd) {
    const int rows = CB - 16 - c0, b0 = c0 + 16;
    const bool ina = qd < rows / 4;
    const int cl = ina ? b0 + 4 * qd : 4 * (qd - rows / 4);
    const int rc = ina ? cl : CB + cl;
    float4* dst = reinterpret_cast<float4*>(ina ? &a[i][cl] : &x[i][cl]);
    const float4 old = *dst;
    float4 acc = ina ? make_float4(0.f, 0.f, 0.f, 0.f) : old;
#pragma unroll
    for (int m4 = 0; m4 < 16; m4 += 4) {
      const float4 pm = *reinterpret_cast<const float4*>(&P[i - 16][m4]);
      const float pj[4] = {pm.x, pm.y, pm.z, pm.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 w = *reinterpret_cast<const float4*>(&R[m4 + u][rc]);
        acc.x = fmaf(pj[u], w.x, acc.x); acc.y = fmaf(pj[u], w.y, acc.y);
        acc.z = fmaf(pj[u], w.z, acc.z); acc.w = fmaf(pj[u], w.w, acc.w);
      }
    }
    if (ina) acc = make_float4(old.x - acc.x, old.y - acc.y, old.z - acc.z, old.w - acc.w);
    *dst = acc;
  };

#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    const int c0 = 16 * s, rows = CB - 16 - c0, b0 = c0 + 16;
    if (warp == 0) {
      if (s > 0) {
        // the pivot block itself: its 16 columns are the first four items of a row
#pragma unroll
        for (int h = 0; h < 2; ++h) update(c0 - 16, c0 + ((tid + 32 * h) >> 2), tid & 3);
        __syncwarp();
      }
      bool bad;
      if (!leaf16<true>(a, iv, col, c0, bad)) leaf16<false>(a, iv, col, c0, bad);
      if (bad && tid == 0) atomicOr(status, JGQ_STATUS_NOT_PD);
    } else if (s > 0) {
      for (int item = tid - 32; item < (rows + 16) * 16; item += 224) {
        const int i = c0 + (item >> 4), qd = item & 15;
        if (i >= b0 || qd >= 4) update(c0 - 16, i, qd);
      }
    }
    __syncthreads();
    // 48 x 16 elements, three per thread: first the rows below (P), then the earlier columns of the pivot rows of X
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const int u = tid / 16 + 16 * t, c = tid % 16;       // u < rows: row b0 + u, column c of P
      float sum = 0.f;
      if (u < rows) {
        const int i = b0 + u;
#pragma unroll
        for (int m = 0; m < 16; m += 4) {
          const float4 p4 = *reinterpret_cast<const float4*>(&a[i][c0 + m]);
          const float4 w = *reinterpret_cast<const float4*>(&iv[c][m]);
          sum = fmaf(p4.x, w.x, sum); sum = fmaf(p4.y, w.y, sum); sum = fmaf(p4.z, w.z, sum); sum = fmaf(p4.w, w.w, sum);
        }
        P[i - 16][c] = sum;
        R[c][i] = sum;
      } else {
        const int cc = u - rows, rr = c;                    // element (rr, cc) of the pivot rows, cc < c0
#pragma unroll
        for (int m = 0; m < 16; ++m) sum = fmaf(iv[rr][m], x[c0 + m][cc], sum);
        R[rr][CB + cc] = -sum;
        if (c0 + rr < nb) X[(int64_t)(r0 + c0 + rr) * K + r0 + cc] = -sum;
      }
    }
    {
      const int rr = tid / 16, c = tid % 16;
      const float v = iv[rr][c];
      R[rr][CB + c0 + c] = v;
      if (c0 + rr < nb && c0 + c < nb) X[(int64_t)(r0 + c0 + rr) * K + r0 + c0 + c] = v;
    }
    __syncthreads();
  }
}

// acc[i][j] += sum_m U[ty + 16 i][m] V[tx + 16 j][m]
__device__ __forceinline__ void tile_mul_nt(float (&acc)[4][4], const float (*U)[CS], const float (*V)[CS]) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll 4
  for (int m = 0; m < CB; m += 4) {
    float4 u[4], w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      u[i] = *reinterpret_cast<const float4*>(&U[ty + 16 * i][m]);
      w[i] = *reinterpret_cast<const float4*>(&V[tx + 16 * i][m]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fmaf(u[i].x, w[j].x, acc[i][j]); acc[i][j] = fmaf(u[i].y, w[j].y, acc[i][j]);
        acc[i][j] = fmaf(u[i].z, w[j].z, acc[i][j]); acc[i][j] = fmaf(u[i].w, w[j].w, acc[i][j]);
      }
  }
}
// acc[i][j] += sum_m U[ty + 16 i][m] V[m][4 tx + j]
__device__ __forceinline__ void tile_mul_nn(float (&acc)[4][4], const float (*U)[CS], const float (*V)[CS]) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll 4
  for (int m = 0; m < CB; m += 4) {
    float4 u[4], w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      u[i] = *reinterpret_cast<const float4*>(&U[ty + 16 * i][m]);
      w[i] = *reinterpret_cast<const float4*>(&V[m + i][4 * tx]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float ui[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
#pragma unroll
      for (int m2 = 0; m2 < 4; ++m2) {
        acc[i][0] = fmaf(ui[m2], w[m2].x, acc[i][0]); acc[i][1] = fmaf(ui[m2], w[m2].y, acc[i][1]);
        acc[i][2] = fmaf(ui[m2], w[m2].z, acc[i][2]); acc[i][3] = fmaf(ui[m2], w[m2].w, acc[i][3]);
      }
    }
  }
}

// One 64 x 64 tile of panel step kb per CTA.  Blocks [ob, kb) are the earlier panels of the same outer block,
// whose updates have not been applied to this tile yet:
//   row block i > kb:     A[i, kb] <- (A[i, kb] - sum_p A[i, p] A[kb, p]^T) inv^T
//   column block c < kb:  X[kb, c] <- -inv (S[kb, c] + sum_p A[kb, p] X[p, c])
// The sums run before the wait for the diagonal kernel.  The CTA of a row block inside the outer block
// (i < obe) then brings its diagonal block up to date with the tile it holds, A[i, i] -= A[i, kb] A[i, kb]^T,
// so that the next diagonal kernel finds a finished block.  With `mirror` the panel tile is also written transposed above
// the diagonal (A[kb, i], which nothing else uses): the large trailing update reads it there.
__global__ void __launch_bounds__(256)
chol_tiles_kernel(float* A, float* X, int K, int kb, int ob, int obe, int tiles_below, int vec, int mirror) {
  __shared__ __align__(16) float U[CB][CS];
  __shared__ __align__(16) float V[CB][CS];
  const int r0 = kb * CB;
  const int nb = min(CB, K - r0);
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int bid = blockIdx.x;
  const bool below = bid < tiles_below;
  const int ib = kb + 1 + bid;                             // row block of a tile below
  const int i0 = ib * CB;
  const int c0 = (bid - tiles_below) * CB;                 // first column of a tile of the inverse
  float4 fu[4], fv[4];
  float own[4][4], acc[4][4];
  const int p_first = below ? ob : max(ob, bid - tiles_below);
  auto fetch_pair = [&](int p) {
    tile_fetch(fu, A, K, below ? i0 : r0, p * CB, K, K, vec);
    if (below) tile_fetch(fv, A, K, r0, p * CB, K, K, vec);
    else       tile_fetch(fv, X, K, p * CB, c0, K, K, vec);
  };
  // the tile itself is complete but for the outer block's earlier panels
  if (below) tile_fetch(fu, A, K, i0, r0, K, r0 + nb, vec);
  else       tile_fetch(fu, X, K, r0, c0, r0 + nb, K, vec);
  tile_put(U, fu);
  if (p_first < kb) fetch_pair(p_first);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) own[i][j] = below ? U[ty + 16 * i][tx + 16 * j] : U[ty + 16 * i][4 * tx + j];
  for (int p = p_first; p < kb; ++p) {
    __syncthreads();
    tile_put(U, fu);
    tile_put(V, fv);
    __syncthreads();
    if (p + 1 < kb) fetch_pair(p + 1);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    if (below) tile_mul_nt(acc, U, V);
    else       tile_mul_nn(acc, U, V);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) own[i][j] = below ? own[i][j] - acc[i][j] : own[i][j] + acc[i][j];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (below) U[ty + 16 * i][tx + 16 * j] = own[i][j];
      else       U[ty + 16 * i][4 * tx + j] = own[i][j];
      acc[i][j] = 0.f;
    }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tile_fetch(fv, X, K, r0, r0, r0 + nb, r0 + nb, vec);
  tile_put(V, fv);
  __syncthreads();
  if (!below) {
    tile_mul_nn(acc, V, U);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (ty + 16 * i < nb) {
        float* dst = X + (int64_t)(r0 + ty + 16 * i) * K + c0 + 4 * tx;
        if (vec) *reinterpret_cast<float4*>(dst) = make_float4(-acc[i][0], -acc[i][1], -acc[i][2], -acc[i][3]);
        else
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[j] = -acc[i][j];
      }
    return;
  }
  tile_mul_nt(acc, U, V);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + ty + 16 * i < K && tx + 16 * j < nb) A[(int64_t)(i0 + ty + 16 * i) * K + r0 + tx + 16 * j] = acc[i][j];
  const bool diag_next = ib < obe;
  if (!diag_next && !mirror) return;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { U[ty + 16 * i][tx + 16 * j] = acc[i][j]; acc[i][j] = 0.f; }
  __syncthreads();
  if (mirror && !diag_next) {
    // rows of the outer block's own panels are never read transposed
    const int r = tid & 63;
    for (int c = tid >> 6; c < nb; c += 4)
      if (i0 + r < K) A[(int64_t)(r0 + c) * K + i0 + r] = U[r][c];
    return;
  }
  tile_mul_nt(acc, U, U);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + ty + 16 * i < K && i0 + tx + 16 * j < K) A[(int64_t)(i0 + ty + 16 * i) * K + i0 + tx + 16 * j] -= acc[i][j];
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// ---- trailing updates of an outer block, both in one launch -------------------------------------------
//   problem 0:  A[r, c] -= sum_k P[r, k] P[c, k]     lower tiles         problem 1:  S[r, c] += sum_k P[r, k] X[k, c]
// with P the block's panel below it (depth 256).  Plain FP32 multiply-adds, one chain per element in increasing k, then
// one addition: what a tile computes does not depend on its size.  Bound by the FP32 pipe when there are tiles for all
// SMs (128 x 128, 8 x 8 per thread, packed pairs of multiply-adds), by a tile's own latency when there are not (64 x 64,
// 4 x 4).  Stages of 32 in two buffers, 16-byte asynchronous copies, nothing transposed on the way.  An update at K = 4096
// takes 84 us on average (128 x 128 x 8 tiles staged through registers: 104; this loop on k-contiguous rows: 134); the
// stage as a whole 315 -> 277 us at K = 768, 2917 -> 2518 at K = 4096.
struct UpdateParams {
  const float* P; const float* PT; const float* X; float* A; float* S;     // PT: P transposed, rows of stride K as well
  int K, depth, rows, cols0, cols1;      // rows of both; columns of problem 0 (= rows) and 1
  int tiles0, tn1, vec;
};

constexpr int UBK = 32, UKS = UBK + 4;   // stage depth, row stride of a k-contiguous tile

// tile (tm, tn) of the list: problem 0's lower tiles row by row, then problem 1's
__device__ __forceinline__ bool update_tile(const UpdateParams& p, int& tm, int& tn) {
  int t = blockIdx.x;
  if (t >= p.tiles0) {
    t -= p.tiles0;
    tm = t / p.tn1; tn = t % p.tn1;
    return true;
  }
  tm = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((tm + 1) * (tm + 2) / 2 <= t) ++tm;
  while (tm * (tm + 1) / 2 > t) --tm;
  tn = t - tm * (tm + 1) / 2;
  return false;
}

// Two multiply-adds, each rounded like fmaf.
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

// 128 x 128 tiles; both operands lie with their free index contiguous (the mirrored panel, X).  Needs p.vec and full stages.
constexpr int ULS = 128;
__global__ void __launch_bounds__(256, 2)
chol_update_large_kernel(const UpdateParams p) {
  extern __shared__ __align__(16) float usm[];                 // [2][A: UBK x 128, B: UBK x 128]
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  int tm, tn;
  const bool second = update_tile(p, tm, tn);
  const int m0 = tm * 128, n0 = tn * 128, K = p.K;
  const int ncol = second ? p.cols1 : p.cols0;
  const float* Bp = second ? p.X : p.PT;
  auto stage = [&](int kk, int buf) {
    float* As = usm + buf * 2 * UBK * ULS;
    float* Bs = As + UBK * ULS;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = (tid >> 5) + 8 * u, c = 4 * (tid & 31);
      if (m0 + c < p.rows) cp_async16(As + k * ULS + c, p.PT + (int64_t)(kk + k) * K + m0 + c);
      else *reinterpret_cast<float4*>(As + k * ULS + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (n0 + c < ncol) cp_async16(Bs + k * ULS + c, Bp + (int64_t)(kk + k) * K + n0 + c);
      else *reinterpret_cast<float4*>(Bs + k * ULS + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint64_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  stage(0, 0);
  for (int kk = 0, buf = 0; kk < p.depth; kk += UBK, buf ^= 1) {
    if (kk + UBK < p.depth) { stage(kk + UBK, buf ^ 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float* As = usm + buf * 2 * UBK * ULS + 4 * ty;
    const float* Bs = usm + buf * 2 * UBK * ULS + UBK * ULS + 4 * tx;
#pragma unroll 4
    for (int k = 0; k < UBK; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(As + k * ULS), a1 = *reinterpret_cast<const float4*>(As + k * ULS + 64);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(Bs + k * ULS), b1 = *reinterpret_cast<const ulonglong2*>(Bs + k * ULS + 64);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t aa = twice(a[i]);
        fma2(acc[i][0], aa, b0.x); fma2(acc[i][1], aa, b0.y);
        fma2(acc[i][2], aa, b1.x); fma2(acc[i][3], aa, b1.y);
      }
    }
    __syncthreads();
  }
  float* C = second ? p.S : p.A;
  const float sign = second ? 1.f : -1.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = m0 + (i < 4 ? 4 * ty + i : 64 + 4 * ty + i - 4);
    if (r >= p.rows) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = n0 + 64 * h + 4 * tx;
      if (c < ncol) {                                       // ncol % 4 == 0
        float4* dst = reinterpret_cast<float4*>(C + (int64_t)r * K + c);
        const float2 v0 = *reinterpret_cast<const float2*>(&acc[i][2 * h]), v1 = *reinterpret_cast<const float2*>(&acc[i][2 * h + 1]);
        float4 o = *dst;
        o.x = fmaf(sign, v0.x, o.x); o.y = fmaf(sign, v0.y, o.y);
        o.z = fmaf(sign, v1.x, o.z); o.w = fmaf(sign, v1.y, o.w);
        *dst = o;
      }
    }
  }
}

// 64 x 64 tiles for any K.
__global__ void __launch_bounds__(256, 2)
chol_update_kernel(const UpdateParams p) {
  constexpr int B = 64, T = B / 16;                           // elements per thread and direction
  constexpr int NS = B + 4;                                   // row stride of a tile with n contiguous
  constexpr int STAGE = 2 * B * UKS;
  static_assert(B * UKS >= UBK * NS, "either operand layout fits its half of a stage");
  extern __shared__ __align__(16) float usm[];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  int tm, tn;
  const bool second = update_tile(p, tm, tn);
  const int m0 = tm * B, n0 = tn * B, K = p.K;
  const int ncol = second ? p.cols1 : p.cols0;

  auto stage = [&](int kk, int buf) {
    float* As = usm + buf * STAGE;
    float* Bs = As + B * UKS;
    const int kn = min(UBK, p.depth - kk);
    auto rows_kc = [&](float* dst, int r0, int rlim) {        // B rows of P, 32 k each
      if (p.vec && kn == UBK) {
#pragma unroll
        for (int u = 0; u < B / 32; ++u) {
          const int r = (tid >> 3) + 32 * u, c = 4 * (tid & 7);
          if (r0 + r < rlim) cp_async16(dst + r * UKS + c, p.P + (int64_t)(r0 + r) * K + kk + c);
          else *reinterpret_cast<float4*>(dst + r * UKS + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      } else {
        for (int i = tid; i < B * UBK; i += 256) {
          const int r = i / UBK, c = i % UBK;
          dst[r * UKS + c] = (r0 + r < rlim && c < kn) ? p.P[(int64_t)(r0 + r) * K + kk + c] : 0.f;
        }
      }
    };
    rows_kc(As, m0, p.rows);
    if (!second) {
      rows_kc(Bs, n0, p.rows);
    } else if (p.vec && kn == UBK) {
#pragma unroll
      for (int u = 0; u < B / 32; ++u) {
        const int i = tid + 256 * u, r = i / (B / 4), c = 4 * (i % (B / 4));
        if (n0 + c < ncol) cp_async16(Bs + r * NS + c, p.X + (int64_t)(kk + r) * K + n0 + c);
        else *reinterpret_cast<float4*>(Bs + r * NS + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int i = tid; i < UBK * B; i += 256) {
        const int r = i / B, c = i % B;
        Bs[r * NS + c] = (r < kn && n0 + c < ncol) ? p.X[(int64_t)(kk + r) * K + n0 + c] : 0.f;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[T][T];
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) acc[i][j] = 0.f;
  stage(0, 0);
  for (int kk = 0, buf = 0; kk < p.depth; kk += UBK, buf ^= 1) {
    if (kk + UBK < p.depth) { stage(kk + UBK, buf ^ 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float* As = usm + buf * STAGE + ty * UKS;
    const float* Bs = usm + buf * STAGE + B * UKS;
    if (!second) {
#pragma unroll 2
      for (int k = 0; k < UBK; k += 4) {
        float4 u[T];
#pragma unroll
        for (int i = 0; i < T; ++i) u[i] = *reinterpret_cast<const float4*>(As + 16 * i * UKS + k);
#pragma unroll
        for (int j = 0; j < T; ++j) {
          const float4 w = *reinterpret_cast<const float4*>(Bs + (tx + 16 * j) * UKS + k);
#pragma unroll
          for (int i = 0; i < T; ++i) {
            acc[i][j] = fmaf(u[i].x, w.x, acc[i][j]); acc[i][j] = fmaf(u[i].y, w.y, acc[i][j]);
            acc[i][j] = fmaf(u[i].z, w.z, acc[i][j]); acc[i][j] = fmaf(u[i].w, w.w, acc[i][j]);
          }
        }
      }
    } else {
#pragma unroll 2
      for (int k = 0; k < UBK; k += 4) {
        float4 u[T];
#pragma unroll
        for (int i = 0; i < T; ++i) u[i] = *reinterpret_cast<const float4*>(As + 16 * i * UKS + k);
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
          for (int j4 = 0; j4 < T / 4; ++j4) {
            const float4 w = *reinterpret_cast<const float4*>(Bs + (k + k1) * NS + 64 * j4 + 4 * tx);
#pragma unroll
            for (int i = 0; i < T; ++i) {
              const float a = k1 == 0 ? u[i].x : k1 == 1 ? u[i].y : k1 == 2 ? u[i].z : u[i].w;
              acc[i][4 * j4] = fmaf(a, w.x, acc[i][4 * j4]); acc[i][4 * j4 + 1] = fmaf(a, w.y, acc[i][4 * j4 + 1]);
              acc[i][4 * j4 + 2] = fmaf(a, w.z, acc[i][4 * j4 + 2]); acc[i][4 * j4 + 3] = fmaf(a, w.w, acc[i][4 * j4 + 3]);
            }
          }
      }
    }
    __syncthreads();
  }

  float* C = second ? p.S : p.A;
#pragma unroll
  for (int i = 0; i < T; ++i) {
    const int r = m0 + ty + 16 * i;
    if (r >= p.rows) continue;
    float* row = C + (int64_t)r * K;
    if (!second) {
#pragma unroll
      for (int j = 0; j < T; ++j) {
        const int c = n0 + tx + 16 * j;
        if (c < ncol) row[c] -= acc[i][j];
      }
    } else {
#pragma unroll
      for (int j4 = 0; j4 < T / 4; ++j4) {
        const int c = n0 + 64 * j4 + 4 * tx;
        if (p.vec && c + 3 < ncol) {
          float4 o = *reinterpret_cast<const float4*>(row + c);
          o.x += acc[i][4 * j4]; o.y += acc[i][4 * j4 + 1]; o.z += acc[i][4 * j4 + 2]; o.w += acc[i][4 * j4 + 3];
          *reinterpret_cast<float4*>(row + c) = o;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c + j < ncol) row[c + j] += acc[i][4 * j4 + j];
        }
      }
    }
  }
}

template <auto Kern>
static int launch_update_tiles(UpdateParams p, int B, int smem, cudaStream_t s) {
  prefer_shared_carveout<Kern>();
  struct AttrTag {};
  once_per_device<AttrTag>([&]() { return (int)cudaFuncSetAttribute(reinterpret_cast<const void*>(Kern), cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  const int tr = (int)cdiv(p.rows, B);
  p.tiles0 = tr * (tr + 1) / 2;
  p.tn1 = (int)cdiv(p.cols1, B);
  Kern<<<(unsigned)(p.tiles0 + tr * p.tn1), 256, smem, s>>>(p);
  return check_launch("chol_update");
}

// Large tiles from one per SM on (they compute twice as much per byte from shared memory); fewer leave SMs idle
// while the small ones do not.
static bool large_update(int K, int c_end, int depth, int vec) {
  const int64_t tr = cdiv(K - c_end, 128);
  return vec && depth % UBK == 0 && tr * (tr + 1) / 2 + tr * cdiv(c_end, 128) >= (int64_t)sm_count();
}

// ---- final: L[i][j] = X[K-1-j][K-1-i] (i >= j), 0 above the diagonal -----------
__global__ void reverse_transpose_kernel(const float* __restrict__ X, float* __restrict__ L, int K,
                                         int32_t* __restrict__ status) {
  __shared__ float t[32][33];
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
  // load: t[jj][ii] = X[K-1-(j0+jj)][K-1-(i0+ii)], ii fastest
  for (int jj = threadIdx.y; jj < 32; jj += blockDim.y) {
    const int ii = threadIdx.x;
    const int i = i0 + ii, j = j0 + jj;
    float v = 0.f;
    if (i < K && j < K && i >= j) v = X[(int64_t)(K - 1 - j) * K + (K - 1 - i)];
    t[jj][ii] = v;
  }
  __syncthreads();
  bool bad = false;
  for (int ii = threadIdx.y; ii < 32; ii += blockDim.y) {
    const int jj = threadIdx.x;
    const int i = i0 + ii, j = j0 + jj;
    if (i < K && j < K) {
      const float v = t[jj][ii];
      bad |= isnan(v);
      L[(int64_t)i * K + j] = v;
    }
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x == 0)) atomicOr(status, JGQ_STATUS_NAN);
}

}  // namespace jgq

using namespace jgq;

extern "C" size_t jgq_damp_invert_workspace_bytes(int64_t K) {
  if (K <= 0) return 0;
  return align_up((size_t)K * (size_t)K * sizeof(float), 256) + align_up((size_t)K, 256) + 256;
}

extern "C" int jgq_damp_invert(float* W, int64_t N, float* H, int64_t K, float damping, float* L,
                               void* ws, size_t ws_bytes, int32_t* dev_status, void* stream) {
  JGQ_REQUIRE(K > 0 && N >= 0, JGQ_ERR_ARG, "damp_invert: bad shape K=%lld N=%lld", (long long)K, (long long)N);
  JGQ_REQUIRE(K <= 46340, JGQ_ERR_LIMIT, "damp_invert: K=%lld exceeds 46340", (long long)K);
  JGQ_REQUIRE(H && L && ws && dev_status && (W || N == 0), JGQ_ERR_ARG, "damp_invert: null pointer");
  JGQ_REQUIRE(ws_bytes >= jgq_damp_invert_workspace_bytes(K), JGQ_ERR_WORKSPACE,
              "damp_invert: workspace %zu < %zu bytes", ws_bytes, jgq_damp_invert_workspace_bytes(K));
  JGQ_REQUIRE(aligned(ws, 256), JGQ_ERR_ALIGN, "damp_invert: workspace must be 256-byte aligned");
  // A few launches per 64-wide panel whose arguments depend on these values alone: replayed as a graph when they recur
  struct { int tag; float damping; int64_t K, N; const void *W, *H, *L, *ws, *status; } key;
  memset(&key, 0, sizeof(key));
  key.tag = 1; key.damping = damping; key.K = K; key.N = N; key.W = W; key.H = H; key.L = L; key.ws = ws; key.status = dev_status;
  return run_replayed(key, (cudaStream_t)stream, [&](cudaStream_t s) -> int {
  const int Ki = (int)K;
  float* A = (float*)ws;
  uint8_t* dead = (uint8_t*)ws + align_up((size_t)K * K * sizeof(float), 256);
  float* damp_add = (float*)(dead + align_up((size_t)K, 256));
  float* X = H;   // H's storage is reused for the triangular inverse once A is built

  prefer_shared_carveout<diag_stats_kernel>();
  prefer_shared_carveout<build_reversed_kernel>();
  prefer_shared_carveout<zero_dead_rows_kernel>();
  prefer_shared_carveout<chol_diag_kernel>();
  prefer_shared_carveout<chol_tiles_kernel>();
  prefer_shared_carveout<reverse_transpose_kernel>();
  diag_stats_kernel<<<1, 1024, 0, s>>>(H, Ki, damping, dead, damp_add);
  JGQ_LAUNCHED();
  {
    dim3 blk(32, 8), grd((unsigned)cdiv(K, 32), (unsigned)cdiv(K, 8));
    build_reversed_kernel<<<grd, blk, 0, s>>>(H, Ki, dead, damp_add, A);
    JGQ_LAUNCHED();
  }
  if (N > 0) {
    dim3 grd((unsigned)std::min<int64_t>(cdiv(N, 256), 64), (unsigned)K);
    zero_dead_rows_kernel<<<grd, 256, 0, s>>>(W, Ki, N, dead);
    JGQ_LAUNCHED();
  }
  if (cudaMemsetAsync(X, 0, (size_t)K * K * sizeof(float), s) != cudaSuccess)
    return fail(JGQ_ERR_CUDA, "damp_invert: memset failed");

  // Two-level blocking: inside an outer block of COB panels the tile kernel applies the block's earlier
  // panels itself; everything beyond the block gets one update of depth 64 * COB when the block is
  // finished, which is where nearly all the arithmetic is.
  const int vec = (Ki % 4 == 0) && aligned(A, 16) && aligned(X, 16);
  const int nblk = (int)cdiv(K, CB);
  for (int ob = 0; ob < nblk; ob += COB) {
    const int c_begin = ob * CB;                                   // first column of the outer block
    const int c_end = std::min(Ki, (ob + COB) * CB);               // one past its last column
    const bool large = c_end < Ki && large_update(Ki, c_end, c_end - c_begin, vec);
    for (int kb = ob; kb < std::min(nblk, ob + COB); ++kb) {
      const int r1 = std::min(Ki, (kb + 1) * CB);      // first row below the diagonal block
      const int below = Ki - r1;
      const int tiles_below = below > 0 ? (int)cdiv(below, CB) : 0;
      // both launches of a step may be placed while their predecessor is finishing; they wait inside
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(1);
      cfg.blockDim = dim3(256);
      cfg.stream = s;
      cfg.attrs = attr;
      cfg.numAttrs = kb > 0 ? 1 : 0;       // the first one follows a memset, which signals nothing early
      cudaError_t e = cudaLaunchKernelEx(&cfg, chol_diag_kernel, (const float*)A, X, Ki, kb, vec, dev_status);
      note_launches(1);
      if (e == cudaSuccess && tiles_below + kb > 0) {
        cfg.gridDim = dim3((unsigned)(tiles_below + kb));
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, chol_tiles_kernel, A, X, Ki, kb, ob, std::min(nblk, ob + COB), tiles_below, vec, large ? 1 : 0);
        note_launches(1);
      }
      if (e != cudaSuccess) { cudaGetLastError(); return fail(JGQ_ERR_CUDA, "damp_invert: %s", cudaGetErrorString(e)); }
    }
    if (c_end < Ki) {
      // the block's whole panel Pb = A[c_end:, c_begin:c_end] at once:
      // A[c_end:, c_end:] -= Pb Pb^T (lower tiles)   and   S[c_end:, :c_end] += Pb X[c_begin:c_end, :c_end]
      const int below = Ki - c_end, depth = c_end - c_begin;
      UpdateParams up;
      memset(&up, 0, sizeof(up));
      up.P = A + (int64_t)c_end * K + c_begin;
      up.X = X + (int64_t)c_begin * K;
      up.A = A + (int64_t)c_end * K + c_end;
      up.S = X + (int64_t)c_end * K;
      up.K = Ki; up.depth = depth; up.rows = below; up.cols0 = below; up.cols1 = c_end; up.vec = vec;
      up.PT = A + (int64_t)c_begin * K + c_end;
      const int rc = large ? launch_update_tiles<chol_update_large_kernel>(up, 128, 4 * UBK * ULS * (int)sizeof(float), s)
                           : launch_update_tiles<chol_update_kernel>(up, 64, 4 * 64 * UKS * (int)sizeof(float), s);
      if (rc) return rc;
    }
  }
  {
    dim3 blk(32, 8), grd((unsigned)cdiv(K, 32), (unsigned)cdiv(K, 32));
    reverse_transpose_kernel<<<grd, blk, 0, s>>>(X, L, Ki, dev_status);
  }
  return check_launch("damp_invert");
  });
}
