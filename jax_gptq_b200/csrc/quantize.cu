// Blocked column-quantize + error propagation (reference gptq.py:120-153, 199-208).
//
// One launch per block of `bs` input rows.  Output channels (columns of the K x N matrix) never interact: a CTA
// owns 32 of them, one per lane, for the whole block.  What bounds the loop is the chain of K dependent
// quantize steps, so everything else is kept off that chain:
//   * warp 0 walks the rows 16 at a time (a sub-block, in registers) and hands its errors on four at a time; the
//     other warps apply them at once to the next 16 rows, and in between the previous sub-block's errors to the
//     later rows, and write its results;
//   * the two divisions of a step are multiplications with reciprocals kept for the whole block, corrected to the
//     IEEE quotient (divide_exact);
//   * the lazy-batch update  W[end:, :] -= L[end:, start:end] @ errors  never stands between two blocks.  For the next
//     block's rows the helpers sum it up sub-block by sub-block, beside the chain, and leave it in the workspace: the next
//     launch subtracts it when it loads its rows.  The rows behind that are updated by further CTAs of the next
//     launch.  The errors stay in the rows of W they came from.
// For every element the updates are applied one source row at a time in increasing row order with a separately
// rounded multiply and subtract, which is exactly the sequence of roundings the reference's unrolled loop performs,
// so a block is bit-identical to the fp32 oracle given the same inputs.  The lazy-batch update is three TF32
// products per term on the tensor cores (mma.sync, increasing contraction index).
// Measured per 128-row block: alone (N = 32) 84 -> 26 us; with its share of the update, K = N = 4096, 46 + 77 -> 64 us.
// The loop's code is kept short on purpose (groups of four steps, rolled loops): with the steps of a sub-block unrolled,
// three of ten issue slots of the kernel went to instruction fetches and a block took 33 us.
#include "common.cuh"
#include "sgemm.cuh"
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace jgq {

constexpr int SUB = 16;               // rows per sub-block
constexpr int QCH = 32;               // channels per CTA
constexpr int QHELP = 8;               // helper warps beside the chain's: one per row pair of a sub-block
constexpr int QWARPS = 1 + QHELP;
constexpr int QTHREADS = 32 * QWARPS;
constexpr int QES = QCH + 8;          // row stride of the errors: the fragment loads (4 rows x 8 channels) hit 32 banks

// The diagonal block of L: rows in groups of 16; a group keeps the 16 g columns in front of its diagonal
// sub-block (+ 4 of padding), and that sub-block is kept by columns
__host__ __device__ constexpr int ltri_stride(int g) { return SUB * g + 4; }
__host__ __device__ constexpr int ltri_base(int g) { return SUB * SUB * (g * (g - 1) / 2) + 4 * SUB * g; }
constexpr int QL_FLOATS = ltri_base(8);                                  // bs = 128
constexpr int QSMEM_FLOATS = QL_FLOATS + 128 * SUB + 128 * QCH + 2 * SUB * QES + 2 * SUB * QCH + 2 * 128;
constexpr int QSMEM_BYTES = QSMEM_FLOATS * (int)sizeof(float);           // 65 KB: two CTAs per SM, or one beside a Hessian CTA

// tiles of the update behind the block: 128 rows x 64 channels, eight warps of 32 x 32
constexpr int TBM = 128, TBN = 64, TBK = 32, TTHREADS = 256, TSTAGES = 2;
constexpr int TAS = TBK + 4, TBS = TBN + 8;            // row strides: fragment loads hit 32 banks
constexpr int TSTAGE_FLOATS = TBM * TAS + TBK * TBS;
static_assert(TSTAGES * TSTAGE_FLOATS <= QSMEM_FLOATS, "tail tiles use the same shared memory");

// JGQ_TAIL_GEMM=ffma keeps the lazy-batch tail update on the FFMA body, in launches of its own (for comparisons).
static int tail_on_tensor_cores() {
  static const int v = []() { const char* e = getenv("JGQ_TAIL_GEMM"); return (e && !strcmp(e, "ffma")) ? 0 : 1; }();
  return v;
}

// a / b rounded to nearest, given y = 1 / b rounded to nearest: a quotient within a unit in the last place,
// corrected twice with the exact residual (Markstein, IBM J. R&D 34, 1990).  For operands and quotients whose residuals
// stay normal; the callers check that.  About 20 cycles of latency, __fdiv_rn about 50.
__device__ __forceinline__ float divide_exact(float a, float b, float y) {
  float q = __fmul_rn(a, y);
  float e = fmaf(-b, q, a);
  q = fmaf(e, y, q);
  e = fmaf(-b, q, a);
  return fmaf(e, y, q);
}

// Products with near-fp32 accuracy on the tensor cores: every operand is split as x = hi + lo with hi = tf32(x), lo =
// tf32(x - hi), and accumulated as lo*hi + hi*lo + hi*hi.  The split keeps 22 of the 24 significand bits, so it is for
// updates that tolerate 2^-21 relative error per product (the lazy-batch update), not for the Cholesky sweep.
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  const float r = x - __uint_as_float(hi);
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(r));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// split_tf32 in integer arithmetic (the conversion unit is a quarter as wide): rounding half away from zero is an
// addition to the magnitude's bits.  For finite values.
__device__ __forceinline__ void split_tf32_alu(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  lo = (__float_as_uint(__fsub_rn(x, __uint_as_float(hi))) + 0x1000u) & 0xffffe000u;
}

struct QuantParams {
  float* W; const float* L; const float* scale; const float* zero;
  void* Q; uint8_t* codes;
  int K; int64_t N; int start, bs; float maxq;
  int apply_prev;               // 1: the previous block's lazy-batch update is part of this launch
  int nch;                      // CTAs that own channels; the rest are tiles of the update behind this block
  int vec;                      // 16-byte copies of rows of L and W are legal
  float* P;                     // [bs][N]: the lazy-batch update of the next launch's rows
  int make_next;                // 1: write P for the next block
  int rest, tail_tn;            // rows behind this block, channel tiles
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// W[m0 .. + 127 behind the block, n0 .. + 63] -= L[rows, previous block] @ errors of the previous block, three TF32
// products per term.  A rank-128 update is bound by its traffic (96 KB of operands and 64 KB of W read and written per
// tile): two 32-deep stages in flight, two CTAs per SM.  Without any arithmetic the tiles of a K = N = 4096 loop take 0.96 of
// 1.6 ms; the rest is the operands' split and the products' latency, hence one split per operand ahead of three runs of
// eight independent products (the whole loop 2.18 -> 2.05 ms against split and products term by term).
__device__ __forceinline__ void tail_tile(const QuantParams& p, float* smem, int tile) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int m0 = (tile / p.tail_tn) * TBM, n0 = (tile % p.tail_tn) * TBN;
  const int K = p.K, bs = p.bs, prev = p.start - bs, row0 = p.start + bs + m0;
  const int64_t N = p.N;
  const int mrows = min(TBM, p.rest - m0), ncols = (int)((N - n0 < TBN) ? N - n0 : TBN);
  const int wm = (warp & 3) * 32, wn = (warp >> 2) * 32;
  auto stage = [&](int kk, int buf) {
    float* As = smem + buf * TSTAGE_FLOATS;
    float* Bs = As + TBM * TAS;
    const float* A = p.L + (int64_t)row0 * K + prev + kk;
    const float* B = p.W + (int64_t)(prev + kk) * N + n0;
    const int kn = min(TBK, bs - kk);
    if (p.vec && kn == TBK) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = (tid >> 3) + 32 * u, c = 4 * (tid & 7);
        if (r < mrows) cp_async16((uint32_t)__cvta_generic_to_shared(As + r * TAS + c), A + (int64_t)r * K + c);
        else *reinterpret_cast<float4*>(As + r * TAS + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int i = tid; i < TBM * TBK; i += TTHREADS) {
        const int r = i / TBK, c = i % TBK;
        As[r * TAS + c] = (r < mrows && c < kn) ? A[(int64_t)r * K + c] : 0.f;
      }
    }
    if (p.vec && kn == TBK) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = (tid >> 4) + 16 * u, c = 4 * (tid & 15);
        if (c < ncols) cp_async16((uint32_t)__cvta_generic_to_shared(Bs + r * TBS + c), B + (int64_t)r * N + c);
        else *reinterpret_cast<float4*>(Bs + r * TBS + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int i = tid; i < TBK * TBN; i += TTHREADS) {
        const int r = i / TBN, c = i % TBN;
        Bs[r * TBS + c] = (r < kn && c < ncols) ? B[(int64_t)r * N + c] : 0.f;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  stage(0, 0);
  for (int kk = 0, buf = 0; kk < bs; kk += TBK, buf ^= 1) {
    if (kk + TBK < bs) { stage(kk + TBK, buf ^ 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("bar.sync 6, 256;" ::: "memory");
    const float* As = smem + buf * TSTAGE_FLOATS + wm * TAS;
    const float* Bs = smem + buf * TSTAGE_FLOATS + TBM * TAS + wn;
#pragma unroll 2
    for (int k8 = 0; k8 < TBK && kk + k8 < bs; k8 += 8) {
      uint32_t ah[2][4], al[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float* ap = As + (16 * i + g) * TAS + k8 + q;
        split_tf32_alu(ap[0], ah[i][0], al[i][0]);
        split_tf32_alu(ap[8 * TAS], ah[i][1], al[i][1]);
        split_tf32_alu(ap[4], ah[i][2], al[i][2]);
        split_tf32_alu(ap[8 * TAS + 4], ah[i][3], al[i][3]);
      }
      uint32_t bh[4][2], bl[4][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float* bp = Bs + (k8 + q) * TBS + 8 * j + g;
        split_tf32_alu(bp[0], bh[j][0], bl[j][0]);
        split_tf32_alu(bp[4 * TBS], bh[j][1], bl[j][1]);
      }
      // eight independent accumulators between two products of one
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_tf32(acc[i][j], al[i], bh[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_tf32(acc[i][j], ah[i], bl[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_tf32(acc[i][j], ah[i], bh[j]);
    }
    asm volatile("bar.sync 6, 256;" ::: "memory");
  }
  const bool pairs = (N % 2 == 0) && ((reinterpret_cast<uintptr_t>(p.W) & 7) == 0);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = wm + 16 * i + g + 8 * h;
      if (r >= mrows) continue;
      float* C = p.W + (int64_t)(row0 + r) * N + n0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = wn + 8 * j + 2 * q;
        if (pairs && c + 1 < ncols) {
          float2 o = *reinterpret_cast<const float2*>(C + c);
          o.x -= acc[i][j][2 * h]; o.y -= acc[i][j][2 * h + 1];
          *reinterpret_cast<float2*>(C + c) = o;
        } else {
          if (c < ncols) C[c] -= acc[i][j][2 * h];
          if (c + 1 < ncols) C[c + 1] -= acc[i][j][2 * h + 1];
        }
      }
    }
}

template <typename QT>
__global__ void __launch_bounds__(QTHREADS, 2)
gptq_block_kernel(const QuantParams p) {
  extern __shared__ __align__(16) float smem[];
  if ((int)blockIdx.x >= p.nch) {
    if (threadIdx.x >= TTHREADS) return;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tail_tile(p, smem, (int)blockIdx.x - p.nch);
    return;
  }
  float* Ld = smem;                         // the part of the diagonal block below its diagonal sub-blocks
  float* Lt = Ld + QL_FLOATS;               // [bs][SUB] its diagonal sub-blocks, by columns
  float* Wb = Lt + 128 * SUB;               // [bs][QCH] the block's weights
  float* Eb = Wb + 128 * QCH;               // [2][SUB][QES] errors of the current and the previous sub-block
  float* Cb = Eb + 2 * SUB * QES;           // [2][SUB][QCH] their codes
  float2* Dy = reinterpret_cast<float2*>(Cb + 2 * SUB * QCH);      // diagonal of L and its reciprocals

  // Warp 0 of the numbering used below is the hardware's warp 1: nine warps put three on the first scheduler and two on
  // each of the others, and the chain should share its scheduler with as few as possible.
  const int hw_warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = hw_warp < 2 ? hw_warp ^ 1 : hw_warp;
  const int bs = p.bs, start = p.start, K = p.K;
  const int64_t N = p.N;
  const int64_t ch0 = (int64_t)blockIdx.x * QCH, col = ch0 + lane;
  const bool live = col < N;
  const bool whole = ch0 + QCH <= N;        // all 32 channels exist
  const int nsub = (bs + SUB - 1) / SUB;

  // ---- L does not depend on the previous launch: fetch it while that one finishes ----
  for (int r = warp; r < bs; r += QWARPS) {
    const int g = r / SUB, w = SUB * g;
    float* dst = Ld + ltri_base(g) + (r % SUB) * ltri_stride(g);
    const float* src = p.L + (int64_t)(start + r) * K + start;
    if (p.vec) {
      if (4 * lane < w) cp_async16((uint32_t)__cvta_generic_to_shared(dst + 4 * lane), src + 4 * lane);
    } else {
      for (int c = lane; c < w; c += 32) dst[c] = src[c];
    }
  }
  for (int s = 0; s < nsub && threadIdx.x < SUB * SUB; ++s) {      // Lt[16 s + i][ii] = L[16 s + ii][16 s + i]
    const int ii = threadIdx.x / SUB, i = threadIdx.x % SUB, r = SUB * s + ii, c = SUB * s + i;
    Lt[c * SUB + ii] = (r < bs && c < bs) ? p.L[(int64_t)(start + r) * K + start + c] : 0.f;
  }
  if (threadIdx.x < 128) {
    const int r = threadIdx.x;
    const float d = r < bs ? p.L[(int64_t)(start + r) * K + start + r] : 1.f;
    Dy[r] = make_float2(d, __fdiv_rn(1.f, d));
  }
  const float sc = live ? p.scale[col] : 1.f;
  const float zr = live ? p.zero[col] : 0.f;
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- this CTA's columns of W, less the previous block's lazy-batch update ----
  {
    const float* Wsrc = p.W + (int64_t)start * N + ch0;
    const float* Psrc = p.P + ch0;
    if (p.vec && whole) {
      const int c4 = 4 * (threadIdx.x & 7), rt = threadIdx.x >> 3;      // 36 rows at a time
      float4 u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = rt + (QTHREADS / 8) * k;
        if (r < bs) {
          cp_async16((uint32_t)__cvta_generic_to_shared(Wb + r * QCH + c4), Wsrc + (int64_t)r * N + c4);
          if (p.apply_prev) u[k] = *reinterpret_cast<const float4*>(Psrc + (int64_t)r * N + c4);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      if (p.apply_prev) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = rt + (QTHREADS / 8) * k;
          if (r < bs) {
            float4* wp = reinterpret_cast<float4*>(Wb + r * QCH + c4);
            float4 w = *wp;
            w.x -= u[k].x; w.y -= u[k].y; w.z -= u[k].z; w.w -= u[k].w;
            *wp = w;
          }
        }
      }
    } else {
      for (int r = warp; r < bs; r += QWARPS) {
        float w = live ? Wsrc[(int64_t)r * N + lane] : 0.f;
        if (live && p.apply_prev) w -= Psrc[(int64_t)r * N + lane];
        Wb[r * QCH + lane] = w;
      }
    }
  }
  // Quotients whose reciprocal form is exact: scale, pivots and zero in the ranges below (checked once, for the whole
  // CTA), and per step |w| <= 2^60 and |w - q| zero or >= 2^-90.  A sub-block that leaves them is finished with
  // plain divisions.
  bool in_range = sc >= 8.6736173798840355e-19f && sc <= 1.152921504606847e18f && fabsf(zr) <= 1048576.f;     // 2^-60 .. 2^60, 2^20
  if (threadIdx.x < 128) { const float d = Dy[threadIdx.x].x; in_range &= d >= 9.0949470177292824e-13f && d <= 1099511627776.f; }   // 2^-40 .. 2^40
  asm volatile("cp.async.wait_all;" ::: "memory");
  const bool fast_cta = __syncthreads_and(in_range);
  const float ysc = __fdiv_rn(1.f, sc);


  auto write_results = [&](int s, int first, int step) {       // rows of sub-block s: dequantised values, codes, errors
    const float* e = Eb + (s & 1) * SUB * QES;
    const float* c = Cb + (s & 1) * SUB * QCH;
    if (!live) return;
    for (int i = first; i < SUB && SUB * s + i < bs; i += step) {
      const int64_t o = (int64_t)(start + SUB * s + i) * N + col;
      const float cv = c[i * QCH + lane];
      reinterpret_cast<QT*>(p.Q)[o] = from_f32<QT>(__fmul_rn(sc, __fsub_rn(cv, zr)));
      if (p.codes) p.codes[o] = (uint8_t)cv;
      // Not finite: stored as the NaN that survives the operand split of the tail tiles (an infinity's low part would be one)
      const float err = e[i * QES + lane];
      p.W[o] = fabsf(err) <= 3.402823466e38f ? err : __uint_as_float(0x7fc00000u);
    }
  };
  // The helpers' half-warps take two neighbouring rows, two channels per lane: a broadcast of L then feeds two
  // channels, and shared memory, which these updates would otherwise wait for, is read half as often.
  const int hc = 2 * (lane & 15), hr = lane >> 4;
  auto l_row = [&](int r) {
    const int g = r / SUB;
    return reinterpret_cast<const float4*>(Ld + ltri_base(g) + (r % SUB) * ltri_stride(g));
  };
  // four errors, in row order, into the two weights of a lane
  auto take4 = [&](float2& w, const float4& l, const float2& e0, const float2& e1, const float2& e2, const float2& e3) {
    w.x = __fsub_rn(w.x, __fmul_rn(l.x, e0.x)); w.y = __fsub_rn(w.y, __fmul_rn(l.x, e0.y));
    w.x = __fsub_rn(w.x, __fmul_rn(l.y, e1.x)); w.y = __fsub_rn(w.y, __fmul_rn(l.y, e1.y));
    w.x = __fsub_rn(w.x, __fmul_rn(l.z, e2.x)); w.y = __fsub_rn(w.y, __fmul_rn(l.z, e2.y));
    w.x = __fsub_rn(w.x, __fmul_rn(l.w, e3.x)); w.y = __fsub_rn(w.y, __fmul_rn(l.w, e3.y));
  };

  // The next block's rows: helper h sums rows 16 h .. + 15 over the contraction index, sub-block by sub-block, all 32
  // channels; the operand of L for the coming sub-block is fetched one ahead.
  const int fg = lane >> 2, fq = lane & 3;
  const int fr0 = 16 * (warp - 1) + fg, fr1 = fr0 + 8;
  const bool feeds_next = p.make_next && warp > 0 && 16 * (warp - 1) < bs;
  const float* LN = p.L + (int64_t)(start + bs + fr0) * K + start + fq;
  float pacc[4][4], fa[2][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) pacc[j][e] = 0.f;
  auto fetch_next = [&](int s) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k0 = SUB * s + 8 * u, k1 = k0 + 4;
      fa[u][0] = (fr0 < bs && k0 + fq < bs) ? __ldg(LN + k0) : 0.f;
      fa[u][1] = (fr1 < bs && k0 + fq < bs) ? __ldg(LN + (int64_t)8 * K + k0) : 0.f;
      fa[u][2] = (fr0 < bs && k1 + fq < bs) ? __ldg(LN + k1) : 0.f;
      fa[u][3] = (fr1 < bs && k1 + fq < bs) ? __ldg(LN + (int64_t)8 * K + k1) : 0.f;
    }
  };
  auto feed_next = [&](int s) {                 // errors of sub-block s
    const float* e = Eb + (s & 1) * SUB * QES + fg;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k0 = 8 * u + fq, k1 = k0 + 4;
      if (SUB * s + 8 * u < bs) {
        uint32_t ah[4], al[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split_tf32_alu(fa[u][i], ah[i], al[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t bh[2], bl[2];
          split_tf32(SUB * s + k0 < bs ? e[k0 * QES + 8 * j] : 0.f, bh[0], bl[0]);
          split_tf32(SUB * s + k1 < bs ? e[k1 * QES + 8 * j] : 0.f, bh[1], bl[1]);
          mma_tf32(pacc[j], al, bh);
          mma_tf32(pacc[j], ah, bl);
          mma_tf32(pacc[j], ah, bh);
        }
      }
    }
  };
  if (feeds_next) fetch_next(0);

  for (int s = 0; s < nsub; ++s) {
    const int s0 = SUB * s, sn = min(SUB, bs - s0);
    float* eb = Eb + (s & 1) * SUB * QES + lane;
    if (warp == 0) {
      // ---- the chain: quantize row after row, errors into the rows behind ----
      float* cb = Cb + (s & 1) * SUB * QCH + lane;
      const float2* dy = Dy + s0;
      float w[SUB];
#pragma unroll
      for (int i = 0; i < SUB; ++i) w[i] = (i < sn) ? Wb[(s0 + i) * QCH + lane] : 0.f;
      int handed = 0;                         // groups of four errors handed to the other warps
      if (fast_cta && sn == SUB) {
        // Four steps per turn, the remaining rows moving down to w[0] after each (the rows that come up from behind
        // are not part of the sub-block and never used): a turn is short enough to stay in the instruction cache.
        bool ok = true;
        const float4* lcol = reinterpret_cast<const float4*>(Lt + s0 * SUB);
#pragma unroll 1
        for (int t = 0; t < 4; ++t) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 dv = dy[4 * t + j];
            float4 l[4];                      // this step's column of the sub-block, rows 4 t .. (in time for the error)
#pragma unroll
            for (int q = 0; q < 4; ++q) l[q] = lcol[4 * j + q];
            ok &= fabsf(w[j]) <= 1.152921504606847e18f;
            // round(w / scale) by adding and subtracting 1.5 * 2^23; beyond 2^22 the sum only has to stay outside [0, maxq]
            float c = __fsub_rn(__fadd_rn(divide_exact(w[j], sc, ysc), 12582912.f), 12582912.f);
            c = fminf(fmaxf(__fadd_rn(c, zr), 0.f), p.maxq);
            const float r = __fsub_rn(w[j], __fmul_rn(sc, __fsub_rn(c, zr)));
            ok &= (__float_as_uint(fabsf(r)) - 1u) >= 0x12800000u - 1u;         // zero, or at least 2^-90
            const float err = divide_exact(r, dv.x, dv.y);
            eb[(4 * t + j) * QES] = err;
            cb[(4 * t + j) * QCH] = c;
#pragma unroll
            for (int x = j + 1; x < SUB; ++x) {
              const float4 v = l[x / 4];
              w[x] = __fsub_rn(w[x], __fmul_rn(x % 4 == 0 ? v.x : x % 4 == 1 ? v.y : x % 4 == 2 ? v.z : v.w, err));
            }
          }
          if (!__all_sync(0xffffffffu, ok)) break;
          asm volatile("bar.arrive %0, %1;" ::"r"(1 + t), "r"(QTHREADS) : "memory");
          handed = t + 1;
          lcol += 4 * (SUB / 4) + 1;          // four columns on, four rows down
#pragma unroll
          for (int x = 0; x < SUB - 4; ++x) w[x] = w[x + 4];
        }
      }
      if (handed < 4) {
        // the general path, row by row in shared memory
        const float* ls = Lt + s0 * SUB;
#pragma unroll 1
        for (int i = 0; i < sn; ++i) {
          // quantize_value: clip(round(w / scale) + zero, 0, maxq), then scale * (q - zero)
          const float wi = Wb[(s0 + i) * QCH + lane];
          float c = __fadd_rn(rintf(__fdiv_rn(wi, sc)), zr);
          c = fminf(fmaxf(c, 0.f), p.maxq);
          const float qv = __fmul_rn(sc, __fsub_rn(c, zr));
          const float err = __fdiv_rn(__fsub_rn(wi, qv), dy[i].x);
          if (i >= 4 * handed) { eb[i * QES] = err; cb[i * QCH] = c; }
          for (int ii = i + 1; ii < sn; ++ii) {
            float* wp = Wb + (s0 + ii) * QCH + lane;
            *wp = __fsub_rn(*wp, __fmul_rn(ls[i * SUB + ii], err));
          }
        }
        for (int t = handed; t < 4; ++t) asm volatile("bar.arrive %0, %1;" ::"r"(1 + t), "r"(QTHREADS) : "memory");
      }
    } else {
      // ---- beside it: the next sub-block's eight row pairs, one per warp, in registers ----
      const int h = warp - 1;
      const int n0 = s0 + SUB, n_end = min(bs, n0 + SUB);
      const float* eprev = Eb + ((s - 1) & 1) * SUB * QES + hc;
      const float* ecur = Eb + (s & 1) * SUB * QES + hc;
      const bool next = n0 < bs;
      const int rn = min(n0 + 2 * h + hr, n_end - 1);                   // a row past the end repeats the last one, unused
      const float4* ln = l_row(next ? rn : 0);
      float2 ep[SUB], wn = make_float2(0.f, 0.f);
      if (next) wn = *reinterpret_cast<const float2*>(Wb + rn * QCH + hc);
      if (s > 0) {
#pragma unroll
        for (int i = 0; i < SUB; ++i) ep[i] = *reinterpret_cast<const float2*>(eprev + i * QES);
        // the previous sub-block's errors: this warp's pair of the next sub-block first, then the pairs behind that one,
        // as many per turn as are left, and the results
#pragma unroll 1
        for (int r0 = n0 + 2 * h; r0 < bs; r0 += 4 * QHELP) {
          const int r1 = r0 + 2 * QHELP;
          const int ra = min(r0 + hr, bs - 1), rb = min(r1 + hr, bs - 1);
          float2 wa = *reinterpret_cast<const float2*>(Wb + ra * QCH + hc), wb = *reinterpret_cast<const float2*>(Wb + rb * QCH + hc);
          const float4* la = l_row(ra) + 4 * (s - 1);
          const float4* lb = l_row(rb) + 4 * (s - 1);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            take4(wa, la[q], ep[4 * q], ep[4 * q + 1], ep[4 * q + 2], ep[4 * q + 3]);
            take4(wb, lb[q], ep[4 * q], ep[4 * q + 1], ep[4 * q + 2], ep[4 * q + 3]);
          }
          if (r0 == n0 + 2 * h) wn = wa;
          else if (r0 + hr < bs) *reinterpret_cast<float2*>(Wb + ra * QCH + hc) = wa;
          if (r1 + hr < bs) *reinterpret_cast<float2*>(Wb + rb * QCH + hc) = wb;
        }
        write_results(s - 1, h, QHELP);
        if (feeds_next) { feed_next(s - 1); fetch_next(s); }
      }
#pragma unroll 1
      for (int t = 0; t < 4; ++t) {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + t), "r"(QTHREADS) : "memory");
        if (next) {
          float2 e[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) e[i] = *reinterpret_cast<const float2*>(ecur + (4 * t + i) * QES);
          take4(wn, ln[4 * s + t], e[0], e[1], e[2], e[3]);
        }
      }
      if (next && n0 + 2 * h + hr < n_end) *reinterpret_cast<float2*>(Wb + rn * QCH + hc) = wn;
    }
    __syncthreads();
    // the next block's CTAs may be placed (and fetch their part of L) from the last sub-block on
    if (s + 2 == nsub || nsub == 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  write_results(nsub - 1, warp, QWARPS);
  if (feeds_next) {
    feed_next(nsub - 1);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = e < 2 ? fr0 : fr1;
        const int64_t c = ch0 + 8 * j + 2 * fq + (e & 1);
        if (r < bs && c < N) p.P[(int64_t)r * N + c] = pacc[j][e];
      }
  }
}

template <typename QT>
static int run_quantize(float* W, const float* L, const float* scale, const float* zero,
                        int K, int64_t N, int bs, int maxq, QT* Q, uint8_t* codes, float* P, cudaStream_t s) {
  auto kern = gptq_block_kernel<QT>;
  struct AttrTag {};
  once_per_device<AttrTag>([&]() {
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    cudaGetLastError();
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, QSMEM_BYTES);
  });
  const bool fused = tail_on_tensor_cores() != 0;
  QuantParams p;
  memset(&p, 0, sizeof(p));
  p.W = W; p.L = L; p.scale = scale; p.zero = zero; p.Q = Q; p.codes = codes;
  p.K = K; p.N = N; p.bs = bs; p.maxq = (float)maxq;
  p.nch = (int)cdiv(N, QCH);
  p.vec = (K % 4 == 0) && (N % 4 == 0) && (bs % 4 == 0) && aligned(L, 16) && aligned(W, 16) && aligned(P, 16);
  p.tail_tn = (int)cdiv(N, TBN);
  p.P = P;
  for (int start = 0; start < K; start += bs) {
    p.start = start;
    p.apply_prev = fused && start > 0;
    const int rest = K - (start + bs);
    p.make_next = fused && rest > 0;
    p.rest = rest;
    const int tiles = (p.apply_prev && rest > 0) ? (int)cdiv(rest, TBM) * p.tail_tn : 0;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(p.nch + tiles));
    cfg.blockDim = dim3(QTHREADS);
    cfg.dynamicSmemBytes = QSMEM_BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = start > 0 ? 1 : 0;       // the first one reads what other kernels of the stream have written
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    note_launches(1);
    if (e != cudaSuccess) { cudaGetLastError(); return fail(JGQ_ERR_CUDA, "gptq_block: %s", cudaGetErrorString(e)); }
    if (!fused && rest > 0) {
      const int rc = launch_sgemm(true, false, L + (int64_t)(start + bs) * K + start, K, W + (int64_t)start * N, N,
                                  W + (int64_t)(start + bs) * N, N, rest, (int)N, bs, -1.f, 1.f, 0, s);
      if (rc) return rc;
    }
  }
  return JGQ_OK;
}

}  // namespace jgq

using namespace jgq;

extern "C" size_t jgq_gptq_quantize_workspace_bytes(int64_t K, int64_t N, int block_size) {
  if (K <= 0 || N <= 0 || block_size <= 0) return 0;
  return align_up((size_t)block_size * (size_t)N * sizeof(float), 256);
}

extern "C" int jgq_gptq_quantize(float* W, const float* L, const float* scale, const float* zero,
                                 int64_t K, int64_t N, int block_size, int maxq,
                                 void* Q, int q_dtype, uint8_t* codes,
                                 void* ws, size_t ws_bytes, void* stream) {
  JGQ_REQUIRE(K > 0 && N > 0, JGQ_ERR_ARG, "gptq_quantize: bad shape K=%lld N=%lld", (long long)K, (long long)N);
  JGQ_REQUIRE(K <= 46340 && N <= 2147483647LL, JGQ_ERR_LIMIT, "gptq_quantize: shape too large");
  JGQ_REQUIRE(block_size >= 1 && block_size <= 128, JGQ_ERR_ARG, "gptq_quantize: block_size %d not in [1,128]", block_size);
  JGQ_REQUIRE(K % block_size == 0, JGQ_ERR_ARG,
              "gptq_quantize: K=%lld is not a multiple of block_size=%d", (long long)K, block_size);
  JGQ_REQUIRE(maxq >= 1 && maxq <= 255, JGQ_ERR_ARG, "gptq_quantize: maxq %d out of range", maxq);
  JGQ_REQUIRE(q_dtype == JGQ_F32 || q_dtype == JGQ_F16 || q_dtype == JGQ_BF16, JGQ_ERR_ARG,
              "gptq_quantize: Q dtype must be f32/f16/bf16");
  JGQ_REQUIRE(W && L && scale && zero && Q && ws, JGQ_ERR_ARG, "gptq_quantize: null pointer");
  JGQ_REQUIRE(ws_bytes >= jgq_gptq_quantize_workspace_bytes(K, N, block_size), JGQ_ERR_WORKSPACE,
              "gptq_quantize: workspace %zu < %zu bytes", ws_bytes, jgq_gptq_quantize_workspace_bytes(K, N, block_size));
  JGQ_REQUIRE(aligned(ws, 16), JGQ_ERR_ALIGN, "gptq_quantize: workspace must be 16-byte aligned");
  // K / block_size launches whose arguments depend on these values alone: replayed as a graph when they recur
  struct { int tag; int block_size, maxq, q_dtype; int64_t K, N; const void *W, *L, *scale, *zero, *Q, *codes, *ws; } key;
  memset(&key, 0, sizeof(key));
  key.tag = 2; key.block_size = block_size; key.maxq = maxq; key.q_dtype = q_dtype; key.K = K; key.N = N;
  key.W = W; key.L = L; key.scale = scale; key.zero = zero; key.Q = Q; key.codes = codes; key.ws = ws;
  return run_replayed(key, (cudaStream_t)stream, [&](cudaStream_t s) {
    switch (q_dtype) {
      case JGQ_F32:  return run_quantize<float>(W, L, scale, zero, (int)K, N, block_size, maxq, (float*)Q, codes, (float*)ws, s);
      case JGQ_F16:  return run_quantize<__half>(W, L, scale, zero, (int)K, N, block_size, maxq, (__half*)Q, codes, (float*)ws, s);
      default:       return run_quantize<__nv_bfloat16>(W, L, scale, zero, (int)K, N, block_size, maxq, (__nv_bfloat16*)Q, codes, (float*)ws, s);
    }
  });
}
