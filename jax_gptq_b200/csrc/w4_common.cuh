// Device helpers shared by the packed-int4 matmul kernels: MMA wrappers with the nibble
// expansion for f16 / bf16 operands, guarded activation loads, scale / zero loads.
#pragma once
#include "common.cuh"
#include <type_traits>

namespace jgq {

constexpr int WCOLS = 128;          // channels per CTA
constexpr int WWARPS = 4;
constexpr int PSTRIDE = WCOLS + 4;  // floats per partial row: 128 sums + sum_k x (+pad)
// Every forward kernel keeps its int32 tickets (and scheduling words) in the first W4_TICKET_REGION bytes of
// the workspace and its fp32 slices behind them: the kernels share one workspace, and what one of them
// writes as slices must never land on words another one expects to find zero.
constexpr int W4_TICKET_REGION = 16384;

template <typename XT> struct MmaType;
template <> struct MmaType<__half> {
  static constexpr uint32_t kMagic = 0x64006400u;  // 1024 | code
  __device__ static __forceinline__ uint32_t expand(uint32_t v) {
    uint32_t r = (v & 0x000F000Fu) | kMagic;
    __half2 h = __hsub2(*reinterpret_cast<__half2*>(&r), __half2half2(__float2half_rn(1024.f)));
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __device__ static __forceinline__ uint32_t ones() { return 0x3C003C00u; }
  __device__ static __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
};
template <> struct MmaType<__nv_bfloat16> {
  static constexpr uint32_t kMagic = 0x43004300u;  // 128 | code
  __device__ static __forceinline__ uint32_t expand(uint32_t v) {
    uint32_t r = (v & 0x000F000Fu) | kMagic;
    __nv_bfloat162 h = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&r), __float2bfloat162_rn(128.f));
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __device__ static __forceinline__ uint32_t ones() { return 0x3F803F80u; }
  __device__ static __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
};

// 16 packed bytes of byte row `row`, channels c0..c0+15 (zero outside the matrix).
__device__ __forceinline__ uint4 load_codes16(const uint8_t* __restrict__ packed, int64_t row, int64_t KB,
                                              int64_t c0, int64_t N, bool vec) {
  uint4 r = make_uint4(0, 0, 0, 0);
  if (row >= KB || c0 >= N) return r;
  const uint8_t* p = packed + row * N + c0;
  if (vec && c0 + 15 < N) {
    r = __ldg(reinterpret_cast<const uint4*>(p));
  } else {
    uint32_t w[4] = {0, 0, 0, 0};
    for (int b = 0; b < 16; ++b)
      if (c0 + b < N) w[b >> 2] |= (uint32_t)p[b] << (8 * (b & 3));
    r = make_uint4(w[0], w[1], w[2], w[3]);
  }
  return r;
}

// Two consecutive activations x[m, k], x[m, k+1] as one MMA operand register (zero outside).
template <typename XT>
__device__ __forceinline__ uint32_t load_x2(const XT* __restrict__ x, int64_t m, int64_t M, int64_t k, int64_t K) {
  if (m >= M || k >= K) return 0u;      // K is even and k is even: k+1 < K as well
  return *reinterpret_cast<const uint32_t*>(x + m * K + k);
}

// fp32 activations: split into bf16 high and low parts (x = hi + lo + O(2^-17 |x|)).
__device__ __forceinline__ void load_x2_split(const float* __restrict__ x, int64_t m, int64_t M, int64_t k, int64_t K,
                                              uint32_t& hi, uint32_t& lo) {
  hi = 0u; lo = 0u;
  if (m >= M || k >= K) return;
  const float2 v = *reinterpret_cast<const float2*>(x + m * K + k);
  const __nv_bfloat16 h0 = __float2bfloat16_rn(v.x), h1 = __float2bfloat16_rn(v.y);
  const __nv_bfloat16 l0 = __float2bfloat16_rn(v.x - __bfloat162float(h0));
  const __nv_bfloat16 l1 = __float2bfloat16_rn(v.y - __bfloat162float(h1));
  hi = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
  lo = (uint32_t)__bfloat16_as_ushort(l0) | ((uint32_t)__bfloat16_as_ushort(l1) << 16);
}

template <typename T> __device__ __forceinline__ float zs_to_f32(const void* p, int64_t i);
template <> __device__ __forceinline__ float zs_to_f32<float>(const void* p, int64_t i) { return ((const float*)p)[i]; }
template <> __device__ __forceinline__ float zs_to_f32<__half>(const void* p, int64_t i) { return __half2float(((const __half*)p)[i]); }

// Activation fragment (MMA B operand, 16 k x 8 tokens) of one 16-step for lane (g, q):
// token m0 + 8*t + g, contraction k0 + 2q.. and k0 + 8 + 2q..
template <typename XT, int NTOK>
__device__ __forceinline__ void load_xfrags(const XT* __restrict__ x, int64_t m0, int64_t M, int64_t k0, int64_t K,
                                            int g, int q, uint32_t (&b)[NTOK][2], uint32_t (&blo)[NTOK][2]) {
  constexpr bool kSplitX = std::is_same<XT, float>::value;
#pragma unroll
  for (int t = 0; t < NTOK; ++t) {
    const int64_t m = m0 + 8 * t + g;
    if (kSplitX) {
      load_x2_split((const float*)x, m, M, k0 + 2 * q, K, b[t][0], blo[t][0]);
      load_x2_split((const float*)x, m, M, k0 + 8 + 2 * q, K, b[t][1], blo[t][1]);
    } else {
      b[t][0] = load_x2<XT>(x, m, M, k0 + 2 * q, K);
      b[t][1] = load_x2<XT>(x, m, M, k0 + 8 + 2 * q, K);
      blo[t][0] = blo[t][1] = 0u;
    }
  }
}

// mma with the fragment roles of this kernel: D[16 ch x 8 tok] += A[16 ch x 16 k] * B[16 k x 8 tok]
template <typename CT>
__device__ __forceinline__ void mma_wx(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       const uint32_t (&b)[2]) {
  const uint32_t a[4] = {a0, a1, a2, a3};
  MmaType<CT>::mma(d, a, b[0], b[1]);
}

// One 16-step: 8 MMAs per token octet over the 2 x 16 bytes this lane holds, plus the MMA with ones.
template <typename CT, int NTOK, bool kSplitX>
__device__ __forceinline__ void w4_step(float (&acc)[NTOK][8][4], float (&accx)[NTOK][4], const uint4& r0, const uint4& r1,
                                        const uint32_t (&xb)[NTOK][2], const uint32_t (&xlo)[NTOK][2]) {
  const uint32_t w0[4] = {r0.x, r0.y, r0.z, r0.w};
  const uint32_t w1[4] = {r1.x, r1.y, r1.z, r1.w};
#pragma unroll
  for (int wi = 0; wi < 2; ++wi) {
    // words wi (channels 4wi..4wi+3) and wi + 2 (channels 8 + 4wi ..) of both byte rows
    const uint32_t u0 = w0[wi], u0s = u0 >> 4, v0 = w0[wi + 2], v0s = v0 >> 4;
    const uint32_t u1 = w1[wi], u1s = u1 >> 4, v1 = w1[wi + 2], v1s = v1 >> 4;
#pragma unroll
    for (int bi = 0; bi < 4; ++bi) {
      const uint32_t sel = (uint32_t)bi | ((uint32_t)bi << 4) | ((uint32_t)(4 + bi) << 8) | ((uint32_t)(4 + bi) << 12);
      const uint32_t a0 = MmaType<CT>::expand(__byte_perm(u0, u0s, sel));   // channel 4wi+bi,     k 2q..
      const uint32_t a1 = MmaType<CT>::expand(__byte_perm(v0, v0s, sel));   // channel 8+4wi+bi,   k 2q..
      const uint32_t a2 = MmaType<CT>::expand(__byte_perm(u1, u1s, sel));   // channel 4wi+bi,     k 8+2q..
      const uint32_t a3 = MmaType<CT>::expand(__byte_perm(v1, v1s, sel));   // channel 8+4wi+bi,   k 8+2q..
#pragma unroll
      for (int t = 0; t < NTOK; ++t) {
        mma_wx<CT>(acc[t][wi * 4 + bi], a0, a1, a2, a3, xb[t]);
        if (kSplitX) mma_wx<CT>(acc[t][wi * 4 + bi], a0, a1, a2, a3, xlo[t]);
      }
    }
  }
  const uint32_t one = MmaType<CT>::ones();
#pragma unroll
  for (int t = 0; t < NTOK; ++t) {
    mma_wx<CT>(accx[t], one, one, one, one, xb[t]);
    if (kSplitX) mma_wx<CT>(accx[t], one, one, one, one, xlo[t]);
  }
}

template <typename T>
__global__ void xsum_kernel(const T* __restrict__ x, float* __restrict__ xsum, int64_t K) {
  __shared__ float part[8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int64_t m = blockIdx.x;
  float s = 0.f;
  for (int64_t k = threadIdx.x; k < K; k += blockDim.x) s += to_f32<T>(x[m * K + k]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    xsum[m] = t;
  }
}

// sum over k of the two bf16 planes of a split fp32 activation row: exactly what the MMAs see, so that
// the offset of the expanded codes cancels exactly in the epilogue
static __global__ void xsum_planes_kernel(const __nv_bfloat16* __restrict__ P0, const __nv_bfloat16* __restrict__ P1,
                                   float* __restrict__ xsum, int64_t K) {
  __shared__ float part[8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int64_t m = blockIdx.x;
  float s = 0.f;
  for (int64_t k = threadIdx.x; k < K; k += blockDim.x)
    s += __bfloat162float(P0[m * K + k]) + __bfloat162float(P1[m * K + k]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    xsum[m] = t;
  }
}

static __global__ void split_x_bf16_kernel(const float* __restrict__ X, __nv_bfloat16* __restrict__ P0,
                                    __nv_bfloat16* __restrict__ P1, int64_t total) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const float v = X[t];
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    P0[t] = h;
    P1[t] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
}

// Four consecutive values as fp32: one load where `vec`, else what lies below `lim`, zeros behind.
template <typename T>
__device__ __forceinline__ void load4(float (&f)[4], const T* p, uint32_t n, uint32_t lim, bool vec) {
  __align__(16) T e[4];
  if (vec) {
    using V = typename std::conditional<sizeof(T) == 4, float4, uint2>::type;
    *reinterpret_cast<V*>(e) = *reinterpret_cast<const V*>(p + n);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = n + i < lim ? p[n + i] : from_f32<T>(0.f);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = to_f32<T>(e[i]);
}

// The activations of the transposed product: xs = x * scale times a power of two of the token row, as two f16 planes hi + lo
// [M][Np] (zero beyond N), and c[m] = (sum_n x scale zero, the inverse power of two).  PAIRED: channels 0, 2, 1, 3 within each four.
// The power of two brings the largest product of the row to [2^13, 2^14).  The planes then hold 22 bits of every element
// down to 2^-16 of it, whatever the row's magnitude (gradients of a mean over many tokens are far below f16's range).
// One CTA per row, which keeps 4 J THREADS products in registers between the two uses and forms what is longer twice.
template <typename XT, typename ZST, int THREADS, int J, bool PAIRED>
__global__ void __launch_bounds__(THREADS, 2048 / THREADS)
tb_prep_kernel(const XT* __restrict__ x, const ZST* __restrict__ scale, const ZST* __restrict__ zero,
               uint32_t N, uint32_t Np, __half* __restrict__ hi, __half* __restrict__ lo, float2* __restrict__ c, int vec) {
  const int64_t m = blockIdx.x;
  __shared__ float pmax[THREADS / 32], psum[THREADS / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  x += m * N;
  hi += m * Np;
  lo += m * Np;
  float v[J][4], big = 0.f, s = 0.f;
  auto products = [&](float (&p)[4], uint32_t n) {
    float a[4], z[4];
    load4<XT>(p, x, n, N, vec != 0);
    load4<ZST>(a, scale, n, N, vec != 0);
    load4<ZST>(z, zero, n, N, vec != 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[i] = n + i < N ? __fmul_rn(p[i], a[i]) : 0.f;
      big = fmaxf(big, fabsf(p[i]));
      s = fmaf(p[i], z[i], s);
    }
  };
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const uint32_t n = 4 * (threadIdx.x + THREADS * j);
    if (n < N) products(v[j], n);
  }
  for (uint32_t n = 4 * (threadIdx.x + THREADS * J); n < N; n += 4 * THREADS) {
    float p[4];
    products(p, n);
  }
  // fixed-order reductions: lanes by shuffle, warps in index order
  for (int o = 16; o > 0; o >>= 1) {
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  if ((threadIdx.x & 31) == 0) { pmax[threadIdx.x >> 5] = big; psum[threadIdx.x >> 5] = s; }
  __syncthreads();
  for (int w = 0; w < THREADS / 32; ++w) big = fmaxf(big, pmax[w]);
  const uint32_t e = min(max(__float_as_uint(big) >> 23, 14u), 254u);      // biased exponent; rows below 2^-113 get 2^126
  const float up = __uint_as_float((267u - e) << 23);
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < THREADS / 32; ++w) t += psum[w];
    c[m] = make_float2(t, __uint_as_float((e - 13u) << 23));
  }
  auto store = [&](const float (&p)[4], uint32_t n) {
    __half h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float q = p[PAIRED && (i == 1 || i == 2) ? 3 - i : i] * up;
      h[i] = __float2half_rn(q);
      l[i] = __float2half_rn(q - __half2float(h[i]));
    }
    *reinterpret_cast<uint2*>(hi + n) = *reinterpret_cast<const uint2*>(h);
    *reinterpret_cast<uint2*>(lo + n) = *reinterpret_cast<const uint2*>(l);
  };
  const float none[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const uint32_t n = 4 * (threadIdx.x + THREADS * j);
    if (n < N) store(v[j], n);
    else if (n < Np) store(none, n);
  }
  for (uint32_t n = 4 * (threadIdx.x + THREADS * J); n < Np; n += 4 * THREADS) {
    float p[4] = {0.f, 0.f, 0.f, 0.f};
    if (n < N) products(p, n);
    store(p, n);
  }
}

// Blocks as wide as a row needs with few products per thread: 32 registers, so that an SM's 2048 threads hide the loads, which
// is what bounds it (2048 rows of 768 channels with 32 products per thread and half the threads: 4 us more).  Wide ones also
// for few rows, where one row's latency counts (one row of 32000 channels with 256 threads: 12 us more).
template <typename XT, typename ZST, bool PAIRED>
static int launch_tb_prep(const XT* x, const void* scale, const void* zero, int64_t rows, int64_t N, int64_t Np, __half* hi,
                          __half* lo, float2* c, cudaStream_t s) {
  const int vec = N % 4 == 0 && aligned(x, 4 * sizeof(XT)) && aligned(scale, 4 * sizeof(ZST)) && aligned(zero, 4 * sizeof(ZST));
  auto go = [&](auto kern, int threads) {
    kern<<<(unsigned)rows, threads, 0, s>>>(x, (const ZST*)scale, (const ZST*)zero, (uint32_t)N, (uint32_t)Np, hi, lo, c, vec);
    return check_launch("w4_matmul_tb_prep");
  };
  if (N <= 1024) return go(tb_prep_kernel<XT, ZST, 256, 1, PAIRED>, 256);
  if (N > 4096 || rows <= sm_count()) return go(tb_prep_kernel<XT, ZST, 1024, 2, PAIRED>, 1024);
  return N <= 2048 ? go(tb_prep_kernel<XT, ZST, 256, 2, PAIRED>, 256) : go(tb_prep_kernel<XT, ZST, 512, 2, PAIRED>, 512);
}

// 8 codes of one 32-bit word (4 channels x {k even, k odd}) -> four 2-channel registers.
// e02 / e13: k even, channels (0,2) / (1,3);  o02 / o13: k odd.
// The integer / logic pipe is the scarce one (half rate), so the constants come from kernel
// parameters (a mask and an exponent pattern as two immediates would cost two logic instructions
// per register) and the magic offset is removed on the FMA pipe:
//   f16:  0x6400 | c = 1024 + c -> subtract 1024;   0x6400 | c << 4 = 1024 + 16 c -> * 1/16 - 64
//   bf16: 0x4300 | c = 128 + c  -> subtract 128 (a nibble does not fit above bit 3 of a bf16 mantissa
//         without reaching the exponent, so the high nibbles are shifted down)
template <int FMT>
__device__ __forceinline__ void expand_word(uint32_t w, uint32_t mask_lo, uint32_t mask_hi, uint32_t magic,
                                            uint32_t& e02, uint32_t& e13, uint32_t& o02, uint32_t& o13) {
  if (FMT == 0) {
    const uint32_t w8 = w >> 8;
    uint32_t a = (w & mask_lo) | magic, b = (w8 & mask_lo) | magic;
    uint32_t c = (w & mask_hi) | magic, d = (w8 & mask_hi) | magic;
    const __half2 k1024 = __half2half2(__float2half_rn(1024.f));
    const __half2 k16th = __half2half2(__float2half_rn(0.0625f)), k64 = __half2half2(__float2half_rn(-64.f));
    __half2 ra = __hsub2(*reinterpret_cast<__half2*>(&a), k1024), rb = __hsub2(*reinterpret_cast<__half2*>(&b), k1024);
    __half2 rc = __hfma2(*reinterpret_cast<__half2*>(&c), k16th, k64), rd = __hfma2(*reinterpret_cast<__half2*>(&d), k16th, k64);
    e02 = *reinterpret_cast<uint32_t*>(&ra); e13 = *reinterpret_cast<uint32_t*>(&rb);
    o02 = *reinterpret_cast<uint32_t*>(&rc); o13 = *reinterpret_cast<uint32_t*>(&rd);
  } else {
    uint32_t a = (w & mask_lo) | magic, b = ((w >> 8) & mask_lo) | magic;
    uint32_t c = ((w >> 4) & mask_lo) | magic, d = ((w >> 12) & mask_lo) | magic;
    const __nv_bfloat162 k128 = __float2bfloat162_rn(128.f);
    __nv_bfloat162 ra = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&a), k128);
    __nv_bfloat162 rb = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&b), k128);
    __nv_bfloat162 rc = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&c), k128);
    __nv_bfloat162 rd = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&d), k128);
    e02 = *reinterpret_cast<uint32_t*>(&ra); e13 = *reinterpret_cast<uint32_t*>(&rb);
    o02 = *reinterpret_cast<uint32_t*>(&rc); o13 = *reinterpret_cast<uint32_t*>(&rd);
  }
}

}  // namespace jgq
