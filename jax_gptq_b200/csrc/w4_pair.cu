// Packed-int4 product for many tokens on CTA pairs (tcgen05 cta_group::2): the forward product and its transpose.
//
//   forward     out[m, n] = scale[n] * ( sum_k x[m, k] code[k, n]  -  zero[n] * sum_k x[m, k] )
//   transposed  out[m, k] = sum_n xs[m, n] code[k, n]  -  c[m],   xs = x * scale,  c[m] = sum_n xs[m, n] zero[n]
//
// The weights are the MMA's 256 rows (output channels n, or contraction-side outputs k in the transposed product),
// the tokens its columns.  A CTA of the pair expands the nibbles of its own 128 rows and loads its half of the
// tokens; the pair's MMA (M = 256, N = 256, issued by the even CTA) reads both CTAs' shared memory.  What bounds the
// single-CTA kernel at large M is the activations' way to the SMs (64 KB per stage of 1024 tensor clocks) and the
// two 64 KB slots its ring has room for; a pair needs 32 KB per SM and stage, and the ring holds four.
//
// A stage is 64 contraction indices and two blocks of 256 token columns: two halves of a 512-token tile with an
// accumulator each (16-bit activations, forward), or the two 16-bit planes of a 256-token tile on the same
// accumulator (fp32 activations; the scaled activations of the transposed product, hi + lo in f16).
//
// Roles (352 threads per CTA): warp 0 loads raw packed bytes (4 KB per stage), warp 10 the activations (32 KB),
// warps 2-9 expand (two warps per stage, four stages at a time), warp 1 of the even CTA issues the MMAs, warps 2-9
// write the outputs.  In the forward product the expanded operand is stored M-major (16 raw bytes are 16 channels of a
// byte row: two chunks of k = 2j, two of 2j + 1); in the transposed one the same bytes are 16 contraction indices of
// rows 2j and 2j + 1, stored K-major.  Either way the expansion leaves channels in the order 0, 2, 1, 3 within
// each four: the forward epilogue undoes it, the transposed product's activations are prepared in that order.
//
// The kernel in front (sums of the activations, and their planes) lets this one start at once; only what reads its
// results waits for it: the epilogue, and with two planes the activations' producer.
//
// Barriers: raw_full / raw_empty are the CTA's own.  a_full (arrivals of the expanding warps of both CTAs) and x_full
// (bytes of both CTAs' loads) live in the even CTA; a_empty, x_empty and acc exist in both and are signalled by two
// commits each.  No load uses multicast.  Waits are bounded: a timed-out product writes NaN.
//
// Measured (GPU time): forward 2048 x 4096 x 11008, bf16: 292 -> 176 us against the single-CTA kernel, 1.05
// PFLOP/s (of 1.67 measured with cuBLAS in a burst); transposed, 2048 rows on 11008 x 4096: 894 -> 276 us against mma.sync, 1.34
// PFLOP/s executed for two planes.  Without the MMAs a stage takes 0.38 us, with them 0.68: the tensor pipe and the
// shared-memory traffic it shares with the loads bound the rest.  Outputs written straight from the accumulators (two bytes
// per lane and token) cost 15 us per tile more than through shared memory.
#include "umma.cuh"
#include "w4_common.cuh"
#include "w4_plans.cuh"
#include <algorithm>
#include <cstring>

namespace jgq {

constexpr int P_STAGE_K = 64;
constexpr int P_RAW_BYTES = 4096;                    // 64 x 128 codes
constexpr int P_A_BYTES = 128 * P_STAGE_K * 2;       // one CTA's expanded rows
constexpr int P_XBLK_BYTES = 128 * P_STAGE_K * 2;    // one CTA's half of a 256-token block
constexpr int P_X_BYTES = 2 * P_XBLK_BYTES;
constexpr int P_RAW_ST = 8, P_A_ST = 4, P_X_ST = 4;
constexpr int P_DQ_WARPS = 8, P_XWARP = 2 + P_DQ_WARPS;
constexpr int P_THREADS = 32 * (3 + P_DQ_WARPS);
constexpr int P_RING_BYTES = P_RAW_ST * P_RAW_BYTES + P_A_ST * P_A_BYTES + P_X_ST * P_X_BYTES;     // 224 KB
constexpr int P_SMEM_BYTES = P_RING_BYTES + 512;
constexpr int P_TMEM_COLS = 512;

struct PairParams {
  const void* zero; const void* scale; void* out;
  const float* tok;            // [M]: sum_k x[m, k] (forward) or c[m] (transposed)
  int64_t M, N, K;
  int rows, depth;             // weight rows (N or K) and contraction length (K or N)
  int planes, tile, nrp;       // activation planes, tokens per tile, row pairs (256 rows each)
  uint32_t emask_lo, emask_hi, emagic;
};

template <typename XT, typename ZST, int FMT, bool TB>
__global__ void __launch_bounds__(P_THREADS, 1)
w4_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap0,
               const __grid_constant__ CUtensorMap xmap1, const PairParams p) {
  using namespace umma;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  uint8_t* raw_ring = smem;
  uint8_t* a_ring = raw_ring + P_RAW_ST * P_RAW_BYTES;
  uint8_t* x_ring = a_ring + P_A_ST * P_A_BYTES;
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + P_RING_BYTES);
  uint64_t* raw_empty = raw_full + P_RAW_ST;
  uint64_t* a_full = raw_empty + P_RAW_ST;
  uint64_t* a_empty = a_full + P_A_ST;
  uint64_t* x_full = a_empty + P_A_ST;
  uint64_t* x_empty = x_full + P_X_ST;
  uint64_t* acc_bar = x_empty + P_X_ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int unit = blockIdx.x >> 1;
  const int row0 = (unit % p.nrp) * 256 + 128 * (int)rank;      // this CTA's weight rows
  const int64_t m0 = (int64_t)(unit / p.nrp) * p.tile;
  const int ntok = (int)((p.M - m0 < (int64_t)p.tile) ? (p.M - m0) : (int64_t)p.tile);
  const int nblk = (p.planes == 2 || ntok > 256) ? 2 : 1;       // a second token block only if it has tokens
  const int nst = (p.depth + P_STAGE_K - 1) / P_STAGE_K;

  if (threadIdx.x == 0) {
    for (int i = 0; i < P_RAW_ST; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], P_DQ_WARPS / P_A_ST); }
    for (int i = 0; i < P_A_ST; ++i) { mbar_init(&a_full[i], 2 * P_DQ_WARPS / P_A_ST); mbar_init(&a_empty[i], 1); }
    for (int i = 0; i < P_X_ST; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
    mbar_init(acc_bar, 1);
    *abort_flag = (smem_u32(smem) & 1023u) != 0u ? 1 : 0;
    fence_barrier_init();
    prefetch_tensormap(&wmap);
    prefetch_tensormap(&xmap0);
    if (p.planes > 1) prefetch_tensormap(&xmap1);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)P_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                // both CTAs' barriers exist before anyone signals across
  tc_fence_after();
  const uint32_t tmem_acc = *tmem_slot;
  const uint32_t a_full0 = mapa_u32(smem_u32(a_full), 0), x_full0 = mapa_u32(smem_u32(x_full), 0);

  if (*abort_flag == 0) {
  if (warp == 0) {
    // ===================== TMA producer, packed weights =====================
    int issued = 0, rs = 0;
    uint32_t rph = 0;
    for (int i = 0; i < nst; ++i) {
      if (i >= P_RAW_ST && !__all_sync(0xffffffffu, mbar_wait(&raw_empty[rs], rph ^ 1, abort_flag))) break;
      if (lane == 0) {
        mbar_expect_tx(&raw_full[rs], P_RAW_BYTES);
        if (TB) tma_load_2d(raw_ring + rs * P_RAW_BYTES, &wmap, i * P_STAGE_K, row0 / 2, &raw_full[rs]);
        else    tma_load_2d(raw_ring + rs * P_RAW_BYTES, &wmap, row0, i * (P_STAGE_K / 2), &raw_full[rs]);
      }
      __syncwarp();
      issued = i + 1;
      if (++rs == P_RAW_ST) { rs = 0; rph ^= 1; }
    }
    if (*abort_flag && issued > 0) {       // boxes may still be in flight: a bounded time to land
      const long long t0 = clock64();
      while (clock64() - t0 < 20000000LL) {}
    }
  } else if (warp == P_XWARP) {
    // ===================== TMA producer, activations =====================
    if (p.planes == 2) asm volatile("griddepcontrol.wait;" ::: "memory");       // the planes come from the previous kernel
    int issued = 0, xs = 0;
    uint32_t xph = 0;
    for (int i = 0; i < nst; ++i) {
      if (i >= P_X_ST && !__all_sync(0xffffffffu, mbar_wait(&x_empty[xs], xph ^ 1, abort_flag))) break;
      if (lane == 0) {
        if (rank == 0) mbar_expect_tx(&x_full[xs], (uint32_t)(2 * nblk * P_XBLK_BYTES));      // the bytes of both CTAs
        const uint32_t bar = x_full0 + (uint32_t)(xs * 8);
        for (int b = 0; b < nblk; ++b)
          tma_load_2d_pair(x_ring + xs * P_X_BYTES + b * P_XBLK_BYTES, (p.planes == 2 && b == 1) ? &xmap1 : &xmap0,
                           i * P_STAGE_K, (int)m0 + (p.planes == 2 ? 0 : 256 * b) + 128 * (int)rank, bar);
      }
      __syncwarp();
      issued = i + 1;
      if (++xs == P_X_ST) { xs = 0; xph ^= 1; }
    }
    if (*abort_flag && issued > 0) {
      const long long t0 = clock64();
      while (clock64() - t0 < 20000000LL) {}
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (even CTA) =====================
    if (rank == 0) {
      const uint32_t idesc = make_idesc_f16(FMT, TB ? 0 : 1, 0, 256, 256);
      const uint64_t desc_a0 = TB ? make_desc_sw128(0, 16, 1024) : make_desc_sw128(0, 8192, 1024);
      const uint64_t desc_b0 = make_desc_sw128(0, 16, 1024);
      const uint32_t a_step = (TB ? 32 : 2048) >> 4;            // 16 contraction indices further in the A tile
      const uint32_t my_a = smem_u32(a_empty), peer_a = mapa_u32(my_a, 1);
      const uint32_t my_x = smem_u32(x_empty), peer_x = mapa_u32(my_x, 1);
      const uint32_t my_acc = smem_u32(acc_bar), peer_acc = mapa_u32(my_acc, 1);
      bool ok = true;
      int as = 0, xs = 0;
      uint32_t aph = 0, xph = 0;
      for (int i = 0; i < nst && ok; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(&x_full[xs], xph, abort_flag) && mbar_wait_cluster(&a_full[as], aph, abort_flag));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t da0 = desc_a0 + (smem_u32(a_ring + as * P_A_BYTES) >> 4);
          const uint64_t db0 = desc_b0 + (smem_u32(x_ring + xs * P_X_BYTES) >> 4);
#pragma unroll
          for (int k16 = 0; k16 < P_STAGE_K / 16; ++k16) {
            const uint64_t da = da0 + (uint32_t)k16 * a_step, db = db0 + (uint32_t)(k16 * 32 >> 4);
            const uint32_t on = (i > 0 || k16 > 0) ? 1u : 0u;
            mma_f16_ss_pair(tmem_acc, da, db, idesc, on);
            if (nblk == 2) {
              if (p.planes == 2) mma_f16_ss_pair(tmem_acc, da, db + (uint32_t)(P_XBLK_BYTES >> 4), idesc, 1u);
              else               mma_f16_ss_pair(tmem_acc + 256, da, db + (uint32_t)(P_XBLK_BYTES >> 4), idesc, on);
            }
          }
          mma_commit_pair(my_a + (uint32_t)(as * 8)); mma_commit_pair(peer_a + (uint32_t)(as * 8));
          mma_commit_pair(my_x + (uint32_t)(xs * 8)); mma_commit_pair(peer_x + (uint32_t)(xs * 8));
        }
        tc_fence_before();
        __syncwarp();
        if (++as == P_A_ST) { as = 0; aph ^= 1; }
        if (++xs == P_X_ST) { xs = 0; xph ^= 1; }
      }
      if (ok && elect_one()) { mma_commit_pair(my_acc); mma_commit_pair(peer_acc); }
      __syncwarp();
    }
  } else {
    // ===================== nibble expansion (warps 2..9), two warps per stage =====================
    const int dw = warp - 2;
    const int as = dw >> 1;
    const int u0 = (dw & 1) * 4;                      // this warp's four of the eight 16-byte loads per lane
    bool ok = true;
    int rs = as;
    uint32_t rph = 0, aph = 0;
    for (int i = as; i < nst; i += P_A_ST) {
      ok = __all_sync(0xffffffffu, mbar_wait(&raw_full[rs], rph, abort_flag));
      if (!ok) break;
      uint4 v[4];
      const uint32_t rawp = smem_u32(raw_ring + rs * P_RAW_BYTES) + (uint32_t)(u0 * 512 + lane * 16);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[u].x), "=r"(v[u].y), "=r"(v[u].z), "=r"(v[u].w)
                     : "r"(rawp + (uint32_t)(u * 512))
                     : "memory");
      if (i >= P_A_ST) {
        ok = __all_sync(0xffffffffu, mbar_wait(&a_empty[as], aph ^ 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
      }
      uint8_t* at = a_ring + as * P_A_BYTES;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        uint32_t e[8], o[8];     // low nibbles / high nibbles: 16 channels each, in expanded order
        expand_word<FMT>(v[u].x, p.emask_lo, p.emask_hi, p.emagic, e[0], e[1], o[0], o[1]);
        expand_word<FMT>(v[u].y, p.emask_lo, p.emask_hi, p.emagic, e[2], e[3], o[2], o[3]);
        expand_word<FMT>(v[u].z, p.emask_lo, p.emask_hi, p.emagic, e[4], e[5], o[4], o[5]);
        expand_word<FMT>(v[u].w, p.emask_lo, p.emask_hi, p.emagic, e[6], e[7], o[6], o[7]);
        const uint4 e0 = make_uint4(e[0], e[1], e[2], e[3]), e1 = make_uint4(e[4], e[5], e[6], e[7]);
        const uint4 o0 = make_uint4(o[0], o[1], o[2], o[3]), o1 = make_uint4(o[4], o[5], o[6], o[7]);
        if (TB) {
          // raw tile: 64 byte rows x 64 channels; lane = byte row 8 (u0 + u) + lane / 4, channels 16 (lane % 4) ..
          const int re = 2 * (8 * (u0 + u) + (lane >> 2)), ro = re + 1, ch = (lane & 3) * 2;
          const bool flip = (lane >> 2) & 1;          // odd byte rows store their second chunk first: no bank conflict
          const int ca = ch + (flip ? 1 : 0), cb = ch + (flip ? 0 : 1);
          *reinterpret_cast<uint4*>(at + re * 128 + ((ca ^ (re & 7)) << 4)) = flip ? e1 : e0;
          *reinterpret_cast<uint4*>(at + re * 128 + ((cb ^ (re & 7)) << 4)) = flip ? e0 : e1;
          *reinterpret_cast<uint4*>(at + ro * 128 + ((ca ^ (ro & 7)) << 4)) = flip ? o1 : o0;
          *reinterpret_cast<uint4*>(at + ro * 128 + ((cb ^ (ro & 7)) << 4)) = flip ? o0 : o1;
        } else {
          // raw tile: 32 byte rows x 128 channels; lane = byte row 4 (u0 + u) + lane / 8, channels 16 (lane % 8) ..
          const int ke = 2 * (4 * (u0 + u) + (lane >> 3)), ko = ke + 1;
          const int ch0 = (lane & 3) * 2;
          uint8_t* grp = at + ((lane & 7) >> 2) * 8192;
          *reinterpret_cast<uint4*>(grp + ke * 128 + (((ch0 + 0) ^ (ke & 7)) << 4)) = e0;
          *reinterpret_cast<uint4*>(grp + ke * 128 + (((ch0 + 1) ^ (ke & 7)) << 4)) = e1;
          *reinterpret_cast<uint4*>(grp + ko * 128 + (((ch0 + 0) ^ (ko & 7)) << 4)) = o0;
          *reinterpret_cast<uint4*>(grp + ko * 128 + (((ch0 + 1) ^ (ko & 7)) << 4)) = o1;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      // the raw slot goes back only after the fence: its next writer is the async proxy
      if (lane == 0) { mbar_arrive_cluster(a_full0 + (uint32_t)(as * 8)); mbar_arrive(&raw_empty[rs]); }
      aph ^= 1;
      rs += P_A_ST;
      if (rs >= P_RAW_ST) { rs -= P_RAW_ST; rph ^= 1; }
    }

    // ===================== epilogue (warps 2..9) =====================
    // A lane holds one weight row for 32 tokens at a time.  The outputs go through shared memory (the rings are idle: the
    // accumulators are complete, so every MMA has read its operands) as [token][128 rows], so that global memory
    // sees whole 256- or 512-byte pieces of a token's row.
    const bool done = __all_sync(0xffffffffu, mbar_wait(acc_bar, 0, abort_flag));
    tc_fence_after();
    asm volatile("griddepcontrol.wait;" ::: "memory");                       // the kernel that sums the activations
    const int q = warp & 3, half = dw >> 2;
    const int r = 32 * q + lane;                                             // MMA row of this CTA = TMEM lane
    const int lrow = TB ? r : ((r & ~3) | ((r & 1) << 1) | ((r >> 1) & 1));  // forward: channels 0, 2, 1, 3
    const int row = row0 + lrow;
    const int64_t ld = TB ? p.K : p.N;
    float sc = 1.f, zr = 1.f;
    if (!TB && row < p.rows) { sc = zs_to_f32<ZST>(p.scale, row); zr = zs_to_f32<ZST>(p.zero, row); }
    const int span = p.planes == 2 ? 128 : 256;                              // columns per warp
    const int c_begin = half * span, c_end = min(ntok, c_begin + span);
    XT* stage = reinterpret_cast<XT*>(smem);                                 // [token][128]: at most 512 x 256 or 256 x 512 bytes
    for (int c = c_begin; c < c_end; c += 32) {
      uint32_t v[32];
      if (done) {
        tmem_ld_32x32(tmem_acc + ((uint32_t)(32 * q) << 16) + (uint32_t)c, v);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int t = 0; t < 32; ++t) v[t] = 0x7fc00000u;
      }
#pragma unroll
      for (int t4 = 0; t4 < 32; t4 += 4) {
        const float4 tk = *reinterpret_cast<const float4*>(p.tok + m0 + c + t4);        // the array is padded past M
        const float tv[4] = {tk.x, tk.y, tk.z, tk.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          stage[(c + t4 + u) * 128 + lrow] = from_f32<XT>(sc * (__uint_as_float(v[t4 + u]) - zr * tv[u]));
      }
    }
    asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");            // the four warps of these columns
    constexpr int V = 16 / (int)sizeof(XT);                                  // elements per 16-byte piece
    constexpr int LT = 128 / V, TPW = 32 / LT;                               // lanes per token, tokens per warp and step
    const int piece = lane % LT, n_left = p.rows - row0 - piece * V;
    const bool wide = n_left >= V && (ld * (int64_t)sizeof(XT)) % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    for (int c = c_begin + q * TPW + lane / LT; c < c_end; c += 4 * TPW) {
      const uint4 w = *reinterpret_cast<const uint4*>(stage + c * 128 + piece * V);
      XT* dst = reinterpret_cast<XT*>(p.out) + (m0 + c) * ld + row0 + piece * V;
      if (wide) {
        *reinterpret_cast<uint4*>(dst) = w;
      } else {
        const XT* e = reinterpret_cast<const XT*>(&w);
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (i < n_left) dst[i] = e[i];
      }
    }
  }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // the partner may still signal this CTA's barriers or read its shared memory until here
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"((uint32_t)P_TMEM_COLS) : "memory");
  }
}

// xs = x * scale as two f16 planes [M][Np] (zero beyond N), channels 0, 2, 1, 3 within each four, and
// c[m] = sum_n xs[m, n] zero[n].  One CTA per token row, four channels per thread and step.
template <typename XT, typename ZST>
__global__ void __launch_bounds__(256)
pair_tb_prep_kernel(const XT* __restrict__ x, const void* __restrict__ scale, const void* __restrict__ zero,
                    int64_t N, int64_t Np, __half* __restrict__ hi, __half* __restrict__ lo, float* __restrict__ c) {
  const int64_t m = blockIdx.x;
  __shared__ float part[8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  float s = 0.f;
  for (int64_t n = 4 * (int64_t)threadIdx.x; n < Np; n += 1024) {
    __half h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t ni = n + (i == 1 ? 2 : i == 2 ? 1 : i);
      float v = 0.f;
      if (ni < N) {
        v = __fmul_rn(to_f32<XT>(x[m * N + ni]), zs_to_f32<ZST>(scale, ni));
        s = fmaf(v, zs_to_f32<ZST>(zero, ni), s);
      }
      h[i] = __float2half_rn(v);
      l[i] = __float2half_rn(v - __half2float(h[i]));
    }
    *reinterpret_cast<uint2*>(hi + m * Np + n) = *reinterpret_cast<const uint2*>(h);
    *reinterpret_cast<uint2*>(lo + m * Np + n) = *reinterpret_cast<const uint2*>(l);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < 8; ++w) t += part[w];
    c[m] = t;
  }
}

// ------------------------------------------------------------------ host ----
PairPlan plan_w4_pair(int64_t M, int64_t N, int64_t K, int x_dtype, int transpose_b) {
  PairPlan pl;
  memset(&pl, 0, sizeof(pl));
  if (M < 1 || N % 16 != 0 || (!transpose_b && K % 8 != 0)) return pl;
  pl.planes = (transpose_b || x_dtype == JGQ_F32) ? 2 : 1;
  pl.tile = pl.planes == 2 ? 256 : 512;
  pl.rows = (int)(transpose_b ? K : N);
  pl.depth = (int)(transpose_b ? N : K);
  pl.nrp = (int)cdiv(pl.rows, 256);
  const int64_t units = pl.nrp * cdiv(M, pl.tile);
  if (units > (1 << 28)) return pl;
  pl.units = (int)units;
  pl.Np = cdiv(N, P_STAGE_K) * P_STAGE_K;
  pl.plane_bytes = pl.planes == 1 ? 0 : align_up((size_t)M * (transpose_b ? pl.Np : K) * 2, 256);
  pl.ws_bytes = W4_TICKET_REGION + align_up((size_t)M * sizeof(float), 256) + 2 * pl.plane_bytes;
  pl.use = 1;
  return pl;
}

template <typename XT, typename ZST, int FMT, bool TB>
static int launch_pair_inst(const PairPlan& pl, const PairParams& p, const CUtensorMap& wmap, const CUtensorMap& x0,
                            const CUtensorMap& x1, cudaStream_t s) {
  auto kern = w4_pair_kernel<XT, ZST, FMT, TB>;
  struct AttrTag {};
  const int arc = once_per_device<AttrTag>([&]() {
    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 0);
    cudaGetLastError();
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM_BYTES);
  });
  if (arc != 0) return fail(JGQ_ERR_CUDA, "w4_matmul: cannot raise the dynamic shared memory limit");
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(2 * pl.units));
  cfg.blockDim = dim3(P_THREADS);
  cfg.dynamicSmemBytes = P_SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, wmap, x0, x1, p);
  note_launches(1);
  if (e != cudaSuccess) { cudaGetLastError(); return fail(JGQ_ERR_CUDA, "w4_pair: %s", cudaGetErrorString(e)); }
  return JGQ_OK;
}

template <typename XT, typename ZST>
static int launch_pair_type(const PairPlan& pl, PairParams& p, const void* x, const uint8_t* packed, int transpose_b, uint8_t* ws, cudaStream_t s) {
  const int64_t M = p.M, N = p.N, K = p.K;
  float* tok = (float*)(ws + W4_TICKET_REGION);
  uint8_t* planes = ws + W4_TICKET_REGION + align_up((size_t)M * sizeof(float), 256);
  p.tok = tok;
  const void* plane[2] = {x, x};
  if (pl.planes == 2) { plane[0] = planes; plane[1] = planes + pl.plane_bytes; }
  int fmt;
  if (transpose_b) {
    pair_tb_prep_kernel<XT, ZST><<<(unsigned)M, 256, 0, s>>>((const XT*)x, p.scale, p.zero, N, pl.Np, (__half*)plane[0], (__half*)plane[1], tok);
    JGQ_LAUNCHED();
    fmt = 0;
  } else if (pl.planes == 2) {
    const int64_t total = M * K;
    split_x_bf16_kernel<<<(int)std::min<int64_t>(cdiv(total, 256), (int64_t)sm_count() * 8), 256, 0, s>>>(
        (const float*)x, (__nv_bfloat16*)plane[0], (__nv_bfloat16*)plane[1], total);
    JGQ_LAUNCHED();
    xsum_planes_kernel<<<(unsigned)M, 256, 0, s>>>((const __nv_bfloat16*)plane[0], (const __nv_bfloat16*)plane[1], tok, K);
    JGQ_LAUNCHED();
    fmt = 1;
  } else {
    xsum_kernel<XT><<<(unsigned)M, 256, 0, s>>>((const XT*)x, tok, K);
    JGQ_LAUNCHED();
    fmt = std::is_same<XT, __half>::value ? 0 : 1;
  }
  p.emask_lo = 0x000F000Fu; p.emask_hi = 0x00F000F0u;
  p.emagic = fmt == 0 ? 0x64006400u : 0x43004300u;
  CUtensorMap wmap, xm[2];
  int rc = transpose_b ? encode_tmap_2d_u8(&wmap, packed, (uint64_t)N, (uint64_t)(K / 2), (uint64_t)N, 64, 64, 0)
                       : encode_tmap_2d_u8(&wmap, packed, (uint64_t)N, (uint64_t)(K / 2), (uint64_t)N, 128, 32, 0);
  if (rc) return rc;
  const uint64_t cols = transpose_b ? (uint64_t)pl.Np : (uint64_t)K;
  for (int b = 0; b < 2; ++b) {
    rc = encode_tmap_2d_b16(&xm[b], plane[b], cols, (uint64_t)M, cols * 2, P_STAGE_K, 128);
    if (rc) return rc;
  }
  if (transpose_b) return launch_pair_inst<XT, ZST, 0, true>(pl, p, wmap, xm[0], xm[1], s);
  return launch_pair_inst<XT, ZST, std::is_same<XT, __half>::value ? 0 : 1, false>(pl, p, wmap, xm[0], xm[1], s);
}

int launch_w4_pair(const PairPlan& pl, const void* x, int x_dtype, const uint8_t* packed, const void* zero, const void* scale,
                   int zs_dtype, void* out, int64_t M, int64_t N, int64_t K, int transpose_b, void* ws, cudaStream_t s) {
  PairParams p;
  memset(&p, 0, sizeof(p));
  p.zero = zero; p.scale = scale; p.out = out;
  p.M = M; p.N = N; p.K = K;
  p.rows = pl.rows; p.depth = pl.depth; p.planes = pl.planes; p.tile = pl.tile; p.nrp = pl.nrp;
  uint8_t* w = (uint8_t*)ws;
  const bool zf = zs_dtype == JGQ_F32;
#define JGQ_PAIR(XT) return zf ? launch_pair_type<XT, float>(pl, p, x, packed, transpose_b, w, s) : launch_pair_type<XT, __half>(pl, p, x, packed, transpose_b, w, s)
  if (x_dtype == JGQ_F32) { JGQ_PAIR(float); }
  if (x_dtype == JGQ_F16) { JGQ_PAIR(__half); }
  JGQ_PAIR(__nv_bfloat16);
#undef JGQ_PAIR
}

}  // namespace jgq
