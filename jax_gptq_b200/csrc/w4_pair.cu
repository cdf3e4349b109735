// Packed-int4 product for many tokens on CTA pairs (tcgen05 cta_group::2): the forward product and its transpose.
//
//   forward     out[m, n] = scale[n] * ( sum_k x[m, k] code[k, n]  -  zero[n] * sum_k x[m, k] )
//   transposed  out[m, k] = sum_n xs[m, n] code[k, n]  -  c[m],   xs = x * scale,  c[m] = sum_n xs[m, n] zero[n]
//               (xs times a power of two of its row, see tb_prep_kernel, which the epilogue takes off again)
//
// The weights are the MMA's 256 rows (output channels n, or contraction-side outputs k in the transposed product),
// the tokens its columns.  A CTA of the pair expands the nibbles of its own 128 rows and loads its half of the
// tokens; the pair's MMA (M = 256, N = 256, issued by the even CTA) reads both CTAs' shared memory.  What bounds the
// single-CTA kernel at large M is the activations' way to the SMs (64 KB per stage of 1024 tensor clocks) and the
// two 64 KB slots its ring has room for; a pair needs 32 KB per SM and stage, and the ring holds three.
// Up to 256 tokens the block is cut to a multiple of 32: 33 rows, transposed, 4096 x 11008: 125 -> 87 us (blocks of 256: 109).
//
// A stage is 64 contraction indices and one or two blocks of 256 token columns: two neighbouring 256-token tiles of
// the same weight rows with an accumulator each (16-bit activations, forward: the expanded weights are used twice), or
// the two 16-bit planes of one tile on the same accumulator (fp32 activations; the scaled activations of the transposed
// product, hi + lo in f16).
//
// Work: items of two neighbouring tiles (512 tokens) in whole rounds over the pairs of SMs, then what is left, tile by tile
// where that lets every pair take at most one.  A pair's items follow one another without draining the pipeline: there are
// two accumulators, used in turn, and a tile's outputs leave while the next one is multiplied; the last item's are written by
// the expanding warps as well.  (Sharing tiles between pairs along the contraction was measured and dropped: the
// exchange of fp32 parts cost 20 to 200 us.)
//
// Roles (480 threads per CTA): warp 0 loads raw packed bytes (4 KB per stage), warp 10 the activations (32 KB),
// warps 2-9 expand (two warps per stage, four stages at a time), warp 1 of the even CTA issues the MMAs, warps 11-14
// write the outputs (helped by warps 2-9 at the end).  In the forward product the expanded operand is stored M-major (16 raw bytes are 16 channels of a
// byte row: two chunks of k = 2j, two of 2j + 1); in the transposed one the same bytes are 16 contraction indices of
// rows 2j and 2j + 1, stored K-major.  Either way the expansion leaves channels in the order 0, 2, 1, 3 within
// each four: the forward epilogue undoes it, the transposed product's activations are prepared in that order.
//
// The kernel in front (sums of the activations, and their planes) lets this one start at once; only what reads its
// results waits for it: the epilogue, and with two planes the activations' producer.
//
// Barriers: raw_full / raw_empty are the CTA's own.  a_full (arrivals of the expanding warps of both CTAs), x_full
// (bytes of both CTAs' loads) and acc_empty (arrivals of both CTAs' epilogue warps) live in the even CTA; a_empty, x_empty
// and acc_full exist in both and are signalled by two commits each.  No load uses multicast.  Waits are bounded: a timed-out product writes NaN.
//
// Measured (replayed over rotating weights): forward, 2048 x 4096 x 11008, bf16: 291 us on the single-CTA kernel, 177 with a
// tile per pair and launch, 152 now, 1.22 PFLOP/s (of 1.67 measured with cuBLAS in a burst; 175 us in a loop of calls that
// changes its inputs); transposed, 2048 rows on 11008 x 4096: 894 with mma.sync, 275, 244, 1.52 PFLOP/s executed for two
// planes; 512 rows, 11008 x 4096: 137 -> 98.  Up to 256 rows of 16-bit
// activations, where a pair has one or two items, it is even or up to 7 % slower than a tile per launch (256 rows, 11008 x 4096:
// 88 -> 95 us).
// Without the MMAs a stage takes 0.38 us, with them 0.68: the tensor pipe and the
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
constexpr int P_RAW_ST = 8, P_A_ST = 4;
constexpr int P_XRING_BYTES = 6 * P_XBLK_BYTES;      // three slots of two blocks, or six of one
constexpr int P_MAX_XST = 6;
constexpr int P_DQ_WARPS = 8, P_XWARP = 2 + P_DQ_WARPS, P_EPI_WARPS = 4;
constexpr int P_THREADS = 32 * (3 + P_DQ_WARPS + P_EPI_WARPS);
constexpr int P_RING_BYTES = P_RAW_ST * P_RAW_BYTES + P_A_ST * P_A_BYTES + P_XRING_BYTES;     // 192 KB
constexpr int P_OUT_STRIDE = 32 * 4 + 16;            // bytes per token in a warp's output buffer (32 rows, up to fp32)
constexpr int P_OUT_BYTES = P_EPI_WARPS * 32 * P_OUT_STRIDE;
constexpr int P_SMEM_BYTES = P_RING_BYTES + P_OUT_BYTES + 512;
constexpr int P_TMEM_COLS = 512;

struct PairParams {
  const void* zero; const void* scale; void* out;
  const float* tok;            // forward: [M] sum_k x[m, k]; transposed: [M][2] c[m] and the power of two for the sums
  int64_t M, N, K;
  int rows, depth;             // weight rows (N or K) and contraction length (K or N)
  int planes, nrp;             // activation planes, row pairs (256 weight rows each)
  int nst, items, G;           // stages per tile, items, pairs of SMs
  int twos, halves, cols;      // items of two tiles, then single tiles of 512-token blocks, then of the last token column
  int nt;                      // tokens per block: 256; fewer only if all tokens fit one block
  int x_blk, x_slot, x_st;     // activation ring: bytes per block (a CTA's half) and per slot, slots
  uint32_t emask_lo, emask_hi, emagic;
};

struct PairItem { int rp, m0, nh; };            // row pair, first token, tiles taken together (1 or 2)
__device__ __forceinline__ PairItem pair_item(const PairParams& p, int t) {
  PairItem s;
  s.nh = 1;
  if (t < p.twos) {
    s.rp = t % p.nrp; s.m0 = 512 * (t / p.nrp); s.nh = 2;
  } else if (t < p.twos + p.halves) {
    const int u = p.twos + ((t - p.twos) >> 1);
    s.rp = u % p.nrp; s.m0 = 512 * (u / p.nrp) + 256 * ((t - p.twos) & 1);
  } else {
    const int u = t - p.twos - p.halves;        // the other token columns of 256: the last one, or all (two planes)
    s.rp = u % p.nrp; s.m0 = 256 * (p.cols + u / p.nrp);
  }
  return s;
}

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
  uint8_t* out_buf = smem + P_RING_BYTES;
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(out_buf + P_OUT_BYTES);
  uint64_t* raw_empty = raw_full + P_RAW_ST;
  uint64_t* a_full = raw_empty + P_RAW_ST;
  uint64_t* a_empty = a_full + P_A_ST;
  uint64_t* x_full = a_empty + P_A_ST;
  uint64_t* x_empty = x_full + P_MAX_XST;
  uint64_t* acc_full = x_empty + P_MAX_XST;       // [2], and [2]: everything is multiplied
  uint64_t* acc_empty = acc_full + 3;             // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const bool misaligned = (smem_u32(smem) & 1023u) != 0u;       // never, but nothing may be loaded then: the outputs become NaN
  const int w_end = misaligned ? 0 : p.items;                    // items pair, pair + G, ...
  const int nst = p.nst, x_st = p.x_st;

  if (threadIdx.x == 0) {
    for (int i = 0; i < P_RAW_ST; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], P_DQ_WARPS / P_A_ST); }
    for (int i = 0; i < P_A_ST; ++i) { mbar_init(&a_full[i], 2 * P_DQ_WARPS / P_A_ST); mbar_init(&a_empty[i], 1); }
    for (int i = 0; i < P_MAX_XST; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * P_EPI_WARPS); }
    mbar_init(&acc_full[2], 1);
    *abort_flag = misaligned ? 1 : 0;
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
  const uint32_t acc_empty0 = mapa_u32(smem_u32(acc_empty), 0);

  if (warp == 0) {
    // ===================== TMA producer, packed weights =====================
    int issued = 0, rs = 0;
    uint32_t rph = 0;
    bool ok = true;
    for (int t = pair; t < w_end && ok; t += p.G) {
      const PairItem sg = pair_item(p, t);
      const int row0 = sg.rp * 256 + 128 * (int)rank;
      for (int st = 0; st < nst; ++st) {
        if (issued >= P_RAW_ST) ok = __all_sync(0xffffffffu, mbar_wait(&raw_empty[rs], rph ^ 1, abort_flag));
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(&raw_full[rs], P_RAW_BYTES);
          if (TB) tma_load_2d(raw_ring + rs * P_RAW_BYTES, &wmap, st * P_STAGE_K, row0 / 2, &raw_full[rs]);
          else    tma_load_2d(raw_ring + rs * P_RAW_BYTES, &wmap, row0, st * (P_STAGE_K / 2), &raw_full[rs]);
        }
        __syncwarp();
        ++issued;
        if (++rs == P_RAW_ST) { rs = 0; rph ^= 1; }
      }
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
    bool ok = true;
    for (int t = pair; t < w_end && ok; t += p.G) {
      const PairItem sg = pair_item(p, t);
      const int nblk = p.planes == 2 ? 2 : sg.nh;
      for (int st = 0; st < nst; ++st) {
        if (issued >= x_st) ok = __all_sync(0xffffffffu, mbar_wait(&x_empty[xs], xph ^ 1, abort_flag));
        if (!ok) break;
        if (lane == 0) {
          if (rank == 0) mbar_expect_tx(&x_full[xs], (uint32_t)(2 * nblk * p.x_blk));      // the bytes of both CTAs
          const uint32_t bar = x_full0 + (uint32_t)(xs * 8);
          for (int b = 0; b < nblk; ++b)
            tma_load_2d_pair(x_ring + xs * p.x_slot + b * p.x_blk, (p.planes == 2 && b == 1) ? &xmap1 : &xmap0,
                             st * P_STAGE_K, sg.m0 + (p.planes == 2 ? 0 : 256 * b) + (p.nt >> 1) * (int)rank, bar);
        }
        __syncwarp();
        ++issued;
        if (++xs == x_st) { xs = 0; xph ^= 1; }
      }
    }
    if (*abort_flag && issued > 0) {
      const long long t0 = clock64();
      while (clock64() - t0 < 20000000LL) {}
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (even CTA) =====================
    if (rank == 0) {
      const uint32_t idesc = make_idesc_f16(FMT, TB ? 0 : 1, 0, 256, p.nt);
      const uint64_t desc_a0 = TB ? make_desc_sw128(0, 16, 1024) : make_desc_sw128(0, 8192, 1024);
      const uint64_t desc_b0 = make_desc_sw128(0, 16, 1024);
      const uint32_t a_step = (TB ? 32 : 2048) >> 4;            // 16 contraction indices further in the A tile
      const uint32_t my_a = smem_u32(a_empty), peer_a = mapa_u32(my_a, 1);
      const uint32_t my_x = smem_u32(x_empty), peer_x = mapa_u32(my_x, 1);
      const uint32_t my_acc = smem_u32(acc_full), peer_acc = mapa_u32(my_acc, 1);
      bool ok = true;
      int as = 0, xs = 0, use = 0;                // `use`: accumulators handed out so far, in turn
      uint32_t aph = 0, xph = 0;
      for (int t = pair; t < w_end && ok; t += p.G) {
        const PairItem sg = pair_item(p, t);
        const uint32_t tacc0 = tmem_acc + (uint32_t)(256 * (use & 1)), tacc1 = tmem_acc + (uint32_t)(256 * ((use & 1) ^ 1));
        for (int h = 0; h < sg.nh && ok; ++h)     // the epilogue warps of both CTAs have read what was in the accumulator
          if (use + h >= 2)
            ok = __all_sync(0xffffffffu, mbar_wait_cluster(&acc_empty[(use + h) & 1], ((uint32_t)((use + h) >> 1) & 1u) ^ 1u, abort_flag));
        tc_fence_after();
        for (int st = 0; st < nst && ok; ++st) {
          ok = __all_sync(0xffffffffu, mbar_wait(&x_full[xs], xph, abort_flag) && mbar_wait_cluster(&a_full[as], aph, abort_flag));
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t da0 = desc_a0 + (smem_u32(a_ring + as * P_A_BYTES) >> 4);
            const uint64_t db0 = desc_b0 + (smem_u32(x_ring + xs * p.x_slot) >> 4);
#pragma unroll
            for (int k16 = 0; k16 < P_STAGE_K / 16; ++k16) {
              const uint64_t da = da0 + (uint32_t)k16 * a_step, db = db0 + (uint32_t)(k16 * 32 >> 4);
              const uint32_t on = (st > 0 || k16 > 0) ? 1u : 0u;
              mma_f16_ss_pair(tacc0, da, db, idesc, on);
              if (p.planes == 2)    mma_f16_ss_pair(tacc0, da, db + (uint32_t)(p.x_blk >> 4), idesc, 1u);
              else if (sg.nh == 2)  mma_f16_ss_pair(tacc1, da, db + (uint32_t)(p.x_blk >> 4), idesc, on);
            }
            mma_commit_pair(my_a + (uint32_t)(as * 8)); mma_commit_pair(peer_a + (uint32_t)(as * 8));
            mma_commit_pair(my_x + (uint32_t)(xs * 8)); mma_commit_pair(peer_x + (uint32_t)(xs * 8));
            if (st + 1 == nst)
              for (int h = 0; h < sg.nh; ++h) {
                const uint32_t o = (uint32_t)(((use + h) & 1) * 8);
                mma_commit_pair(my_acc + o); mma_commit_pair(peer_acc + o);
              }
          }
          tc_fence_before();
          __syncwarp();
          if (++as == P_A_ST) { as = 0; aph ^= 1; }
          if (++xs == x_st) { xs = 0; xph ^= 1; }
        }
        use += sg.nh;
      }
      if (ok && elect_one()) { mma_commit_pair(my_acc + 16); mma_commit_pair(peer_acc + 16); }
      __syncwarp();
    }
  } else if (warp < P_XWARP) {
    // ===================== nibble expansion (warps 2..9), two warps per stage =====================
    const int dw = warp - 2;
    const int as = dw >> 1;
    const int u0 = (dw & 1) * 4;                      // this warp's four of the eight 16-byte loads per lane
    bool ok = true;
    int rs = as;
    uint32_t rph = 0, aph = 0;
    const int total = pair < w_end ? (w_end - 1 - pair) / p.G * nst + nst : 0;      // stages of all items
    for (int i = as; i < total; i += P_A_ST) {
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
  }

  // ===================== outputs (warps 11..14; for the last item warps 2..9 as well) =====================
  // A warp has 32 weight rows, one per lane.  The outputs of 32 tokens at a time go through its own shared memory as
  // [token][32 rows], so that global memory sees 16-byte pieces of a token's row.
  if (warp > 1 && warp != P_XWARP) {
    const bool helper = warp < P_XWARP;
    const int q = warp & 3;                                                  // TMEM lanes 32 q .. + 31
    const int share = helper ? 1 + ((warp - 2) >> 2) : 0;                    // of the three warps with this q
    const int lrow = TB ? lane : ((lane & ~3) | ((lane & 1) << 1) | ((lane >> 1) & 1));      // forward: channels 0, 2, 1, 3
    const int64_t ld = TB ? p.K : p.N;
    // helpers use the A ring: by then every MMA has read its operands
    uint8_t* buf = helper ? a_ring + (warp - 2) * 32 * P_OUT_STRIDE : out_buf + (warp - P_XWARP - 1) * 32 * P_OUT_STRIDE;
    constexpr int V = 16 / (int)sizeof(XT);                                  // elements per 16-byte piece
    constexpr int LT = 32 / V, TPW = 32 / LT;                                // lanes per token, tokens per step
    asm volatile("griddepcontrol.wait;" ::: "memory");                       // the kernel that sums the activations
    int use = 0;
    for (int t = pair; t < p.items; t += p.G) {
      const PairItem it = pair_item(p, t);
      const bool final_item = t + p.G >= p.items;
      if (helper && !final_item) { use += it.nh; continue; }
      const int row32 = it.rp * 256 + 128 * (int)rank + 32 * q;
      const int row = row32 + lrow;
      float sc = 1.f, zr = 1.f;
      if (!TB && row < p.rows) { sc = zs_to_f32<ZST>(p.scale, row); zr = zs_to_f32<ZST>(p.zero, row); }
      const int piece = lane % LT, n_left = p.rows - row32 - piece * V;
      const bool wide = n_left >= V && (ld * (int64_t)sizeof(XT)) % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
      for (int h = 0; h < it.nh; ++h, ++use) {
        const int b = use & 1, m0 = it.m0 + 256 * h;
        // A helper has not followed acc_full's phases and could take an earlier one for the last: it waits for the end.
        const bool done = __all_sync(0xffffffffu, mbar_wait_long(helper ? &acc_full[2] : &acc_full[b],
                                                                 helper ? 0u : (uint32_t)(use >> 1) & 1u, abort_flag));
        tc_fence_after();
        const int ntok = (int)min((int64_t)256, p.M - m0);
        for (int c = final_item ? 32 * share : 0; c < ntok; c += final_item ? 96 : 32) {
          // one value per token comes by shuffle, a pair through the 16 bytes that every token's row of the buffer has left
          float tok = 0.f;
          if (TB) {
            if (c + lane < ntok)
              *reinterpret_cast<float2*>(buf + lane * P_OUT_STRIDE + 128) = *reinterpret_cast<const float2*>(p.tok + 2 * (int64_t)(m0 + c + lane));
            __syncwarp();
          } else if (c + lane < ntok) {
            tok = p.tok[m0 + c + lane];
          }
          uint32_t v[32];
          if (done) {
            tmem_ld_32x32(tmem_acc + (uint32_t)(256 * b) + ((uint32_t)(32 * q) << 16) + (uint32_t)c, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0x7fc00000u;
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            float o;
            if (TB) {
              const float2 t = *reinterpret_cast<const float2*>(buf + i * P_OUT_STRIDE + 128);
              o = fmaf(__uint_as_float(v[i]), t.y, -t.x);
            } else {
              o = sc * (__uint_as_float(v[i]) - zr * __shfl_sync(0xffffffffu, tok, i));
            }
            *reinterpret_cast<XT*>(buf + i * P_OUT_STRIDE + lrow * (int)sizeof(XT)) = from_f32<XT>(o);
          }
          __syncwarp();
#pragma unroll
          for (int i0 = 0; i0 < 32; i0 += TPW) {
            const int i = i0 + lane / LT;
            if (c + i < ntok) {
              const uint4 w = *reinterpret_cast<const uint4*>(buf + i * P_OUT_STRIDE + piece * 16);
              XT* dst = reinterpret_cast<XT*>(p.out) + (int64_t)(m0 + c + i) * ld + row32 + piece * V;
              if (wide) {
                *reinterpret_cast<uint4*>(dst) = w;
              } else {
                const XT* e = reinterpret_cast<const XT*>(&w);
#pragma unroll
                for (int x = 0; x < V; ++x)
                  if (x < n_left) dst[x] = e[x];
              }
            }
          }
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (!helper && lane == 0) mbar_arrive_cluster(acc_empty0 + (uint32_t)(b * 8));
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

// ------------------------------------------------------------------ host ----
PairPlan plan_w4_pair(int64_t M, int64_t N, int64_t K, int x_dtype, int transpose_b) {
  PairPlan pl;
  memset(&pl, 0, sizeof(pl));
  if (M < 1 || N % 16 != 0 || (!transpose_b && K % 8 != 0)) return pl;
  pl.planes = (transpose_b || x_dtype == JGQ_F32) ? 2 : 1;
  pl.rows = (int)(transpose_b ? K : N);
  pl.depth = (int)(transpose_b ? N : K);
  pl.nrp = (int)cdiv(pl.rows, 256);
  pl.nt = (int)std::min<int64_t>(256, cdiv(M, 32) * 32);
  const int64_t cols = cdiv(M, 256), tiles = pl.nrp * cols;
  if (tiles > (1 << 28)) return pl;
  const int pairs = std::max(1, sm_count() / 2);
  const int64_t blocks = pl.planes == 2 ? 0 : pl.nrp * (cols / 2);               // of two tiles
  const int64_t left = blocks % pairs, odd = tiles - 2 * blocks;
  const bool halve = 2 * left + odd <= pairs;                                     // what whole rounds leave fits one more round of single tiles
  pl.twos = (int)(halve ? blocks - left : blocks);
  pl.halves = (int)(halve ? 2 * left : 0);
  pl.cols = (int)(pl.planes == 2 ? 0 : cols / 2 * 2);
  pl.items = (int)(pl.twos + pl.halves + odd);
  pl.G = std::min(pairs, pl.items);
  // Estimate of the forward product (see w4_pair_choice): per round the stages and the outputs of a tile, more with its
  // tokens; 0.68 us a stage for two tiles at once.
  const double nst = (double)cdiv(pl.depth, P_STAGE_K), nt = pl.nt, two = 0.68 * nst + 4.0;
  const double one = pl.planes == 2 ? (0.50 + 0.00069 * nt) * nst + 0.0168 * nt : (0.475 + 0.00028 * nt) * nst + 0.0121 * nt;
  const int64_t rounds = cdiv(pl.twos, pairs), room = rounds * pairs - pl.twos;
  pl.us = (double)rounds * two + (double)cdiv(std::max<int64_t>(0, pl.halves + odd - room), pairs) * one + (pl.planes == 2 ? 7.2 : 5.9);
  pl.Np = cdiv(N, P_STAGE_K) * P_STAGE_K;
  pl.plane_bytes = pl.planes == 1 ? 0 : align_up((size_t)M * (transpose_b ? pl.Np : K) * 2, 256);
  pl.tok_bytes = align_up((size_t)M * (transpose_b ? sizeof(float2) : sizeof(float)), 256);
  pl.ws_bytes = W4_TICKET_REGION + pl.tok_bytes + 2 * pl.plane_bytes;
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
  cfg.gridDim = dim3((unsigned)(2 * pl.G));
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
  uint8_t* planes = ws + W4_TICKET_REGION + pl.tok_bytes;
  p.tok = tok;
  const void* plane[2] = {x, x};
  if (pl.planes == 2) { plane[0] = planes; plane[1] = planes + pl.plane_bytes; }
  int fmt;
  if (transpose_b) {
    const int rc = launch_tb_prep<XT, ZST, true>((const XT*)x, p.scale, p.zero, M, N, pl.Np, (__half*)plane[0], (__half*)plane[1], (float2*)tok, s);
    if (rc) return rc;
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
    rc = encode_tmap_2d_b16(&xm[b], plane[b], cols, (uint64_t)M, cols * 2, P_STAGE_K, (uint32_t)pl.nt / 2);
    if (rc) return rc;
  }
  if (transpose_b) return launch_pair_inst<XT, ZST, 0, true>(pl, p, wmap, xm[0], xm[1], s);
  return launch_pair_inst<XT, ZST, std::is_same<XT, __half>::value ? 0 : 1, false>(pl, p, wmap, xm[0], xm[1], s);
}

int launch_w4_pair(const PairPlan& pl, const void* x, int x_dtype, const uint8_t* packed, const void* zero, const void* scale,
                   int zs_dtype, void* out, int64_t M, int64_t N, int64_t K, int transpose_b, void* ws, cudaStream_t s) {
  PairParams p;
  memset(&p, 0, sizeof(p));
  p.nst = (int)cdiv(pl.depth, P_STAGE_K);
  p.items = pl.items; p.twos = pl.twos; p.halves = pl.halves; p.cols = pl.cols; p.G = pl.G;
  p.nt = pl.nt;
  p.x_blk = pl.nt / 2 * P_STAGE_K * 2;
  p.x_slot = (pl.planes == 2 || pl.twos > 0) ? 2 * p.x_blk : p.x_blk;
  p.x_st = std::min(P_MAX_XST, P_XRING_BYTES / p.x_slot);
  p.zero = zero; p.scale = scale; p.out = out;
  p.M = M; p.N = N; p.K = K;
  p.rows = pl.rows; p.depth = pl.depth; p.planes = pl.planes; p.nrp = pl.nrp;
  uint8_t* w = (uint8_t*)ws;
  const bool zf = zs_dtype == JGQ_F32;
#define JGQ_PAIR(XT) return zf ? launch_pair_type<XT, float>(pl, p, x, packed, transpose_b, w, s) : launch_pair_type<XT, __half>(pl, p, x, packed, transpose_b, w, s)
  if (x_dtype == JGQ_F32) { JGQ_PAIR(float); }
  if (x_dtype == JGQ_F16) { JGQ_PAIR(__half); }
  JGQ_PAIR(__nv_bfloat16);
#undef JGQ_PAIR
}

}  // namespace jgq
