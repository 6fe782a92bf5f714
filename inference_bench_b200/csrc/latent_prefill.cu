// Latent attention of prompt portions on the sm_100a tensor cores, with keys and values made per head.
//
// A cached row [latent c (rank) | key part r (rot)] stands for every head's key [Wuk c | r] and value Wuv c. For decoded tokens the maps go
// to the query and to the weighted sum of latents (latent_attention_mma.cu): 2 rank + rot multiplies for a (query, key) pair and head, and the
// cache is read once for all heads. A prompt portion has many queries a key, and there the maps are cheaper on the keys: one product
// [keys, rank] x [heads (dim + vdim), rank], then dim + rot + vdim multiplies a pair (320 against 1,088 at heads of 128 + 64 and a latent of
// 512), and an accumulator of vdim columns, which tensor memory holds beside two score tiles. The steps:
//   latent_gather_kernel    the rows that a step's portions see, out of the pages into [rows][rank] and [rows][64] (the key part, zeros
//                           behind it); every request's rows start at a multiple of 64, so a tile of 64 keys holds one request's rows only
//   ib_gemm_bf16_2cta       keys and values of all heads, [rows][heads * dim | heads * vdim] in bfloat16 (gemm_tcgen05_2cta.cu)
//   latent_prefill_kernel   a CTA per 128 query rows of one head: the roles of attention_prefill_ws.cu (four softmax warps, a warp that issues
//                           the MMAs one score tile ahead, a warp each for the key and value tiles), with a query of dim + rot values
// Bound by the softmax warps' chain from a score tile to the next (two CTAs an SM fill each other's gaps), then by the scores' operand reads.
// Which segments of a step come here is decided in parts/latent.py. Measured, 16 heads of 128 + 64 on a latent of 512: 2,048 tokens 8 + 19 + 47 us
// (gather, product, attention) where the maps to the latents' space and attention there took 70 + 666; 333 tokens of three requests behind 116 to
// 583 cached positions 8 + 19 + 25 against 31 + 80; 64 tokens behind 900 8 + 15 + 25 against 21 + 92; 32 tokens alone 9 + 13 + 11 against 19 + 17.
#include <cuda.h>

#include <type_traits>

#include "kv_view.cuh"
#include "mma_tiles.cuh"
#include "sm100.cuh"
#include "tma_host.cuh"

namespace {

constexpr int BM = 128, BN = 64;
constexpr int kSoftmaxWarps = 4, kThreads = (kSoftmaxWarps + 3) * 32;
constexpr float kRescaleThreshold = 8.f;  // log2 units
constexpr int KS = 2;                     // buffers for key tiles: one goes with each score tile
constexpr int kRot = 64;                  // columns of the key part's block
constexpr int kGatherRows = 8;

__device__ __forceinline__ uint32_t blk_offset(int rows, int r, int cc) {  // 16-byte chunk cc of row r in [rows][64]-element blocks, 128-byte swizzle
  return (uint32_t)((cc >> 3) * rows * 128 + r * 128 + (((cc & 7) ^ (r & 7)) << 4));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {   // round to nearest even, one instruction
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void bar_sync_softmax() { asm volatile("bar.sync 1, %0;" ::"n"(kSoftmaxWarps * 32) : "memory"); }

// blocks [n][2]: the segment and the first position of every 64 rows.
// A warp copies a row at a time; rows outside what the segment sees are zero. It does not let its dependents start early: the product that follows takes
// tensor memory before it waits, and must not do so while a product before this kernel may still be waiting for its own.
__global__ void __launch_bounds__(256) latent_gather_kernel(IbKvView kv, const int* __restrict__ blocks, const int* __restrict__ seg_start, const int* __restrict__ seg_pos0,
                                                            int window, int rank, int rot, __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ r_out,
                                                            unsigned* __restrict__ status) {
  ib::pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * kGatherRows + warp;
  const int block = (int)(row / BN), seg = blocks[2 * block], key = blocks[2 * block + 1] + (int)(row % BN);
  const int limit = seg_pos0[seg] + seg_start[seg + 1] - seg_start[seg];
  const uint4* src = nullptr;
  if (key < limit && key >= ib::first_visible(seg_pos0[seg], window)) {   // (pages before the window may be gone)
    const long long off = ib::kv_offset(kv, seg, key, 0);
    if (off < 0) {
      if (lane == 0) atomicOr(status, IB_ERR_BAD_PAGE);
    } else {
      src = (const uint4*)((const __nv_bfloat16*)kv.base + off);
    }
  }
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4* dst = (uint4*)(x + row * rank);
  for (int c = lane; c < rank / 8; c += 32) dst[c] = src ? src[c] : zero;
  if (r_out && lane < kRot / 8) ((uint4*)(r_out + row * kRot))[lane] = src && lane < rot / 8 ? src[rank / 8 + lane] : zero;
}

template <int DIM, int RB, int VD>
struct Smem {
  static constexpr int kQ = BM * (DIM + RB) * 2, kK = BN * (DIM + RB) * 2, kV = BN * VD * 2;
  // buffers for value tiles: what two CTAs an SM leave room for. One is enough: a tile's softmax lies between two uses (heads of 128 + 64, 2,048
  // tokens of 16 heads: 54 us with three buffers and one CTA an SM, 47 with one and two).
  static constexpr int kRoom = (112 * 1024 - kQ - KS * kK) / kV, VS = kRoom < 1 ? 1 : kRoom > 3 ? 3 : kRoom;
  static constexpr int oQ = 0, oK = kQ, oV = kQ + KS * kK, oBar = oV + VS * kV;
  static constexpr int kBars = KS + 2 * VS + 5;   // k_full[KS] v_full[VS] v_empty[VS] s_full[2] p_full[2] q_full; then the tmem slot and the flag
  static constexpr int kBytes = oBar + kBars * 8 + 16;
  static_assert(kBytes <= 113 * 1024, "two CTAs must fit one SM");
};

// tiles [n][4]: the first token of a tile of up to 128 consecutive tokens of one request, their number, the first one's position, and the
// row of the key matrices at which the request's position 0 would lie (its first gathered row minus its first gathered position). RB: columns
// of the turned part's block, 64 (zeros behind a part of fewer values) or 0.
template <int DIM, int RB, int VD>
__global__ void __launch_bounds__(kThreads, 2)
    latent_prefill_kernel(const __nv_bfloat16* __restrict__ q_nope, const float* __restrict__ q_rot, int q_rot_row, int rot, const int4* __restrict__ tiles,
                          const __grid_constant__ CUtensorMap kv_map, const __grid_constant__ CUtensorMap r_map, int window, float scale_log2e,
                          const float* __restrict__ sink_values, IbAttnTail tail, __nv_bfloat16* __restrict__ out, int heads, unsigned long long wait_ns,
                          unsigned* __restrict__ status) {
  using SM = Smem<DIM, RB, VD>;
  constexpr int VS = SM::VS;
  constexpr int CPR = DIM / 8, DB = DIM / 64;
  constexpr int kTmemCols = 256;            // S0 [0,64) | S1 [64,128) | O [128, 128+VD); P_j lies over the first 32 columns of S_j
  extern __shared__ __align__(1024) uint8_t sm[];
  if (sm100::smem_u32(sm) & 1023u) {
    if (threadIdx.x == 0) atomicOr(status, IB_ERR_INTERNAL);
    return;
  }
  const uint32_t q_s = sm100::smem_u32(sm + SM::oQ), k_s = sm100::smem_u32(sm + SM::oK), v_s = sm100::smem_u32(sm + SM::oV);
  uint64_t* bars = (uint64_t*)(sm + SM::oBar);
  uint64_t *k_full = bars, *v_full = bars + KS, *v_empty = bars + KS + VS, *s_full = bars + KS + 2 * VS, *p_full = s_full + 2, *q_full = s_full + 4;
  uint32_t* tmem_slot = (uint32_t*)(bars + SM::kBars);
  volatile int* gave_up = (volatile int*)(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < KS; i++) sm100::mbar_init(&k_full[i], 1);
    for (int i = 0; i < VS; i++) {
      sm100::mbar_init(&v_full[i], 1);
      sm100::mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      sm100::mbar_init(&s_full[i], 1);
      sm100::mbar_init(&p_full[i], kSoftmaxWarps);
    }
    sm100::mbar_init(q_full, 1);
    *gave_up = 0;
    sm100::fence_barrier_init();
  }
  if (warp == kSoftmaxWarps) {
    sm100::tmem_alloc(tmem_slot, kTmemCols);
    sm100::tmem_relinquish();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  ib::pdl_launch_dependents();   // only now: the product that follows must not take tensor memory that a CTA of this kernel still waits for
  const uint32_t tmem = *tmem_slot;
  ib::pdl_wait();

  const int h = blockIdx.x;
  const int4 tile = tiles[blockIdx.y];
  const int t0 = tile.x, rows = tile.y, pos_first = tile.z, pos_last = pos_first + rows - 1;
  const int key_lo = ib::first_visible(pos_first, window);   // of the tile's rows, the first sees the earliest key
  const int lo_last = ib::first_visible(pos_last, window);   // a tile of keys from here on is seen by every row whose position has come
  const int kt_begin = key_lo / BN, n_kt = pos_last / BN + 1 - kt_begin;
  // a wait that ran out: say so once, and from then on nobody waits (the results are void, the status says so)
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (sm100::mbar_try_wait(bar, parity) || *gave_up) return;
    if (!sm100::mbar_wait(bar, parity, wait_ns)) {
      *gave_up = 1;
      atomicOr(status, IB_ERR_WAIT_TIMEOUT);
    }
  };

  if (warp > kSoftmaxWarps) {
    // ------------------------------------------------------------ the copying warps: one for the key tiles, one for the value tiles
    if (lane == 0) {
      const bool keys = warp == kSoftmaxWarps + 1;
      sm100::prefetch_tensormap(&kv_map);
      int st = 0;
      uint32_t par = 1;   // the parity to wait for before a buffer is filled again: of s_full (keys), of v_empty (values)
      for (int j = 0; j < n_kt; j++) {
        const int row = tile.w + (kt_begin + j) * BN;
        if (keys) {
          if (j >= KS) wait(&s_full[st], par);   // the MMA warp's commit to s_full says that the scores of tile j - 2 are there and the buffer is free
          uint8_t* dst = sm + SM::oK + st * SM::kK;
          sm100::mbar_arrive_expect_tx(&k_full[st], SM::kK);
#pragma unroll
          for (int b = 0; b < DB; b++) sm100::tma_load_2d(dst + b * BN * 128, &kv_map, h * DIM + b * 64, row, &k_full[st]);
          if (RB) sm100::tma_load_2d(dst + DB * BN * 128, &r_map, 0, row, &k_full[st]);
          if (++st == KS) st = 0, par ^= 1;
        } else {
          wait(&v_empty[st], par);
          uint8_t* dst = sm + SM::oV + st * SM::kV;
          sm100::mbar_arrive_expect_tx(&v_full[st], SM::kV);
#pragma unroll
          for (int b = 0; b < VD / 64; b++) sm100::tma_load_2d(dst + b * BN * 128, &kv_map, heads * DIM + h * VD + b * 64, row, &v_full[st]);
          if (++st == VS) st = 0, par ^= 1;
        }
      }
    }
  } else if (warp == kSoftmaxWarps) {
    // ------------------------------------------------------------ the MMA warp (one lane issues)
    if (lane == 0) {
      constexpr uint32_t idesc_s = sm100::idesc_bf16_f32(BM, BN);
      constexpr uint32_t idesc_o = sm100::idesc_bf16_f32_b_mn(BM, VD);
      const uint64_t dq0 = sm100::smem_desc_sw128(q_s), dk0 = sm100::smem_desc_sw128(k_s), dv0 = sm100::smem_desc_sw128_mn(v_s, BN * 128);
      int ks = 0, vs = 0;
      uint32_t k_par = 0, v_par = 0;
      auto issue_s = [&](int j) {  // S_j = Q K_j^T into S buffer j & 1 (= K buffer ks); its commit also frees the K buffer
        wait(&k_full[ks], k_par);
        sm100::tc_fence_after();
        const uint64_t dk = dk0 + (uint64_t)(ks * (SM::kK >> 4));
#pragma unroll
        for (int kk = 0; kk < (DIM + RB) / 16; kk++) {
          const uint64_t step = (uint64_t)(2 * (kk & 3));
          sm100::mma_bf16_ss(tmem + ks * BN, dq0 + (uint64_t)(((kk >> 2) * BM * 128) >> 4) + step, dk + (uint64_t)(((kk >> 2) * BN * 128) >> 4) + step,
                             idesc_s, kk != 0);
        }
        sm100::mma_commit(&s_full[ks]);
        if (++ks == KS) ks = 0, k_par ^= 1;
      };
      wait(q_full, 0);
      issue_s(0);
      for (int j = 0; j < n_kt; j++) {
        if (j + 1 < n_kt) issue_s(j + 1);
        wait(&p_full[j & 1], (j >> 1) & 1);
        wait(&v_full[vs], v_par);
        sm100::tc_fence_after();
        const uint64_t dv = dv0 + (uint64_t)(vs * (SM::kV >> 4));
#pragma unroll
        for (int kstep = 0; kstep < BN / 16; kstep++)   // O += P_j V_j, P from tensor memory: 16 keys = 8 columns per step
          sm100::mma_bf16_ts(tmem + 2 * BN, tmem + (j & 1) * BN + kstep * 8, dv + (uint64_t)((kstep * 16 * 128) >> 4), idesc_o, (j | kstep) != 0);
        sm100::mma_commit(&v_empty[vs]);   // O has tile j, and the V buffer is free
        if (++vs == VS) vs = 0, v_par ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------ the softmax warps: thread = query row
    const int row = tid;
    const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16);
    const int my_pos = pos_first + row;
    const int my_lo = ib::first_visible(my_pos, window);
    for (int idx = tid; idx < BM * CPR; idx += kSoftmaxWarps * 32) {
      const int r = idx / CPR, cc = idx % CPR;
      const uint32_t d = q_s + blk_offset(BM, r, cc);
      if (r < rows)
        mt::cp_async16(d, q_nope + ((size_t)(t0 + r) * heads + h) * DIM + cc * 8);
      else
        mt::st_shared_zero16(d);
    }
    for (int idx = tid; idx < BM * (RB / 8); idx += kSoftmaxWarps * 32) {   // the turned part, float32 in memory
      const int r = idx / 8, cc = idx % 8;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < rows && cc < rot / 8) {
        const float* src = q_rot + ((size_t)(t0 + r) * heads + h) * q_rot_row + cc * 8;
        const float4 a = *(const float4*)src, b = *(const float4*)(src + 4);
        v = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
      }
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(q_s + DB * BM * 128 + blk_offset(BM, r, cc)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    }
    mt::cp_async_commit();
    mt::cp_async_wait<0>();
    sm100::fence_proxy_async();
    bar_sync_softmax();
    if (tid == 0) sm100::mbar_arrive(q_full);

    float m_ref = -INFINITY, l = 0.f;
    for (int j = 0; j < n_kt; j++) {
      wait(&s_full[j & 1], (j >> 1) & 1);
      sm100::tc_fence_after();
      uint32_t sr[BN];
      sm100::tmem_ld_32x32b_x32(t_lane + (j & 1) * BN, sr);
      sm100::tmem_ld_32x32b_x32(t_lane + (j & 1) * BN + 32, sr + 32);
      sm100::tmem_ld_wait();
      const int key0 = (kt_begin + j) * BN;
      const bool need_mask = key0 + BN - 1 > pos_first || key0 < lo_last;
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < BN; c++) {
          const int key = key0 + c;
          if (key > my_pos || key < my_lo) sr[c] = 0xff800000u;  // -inf
        }
      }
      // the maximum of the raw products (the positive scale is applied once below): four chains of three-input maxima
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < BN; c += 8) {
#pragma unroll
        for (int e = 0; e < 4; e++) mx[e] = max3(mx[e], __uint_as_float(sr[c + 2 * e]), __uint_as_float(sr[c + 2 * e + 1]));
      }
      const float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2e;
      // the reference maximum moves only when a row's maximum grew a lot (or at the first tile); then O,
      // which P V of the tile before may still be adding to, is rescaled once that MMA has finished
      const bool grow = tile_max > m_ref + kRescaleThreshold || (m_ref == -INFINITY && tile_max > -INFINITY);
      if (j == 0) {
        m_ref = tile_max;
      } else if (__any_sync(0xffffffffu, grow)) {
        // P V of tile t commits to v_empty[t % VS]. A parity wait tells a phase from the one before it only; here the barrier
        // of tile j - 1 has seen tile j - 1 - VS (S_j is ready, and P V of tile j - 2 was issued before it) and cannot have
        // seen tile j - 1 + VS (its P is not written yet), so the parity of tile j - 1 is not mistaken.
        wait(&v_empty[(j - 1) % VS], ((j - 1) / VS) & 1);
        sm100::tc_fence_after();
        const float m_new = grow ? fmaxf(m_ref, tile_max) : m_ref;
        const float f = m_new == -INFINITY ? 1.f : ex2(m_ref - m_new);  // 1 for rows that keep their reference, 0 when it was -inf
        l *= f;
        m_ref = m_new;
#pragma unroll 1
        for (int c0 = 0; c0 < VD; c0 += 32) {
          uint32_t o[32];
          sm100::tmem_ld_32x32b_x32(t_lane + 2 * BN + c0, o);
          sm100::tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; c++) o[c] = __float_as_uint(__uint_as_float(o[c]) * f);
          sm100::tmem_st_32x32b_x32(t_lane + 2 * BN + c0, o);
        }
        sm100::tmem_st_wait();
      }
      const float mu = m_ref == -INFINITY ? 0.f : m_ref;
      // P = 2^(S - m_ref) as bfloat16, two to a column, over the first 32 columns of S_j
      uint32_t w[BN / 2];
      const float2 sc2 = make_float2(scale_log2e, scale_log2e), nmu2 = make_float2(-mu, -mu);
      float2 la = make_float2(0.f, 0.f), lb = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < BN; c += 4) {
        const float2 a = __ffma2_rn(make_float2(__uint_as_float(sr[c]), __uint_as_float(sr[c + 1])), sc2, nmu2);
        const float2 b = __ffma2_rn(make_float2(__uint_as_float(sr[c + 2]), __uint_as_float(sr[c + 3])), sc2, nmu2);
        const float2 pa = make_float2(ex2(a.x), ex2(a.y));
        const float2 pb = make_float2(ex2(b.x), ex2(b.y));
        la = __fadd2_rn(la, pa);
        lb = __fadd2_rn(lb, pb);
        w[c / 2] = pack_bf16x2(pa.x, pa.y);
        w[c / 2 + 1] = pack_bf16x2(pb.x, pb.y);
      }
      l += (la.x + la.y) + (lb.x + lb.y);
      sm100::tmem_st_32x32b_x32(t_lane + (j & 1) * BN, w);
      sm100::tmem_st_wait();
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&p_full[j & 1]);
    }
    // ---- O / l -> out
    wait(&v_empty[(n_kt - 1) % VS], ((n_kt - 1) / VS) & 1);
    sm100::tc_fence_after();
    if (!*gave_up) {
      // the sink's weight in the units of the running sum
      if (sink_values) l += ex2(sink_values[h] * 1.4426950408889634f - m_ref);
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (row < rows) inv *= ib::tail_factor(tail, t0 + row, h);
      __nv_bfloat16* dst = out + ((size_t)(t0 + row) * heads + h) * VD;
#pragma unroll 1
      for (int c0 = 0; c0 < VD; c0 += 32) {
        uint32_t o[32];
        sm100::tmem_ld_32x32b_x32(t_lane + 2 * BN + c0, o);
        sm100::tmem_ld_wait();
        if (row < rows) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 v;
            v.x = mt::pack_bf16(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv);
            v.y = mt::pack_bf16(__uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
            v.z = mt::pack_bf16(__uint_as_float(o[c + 4]) * inv, __uint_as_float(o[c + 5]) * inv);
            v.w = mt::pack_bf16(__uint_as_float(o[c + 6]) * inv, __uint_as_float(o[c + 7]) * inv);
            *(uint4*)(dst + c0 + c) = v;
          }
        }
      }
    }
  }
  // every role is done: the MMAs have finished (the softmax threads waited for the last one), copies have landed (every tile was used)
  sm100::tc_fence_before();
  __syncthreads();
  if (warp == kSoftmaxWarps) {
    __syncwarp();
    sm100::tmem_dealloc(tmem, kTmemCols);
  }
}

int make_map(CUtensorMap* m, const void* ptr, long long rows, int cols) {   // boxes of 64 rows of 64 values
  tma_host::EncodeTiledFn fn = tma_host::encode_fn();
  IB_CHECK_ARG(fn, "latent_prefill: the driver has no cuTensorMapEncodeTiled");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {64, BN};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  IB_CHECK_ARG(r == CUDA_SUCCESS, "latent_prefill: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

bool sizes_fit(int dim, int rot, int vdim) { return (dim == 64 || dim == 128) && (vdim == 64 || vdim == 128) && rot >= 0 && rot <= kRot && rot % 8 == 0; }

}  // namespace

extern "C" int ib_latent_prefill_supports(int dim, int rot, int vdim, int rank) { return sizes_fit(dim, rot, vdim) && rank > 0 && rank % 8 == 0; }

// The cached rows of `blocks` [n_blocks][2] (segment, first position; 64 rows each) -> x [64 n_blocks, rank] and r [64 n_blocks, 64] bfloat16
// (r: the key part's rot values, zeros behind them; null with rot = 0). Rows past a segment's last position of the step are zero, and with a window those
// that its first token does not see.
extern "C" int ib_latent_gather(const IbKvView* kv, const int* blocks, int n_blocks, const int* seg_start, const int* seg_pos0, int window, int rank, int rot, void* x, void* r,
                                unsigned* status, cudaStream_t stream) {
  if (n_blocks == 0) return 0;
  IB_CHECK_ARG(kv && kv->base && kv->block_table && kv->dtype == IB_BF16 && kv->head_dim == rank + rot && kv->kv_heads == 1 && kv->page_size > 0 && kv->num_pages > 0,
               "latent_gather: a bfloat16 view of rows of %d + %d values is needed", rank, rot);
  IB_CHECK_ARG(n_blocks > 0 && rank > 0 && rank % 8 == 0 && rot >= 0 && rot <= kRot && rot % 8 == 0 && (rot == 0) == (r == nullptr), "latent_gather: bad sizes %d, %d, %d", n_blocks,
               rank, rot);
  IB_CHECK_ARG((uintptr_t)kv->base % 16 == 0 && kv->page_stride % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)r % 16 == 0, "latent_gather: rows must start on 16 bytes");
  ib::launch(latent_gather_kernel, dim3(n_blocks * (BN / kGatherRows)), 256, 0, stream, *kv, blocks, seg_start, seg_pos0, window, rank, rot, (__nv_bfloat16*)x, (__nv_bfloat16*)r, status);
  IB_CHECK_LAUNCH("latent_gather");
  return 0;
}

// q_nope [T, heads, dim] bfloat16, q_rot float32 with q_rot_row values between consecutive heads (rot of them read), keys_values [rows, heads
// dim + heads vdim] bfloat16, key_part [rows, 64] bfloat16 -> out [T, heads, vdim] bfloat16 for the tokens of `tiles` [n_tiles][4] (see the
// kernel). sink_values: float32 [heads] or null; tail: the gate (its other fields are not read).
extern "C" int ib_latent_prefill(const void* q_nope, const float* q_rot, int q_rot_row, const int* tiles, int n_tiles, const void* keys_values, const void* key_part,
                                 long long rows, int window, float scale, const float* sink_values, const IbAttnTail* tail_in, void* out, int heads, int dim, int rot,
                                 int vdim, unsigned* status, cudaStream_t stream) {
  if (n_tiles == 0) return 0;
  IB_CHECK_ARG(sizes_fit(dim, rot, vdim), "latent_prefill: head sizes %d + %d and %d (64 or 128, and a turned part of up to 64 that is a multiple of 8)", dim, rot, vdim);
  IB_CHECK_ARG(q_nope && tiles && keys_values && out && (rot == 0 || (q_rot && key_part)) && n_tiles > 0 && n_tiles <= 65535 && heads > 0 && rows > 0 && rows <= 0x7fffffffll && window >= 0,
               "latent_prefill: a null pointer or bad sizes (%d tiles, %d heads, %lld rows)", n_tiles, heads, rows);
  IB_CHECK_ARG(((uintptr_t)q_nope | (uintptr_t)q_rot | (uintptr_t)tiles | (uintptr_t)keys_values | (uintptr_t)key_part | (uintptr_t)out) % 16 == 0 && q_rot_row % 4 == 0,
               "latent_prefill: operands must be 16-byte aligned");
  IbAttnTail tail{};
  if (tail_in) tail.gate = tail_in->gate, tail.gate_parts = tail_in->gate_parts, tail.gate_row = tail_in->gate_row, tail.gate_stride = tail_in->gate_stride;
  CUtensorMap km, rm;
  if (make_map(&km, keys_values, rows, heads * (dim + vdim))) return 1;
  if (make_map(&rm, rot ? key_part : keys_values, rows, rot ? kRot : heads * (dim + vdim))) return 1;
  auto sized = [&](auto d, auto r, auto v) -> int {
    constexpr int D = decltype(d)::value, R = decltype(r)::value, V = decltype(v)::value, bytes = Smem<D, R, V>::kBytes;
    static bool configured = false;
    if (!configured) {
      cudaError_t e = cudaFuncSetAttribute(latent_prefill_kernel<D, R, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      IB_CHECK_ARG(e == cudaSuccess, "latent_prefill: cannot reserve %d bytes of shared memory: %s", bytes, cudaGetErrorString(e));
      configured = true;
    }
    ib::launch(latent_prefill_kernel<D, R, V>, dim3(heads, n_tiles), kThreads, bytes, stream, (const __nv_bfloat16*)q_nope, q_rot, q_rot_row, rot, (const int4*)tiles, km, rm, window,
               scale * 1.4426950408889634f, sink_values, tail, (__nv_bfloat16*)out, heads, ib_wait_limit_ns(), status);
    return 0;
  };
  using std::integral_constant;
  const integral_constant<int, 64> c64{};
  const integral_constant<int, 128> c128{};
  auto with_values = [&](auto d, auto r) { return vdim == 128 ? sized(d, r, c128) : sized(d, r, c64); };
  auto with_part = [&](auto d) { return rot ? with_values(d, integral_constant<int, kRot>{}) : with_values(d, integral_constant<int, 0>{}); };
  const int bad = dim == 128 ? with_part(c128) : with_part(c64);
  if (bad) return bad;
  IB_CHECK_LAUNCH("latent_prefill");
  return 0;
}
