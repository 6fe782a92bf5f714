// The large-tile matrix product on CTA pairs: out[t][n] = sum_k x[t][k] * w[n][k], bfloat16 operands,
// float32 accumulation, for prompts (256 tokens per tile; 128 with the SwiGLU epilogue).
//
// Two CTAs of a cluster (two neighbouring SMs) work on one 256 (rows of W) x 256 (tokens) tile with
// tcgen05.mma.cta_group::2: each CTA loads its own 128 rows of W and its own 128 of the 256 tokens,
// the MMA reads both halves of the token tile from the two SMs' shared memory, and each CTA's
// tensor memory receives the 128 x 256 block of its rows. Per FLOP this moves half the token-tile
// bytes of the single-CTA kernel, which is what limits that one. With two accumulators per CTA
// (gate rows and up rows of a SwiGLU feed-forward) the epilogue writes silu(gate) * up directly.
//
// Roles per CTA: warp 0 issues its TMA loads (completion is counted on the leader CTA's barrier),
// warp 1 of the leader CTA issues the MMAs for the pair and signals both CTAs' barriers, warps 2-5
// store this CTA's accumulator rows. No load uses cluster multicast. Every wait is bounded.
// The reference's equivalent is its mma.sync tile kernel (crates/kir/src/cuda/gemm/core.rs:14-155).
#include <cuda.h>

#include <cuda_bf16.h>

#include "entries.h"
#include "kv_view.cuh"
#include "sm100.cuh"
#include "tma_host.cuh"

namespace {

constexpr int BM = 128;      // rows of W per CTA (256 per pair)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int kThreads = 192;
// EPI_ADD adds where the stream lies, in L2: a read, an addition and a store by the epilogue's threads took 4 to 6 us more than a store alone, since a
// tile's last trip to memory has nothing behind it (1,003 tokens of 4,096 x 4,096: 41.0 us, 34.8 now; 2,048 of 1,024 x 2,048: 28.7 and 24.6). Such an
// addition takes numbers below 2^-126 for zero, in the stream and in the sum. With a product of 2^-100 and more neither can matter: a number below 2^-126 in the
// stream is less than half of the product's last place, and a sum of the product (a multiple of 2^-123) and a number of at least 2^-102 (a multiple of 2^-125) is
// zero or at least 2^-125. Where a thread has a smaller
// product among its 32 it adds them itself, so the sums are the bits of an IEEE addition.
// (Whole 32s are looked at and added without a test a token, which pays for the look: warm, additions of every product in L2 | now, 300 tokens of 1,024 x 3,072
// 21.7 | 21.6 us, 2,048 of 4,096 x 4,096 53.1 | 52.7, of 4,096 x 12,288 141.1 | 140.3.)
constexpr float kAddInL2 = 0x1p-100f;
constexpr int EPI_STORE = 0, EPI_SWIGLU = 1, EPI_ADD = 2;   // float32 out; bfloat16 silu(gate) * up; float32 out += product
constexpr int EPI_QKV = 3;   // the q/k/v projection finished in the epilogue: per-head norm, rotation, queries out, keys and values into the cache
constexpr int EPI_CLAMPED = 6;   // EPI_SWIGLU with clamped halves (ib::clamped_glu): the limit in QkvEpi::act_pq[0], the slope in QkvEpi::act_slope
constexpr bool epi_gated(int epi) { return epi == EPI_SWIGLU || epi == EPI_CLAMPED; }
constexpr int EPI_GLU16 = 8, EPI_CLAMPED16 = 9;   // EPI_SWIGLU and EPI_CLAMPED with gate and up rows in one accumulator, sixteen of each in turn
constexpr bool epi_16(int epi) { return epi == EPI_GLU16 || epi == EPI_CLAMPED16; }
constexpr int EPI_RELU2 = 5;   // bfloat16 max(product, 0)^2
constexpr int EPI_BF16 = 7;    // the product rounded to bfloat16, tokens and matrix rows exchanged as for EPI_QKV (a thread writes a token's row piece by piece)
constexpr int EPI_XIELU = 4;   // bfloat16 xielu(product) with the activation's two numbers (QkvEpi::act_pq)
constexpr int kQkvHead = 128;   // head size of the EPI_QKV form: a head is 128 accumulator columns
constexpr uint32_t kPeerBitMask = 0xFEFFFFFFu;   // clears the bit that tells the two CTAs of a pair apart in a shared::cluster address

constexpr int kMaxGroups = 256;   // matrices of one launch of the regrouped form (PairGroups)

// BN: tokens per tile = accumulator columns (each CTA loads half of them)
template <int MT, int BN>
struct Tile {
  static constexpr int kABytes = BM * BK * 2, kBBytes = (BN / 2) * BK * 2;
  static constexpr int kStageBytes = MT * kABytes + kBBytes;
  static constexpr int kStages = (200 * 1024) / kStageBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /* alignment slack */ + 256 /* barriers */ + 1024 /* norm scales of EPI_QKV */ +
                                    2 * (kMaxGroups + 1) * 4 /* the groups' table */;
  static constexpr int kAccSets = 512 / (MT * BN);   // accumulator sets that fit tensor memory
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {   // round to nearest even
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm100::smem_u32(slot)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc2(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// TMA tile load whose completion bytes are counted on the barrier at the same offset in the pair's leader CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          sm100::smem_u32(smem_dst)),
      "l"(m), "r"(x), "r"(y), "r"(sm100::smem_u32(bar) & kPeerBitMask)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* m, int x, int y, int z, int w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          sm100::smem_u32(smem_dst)),
      "l"(m), "r"(x), "r"(y), "r"(z), "r"(w), "r"(sm100::smem_u32(bar) & kPeerBitMask)
      : "memory");
}
__device__ __forceinline__ void mma_bf16_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(sm100::smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

// Arrive on the barrier at this offset in the pair's leader CTA (from either CTA).
__device__ __forceinline__ void arrive_on_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(sm100::smem_u32(bar) & kPeerBitMask) : "memory");
}

// Regrouped rows (routed experts): rows offsets[e] .. offsets[e + 1] of x go through matrix e, rows e * w_rows .. of w. tiles[e] is the first token tile of
// group e and tiles[n] their number; a tile never crosses a group's end (rows past it are multiplied and not stored). n = 0: one matrix for all.
// The table is read into shared memory once, after the wait for the kernels before; a tile's group is a search in it. Bound by memory at up to a few
// hundred rows a group, so the tiles go group by group: with all groups' token tiles under one block of rows after the other, 12,288 rows of 64 groups, 2,816 x
// 2,048 each, read 1.17 GB (the rows of x again and again) where 0.79 are there, 203 us; in this order 156 (5.1 TB/s; single CTAs 238), the 2,048 x
// 1,408 product behind it 115 and 92 (166). 49,152 rows: 538 and 420 (711), 302 and 240 (557; 1.2 PFLOP/s).
struct PairGroups {
  const int* offsets;
  const int* tiles;
  int n, w_rows;
};

// What the EPI_QKV epilogue works with. The product is taken the other way round there: the tokens are the
// rows of the MMA (tensor-memory lanes: a thread of the epilogue owns a token) and the rows of the fused
// [q | k | v] weight are its columns, so that a head's 128 values of a token sit in one thread: the norm is a
// sum inside the thread, the rotation partner (d + 64) is the thread's own, and a token's head goes out as one
// contiguous row. What `qk_norm_rope_kv` computes from the stored product, with the same formulas:
// per-head RMSNorm of q and k heads (scales or null), half rotation by the step's tables (or null), queries
// as bfloat16 [tokens][heads * 128], keys and values into the paged cache at the token's position.
struct QkvEpi {
  const float* q_norm_w;
  const float* k_norm_w;
  float eps;
  const float* cos_t;   // [tokens][64]
  const float* sin_t;
  const int* positions;
  const int* seg_of_token;
  __nv_bfloat16* q_out;
  IbKvView kv;
  int write_kv;
  int heads;
  const float* act_pq;   // EPI_XIELU: the activation's two numbers (p, q); EPI_CLAMPED: the limit; float32 on the device
  float act_slope;       // EPI_CLAMPED
};

// Persistent: each CTA pair walks tiles pair, pair + n_pairs, ... (token tiles vary fastest, so the
// pairs that work at the same time share rows of W). The TMA warps run ahead into the next tile
// while the accumulator of the last one is stored; with one accumulator per tile (MT = 1) tensor
// memory holds two of them, so the next tile's MMAs also run during that store.
template <int MT, int EPI, int BN>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_2cta_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_x16, void* __restrict__ out_, int T, int N,
                     int K, int token_tiles, int total_tiles, int second_off, unsigned long long wait_ns, unsigned* __restrict__ status, const QkvEpi qe, const PairGroups grp) {
  using TL = Tile<MT, BN>;
  constexpr int STAGES = TL::kStages;
  constexpr int BNH = BN / 2;
  constexpr int NBUF = TL::kAccSets >= 2 ? 2 : 1;   // accumulator sets in use
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = sm100::smem_u32(smem_raw);
  uint8_t* tiles = smem_raw + (((raw + 1023u) & ~1023u) - raw);   // the same offset in both CTAs: same kernel, same launch
  uint64_t* full = (uint64_t*)(tiles + STAGES * TL::kStageBytes);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;   // [NBUF]
  uint64_t* acc_empty = acc_full + 2;    // [NBUF], used in the leader CTA
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  float* norm_s = (float*)(tiles + STAGES * TL::kStageBytes + 256);   // EPI_QKV: q scales [128], k scales [128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();          // 0 = leader
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int nkt = (K + BK - 1) / BK;
  constexpr int kColsPerPair = epi_16(EPI) ? BM : epi_gated(EPI) ? 2 * BM : 2 * BM * MT;

  int* g_off = (int*)(tiles + STAGES * TL::kStageBytes + 256 + 1024);   // [kMaxGroups + 1]
  int* g_tile = g_off + kMaxGroups + 1;
  ib::pdl_launch_dependents();
  if (grp.n) {   // the table is the work of the kernels before
    ib::pdl_wait();
    for (int i = threadIdx.x; i <= grp.n; i += kThreads) g_off[i] = grp.offsets[i], g_tile[i] = grp.tiles[i];
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      sm100::mbar_init(&full[s], 1);
      sm100::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      sm100::mbar_init(&acc_full[b], 1);
      sm100::mbar_init(&acc_empty[b], 8);   // four epilogue warps in each of the two CTAs
    }
    sm100::fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc2(tmem_slot, 512);
    tmem_relinquish2();
  }
  if constexpr (EPI == EPI_QKV) {   // the norm scales are weights: nothing earlier in the stream writes them
    for (int i = threadIdx.x; i < 2 * kQkvHead; i += kThreads) {
      const float* src = i < kQkvHead ? qe.q_norm_w : qe.k_norm_w;
      norm_s[i] = src ? src[i % kQkvHead] : 1.f;
    }
  }
  sm100::tc_fence_before();
  __syncthreads();
  cluster_sync();   // both CTAs' barriers exist before either signals the other's
  sm100::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  const int row_blocks = (N + kColsPerPair - 1) / kColsPerPair;
  if (grp.n) total_tiles = g_tile[grp.n] * row_blocks;
  // a tile: its block of rows of W, its first token, one past its last, its group and where the group's matrix begins
  struct Place {
    int rb, t0, t_end, group, w0;
  };
  auto place = [&](int tile) {
    if (!grp.n) return Place{tile / token_tiles, tile % token_tiles * BN, T, 0, 0};
    // group by group, so that its rows of x and its matrix come from memory once: every block of the matrix with all of the group's token tiles in turn
    int lo = 0, hi = grp.n;   // the last group whose first tile is at or before this one
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (g_tile[mid] * row_blocks <= tile) lo = mid;
      else hi = mid;
    }
    const int in = tile - g_tile[lo] * row_blocks, own = g_tile[lo + 1] - g_tile[lo], rb = in / own;
    return Place{rb, g_off[lo] + (in - rb * own) * BN, g_off[lo + 1], lo, lo * grp.w_rows};
  };
  // Regrouped rows in tiles of 256: a tile is loaded and multiplied only as far as its rows go, in steps of 32 (each CTA has half of them; tmap_x brings
  // 64 rows, tmap_x16 sixteen). Otherwise the tile's full width, in one load.
  constexpr bool kTrims = MT == 1 && BN == 256;
  auto width = [&](const Place& p) { return kTrims && grp.n ? min(BN, (p.t_end - p.t0 + 31) & ~31) : BN; };
  // W rows of accumulator m of this CTA for the pair's row block rb: plain tiles stack 256-row pairs;
  // SwiGLU takes gate rows and, second_off on, up rows
  auto w_row = [&](int rb, int m) {
    const int n_pair = rb * kColsPerPair;
    return epi_gated(EPI) ? n_pair + (int)rank * BM + m * second_off : n_pair + m * 2 * BM + (int)rank * BM;
  };

  if (warp == 0) {
    if (sm100::elect_one()) {
      sm100::prefetch_tensormap(&tmap_w);
      sm100::prefetch_tensormap(&tmap_x);
      bool waited = false, ok = true;
      int it = 0;   // k-tiles sent so far, over all tiles: stage = it % STAGES
      for (int tile = pair; tile < total_tiles && ok; tile += n_pairs) {
        const Place at = place(tile);
        const int wide = width(at);
        for (int i = 0; i < nkt; i++, it++) {
          const int s = it % STAGES;
          if (!sm100::mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, wait_ns)) {
            atomicOr(status, IB_ERR_WAIT_TIMEOUT);
            ok = false;
            break;
          }
          uint8_t* a = tiles + s * TL::kStageBytes;
          if (rank == 0) sm100::mbar_arrive_expect_tx(&full[s], 2 * MT * TL::kABytes + wide * BK * 2);   // the leader counts both CTAs' bytes
          if ((EPI == EPI_QKV || EPI == EPI_BF16) && !waited) {   // there the rows are the tokens, which the kernel before wrote
            ib::pdl_wait();
            waited = true;
          }
          if constexpr (epi_16(EPI)) {   // sixteen gate rows, the sixteen up rows that go with them, four times
            const int first = (at.w0 + at.rb * kColsPerPair + (int)rank * (BM / 2)) / 16;
#pragma unroll
            for (int e = 0; e < 4; e++) tma_load_4d_pair(a + e * 32 * BK * 2, &tmap_w, i * BK, 0, first + e, 0, &full[s]);
          } else {
#pragma unroll
            for (int m = 0; m < MT; m++) tma_load_2d_pair(a + m * TL::kABytes, &tmap_w, i * BK, at.w0 + w_row(at.rb, m), &full[s]);
          }
          if (!waited) {   // the weights above do not depend on earlier kernels; x does
            ib::pdl_wait();
            waited = true;
          }
          if (kTrims && grp.n) {
            const int half = wide / 2, first = at.t0 + (int)rank * half;
            uint8_t* xs = a + MT * TL::kABytes;
            int r = 0;
            for (; r + 64 <= half; r += 64) tma_load_2d_pair(xs + r * BK * 2, &tmap_x, i * BK, first + r, &full[s]);
            for (; r < half; r += 16) tma_load_2d_pair(xs + r * BK * 2, &tmap_x16, i * BK, first + r, &full[s]);
          } else {
            tma_load_2d_pair(a + MT * TL::kABytes, &tmap_x, i * BK, at.t0 + (int)rank * BNH, &full[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && sm100::elect_one()) {
      bool ok = true;
      int it = 0, tl = 0;
      for (int tile = pair; tile < total_tiles && ok; tile += n_pairs, tl++) {
        const int b = tl % NBUF;
        if (tl >= NBUF && !sm100::mbar_wait(&acc_empty[b], ((tl / NBUF) - 1) & 1, wait_ns)) {   // the accumulator's last contents have been stored
          atomicOr(status, IB_ERR_WAIT_TIMEOUT);
          ok = false;
          break;
        }
        sm100::tc_fence_after();
        const uint32_t idesc = sm100::idesc_bf16_f32(2 * BM, kTrims && grp.n ? width(place(tile)) : BN);
        for (int i = 0; i < nkt; i++, it++) {
          const int s = it % STAGES;
          if (!sm100::mbar_wait(&full[s], (it / STAGES) & 1, wait_ns)) {
            atomicOr(status, IB_ERR_WAIT_TIMEOUT);
            ok = false;
            break;
          }
          sm100::tc_fence_after();
          const uint32_t a_addr = sm100::smem_u32(tiles + s * TL::kStageBytes);
          const uint64_t db = sm100::smem_desc_sw128(a_addr + MT * TL::kABytes);
#pragma unroll
          for (int m = 0; m < MT; m++) {
            const uint64_t da = sm100::smem_desc_sw128(a_addr + m * TL::kABytes);
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; k++) mma_bf16_ss_pair(tmem + b * MT * BN + m * BN, da + 2 * k, db + 2 * k, idesc, (i | k) != 0);
          }
          mma_commit_pair(&empty[s]);
        }
        if (ok) mma_commit_pair(&acc_full[b]);
      }
    }
  } else {
    const int q = warp & 3;
    ib::pdl_wait();
    const uint32_t lane_addr = tmem + ((uint32_t)(q * 32) << 16);
    int tl = 0;
    for (int tile = pair; tile < total_tiles; tile += n_pairs, tl++) {
      const int b = tl % NBUF;
      const Place at = place(tile);
      const int t0 = at.t0, n_pair = at.rb * kColsPerPair, t_end = at.t_end;
      bool ok = sm100::mbar_wait(&acc_full[b], (tl / NBUF) & 1, wait_ns);
      if (!ok && lane == 0) atomicOr(status, IB_ERR_WAIT_TIMEOUT);
      sm100::tc_fence_after();
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if constexpr (EPI == EPI_QKV) {
        // this thread's token, and the (up to) two heads of the tile: columns [0,128) and [128,256) of the accumulator
        const int tok = n_pair + (int)rank * BM + q * 32 + lane;
        const bool live = tok < N;
        const int kvh = qe.kv.kv_heads;
        int pos = 0, seg = 0;
        if (live && qe.write_kv) {
          pos = qe.positions[tok];
          seg = qe.seg_of_token[tok];
        }
        const float* cs = qe.cos_t ? qe.cos_t + (size_t)tok * (kQkvHead / 2) : nullptr;
        const float* sn = qe.sin_t ? qe.sin_t + (size_t)tok * (kQkvHead / 2) : nullptr;
#pragma unroll 1
        for (int hh = 0; hh < BN / kQkvHead; hh++) {
          const int j = t0 / kQkvHead + hh;   // head slot: q heads, then k heads, then v heads
          if (j * kQkvHead >= T) break;
          const bool is_q = j < qe.heads, is_k = !is_q && j < qe.heads + kvh;
          if (!is_q && !qe.write_kv) continue;
          const uint32_t col0 = lane_addr + b * MT * BN + hh * kQkvHead;
          const float* nw = is_q ? (qe.q_norm_w ? norm_s : nullptr) : (is_k && qe.k_norm_w ? norm_s + kQkvHead : nullptr);
          float inv = 1.f;
          if (nw) {   // sum of squares over the head, d rising (uniform branch: every lane of the warp reads tensor memory)
            float ss = 0.f;
#pragma unroll 1
            for (int c0 = 0; c0 < kQkvHead; c0 += 32) {
              uint32_t r[32];
              sm100::tmem_ld_32x32b_x32(col0 + c0, r);
              sm100::tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 32; c++) ss = __fmaf_rn(__uint_as_float(r[c]), __uint_as_float(r[c]), ss);
            }
            inv = rsqrtf(ss / (float)kQkvHead + qe.eps);
          }
          // destination row of this token's head
          __nv_bfloat16* dst = nullptr;
          if (live) {
            if (is_q) {
              dst = qe.q_out + ((size_t)tok * qe.heads + j) * kQkvHead;
            } else {
              const long long off = ib::kv_offset(qe.kv, seg, pos, is_k ? j - qe.heads : j - qe.heads - kvh);
              if (off < 0)
                atomicOr(status, IB_ERR_BAD_PAGE);
              else
                dst = (__nv_bfloat16*)qe.kv.base + off + (is_k ? 0 : qe.kv.v_offset);
            }
          }
          const bool turn = (is_q || is_k) && cs != nullptr;
#pragma unroll 1
          for (int c0 = 0; c0 < kQkvHead / 2; c0 += 32) {   // values d = c0 + c and their rotation partners d + 64
            uint32_t lo[32], hi[32];
            sm100::tmem_ld_32x32b_x32(col0 + c0, lo);
            sm100::tmem_ld_32x32b_x32(col0 + kQkvHead / 2 + c0, hi);
            sm100::tmem_ld_wait();
            if (dst) {
#pragma unroll
              for (int c4 = 0; c4 < 32; c4 += 4) {
                float a[4], bb[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                  a[e] = __uint_as_float(lo[c4 + e]);
                  bb[e] = __uint_as_float(hi[c4 + e]);
                  if (nw) {
                    a[e] = nw[c0 + c4 + e] * (a[e] * inv);
                    bb[e] = nw[kQkvHead / 2 + c0 + c4 + e] * (bb[e] * inv);
                  }
                }
                if (turn) {
                  const float4 c = *(const float4*)(cs + c0 + c4), sgn = *(const float4*)(sn + c0 + c4);
                  const float cv[4] = {c.x, c.y, c.z, c.w}, sv[4] = {sgn.x, sgn.y, sgn.z, sgn.w};
#pragma unroll
                  for (int e = 0; e < 4; e++) {
                    const float x0 = a[e], x1 = bb[e];
                    a[e] = __fmaf_rn(x1, -sv[e], __fmul_rn(x0, cv[e]));
                    bb[e] = __fmaf_rn(x0, sv[e], __fmul_rn(x1, cv[e]));
                  }
                }
                lo[c4 / 2] = pack_bf16x2(a[0], a[1]);
                lo[c4 / 2 + 1] = pack_bf16x2(a[2], a[3]);
                hi[c4 / 2] = pack_bf16x2(bb[0], bb[1]);
                hi[c4 / 2 + 1] = pack_bf16x2(bb[2], bb[3]);
              }
#pragma unroll
              for (int v = 0; v < 4; v++) {
                *(uint4*)(dst + c0 + 8 * v) = make_uint4(lo[4 * v], lo[4 * v + 1], lo[4 * v + 2], lo[4 * v + 3]);
                *(uint4*)(dst + kQkvHead / 2 + c0 + 8 * v) = make_uint4(hi[4 * v], hi[4 * v + 1], hi[4 * v + 2], hi[4 * v + 3]);
              }
            }
          }
        }
      } else if constexpr (EPI == EPI_BF16) {
        const int tok = n_pair + (int)rank * BM + q * 32 + lane;
        __nv_bfloat16* dst = (__nv_bfloat16*)out_ + (size_t)tok * T + t0;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
          uint32_t r[32];
          sm100::tmem_ld_32x32b_x32(lane_addr + b * MT * BN + c0, r);
          sm100::tmem_ld_wait();
          if (tok < N) {
#pragma unroll
            for (int c = 0; c < 32; c += 8)
              if (t0 + c0 + c < T)   // (T is a multiple of 8)
                *(uint4*)(dst + c0 + c) = make_uint4(pack_bf16x2(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), pack_bf16x2(__uint_as_float(r[c + 2]), __uint_as_float(r[c + 3])),
                                                     pack_bf16x2(__uint_as_float(r[c + 4]), __uint_as_float(r[c + 5])), pack_bf16x2(__uint_as_float(r[c + 6]), __uint_as_float(r[c + 7])));
          }
        }
      } else if constexpr (EPI == EPI_STORE || EPI == EPI_ADD || EPI == EPI_XIELU || EPI == EPI_RELU2) {
        float* dst = (float*)out_;
        __nv_bfloat16* dst_act = (__nv_bfloat16*)out_;
        float ap = 0.f, an = 0.f;
        if constexpr (EPI == EPI_XIELU) ap = ib::softplus(qe.act_pq[0]), an = 0.5f + ib::softplus(qe.act_pq[1]);
#pragma unroll 1
        for (int m = 0; m < MT; m++) {
          const int n = n_pair + m * 2 * BM + (int)rank * BM + q * 32 + lane;
#pragma unroll 1
          for (int c0 = 0; c0 < width(at); c0 += 32) {
            uint32_t r[32];
            sm100::tmem_ld_32x32b_x32(lane_addr + b * MT * BN + m * BN + c0, r);
            sm100::tmem_ld_wait();
            if constexpr (EPI == EPI_ADD) {
              const bool whole = t0 + c0 + 32 <= t_end;
              float least = INFINITY;
              if (whole) {
#pragma unroll
                for (int c = 0; c < 32; c += 2) least = fminf(fminf(least, fabsf(__uint_as_float(r[c]))), fabsf(__uint_as_float(r[c + 1])));
              } else {
#pragma unroll
                for (int c = 0; c < 32; c++) least = fminf(least, t0 + c0 + c < t_end ? fabsf(__uint_as_float(r[c])) : INFINITY);
              }
              // every element belongs to one thread of one launch: one addition, the same sum in every run
              auto add = [&](int t, uint32_t v) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(dst + (size_t)t * N + n), "f"(__uint_as_float(v)) : "memory"); };
              if (n < N) {
                if (least < kAddInL2) {
#pragma unroll
                  for (int c = 0; c < 32; c++)
                    if (t0 + c0 + c < t_end) dst[(size_t)(t0 + c0 + c) * N + n] += __uint_as_float(r[c]);
                } else if (whole) {
#pragma unroll
                  for (int c = 0; c < 32; c++) add(t0 + c0 + c, r[c]);
                } else {
#pragma unroll
                  for (int c = 0; c < 32; c++)
                    if (t0 + c0 + c < t_end) add(t0 + c0 + c, r[c]);
                }
              }
              __syncwarp();   // (the next load from tensor memory is the whole warp's)
            } else if (n < N) {
#pragma unroll
              for (int c = 0; c < 32; c++) {
                const int t = t0 + c0 + c;
                if (t < t_end) {
                  if constexpr (EPI == EPI_XIELU)
                    dst_act[(size_t)t * N + n] = __float2bfloat16_rn(ib::xielu(__uint_as_float(r[c]), ap, an));
                  else if constexpr (EPI == EPI_RELU2)
                    dst_act[(size_t)t * N + n] = __float2bfloat16_rn(ib::relu2(__uint_as_float(r[c])));
                  else
                    dst[(size_t)t * N + n] = __uint_as_float(r[c]);
                }
              }
            }
          }
        }
      } else if constexpr (epi_16(EPI)) {
        // Lane l holds gate row l or, from 16 on, up row l - 16 of the warp's sixteen: one exchange gives each half of the lanes both numbers of every
        // second token. No branch stands between the numbers: a thread's sixteen run side by side.
        const float limit = EPI == EPI_CLAMPED16 ? qe.act_pq[at.group] : 0.f;
        const int n = n_pair + (int)rank * (BM / 2) + q * 16 + (lane & 15), wide = width(at), up = lane >> 4;
        __nv_bfloat16* dst = (__nv_bfloat16*)out_;
#pragma unroll 1
        for (int c0 = 0; c0 < wide; c0 += 32) {
          uint32_t r[32];
          sm100::tmem_ld_32x32b_x32(lane_addr + b * BN + c0, r);
          sm100::tmem_ld_wait();
          __nv_bfloat16 v[16];
#pragma unroll
          for (int c = 0; c < 16; c++) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? r[2 * c] : r[2 * c + 1], 16);
            const float gv = __uint_as_float(up ? got : r[2 * c]), uv = __uint_as_float(up ? r[2 * c + 1] : got);
            if constexpr (EPI == EPI_CLAMPED16) v[c] = __float2bfloat16_rn(ib::clamped_glu<true>(gv, uv, limit, qe.act_slope));
            else v[c] = __float2bfloat16_rn(__fdividef(gv, 1.f + __expf(-gv)) * uv);
          }
          if (n < N) {
#pragma unroll
            for (int c = 0; c < 16; c++) {
              const int t = t0 + c0 + 2 * c + up;
              if (t < t_end) dst[(size_t)t * N + n] = v[c];
            }
          }
        }
      } else {
        __nv_bfloat16* dst = (__nv_bfloat16*)out_;
        const float limit = EPI == EPI_CLAMPED ? qe.act_pq[at.group] : 0.f;
        const int n = n_pair + (int)rank * BM + q * 32 + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
          uint32_t g[32], u[32];
          sm100::tmem_ld_32x32b_x32(lane_addr + b * MT * BN + c0, g);
          sm100::tmem_ld_32x32b_x32(lane_addr + b * MT * BN + BN + c0, u);
          sm100::tmem_ld_wait();
          // All 32 are made before the first is stored: a branch a token kept them from running side by side (2,048 tokens of 12,288 x 4,096
          // 259 -> 253 us, of 3,072 x 1,024 40 -> 32; 1,003 tokens 148.5 -> 144.4 and 30 -> 26).
#pragma unroll
          for (int c = 0; c < 32; c++) {
            const float gv = __uint_as_float(g[c]), uv = __uint_as_float(u[c]);
            if constexpr (EPI == EPI_CLAMPED) g[c] = __float_as_uint(ib::clamped_glu<true>(gv, uv, limit, qe.act_slope));
            else g[c] = __float_as_uint(__fdividef(gv, 1.f + __expf(-gv)) * uv);
          }
          if (n < N) {
#pragma unroll
            for (int c = 0; c < 32; c++) {
              const int t = t0 + c0 + c;
              if (t < t_end) dst[(size_t)t * N + n] = __float2bfloat16_rn(__uint_as_float(g[c]));
            }
          }
        }
      }
      // this warp has read its part of the accumulator: tell the leader's MMA warp
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_on_leader(&acc_empty[b]);
    }
  }
  sm100::tc_fence_before();
  __syncthreads();
  cluster_sync();   // neither CTA leaves (or frees tensor memory) while its partner may still signal it
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc2(tmem, 512);
  }
}

int make_tmap(CUtensorMap* m, const void* ptr, int rows, int K, int box_rows) {
  tma_host::EncodeTiledFn fn = tma_host::encode_fn();
  IB_CHECK_ARG(fn, "gemm_tcgen05_2cta: the driver has no cuTensorMapEncodeTiled");
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  IB_CHECK_ARG(r == CUDA_SUCCESS, "gemm_tcgen05_2cta: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

// The [E][2 I][K] gate and up rows as (k, sixteen rows, sixteens, gate or up): a box brings sixteen gate rows and the up rows that go with them. The last
// sixteens, whose up rows would lie behind the buffer, are outside.
int make_tmap_glu16(CUtensorMap* m, const void* ptr, int rows, int I, int K) {
  tma_host::EncodeTiledFn fn = tma_host::encode_fn();
  IB_CHECK_ARG(fn, "gemm_tcgen05_2cta: the driver has no cuTensorMapEncodeTiled");
  IB_CHECK_ARG(I % 16 == 0 && rows % (2 * I) == 0, "gemm_tcgen05_2cta: %d gate rows are no whole sixteens", I);
  const cuuint64_t row = (cuuint64_t)K * 2;
  cuuint64_t dims[4] = {(cuuint64_t)K, 16, (cuuint64_t)(rows - I) / 16, 2};
  cuuint64_t strides[3] = {row, row * 16, row * I};
  cuuint32_t box[4] = {(cuuint32_t)BK, 16, 1, 2};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  IB_CHECK_ARG(r == CUDA_SUCCESS, "gemm_tcgen05_2cta: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

template <int MT, int EPI, int BN>
int launch(const void* x, const void* w, void* out, int T, int N, int K, int w_rows, int second_off, unsigned* status, cudaStream_t stream,
           const QkvEpi& qe = QkvEpi{}, const PairGroups& grp = PairGroups{}) {
  using TL = Tile<MT, BN>;
  IB_CHECK_ARG(T > 0 && N > 0 && K > 0 && K % 8 == 0, "gemm_tcgen05_2cta: bad sizes T=%d N=%d K=%d (K must be a multiple of 8)", T, N, K);
  IB_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0, "gemm_tcgen05_2cta: operands must be 16-byte aligned");
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_2cta_kernel<MT, EPI, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, TL::kSmemBytes);
    IB_CHECK_ARG(e == cudaSuccess, "gemm_tcgen05_2cta: cannot reserve %d bytes of shared memory: %s", TL::kSmemBytes, cudaGetErrorString(e));
    configured = true;
  }
  CUtensorMap tw, tx, tx16;
  const bool trims = MT == 1 && BN == 256 && grp.n;
  if (epi_16(EPI) ? make_tmap_glu16(&tw, w, w_rows, N, K) : make_tmap(&tw, w, w_rows, K, BM)) return 1;
  if (make_tmap(&tx, x, T, K, trims ? 64 : BN / 2)) return 1;
  if (!trims) tx16 = tx;
  else if (make_tmap(&tx16, x, T, K, 16)) return 1;
  const int cols_per_pair = epi_16(EPI) ? BM : epi_gated(EPI) ? 2 * BM : 2 * BM * MT;
  const int token_tiles = grp.n ? T / BN + grp.n : (T + BN - 1) / BN, row_blocks = (N + cols_per_pair - 1) / cols_per_pair;
  const int total_tiles = token_tiles * row_blocks;
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  const int n_pairs = total_tiles < sm_count / 2 ? total_tiles : sm_count / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * n_pairs);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = TL::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = ib_pdl_enabled();
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_2cta_kernel<MT, EPI, BN>, tw, tx, tx16, out, T, N, K, token_tiles, total_tiles, second_off, ib_wait_limit_ns(), status, qe, grp);
  IB_CHECK_ARG(e == cudaSuccess, "gemm_tcgen05_2cta: launch failed: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace

// x [T, K], w [N, K] bfloat16 -> out [T, N] float32, 256 x 256 tiles on CTA pairs (meant for T >= 256).
extern "C" int ib_gemm_tcgen05_2cta(const void* x, const void* w, float* out, int T, int N, int K, unsigned* status, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  return launch<1, EPI_STORE, 256>(x, w, out, T, N, K, N, 0, status, stream);
}

// The same product added to what out [T, N] float32 holds (the residual stream), in place.
extern "C" int ib_gemm_tcgen05_2cta_add(const void* x, const void* w, float* out, int T, int N, int K, unsigned* status, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  return launch<1, EPI_ADD, 256>(x, w, out, T, N, K, N, 0, status, stream);
}

// x [T, K], w [N, K] bfloat16 -> out [T, N] bfloat16: the product, rounded once (N a multiple of 8). The tokens are the rows of the MMA, so that
// a thread of the epilogue owns a token and stores 16 bytes at a time.
extern "C" int ib_gemm_bf16_2cta(const void* x, const void* w, void* out, int T, int N, int K, unsigned* status, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  IB_CHECK_ARG(N % 8 == 0 && ((uintptr_t)out & 15) == 0, "gemm_bf16_2cta: rows of %d values must start on 16 bytes", N);
  return launch<1, EPI_BF16, 256>(w, x, out, N, T, K, T, 0, status, stream);
}

// x [T, K], w [N, K] bfloat16 -> act [T, N] bfloat16 = max(x w^T, 0)^2, with the activation in the epilogue.
extern "C" int ib_gemm_relu2_tcgen05_2cta(const void* x, const void* w, void* act, int T, int N, int K, unsigned* status, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  return launch<1, EPI_RELU2, 256>(x, w, act, T, N, K, N, 0, status, stream);
}

// x [T, K], w [N, K] bfloat16 -> act [T, N] bfloat16 = xielu(x w^T) with the two numbers pq (float32, on the device): the product of
// ib_gemm_tcgen05_2cta with the activation in its epilogue.
extern "C" int ib_gemm_xielu_tcgen05_2cta(const void* x, const void* w, void* act, int T, int N, int K, const float* pq, unsigned* status, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  IB_CHECK_ARG(pq, "gemm_xielu_tcgen05_2cta: the activation's two numbers are missing");
  QkvEpi qe{};
  qe.act_pq = pq;
  return launch<1, EPI_XIELU, 256>(x, w, act, T, N, K, N, 0, status, stream, qe);
}

// w [2*I, K] = gate rows then up rows -> act [T, I] bfloat16 = silu(x gate^T) * (x up^T), on CTA pairs.
// limit: null, or one float32 on the device: clamped halves instead, with the sigmoid's slope.
extern "C" int ib_gemm_swiglu_tcgen05_2cta(const void* x, const void* w, void* act, int T, int I, int K, const float* limit, float slope, unsigned* status, cudaStream_t stream) {
  if (T == 0 || I == 0) return 0;
  if (limit) {
    QkvEpi qe{};
    qe.act_pq = limit, qe.act_slope = slope;
    return launch<2, EPI_CLAMPED, 128>(x, w, act, T, I, K, 2 * I, I, status, stream, qe);
  }
  return launch<2, EPI_SWIGLU, 128>(x, w, act, T, I, K, 2 * I, I, status, stream);
}

// The products of regrouped rows on CTA pairs, tiles of `tile` rows, 128 or 256 (the table: ib_moe_sort with tile_rows = tile): x [R, K] bfloat16 and w [E, N or 2 I, K];
// offsets, tiles [E + 1] (see PairGroups). Store: out [R, N] float32; act 2: [R, N] bfloat16 max(product, 0)^2.
extern "C" int ib_gemm_grouped_2cta(const void* x, const void* w, void* out, int R, int N, int K, const int* offsets, const int* tiles, int E, int tile, int act, unsigned* status,
                                    cudaStream_t stream) {
  if (R == 0 || N == 0) return 0;
  IB_CHECK_ARG(E > 0 && E <= kMaxGroups && offsets && tiles && (act == 0 || act == 2), "gemm_grouped_2cta: %d groups (up to %d) or activation %d", E, kMaxGroups, act);
  IB_CHECK_ARG(tile == 128 || tile == 256, "gemm_grouped_2cta: tiles of %d rows (128 and 256 are built)", tile);
  IB_CHECK_ARG((long long)E * N < (1ll << 31), "gemm_grouped_2cta: %d matrices of %d rows", E, N);
  const PairGroups grp{offsets, tiles, E, N};
  if (tile == 256 && act == 2) return launch<1, EPI_RELU2, 256>(x, w, out, R, N, K, E * N, 0, status, stream, QkvEpi{}, grp);
  if (tile == 256) return launch<1, EPI_STORE, 256>(x, w, out, R, N, K, E * N, 0, status, stream, QkvEpi{}, grp);
  if (act == 2) return launch<2, EPI_RELU2, 128>(x, w, out, R, N, K, E * N, BM * 2, status, stream, QkvEpi{}, grp);
  return launch<2, EPI_STORE, 128>(x, w, out, R, N, K, E * N, BM * 2, status, stream, QkvEpi{}, grp);
}

// act [R, I] bfloat16 = silu(gate) * up per group, w [E, 2 I, K] = every group's gate rows then its up rows; limits: null, or float32 [E]: clamped halves.
extern "C" int ib_gemm_grouped_swiglu_2cta(const void* x, const void* w, void* act, int R, int I, int K, const int* offsets, const int* tiles, int E, int tile, const float* limits,
                                           float slope, unsigned* status, cudaStream_t stream) {
  if (R == 0 || I == 0) return 0;
  IB_CHECK_ARG(E > 0 && E <= kMaxGroups && offsets && tiles, "gemm_grouped_swiglu_2cta: %d groups (up to %d)", E, kMaxGroups);
  IB_CHECK_ARG(tile == 128 || (tile == 256 && I % 16 == 0), "gemm_grouped_swiglu_2cta: tiles of %d rows with %d gate rows (128, or 256 with a multiple of 16)", tile, I);
  IB_CHECK_ARG((long long)E * 2 * I < (1ll << 31), "gemm_grouped_swiglu_2cta: %d matrices of %d rows", E, 2 * I);
  const PairGroups grp{offsets, tiles, E, 2 * I};
  QkvEpi qe{};
  qe.act_pq = limits, qe.act_slope = slope;
  if (tile == 256 && limits) return launch<1, EPI_CLAMPED16, 256>(x, w, act, R, I, K, E * 2 * I, I, status, stream, qe, grp);
  if (tile == 256) return launch<1, EPI_GLU16, 256>(x, w, act, R, I, K, E * 2 * I, I, status, stream, qe, grp);
  if (limits) return launch<2, EPI_CLAMPED, 128>(x, w, act, R, I, K, E * 2 * I, I, status, stream, qe, grp);
  return launch<2, EPI_SWIGLU, 128>(x, w, act, R, I, K, E * 2 * I, I, status, stream, qe, grp);
}

// The q/k/v projection with its epilogue: x [T, K] bfloat16 and w [(heads + 2 kv_heads) * 128, K] bfloat16 (q rows, k rows, v rows)
// -> q_out [T, heads * 128] bfloat16 normed and turned, and (write_kv) keys and values of each token at its position
// in the paged cache; what ib_gemm_tcgen05_2cta followed by ib_qk_norm_rope_kv gives, without the float32 product
// in memory between them. Head size 128, a bfloat16 cache, the whole head turned (cos_t, sin_t [T, 64]) or none of it.
extern "C" int ib_gemm_qkv_tcgen05_2cta(const void* x, const void* w, int T, int K, const float* q_norm_w, const float* k_norm_w, float eps,
                                        const float* cos_t, const float* sin_t, const int* positions, const int* seg_of_token, void* q_out,
                                        const IbKvView* kv, int write_kv, int heads, unsigned* status, cudaStream_t stream) {
  if (T == 0) return 0;
  IB_CHECK_ARG(kv && q_out && positions && seg_of_token, "gemm_qkv_tcgen05_2cta: a null pointer");
  IB_CHECK_ARG(kv->head_dim == kQkvHead, "gemm_qkv_tcgen05_2cta: head size %d (this form has 128)", kv->head_dim);
  IB_CHECK_ARG(!write_kv || (kv->base && kv->block_table && kv->dtype == IB_BF16), "gemm_qkv_tcgen05_2cta: the cache must be bfloat16");
  IB_CHECK_ARG(heads > 0 && kv->kv_heads > 0, "gemm_qkv_tcgen05_2cta: %d heads, %d kv heads", heads, kv->kv_heads);
  IB_CHECK_ARG((cos_t == nullptr) == (sin_t == nullptr), "gemm_qkv_tcgen05_2cta: one rotation table without the other");
  IB_CHECK_ARG(((uintptr_t)q_out & 15) == 0 && ((uintptr_t)kv->base & 15) == 0 && ((uintptr_t)cos_t & 15) == 0 && ((uintptr_t)sin_t & 15) == 0,
               "gemm_qkv_tcgen05_2cta: outputs and tables must be 16-byte aligned");
  QkvEpi qe = {q_norm_w, k_norm_w, eps, cos_t, sin_t, positions, seg_of_token, (__nv_bfloat16*)q_out, *kv, write_kv, heads};
  const int N = (heads + 2 * kv->kv_heads) * kQkvHead;
  // the other way round: the tokens are the rows of the product, the weight's rows its columns
  return launch<1, EPI_QKV, 256>(w, x, nullptr, N, T, K, T, 0, status, stream, qe);
}
