// Causal attention of prompt portions in float32: the true 32-bit path, for heads of 64 or 128 whose keys are as large as their values.
//
// s = q . k * scale in one chain of FMAs over the head, softmax with a running maximum and sum, o = sum_j p_j v_j: what
// attention_generic_kernel computes, with its window, blocks of positions, kept first positions, cap, sink, gate and factor. There a warp
// holds one query row and every lane reads a key row of its own, so a portion reads each key once a row and the FMA units wait for it
// (259 + 518 tokens of 16 heads of 128: 1,610 us a layer). Here a CTA holds 64 rows of one head over tiles of 64 keys in shared memory, a
// thread 4 x 4 scores and 4 rows of 8 outputs: 138 us. What bounds it is shared-memory reads (8 of 16 bytes for 64 FMAs in the scores, 12
// for 128 in the sum) and, for few portions, the longest row tile's chain of key tiles; where the next tile's keys lie is looked up a tile
// ahead (looked up where it is needed, the same work took 232 us with tiles of 32 keys, 169 a tile ahead).
//
// Key tiles start at multiples of 64 positions, and a row's maximum, sum and output advance in runs of 32 keys, each operation and its place as
// in attention_generic_kernel: a position's bits are the same in a portion, alone and as a decoded token, however a prompt is cut. (One
// advance for all 64 keys of a tile took 132 us.) Reference: crates/kir/src/cuda/attention/flash_mma.rs:193 (the causal mask and window).
#include <type_traits>

#include "kv_view.cuh"

namespace {

constexpr int BQ = 64, BKEYS = 64, TILE_THREADS = 256, QTILE = 128;   // QTILE: rows of a work item (two CTAs)

struct Variant {
  int window;      // > 0: a position sees itself and the window - 1 before it; < 0: the earlier positions of its own block of -window; 0: all
  int keep;        // with a window: the first positions that are seen as well
  float scale, softcap;
  int sink;        // 1: the softmax's denominator has one more term, of score sink_values[head] (null: 0)
  const float* sink_values;
};

template <int HD>
constexpr size_t prompt_f32_smem() {
  return sizeof(float) * (BQ * (HD + 4) + BKEYS * (HD + 4) + BKEYS * HD + BQ * (BKEYS + 4)) + 2 * BKEYS * sizeof(long long);
}

template <int HD>
__global__ void __launch_bounds__(TILE_THREADS)
attention_prompt_f32_kernel(const float* __restrict__ q, IbKvView kv, const int* __restrict__ tile_seg, const int* __restrict__ tile_row0, const int* __restrict__ seg_start,
                            const int* __restrict__ seg_pos0, Variant va, IbAttnTail tail, float* __restrict__ out, int heads, unsigned* __restrict__ status) {
  constexpr int QL = HD + 4, PL = BKEYS + 4, NC = HD / 64;
  extern __shared__ __align__(16) float sm[];
  float *qs = sm, *ks = qs + BQ * QL, *vs = ks + BKEYS * QL, *ps = vs + BKEYS * HD;
  long long* offs = (long long*)(ps + BQ * PL);   // [2][BKEYS]
  ib::pdl_launch_dependents();
  ib::pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
  const int item = blockIdx.x / (QTILE / BQ), h = blockIdx.y;
  const int seg = tile_seg[item], row0 = tile_row0[item] + (blockIdx.x % (QTILE / BQ)) * BQ;
  const int first = seg_start[seg], len = seg_start[seg + 1] - first;
  if (row0 >= len) return;
  const int rows = min(BQ, len - row0), t0 = first + row0, pos0 = seg_pos0[seg] + row0, last = pos0 + rows - 1;
  const int kvhead = h / (heads / kv.kv_heads);
  const int lo0 = ib::first_visible(pos0, va.window);          // the first row sees the earliest keys
  const int keep = va.window > 0 ? va.keep : 0;

  for (int e = tid; e < BQ * (HD / 4); e += TILE_THREADS) {
    const int r = e / (HD / 4), c = e % (HD / 4) * 4;
    *(float4*)&qs[r * QL + c] = r < rows ? *(const float4*)(q + ((size_t)(t0 + r) * heads + h) * HD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // Where a tile's 64 keys lie (one lane of the first two warps each, a tile ahead of their use, so that nothing waits for the block
  // table); -1: no query of the tile sees the key, or its page is missing.
  auto look_up = [&](int k0, int buf) {
    if (tid < BKEYS) {
      const int key = k0 + tid;
      long long off = -1;
      if (key <= last && (key >= lo0 || key < keep)) {
        off = ib::kv_offset(kv, seg, key, kvhead);
        if (off < 0) atomicOr(status, IB_ERR_BAD_PAGE);
      }
      offs[buf * BKEYS + tid] = off;
    }
  };
  // A tile's keys or values to shared memory, a row a warp at a time; rows that are not read are zero.
  auto load = [&](float* dst, int stride, int buf, long long plane) {
#pragma unroll
    for (int u = 0; u < BKEYS / 8; u++) {
      const int j = u * 8 + warp;
      const long long off = offs[buf * BKEYS + j];
      const float* src = (const float*)kv.base + (off < 0 ? 0 : off + plane) + lane * (HD / 32);
      const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + j * stride + lane * (HD / 32));
      if constexpr (HD == 128) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(off < 0 ? 0 : 16) : "memory");
      else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(to), "l"(src), "r"(off < 0 ? 0 : 8) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float o[4][4 * NC], m[4], l[4];
  int lo[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    m[i] = va.sink ? (va.sink_values ? va.sink_values[h] : 0.f) : -INFINITY, l[i] = va.sink ? 1.f : 0.f;
    lo[i] = ib::first_visible(pos0 + ty + 16 * i, va.window);
#pragma unroll
    for (int c = 0; c < 4 * NC; c++) o[i][c] = 0.f;
  }
  // tiles: those that hold kept keys, then those from the first row's first key on
  const int kept_tiles = (min(keep, lo0) + BKEYS - 1) / BKEYS, from = max(kept_tiles, lo0 / BKEYS), n = kept_tiles + (last / BKEYS - from + 1);
  auto start = [&](int i) { return (i < kept_tiles ? i : from + i - kept_tiles) * BKEYS; };
  look_up(start(0), 0);
  __syncthreads();
  load(ks, QL, 0, 0);
  load(vs, HD, 0, kv.v_offset);
  for (int it = 0; it < n; it++) {
    const int k0 = start(it), buf = it & 1;
    asm volatile("cp.async.wait_group 1;" ::: "memory");   // the keys; the values may still travel
    __syncthreads();
    if (it + 1 < n) look_up(start(it + 1), buf ^ 1);
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) s[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < HD; d += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = *(const float4*)&qs[(ty + 16 * i) * QL + d];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = *(const float4*)&ks[(tx + 16 * j) * QL + d];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
    }
    const bool whole = k0 + BKEYS - 1 <= pos0 && (k0 >= ib::first_visible(last, va.window) || k0 + BKEYS <= keep);   // every row sees every key
    float corr[4][2];   // what the sums so far are multiplied by before each run of 32 keys
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int pos = pos0 + ty + 16 * i;
      float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int key = k0 + tx + 16 * j;
        s[i][j] = __fmul_rn(s[i][j], va.scale);
        if (va.softcap > 0.f) s[i][j] = __fmul_rn(va.softcap, tanhf(s[i][j] / va.softcap));
        if (offs[buf * BKEYS + tx + 16 * j] < 0 || key > pos || (key < lo[i] && key >= keep)) s[i][j] = -INFINITY;
        top[j >> 1] = fmaxf(top[j >> 1], s[i][j]);
      }
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) top[0] = fmaxf(top[0], __shfl_xor_sync(0xffffffffu, top[0], x)), top[1] = fmaxf(top[1], __shfl_xor_sync(0xffffffffu, top[1], x));
#pragma unroll
      for (int run = 0; run < 2; run++) {
        const float m_new = fmaxf(m[i], top[run]);
        corr[i][run] = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);   // (nothing seen so far: the sums are zero)
        float p[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int j = 2 * run + e;
          p[e] = s[i][j] == -INFINITY ? -0.f : expf(s[i][j] - m_new);   // (-0 marks a key that the row does not see)
          ps[(ty + 16 * i) * PL + tx + 16 * j] = p[e];
        }
        float sum = p[0] + p[1];
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        l[i] = __fmaf_rn(l[i], corr[i][run], sum), m[i] = m_new;
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // the values are here, and nobody reads the keys any more
    if (it + 1 < n) load(ks, QL, buf ^ 1, 0);
    auto add = [&](auto guard) {
#pragma unroll 1
      for (int run = 0; run < 2; run++) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int c = 0; c < 4 * NC; c++) o[i][c] = __fmul_rn(o[i][c], run ? corr[i][1] : corr[i][0]);
#pragma unroll 2
        for (int j = 32 * run; j < 32 * run + 32; j += 4) {
          float4 p[4];
#pragma unroll
          for (int i = 0; i < 4; i++) p[i] = *(const float4*)&ps[(ty + 16 * i) * PL + j];
#pragma unroll
          for (int jj = 0; jj < 4; jj++)
#pragma unroll
            for (int c = 0; c < NC; c++) {
              const float4 v = *(const float4*)&vs[(j + jj) * HD + c * 64 + tx * 4];
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const float w = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
                // (a key that a row does not see adds nothing to it, whatever its value holds)
                if (!decltype(guard)::value || __float_as_uint(w) != 0x80000000u) {
                  o[i][4 * c] = fmaf(w, v.x, o[i][4 * c]), o[i][4 * c + 1] = fmaf(w, v.y, o[i][4 * c + 1]);
                  o[i][4 * c + 2] = fmaf(w, v.z, o[i][4 * c + 2]), o[i][4 * c + 3] = fmaf(w, v.w, o[i][4 * c + 3]);
                }
              }
            }
        }
      }
    };
    if (whole) add(std::false_type{});
    else add(std::true_type{});
    __syncthreads();   // nobody reads the values any more
    if (it + 1 < n) load(vs, HD, buf ^ 1, kv.v_offset);
  }
  const int out_row = tail.out_row ? tail.out_row : heads * HD;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = ty + 16 * i;
    if (r >= rows) continue;
    float f = (l[i] > 0.f ? 1.f / l[i] : 0.f) * (tail.out_scale != 0.f ? tail.out_scale : 1.f);
    if (tail.gate) {
      const float* g = tail.gate + (size_t)(t0 + r) * tail.gate_row + h;
      float z = g[0];
      for (int p = 1; p < tail.gate_parts; p++) z += g[(size_t)p * tail.gate_stride];
      f *= 1.f / (1.f + expf(-z));
    }
    float* to = out + (size_t)(t0 + r) * out_row + (size_t)h * HD + tx * 4;
#pragma unroll
    for (int c = 0; c < NC; c++) *(float4*)(to + c * 64) = make_float4(o[i][4 * c] * f, o[i][4 * c + 1] * f, o[i][4 * c + 2] * f, o[i][4 * c + 3] * f);
  }
}

}  // namespace

// q [T, heads * HD], out rows of tail->out_row (null: heads * HD) float32; tile_seg, tile_row0 [n_tiles]: segments and first rows of the
// portions' tiles of 128 rows. window < 0: blocks of -window positions. tail: sink values, gate, factor and output row (`diff` is not read).
extern "C" int ib_attention_prompt_f32(const float* q, const IbKvView* kv, const int* tile_seg, const int* tile_row0, int n_tiles, const int* seg_start, const int* seg_pos0,
                                       int window, float scale, float* out, int heads, float softcap, int sink, const IbAttnTail* tail, int keep, unsigned* status,
                                       cudaStream_t stream) {
  if (n_tiles == 0) return 0;
  IB_CHECK_ARG(kv && kv->base && kv->block_table && kv->dtype == IB_F32 && (kv->head_dim == 64 || kv->head_dim == 128), "attention_prompt_f32: a float32 view with heads of 64 or 128 is needed");
  IB_CHECK_ARG(kv->kv_heads > 0 && heads > 0 && heads % kv->kv_heads == 0 && heads <= 65535, "attention_prompt_f32: %d query heads are not a multiple of %d kv heads", heads, kv->kv_heads);
  IB_CHECK_ARG(n_tiles > 0 && kv->page_size > 0 && kv->num_pages > 0 && kv->table_stride > 0 && keep >= 0, "attention_prompt_f32: bad sizes");
  IbAttnTail t = tail ? *tail : IbAttnTail{};
  IB_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)kv->base % 16 == 0 && kv->page_stride % 4 == 0 && kv->v_offset % 4 == 0 && t.out_row % 4 == 0 &&
                   (t.out_row == 0 || t.out_row >= heads * kv->head_dim),
               "attention_prompt_f32: rows must start on 16 bytes and hold all heads");
  IB_CHECK_ARG(sink || !t.sink_values, "attention_prompt_f32: sink values without a sink");
  const Variant va{window, keep, scale, softcap, sink, t.sink_values};
  auto go = [&](auto kernel, size_t bytes) -> int {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    IB_CHECK_ARG(e == cudaSuccess, "attention_prompt_f32: %s", cudaGetErrorString(e));
    ib::launch(kernel, dim3(n_tiles * (QTILE / BQ), heads), TILE_THREADS, bytes, stream, q, *kv, tile_seg, tile_row0, seg_start, seg_pos0, va, t, out, heads, status);
    return 0;
  };
  if (kv->head_dim == 128 ? go(attention_prompt_f32_kernel<128>, prompt_f32_smem<128>()) : go(attention_prompt_f32_kernel<64>, prompt_f32_smem<64>())) return 1;
  IB_CHECK_LAUNCH("attention_prompt_f32");
  return 0;
}
