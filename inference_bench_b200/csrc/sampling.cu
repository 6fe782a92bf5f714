// Next-token choice on the device, one thread-block cluster per logits row.
//
// Temperature 0: argmax, the lowest index winning ties. Otherwise Gumbel-max over the candidates
// that survive top-k, top-p and min-p, on v = logit / T: token = argmax_i (v_i + g_i),
// g_i = -ln(-ln u_i), u_i from an integer hash of (seed, step, i). Same semantics and the same
// hash as the reference's sample_rows (crates/kir/tests/golden/prims/prims_sm120.cu:34-39,
// 51-163, 208-250); the thresholds here are found digit by digit of the value's bits, four at a
// time, by count (top-k) or by mass (top-p). Counts are exact; mass is summed in an order that follows
// from the vocabulary alone. So a row's token depends neither on thread timing nor on the rows beside it.
#include "common.cuh"

namespace {

constexpr int kThreads = 512, kWarpsOfRow = kThreads / 32;
constexpr int kCtasOfSm = 3;         // CTAs that may share an SM
constexpr int kMaxParts = 8;         // of a row: its vocabulary is cut into 1, 2, 4 or 8 parts, which its cluster's CTAs share
constexpr int kPartValues = 4096;    // the least number of values in a part

struct RowParams {  // six 32-bit words per row, as the reference packs them (crates/specrt/src/runtime/step.rs:76-85)
  float inv_temp;   // 0 = greedy
  unsigned seed;
  unsigned step;
  int top_k;    // 0 = off
  float top_p;  // 1 = off
  float min_p;  // 0 = off
};

__device__ __forceinline__ float gumbel(unsigned seed, unsigned step, unsigned i) {
  unsigned x = seed * 747796405u + step * 2891336453u + i * 2246822519u + 1u;
  x ^= x >> 16;
  x *= 2246822507u;
  x ^= x >> 13;
  x *= 3266489909u;
  x ^= x >> 16;
  float u = ((float)(x >> 8) + 0.5f) / 16777216.0f;
  return -logf(-logf(u));
}

// Monotone map float -> unsigned (larger float, larger key), zeros of both signs alike.
__device__ __forceinline__ unsigned order_key(float v) {
  unsigned b = __float_as_uint(v + 0.f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float order_value(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

__device__ __forceinline__ void better(float& bv, int& bi, float ov, int oi) {  // the lowest index wins ties
  if (ov > bv || (ov == bv && oi < bi)) {
    bv = ov;
    bi = oi;
  }
}

// What the CTAs of a row's cluster exchange: each leaves its part, and after one cluster barrier every one reads all of them, in the order of the ranks.
// Two places are used in turn: a CTA writes a place again only behind the barrier after the one that its readers passed.
struct RowShared {
  float warp_part[kMaxParts][kWarpsOfRow][16];   // (of the CTA's own parts)
  int warp_index[kWarpsOfRow];
  float part[2][kMaxParts][16];
  float part_index[2];   // (bits of whole numbers)
  float total[16];
  float bins[16][kThreads];   // a thread's sixteen sums of a pass
};

// Of the row a CTA has `own` parts in a row, of `share` values each (the row's last ones may have fewer, or none). p = own: where its values end.
__device__ __forceinline__ int part_begin(int V, int share, int own, int p) { return min(V, ((int)blockIdx.x * own + p) * share); }

// f(i, value) for the values begin .. end - 1 of the row: four neighbours a thread, in one access where the row starts on 16 bytes, U such fours requested
// together. Which thread gets which values in which order does not depend on where the row starts.
template <int U, class F>
__device__ __forceinline__ void each_value(const float* __restrict__ row, int begin, int end, F f) {
  const int quads = (end - begin) / 4;
  const float* src = row + begin;
  const bool wide = ((uintptr_t)src & 15) == 0;
  for (int q0 = threadIdx.x; q0 < quads; q0 += U * kThreads) {
    float4 v[U];
    if (wide) {
#pragma unroll
      for (int u = 0; u < U; u++)
        if (q0 + u * kThreads < quads) v[u] = ((const float4*)src)[q0 + u * kThreads];
    } else {
#pragma unroll
      for (int u = 0; u < U; u++) {
        const float* at = src + 4 * (q0 + u * kThreads);
        if (q0 + u * kThreads < quads) v[u] = make_float4(at[0], at[1], at[2], at[3]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = begin + 4 * (q0 + u * kThreads);
      if (q0 + u * kThreads < quads) f(i, v[u].x), f(i + 1, v[u].y), f(i + 2, v[u].z), f(i + 3, v[u].w);
    }
  }
  const int i = begin + 4 * quads + threadIdx.x;
  if (i < end) f(i, row[i]);
}

// A warp's sums of sixteen values of every thread, to its place for the CTA's part p.
__device__ __forceinline__ void warp_sums(float (&s)[16], RowShared& sh, int p) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 1; o >>= 1) {   // lanes halve the values between them: lane (l4 l3 l2 l1 l0) ends with value l4 l3 l2 l1
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o / 2; i++) {
      const float give = up ? s[i] : s[i + o / 2], keep = up ? s[i + o / 2] : s[i];
      s[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
  if (!(lane & 1)) sh.warp_part[p][warp][lane >> 1] = s[0];
}

// The sums over the row of what the warps left for `own` parts a CTA, added part by part, in sh.total for all threads; `turn` is 0 and 1 from call to call.
__device__ __forceinline__ void row_sums(RowShared& sh, int own, int turn) {
  __syncthreads();
  const int j = threadIdx.x & 15, p = threadIdx.x >> 4, ctas = gridDim.x;
  if (p < own) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kWarpsOfRow; w++) t += sh.warp_part[p][w][j];
    sh.part[turn][p][j] = t;
  }
  if (ctas > 1) {
    __syncwarp();
    ib::cluster_sync();
  } else if (own > 1) {
    __syncthreads();
  }
  if (threadIdx.x < 16) {   // (all parts are requested before the first is added; own is a power of two)
    const int parts = ctas * own, lg = 31 - __clz(own);
    float v[kMaxParts], t = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxParts; i++)
      if (i < parts) v[i] = ctas > 1 ? ib::peer_ld(&sh.part[turn][i & (own - 1)][j], i >> lg) : sh.part[turn][i][j];
#pragma unroll
    for (int i = 0; i < kMaxParts; i++)
      if (i < parts) t += v[i];
    sh.total[j] = t;
  }
  __syncthreads();
}

// The best (value, index) of the cluster, in the first warp of every CTA.
__device__ __forceinline__ void cluster_best(float& bv, int& bi, RowShared& sh, int ctas, int turn) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) better(bv, bi, __shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o));
  if (lane == 0) sh.warp_part[0][warp][0] = bv, sh.warp_index[warp] = bi;
  __syncthreads();
  if (warp == 0) {
    bv = lane < kWarpsOfRow ? sh.warp_part[0][lane][0] : -INFINITY;
    bi = lane < kWarpsOfRow ? sh.warp_index[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) better(bv, bi, __shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o));
    if (lane == 0) sh.part[turn][0][0] = bv, sh.part_index[turn] = __int_as_float(bi);
  }
  __syncwarp();
  if (ctas == 1) return;
  ib::cluster_sync();
  if (warp == 0)
    for (int c = 0; c < ctas; c++) better(bv, bi, ib::peer_ld(&sh.part[turn][0][0], c), __float_as_int(ib::peer_ld(&sh.part_index[turn], c)));
}

// The largest key t of lo .. hi - 1 with at least `target` of weight in the values of key t and above (lo when there is none), the weight being a count or
// the mass e^(v - m). A pass looks at the sixteen parts of the interval that is left; what lies above it is known from the passes before.
// FRACTION: target is a share of the weight of lo and above. WHOLE: the CTA's values are summed as one part (counts are exact in any order).
template <bool MASS, bool FRACTION, bool WHOLE>
__device__ __forceinline__ unsigned search(const float* row, int V, int share, int all, float inv_temp, float m, unsigned lo, unsigned long long hi, float target, RowShared& sh, int& turn) {
  float above = 0.f;   // the weight of hi and above
  bool first = true;
  while (lo + 1ull < hi) {
    const int bits = 64 - __clzll((long long)(hi - lo - 1)), shift = bits > 4 ? bits - 4 : 0;
    const int own = WHOLE ? 1 : all;
#pragma unroll 1
    for (int p = 0; p < own; p++) {
#pragma unroll
      for (int j = 0; j < 16; j++) sh.bins[j][threadIdx.x] = 0.f;
      each_value<2>(row, part_begin(V, share, all, p), part_begin(V, share, all, WHOLE ? all : p + 1), [&](int, float x) {
        const float v = x * inv_temp;
        const unsigned key = order_key(v);
        if (key < lo || key >= hi) return;
        sh.bins[(key - lo) >> shift][threadIdx.x] += MASS ? expf(v - m) : 1.f;
      });
      float s[16];   // of sixteenth j of the interval and above
#pragma unroll
      for (int j = 15; j >= 0; j--) s[j] = sh.bins[j][threadIdx.x] + (j < 15 ? s[j + 1] : 0.f);
      warp_sums(s, sh, p);
    }
    row_sums(sh, own, turn);
    turn ^= 1;
    if (FRACTION && first) target *= sh.total[0];
    first = false;
    int best = 0;
    float next = above;
#pragma unroll
    for (int j = 1; j < 16; j++)
      if (above + sh.total[j] >= target) best = j;
    if (best < 15) next = above + sh.total[best + 1];
    hi = min(hi, (unsigned long long)lo + ((unsigned long long)(best + 1) << shift));
    lo += (unsigned)best << shift;
    above = next;
  }
  return lo;
}

// One row. All of a greedy row is one pass over its logits; a threshold is eight passes of four bits each over logits that stay in L2, and what a pass costs
// is its reductions, not its reads. A row of 151,936 took 929 us with top-p, 222 with top-k and 885 with both and min-p, by one CTA and a pass for every step of a
// bisection, and a greedy one 17 us in three kernels: 51, 45, 71 and 12 us so (64 rows: 1,000, 240, 941 and 36 against 129, 92, 166 and 18; caches cold). Where a
// CTA has several parts of a row their masses are summed one after the other: 64 rows with top-p took 113 us in an order that followed the number of CTAs, and the
// token of a row could then change with the number of rows.
// With `status` the step's status word is copied to tokens[rows], so the host gets it in the transfer that brings the tokens.
// PER_SM: how many CTAs share an SM, by the registers a thread may have.
template <int PER_SM>
__global__ void __launch_bounds__(kThreads, PER_SM) sample_kernel(const float* __restrict__ logits, int V, int share, int own, const RowParams* __restrict__ params,
                                                                  int* __restrict__ tokens, const unsigned* __restrict__ status) {
  __shared__ RowShared sh;
  ib::pdl_launch_dependents();
  ib::pdl_wait();
  const int r = blockIdx.y, ctas = gridDim.x, rank = blockIdx.x;
  const float* row = logits + (size_t)r * V;
  __shared__ RowParams p;   // (six registers a thread less through all passes)
  if (threadIdx.x < sizeof(RowParams) / 4) ((int*)&p)[threadIdx.x] = ((const int*)(params + r))[threadIdx.x];
  __syncthreads();
  const bool sampling = p.inv_temp > 0.f;
  const int begin = part_begin(V, share, own, 0), end = part_begin(V, share, own, own);
  int turn = 0;
  float thr = -INFINITY;
  const bool use_k = p.top_k > 0 && p.top_k < V, use_p = p.top_p < 1.f, use_m = p.min_p > 0.f;
  if (sampling && (use_k || use_p || use_m)) {   // (the same for all CTAs of the row)
    float m = -INFINITY;
    if (use_p || use_m) {
      int none = 0;
      each_value<4>(row, begin, end, [&](int, float x) { m = fmaxf(m, x * p.inv_temp); });
      cluster_best(m, none, sh, ctas, turn);
      turn ^= 1;
      if (threadIdx.x == 0) sh.total[0] = m;
      __syncthreads();
      m = sh.total[0];
    }
    if (use_k) thr = order_value(search<false, false, true>(row, V, share, own, p.inv_temp, m, 0u, 1ull << 32, (float)p.top_k, sh, turn));
    if (use_p) {   // the largest threshold whose candidates (also above the top-k threshold) hold mass >= top_p * total
      const float lo = thr > -INFINITY ? thr : m - 88.f;
      const unsigned key_lo = order_key(lo);
      const unsigned long long key_hi = order_key(nextafterf(m, INFINITY));
      const float part = fmaxf(p.top_p, 1e-9f);
      thr = fmaxf(thr, order_value(own == 1 ? search<true, true, true>(row, V, share, own, p.inv_temp, m, key_lo, key_hi, part, sh, turn)
                                            : search<true, true, false>(row, V, share, own, p.inv_temp, m, key_lo, key_hi, part, sh, turn)));
    }
    if (use_m) thr = fmaxf(thr, m + logf(p.min_p));
  }
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  if (sampling)
    each_value<4>(row, begin, end, [&](int i, float x) {
      const float v = x * p.inv_temp;
      if (!(v < thr)) better(bv, bi, v + gumbel(p.seed, p.step, (unsigned)i), i);
    });
  else
    each_value<4>(row, begin, end, [&](int i, float x) { better(bv, bi, x, i); });
  cluster_best(bv, bi, sh, ctas, turn);
  if (rank == 0 && threadIdx.x == 0) {
    tokens[r] = bi == 0x7fffffff ? 0 : bi;
    if (status && r == 0) tokens[gridDim.y] = (int)*status;
  }
  if (ctas > 1) {   // nobody leaves while its part may still be read
    __syncwarp();
    ib::cluster_sync();
  }
}

// After a decode step: feed every row's sampled token back as its next input, move its position on
// by one, count its sampling step, and log the token. With this at the end of a captured decode
// step the graph can be replayed many times with no host work in between; the host reads the log
// afterwards (the reference's argmax_advance does the same for one row:
// crates/kir/tests/golden/prims/prims_sm120.cu:252-294).
// host: null, or pinned memory of rows + 1 words that receives the tokens and what stands behind them in `sampled` (the status word's value): a step that
// the host waits for needs no copy behind it.
__global__ void advance_rows_kernel(const int* __restrict__ sampled, int* __restrict__ token_in, int* __restrict__ positions,
                                    int* __restrict__ pos0, RowParams* __restrict__ params, int* __restrict__ history, int* __restrict__ count,
                                    int rows, int history_len, int* __restrict__ host) {
  // No early launch of the kernels that follow: the attention kernels of the next step read
  // `positions` before their own dependency wait, so nothing of the next step may start before
  // the rows are written. The next kernel starts when this one has finished.
  ib::pdl_wait();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int c = count[0];
  if (i < rows) {
    int tok = sampled[i];
    token_in[i] = tok;
    positions[i] += 1;
    pos0[i] += 1;
    params[i].step += 1;
    if (c < history_len) history[(size_t)c * rows + i] = tok;
    if (host) host[i] = tok;
  }
  if (host && i == 0) host[rows] = sampled[rows];
  __syncthreads();
  if (i == 0) count[0] = c + 1;
}

// A captured step's inputs from pinned host memory: the host writes them, the step's first kernel fetches them. Bound by one trip over the bus; a copy in
// front of the step is another call (6 us on the host for 1 row, 16 for 64) and 8 us on the device. With the tokens written back by advance_rows a step
// that the host waits for takes 441 -> 427 us (1 row of twelve 0.6B layers), 569 -> 552 (8 rows of five 8B layers), 743 -> 728 (64 rows of three). No
// early launch of the kernels that follow, as above: they read positions and tables before their own wait.
__global__ void __launch_bounds__(256) fetch_ints_kernel(const int4* host, int4* __restrict__ dev, int n4) {
  ib::pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n4) dev[i] = __ldcv(host + i);
}

}  // namespace

// host: pinned memory that the device can read, dev: device memory; n ints, a multiple of four, both on 16 bytes.
extern "C" int ib_fetch_ints(const int* host, int* dev, int n, cudaStream_t stream) {
  if (n == 0) return 0;
  IB_CHECK_ARG(n > 0 && n % 4 == 0 && host && dev && (((uintptr_t)host | (uintptr_t)dev) & 15) == 0, "fetch_ints: %d ints (a multiple of four, on 16 bytes)", n);
  ib::launch(fetch_ints_kernel, (n / 4 + 255) / 256, 256, 0, stream, (const int4*)host, (int4*)dev, n / 4);
  IB_CHECK_LAUNCH("fetch_ints");
  return 0;
}

extern "C" int ib_advance_rows(const int* sampled, int* token_in, int* positions, int* pos0, void* params, int* history, int* count, int rows,
                               int history_len, int* host, cudaStream_t stream) {
  if (rows == 0) return 0;
  IB_CHECK_ARG(rows > 0 && rows <= 1024 && history_len >= 0, "advance_rows: bad sizes rows=%d history=%d", rows, history_len);
  ib::launch(advance_rows_kernel, 1, 1024, 0, stream, sampled, token_in, positions, pos0, (RowParams*)params, history, count, rows, history_len, host);
  IB_CHECK_LAUNCH("advance_rows");
  return 0;
}

namespace {

// How many rows of 1 << lg CTAs the device runs at once (a cluster's CTAs lie in one group of SMs, so this is less than the CTAs that fit).
template <int PER_SM>
int rows_at_once(int lg) {
  static int known[4] = {};
  if (!known[lg]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << lg, 65535);
    cfg.blockDim = kThreads;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1u << lg, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, sample_kernel<PER_SM>, &cfg) != cudaSuccess) cudaGetLastError(), n = 0;
    known[lg] = n > 0 ? n : 1;
  }
  return known[lg];
}

}  // namespace

// logits float32 [rows, V], params [rows] of six words -> tokens int32 [rows].
// status: null, or the device status word, whose value is then stored in tokens[rows] (tokens has rows + 1 entries).
extern "C" int ib_sample_rows(const float* logits, int rows, int V, const void* params, int* tokens, const unsigned* status, cudaStream_t stream) {
  if (rows == 0) return 0;
  IB_CHECK_ARG(rows > 0 && rows <= 65535 && V > 0, "sample_rows: bad sizes rows=%d V=%d", rows, V);
  // The parts follow from the vocabulary alone. The CTAs that share them: as many as leave all rows running at once, three CTAs an SM: 64 rows of 151,936 with
  // top-p take 311 us on 1 CTA a row, 182 on 2, 143 on 4, 177 on 8; 160 rows 463 | 345 | 307 | 355; 128 rows of 32,768 114 | 105 | 120 | 159; 38 rows of 151,936
  // 307 | 178 | 137 | 112. And no more CTAs an SM than that takes: where three fit, some SMs are given three and others one. 64 rows of 151,936, logits in L2,
  // three | two an SM: drawn without a filter 44 | 32 us, top-k 129 | 85, top-p 172 | 122; 128 rows 86 | 62, 220 | 141, 309 | 212.
  int parts = 1, lg = 0;
  while (parts < kMaxParts && 2 * parts * kPartValues <= V) parts *= 2;
  while (1 << lg < parts && rows <= rows_at_once<kCtasOfSm>(lg + 1)) lg++;
  const int ctas = 1 << lg;
  ib::launch_cluster(rows <= rows_at_once<2>(lg) ? sample_kernel<2> : sample_kernel<kCtasOfSm>, dim3(ctas, rows), dim3(ctas), kThreads, 0, stream, logits, V,
                     ((V + parts - 1) / parts + 3) & ~3, parts / ctas, (const RowParams*)params, tokens, status);
  IB_CHECK_LAUNCH("sample_rows");
  return 0;
}
