// out[t][n] = sum_k x[t][k] * w[n][k] in float32 FMA arithmetic, for any T, N, K.
//
// This is the matrix product of the true 32-bit path (float32 inputs; no tensor-core mode of
// reduced precision), and with bfloat16 inputs it is the plain reference of the tcgen05 kernel.
// Every output element is the sum (c0 + c1) + (c2 + c3) of four sequential chains of FMAs, chain g over the
// k's with (k / 16) % 4 == g in ascending order, whatever the tile: a row's result does not depend on which
// other rows share the launch. The reference's equivalent is its 64x64x16 float32 tile
// (crates/kir/src/cuda/prelude.cu:213-276).
//
// What bounds it is the FMA units and the shared-memory reads that feed them where the product is large (128 lanes an SM; 73 TFLOP/s measured
// for FMAs on two registers, 49 on three), and too few threads where it is not: one chain an output left a product of 777 x 1,024 x 2,048 with
// three warps an SM. Hence four groups of 64 threads a tile, each with its own chain; their sums meet in shared memory at the end. A thread
// holds TM x TN outputs and reads four k's of a row in one 16-byte access (rows are 68 values apart, so eight neighbouring rows meet every
// bank once); three stages of 64 k's arrive by cp.async. 16 x 64 and smaller tiles are bound by the shared-memory reads (16 bytes a lane, 4 cycles
// of the SM's port a warp), larger ones by how the FMAs' operands leave the registers.
#include "common.cuh"

namespace {

constexpr int GROUPS = 4, GROUP_THREADS = 64, THREADS = GROUPS * GROUP_THREADS, GK = 16, BK = GROUPS * GK, STAGES = 3;

__device__ __forceinline__ float4 read4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 read4(const __nv_bfloat16* p) {
  const uint2 v = *(const uint2*)p;
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}

template <typename E>
struct Row {   // a staged row's length: 68 float32 or 72 bfloat16 (eight rows of 16 or 8 bytes meet different banks)
  static constexpr int LEN = sizeof(E) == 4 ? BK + 4 : BK + 8;
};

// rows r0 .. r0 + R - 1 of src [n][K], columns k0 .. k0 + BK - 1, into dst [R][LEN]; what lies outside is zero. VEC: rows start on 16
// bytes, so 16-byte asynchronous copies are used (a copy that crosses the row's end brings zeros behind it).
template <typename E, int R, bool VEC>
__device__ __forceinline__ void stage_rows(E* dst, const E* __restrict__ src, int r0, int n, int k0, int K, int tid) {
  constexpr int LEN = Row<E>::LEN;
  if constexpr (VEC) {
    constexpr int PER = 16 / sizeof(E), QUADS = BK / PER, STEP = THREADS / QUADS;   // rows a pass of all threads brings
    const int r = tid / QUADS, q = tid % QUADS, k = k0 + q * PER, left = max(0, min(16, (K - k) * (int)sizeof(E)));
    const E* from = src + (size_t)(r0 + r) * K + k;
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + r * LEN + q * PER);
#pragma unroll
    for (int u = 0; u < (R + STEP - 1) / STEP; u++) {
      const bool in = r0 + r + u * STEP < n && left > 0;
      if (R % STEP == 0 || r + u * STEP < R)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + u * STEP * LEN * (int)sizeof(E)), "l"(in ? from + (size_t)u * STEP * K : src), "r"(in ? left : 0)
                     : "memory");
    }
  } else {
    for (int e = tid; e < R * BK; e += THREADS) {
      const int r = e / BK, k = e % BK;
      dst[r * LEN + k] = r0 + r < n && k0 + k < K ? src[(size_t)(r0 + r) * K + k0 + k] : (E)0.f;
    }
  }
}

template <typename X, typename W, int BM, int BN>
constexpr size_t smem_bytes() {
  const size_t stages = STAGES * (BM * Row<X>::LEN * sizeof(X) + BN * Row<W>::LEN * sizeof(W)), sums = (size_t)GROUPS * BM * (BN + 4) * 4;
  return stages > sums ? stages : sums;
}

template <typename X, typename W, int BM, int BN, int TM, int TN, bool VEC, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) gemm_simt_kernel(const X* __restrict__ x, const W* __restrict__ w, float* __restrict__ out, int T, int N, int K) {
  static_assert((BM / TM) * (BN / TN) == GROUP_THREADS, "a group of 64 threads covers the tile");
  constexpr int COLS = BN / TN, ROWS = BM / TM;   // thread (ty, tx) holds rows ty + ROWS i and columns tx + COLS j
  constexpr int XL = Row<X>::LEN, WL = Row<W>::LEN;
  extern __shared__ __align__(16) unsigned char smem[];
  X* xs = (X*)smem;
  W* ws = (W*)(smem + STAGES * BM * XL * sizeof(X));
  ib::pdl_launch_dependents();
  ib::pdl_wait();
  const int tid = threadIdx.x, group = tid / GROUP_THREADS, lane = tid % GROUP_THREADS, ty = lane / COLS, tx = lane % COLS;
  const int t0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.f;

  const int steps = (K + BK - 1) / BK;
  auto fill = [&](int s) {
    if (s < steps) {
      stage_rows<X, BM, VEC>(xs + (s % STAGES) * BM * XL, x, t0, T, s * BK, K, tid);
      stage_rows<W, BN, VEC>(ws + (s % STAGES) * BN * WL, w, n0, N, s * BK, K, tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) fill(s);
  for (int s = 0; s < steps; s++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    fill(s + STAGES - 1);   // into the buffer whose readers passed the barrier
    const X* xa = xs + (s % STAGES) * BM * XL + ty * XL + group * GK;
    const W* wb = ws + (s % STAGES) * BN * WL + tx * WL + group * GK;
    // (k's past the end are zeros in both operands: an FMA with them leaves a sum as it is)
#pragma unroll
    for (int q = 0; q < GK; q += 4) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; i++) a[i] = read4(xa + i * ROWS * XL + q);
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const float4 b = read4(wb + j * COLS * WL + q);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* sums = (float*)smem;   // [GROUPS][BM][BN + 4]
  constexpr int SL = BN + 4;
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) sums[(group * BM + ty + ROWS * i) * SL + tx + COLS * j] = acc[i][j];
  __syncthreads();
  const bool wide = N % 4 == 0 && (uintptr_t)out % 16 == 0;
#pragma unroll
  for (int e = tid; e < BM * BN / 4; e += THREADS) {
    const int r = e / (BN / 4), c = e % (BN / 4) * 4, t = t0 + r, n = n0 + c;
    if (t >= T || n >= N) continue;
    float4 v[GROUPS];
#pragma unroll
    for (int g = 0; g < GROUPS; g++) v[g] = *(const float4*)&sums[(g * BM + r) * SL + c];
    const float4 o = make_float4((v[0].x + v[1].x) + (v[2].x + v[3].x), (v[0].y + v[1].y) + (v[2].y + v[3].y), (v[0].z + v[1].z) + (v[2].z + v[3].z),
                                 (v[0].w + v[1].w) + (v[2].w + v[3].w));
    float* to = out + (size_t)t * N + n;
    if (wide) {
      *(float4*)to = o;
    } else {
      to[0] = o.x;
      if (n + 1 < N) to[1] = o.y;
      if (n + 2 < N) to[2] = o.z;
      if (n + 3 < N) to[3] = o.w;
    }
  }
}

template <typename X, typename W, int BM, int BN, int TM, int TN, int MINB = 2>
int run(const X* x, const W* w, float* out, int T, int N, int K, cudaStream_t stream) {
  const bool vec = (size_t)K * sizeof(X) % 16 == 0 && (size_t)K * sizeof(W) % 16 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0;
  dim3 grid((N + BN - 1) / BN, (T + BM - 1) / BM);
  IB_CHECK_ARG(grid.y <= 65535, "gemm_simt: T=%d rows exceed the grid limit", T);
  constexpr size_t bytes = smem_bytes<X, W, BM, BN>();
  auto kernel = vec ? gemm_simt_kernel<X, W, BM, BN, TM, TN, true, MINB> : gemm_simt_kernel<X, W, BM, BN, TM, TN, false, MINB>;
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    IB_CHECK_ARG(e == cudaSuccess, "gemm_simt: %s", cudaGetErrorString(e));
  }
  ib::launch(kernel, grid, THREADS, bytes, stream, x, w, out, T, N, K);
  return 0;
}

// The larger the tile, the fewer shared-memory reads an FMA costs, and the worse its CTAs fill the SMs: a tile's last round of CTAs takes as long as
// a full one. So the form is the one with the least of rounds x (a tile's FMAs / the rate of a full SM) over the sizes; the rates, in FMAs an
// SM and us, are those of 2,048 x 4,096 x 4,096 rows, columns and k's (64 x 128: 1,565 us, 44 TFLOP/s; 64 x 64: 1,683; 32 x 64: 1,819; 32 x 32:
// 2,034), with which a product of 40 to 777 rows takes 7 to 12 us more than said here, whatever the tile. Measured (us, the tile by a count of
// CTAs alone before | now): 777 x 1,024 x 2,048 113 | 94 (143 tiles of 64 x 96 where 64 x 64 makes 208); 777 x 1,024 x 3,072 166 | 137;
// 777 x 6,144 x 1,024 288 | 257; 777 x 4,096 x 1,024 195 | 180; 300 x 1,024 x 2,048 68 | 57; 100 x 6,144 x 1,024 61 | 47. (Two-wide FMAs, tiles stored
// k by k, operands read a step ahead and two tiles an SM were all slower: 29 to 43 TFLOP/s at the large size; registers alone reach 66.)
// Up to 16 rows a tile has 16, and as many columns as leave every SM a CTA (2 x 32,768 x 1,024: 50 us against 230; 8 x 1,024 x 3,072: 26 against 236).
constexpr int SMS = 148;
struct Form {
  int bm, bn, per_sm;   // rows and columns of a tile, CTAs that share an SM
  float rate;
};
constexpr Form FORMS[] = {{16, 16, 2, 45e3f},   {16, 64, 2, 93e3f},  {32, 32, 2, 115e3f}, {32, 64, 2, 129e3f},  {48, 64, 1, 125e3f},
                          {64, 64, 1, 140e3f}, {40, 128, 1, 140e3f}, {48, 128, 1, 146e3f}, {56, 128, 1, 150e3f}, {64, 96, 1, 150e3f}, {64, 128, 1, 150e3f}};

inline int best_form(int T, int N) {
  int best = 0;
  float least = 0.f;
  for (int i = 0; i < (int)(sizeof(FORMS) / sizeof(FORMS[0])); i++) {
    const Form& f = FORMS[i];
    const long long tiles = (long long)((N + f.bn - 1) / f.bn) * ((T + f.bm - 1) / f.bm);
    const float rate = f.per_sm > 1 && tiles <= SMS ? 0.75f * f.rate : f.rate;   // (an SM with one of its two)
    const float cost = (float)((tiles + SMS - 1) / SMS) * (float)(f.bm * f.bn) / rate;
    if (i == 0 || cost < least) best = i, least = cost;
  }
  return best;
}

template <typename X, typename W>
int go(const X* x, const W* w, float* out, int T, int N, int K, cudaStream_t stream) {
  if (T <= 16) {
    if ((N + 63) / 64 >= SMS) return run<X, W, 16, 64, 2, 8>(x, w, out, T, N, K, stream);
    return run<X, W, 16, 16, 2, 2>(x, w, out, T, N, K, stream);
  }
  switch (best_form(T, N)) {   // (one CTA an SM: 48 and more sums and the operands of a thread do not fit 128 registers)
    case 0: return run<X, W, 16, 16, 2, 2>(x, w, out, T, N, K, stream);
    case 1: return run<X, W, 16, 64, 2, 8>(x, w, out, T, N, K, stream);
    case 2: return run<X, W, 32, 32, 4, 4>(x, w, out, T, N, K, stream);
    case 3: return run<X, W, 32, 64, 4, 8>(x, w, out, T, N, K, stream);
    case 4: return run<X, W, 48, 64, 6, 8, 1>(x, w, out, T, N, K, stream);
    case 5: return run<X, W, 64, 64, 8, 8, 1>(x, w, out, T, N, K, stream);
    case 6: return run<X, W, 40, 128, 5, 16, 1>(x, w, out, T, N, K, stream);
    case 7: return run<X, W, 48, 128, 6, 16, 1>(x, w, out, T, N, K, stream);
    case 8: return run<X, W, 56, 128, 7, 16, 1>(x, w, out, T, N, K, stream);
    case 9: return run<X, W, 64, 96, 8, 12, 1>(x, w, out, T, N, K, stream);
    default: return run<X, W, 64, 128, 8, 16, 1>(x, w, out, T, N, K, stream);
  }
}

}  // namespace

extern "C" int ib_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, float* out, int T, int N, int K, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  IB_CHECK_ARG(T > 0 && N > 0 && K > 0, "gemm_simt: bad sizes T=%d N=%d K=%d", T, N, K);
  int bad;
  if (x_dtype == IB_F32 && w_dtype == IB_F32)
    bad = go((const float*)x, (const float*)w, out, T, N, K, stream);
  else if (x_dtype == IB_BF16 && w_dtype == IB_BF16)
    bad = go((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, T, N, K, stream);
  else if (x_dtype == IB_F32 && w_dtype == IB_BF16)
    bad = go((const float*)x, (const __nv_bfloat16*)w, out, T, N, K, stream);
  else
    return ib_set_error("gemm_simt: unsupported dtypes x=%d w=%d", x_dtype, w_dtype);
  if (bad) return bad;
  IB_CHECK_LAUNCH("gemm_simt");
  return 0;
}
