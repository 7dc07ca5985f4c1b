// Plain matrix product for the true 32-bit path and for weights that are stored in 32-bit:
//   out[m,n] = sum_k A[m,k] * W[n,k] (+ bias[n])        weights are [out, in], as in the checkpoint
// FFMA only, no tensor cores and no reduced-precision mode.  The order in which an output's products are added follows
// from K alone, so its value depends on its own row of A and row of W only: the same bits whether the row comes alone, in a
// prompt or in a batch.  k_linear_plain (bfloat16 activations or weights): one accumulator over k = 0..K-1 in ascending
// order.  All in float32: see k_linear_f32_few and k_linear_f32_tile.
//
// Counterpart in the reference: k_gemm_f16 (src/kernels.cu:1410-1431; 16x16 tiles, one output per
// thread, f32 accumulate) with k_bias (:390-393) and k_add (:75-78) behind it.
#include "common.cuh"

enum { LIN_STORE = 0, LIN_ACCUM = 1 };

template <typename TA, typename TW, typename TO, int MODE>
__global__ void __launch_bounds__(256)
k_linear_plain(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias,
               TO* __restrict__ out, int M, int N, int K, int lda, int ldo) {
  cima_pdl_wait();
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;       // 16 x 16 threads, 4 x 4 outputs each
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 x 16 elements of each operand, 4 per thread: thread -> (row = idx / 16, k = idx % 16)
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int idx = threadIdx.x + r * 256;
      const int row = idx >> 4, kk = idx & 15;
      const int k = k0 + kk;
      float a = 0.f, w = 0.f;
      if (k < K) {
        if (m0 + row < M) a = cima_to_f32<TA>(A[(size_t)(m0 + row) * lda + k]);
        if (n0 + row < N) w = cima_to_f32<TW>(W[(size_t)(n0 + row) * K + k]);
      }
      As[kk][row] = a;
      Ws[kk][row] = w;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; j++) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      TO* o = out + (size_t)m * ldo + n;
      if (MODE == LIN_ACCUM) *o = cima_from_f32<TO>(cima_to_f32<TO>(*o) + v);
      else *o = cima_from_f32<TO>(v);
    }
  }
}

// ---------------------------------------------------------------------------------------------------- all in float32
// The 32-bit path's own product.  An output's sum over k is cut into F32_GROUPS ranges of k (f32_group_len, from K alone; sums of
// at most F32_ONE_RANGE stay one range, as there is little to share); a range is added up in ascending k by one accumulator, and
// the ranges' sums are added in their order.  Both kernels below follow that order, so a row's bits depend on its own row of A and
// the weights only: the same alone, in a prompt or in a batch, whatever tile or split serves it.  (One accumulator over all of K left a decode step one thread per output feature:
// 75 us a product at the 0.5B shape, 0.3 TB/s.  Eight ranges give eight times the threads, and a shorter chain of roundings.)
constexpr int F32_GROUPS = 8, F32_ONE_RANGE = 512;
__host__ __device__ inline int f32_group_len(int K) { return ((K <= F32_ONE_RANGE ? K : (K + F32_GROUPS - 1) / F32_GROUPS) + 15) & ~15; }

__device__ __forceinline__ void f32_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void f32_finish(float* o, float v, const float* bias, int n, int mode) {
  if (bias) v += bias[n];
  *o = mode == LIN_ACCUM ? *o + v : v;
}

// At most 8 rows (a decode step): the weights' bytes are the floor; at a third to a half of the bandwidth it stands between its loads'
// latency and shared memory.  A block takes 8 output features, a warp one range of k of
// them: its pieces of the 8 weight rows travel through shared memory by cp.async, 256-byte runs of a row at a time, up
// to FEW_STAGES pieces in flight, the first ones before the kernel ahead has finished where the caller says that it does not write them (`early`).  Lane =
// (feature, row mod 4): a lane walks its feature's range in order for one or two rows of A.  8 features a block and not more:
// a narrow product (896 features) still covers 112 SMs, and a wide one keeps several blocks on each.  A sum of one range has no
// work for a second warp, so there (ONE) each warp takes 8 features of its own, as many warps a block as leave a block for every SM
// (16,384 features of 512 k, one row: 17 us; with one working warp of 8 a block 51).  Measured inside a decode
// step of the 0.5B shape, 2 rows: 9.3 us a product on average, 2.2 TB/s (74.8 us and 0.27 TB/s with a thread an output feature).
constexpr int FEW_ROWS = 8, FEW_F = 8, FEW_K = 64, FEW_PITCH = FEW_K + 4, FEW_STAGES = 4, FEW_WARPS = F32_GROUPS;

template <int MR, bool VEC, bool ONE>        // MR: rows of A a lane takes (rows r, r + 4)
__global__ void __launch_bounds__(32 * FEW_WARPS)
k_linear_f32_few(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out,
                 int M, int N, int K, int lda, int ldo, int mode, int stages, int early) {
  extern __shared__ __align__(16) float few_smem[];
  __shared__ float red[FEW_WARPS][FEW_ROWS][FEW_F];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n0 = (ONE ? blockIdx.x * (blockDim.x >> 5) + warp : blockIdx.x) * FEW_F;
  const int len = f32_group_len(K), k0 = ONE ? 0 : min(K, warp * len), kn = min(K, k0 + len) - k0, chunks = (kn + FEW_K - 1) / FEW_K;
  const int unit = (FEW_F + M) * FEW_PITCH;             // a stage: 8 rows of W, then M rows of A
  float* mine = few_smem + (size_t)warp * stages * unit;
  // half a warp brings a piece of one row (from k0 + c FEW_K on) to dst; what lies beyond the range is zero
  const int half = lane >> 4, at = 4 * (lane & 15);
  auto piece = [&](float* dst, const float* src, int c) {
    const int left = kn - c * FEW_K - at;
    src += k0 + c * FEW_K + at;
    if constexpr (VEC) {
      if (left > 0) f32_copy16(dst + at, src);
      else *reinterpret_cast<float4*>(dst + at) = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++) dst[at + e] = e < left ? src[e] : 0.f;
    }
  };
  auto weights = [&](int c) {
    float* s = mine + (c % stages) * unit;
#pragma unroll
    for (int f = half; f < FEW_F; f += 2) piece(s + f * FEW_PITCH, W + (size_t)min(n0 + f, N - 1) * K, c);
  };
  auto rows = [&](int c) {
    float* s = mine + (c % stages) * unit + FEW_F * FEW_PITCH;
    for (int m = half; m < M; m += 2) piece(s + m * FEW_PITCH, A + (size_t)m * lda, c);
  };
  if (!early) cima_pdl_wait();
  for (int c = 0; c < min(stages, chunks); c++) weights(c);
  if (early) cima_pdl_wait();
  for (int c = 0; c < stages; c++) {
    if (c < chunks) rows(c);
    f32_commit();                                       // (the first of these groups holds all the weights requested above)
  }
  const int f = lane & 7, r = lane >> 3;
  const bool live = r < M;
  float acc[MR];
#pragma unroll
  for (int i = 0; i < MR; i++) acc[i] = 0.f;
  for (int c = 0; c < chunks; c++) {
    if (stages == FEW_STAGES) f32_wait<FEW_STAGES - 1>();
    else if (stages == 2) f32_wait<1>();
    else f32_wait<0>();
    __syncwarp();
    const float* s = mine + (c % stages) * unit;
    if (live) {
      const float *w = s + f * FEW_PITCH, *a = s + (FEW_F + r) * FEW_PITCH;
      const bool two = MR > 1 && r + 4 < M;
      const float* a2 = two ? a + 4 * FEW_PITCH : a;
      const int kc = (min(FEW_K, kn - c * FEW_K) + 3) & ~3;
#pragma unroll 8
      for (int k = 0; k < kc; k += 4) {
        const float4 x = *reinterpret_cast<const float4*>(w + k), y = *reinterpret_cast<const float4*>(a + k);
        acc[0] = fmaf(y.x, x.x, acc[0]); acc[0] = fmaf(y.y, x.y, acc[0]);
        acc[0] = fmaf(y.z, x.z, acc[0]); acc[0] = fmaf(y.w, x.w, acc[0]);
        if constexpr (MR > 1) {
          const float4 z = *reinterpret_cast<const float4*>(a2 + k);
          acc[1] = fmaf(z.x, x.x, acc[1]); acc[1] = fmaf(z.y, x.y, acc[1]);
          acc[1] = fmaf(z.z, x.z, acc[1]); acc[1] = fmaf(z.w, x.w, acc[1]);
        }
      }
    }
    __syncwarp();                                       // the stage has been read by every lane
    if (c + stages < chunks) { weights(c + stages); rows(c + stages); }
    f32_commit();
  }
  f32_wait<0>();
  cima_pdl_trigger();
  if constexpr (ONE) {
    if (live && n0 + f < N) {
      f32_finish(out + (size_t)r * ldo + n0 + f, acc[0], bias, n0 + f, mode);
      if (MR > 1 && r + 4 < M) f32_finish(out + (size_t)(r + 4) * ldo + n0 + f, acc[MR - 1], bias, n0 + f, mode);
    }
    return;
  }
  if (live) {
    red[warp][r][f] = acc[0];
    if (MR > 1 && r + 4 < M) red[warp][r + 4][f] = acc[MR - 1];
  }
  __syncthreads();
  const int m = threadIdx.x / FEW_F, n = n0 + threadIdx.x % FEW_F;
  if (m < M && n < N) {
    float v = red[0][m][threadIdx.x % FEW_F];
#pragma unroll
    for (int g = 1; g < FEW_WARPS; g++) v += red[g][m][threadIdx.x % FEW_F];
    f32_finish(out + (size_t)m * ldo + n, v, bias, n, mode);
  }
}

// More rows: bound by shared memory (64-row tiles, 398 rows of 9,728 x 896: 89 % of its rate, issue slots 69 %).  Tiles of BM x 128 outputs, 256 threads with BM / 16 x 8 outputs each.  The next 16 k travel
// through registers while the current ones are multiplied.  (Products two at a time, fma.rn.f32x2, want every value of A twice in
// shared memory and were no faster.)  SPLIT: a cluster of 8 blocks shares a tile, a range of k each, and adds the ranges' sums in
// order through distributed shared memory (see launch_f32 for when).  Measured inside a prompt step of the 0.5B shape, 201 + 197
// rows: 112 us a product on average, 26 TFLOP/s (322 us with tiles of 64 x 64 and 4 x 4 a thread); by themselves, alone and shared: 1,152 x 896 95 and 30 us, 9,728 x 896 187 and
// 186, 896 x 4,864 491 and 124; tiles of 64 rows for 37 rows of 1,152 x 896: 11.5, of 128: 17.
constexpr int F32_BN = 128, F32_BK = 16, F32_WROW = F32_BN + 4;

template <int BM>
constexpr int f32_tile_floats() { return 2 * F32_BK * (BM + 4 + F32_WROW); }
template <int BM, bool SPLIT>
constexpr size_t f32_tile_smem() {
  const size_t stage = f32_tile_floats<BM>() * sizeof(float), tile = SPLIT ? (size_t)BM * (F32_BN + 4) * sizeof(float) : 0;
  return stage > tile ? stage : tile;
}

template <int BM, bool SPLIT, bool VEC>
__global__ void __launch_bounds__(256, SPLIT ? 2 : 1)
k_linear_f32_tile(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out,
                  int M, int N, int K, int lda, int ldo, int mode) {
  constexpr int TM = BM / 16, AROW = BM + 4;
  constexpr int NA = (BM * F32_BK / 4 + 255) / 256, NW = F32_BN * F32_BK / 4 / 256;      // 16-byte pieces a thread moves
  extern __shared__ __align__(16) float f32_smem[];
  float* As = f32_smem;                                 // [2][F32_BK][AROW]
  float* Ws = f32_smem + 2 * F32_BK * AROW;             // [2][F32_BK][F32_WROW]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int rank = SPLIT ? blockIdx.x % F32_GROUPS : 0;
  const int m0 = blockIdx.y * BM, n0 = (SPLIT ? blockIdx.x / F32_GROUPS : blockIdx.x) * F32_BN;
  const int len = f32_group_len(K);
  const int kbeg = SPLIT ? min(K, rank * len) : 0, kend = SPLIT ? min(K, kbeg + len) : K;
  cima_pdl_wait();

  float4 ra[NA], rw[NW];
  auto load4 = [&](const float* p, int k) {              // four values of a row from k on; zero beyond the range
    if constexpr (VEC) return k < kend ? *reinterpret_cast<const float4*>(p + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    else return make_float4(k < kend ? p[k] : 0.f, k + 1 < kend ? p[k + 1] : 0.f, k + 2 < kend ? p[k + 2] : 0.f, k + 3 < kend ? p[k + 3] : 0.f);
  };
  auto fetch = [&](int k) {
#pragma unroll
    for (int i = 0; i < NA; i++) {
      const int idx = tid + 256 * i;
      if (BM * F32_BK / 4 >= 256 * (i + 1) || idx < BM * F32_BK / 4) ra[i] = load4(A + (size_t)min(m0 + idx / 4, M - 1) * lda, k + 4 * (idx % 4));
    }
#pragma unroll
    for (int i = 0; i < NW; i++) {
      const int idx = tid + 256 * i;
      rw[i] = load4(W + (size_t)min(n0 + idx / 4, N - 1) * K, k + 4 * (idx % 4));
    }
  };
  auto place = [&](int buf) {
#pragma unroll
    for (int i = 0; i < NA; i++) {
      const int idx = tid + 256 * i;
      if (BM * F32_BK / 4 >= 256 * (i + 1) || idx < BM * F32_BK / 4) {
        float* p = As + (buf * F32_BK + 4 * (idx % 4)) * AROW + idx / 4;
        p[0] = ra[i].x; p[AROW] = ra[i].y; p[2 * AROW] = ra[i].z; p[3 * AROW] = ra[i].w;
      }
    }
#pragma unroll
    for (int i = 0; i < NW; i++) {
      const int idx = tid + 256 * i;
      float* p = Ws + (buf * F32_BK + 4 * (idx % 4)) * F32_WROW + idx / 4;
      p[0] = rw[i].x; p[F32_WROW] = rw[i].y; p[2 * F32_WROW] = rw[i].z; p[3 * F32_WROW] = rw[i].w;
    }
  };

  float acc[TM][8], total[SPLIT ? 1 : TM][SPLIT ? 1 : 8];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) {
      acc[i][j] = 0.f;
      if constexpr (!SPLIT) total[i][j] = 0.f;
    }
  const int tiles = kend > kbeg ? (kend - kbeg + F32_BK - 1) / F32_BK : 0;
  const int per = len / F32_BK;                         // tiles of a range (SPLIT: the only one)
  if (tiles > 0) { fetch(kbeg); place(0); }
  int until = per;
  for (int t = 0; t < tiles; t++) {
    const int buf = t & 1;
    if (t + 1 < tiles) fetch(kbeg + (t + 1) * F32_BK);
    __syncthreads();
    const float *as = As + buf * F32_BK * AROW + TM * ty, *ws = Ws + buf * F32_BK * F32_WROW + 4 * tx;
#pragma unroll
    for (int k = 0; k < F32_BK; k++) {
      float a[TM], w[8];
      if constexpr (TM >= 4) {
#pragma unroll
        for (int i = 0; i < TM; i += 4) {
          const float4 v = *reinterpret_cast<const float4*>(as + k * AROW + i);
          a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
        }
      } else {
        const float2 v = *reinterpret_cast<const float2*>(as + k * AROW);
        a[0] = v.x; a[1] = v.y;
      }
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(ws + k * F32_WROW + 16 * j);
        w[j] = v.x; w[j + 1] = v.y; w[j + 2] = v.z; w[j + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    if constexpr (!SPLIT) {
      if (--until == 0 || t + 1 == tiles) {             // a range is complete
        until = per;
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < 8; j++) {
            total[i][j] += acc[i][j];
            acc[i][j] = 0.f;
          }
      }
    }
    if (t + 1 < tiles) place(buf ^ 1);                  // (last read before the barrier above)
  }
  cima_pdl_trigger();
  const bool wide = ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  auto store4 = [&](int m, int n, float4 v) {
    if (m >= M || n >= N) return;
    float* o = out + (size_t)m * ldo + n;
    if (wide && n + 3 < N) {
      if (bias) { v.x += bias[n]; v.y += bias[n + 1]; v.z += bias[n + 2]; v.w += bias[n + 3]; }
      if (mode == LIN_ACCUM) {
        const float4 c = *reinterpret_cast<const float4*>(o);
        v.x = c.x + v.x; v.y = c.y + v.y; v.z = c.z + v.z; v.w = c.w + v.w;
      }
      *reinterpret_cast<float4*>(o) = v;
    } else {
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (n + j < N) f32_finish(o + j, e[j], bias, n + j, mode);
    }
  };
  if constexpr (SPLIT) {
    constexpr int ROW = F32_BN + 4;
    __syncthreads();                                    // the stages are free: the tile takes their place
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        *reinterpret_cast<float4*>(f32_smem + (ty * TM + i) * ROW + 64 * j + 4 * tx) = make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
      }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    const unsigned base = (unsigned)__cvta_generic_to_shared(f32_smem);
    constexpr int MINE = BM / F32_GROUPS;               // rows of the tile that this block finishes
    for (int idx = tid; idx < MINE * (F32_BN / 4); idx += 256) {
      const int m = rank * MINE + idx / (F32_BN / 4), n = 4 * (idx % (F32_BN / 4));
      float4 s[F32_GROUPS];
#pragma unroll
      for (int g = 0; g < F32_GROUPS; g++) {
        unsigned at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base + (unsigned)((m * ROW + n) * sizeof(float))), "r"(g));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(s[g].x), "=f"(s[g].y), "=f"(s[g].z), "=f"(s[g].w) : "r"(at) : "memory");
      }
      float4 v = s[0];
#pragma unroll
      for (int g = 1; g < F32_GROUPS; g++) { v.x += s[g].x; v.y += s[g].y; v.z += s[g].z; v.w += s[g].w; }
      store4(m0 + m, n0 + n, v);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");      // nobody leaves while its tile is read
  } else {
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
        store4(m0 + ty * TM + i, n0 + 64 * j + 4 * tx, make_float4(total[i][4 * j], total[i][4 * j + 1], total[i][4 * j + 2], total[i][4 * j + 3]));
  }
}

template <typename Kern>
static int f32_allow(Kern kern, size_t smem) {
  if (smem <= 44 * 1024) return 0;                      // (48 KB are a kernel's without asking, its own static arrays among them)
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e == cudaSuccess ? 0 : cima_fail((int)e, "linear_plain: %zu bytes of shared memory are not available: %s", smem, cudaGetErrorString(e));
}

template <int BM, bool SPLIT, bool VEC>
static int launch_f32_tile(const float* A, const float* W, const float* bias, float* out, int mode, int M, int N, int K, int lda, int ldo,
                           cudaStream_t stream) {
  constexpr size_t smem = f32_tile_smem<BM, SPLIT>();
  auto kern = k_linear_f32_tile<BM, SPLIT, VEC>;
  if (int rc = f32_allow(kern, smem)) return rc;
  const dim3 grid((unsigned)((N + F32_BN - 1) / F32_BN) * (SPLIT ? F32_GROUPS : 1), (unsigned)((M + BM - 1) / BM));
  return cima_launch(kern, grid, dim3(256), smem, stream, SPLIT ? F32_GROUPS : 1, A, W, bias, out, M, N, K, lda, ldo, mode);
}

template <bool VEC>
static int launch_f32(const float* A, const float* W, const float* bias, float* out, int mode, int M, int N, int K, int lda, int ldo,
                      int early, cudaStream_t stream) {
  if (M <= FEW_ROWS) {
    const bool one = K <= F32_ONE_RANGE;
    const int parts = (N + FEW_F - 1) / FEW_F, warps = one ? max(1, min(FEW_WARPS, parts / 148)) : FEW_WARPS;
    const int chunks = (f32_group_len(K) + FEW_K - 1) / FEW_K, unit = (FEW_F + M) * FEW_PITCH * (int)sizeof(float) * warps;
    const int blocks = one ? (parts + warps - 1) / warps : parts;
    // the most pieces in flight that leave room for two blocks on an SM: its own, or the next launch's, whose weights are then
    // requested while this one ends
    const int room = 110 * 1024;
    const int stages = chunks >= FEW_STAGES && FEW_STAGES * unit <= room ? FEW_STAGES : chunks >= 2 ? 2 : 1;
    const size_t smem = (size_t)stages * unit;
    auto kern = one ? (M <= 4 ? k_linear_f32_few<1, VEC, true> : k_linear_f32_few<2, VEC, true>) : M <= 4 ? k_linear_f32_few<1, VEC, false> : k_linear_f32_few<2, VEC, false>;
    if (int rc = f32_allow(kern, smem)) return rc;
    return cima_launch(kern, dim3((unsigned)blocks), dim3(32 * warps), smem, stream, 1, A, W, bias, out, M, N, K, lda, ldo, mode, stages, early);
  }
  // The tile's rows, and whether clusters share a tile, by the time of the SM that gets the most blocks: a block's rows (a lower tile
  // reads more of shared memory for a product: measured at 0.9 and 0.7 of the rate), an eighth of them where a cluster shares the tile (and
  // a sixth more for the sums' way through the cluster).
  const long long nt = (N + F32_BN - 1) / F32_BN;
  int bm = 128;
  bool split = false;
  double best = 1e30;
  for (int rows = 128; rows >= 32; rows /= 2)
    for (int shared = 0; shared < 2; shared++) {
      if (shared && K <= F32_ONE_RANGE) continue;
      const long long blocks = nt * ((M + rows - 1) / rows) * (shared ? F32_GROUPS : 1);
      const double cost = (double)((blocks + 147) / 148) * rows * (rows == 128 ? 1.0 : rows == 64 ? 1.1 : 1.4) * (shared ? 1.17 / F32_GROUPS : 1.0);
      if (cost < best) { best = cost; bm = rows; split = shared; }
    }
#define F32_RUN(BM) return split ? launch_f32_tile<BM, true, VEC>(A, W, bias, out, mode, M, N, K, lda, ldo, stream) \
                                 : launch_f32_tile<BM, false, VEC>(A, W, bias, out, mode, M, N, K, lda, ldo, stream)
  if (bm == 32) F32_RUN(32);
  if (bm == 64) F32_RUN(64);
  F32_RUN(128);
#undef F32_RUN
}

template <typename TA, typename TW, typename TO>
static int launch_plain(const void* A, const void* W, const float* bias, void* out, int mode, int M, int N, int K,
                        int lda, int ldo, int early, cudaStream_t stream) {
  if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4 && sizeof(TO) == 4) {
    const bool vec = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    const int rc = vec ? launch_f32<true>((const float*)A, (const float*)W, bias, (float*)out, mode, M, N, K, lda, ldo, early, stream)
                       : launch_f32<false>((const float*)A, (const float*)W, bias, (float*)out, mode, M, N, K, lda, ldo, early, stream);
    return rc ? rc : cima_launch_result();
  } else {
  dim3 grid((N + 63) / 64, (M + 63) / 64);
  if (mode == LIN_STORE)
    { int rc_ = cima_launch(k_linear_plain<TA, TW, TO, LIN_STORE>, dim3(grid), dim3(256), (size_t)(0), stream, 1, (const TA*)A, (const TW*)W, bias, (TO*)out, M, N, K, lda, ldo); if (rc_) return rc_; }
  else
    { int rc_ = cima_launch(k_linear_plain<TA, TW, TO, LIN_ACCUM>, dim3(grid), dim3(256), (size_t)(0), stream, 1, (const TA*)A, (const TW*)W, bias, (TO*)out, M, N, K, lda, ldo); if (rc_) return rc_; }
  return cima_launch_result();
  }
}

// mode 0: out = A W^T (+ bias), stored as out_dtype.  mode 1: out += A W^T (+ bias); out must be float32.
// early != 0: the kernel launched just before this one on the stream does not write W, so W may be read while it finishes.
extern "C" int cima_linear_plain(const void* A, int a_dtype, const void* W, int w_dtype, const float* bias,
                                 void* out, int out_dtype, int mode, int M, int N, int K, int lda, int ldo,
                                 int early, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (N <= 0 || K <= 0) return cima_fail(CIMA_E_SIZE, "linear_plain: N %d and K %d must be positive", N, K);
  if (lda < K || ldo < N) return cima_fail(CIMA_E_SIZE, "linear_plain: leading dimensions (%d, %d) are smaller than the rows (%d, %d)", lda, ldo, K, N);
  if (mode != LIN_STORE && mode != LIN_ACCUM) return cima_fail(CIMA_E_ARG, "linear_plain: mode %d is neither store (0) nor accumulate (1)", mode);
  if (mode == LIN_ACCUM && out_dtype != CIMA_F32) return cima_fail(CIMA_E_DTYPE, "linear_plain: accumulation needs a float32 output");
  if ((long long)((M + 63) / 64) > 65535) return cima_fail(CIMA_E_SIZE, "linear_plain: %d rows exceed one launch; the caller cuts them", M);
  const int key = a_dtype * 4 + w_dtype * 2 + out_dtype;
  switch (key) {
    case 0: return launch_plain<float, float, float>(A, W, bias, out, mode, M, N, K, lda, ldo, early, stream);
    case 4 + 0 + 0: return launch_plain<__nv_bfloat16, float, float>(A, W, bias, out, mode, M, N, K, lda, ldo, early, stream);
    case 4 + 0 + 1: return launch_plain<__nv_bfloat16, float, __nv_bfloat16>(A, W, bias, out, mode, M, N, K, lda, ldo, early, stream);
    case 4 + 2 + 0: return launch_plain<__nv_bfloat16, __nv_bfloat16, float>(A, W, bias, out, mode, M, N, K, lda, ldo, early, stream);
    case 4 + 2 + 1: return launch_plain<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(A, W, bias, out, mode, M, N, K, lda, ldo, early, stream);
    default:
      return cima_fail(CIMA_E_DTYPE, "linear_plain: dtypes (A %d, W %d, out %d) are not a supported combination", a_dtype, w_dtype, out_dtype);
  }
}
