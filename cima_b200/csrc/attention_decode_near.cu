// Decode attention of near contexts (bfloat16, one new query a sequence, up to 8 query heads a kv head): keys and values go
// straight to registers, and the blocks that share a sequence and kv head are a thread-block cluster that merges its results
// itself, so one launch does what the split kernel and its merge do in two.
//
// What bounds a step's attention over some hundred or thousand positions is not bytes but the chain: launch, a page's way to
// shared memory, a few instructions a key, the merge.  attention_decode.cu walks its pages one after another through shared
// memory (about 850 instructions a warp and page, 24 KB of code that is fetched anew at every launch).  Here a warp takes 16
// keys at a time and a block 128: lane (g, t) loads dims 32 d + 8 t .. + 7 of keys g and g + 8, 16 bytes each, which serve as
// operands as they are (a sum over dims does not care about their order); S = K Q^T has the keys as its 16 rows and the
// group's heads as its 8 columns, O = V^T P^T the dims as rows, V and P transposed by movmatrix.  The first round's loads are issued
// before the wait for the projection kernel, but for the newest position's, and each later round's as soon as its
// registers are free.  Scores, maxima, exponentials and sums are float32, base 2; probabilities are rounded to bfloat16 as the
// operand of P V only.  Warps, then the cluster's blocks, are merged in a fixed order.
//
// Measured inside the decode step (us a layer against the split kernel and its merge): 0.5B shape, one sequence of 40 / 300 /
// 1,000 positions -0.7 / -2.6 / -2.5; 1.5B, 100 / 4,000 -3.7 / -3.5, five of 340 -4.0; 7B, one of 2,000 -4.7, 8 of 300 / 2,048 /
// 24,000 -5.2 / -6.8 / -6.7, 32 of 270 -5.3.  (kernels.py, near_cluster and near_context: which cluster, and up to where.)
#include "common.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace {

constexpr int PS = 64;            // keys per page
constexpr int WARPS = 8;

__device__ __forceinline__ uint4 ld_once16(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transposed(uint32_t v) {
  uint32_t r;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// early: the kernel launched just before this one has written nothing that this one reads but qkv and, in the cache, the newest position
// (seq_len[b] - 1) of each sequence: every other position is read before the wait on that kernel, its own page's included.
// (attention_decode.cu asks for less: it leaves the newest position's whole page until after the wait.)  qkv is not __restrict__, since that
// kernel may write it during this one's life: its reads must stay behind the wait.
template <int HD>
__global__ void __launch_bounds__(WARPS * 32)
k_attention_near(const __nv_bfloat16* qkv, int ld, const __nv_bfloat16* cache, CimaPaged pg, const int* __restrict__ seq_slot,
                 const int* __restrict__ seq_len, __nv_bfloat16* __restrict__ out, int ldo, int nh, int nkv, float scale, int window, int early) {
  if (!early) cima_pdl_wait();
  __shared__ float so[WARPS][8][HD + 1];             // the warps' results; then [0]: the block's
  __shared__ float2 ml[WARPS][8];                    // their maxima and sums; then [0]: the block's
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int kvh = blockIdx.y, b = blockIdx.z, G = nh / nkv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int len = seq_len[b], slot = seq_slot[b];
  const int lo = window > 0 && len > window ? len - window : 0;
  const int first = lo / 16, chunks = (len - 1) / 16 - first + 1;           // pieces of 16 keys
  const int c0 = first + chunks * rank / CL, c1 = first + chunks * (rank + 1) / CL;
  const __nv_bfloat16* kbase = cache + (size_t)kvh * (PS * HD) + 8 * t;
  const size_t v_off = (size_t)nkv * (PS * HD);

  auto place = [&](int c) {
    int e = c >> 2;
    if (pg.ring) e %= pg.ring;
    return kbase + (size_t)pg.table[(size_t)slot * pg.width + e] * 2 * nkv * (PS * HD) + (c & 3) * 16 * HD;
  };
  // Rows that are not loaded keep what the registers hold (0, or an earlier key's): a key's score is then masked.  A value's weight is 0, which
  // an earlier key's infinity would turn into NaN, so a later round clears its values (`clear`).
  uint4 kf[HD / 32][2] = {}, vf[HD / 32][2] = {};
  auto load = [&](uint4 (&r)[HD / 32][2], const __nv_bfloat16* src, int c, int from, int to, bool clear = false) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int key = c * 16 + g + 8 * h;
      if (key >= from && key < to) {
#pragma unroll
        for (int d = 0; d < HD / 32; d++) r[d][h] = ld_once16(src + (g + 8 * h) * HD + 32 * d);
      } else if (clear) {
#pragma unroll
        for (int d = 0; d < HD / 32; d++) r[d][h] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };

  int c = c0 + warp;
  const bool busy = c < c1;
  const __nv_bfloat16* src = nullptr;
  if (busy) {
    src = place(c);
    load(kf, src, c, lo, early ? len - 1 : len);
    load(vf, src + v_off, c, lo, early ? len - 1 : len);
  }
  if (early) cima_pdl_wait();

  float o[HD / 16][4];
#pragma unroll
  for (int j = 0; j < HD / 16; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float mr[2] = {-INFINITY, -INFINITY}, lr[2] = {0.f, 0.f};
  if (busy) {
    if (early && c * 16 + 16 >= len) {                // the newest position: the kernel before has written it by now
      load(kf, src, c, len - 1, len);
      load(vf, src + v_off, c, len - 1, len);
    }
    uint4 q[HD / 32] = {};
    if (g < G) {
#pragma unroll
      for (int d = 0; d < HD / 32; d++) q[d] = *reinterpret_cast<const uint4*>(qkv + (size_t)b * ld + (size_t)(kvh * G + g) * HD + 32 * d + 8 * t);
    }
    const float sc2 = scale * 1.4426950408889634f;    // scores and maxima are in the base-2 domain
#pragma unroll 1
    for (; c < c1; c += WARPS) {
      const bool more = c + WARPS < c1;
      if (more) src = place(c + WARPS);
      // S = K Q^T: (key g, heads 2t, 2t + 1), (key g + 8, the same)
      float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int d = 0; d < HD / 32; d++) {
        mma(sa, kf[d][0].x, kf[d][1].x, kf[d][0].y, kf[d][1].y, q[d].x, q[d].y);
        mma(sb, kf[d][0].z, kf[d][1].z, kf[d][0].w, kf[d][1].w, q[d].z, q[d].w);
      }
      if (more) load(kf, src, c + WARPS, lo, len);
      const int key = c * 16 + g;
      // Probabilities against the 16 keys' own maximum, whose key's is 1 and so has no rounding to bfloat16, and the 16 keys' sum from 0, brought
      // to the running maximum by float32 multiply-adds: against the running maximum the result was the further from 64 bits the fewer
      // warps shared the keys (relative error at 2,000 positions in clusters of 16 / 4 / 1: 1.94 / 2.04 / 2.14e-3), further than the splits
      // where those are more than the blocks.
      float p[4], corr[2], f[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float v0 = key >= lo && key < len ? (sa[j] + sb[j]) * sc2 : -INFINITY;
        const float v1 = key + 8 >= lo && key + 8 < len ? (sa[j + 2] + sb[j + 2]) * sc2 : -INFINITY;
        float mx = fmaxf(v0, v1);
#pragma unroll
        for (int x = 4; x < 32; x *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
        const float own = mx == -INFINITY ? 0.f : mx, mn = fmaxf(mr[j], mx), ms = mn == -INFINITY ? 0.f : mn;
        p[j] = ex2(v0 - own);
        p[j + 2] = ex2(v1 - own);
        corr[j] = ex2(mr[j] - ms);
        f[j] = ex2(mx - ms);
        mr[j] = mn;
        lr[j] = fmaf(lr[j], corr[j], (p[j] + p[j + 2]) * f[j]);
      }
      const uint32_t b0 = transposed(pack2(p[0], p[1])), b1 = transposed(pack2(p[2], p[3]));
      // O = V^T P^T: tile (d, e) holds dims 32 d + 8 (g / 2) + g % 2 + 4 e (rows g) and those + 2 (rows g + 8)
#pragma unroll
      for (int d = 0; d < HD / 32; d++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
          float s16[4] = {0.f, 0.f, 0.f, 0.f};
          if (e == 0) mma(s16, transposed(vf[d][0].x), transposed(vf[d][0].y), transposed(vf[d][1].x), transposed(vf[d][1].y), b0, b1);
          else mma(s16, transposed(vf[d][0].z), transposed(vf[d][0].w), transposed(vf[d][1].z), transposed(vf[d][1].w), b0, b1);
#pragma unroll
          for (int i = 0; i < 4; i++) o[2 * d + e][i] = fmaf(o[2 * d + e][i], corr[i & 1], s16[i] * f[i & 1]);
        }
      }
      if (more) load(vf, src + v_off, c + WARPS, lo, len, true);
    }
  }
  cima_pdl_trigger();

  // the warps' results side by side
#pragma unroll
  for (int j = 0; j < 2; j++) {
    float l = lr[j];
#pragma unroll
    for (int x = 4; x < 32; x *= 2) l += __shfl_xor_sync(0xffffffffu, l, x);
    float* row = &so[warp][2 * t + j][8 * (g >> 1) + (g & 1)];
#pragma unroll
    for (int i = 0; i < HD / 16; i++) {
      row[32 * (i >> 1) + 4 * (i & 1)] = o[i][j];
      row[32 * (i >> 1) + 4 * (i & 1) + 2] = o[i][j + 2];
    }
    if (g == 0) ml[warp][2 * t + j] = make_float2(mr[j], l);
  }
  __syncthreads();
  // a warp a head: the warps' factors in lanes 0 .. 7, the sum over the warps dim by dim
  float mine[HD / 32], M = -INFINITY, l = 0.f;
  {
    const float2 w = lane < WARPS ? ml[lane][warp] : make_float2(-INFINITY, 0.f);
    M = w.x;
#pragma unroll
    for (int x = 4; x > 0; x >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, x));
    M = __shfl_sync(0xffffffffu, M, 0);
    const float f = ex2(w.x - (M == -INFINITY ? 0.f : M));
    l = f * w.y;
#pragma unroll
    for (int x = 4; x > 0; x >>= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
    l = __shfl_sync(0xffffffffu, l, 0);
#pragma unroll
    for (int i = 0; i < HD / 32; i++) mine[i] = 0.f;
#pragma unroll 4
    for (int w2 = 0; w2 < WARPS; w2++) {
      const float fw = __shfl_sync(0xffffffffu, f, w2);
#pragma unroll
      for (int i = 0; i < HD / 32; i++) mine[i] += fw * so[w2][warp][lane + 32 * i];
    }
  }
  if (CL > 1) {
    __syncthreads();                                  // every warp has read the others' results: the block's take their place
#pragma unroll
    for (int i = 0; i < HD / 32; i++) so[0][warp][lane + 32 * i] = mine[i];
    if (lane == 0) ml[0][warp] = make_float2(M, l);
    cluster.sync();
    // head `warp` is finished by the block whose rank is warp % CL
    if (warp % CL == rank) {
      const float2 w = lane < CL ? *cluster.map_shared_rank(&ml[0][warp], lane) : make_float2(-INFINITY, 0.f);
      M = w.x;
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, x));
      const float f = ex2(w.x - (M == -INFINITY ? 0.f : M));
      l = f * w.y;
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
      for (int i = 0; i < HD / 32; i++) mine[i] = 0.f;
#pragma unroll 4
      for (int r = 0; r < CL; r++) {
        const float fw = __shfl_sync(0xffffffffu, f, r);
        const float* theirs = cluster.map_shared_rank(&so[0][warp][lane], r);
#pragma unroll
        for (int i = 0; i < HD / 32; i++) mine[i] += fw * theirs[32 * i];
      }
      M = __shfl_sync(0xffffffffu, M, 0);
      l = __shfl_sync(0xffffffffu, l, 0);
    }
  }
  if (warp < G && warp % CL == rank) {
    const int h = kvh * G + warp;
    const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
    for (int i = 0; i < HD / 32; i++) out[(size_t)b * ldo + (size_t)h * HD + lane + 32 * i] = __float2bfloat16_rn(mine[i] * inv);
  }
  if (CL > 1) cluster.sync();                         // a block's shared memory outlives the others' reads of it
}

// Clusters of more than 8 blocks are more than every device has to offer: this one may.
template <int HD>
cudaError_t allow_near(int cluster) {
  if (cluster <= 8) return cudaSuccess;
  static bool allowed[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && (dev < 0 || dev >= 64 || !allowed[dev])) {
    e = cudaFuncSetAttribute(k_attention_near<HD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess && dev >= 0 && dev < 64) allowed[dev] = true;
  }
  return e;
}

// Clusters of `cluster` blocks that the current device holds at once; 0 where it cannot place one, or cannot say.
template <int HD>
int near_room(int cluster) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(WARPS * 32);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (allow_near<HD>(cluster) == cudaSuccess && cudaOccupancyMaxActiveClusters(&n, k_attention_near<HD>, &cfg) == cudaSuccess) return n;
  cudaGetLastError();                                 // (what is no launch's error must not become one)
  return 0;
}

template <int HD>
int launch_near(const void* qkv, int ld, const void* cache, CimaPaged pg, const int* seq_slot, const int* seq_len, void* out, int ldo, int B, int nh,
                int nkv, float scale, int window, int cluster, int early, cudaStream_t stream) {
  if (const cudaError_t e = allow_near<HD>(cluster)) return cima_fail((int)e, "attention_decode_near: a cluster of %d blocks: %s", cluster, cudaGetErrorString(e));
  const int rc = cima_launch(k_attention_near<HD>, dim3(cluster, nkv, B), dim3(WARPS * 32), 0, stream, cluster, (const __nv_bfloat16*)qkv, ld,
                             (const __nv_bfloat16*)cache, pg, seq_slot, seq_len, (__nv_bfloat16*)out, ldo, nh, nkv, scale, window, early);
  return rc ? rc : cima_launch_result();
}

}  // namespace

// One query row a sequence (row b of qkv belongs to sequence b), pages of 64 with keys | values, head sizes 64 and 128, at most 8
// query heads a kv head; any window (without kept first positions); `cluster` blocks (1, 2, 4, 8 or 16) share a sequence and kv
// head.  early: see k_attention_near (more is asked of the kernel before than by cima_attention_decode).  The other arguments are
// cima_attention_decode's.
extern "C" int cima_attention_decode_near(const void* qkv, int ld, const void* cache, const int* table, int table_width, int ring, const int* seq_slot,
                                          const int* seq_len, void* out, int ldo, int B, int nh, int nkv, int hd, float scale, int window,
                                          int cluster, int early, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (hd != 64 && hd != 128) return cima_fail(CIMA_E_SIZE, "attention_decode_near: head_dim %d; this kernel takes 64 and 128", hd);
  if (nh <= 0 || nkv <= 0 || nh % nkv || nh / nkv > 8) return cima_fail(CIMA_E_SIZE, "attention_decode_near: %d heads are not 1 to 8 times %d kv heads", nh, nkv);
  if (cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8 && cluster != 16) return cima_fail(CIMA_E_ARG, "attention_decode_near: a cluster of %d; 1, 2, 4, 8 and 16 are possible", cluster);
  if (B > 65535 || nkv > 65535) return cima_fail(CIMA_E_SIZE, "attention_decode_near: %d sequences exceed one launch", B);
  if (ld % 8 || ((uintptr_t)qkv & 15) || ((uintptr_t)cache & 15)) return cima_fail(CIMA_E_ARG, "attention_decode_near: qkv rows and the cache must be 16-byte aligned");
  const CimaPaged pg{table, table_width, ring, PS, nkv, hd, 2};
  return (hd == 64 ? launch_near<64> : launch_near<128>)(qkv, ld, cache, pg, seq_slot, seq_len, out, ldo, B, nh, nkv, scale, window, cluster, early, stream);
}

// room[0 .. 3]: clusters of 16, 8, 4 and 2 blocks that the current device holds at once (they follow from how its SMs are grouped, which
// differs from one device to the next).
extern "C" int cima_attention_decode_near_room(int hd, int* room) {
  if (hd != 64 && hd != 128) return cima_fail(CIMA_E_SIZE, "attention_decode_near: head_dim %d; this kernel takes 64 and 128", hd);
  for (int i = 0; i < 4; i++) room[i] = hd == 64 ? near_room<64>(16 >> i) : near_room<128>(16 >> i);
  return 0;
}
