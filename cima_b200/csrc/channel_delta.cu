// The delta rule with a decay a key channel (see recurrence.cu), 16 tokens at a time: bfloat16 values of a long step.
//   S <- diag(g_t) S;  u = beta_t (v - S^T k);  S <- S + k u^T;  o = S^T q            q, k, g, beta float32, S float32
// With G_t = g_1 .. g_t of the chunk (a vector over the key channels), R_s = g_(s+1) .. g_16, the state S0 in front of it and
//   a_ts = k_t . (g_(s+1) .. g_t k_s)  (s < t),      m_ts = q_t . (g_(s+1) .. g_t k_s)  (s <= t)
//   (I + A) U = rhs,   A_ts = beta_t a_ts,   rhs_t = beta_t (v_t - (G_t k_t)^T S0)
//   o_t = (G_t q_t)^T S0 + sum_{s <= t} m_ts u_s
//   S   = diag(G_16) S0 + sum_s (R_s k_s) u_s^T
// so the chain from token to token (880 cycles each in the walk of recurrence.cu, two reductions over lanes and the reads of
// k, q and g for every four columns) becomes one from chunk to chunk.  Every factor is a product of decays between 0 and 1, in the
// order the walk multiplies them: nothing is divided by, nothing overflows, and a decay of 0 is no special case.  The products
// run on the tensor cores (mma.m16n8k16) without giving up float32: both operands enter as sums of three bfloat16 terms, which
// hold their 24 bits, in all pairs but those below 2^-24, summed in float32.  Bound by the issue of mma.sync in the column warps
// (312 a chunk), so it gains where there are several sequences.  12 heads of 128 x 128, walk and chunks: sequences of 900, 883,
// 531 and 1,080 tokens 500 and 335 us; 16 of 300: 567 and 302; 64 of 128: 869 and 510; one of 2,048: 631 and 620.
//   Warps 0 .. 3 own 16 columns each and keep S^T [16 columns][dim] as the accumulators of the update; two neighbouring
//   accumulator tiles are the A operand of the next chunk's product.  The others run ahead, a barrier a chunk between the stages:
//   warp 9 loads the rows of chunk j + 4, warps 4 and 5 make a and m of chunk j + 2 (half of the s each, 4 channels a lane, a
//   running product a value of s), warps 6 and 7 the split vectors G k, G q and R k of chunk j + 1, and warp 8 turns a into
//   T = (I + A)^-1 there, while chunk j is worked on.
#include "common.cuh"
#include "delta_chunk.cuh"

namespace {
constexpr int CD_COL_WARPS = 4, CD_COLS = 16 * CD_COL_WARPS, CD_THREADS = 32 * (CD_COL_WARPS + 6), CD_ROWS = 4, CD_VALUES = 5;
constexpr int CD_TROW = 24, CD_VROW = CD_COLS + 8;      // padded rows of the 16 x 16 matrices' terms and of v

template <int DIMP>
struct __align__(16) CdShared {
  float k[CD_ROWS][DC_T][DIMP + 4], q[CD_ROWS][DC_T][DIMP + 4], g[CD_ROWS][DC_T][DIMP + 4];
  bf16 v[CD_VALUES][DC_T][CD_VROW];
  bf16 K[2][3][DC_T][DIMP + 8], Q[2][3][DC_T][DIMP + 8], W[2][3][DC_T][DIMP + 8];      // the terms of G k, G q and R k
  bf16 T[2][3][DC_T][CD_TROW], M[2][3][DC_T][CD_TROW];  // the terms of the inverse and of m, [t][s]
  float a[2][DC_T][DC_T + 4], m[2][DC_T][DC_T + 4], A[DC_T][DC_T + 4];
  float beta[CD_VALUES][DC_T], gc[2][DIMP];             // gc: G_16
};

// a and m of one chunk for half of the s: 0, 3, 4, 7, .. (half 0) or 1, 2, 5, 6, .. (half 1), 60 pairs each.  (The tokens stay a
// loop: written out sixteen times, the two halves were 128 KB of instructions.)
template <int DIMP>
__device__ __forceinline__ void cd_pairs(CdShared<DIMP>& sm, int stage, int buf, int nt, int lane, int half) {
  const bool have = 4 * lane < DIMP;
  float w[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int e = 0; e < 4; e++) w[i][e] = 0.f;
#pragma unroll 1
  for (int t0 = 0; t0 < DC_T; t0 += 2) {                  // two tokens' sums handed over together
    float x[32];                                          // token u: 16 u + 2 i: a of the i-th s, 16 u + 2 i + 1: m
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int t = t0 + u;
      float4 g4 = make_float4(1.f, 1.f, 1.f, 1.f), k4 = make_float4(0.f, 0.f, 0.f, 0.f), q4 = k4;      // a token beyond the end does nothing
      if (have && t < nt) {
        g4 = *reinterpret_cast<const float4*>(&sm.g[stage][t][4 * lane]);
        k4 = *reinterpret_cast<const float4*>(&sm.k[stage][t][4 * lane]);
        q4 = *reinterpret_cast<const float4*>(&sm.q[stage][t][4 * lane]);
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int s = 2 * i + ((i & 1) ? 1 - half : half);
        if (s == t) {                                     // (before its own token w is 0, and so are its sums)
          w[i][0] = k4.x; w[i][1] = k4.y; w[i][2] = k4.z; w[i][3] = k4.w;
        } else {
          w[i][0] *= g4.x; w[i][1] *= g4.y; w[i][2] *= g4.z; w[i][3] *= g4.w;
        }
        const float a = fmaf(k4.x, w[i][0], fmaf(k4.y, w[i][1], fmaf(k4.z, w[i][2], k4.w * w[i][3])));
        x[16 * u + 2 * i] = s == t ? 0.f : a;
        x[16 * u + 2 * i + 1] = fmaf(q4.x, w[i][0], fmaf(q4.y, w[i][1], fmaf(q4.z, w[i][2], q4.w * w[i][3])));
      }
    }
    // handed over by halves: the lane's number says which of the 32 sums it ends up with
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
      const bool upper = lane & d;
#pragma unroll
      for (int c = 0; c < d; c++) {
        const float mine = upper ? x[c + d] : x[c], other = upper ? x[c] : x[c + d];
        x[c] = mine + __shfl_xor_sync(0xffffffffu, other, d);
      }
    }
    const int i = (lane >> 1) & 7, s = 2 * i + ((i & 1) ? 1 - half : half), t = t0 + (lane >> 4);
    if (lane & 1) sm.m[buf][t][s] = x[0];
    else sm.a[buf][t][s] = x[0];
  }
}

template <int DIMP>
__global__ void __launch_bounds__(CD_THREADS, 1)
k_channel_delta(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk, const bf16* __restrict__ v, int ldv,
                const float* __restrict__ g, const float* __restrict__ beta, float* __restrict__ state, const int* __restrict__ seq_slot,
                const int* __restrict__ seq_first_row, float* __restrict__ out, int heads, int kv_heads, int dim, int vdim) {
  extern __shared__ __align__(16) unsigned char cd_smem[];
  CdShared<DIMP>& sm = *reinterpret_cast<CdShared<DIMP>*>(cd_smem);
  constexpr int KS = DIMP / 16, NT = DIMP / 8;
  const int seq = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * CD_COLS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g8 = lane >> 2, t4 = lane & 3;              // a fragment's row (and row + 8) and pair of columns
  const int kvh = h / (heads / kv_heads);
  cima_pdl_wait();
  const int first = seq_first_row[seq], n = seq_first_row[seq + 1] - first;
  const int chunks = (n + DC_T - 1) / DC_T;
  // what no copy reaches (channels and columns beyond the sizes) stays zero
  for (int i = threadIdx.x; i < (int)(sizeof(sm.k) + sizeof(sm.q) + sizeof(sm.g) + sizeof(sm.v)) / 16; i += CD_THREADS)
    reinterpret_cast<uint4*>(&sm)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();

  // Every warp meets a barrier at the start of step j = -3 .. chunks - 1 and works on its own chunk of that step, if there is one.
  if (warp == CD_COL_WARPS + 5) {
    // ------------------------------------------------------------------------------------------ the rows of chunk j + 4
    // Beyond a sequence's end the last token's rows are copied again: nobody reads q, k and g there, and v meets a step size of 0.
    auto load = [&](int c) {
      if (c < chunks) {
        const int stage = c % CD_ROWS, vs = c % CD_VALUES, t0 = c * DC_T;
        for (int t = 0; t < DC_T; t++) {
          const size_t row = (size_t)(first + min(t0 + t, n - 1));
          if (4 * lane < dim) {
            dc_copy16((unsigned)__cvta_generic_to_shared(&sm.k[stage][t][4 * lane]), k + row * ldk + (size_t)kvh * dim + 4 * lane);
            dc_copy16((unsigned)__cvta_generic_to_shared(&sm.q[stage][t][4 * lane]), q + row * ldq + (size_t)kvh * dim + 4 * lane);
            dc_copy16((unsigned)__cvta_generic_to_shared(&sm.g[stage][t][4 * lane]), g + (row * heads + h) * dim + 4 * lane);
          }
        }
        const int vd = (lane % (CD_COLS / 8)) * 8;
        for (int t = lane / (CD_COLS / 8); t < DC_T; t += 32 / (CD_COLS / 8))
          if (col0 + vd < vdim)
            dc_copy16((unsigned)__cvta_generic_to_shared(&sm.v[vs][t][vd]), v + (size_t)(first + min(t0 + t, n - 1)) * ldv + (size_t)h * vdim + col0 + vd);
        if (lane < DC_T) sm.beta[vs][lane] = t0 + lane < n ? beta[(size_t)(first + t0 + lane) * heads + h] : 0.f;
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    load(0);
    for (int j = -3; j < chunks; j++) {
      __syncthreads();
      load(j + 4);                                      // (into the place of rows that were last read at step j - 1)
      asm volatile("cp.async.wait_group 1;\n" ::);      // chunk j + 3 is there at the next barrier
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    return;
  }
  if (warp >= CD_COL_WARPS && warp < CD_COL_WARPS + 2) {
    // ------------------------------------------------------------------------------------------ a and m of chunk j + 2
    for (int j = -3; j < chunks; j++) {
      __syncthreads();
      const int c = j + 2;
      if (c < 0 || c >= chunks) continue;
      cd_pairs<DIMP>(sm, c % CD_ROWS, c & 1, min(DC_T, n - c * DC_T), lane, warp - CD_COL_WARPS);
    }
    return;
  }
  if (warp >= CD_COL_WARPS + 2 && warp < CD_COL_WARPS + 4) {
    // ------------------------------------------------------------------------------------------ G k, G q, R k of chunk j + 1
    const int d = 2 * ((warp - CD_COL_WARPS - 2) * 32 + lane);      // two neighbouring channels a lane
    for (int j = -3; j < chunks; j++) {
      __syncthreads();
      const int c = j + 1;
      if (c < 0 || c >= chunks || d >= DIMP) continue;
      const int stage = c % CD_ROWS, buf = c & 1, nt = min(DC_T, n - c * DC_T);
      auto put = [&](bf16 (&to)[3][DC_T][DIMP + 8], int t, float x, float y) {
        uint32_t hi, mid, lo;
        dc_split(x, y, hi, mid, lo);
        *reinterpret_cast<uint32_t*>(&to[0][t][d]) = hi;
        *reinterpret_cast<uint32_t*>(&to[1][t][d]) = mid;
        *reinterpret_cast<uint32_t*>(&to[2][t][d]) = lo;
      };
      float2 G = make_float2(1.f, 1.f), R = G;
#pragma unroll 4
      for (int t = 0; t < DC_T; t++) {
        float2 kk = make_float2(0.f, 0.f), qq = kk;
        if (t < nt) {
          const float2 gg = *reinterpret_cast<const float2*>(&sm.g[stage][t][d]);
          kk = *reinterpret_cast<const float2*>(&sm.k[stage][t][d]);
          qq = *reinterpret_cast<const float2*>(&sm.q[stage][t][d]);
          G.x *= gg.x; G.y *= gg.y;
        }
        put(sm.K[buf], t, G.x * kk.x, G.y * kk.y);
        put(sm.Q[buf], t, G.x * qq.x, G.y * qq.y);
      }
      *reinterpret_cast<float2*>(&sm.gc[buf][d]) = G;
#pragma unroll 4
      for (int s = DC_T - 1; s >= 0; s--) {
        float2 kk = make_float2(0.f, 0.f), gg = make_float2(1.f, 1.f);
        if (s < nt) {
          kk = *reinterpret_cast<const float2*>(&sm.k[stage][s][d]);
          gg = *reinterpret_cast<const float2*>(&sm.g[stage][s][d]);
        }
        put(sm.W[buf], s, R.x * kk.x, R.y * kk.y);
        R.x *= gg.x; R.y *= gg.y;
      }
    }
    return;
  }
  if (warp == CD_COL_WARPS + 4) {
    // ------------------------------------------------------------------------------------------ T and m's terms of chunk j + 1
    for (int j = -3; j < chunks; j++) {
      __syncthreads();
      const int c = j + 1;
      if (c < 0 || c >= chunks) continue;
      const int buf = c & 1, vs = c % CD_VALUES;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int t = g8 + 8 * e;
        const float be = sm.beta[vs][t];
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const int s2 = 8 * x + 2 * t4;
          const float2 a = *reinterpret_cast<const float2*>(&sm.a[buf][t][s2]), m = *reinterpret_cast<const float2*>(&sm.m[buf][t][s2]);
          *reinterpret_cast<float2*>(&sm.A[t][s2]) = make_float2(be * a.x, be * a.y);      // (0 for s >= t)
          uint32_t hi, mid, lo;
          dc_split(m.x, m.y, hi, mid, lo);
          *reinterpret_cast<uint32_t*>(&sm.M[buf][0][t][s2]) = hi;
          *reinterpret_cast<uint32_t*>(&sm.M[buf][1][t][s2]) = mid;
          *reinterpret_cast<uint32_t*>(&sm.M[buf][2][t][s2]) = lo;
        }
      }
      __syncwarp();
      // column `lane` of T: T[t] = e_t - sum_{s < t} A[t][s] T[s]
      const int col = lane & 15;
      float T[DC_T];
#pragma unroll
      for (int t = 0; t < DC_T; t++) {
        float s0 = t == col ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
        for (int x = 0; x < t; x += 4) {
          const float4 A4 = *reinterpret_cast<const float4*>(&sm.A[t][x]);
          s0 = fmaf(-A4.x, T[x], s0);
          if (x + 1 < t) s1 = fmaf(-A4.y, T[x + 1], s1);
          if (x + 2 < t) s0 = fmaf(-A4.z, T[x + 2], s0);
          if (x + 3 < t) s1 = fmaf(-A4.w, T[x + 3], s1);
        }
        T[t] = s0 + s1;
      }
      if (lane < DC_T) {
#pragma unroll
        for (int t = 0; t < DC_T; t++) {
          const bf16 hi = __float2bfloat16_rn(T[t]);
          const float r1 = T[t] - __bfloat162float(hi);
          const bf16 mid = __float2bfloat16_rn(r1);
          sm.T[buf][0][t][col] = hi;
          sm.T[buf][1][t][col] = mid;
          sm.T[buf][2][t][col] = __float2bfloat16_rn(r1 - __bfloat162float(mid));
        }
      }
      __syncwarp();                                     // (A is written again by other lanes)
    }
    return;
  }

  // ---------------------------------------------------------------------------------------------- 16 columns of the state
  // where the lane's pieces of a B operand lie for ldmatrix (rows of n, k contiguous; and its transposed form)
  const int b_row = (lane & 7) + 8 * (lane >> 4), b_col = 8 * ((lane >> 3) & 1);
  const int bt_row = (lane & 7) + 8 * ((lane >> 3) & 1), bt_col = 8 * (lane >> 4);
  // acc[j]: S^T, rows (columns of S) c0 = g8 and c0 + 8, dims 8 j + 2 t4 and the next
  const int c0 = warp * 16 + g8;
  float* st = state + (((size_t)seq_slot[seq] * heads + h) * dim) * (size_t)vdim + col0 + c0;
  const bool in0 = col0 + c0 < vdim, in1 = col0 + c0 + 8 < vdim;
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; j++)
#pragma unroll
    for (int y = 0; y < 2; y++) {
      const int d = 8 * j + 2 * t4 + y;
      acc[j][y] = in0 && d < dim ? st[(size_t)d * vdim] : 0.f;
      acc[j][2 + y] = in1 && d < dim ? st[(size_t)d * vdim + 8] : 0.f;
    }
  for (int j = -3; j < 0; j++) __syncthreads();         // (the other warps' first chunks)
  for (int c = 0; c < chunks; c++) {
    __syncthreads();
    const int vs = c % CD_VALUES, buf = c & 1, t0 = c * DC_T;
    // (G k)^T S0 and (G q)^T S0, transposed: the largest terms' product apart from the small ones.  Products that add to one
    // sum wait for each other, so four sums take turns.
    float ph[2][4] = {}, pl[2][4] = {}, rh[2][4] = {}, rl[2][4] = {};
#pragma unroll
    for (int j = 0; j < KS; j++) {
      uint32_t hi[4], mid[4], lo[4], bk[3][4], bq[3][4];
#pragma unroll
      for (int m = 0; m < 3; m++) {
        dc_ldmatrix(bk[m], &sm.K[buf][m][b_row][j * 16 + b_col]);
        dc_ldmatrix(bq[m], &sm.Q[buf][m][b_row][j * 16 + b_col]);
      }
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int e = 0; e < 2; e++)
          dc_split(acc[2 * j + x][2 * e], acc[2 * j + x][2 * e + 1], hi[2 * x + e], mid[2 * x + e], lo[2 * x + e]);
      auto turn = [&](float (&p)[2][4], float (&r)[2][4], const uint32_t (&a)[4], int m) {
#pragma unroll
        for (int x = 0; x < 2; x++) {
          dc_mma(p[x], a, bk[m][2 * x], bk[m][2 * x + 1]);
          dc_mma(r[x], a, bq[m][2 * x], bq[m][2 * x + 1]);
        }
      };
      turn(pl, rl, lo, 0);
      turn(ph, rh, hi, 0);
      turn(pl, rl, hi, 2);
      turn(pl, rl, mid, 1);
      turn(pl, rl, mid, 0);
      turn(pl, rl, hi, 1);
    }
    // rhs^T: columns c0, c0 + 8; tokens 8 x + 2 t4, + 1; as A operand of U^T = rhs^T T^T
    uint32_t hi[4], mid[4], lo[4];
#pragma unroll
    for (int x = 0; x < 2; x++) {
      const int t = 8 * x + 2 * t4;
      const float be0 = sm.beta[vs][t], be1 = sm.beta[vs][t + 1];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const float v0 = __bfloat162float(sm.v[vs][t][c0 + 8 * e]), v1 = __bfloat162float(sm.v[vs][t + 1][c0 + 8 * e]);
        dc_split(be0 * (v0 - (ph[x][2 * e] + pl[x][2 * e])), be1 * (v1 - (ph[x][2 * e + 1] + pl[x][2 * e + 1])),
                 hi[2 * x + e], mid[2 * x + e], lo[2 * x + e]);
      }
    }
    auto product = [&](float (&o)[2][4], const bf16 (&B)[3][DC_T][CD_TROW]) {
      float small[2][4] = {};
      uint32_t b[2][3][2];
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int m = 0; m < 3; m++) {
          b[x][m][0] = *reinterpret_cast<const uint32_t*>(&B[m][8 * x + g8][2 * t4]);
          b[x][m][1] = *reinterpret_cast<const uint32_t*>(&B[m][8 * x + g8][2 * t4 + 8]);
        }
      auto turn = [&](float (&to)[2][4], const uint32_t (&a)[4], int m) {
#pragma unroll
        for (int x = 0; x < 2; x++) dc_mma(to[x], a, b[x][m][0], b[x][m][1]);
      };
      turn(small, lo, 0);
      turn(o, hi, 0);
      turn(small, hi, 2);
      turn(small, mid, 1);
      turn(small, mid, 0);
      turn(small, hi, 1);
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int e = 0; e < 4; e++) o[x][e] += small[x][e];
    };
    float U[2][4] = {};
    product(U, sm.T[buf]);
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int e = 0; e < 2; e++) dc_split(U[x][2 * e], U[x][2 * e + 1], hi[2 * x + e], mid[2 * x + e], lo[2 * x + e]);
    float o[2][4];
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int e = 0; e < 4; e++) o[x][e] = rh[x][e] + rl[x][e];
    product(o, sm.M[buf]);
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < 2; y++) {
        const int t = t0 + 8 * x + 2 * t4 + y;
        if (t < n) {
          float* dst = out + ((size_t)(first + t) * heads + h) * vdim + col0 + c0;
          if (in0) dst[0] = o[x][y];
          if (in1) dst[8] = o[x][2 + y];
        }
      }
    // S^T <- S^T diag(G_16) + U^T (R k)
#pragma unroll
    for (int j = 0; j < NT; j += 4) {
      uint32_t b[2][3][4];
      float add[4][4] = {};
#pragma unroll
      for (int y = 0; y < 2; y++)
#pragma unroll
        for (int m = 0; m < 3; m++) dc_ldmatrix_trans(b[y][m], &sm.W[buf][m][bt_row][(j + 2 * y) * 8 + bt_col]);
      auto turn = [&](const uint32_t (&a)[4], int m) {
#pragma unroll
        for (int x = 0; x < 4; x++) dc_mma(add[x], a, b[x >> 1][m][2 * (x & 1)], b[x >> 1][m][2 * (x & 1) + 1]);
      };
      turn(lo, 0);
      turn(hi, 2);
      turn(mid, 1);
      turn(mid, 0);
      turn(hi, 1);
      turn(hi, 0);
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const float2 G = *reinterpret_cast<const float2*>(&sm.gc[buf][8 * (j + x) + 2 * t4]);
        acc[j + x][0] = fmaf(G.x, acc[j + x][0], add[x][0]); acc[j + x][1] = fmaf(G.y, acc[j + x][1], add[x][1]);
        acc[j + x][2] = fmaf(G.x, acc[j + x][2], add[x][2]); acc[j + x][3] = fmaf(G.y, acc[j + x][3], add[x][3]);
      }
    }
  }
  cima_pdl_trigger();
#pragma unroll
  for (int j = 0; j < NT; j++)
#pragma unroll
    for (int y = 0; y < 2; y++) {
      const int d = 8 * j + 2 * t4 + y;
      if (in0 && d < dim) st[(size_t)d * vdim] = acc[j][y];
      if (in1 && d < dim) st[(size_t)d * vdim + 8] = acc[j][2 + y];
    }
}

template <int DIMP>
int launch_channel_delta(const float* q, int ldq, const float* k, int ldk, const void* v, int ldv, const float* g, const float* beta, float* state,
                         const int* seq_slot, const int* seq_first_row, float* out, int n_seqs, int heads, int kv_heads, int dim, int vdim,
                         cudaStream_t stream) {
  typedef CdShared<DIMP> Sh;
  static_assert(offsetof(Sh, q) % 16 == 0 && offsetof(Sh, g) % 16 == 0 && offsetof(Sh, v) % 16 == 0 && offsetof(Sh, K) % 16 == 0 && offsetof(Sh, Q) % 16 == 0 &&
                offsetof(Sh, W) % 16 == 0 && offsetof(Sh, T) % 4 == 0 && offsetof(Sh, M) % 4 == 0 && offsetof(Sh, a) % 8 == 0 && offsetof(Sh, m) % 8 == 0 &&
                offsetof(Sh, A) % 16 == 0 && offsetof(Sh, gc) % 8 == 0 && (DIMP + 8) * 2 % 16 == 0 && CD_VROW * 2 % 16 == 0,
                "what is read 16 (8, 4) bytes at a time starts there");
  constexpr size_t smem = sizeof(Sh);
  const cudaError_t e = cudaFuncSetAttribute(k_channel_delta<DIMP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cima_fail((int)e, "channel_delta: cannot raise shared memory to %zu bytes: %s", smem, cudaGetErrorString(e));
  const dim3 grid((vdim + CD_COLS - 1) / CD_COLS, heads, n_seqs);
  return cima_launch(k_channel_delta<DIMP>, grid, dim3(CD_THREADS), smem, stream, 1, q, ldq, k, ldk, (const bf16*)v, ldv, g, beta, state, seq_slot,
                     seq_first_row, out, heads, kv_heads, dim, vdim);
}
}  // namespace

// The delta rule of cima_recurrence for bfloat16 values, 16 tokens at a time: q, k float32 rows of kv_heads * dim values (strides in
// multiples of 4, 16-byte aligned), v bfloat16 rows of heads * vdim (stride and vdim multiples of 8), g [T, heads * dim], beta [T, heads],
// out [T, heads * vdim] float32; dim a multiple of 4, at most 128.
extern "C" int cima_channel_delta(const float* q, int ldq, const float* k, int ldk, const void* v, int ldv, const float* g, const float* beta,
                                  float* state, const int* seq_slot, const int* seq_first_row, float* out, int T, int n_seqs, int heads,
                                  int kv_heads, int dim, int vdim, cudaStream_t stream) {
  if (T <= 0 || n_seqs <= 0) return 0;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads > 65535 || n_seqs > 65535)
    return cima_fail(CIMA_E_SIZE, "channel_delta: %d heads on %d key heads in %d sequences are not accepted", heads, kv_heads, n_seqs);
  if (dim <= 0 || dim > 128 || dim % 4 || vdim <= 0 || vdim % 8) return cima_fail(CIMA_E_SIZE, "channel_delta: key size %d must be a multiple of 4 up to 128 and value size %d a multiple of 8", dim, vdim);
  if (!q || !k || !v || !g || !beta || !state || !out) return cima_fail(CIMA_E_ARG, "channel_delta: the rows, the state and the output are needed");
  if (ldq % 4 || ldk % 4 || ldv % 8 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)g) & 15))
    return cima_fail(CIMA_E_ARG, "channel_delta: rows of strides %d, %d and %d must start on 16 bytes", ldq, ldk, ldv);
  const int rc = dim <= 64 ? launch_channel_delta<64>(q, ldq, k, ldk, v, ldv, g, beta, state, seq_slot, seq_first_row, out, n_seqs, heads, kv_heads, dim, vdim, stream)
                           : launch_channel_delta<128>(q, ldq, k, ldk, v, ldv, g, beta, state, seq_slot, seq_first_row, out, n_seqs, heads, kv_heads, dim, vdim, stream);
  return rc ? rc : cima_launch_result();
}
