// Plain causal grouped-query attention, all sums in float32: the attention of the true 32-bit path (k_attention_f32, head sizes
// up to 256), and the fallback for head sizes that no other kernel takes (k_attention_plain: one warp per (query row, head),
// keys visited one by one with a running (max, sum, accumulator)).  Two sources of keys and values:
//   step  - the step's own qkv buffer (a prompt that starts at position 0: key j of a sequence is
//           its row j), used for prefill;
//   cache - the layer's pages through the slot's block table, used for decoding.
// Head h reads kv head h / (heads / kv_heads); score = q.k * scale; a query at position p sees
// keys j <= p, and with window w > 0 only p - j < w (src/kernels.cu:458-491, :700-712); with `keep_first` f > 0 the
// first f positions stay visible beyond the window (at their own positions).  `v_group` neighbouring key heads share
// one value head (1: a value head for every key head): value head = key head / v_group, and a row of the step holds
// nkv / v_group value heads behind its key heads.
// A head's softmax may hold one more entry without a value: `sink` entries of score 0, or exp(head_sink[h]).
// `gate_col` > 0: the row's own buffer holds a gate value for every value of the result from that column on (heads of hd
// values like the queries'); the result leaves times the gate's sigmoid.
// `slopes` (or null), one number a head: slopes[h] * (p - j) is taken off the scaled score of key j for a query at position p.
// A row's result depends only on its own sequence: same bits alone or in any batch.
#include "common.cuh"

template <typename TA, bool FROM_CACHE, int NI>       // NI: values of a head per lane (head_dim <= 32 NI)
__global__ void __launch_bounds__(128)
k_attention_plain(const TA* __restrict__ qkv, int ld, const TA* __restrict__ cache, CimaPaged pg,
                  const int* __restrict__ row_pos, const int* __restrict__ row_seq,
                  const int* __restrict__ seq_slot, const int* __restrict__ seq_first_row,
                  TA* __restrict__ out, int ldo, int T, int nh, int nkv, int hd, float scale, int window, float sink, int keep_first, int v_group,
                  const float* __restrict__ head_sink, int gate_col, const float* __restrict__ slopes) {
  cima_pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  const int h = blockIdx.y;
  if (row >= T) return;
  const int kvh = h / (nh / nkv);
  const int pos = row_pos[row];
  const int seq = row_seq[row];
  const int slot = FROM_CACHE ? seq_slot[seq] : 0;
  const int first = FROM_CACHE ? 0 : seq_first_row[seq];
  const int vh = kvh / v_group;
  const int kcol = (nh + kvh) * hd, vcol = (nh + nkv + vh) * hd;

  float q[NI], acc[NI];
  const TA* qp = qkv + (size_t)row * ld + (size_t)h * hd;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int d = lane + 32 * i;
    q[i] = d < hd ? cima_to_f32<TA>(qp[d]) : 0.f;
    acc[i] = 0.f;
  }
  const float slope = slopes ? slopes[h] : 0.f;
  float m = -1e30f, l = 0.f;
  const int lo = (window > 0 && pos + 1 > window) ? pos + 1 - window : 0;
  const int kept = min(keep_first, lo);         // the first positions that stay visible below the window
  for (int j = kept > 0 ? 0 : lo; j <= pos; j++) {
    if (j == kept && j < lo) j = lo;
    const TA *kp, *vp;
    if (FROM_CACHE) {
      kp = cache + pg.offset(slot, j, 0, kvh);
      vp = cache + pg.offset(slot, j, 1, vh);
    } else {
      kp = qkv + (size_t)(first + j) * ld + kcol;
      vp = qkv + (size_t)(first + j) * ld + vcol;
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int d = lane + 32 * i;
      if (d < hd) s = fmaf(q[i], cima_to_f32<TA>(kp[d]), s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s = s * scale - slope * (float)(pos - j);
    const float m2 = fmaxf(m, s);
    const float corr = expf(m - m2), p = expf(s - m2);
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int d = lane + 32 * i;
      if (d < hd) acc[i] = acc[i] * corr + p * cima_to_f32<TA>(vp[d]);
    }
    l = l * corr + p;
    m = m2;
  }
  TA* op = out + (size_t)row * ldo + (size_t)h * hd;
  // `sink` entries of score 0 that carry no value (0: an ordinary softmax); or, with `head_sink`, one entry whose score is
  // the head's own number (neither scaled nor attached to a value)
  // (without either nothing is added: the exponential of a low maximum is infinite, and 0 times that no number)
  if (head_sink) l += expf(head_sink[h] - m);
  else if (sink != 0.f) l += sink * expf(-m);
  const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int d = lane + 32 * i;
    if (d < hd) {
      const float gate = gate_col > 0 ? cima_sigmoid(cima_to_f32<TA>(qkv[(size_t)row * ld + gate_col + (size_t)h * hd + d])) : 1.0f;
      op[d] = cima_from_f32<TA>(acc[i] * inv * gate);
    }
  }
}

// ---------------------------------------------------------------------------------------------------- float32, head sizes up to 256
// The attention of the 32-bit path.  Keys are taken in pieces of 32 neighbouring positions (32 b .. 32 b + 31): a piece has a
// maximum, a sum and a weighted sum of values of its own, added up in ascending position, and the pieces are merged in
// ascending b.  A result therefore depends on its own sequence and position only, whoever computes it: the same bits whole,
// token by token or in a batch, from the step's rows or from pages.  (A warp that walked one key after another took 294 us at
// 200 positions, a chain of some 1.4 us a key; bound by latency.)
//
// A block owns up to QV query vectors of one sequence and key head: neighbouring rows times the heads that share the key head,
// so that a piece's keys and values serve them all.  Its teams of warps take the pieces in turn, each team through its own shared
// memory (cp.async), a lane a key for the scores and a lane NI dims for the weighted sums, the vectors in eights over the team's
// warps; what a round of pieces gives is merged by the block in their order.  Rows, teams and warps a team: launch_attention_f32.
// Measured, us (a warp that walks one key after another): 14 heads of 64 on 2, one row at 100 positions 11.8 (75), at 1,000: 43 (721), two
// prompts of 200 rows 57 (135), one of 1,000: 304 (1,171).  A sequence of a dozen positions or fewer does not repay a piece's own chain: one
// row at 8 positions 10 (8.7), a prompt of 5 rows 8.9 (5.4); it stays here, as its later rows' bits follow from this order.
constexpr int AF_KEYS = 32;

struct AfArgs {
  const float *qkv, *cache, *head_sink, *slopes;
  const int *row_pos, *row_seq, *seq_slot, *seq_first_row;
  float* out;
  CimaPaged pg;
  int ld, ldo, T, nh, nkv, hd, window, keep_first, v_group, gate_col, rows, heads, team;      // a block's rows, and heads of a key head; warps of a team
  float scale, sink;
};

template <int HDP> constexpr int AF_QV = HDP <= 64 ? 32 : HDP <= 128 ? 24 : 16;
template <int HDP> constexpr int AF_THREADS = HDP <= 128 ? 256 : 128;
static size_t af_smem(int hdp, int teams, int team, int qv) {
  return sizeof(float) * ((size_t)teams * 2 * AF_KEYS * (hdp + 4) + (size_t)2 * qv * hdp + (size_t)teams * qv * (hdp + 4) + (size_t)teams * team * 8 * AF_KEYS);
}

template <int HDP, bool FROM_CACHE, bool VEC>
__global__ void __launch_bounds__(AF_THREADS<HDP>)
k_attention_f32(const __grid_constant__ AfArgs a) {
  constexpr int NI = HDP / 32, PITCH = HDP + 4, QVM = AF_QV<HDP>;
  extern __shared__ __align__(16) float af[];
  __shared__ float s_m[8][QVM], s_l[8][QVM], s_c[8][QVM], s_k[8][QVM], run_m[QVM], run_l[QVM];
  __shared__ int s_any[8][QVM];
  cima_pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  const int teams = warps / a.team, slot_of = warp / a.team, member = warp - slot_of * a.team;
  const int group = a.nh / a.nkv, per_kv = (group + a.heads - 1) / a.heads;      // blocks of heads of one key head
  const int kvh = blockIdx.y / per_kv, h0 = kvh * group + (blockIdx.y % per_kv) * a.heads;
  const int heads = min(a.heads, (kvh + 1) * group - h0), vh = kvh / a.v_group;
  const int qvs_max = a.rows * a.heads, hd = a.hd, hdr = (hd + 3) & ~3;
  float* Kt = af + (size_t)slot_of * 2 * AF_KEYS * PITCH;
  float* Vt = Kt + AF_KEYS * PITCH;
  float* Q = af + (size_t)teams * 2 * AF_KEYS * PITCH;          // [qv][HDP]
  float* O = Q + (size_t)qvs_max * HDP;                          // [qv][HDP], the running weighted sums
  float* part = O + (size_t)qvs_max * HDP;                       // [team][qv][PITCH], a round's pieces
  float* P = part + (size_t)teams * qvs_max * PITCH + (size_t)warp * 8 * AF_KEYS;      // [8][32], the warp's weights
  const int t0 = blockIdx.x * a.rows, t1 = min(a.T, t0 + a.rows);

  for (int r0 = t0; r0 < t1;) {                          // rows of one sequence at a time
    const int seq = a.row_seq[r0];
    int r1 = r0 + 1;
    while (r1 < t1 && a.row_seq[r1] == seq) r1++;
    const int qvs = (r1 - r0) * heads;                   // vector i: row r0 + i / heads, head h0 + i % heads
    const int slot = FROM_CACHE ? a.seq_slot[seq] : 0, first = FROM_CACHE ? 0 : a.seq_first_row[seq];
    int pmin = a.row_pos[r0], pmax = pmin;
    for (int r = r0 + 1; r < r1; r++) { const int p = a.row_pos[r]; pmin = min(pmin, p); pmax = max(pmax, p); }
    const int lo = a.window > 0 && pmin + 1 > a.window ? pmin + 1 - a.window : 0, kept = min(a.keep_first, lo);
    const int b0 = lo / AF_KEYS, kept_pieces = min((kept + AF_KEYS - 1) / AF_KEYS, b0), pieces = kept_pieces + pmax / AF_KEYS - b0 + 1;
    __syncthreads();                                     // the sequence before is done with Q, O and the running sums
    for (int i = tid; i < qvs * HDP; i += blockDim.x) {
      const int v = i / HDP, d = i - v * HDP;
      Q[i] = d < hd ? a.qkv[(size_t)(r0 + v / heads) * a.ld + (size_t)(h0 + v % heads) * hd + d] : 0.f;
      O[i] = 0.f;
    }
    for (int i = tid; i < qvs; i += blockDim.x) { run_m[i] = -1e30f; run_l[i] = 0.f; }
    __syncthreads();
    for (int base = 0; base < pieces; base += teams) {
      const int mine = base + slot_of;
      const int b = mine < kept_pieces ? mine : b0 + mine - kept_pieces;
      const int j = b * AF_KEYS + lane;
      // what no row sees is not read (pages may hold anything there), and its place in shared memory not used
      const bool seen = mine < pieces && j <= pmax && (j >= lo || j < kept);
      const unsigned have = __ballot_sync(0xffffffffu, seen);
      const int keys = 32 - __clz(have);                 // behind the last one that is seen
      if (mine < pieces) {
        const float *kp = nullptr, *vp = nullptr;
        if (seen) {
          if (FROM_CACHE) {
            const size_t at = a.pg.offset(slot, j, 0, kvh);
            kp = a.cache + at;
            vp = vh == kvh ? kp + a.pg.value_offset() : a.cache + a.pg.offset(slot, j, 1, vh);
          } else {
            kp = a.qkv + (size_t)(first + j) * a.ld + (size_t)(a.nh + kvh) * hd;
            vp = a.qkv + (size_t)(first + j) * a.ld + (size_t)(a.nh + a.nkv + vh) * hd;
          }
        }
        auto bring = [&](int key) {
          const float* ks = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(kp), key));
          const float* vs = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(vp), key));
          const bool ok = have >> key & 1;
          if constexpr (VEC) {
            for (int d = 4 * lane; d < HDP; d += 128) {
              if (ok && d < hd) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(Kt + key * PITCH + d)), "l"(ks + d));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(Vt + key * PITCH + d)), "l"(vs + d));
              } else {
                *reinterpret_cast<float4*>(Kt + key * PITCH + d) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(Vt + key * PITCH + d) = make_float4(0.f, 0.f, 0.f, 0.f);
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < NI; i++) {
              const int d = lane + 32 * i;
              Kt[key * PITCH + d] = ok && d < hd ? ks[d] : 0.f;
              Vt[key * PITCH + d] = ok && d < hd ? vs[d] : 0.f;
            }
          }
        };
        if (a.team == 1 && keys == AF_KEYS) {
          for (int key = 0; key < AF_KEYS; key++) bring(key);
        } else {
          for (int key = member; key < keys; key += a.team) bring(key);
        }
        if constexpr (VEC) asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
      }
      if (a.team > 1) __syncthreads();
      else __syncwarp();
      if (mine < pieces) {
        float* mypart = part + (size_t)slot_of * qvs_max * PITCH;
        for (int v0 = 8 * member; v0 < qvs; v0 += 8 * a.team) {      // eight query vectors at a time
          float s[8];
          const float* q[8];
#pragma unroll
          for (int x = 0; x < 8; x++) { s[x] = 0.f; q[x] = Q + (size_t)min(v0 + x, qvs - 1) * HDP; }
#pragma unroll 2
          for (int d = 0; d < hdr; d += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(Kt + lane * PITCH + d);
#pragma unroll
            for (int x = 0; x < 8; x++) {
              const float4 q4 = *reinterpret_cast<const float4*>(q[x] + d);
              s[x] = fmaf(q4.x, k4.x, s[x]); s[x] = fmaf(q4.y, k4.y, s[x]);
              s[x] = fmaf(q4.z, k4.z, s[x]); s[x] = fmaf(q4.w, k4.w, s[x]);
            }
          }
          unsigned vis[8], all = 0xffffffffu;
#pragma unroll
          for (int x = 0; x < 8; x++) {
            const int v = min(v0 + x, qvs - 1), h = h0 + v % heads, pos = a.row_pos[r0 + v / heads];
            const int from = a.window > 0 && pos + 1 > a.window ? pos + 1 - a.window : 0;
            const bool see = j <= pos && (j >= from || j < a.keep_first);
            s[x] = s[x] * a.scale - (a.slopes ? a.slopes[h] : 0.f) * (float)(pos - j);
            vis[x] = __ballot_sync(0xffffffffu, see);
            all &= vis[x];
            float m = see ? fmaxf(s[x], -1e30f) : -1e30f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const float p = see ? expf(s[x] - m) : 0.f;
            float l = p;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            P[x * AF_KEYS + lane] = p;
            if (lane == 0 && v0 + x < qvs) { s_m[slot_of][v] = m; s_l[slot_of][v] = l; s_any[slot_of][v] = vis[x] != 0u; }
          }
          __syncwarp();
          float o[8][NI];
#pragma unroll
          for (int x = 0; x < 8; x++)
#pragma unroll
            for (int i = 0; i < NI; i++) o[x][i] = 0.f;
          auto weigh = [&](int k, bool whole) {
            float vv[4][NI];
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
              for (int i = 0; i < NI; i++) vv[e][i] = Vt[(k + e) * PITCH + lane + 32 * i];
#pragma unroll
            for (int x = 0; x < 8; x++) {
              const float4 p4 = *reinterpret_cast<const float4*>(P + x * AF_KEYS + k);
              const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
              for (int e = 0; e < 4; e++)
                if (whole || (vis[x] >> (k + e) & 1)) {
#pragma unroll
                  for (int i = 0; i < NI; i++) o[x][i] = fmaf(p[e], vv[e][i], o[x][i]);
                }
            }
          };
          if (all == 0xffffffffu) {
#pragma unroll 2
            for (int k = 0; k < AF_KEYS; k += 4) weigh(k, true);
          } else {                                       // a value that the row does not see stays out, whatever it is
#pragma unroll 1
            for (int k = 0; k < keys; k += 4) weigh(k, false);
          }
#pragma unroll
          for (int x = 0; x < 8; x++)
            if (v0 + x < qvs) {
#pragma unroll
              for (int i = 0; i < NI; i++) mypart[(size_t)(v0 + x) * PITCH + lane + 32 * i] = o[x][i];
            }
          __syncwarp();                                  // the weights have been read
        }
      }
      __syncthreads();
      const int there = min(teams, pieces - base);
      for (int v = tid; v < qvs; v += blockDim.x) {      // the factors of the round's pieces, in their order
        float m = run_m[v], l = run_l[v];
        for (int w = 0; w < there; w++) {
          float c = 1.f, k = 0.f;
          if (s_any[w][v]) {
            const float m2 = fmaxf(m, s_m[w][v]);
            c = expf(m - m2); k = expf(s_m[w][v] - m2);
            l = l * c + s_l[w][v] * k;
            m = m2;
          }
          s_c[w][v] = c; s_k[w][v] = k;
        }
        run_m[v] = m; run_l[v] = l;
      }
      __syncthreads();
      for (int i = tid; i < qvs * HDP; i += blockDim.x) {
        const int v = i / HDP, d = i - v * HDP;
        float acc = O[i];
        for (int w = 0; w < there; w++)
          if (s_any[w][v]) acc = fmaf(part[((size_t)w * qvs_max + v) * PITCH + d], s_k[w][v], acc * s_c[w][v]);
        O[i] = acc;
      }
      __syncthreads();
    }
    for (int i = tid; i < qvs * HDP; i += blockDim.x) {
      const int v = i / HDP, d = i - v * HDP;
      if (d >= hd) continue;
      const int row = r0 + v / heads, h = h0 + v % heads;
      const float m = run_m[v];
      float l = run_l[v];
      if (a.head_sink) l += expf(a.head_sink[h] - m);
      else if (a.sink != 0.f) l += a.sink * expf(-m);    // (see k_attention_plain)
      const float gate = a.gate_col > 0 ? cima_sigmoid(a.qkv[(size_t)row * a.ld + a.gate_col + (size_t)h * hd + d]) : 1.0f;
      a.out[(size_t)row * a.ldo + (size_t)h * hd + d] = O[i] * (l > 0.f ? 1.0f / l : 0.f) * gate;
    }
    r0 = r1;
  }
}

// The same sums for steps of few rows (a decode step), head sizes 64 and 128, all keys visible below a row's position but for a window's.
// A block owns ONE head of one row, a warp a piece, its keys and values straight to registers: a lane a key for the scores, a lane
// HD / 32 neighbouring dims for the weighted sum.  What bounds such a step is the chain and not the bytes: the kernel above takes
// 13 us for one or two rows at 200 positions, most of it the pieces' way through shared memory and the seven heads of a key
// head one after the other; here each head has a block, and its keys are read from L2 as often as heads share them.  The order of
// every sum is the other kernel's.  Measured, us a decode step of the 0.5B shape in 32 bits, the kernel above / this one: one row at
// 10 / 1,000 / 8,000 positions 1,332 / 1,190, 2,151 / 1,601, 8,998 / 5,067, two at 205 1,428 / 1,260, 8 at 300 1,824 / 1,550, 20 at 1,500
// 4,498 / 3,948.
// (Volatile, so that a batch of loads stays in front of the sums it is asked for: left to the compiler, each waits for its own.)
__device__ __forceinline__ float4 ld_f4(const float* p, bool ok) {
  float4 v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %5, 0;\nmov.b32 %0, 0;\nmov.b32 %1, 0;\nmov.b32 %2, 0;\nmov.b32 %3, 0;\n@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"
               : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w) : "l"(p), "r"((int)ok));
  return v;
}
__device__ __forceinline__ float2 ld_f2(const float* p, bool ok) {
  float2 v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %3, 0;\nmov.b32 %0, 0;\nmov.b32 %1, 0;\n@p ld.global.v2.f32 {%0, %1}, [%2];\n}\n"
               : "=&f"(v.x), "=&f"(v.y) : "l"(p), "r"((int)ok));
  return v;
}
template <int HD>
__global__ void __launch_bounds__(256)
k_attention_f32_row(const __grid_constant__ AfArgs a) {
  constexpr int NI = HD / 32, PARTS = HD / 64, BATCH = AF_KEYS / PARTS;      // K in pieces of 64 dims, V in batches of so many keys
  __shared__ __align__(16) float q[HD];
  __shared__ float part[8][HD], s_m[8], s_l[8];
  __shared__ int s_any[8];
  cima_pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = blockIdx.x, h = blockIdx.y, kvh = h / (a.nh / a.nkv);
  const int pos = a.row_pos[row], slot = a.seq_slot[a.row_seq[row]];
  const int lo = a.window > 0 && pos + 1 > a.window ? pos + 1 - a.window : 0, b0 = lo / AF_KEYS, pieces = pos / AF_KEYS - b0 + 1;
  if (tid < HD) q[tid] = a.qkv[(size_t)row * a.ld + (size_t)h * HD + tid];
  __syncthreads();
  float m = -1e30f, l = 0.f, acc = 0.f;                  // of dim `tid`, over the pieces so far
  for (int base = 0; base < pieces; base += 8) {
    if (base + warp < pieces) {
      const int j0 = (b0 + base + warp) * AF_KEYS, j = j0 + lane;
      const bool see = j <= pos && j >= lo;
      const unsigned vis = __ballot_sync(0xffffffffu, see);
      const float* kp = a.cache + a.pg.offset(slot, j0, 0, kvh);      // (a piece lies in one page)
      const float* vp = kp + a.pg.value_offset() + NI * lane;
      kp += (size_t)lane * HD;
      float s = 0.f;
      float v[BATCH][NI];
      auto values = [&](int from) {
#pragma unroll
        for (int k = 0; k < BATCH; k++) {
          const bool ok = vis >> (from + k) & 1;         // (what no row sees is not read)
          if constexpr (NI == 2) {
            const float2 x = ld_f2(vp + (size_t)(from + k) * HD, ok);
            v[k][0] = x.x; v[k][1] = x.y;
          } else {
            const float4 x = ld_f4(vp + (size_t)(from + k) * HD, ok);
            v[k][0] = x.x; v[k][1] = x.y; v[k][2] = x.z; v[k][3] = x.w;
          }
        }
      };
#pragma unroll 1
      for (int part0 = 0; part0 < HD; part0 += 64) {
        float4 k4[16];
#pragma unroll
        for (int i = 0; i < 16; i++) k4[i] = ld_f4(kp + part0 + 4 * i, see);
        if (part0 + 64 == HD) values(0);                 // on their way while the scores are made
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const float4 q4 = *reinterpret_cast<const float4*>(q + part0 + 4 * i);
          s = fmaf(q4.x, k4[i].x, s); s = fmaf(q4.y, k4[i].y, s);
          s = fmaf(q4.z, k4[i].z, s); s = fmaf(q4.w, k4[i].w, s);
        }
      }
      s *= a.scale;
      float mp = see ? fmaxf(s, -1e30f) : -1e30f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, o));
      const float p = see ? expf(s - mp) : 0.f;
      float lp = p;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) lp += __shfl_xor_sync(0xffffffffu, lp, o);
      float o[NI];
#pragma unroll
      for (int i = 0; i < NI; i++) o[i] = 0.f;
#pragma unroll
      for (int from = 0; from < AF_KEYS; from += BATCH) {
        if (from > 0) values(from);
#pragma unroll
        for (int k = 0; k < BATCH; k++) {
          const float pk = __shfl_sync(0xffffffffu, p, from + k);
          if (vis >> (from + k) & 1) {
#pragma unroll
            for (int i = 0; i < NI; i++) o[i] = fmaf(pk, v[k][i], o[i]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < NI; i++) part[warp][NI * lane + i] = o[i];
      if (lane == 0) { s_m[warp] = mp; s_l[warp] = lp; s_any[warp] = vis != 0u; }
    }
    __syncthreads();
    if (tid < HD) {
      const int there = min(8, pieces - base);
      for (int w = 0; w < there; w++)
        if (s_any[w]) {
          const float m2 = fmaxf(m, s_m[w]), c = expf(m - m2), k = expf(s_m[w] - m2);
          l = l * c + s_l[w] * k;
          m = m2;
          acc = fmaf(part[w][tid], k, acc * c);
        }
    }
    __syncthreads();
  }
  if (tid < HD) a.out[(size_t)row * a.ldo + (size_t)h * HD + tid] = acc * (l > 0.f ? 1.0f / l : 0.f);
}

// max_keys: positions of the longest sequence after the step.  The bits do not depend on rows, teams or warps.
template <int HDP, bool FROM_CACHE>
static int launch_attention_f32(AfArgs a, bool vec, int n_seqs, int max_keys, cudaStream_t stream) {
  const int group = a.nh / a.nkv;
  a.heads = group < AF_QV<HDP> ? group : AF_QV<HDP>;
  const int per_kv = (group + a.heads - 1) / a.heads;
  // Few rows: a row a block, so that rows do not wait for one another; many: as many rows as share a block's keys, and no more than a
  // sequence has (64 sequences' decode rows in blocks of 32 took 917 us, one after another in each block; 201 so).
  const bool few = (long long)a.T * a.nkv * per_kv <= 592;
  const int vectors = AF_QV<HDP>;
  const int average = (a.T + n_seqs - 1) / n_seqs, most = max(1, vectors / a.heads), parts = (average + most - 1) / most;
  a.rows = few ? 1 : (average + parts - 1) / parts;
  // A team a piece, no more than there are pieces (a team's shared memory is another block's: 16 prompts of 20 rows, 32 heads of 64, took 148 us; 29 so),
  // and the spare warps are the teams': they share its loads and vectors.
  int teams = HDP <= 64 ? (few ? 8 : 4) : HDP <= 128 ? 4 : 2;
  while (teams > 1 && (teams - 1) * AF_KEYS >= max_keys) teams--;
  for (;; teams--) {
    a.team = AF_THREADS<HDP> / 32 / teams;
    if (teams == 1 || af_smem(HDP, teams, a.team, a.rows * a.heads) <= 220 * 1024) break;
  }
  const int warps = teams * a.team;
  const size_t smem = af_smem(HDP, teams, a.team, a.rows * a.heads);
  auto kern = vec ? k_attention_f32<HDP, FROM_CACHE, true> : k_attention_f32<HDP, FROM_CACHE, false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cima_fail((int)e, "attention_plain: %zu bytes of shared memory are not available: %s", smem, cudaGetErrorString(e));
  const dim3 grid((unsigned)((a.T + a.rows - 1) / a.rows), (unsigned)(a.nkv * per_kv));
  return cima_launch(kern, grid, dim3(32 * warps), smem, stream, 1, a);
}

// from_cache 0: keys/values of the step (seq_first_row needed); 1: of the cache (table, seq_slot needed).
// n_seqs: sequences of the step; max_keys: positions of the longest after it (0: not known).  Neither changes a result.
extern "C" int cima_attention_plain(const void* qkv, int dtype, int ld, const void* cache, const int* table,
                                    int table_width, int ring, int page_size, const int* row_pos,
                                    const int* row_seq, const int* seq_slot, const int* seq_first_row, void* out,
                                    int ldo, int T, int nh, int nkv, int hd, float scale, int window,
                                    int from_cache, int planes, float sink, int keep_first, int v_group, const float* head_sink,
                                    int gate_col, const float* slopes, int n_seqs, int max_keys, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (hd <= 0 || hd > 1024) return cima_fail(CIMA_E_SIZE, "attention_plain: head_dim %d is outside 1..1024", hd);
  if (planes != 1 && planes != 2) return cima_fail(CIMA_E_ARG, "attention_plain: %d planes; pages hold keys | values (2) or one shared vector (1)", planes);
  if (nh <= 0 || nkv <= 0 || nh % nkv) return cima_fail(CIMA_E_SIZE, "attention_plain: %d heads are not a multiple of %d kv heads", nh, nkv);
  if (nh > 65535) return cima_fail(CIMA_E_SIZE, "attention_plain: %d heads exceed one launch", nh);
  if (keep_first < 0 || v_group < 1 || nkv % v_group) return cima_fail(CIMA_E_ARG, "attention_plain: keep_first %d must not be negative and %d kv heads be a multiple of v_group %d", keep_first, nkv, v_group);
  if (from_cache && (!cache || !table)) return cima_fail(CIMA_E_ARG, "attention_plain: decoding needs the cache and its block table");
  if (gate_col < 0 || (gate_col > 0 && gate_col + nh * hd > ld)) return cima_fail(CIMA_E_ARG, "attention_plain: %d gate values from column %d on exceed the rows of %d", nh * hd, gate_col, ld);
  CimaPaged pg{table, table_width, ring, page_size, nkv, hd, planes};
  if (n_seqs <= 0) n_seqs = T;
  if (max_keys <= 0) max_keys = from_cache ? 0x7fffffff : T;
  if (dtype == CIMA_F32 && hd <= 256) {
    AfArgs a{(const float*)qkv, (const float*)cache, head_sink, slopes, row_pos, row_seq, seq_slot, seq_first_row, (float*)out, pg,
             ld, ldo, T, nh, nkv, hd, window, keep_first, v_group, gate_col, 1, 1, 1, scale, sink};
    const bool vec = hd % 4 == 0 && (from_cache || ld % 4 == 0) && ((from_cache ? (uintptr_t)cache : (uintptr_t)qkv) & 15) == 0;
    int rc;
    // One head of one row a block up to 296 of them, two an SM at head size 64 (98 registers); at 128 (170 registers) an SM holds one and more
    // than 148 run in two waves, which still beat the other kernel at every length.  us a layer against it at 10 / 100 / 1,000 / 8,000 positions:
    // 280 blocks of 64 (20 rows of 14 heads) -4.7 / -5.8 / -16 / -116, 288 of 128 (24 rows of 12 heads) -3.4 / -1.5 / -23 / -161, 280 of 128
    // (10 rows of 28 heads) -7.1 / -2.8 / -27 / -186; with one long row beside short ones more.  336 lose (64: 1,000 positions +8.4,
    // 8,000 +105; 128: 100 positions +3.1, 8,000 +118): there the heads that share keys share a block.
    if (from_cache && (hd == 64 || hd == 128) && (long long)T * nh <= 296 && T <= n_seqs && page_size % AF_KEYS == 0 && planes == 2 && ((uintptr_t)cache & 15) == 0 &&
        sink == 0.f && keep_first == 0 && v_group == 1 && !head_sink && gate_col == 0 && !slopes) {
      rc = hd == 64 ? cima_launch(k_attention_f32_row<64>, dim3(T, nh), dim3(256), (size_t)0, stream, 1, a) : cima_launch(k_attention_f32_row<128>, dim3(T, nh), dim3(256), (size_t)0, stream, 1, a);
      return rc ? rc : cima_launch_result();
    }
    if (hd <= 64) rc = from_cache ? launch_attention_f32<64, true>(a, vec, n_seqs, max_keys, stream) : launch_attention_f32<64, false>(a, vec, n_seqs, max_keys, stream);
    else if (hd <= 128) rc = from_cache ? launch_attention_f32<128, true>(a, vec, n_seqs, max_keys, stream) : launch_attention_f32<128, false>(a, vec, n_seqs, max_keys, stream);
    else rc = from_cache ? launch_attention_f32<256, true>(a, vec, n_seqs, max_keys, stream) : launch_attention_f32<256, false>(a, vec, n_seqs, max_keys, stream);
    return rc ? rc : cima_launch_result();
  }
  dim3 grid((T + 3) / 4, nh);
#define LAUNCH_NI(TA, FC, NI) cima_launch(k_attention_plain<TA, FC, NI>, dim3(grid), dim3(128), (size_t)(0), stream, 1, (const TA*)qkv, ld, (const TA*)cache, pg, \
    row_pos, row_seq, seq_slot, seq_first_row, (TA*)out, ldo, T, nh, nkv, hd, scale, window, sink, keep_first, v_group, head_sink, gate_col, slopes)
  int rc;
  if (dtype == CIMA_F32) rc = from_cache ? LAUNCH_NI(float, true, 32) : LAUNCH_NI(float, false, 32);
  else if (dtype != CIMA_BF16) return cima_fail(CIMA_E_DTYPE, "attention_plain: dtype code %d is neither float32 nor bfloat16", dtype);
  else if (hd <= 256) rc = from_cache ? LAUNCH_NI(__nv_bfloat16, true, 8) : LAUNCH_NI(__nv_bfloat16, false, 8);
  else rc = from_cache ? LAUNCH_NI(__nv_bfloat16, true, 32) : LAUNCH_NI(__nv_bfloat16, false, 32);
  if (rc) return rc;
#undef LAUNCH_NI
  return cima_launch_result();
}
