// The linear scan of sequence_state.cu over prompt portions, sixteen tokens at a time, and over single tokens (at the end):
//
//   S_t = D_t S_(t-1) + k_t u_t^T,  o_t = S_t^T q_t          per request and head, S is [d, dv], float32
//   u_t = v_t, gain_t v_t (row gates), or beta_t (v_t - (D_t S_(t-1))^T k_t) (delta rule)
//
// Token after token a scan is a chain of dependent steps: a few instructions, a shuffle tree, 0.27 to 0.47 us a token.  Cut
// into chunks of C = 16 tokens with S_0 the state before a chunk, G_t = D_t ... D_1 and E_s = D_C ... D_(s+1):
//
//   o_t = (G_t q_t)^T S_0 + sum_(s <= t) A_ts u_s,            A_ts = q_t . (D_t ... D_(s+1) k_s)
//   S_C = G_C S_0 + sum_s (E_s k_s) u_s^T
//   delta rule: w_t = v_t - (G_t k_t)^T S_0,  u_t = sum_(s <= t) T_ts w_s,   T = (I + tril(beta B, -1))^-1 diag(beta),
//               B_ts = k_t . (D_t ... D_(s+1) k_s)            (the forward substitution of u_t, its steps gathered in T)
//
// Only products of decays between two tokens of a chunk are formed, never a quotient of two, so nothing overflows that
// the recurrence does not, and every sum is over float32 products of float32 factors.  What does not depend on the
// state is made for all chunks at once by a first kernel: per chunk and head a record of G_t q_t, E_s k_s, (G_t k_t,) A, (T)
// and G_C, in float32.  The second walks the chunks.
#include "common.cuh"

namespace b200 {

constexpr int kChunkTokens = 16;
constexpr int kChunkCols = 32;           // value columns a CTA owns
constexpr int kChunkMaxDim = 128;

enum ChunkGate : int { CHUNK_HEAD = 0, CHUNK_CHANNEL = 1, CHUNK_ROW = 2, CHUNK_TOKEN = 3 };

struct ChunkParams {
  const void* q; const void* k; const void* v;
  int ldq, ldk, ldv;
  const float* gate;                               // [n, H * d] (channel)
  const float* decay;                              // [H] (head)
  const float* row_decay; const float* row_gain;   // [n, H] (row: both; token: the first)
  const float* beta;                               // [n, H] (delta rule)
  float* state;                                    // [slots, H, d, dv]
  float* norm_state; float* norm_out;              // [slots, H, d], [n, H] (row)
  float* out;                                      // [n, H * dv]
  float* records;                                  // [chunks][H][record_floats]
  const int* q_start; const int* slots;
  int entries, H, Hqk, d, dp, dv, act;             // dp: d rounded up to 32, 64 or 128
  float q_scale;
  int skip, most;                                  // of every request: tokens before this launch's, tokens in it at most
};

// The rows of a request that a launch scans.
struct Portion { int first, count; };
__device__ __forceinline__ Portion portion_of(const ChunkParams& p, int entry) {
  const int first = p.q_start[entry], count = p.q_start[entry + 1] - first, skip = min(p.skip, count);
  return {first + skip, min(p.most, count - skip)};
}

// A record: Q [16][dp], K [16][dp], (KF [16][dp],) A [16][16], (T [16][16],) whole [dp].
__host__ __device__ constexpr int record_floats(int dp, bool delta) {
  return (delta ? 3 : 2) * kChunkTokens * dp + (delta ? 2 : 1) * kChunkTokens * kChunkTokens + dp;
}

// (as in sequence_state.cu: SiLU of a value that was stored in 16 bits with the hardware's exponential and reciprocal)
template <typename T> __device__ __forceinline__ float chunk_silu(float x) {
  if constexpr (sizeof(T) == 2) return __fdividef(x, 1.f + __expf(-x));
  else return x / (1.f + expf(-x));
}

// ---------------------------------------------------------------------------------------------------- the records
// One CTA per chunk and head.  A and B in sixteen blocks of four by four tokens, eight threads a block with a share of the
// channels each (four neighbouring ones at a time).  Decays of one number a token multiply the finished products.  Decays
// per channel: in a block on the diagonal k_s runs through the decays up to every t; below it q_t takes the decays from its
// block's first token on, k_s those up to its block's last, and the blocks between theirs, so that a product of decays is
// formed once a row and not once a pair.  The eight threads' sums are exchanged so that each finishes two pairs of tokens.
template <typename T, bool DELTA, int GATE>
__global__ void __launch_bounds__(128) scan_chunk_records_kernel(const ChunkParams p) {
  constexpr int C = kChunkTokens, D = kChunkMaxDim;
  __shared__ __align__(16) float qs[C][D], ks[C][D], gs[GATE == CHUNK_CHANNEL ? C : 1][D];
  __shared__ __align__(16) float block_decay[GATE == CHUNK_CHANNEL ? 4 : 1][D];
  __shared__ float as[C][C], bs[C][C], ts[C][C], alpha[C], gain[C], between[C][C];
  pdl_trigger();
  pdl_wait();
  int entry = 0, chunk = blockIdx.x, first = 0, count = 0;
  for (;; ++entry) {
    if (entry == p.entries) return;
    const Portion portion = portion_of(p, entry);
    first = portion.first;
    count = portion.count;
    const int chunks = (count + C - 1) / C;
    if (chunk < chunks) break;
    chunk -= chunks;
  }
  first += chunk * C;
  count = min(C, count - chunk * C);
  const int h = blockIdx.y, hqk = h / (p.H / p.Hqk), d = p.d, dp = p.dp, tid = threadIdx.x;
  const T* qg = static_cast<const T*>(p.q) + static_cast<size_t>(first) * p.ldq + hqk * d + tid;
  const T* kg = static_cast<const T*>(p.k) + static_cast<size_t>(first) * p.ldk + hqk * d + tid;
  const float* gg = p.gate + static_cast<size_t>(first) * p.H * d + h * d + tid;
  float* record = p.records + (static_cast<size_t>(blockIdx.x) * p.H + h) * record_floats(dp, DELTA);
  if (tid < C) {
    const size_t at = static_cast<size_t>(first + tid) * p.H + h;
    alpha[tid] = tid >= count ? 1.f : (GATE == CHUNK_HEAD ? p.decay[h] : GATE == CHUNK_CHANNEL ? 1.f : p.row_decay[at]);
    gain[tid] = tid >= count ? 0.f : (DELTA ? p.beta[at] : (GATE == CHUNK_ROW ? p.row_gain[at] : 1.f));
  }
  float q[C], k[C], g[GATE == CHUNK_CHANNEL ? C : 1];
  {
    T rq[C], rk[C];                 // all of a channel's rows are on their way before the first is used
#pragma unroll
    for (int t = 0; t < C; ++t) {
      const bool ok = t < count && tid < d;
      rq[t] = ok ? qg[static_cast<size_t>(t) * p.ldq] : from_float<T>(0.f);
      rk[t] = ok ? kg[static_cast<size_t>(t) * p.ldk] : from_float<T>(0.f);
      if (GATE == CHUNK_CHANNEL) g[t] = ok ? gg[static_cast<size_t>(t) * p.H * d] : 1.f;
    }
#pragma unroll
    for (int t = 0; t < C; ++t) {
      q[t] = to_float(rq[t]);
      k[t] = to_float(rk[t]);
      if (p.act) { q[t] = chunk_silu<T>(q[t]); k[t] = chunk_silu<T>(k[t]); }
      q[t] *= p.q_scale;
      qs[t][tid] = q[t];
      ks[t][tid] = k[t];
    }
  }
  if (GATE == CHUNK_CHANNEL) {
    float through = 1.f;
#pragma unroll
    for (int t = 0; t < C; ++t) {
      gs[t][tid] = g[t];
      through *= g[t];
      if (t % 4 == 3) {
        block_decay[t / 4][tid] = through;
        through = 1.f;
      }
    }
  }
  __syncthreads();
  if (tid < dp) {                   // the decays up to a token on q (and k), those behind it on k
    float* to = record + tid;
    float f = 1.f;
#pragma unroll
    for (int t = 0; t < C; ++t) {
      f *= GATE == CHUNK_CHANNEL ? g[GATE == CHUNK_CHANNEL ? t : 0] : alpha[t];
      to[t * dp] = q[t] * f;
      if (DELTA) to[(2 * C + t) * dp] = k[t] * f;
    }
    record[record_floats(dp, DELTA) - dp + tid] = f;
    f = 1.f;
#pragma unroll
    for (int t = C - 1; t >= 0; --t) {
      to[(C + t) * dp] = k[t] * (GATE == CHUNK_ROW ? f * gain[t] : f);
      f *= GATE == CHUNK_CHANNEL ? g[GATE == CHUNK_CHANNEL ? t : 0] : alpha[t];
    }
  }
  if (GATE != CHUNK_CHANNEL) {      // the decays between two tokens, times the earlier one's gain (row gates)
    for (int idx = tid; idx < C * C; idx += 128) {
      const int t = idx / C, s = idx % C;
      float g = GATE == CHUNK_ROW ? gain[s] : 1.f;
      for (int r = s + 1; r <= t; ++r) g *= alpha[r];
      between[t][s] = g;
    }
    __syncthreads();
  }
  const int ti = tid / 32, si = tid / 8 % 4, part = tid % 8;
  float a[16], b[DELTA ? 16 : 1];
#pragma unroll
  for (int v = 0; v < 16; ++v) {
    a[v] = 0.f;
    if (DELTA) b[v] = 0.f;
  }
  auto dot = [](const float4& x, const float4& y, float acc) { return fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, acc)))); };
  auto scale = [](float4& x, const float4& g) { x.x *= g.x; x.y *= g.y; x.z *= g.z; x.w *= g.w; };
  if (si <= ti) {
#pragma unroll 1
    for (int c = part * 4; c < d; c += 32) {            // channels from d on hold zeros
      float4 q[4], k[4], kq[DELTA ? 4 : 1];    // (rows of the tokens, not the channel's values above)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[i] = *reinterpret_cast<const float4*>(&qs[ti * 4 + i][c]);
        k[i] = *reinterpret_cast<const float4*>(&ks[si * 4 + i][c]);
        if (DELTA) kq[i] = *reinterpret_cast<const float4*>(&ks[ti * 4 + i][c]);
      }
      if (GATE == CHUNK_CHANNEL && ti == si) {
        float4 g[4];
#pragma unroll
        for (int i = 1; i < 4; ++i) g[i] = *reinterpret_cast<const float4*>(&gs[ti * 4 + i][c]);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          float4 run = k[s];
#pragma unroll
          for (int t = s; t < 4; ++t) {
            if (t > s) scale(run, g[t]);
            a[t * 4 + s] = dot(q[t], run, a[t * 4 + s]);
            if (DELTA) b[t * 4 + s] = dot(kq[t], run, b[t * 4 + s]);
          }
        }
        continue;
      }
      if (GATE == CHUNK_CHANNEL) {
        float4 g = make_float4(1.f, 1.f, 1.f, 1.f);
        for (int i = si + 1; i < ti; ++i) scale(g, *reinterpret_cast<const float4*>(&block_decay[i][c]));
#pragma unroll
        for (int s = 3; s >= 0; --s) {                  // behind token s up to its block's last, and through the blocks between
          scale(k[s], g);
          if (s > 0) scale(g, *reinterpret_cast<const float4*>(&gs[si * 4 + s][c]));
        }
        g = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          scale(g, *reinterpret_cast<const float4*>(&gs[ti * 4 + t][c]));
          scale(q[t], g);
          if (DELTA) scale(kq[t], g);
        }
      }
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          a[t * 4 + s] = dot(q[t], k[s], a[t * 4 + s]);
          if (DELTA) b[t * 4 + s] = dot(kq[t], k[s], b[t * 4 + s]);
        }
    }
  }
  auto share_out = [&](float (&x)[16]) -> int {         // the number of the first of the two sums that end up here, in x[0] and x[1]
    int held = 0;
#pragma unroll
    for (int o = 4, keep = 8; o > 0; o >>= 1, keep >>= 1) {
      const bool upper = (tid & o) != 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i < keep) {
          const float send = upper ? x[i] : x[i + keep];
          x[i] = (upper ? x[i + keep] : x[i]) + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      held += upper ? keep : 0;
    }
    return held;
  };
  const int held = share_out(a);
  if constexpr (DELTA) share_out(b);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = ti * 4 + (held + e) / 4, s = si * 4 + (held + e) % 4;
    const float g = GATE == CHUNK_CHANNEL ? 1.f : (s <= t ? between[t][s] : 0.f);
    as[t][s] = s <= t ? a[e] * g : 0.f;
    if (DELTA) bs[t][s] = s <= t ? b[e] * g : 0.f;
  }
  __syncthreads();
  if (DELTA && tid < C) {           // column tid of T, by forward substitution
    float x[C];
#pragma unroll
    for (int t = 0; t < C; ++t) {
      float sum = t == tid ? 1.f : 0.f;
#pragma unroll
      for (int s = 0; s < C; ++s)
        if (s < t && s >= tid) sum = fmaf(-bs[t][s], x[s], sum);
      x[t] = t < tid ? 0.f : gain[t] * sum;
      ts[t][tid] = x[t];
    }
  }
  __syncthreads();
  float* to = record + (DELTA ? 3 : 2) * C * dp;
  for (int idx = tid; idx < C * C; idx += 128) {
    to[idx] = as[idx / C][idx % C];
    if (DELTA) to[C * C + idx] = ts[idx / C][idx % C];
  }
}

// ---------------------------------------------------------------------------------------------------- the chunks
// One CTA per request, head and 32 value columns.  Warp w holds rows 16 w .. 16 w + 15 of the state, a lane four rows and
// four columns of them, in registers for the whole portion.  Records come two chunks ahead by asynchronous copies into a ring
// of three.  Per chunk:
//   every warp multiplies its rows of the state with all sixteen q (k); the lanes that share columns exchange sums, the
//   warps' sums meet in shared memory;
//   o and u are finished with A and T, a warp a token, a lane a column; the state takes its sixteen updates.
// Bound by the latency of a chunk's steps (two to four barriers; 2.2 us a chunk) and by the reads of shared memory beside
// them, where a value that all lanes read alike costs as much as one each: it meets four columns a lane.  With rows that
// this kernel's threads fetched and scaled themselves a chunk took 3.9 us.  2,048 tokens of 32 heads of 128 x 128, records and
// chunks: 39 + 280 us with one decay a head (685 token by token), 80 + 390 with the delta rule and decays per channel (958);
// three portions of 578 tokens: 46 + 164 with decays per channel (542), 33 + 212 with row gates (438).
// ROW: the normaliser is one more column, behind the last value column, whose value is 1 for every token.
constexpr int kRing = 3;
template <typename TV, bool DELTA, bool ROW, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) scan_chunk_kernel(const ChunkParams p) {
  constexpr int C = kChunkTokens, NC = kChunkCols, DP = WARPS * 16, THREADS = WARPS * 32, RECORD = record_floats(DP, DELTA);
  constexpr int VPT = C / WARPS;                        // value elements a thread stages, tokens it finishes
  extern __shared__ __align__(16) float smem[];
  float* ring = smem;                                   // [kRing][RECORD]
  float* vs = ring + kRing * RECORD;                    // [2][C][NC]
  float* us = vs + 2 * C * NC;                          // [C][NC] (delta rule)
  float* red = us + (DELTA ? C * NC : 0);               // [WARPS][C][NC]
  float* redk = red + WARPS * C * NC;                   // [WARPS][C][NC] (delta rule)
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int d = p.d, dv = p.dv, columns = dv + (ROW ? 1 : 0), col_blocks = (columns + NC - 1) / NC;
  const int h = blockIdx.x / col_blocks, col0 = blockIdx.x % col_blocks * NC, col = col0 + lane, entry = blockIdx.y;
  const Portion portion = portion_of(p, entry);
  const int t_begin = portion.first, t_end = t_begin + portion.count;
  if (t_begin >= t_end) return;
  int slot0 = 0;                                        // this request's first record
  for (int e = 0; e < entry; ++e) slot0 += (portion_of(p, e).count + C - 1) / C;
  const int chunks = (t_end - t_begin + C - 1) / C;
  const bool is_norm = ROW && col == dv, live = col < dv || is_norm;
  const size_t head = static_cast<size_t>(p.slots[entry]) * p.H + h;

  auto ask = [&](int chunk) {                           // a group of copies per call, empty past the last chunk
    if (chunk < chunks) {
      const float* src = p.records + (static_cast<size_t>(slot0 + chunk) * p.H + h) * RECORD;
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(ring + chunk % kRing * RECORD));
#pragma unroll
      for (int i = 0; i < (RECORD / 4 + THREADS - 1) / THREADS; ++i) {
        const int at = tid + i * THREADS;
        if (at < RECORD / 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + at * 16), "l"(src + at * 4) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  ask(0);
  ask(1);
  const TV* vg = static_cast<const TV*>(p.v) + static_cast<size_t>(h) * dv + col;
  TV rv[VPT];                       // kept in the storage type: a conversion right behind the load would wait for it
  auto fetch_values = [&](int t0) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int t = t0 + warp + i * WARPS;
      rv[i] = t < t_end && col < dv ? vg[static_cast<size_t>(t) * p.ldv] : from_float<TV>(t < t_end && is_norm ? 1.f : 0.f);
    }
  };
  fetch_values(t_begin);

  // the lane's part of the state: rows row0 .. row0 + 3, columns col0 + cl .. + 3
  const int cl = lane % 8 * 4, row0 = warp * 16 + lane / 8 * 4;
  auto cell = [&](int r, int c) -> float* {             // null where there is none
    if (r >= d) return nullptr;
    if (ROW && c == dv) return p.norm_state + head * d + r;
    return c < dv ? p.state + (head * d + r) * dv + c : nullptr;
  };
  float2 S[4][2];                                       // [column][pair of rows]
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float* x = cell(row0 + 2 * i, col0 + cl + c);
      const float* y = cell(row0 + 2 * i + 1, col0 + cl + c);
      S[c][i] = make_float2(x ? *x : 0.f, y ? *y : 0.f);
    }

  // x[t] . S over the warp's rows for the sixteen t, into to[warp][t][column]
  auto times_state = [&](const float* x, float* to) {
    const bool upper2 = (lane & 16) != 0, upper1 = (lane & 8) != 0;
#pragma unroll
    for (int t0 = 0; t0 < C; t0 += 4) {
      float part[4][4];                                 // [token][column]
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float4 v = *reinterpret_cast<const float4*>(x + (t0 + t) * DP + row0);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 a = __ffma2_rn(make_float2(v.z, v.w), S[c][1], __fmul2_rn(make_float2(v.x, v.y), S[c][0]));
          part[t][c] = a.x + a.y;
        }
      }
      // the four lanes of a column share the four tokens out: the lane of rows 4 r keeps token r
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float send = upper2 ? part[t][c] : part[t + 2][c];
          part[t][c] = (upper2 ? part[t + 2][c] : part[t][c]) + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float send = upper1 ? part[0][c] : part[1][c];
        part[0][c] = (upper1 ? part[1][c] : part[0][c]) + __shfl_xor_sync(0xffffffffu, send, 8);
      }
      *reinterpret_cast<float4*>(to + (warp * C + t0 + lane / 8) * NC + cl) = make_float4(part[0][0], part[0][1], part[0][2], part[0][3]);
    }
  };
  auto update_state = [&](const float* kt, const float* whole, const float* u) {
    const float4 f = *reinterpret_cast<const float4*>(whole + row0);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      S[c][0] = __fmul2_rn(S[c][0], make_float2(f.x, f.y));
      S[c][1] = __fmul2_rn(S[c][1], make_float2(f.z, f.w));
    }
#pragma unroll
    for (int s = 0; s < C; ++s) {
      const float4 k = *reinterpret_cast<const float4*>(kt + s * DP + row0);
      const float4 x = *reinterpret_cast<const float4*>(u + s * NC + cl);
      const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        S[c][0] = __ffma2_rn(make_float2(k.x, k.y), make_float2(xs[c], xs[c]), S[c][0]);
        S[c][1] = __ffma2_rn(make_float2(k.z, k.w), make_float2(xs[c], xs[c]), S[c][1]);
      }
    }
  };

  // sum over s <= t of row[s] * u[s][lane], added to x: the row is the same for all lanes
  auto combine = [&](const float* row, const float* u, int t, float x) {
#pragma unroll
    for (int s = 0; s < C; s += 4) {
      const float4 a = *reinterpret_cast<const float4*>(row + s);
      if (s <= t) x = fmaf(a.x, u[s * NC + lane], x);            // (later tokens' rows are not touched: they may hold anything)
      if (s + 1 <= t) x = fmaf(a.y, u[(s + 1) * NC + lane], x);
      if (s + 2 <= t) x = fmaf(a.z, u[(s + 2) * NC + lane], x);
      if (s + 3 <= t) x = fmaf(a.w, u[(s + 3) * NC + lane], x);
    }
    return x;
  };
  auto gathered = [&](const float* parts, int t) {
    float x = 0.f;
#pragma unroll
    for (int part = 0; part < WARPS; ++part) x += parts[(part * C + t) * NC + lane];
    return x;
  };

  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int t0 = t_begin + chunk * C, count = min(C, t_end - t0);
    const float* record = ring + chunk % kRing * RECORD;
    const float* am = record + (DELTA ? 3 : 2) * C * DP;
    const float* whole = record + RECORD - DP;
    float* v = vs + (chunk & 1) * C * NC;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float x = to_float(rv[i]);
      if (p.act) x = chunk_silu<TV>(x);
      v[(warp + i * WARPS) * NC + lane] = x;
    }
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();                                    // the record and the values are there; the chunk before has been read
    ask(chunk + 2);
    fetch_values(t0 + C);
    times_state(record, red);
    if constexpr (DELTA) times_state(record + 2 * C * DP, redk);
    else update_state(record + C * DP, whole, v);
    __syncthreads();                                    // the warps' sums are there
    if constexpr (DELTA) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int t = warp + i * WARPS;
        v[t * NC + lane] -= gathered(redk, t);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int t = warp + i * WARPS;
        us[t * NC + lane] = combine(am + C * C + t * C, v, t, 0.f);
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int t = warp + i * WARPS;
      const float o = combine(am + t * C, DELTA ? us : v, t, gathered(red, t));
      if (live && t < count) {
        if (is_norm) p.norm_out[static_cast<size_t>(t0 + t) * p.H + h] = o;
        else p.out[(static_cast<size_t>(t0 + t) * p.H + h) * dv + col] = o;
      }
    }
    if constexpr (DELTA) update_state(record + C * DP, whole, us);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float* x = cell(row0 + 2 * i, col0 + cl + c);
      float* y = cell(row0 + 2 * i + 1, col0 + cl + c);
      if (x) *x = S[c][i].x;
      if (y) *y = S[c][i].y;
    }
}

template <typename TV, bool DELTA, bool ROW, int WARPS>
int launch_chunks(const ChunkParams& p, cudaStream_t stream) {
  constexpr int C = kChunkTokens, NC = kChunkCols;
  constexpr size_t smem = sizeof(float) * (kRing * record_floats(WARPS * 16, DELTA) + (DELTA ? 3 : 2) * C * NC + (DELTA ? 2 : 1) * WARPS * C * NC);
  static DeviceOnce once;
  const int status = configure_once(once, scan_chunk_kernel<TV, DELTA, ROW, WARPS>, smem);
  if (status) return status;
  const int columns = p.dv + (ROW ? 1 : 0);
  launch(scan_chunk_kernel<TV, DELTA, ROW, WARPS>, dim3(p.H * ((columns + NC - 1) / NC), p.entries), dim3(WARPS * 32), smem, stream, p);
  return launch_status();
}

inline int padded_dim(int d) { return d <= 32 ? 32 : (d <= 64 ? 64 : 128); }

template <typename T, typename TV, bool DELTA, int GATE>
int run_chunks(ChunkParams p, int chunks, cudaStream_t stream) {
  constexpr bool ROW = GATE == CHUNK_ROW;
  p.dp = padded_dim(p.d);
  launch(scan_chunk_records_kernel<T, DELTA, GATE>, dim3(chunks, p.H), dim3(128), 0, stream, p);
  if (int e = launch_status()) return e;
  if (p.dp == 32) return launch_chunks<TV, DELTA, ROW, 2>(p, stream);
  if (p.dp == 64) return launch_chunks<TV, DELTA, ROW, 4>(p, stream);
  return launch_chunks<TV, DELTA, ROW, 8>(p, stream);
}

// ---------------------------------------------------------------------------------------------------- single tokens
// A decode step moves every request's state in and out and does next to nothing with it: one CTA per request, head and 128
// value columns holds the whole tile in registers, a warp 16 rows of it, a lane four columns of each, with all of its 16-byte
// reads on their way at once (64 KB a CTA, two CTAs an SM).  Sums over rows meet in shared memory once: the delta rule's
// read-out is formed as (D S)^T q + u (k . q) beside (D S)^T k, so one barrier serves both.  ROW: the normaliser's row is kept by the
// first 128 threads.  Bound by memory: 32 requests of 16 heads of 128 x 128 (67 MB) 13.8 us, 13.3 with the delta rule (20.9 and 23.8
// with the token-by-token kernel, whose lanes move 32 bytes of a row at a time); 8 requests of 32 heads 7.9 us, 8.8 with row gates
// (13.4 and 14.0).
template <typename T, typename TV, bool DELTA, int GATE>
__global__ void __launch_bounds__(256, 2) scan_single_kernel(const ChunkParams p) {
  constexpr bool ROW = GATE == CHUNK_ROW;
  __shared__ __align__(16) float ks[kChunkMaxDim], qs[kChunkMaxDim], gs[kChunkMaxDim];
  __shared__ __align__(16) float4 sum_k[DELTA ? 8 : 1][32], sum_q[8][32];
  __shared__ float scratch[32];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.x, entry = blockIdx.y, d = p.d, dv = p.dv;
  const int c = blockIdx.z * 128 + lane * 4, hqk = h / (p.H / p.Hqk);
  const size_t row = p.q_start[entry], head = static_cast<size_t>(p.slots[entry]) * p.H + h;
  const bool on = c < dv;                         // dv is a multiple of four here
  float* base = p.state + head * d * dv + c;
  float4 S[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = warp * 16 + i;
    S[i] = on && r < d ? *reinterpret_cast<const float4*>(base + static_cast<size_t>(r) * dv) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float all = GATE == CHUNK_HEAD ? p.decay[h] : (GATE == CHUNK_CHANNEL ? 1.f : p.row_decay[row * p.H + h]);
  const float gain = DELTA ? p.beta[row * p.H + h] : (ROW ? p.row_gain[row * p.H + h] : 1.f);
  float n = 0.f, kq = 0.f;
  if (tid < kChunkMaxDim) {
    float q = 0.f, k = 0.f, g = all;
    if (tid < d) {
      q = to_float(static_cast<const T*>(p.q)[row * p.ldq + hqk * d + tid]);
      k = to_float(static_cast<const T*>(p.k)[row * p.ldk + hqk * d + tid]);
      if (p.act) { q = chunk_silu<T>(q); k = chunk_silu<T>(k); }
      q *= p.q_scale;
      if (GATE == CHUNK_CHANNEL) g = p.gate[row * p.H * d + h * d + tid];
      if (ROW && blockIdx.z == 0) {
        n = fmaf(gain, k, all * p.norm_state[head * d + tid]);
        p.norm_state[head * d + tid] = n;
      }
    }
    ks[tid] = k;
    qs[tid] = q;
    gs[tid] = g;
    n *= q;
    kq = k * q;
  }
  float u[4] = {0.f, 0.f, 0.f, 0.f};
  if (on) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      u[e] = to_float(static_cast<const TV*>(p.v)[row * p.ldv + h * dv + c + e]);
      if (p.act) u[e] = chunk_silu<TV>(u[e]);
      if (ROW) u[e] *= gain;
    }
  }
  __syncthreads();
  if (DELTA) kq = block_sum(kq, scratch);
  if (ROW && blockIdx.z == 0) {
    n = block_sum(n, scratch);
    if (tid == 0) p.norm_out[row * p.H + h] = n;
  }
  float4 dk = make_float4(0.f, 0.f, 0.f, 0.f), dq = dk;
  auto add = [](float4& x, float f, const float4& y) {
    x.x = fmaf(f, y.x, x.x); x.y = fmaf(f, y.y, x.y); x.z = fmaf(f, y.z, x.z); x.w = fmaf(f, y.w, x.w);
  };
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = warp * 16 + i;
    const float g = gs[r], k = ks[r];
    S[i].x *= g; S[i].y *= g; S[i].z *= g; S[i].w *= g;
    if (DELTA) add(dk, k, S[i]);
    else add(S[i], k, make_float4(u[0], u[1], u[2], u[3]));
    add(dq, qs[r], S[i]);
  }
  if (DELTA) sum_k[warp][lane] = dk;
  sum_q[warp][lane] = dq;
  __syncthreads();
  if (DELTA) {
    dk = sum_k[0][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) add(dk, 1.f, sum_k[w][lane]);
    u[0] = gain * (u[0] - dk.x); u[1] = gain * (u[1] - dk.y); u[2] = gain * (u[2] - dk.z); u[3] = gain * (u[3] - dk.w);
#pragma unroll
    for (int i = 0; i < 16; ++i) add(S[i], ks[warp * 16 + i], make_float4(u[0], u[1], u[2], u[3]));
  }
  if (!on) return;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = warp * 16 + i;
    if (r < d) *reinterpret_cast<float4*>(base + static_cast<size_t>(r) * dv) = S[i];
  }
  if (warp == 0) {
    dq = sum_q[0][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) add(dq, 1.f, sum_q[w][lane]);
    if (DELTA) add(dq, kq, make_float4(u[0], u[1], u[2], u[3]));
    *reinterpret_cast<float4*>(p.out + (row * p.H + h) * dv + c) = dq;
  }
}

template <typename T, typename TV, bool DELTA, int GATE>
int run_single(const ChunkParams& p, cudaStream_t stream) {
  launch(scan_single_kernel<T, TV, DELTA, GATE>, dim3(p.H, p.entries, (p.dv + 127) / 128), dim3(256), 0, stream, p);
  return launch_status();
}

// CHUNKS: portions; else one token a request.
template <bool CHUNKS, typename T, typename TV, bool DELTA, int GATE>
int run_form(const ChunkParams& p, int chunks, cudaStream_t stream) {
  if constexpr (CHUNKS) return run_chunks<T, TV, DELTA, GATE>(p, chunks, stream);
  else return run_single<T, TV, DELTA, GATE>(p, stream);
}

template <bool CHUNKS>
int scan_form(const ChunkParams& p, int chunks, int dtype, int v_dtype, cudaStream_t stream) {
  if (p.entries <= 0 || chunks <= 0) return 0;
  if (p.H <= 0 || p.Hqk <= 0 || p.H % p.Hqk != 0 || p.d <= 0 || p.dv <= 0 || p.d > kChunkMaxDim) return B200_ERR_BAD_SIZE;
  if ((p.gate != nullptr) + (p.decay != nullptr) + (p.row_decay != nullptr) != 1) return B200_ERR_BAD_SIZE;
  if (p.entries > 65535 || p.H > 65535) return B200_ERR_TOO_LARGE;
  if (p.beta != nullptr && p.row_gain == nullptr && dtype == kF32 && v_dtype == kF32) {
    if (p.gate != nullptr) return run_form<CHUNKS, float, float, true, CHUNK_CHANNEL>(p, chunks, stream);
    if (p.row_decay != nullptr) return run_form<CHUNKS, float, float, true, CHUNK_TOKEN>(p, chunks, stream);
  } else if (p.beta == nullptr && v_dtype == kBF16) {
    if (p.decay != nullptr && dtype == kF32) return run_form<CHUNKS, float, __nv_bfloat16, false, CHUNK_HEAD>(p, chunks, stream);
    if (p.decay != nullptr && dtype == kBF16) return run_form<CHUNKS, __nv_bfloat16, __nv_bfloat16, false, CHUNK_HEAD>(p, chunks, stream);
    if (p.gate != nullptr && dtype == kBF16) return run_form<CHUNKS, __nv_bfloat16, __nv_bfloat16, false, CHUNK_CHANNEL>(p, chunks, stream);
    if (p.row_decay != nullptr && p.row_gain != nullptr && p.norm_state != nullptr && p.norm_out != nullptr && dtype == kBF16)
      return run_form<CHUNKS, __nv_bfloat16, __nv_bfloat16, false, CHUNK_ROW>(p, chunks, stream);
  }
  return B200_ERR_BAD_DTYPE;
}

}  // namespace b200

// The forms of the scan that portions of prompts meet beside 16-bit activations: float32 q, k, v with the delta rule (a decay per
// channel: gate, or per token: row_decay), float32 q, k beside bfloat16 v or bfloat16 rows with one decay a head (decay), bfloat16
// rows with a decay per channel (gate) or with row gates (row_decay and row_gain; norm_state, norm_out).  Key sizes up to 128.
// Of every request's tokens the launch takes those from `skip` on, `most` at most (both multiples of 16 where a request goes on behind
// them): a long portion's records need not all be there at once, its state goes from launch to launch in the request's slot.
// `chunks`: at least the number of chunks of 16 tokens of all requests in it; records: chunks * H * b200_scan_chunks_record_floats(d,
// delta) floats, 16-byte aligned.
extern "C" long b200_scan_chunks_record_floats(int d, int delta) { return b200::record_floats(b200::padded_dim(d), delta != 0); }

extern "C" int b200_scan_chunks(const void* q, const void* k, const void* v, int ldq, int ldk, int ldv, const float* gate,
                                const float* decay, const float* row_decay, const float* row_gain, const float* beta, float* state,
                                float* norm_state, float* norm_out, float* out, float* records, const int* q_start, const int* slots,
                                int entries, int chunks, int skip, int most, int H, int Hqk, int d, int dv, int act, float q_scale,
                                int dtype, int v_dtype, cudaStream_t stream) {
  using namespace b200;
  if (skip < 0 || most <= 0 || skip % kChunkTokens != 0) return B200_ERR_BAD_SIZE;
  const ChunkParams p{q, k, v, ldq, ldk, ldv, gate, decay, row_decay, row_gain, beta, state, norm_state, norm_out, out, records,
                      q_start, slots, entries, H, Hqk, d, 0, dv, act, q_scale, skip, most};
  return scan_form<true>(p, chunks, dtype, v_dtype, stream);
}

// The same forms for batches in which every request has one token; value sizes that are multiples of four, states and outputs
// that start on 16-byte boundaries.
extern "C" int b200_scan_single(const void* q, const void* k, const void* v, int ldq, int ldk, int ldv, const float* gate,
                                const float* decay, const float* row_decay, const float* row_gain, const float* beta, float* state,
                                float* norm_state, float* norm_out, float* out, const int* q_start, const int* slots,
                                int entries, int H, int Hqk, int d, int dv, int act, float q_scale, int dtype, int v_dtype,
                                cudaStream_t stream) {
  using namespace b200;
  if (dv % 4 != 0 || ((reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(out)) & 15)) return B200_ERR_BAD_SIZE;
  const ChunkParams p{q, k, v, ldq, ldk, ldv, gate, decay, row_decay, row_gain, beta, state, norm_state, norm_out, out, nullptr,
                      q_start, slots, entries, H, Hqk, d, 0, dv, act, q_scale, 0, 1};
  return scan_form<false>(p, 1, dtype, v_dtype, stream);
}
