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
// the recurrence does not.  What does not depend on the state is made for all chunks at once by a first kernel, in float32: per chunk and
// head a record of G_t q_t, E_s k_s, (G_t k_t,) A, (T), each number as three bfloat16 that hold its 24 bits, and G_C.  The second walks the
// chunks on the tensor cores, its sums in float32.
#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

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
  void* records;                                   // [chunks][H][record_bytes]
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

// A record: Q, K, (KF,) each three planes of bfloat16 [16][dp + 8] that add up to the float32 numbers, A, (T,) each three planes
// [16][24] (rows 16 bytes longer than their numbers: ldmatrix then reads eight of them from different banks), whole [dp] floats.
__host__ __device__ constexpr int record_pitch(int dp) { return dp + 8; }
constexpr int kSmallPitch = kChunkTokens + 8;
__host__ __device__ constexpr int record_bytes(int dp, bool delta) {
  return (delta ? 9 : 6) * kChunkTokens * record_pitch(dp) * 2 + (delta ? 6 : 3) * kChunkTokens * kSmallPitch * 2 + dp * 4;
}
// x as the sum of three bfloat16, `plane` numbers apart.  The first is at most the largest bfloat16, so that every finite number has such parts; an
// infinity or NaN is the second one (number_of_parts).
__device__ __forceinline__ void store_parts(__nv_bfloat16* to, int plane, float x) {
  uint16_t bits;
  asm("cvt.rn.satfinite.bf16.f32 %0, %1;\n" : "=h"(bits) : "f"(x));
  __nv_bfloat16 part = __ushort_as_bfloat16(bits);
  to[0] = part;
  x -= __bfloat162float(part);
  part = __float2bfloat16_rn(x);
  to[plane] = part;
  to[2 * plane] = __float2bfloat16_rn(x - __bfloat162float(part));
}
__device__ __forceinline__ float number_of_parts(const __nv_bfloat16* at, int plane) {
  const float second = __bfloat162float(at[plane]);
  return isfinite(second) ? (__bfloat162float(at[2 * plane]) + second) + __bfloat162float(at[0]) : second;
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
  unsigned char* record = reinterpret_cast<unsigned char*>(p.records) + (static_cast<size_t>(blockIdx.x) * p.H + h) * record_bytes(dp, DELTA);
  const int pitch = record_pitch(dp), plane = C * pitch;
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
    __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(record) + tid;
    float f = 1.f;
#pragma unroll
    for (int t = 0; t < C; ++t) {
      f *= GATE == CHUNK_CHANNEL ? g[GATE == CHUNK_CHANNEL ? t : 0] : alpha[t];
      store_parts(to + t * pitch, plane, q[t] * f);
      if (DELTA) store_parts(to + 6 * plane + t * pitch, plane, k[t] * f);
    }
    reinterpret_cast<float*>(record + record_bytes(dp, DELTA))[tid - dp] = f;
    f = 1.f;
#pragma unroll
    for (int t = C - 1; t >= 0; --t) {
      store_parts(to + 3 * plane + t * pitch, plane, k[t] * (GATE == CHUNK_ROW ? f * gain[t] : f));
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
  __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(record) + (DELTA ? 9 : 6) * plane;
  for (int idx = tid; idx < C * C; idx += 128) {
    const int at = idx / C * kSmallPitch + idx % C;
    store_parts(to + at, C * kSmallPitch, as[idx / C][idx % C]);
    if (DELTA) store_parts(to + 3 * C * kSmallPitch + at, C * kSmallPitch, ts[idx / C][idx % C]);
  }
}

// ---------------------------------------------------------------------------------------------------- the chunks
// One CTA per request, head and 32 value columns; two warps hold 16 columns of the state, transposed, half of the rows each, in registers
// for the whole portion, laid out as the accumulators of mma.sync m16n8k16 (16 columns x 8 rows a tile).  So the state is the row operand
// of S^T q (k) as it stands and its update is accumulated in its own layout; the two warps exchange their halves' sums.  A chunk's
// record arrives by one bulk copy, one or two chunks ahead.
// Float32 factors are sums of three bfloat16 (24 bits); of the nine products of two, the six that reach 2^-24 of the whole are formed on the
// tensor cores.  Those truncate the sums they accumulate, so every leading product (largest part with largest part) is summed by itself from zero
// and added in float32, and so is what a chunk adds to the state.  Errors against 64 bits over 400 to 2,000 tokens of 8 to 32 heads, all forms:
// 0.80 to 1.00 of the FMA kernel's that this one replaced in the read-outs, 0.76 to 1.00 in the states.
// Bound by the issue of the two warps' instructions: 102 (VSPLIT) or 75 matrix instructions a chunk and warp, 156 with the delta rule, 8.2 clocks each,
// and about as many others.  With records, 2,048 tokens of 32 heads of 128 x 128: one decay a head 262 us (317 with the FMA kernel, whose warps held
// 16 rows x 32 columns each and exchanged every sum), delta rule with decays per channel 352 (460); 16 heads 232 and 300 (299, 424); three portions of
// 578 tokens, 32 heads: decays per channel 159 (217), row gates 172 (250); one of 1,733 with row gates 213 (354).
// ROW: the normaliser is one more column, behind the last value column, whose value is 1 for every token.
// A number that is not finite has no three parts whose products add up to its own, nor has one beyond the largest bfloat16, and beside weights of
// 0 such a value would reach the tokens before its own.  Any of them leaves a read-out or a cell of the state that is not finite; these are
// looked at, and the CTA then takes its portion once more from its first token in float32 (scan_plainly).
struct Triple { uint32_t part[3]; };        // two neighbouring values: three bfloat16 pairs that add up to them, largest first
__device__ __forceinline__ Triple split_pair(float x, float y) {
  Triple s;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    s.part[i] = pack_bf16(x, y);
    x -= __uint_as_float(s.part[i] << 16);
    y -= __uint_as_float(s.part[i] & 0xffff0000u);
  }
  return s;
}
// the accumulators of two neighbouring tiles (16 columns x 16 rows or tokens) as three row operands of 16 x 16
__device__ __forceinline__ void split_tiles(const float (&lo)[4], const float (&hi)[4], uint32_t (&a)[3][4]) {
  const Triple x[4] = {split_pair(lo[0], lo[1]), split_pair(lo[2], lo[3]), split_pair(hi[0], hi[1]), split_pair(hi[2], hi[3])};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) a[i][j] = x[j].part[i];
}
// (as mma_bf16, but free to be moved among other instructions: nothing but registers go in and out)
__device__ __forceinline__ void mma_free(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// which parts of the two factors make the six products, smallest first; with one part only of the first factor, three
__device__ constexpr int kPartA[6] = {2, 0, 1, 1, 0, 0}, kPartB[6] = {0, 2, 1, 0, 1, 0};

// One CTA's portion with every sum over float32 products: a warp has a quarter of the rows, a lane a column.  For portions with numbers that the
// tensor cores cannot take, so written for few registers beside the kernel that calls it, not for speed.  `shared`: 6 * 16 * 32 floats.
template <typename TV, bool DELTA, bool ROW, bool VSPLIT, int DP>
__device__ __noinline__ void scan_plainly(const ChunkParams& p, int entry, int h, int col0, int slot0, float* shared) {
  constexpr int C = kChunkTokens, NC = kChunkCols, RECORD = record_bytes(DP, DELTA), PITCH = record_pitch(DP), ROWS = DP / 4;
  float* us = shared;                                   // [C][NC]
  float* vs = us + C * NC;                              // [C][NC]
  float* red = vs + C * NC;                             // [4][C][NC]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, col = col0 + lane, row0 = warp * ROWS;
  const Portion portion = portion_of(p, entry);
  const size_t head = static_cast<size_t>(p.slots[entry]) * p.H + h;
  const bool norm = ROW && col == p.dv, live = col < p.dv || norm;
  auto cell = [&](int r) { return norm ? p.norm_state + head * p.d + r : p.state + (head * p.d + r) * p.dv + col; };
  float S[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) S[r] = live && row0 + r < p.d ? *cell(row0 + r) : 0.f;
  auto times_state = [&](const __nv_bfloat16* rows) {   // into `red`: this warp's rows' share of all tokens' sums
#pragma unroll 1
    for (int s = 0; s < C; ++s) {
      float x = 0.f;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) x = fmaf(S[r], number_of_parts(rows + s * PITCH + row0 + r, C * PITCH), x);
      red[(warp * C + s) * NC + lane] = x;
    }
  };
  auto whole_sum = [&](int s) { return (red[s * NC + lane] + red[(C + s) * NC + lane]) + (red[(2 * C + s) * NC + lane] + red[(3 * C + s) * NC + lane]); };
  auto up_to_now = [&](const __nv_bfloat16* m, const float* x, int s, float sum) {
#pragma unroll 1
    for (int e = 0; e <= s; ++e) sum = fmaf(number_of_parts(m + s * kSmallPitch + e, C * kSmallPitch), x[e * NC + lane], sum);
    return sum;
  };
#pragma unroll 1
  for (int first = 0; first < portion.count; first += C) {
    const int tokens = min(C, portion.count - first);
    const unsigned char* record = static_cast<const unsigned char*>(p.records) + (static_cast<size_t>(slot0 + first / C) * p.H + h) * RECORD;
    const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(record);
    const __nv_bfloat16* small = rows + (DELTA ? 9 : 6) * C * PITCH;
    const float* whole = reinterpret_cast<const float*>(record + RECORD) - DP;
    __syncthreads();
#pragma unroll 1
    for (int s = warp; s < C; s += 4) {
      float x = norm && s < tokens ? 1.f : 0.f;
      if (col < p.dv && s < tokens) {
        x = to_float(static_cast<const TV*>(p.v)[static_cast<size_t>(portion.first + first + s) * p.ldv + static_cast<size_t>(h) * p.dv + col]);
        if (VSPLIT && p.act) x = chunk_silu<TV>(x);
      }
      (DELTA ? vs : us)[s * NC + lane] = x;
    }
    if constexpr (DELTA) {
      times_state(rows + 6 * C * PITCH);
      __syncthreads();
#pragma unroll 1
      for (int s = warp; s < C; s += 4) vs[s * NC + lane] -= whole_sum(s);
      __syncthreads();
#pragma unroll 1
      for (int s = warp; s < C; s += 4) us[s * NC + lane] = up_to_now(small + 3 * C * kSmallPitch, vs, s, 0.f);
    }
    times_state(rows);
    __syncthreads();
#pragma unroll 1
    for (int s = warp; s < tokens; s += 4) {
      const float o = up_to_now(small, us, s, whole_sum(s));
      const size_t at = static_cast<size_t>(portion.first + first + s) * p.H + h;
      if (norm) p.norm_out[at] = o;
      else if (live) p.out[at * p.dv + col] = o;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) S[r] *= whole[row0 + r];
#pragma unroll 1
    for (int s = 0; s < tokens; ++s) {
      const float u = us[s * NC + lane];
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (row0 + r < p.d) S[r] = fmaf(number_of_parts(rows + 3 * C * PITCH + s * PITCH + row0 + r, C * PITCH), u, S[r]);     // (rows that are not there stay 0)
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
    if (live && row0 + r < p.d) *cell(row0 + r) = S[r];
}

constexpr int kChunkTiles = kChunkCols / 16, kChunkThreads = kChunkTiles * 64;
// records in shared memory: as many as leave room for two CTAs an SM
__host__ __device__ constexpr int record_ring(bool delta) { return delta ? 2 : 3; }
__device__ int g_scan_error = 0;
// Registers a thread.  Under another bound the compiler puts a chunk's instructions in another order, and its time follows: 2,048 tokens of 32 heads of
// 128, one decay a head 205 to 217 us between 154 and 200 registers, delta rule 346 to 427 between 152 and 200; the best of them each.  Left to
// itself it makes room for a third CTA an SM that the records do not leave (row gates 128 registers: 367 us, 239).  Small states need no bound but one (8 heads of 32, 509 tokens, a decay
// a head: 30.3 us without, 26.0 with 96).
constexpr int chunk_registers(int dt, bool delta, bool row) {
  if (dt < 8) return dt == 2 && !delta && !row ? 96 : 255;
  return delta ? 176 : (row ? 172 : 156);
}
template <typename TV, bool DELTA, bool ROW, bool VSPLIT, int DT>
__global__ void __launch_bounds__(kChunkThreads) __maxnreg__(chunk_registers(DT, DELTA, ROW))
scan_chunk_kernel(const __grid_constant__ ChunkParams p) {
  constexpr int C = kChunkTokens, DP = DT * 16, RECORD = record_bytes(DP, DELTA), RING = record_ring(DELTA), PITCH = record_pitch(DP) * 2, HT = DT / 2;
  constexpr int PLANE = C * PITCH, SMALL = C * kSmallPitch * 2, UPARTS = VSPLIT || DELTA ? 3 : 1;
  extern __shared__ __align__(16) unsigned char ring[];   // [RING][RECORD]
  __shared__ __align__(8) uint64_t full[RING];
  __shared__ float4 handed[DELTA ? 3 : 1][kChunkTiles][2][32];     // sums over half of the rows for the other half's warp: of a read-out, of w
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, tile = warp >> 1, half = warp & 1;
  if (tid == 0) {
    for (int i = 0; i < RING; ++i) mbar_init(full + i, 1);
    fence_barrier_init();
  }
  pdl_wait();
  const int d = p.d, dv = p.dv, columns = dv + (ROW ? 1 : 0), col_blocks = (columns + kChunkCols - 1) / kChunkCols;
  const int h = blockIdx.x / col_blocks, col0 = blockIdx.x % col_blocks * kChunkCols + tile * 16, entry = blockIdx.y;
  const Portion portion = portion_of(p, entry);
  const int t_begin = portion.first, t_end = t_begin + portion.count;
  if (t_begin >= t_end) return;
  int slot0 = 0;                                        // this request's first record
  for (int e = 0; e < entry; ++e) slot0 += (portion_of(p, e).count + C - 1) / C;
  const int chunks = (t_end - t_begin + C - 1) / C;
  const size_t head = static_cast<size_t>(p.slots[entry]) * p.H + h;
  __syncthreads();                                      // the barriers are there

  const unsigned char* next_record = static_cast<const unsigned char*>(p.records) + (static_cast<size_t>(slot0) * p.H + h) * RECORD;
  int next_slot = 0, left = chunks;                     // of the records still to be asked for
  auto ask = [&]() {                                    // one thread
    if (left > 0) {
      mbar_expect_tx(full + next_slot, RECORD);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_addr(ring + next_slot * RECORD)),
                   "l"(next_record), "r"(RECORD), "r"(smem_addr(full + next_slot))
                   : "memory");
      next_record += static_cast<size_t>(p.H) * RECORD;
      next_slot = next_slot + 1 == RING ? 0 : next_slot + 1;
      --left;
    }
  };
  if (tid == 0)
    for (int i = 1; i < RING; ++i) ask();
  // this lane's columns: col0 + g and 8 further on; its tokens of a chunk: 2 t, 2 t + 1 and 8 further on; its rows of tile j: row0 + 8 j + 2 t, + 1
  const bool working = col0 < columns;
  const int row0 = half * (DP / 2);
  TV rv[2][4];                      // kept in the storage type: a conversion right behind the load would wait for it
  const TV* vg = static_cast<const TV*>(p.v) + static_cast<size_t>(h) * dv + col0 + g;
  auto fetch_values = [&](int t0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int tok = t0 + (i >> 2) * 8 + 2 * t + (i & 1), c = ((i >> 1) & 1) * 8;
      rv[i >> 2][i & 3] = tok < t_end && col0 + g + c < dv ? vg[static_cast<size_t>(tok) * p.ldv + c]
                                                           : from_float<TV>(ROW && tok < t_end && col0 + g + c == dv ? 1.f : 0.f);
    }
  };
  fetch_values(t_begin);
  auto cell = [&](int r, int c) -> float* {             // null where there is none
    if (r >= d) return nullptr;
    if (ROW && c == dv) return p.norm_state + head * d + r;
    return c < dv ? p.state + (head * d + r) * dv + c : nullptr;
  };
  float S[2 * HT][4];
#pragma unroll
  for (int j = 0; j < 2 * HT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float* x = cell(row0 + 8 * j + 2 * t + (e & 1), col0 + g + (e >> 1) * 8);
      S[j][e] = x ? *x : 0.f;
    }
  // ldmatrix: rows of column operands whose K runs along them (q, k: tokens; A, T: tokens), and of k as rows of K, which it transposes
  const int row_n = (lane >> 4) * 8 + (lane & 7), half_n = ((lane >> 3) & 1) * 16;
  const int row_k = ((lane >> 3) & 1) * 8 + (lane & 7), half_k = (lane >> 4) * 16;
  auto load_n = [&](uint32_t (&r)[4], uint32_t base, int pitch, int step) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(base + row_n * pitch + step * 32 + half_n));
  };
  auto load_k = [&](uint32_t (&r)[4], uint32_t base, int step) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(base + row_k * PITCH + step * 32 + half_k));
  };
  auto pair_barrier = [&]() { asm volatile("bar.sync %0, 64;\n" ::"r"(tile + 1) : "memory"); };

  // S^T x over this warp's rows for the sixteen rows of x (three planes from `planes` on): [tile of tokens][accumulator]
  auto times_state = [&](uint32_t planes, float (&out)[2][4]) {
    float lead[HT][2][4] = {}, rest[2][2][4] = {};      // (a leading product's sum is truncated once, not again by those behind it)
    uint32_t ahead[3][4];                               // the next step's rows: asked for under this one's products
    planes += row0 * 2;
#pragma unroll
    for (int i = 0; i < 3; ++i) load_n(ahead[i], planes + i * PLANE, PITCH, 0);
#pragma unroll
    for (int ks = 0; ks < HT; ++ks) {
      uint32_t a[3][4], b[3][4];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) b[i][j] = ahead[i][j];
      if (ks + 1 < HT) {
#pragma unroll
        for (int i = 0; i < 3; ++i) load_n(ahead[i], planes + i * PLANE, PITCH, ks + 1);
      }
      split_tiles(S[2 * ks], S[2 * ks + 1], a);
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma_free(i == 5 ? lead[ks][nt] : rest[i & 1][nt], a[kPartA[i]], b[kPartB[i]][2 * nt], b[kPartB[i]][2 * nt + 1]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int n = 1; n < HT; n *= 2)
#pragma unroll
          for (int ks = 0; ks + n < HT; ks += 2 * n) lead[ks][nt][e] += lead[ks + n][nt][e];
        out[nt][e] = (rest[0][nt][e] + rest[1][nt][e]) + lead[0][nt][e];
      }
  };
  // out[t] += sum over s <= t of M[t][s] x[s] for eight tokens from `first` on, M in three planes; x as row operands in `parts` planes
  auto up_to_now = [&](uint32_t m, int first, const uint32_t (&a)[3][4], int parts, float (&out)[4]) {
    uint32_t b[3][2];
#pragma unroll
    for (int i = 0; i < 3; ++i)
      asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n"
                   : "=r"(b[i][0]), "=r"(b[i][1])
                   : "r"(m + i * SMALL + (first + (lane & 7)) * (kSmallPitch * 2) + half_n));
    float lead[4] = {}, rest[2][4] = {};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      if (kPartA[i] >= parts) continue;
      mma_free(i == 5 ? lead : rest[i & 1], a[kPartA[i]], b[kPartB[i]][0], b[kPartB[i]][1]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) out[e] += (rest[0][e] + rest[1][e]) + lead[e];
  };

  int slot = 0;
  uint32_t phase = 0;
  float doubt = 0.f;                                    // NaN once something has not been finite
  for (int t0 = t_begin; t0 < t_end; t0 += C) {
    const bool ok = mbar_wait(full + slot, phase);
    if (!__syncthreads_and(ok)) {                       // (the record is there; the one before has been read)
      if (tid == 0) {                                   // (copies on their way still get their time)
        atomicExch(&g_scan_error, 1);
        for (int i = 0; i < RING; ++i) mbar_wait(full + i, i < slot ? phase ^ 1 : phase);
      }
      return;
    }
    if (tid == 0) ask();
    const unsigned char* record_at = ring + slot * RECORD;
    if (++slot == RING) { slot = 0; phase ^= 1; }
    if (!working) continue;
    const uint32_t record = smem_addr(record_at), small = record + (DELTA ? 9 : 6) * PLANE;
    const float* whole = reinterpret_cast<const float*>(record_at + RECORD - DP * 4) + row0 + 2 * t;
    float u[2][4], o[2][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float x = to_float(rv[i >> 2][i & 3]);
      if (VSPLIT && p.act) x = chunk_silu<TV>(x);
      u[i >> 2][i & 3] = x;
    }
    fetch_values(t0 + C);
    uint32_t a[3][4];
    if constexpr (DELTA) {
      float w[2][4];
      times_state(record + 6 * PLANE, w);
      handed[1][tile][half][lane] = make_float4(w[0][0], w[0][1], w[0][2], w[0][3]);
      handed[2][tile][half][lane] = make_float4(w[1][0], w[1][1], w[1][2], w[1][3]);
      pair_barrier();
      float sums[2][2][4];                              // both warps add the halves up in their order
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = handed[1 + (i & 1)][tile][i >> 1][lane];
        sums[i >> 1][i & 1][0] = x.x; sums[i >> 1][i & 1][1] = x.y; sums[i >> 1][i & 1][2] = x.z; sums[i >> 1][i & 1][3] = x.w;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        w[i >> 2][i & 3] = u[i >> 2][i & 3] - (sums[0][i >> 2][i & 3] + sums[1][i >> 2][i & 3]);
        u[i >> 2][i & 3] = 0.f;
      }
      split_tiles(w[0], w[1], a);
      up_to_now(small + 3 * SMALL, 0, a, 3, u[0]);
      up_to_now(small + 3 * SMALL, 8, a, 3, u[1]);
    }
    if constexpr (UPARTS == 3) {
      split_tiles(u[0], u[1], a);
    } else {                                            // the values are bfloat16
      a[0][0] = pack_bf16(u[0][0], u[0][1]);
      a[0][1] = pack_bf16(u[0][2], u[0][3]);
      a[0][2] = pack_bf16(u[1][0], u[1][1]);
      a[0][3] = pack_bf16(u[1][2], u[1][3]);
    }
    times_state(record, o);
    // each of the two warps finishes eight tokens of the read-out
    handed[0][tile][half][lane] = half ? make_float4(o[0][0], o[0][1], o[0][2], o[0][3]) : make_float4(o[1][0], o[1][1], o[1][2], o[1][3]);
    // the state takes its decay and the sixteen tokens' updates, four tiles of eight rows at a time
    uint32_t ahead[3][2][4];
    constexpr int GROUP = HT > 1 ? 4 : 2;               // tiles at a time
#pragma unroll
    for (int i = 0; i < 3 * GROUP / 2; ++i) load_k(ahead[i / (GROUP / 2)][i % (GROUP / 2)], record + (3 + i / (GROUP / 2)) * PLANE + row0 * 2, i % (GROUP / 2));
#pragma unroll
    for (int j = 0; j < 2 * HT; j += GROUP) {
      float sum[GROUP][4] = {}, top[GROUP][4] = {};
      uint32_t b[3][2][4];
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) b[i >> 1][i & 1][x] = ahead[i >> 1][i & 1][x];
      if (j + GROUP < 2 * HT) {
#pragma unroll
        for (int i = 0; i < 6; ++i) load_k(ahead[i >> 1][i & 1], record + (3 + (i >> 1)) * PLANE + row0 * 2, j / 2 + 2 + (i & 1));
      }
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        if (kPartA[i] >= UPARTS) continue;
#pragma unroll
        for (int x = 0; x < GROUP; ++x) mma_free(i == 5 ? top[x] : sum[x], a[kPartA[i]], b[kPartB[i]][x >> 1][(x & 1) * 2], b[kPartB[i]][x >> 1][(x & 1) * 2 + 1]);
      }
#pragma unroll
      for (int x = 0; x < GROUP; ++x) {
        const float2 f = *reinterpret_cast<const float2*>(whole + 8 * (j + x));
        S[j + x][0] = fmaf(S[j + x][0], f.x, sum[x][0]) + top[x][0];
        S[j + x][1] = fmaf(S[j + x][1], f.y, sum[x][1]) + top[x][1];
        S[j + x][2] = fmaf(S[j + x][2], f.x, sum[x][2]) + top[x][2];
        S[j + x][3] = fmaf(S[j + x][3], f.y, sum[x][3]) + top[x][3];
      }
    }
    pair_barrier();
    const float4 other = handed[0][tile][half ^ 1][lane];
    float mine[4] = {other.x + (half ? o[1][0] : o[0][0]), other.y + (half ? o[1][1] : o[0][1]), other.z + (half ? o[1][2] : o[0][2]),
                     other.w + (half ? o[1][3] : o[0][3])};
    up_to_now(small, half * 8, a, UPARTS, mine);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      doubt = fmaf(mine[i], 0.f, doubt);
      const int tok = t0 + half * 8 + 2 * t + (i & 1), c = col0 + g + (i >> 1) * 8;
      if (tok >= t_end) continue;
      if (c < dv) p.out[(static_cast<size_t>(tok) * p.H + h) * dv + c] = mine[i];
      else if (ROW && c == dv) p.norm_out[static_cast<size_t>(tok) * p.H + h] = mine[i];
    }
  }
#pragma unroll
  for (int j = 0; j < 2 * HT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) doubt = fmaf(S[j][e], 0.f, doubt);
  if (__syncthreads_or(doubt != 0.f)) {                 // (nothing of the state has been written)
    scan_plainly<TV, DELTA, ROW, VSPLIT, DP>(p, entry, h, blockIdx.x % col_blocks * kChunkCols, slot0, reinterpret_cast<float*>(ring));
    return;
  }
  if (!working) return;
#pragma unroll
  for (int j = 0; j < 2 * HT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float* x = cell(row0 + 8 * j + 2 * t + (e & 1), col0 + g + (e >> 1) * 8);
      if (x) *x = S[j][e];
    }
}

template <typename TV, bool DELTA, bool ROW, bool VSPLIT, int DT>
int launch_chunks(const ChunkParams& p, cudaStream_t stream) {
  constexpr size_t smem = record_ring(DELTA) * record_bytes(DT * 16, DELTA);
  static DeviceOnce once;
  const int status = configure_once(once, scan_chunk_kernel<TV, DELTA, ROW, VSPLIT, DT>, smem + 8 * 1024);      // (the kernel's own arrays count too)
  if (status) return status;
  const int columns = p.dv + (ROW ? 1 : 0);
  launch(scan_chunk_kernel<TV, DELTA, ROW, VSPLIT, DT>, dim3(p.H * ((columns + kChunkCols - 1) / kChunkCols), p.entries), dim3(kChunkThreads), smem, stream, p);
  return launch_status();
}

inline int padded_dim(int d) { return d <= 32 ? 32 : (d <= 64 ? 64 : 128); }

template <typename TV, bool DELTA, bool ROW, bool VSPLIT>
int launch_chunks_of(const ChunkParams& p, cudaStream_t stream) {
  if (p.dp == 32) return launch_chunks<TV, DELTA, ROW, VSPLIT, 2>(p, stream);
  if (p.dp == 64) return launch_chunks<TV, DELTA, ROW, VSPLIT, 4>(p, stream);
  return launch_chunks<TV, DELTA, ROW, VSPLIT, 8>(p, stream);
}

template <typename T, typename TV, bool DELTA, int GATE>
int run_chunks(ChunkParams p, int chunks, cudaStream_t stream) {
  constexpr bool ROW = GATE == CHUNK_ROW;
  p.dp = padded_dim(p.d);
  launch(scan_chunk_records_kernel<T, DELTA, GATE>, dim3(chunks, p.H), dim3(128), 0, stream, p);
  if (int e = launch_status()) return e;
  if constexpr (!DELTA) {
    if (!p.act) return launch_chunks_of<TV, DELTA, ROW, false>(p, stream);
  }
  return launch_chunks_of<TV, DELTA, ROW, true>(p, stream);
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
extern "C" long b200_scan_chunks_record_floats(int d, int delta) { return b200::record_bytes(b200::padded_dim(d), delta != 0) / 4; }

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

// Read and clear the error flag set by a bounded wait that ran out.  Synchronises the device.
extern "C" int b200_scan_chunks_error() {
  int v = 0, zero = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  cudaMemcpyFromSymbol(&v, b200::g_scan_error, sizeof(int));
  cudaMemcpyToSymbol(b200::g_scan_error, &zero, sizeof(int));
  return v;
}
