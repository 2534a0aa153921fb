// Causal attention over the paged cache on CUDA cores, 32-bit arithmetic throughout.
// It serves prompt portions and single decoded tokens alike: every query token is
// handled by itself (one warp per token and query head), reading keys 0..p of its
// request through the block table, in tiles of 32 keys that start at key 0.  The
// order of every sum is therefore a function of the token's own position only, so a
// token's output is bit-identical however the batch was cut.
//
// Formula (mini_llm/nn/attention.py:95-99, 231-248): S = q.k^T * scale, key t visible
// iff t <= p (and t > p - window when a window is set), P = softmax(S), o = P.v;
// query head j reads KV head j / (nq / nkv)  (mini_llm/nn/attention.py:18-33).
//
// Optional rules on the scores, each a parameter: a soft cap (S <- cap * tanh(S / cap)), a
// bias by distance (S <- S - slope_j * (p - t) with one slope per query head), and a sink
// (a virtual key that carries no value, of score 0 or of a number per query head that the scale does not touch: the weights
// become exp(S) / (exp(sink) + sum exp(S))).
// Values may have a head size `dv` of their own.  Two further rules: a bias by the logarithm of the distance
// (S <- S - r1_j * ln(1 + r2_j * (p - t)) with two numbers per query head) and a mask in blocks (`chunk` > 0: position p
// sees t only if floor(p / chunk) = floor(t / chunk), blocks counted from position 0 of the sequence).
//
// Two kernels keep that order bit for bit: one warp per token and head (single decoded tokens, and every size), and tiles
// of query rows that share the keys and values of a prompt portion (float32).
#include <type_traits>

#include "common.cuh"

namespace b200 {

// What the rules make of a product q . k: every rounding is spelled out, so that the kernels cannot differ in it.
struct ScoreRules {
  float scale, softcap, inv_cap, slope, r1, r2;
  bool log_bias;
  __device__ __forceinline__ float operator()(float dot, int distance) const {
    float s = __fmul_rn(dot, scale);
    if (softcap > 0.f) s = __fmul_rn(softcap, tanhf(__fmul_rn(s, inv_cap)));
    s = __fmaf_rn(-slope, static_cast<float>(distance), s);
    if (log_bias) s = __fmaf_rn(-r1, log1pf(__fmul_rn(r2, static_cast<float>(distance))), s);
    return s;
  }
};

// One warp per token and head.  kMaxChunks x 32 columns of values at most; the key size is bounded by shared memory only
template <typename T, int kMaxChunks>
__global__ void __launch_bounds__(128)
paged_attention_simt_kernel(const T* __restrict__ q, const T* __restrict__ k_pool,
                            const T* __restrict__ v_pool, T* __restrict__ out,
                            const int* __restrict__ positions, const int* __restrict__ token_entry,
                            const int* __restrict__ block_table, int table_stride, int page_size,
                            int nq, int nkv, int d, float scale, int window, int dv, float softcap,
                            const float* __restrict__ slopes, int sink, int v_row, int chunk,
                            const float* __restrict__ log_r1, const float* __restrict__ log_r2,
                            const float* __restrict__ sinks) {
  extern __shared__ float smem[];
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int token = blockIdx.x;
  const int head = blockIdx.y * 4 + warp;
  if (head >= nq) return;
  const int kvh = head / (nq / nkv);
  const int p = positions[token];
  const int* table = block_table + static_cast<size_t>(token_entry[token]) * table_stride;
  float* qs = smem + warp * d;
  const T* qrow = q + (static_cast<size_t>(token) * nq + head) * d;
  for (int i = lane; i < d; i += 32) qs[i] = to_float(qrow[i]);
  __syncwarp();

  int w0 = window > 0 ? max(0, p - window + 1) : 0;
  if (chunk > 0) w0 = max(w0, p / chunk * chunk);
  // the sink is a key of score 0 (or sinks[head]) and value 0 that every row sees: it starts the running maximum and sum
  float m = sink ? 0.f : -INFINITY, l = sink || sinks != nullptr ? 1.f : 0.f;
  if (sinks != nullptr) m = sinks[head];
  const ScoreRules rules{scale, softcap, softcap > 0.f ? 1.f / softcap : 0.f, slopes ? slopes[head] : 0.f,
                         log_r1 ? log_r1[head] : 0.f, log_r2 ? log_r2[head] : 0.f, log_r1 != nullptr};
  float acc[kMaxChunks];
#pragma unroll
  for (int c = 0; c < kMaxChunks; ++c) acc[c] = 0.f;

  constexpr int VN = Vec<T>::n;
  for (int t0 = (w0 / 32) * 32; t0 <= p; t0 += 32) {
    const int t = t0 + lane;
    bool valid = t <= p && t >= w0;
    float s = -INFINITY;
    const int page = valid ? table[t / page_size] : -1;
    valid = valid && page >= 0;      // a page given back (window) or a padding row without pages
    if (valid) {
      const T* krow = k_pool + ((static_cast<size_t>(page) * nkv + kvh) * page_size + t % page_size) * d;
      float dot = 0.f;
      if (d % VN == 0) {         // rows of keys then start on 16-byte boundaries
#pragma unroll 8
        for (int i = 0; i < d; i += VN) {
          float f[VN];
          Vec<T>::unpack(*reinterpret_cast<const typename Vec<T>::type*>(krow + i), f);
#pragma unroll
          for (int e = 0; e < VN; ++e) dot = fmaf(qs[i + e], f[e], dot);
        }
      } else {
        for (int i = 0; i < d; ++i) dot = fmaf(qs[i], to_float(krow[i]), dot);
      }
      s = rules(dot, p - t);
    }
    const float m_tile = warp_max(s);
    if (m_tile == -INFINITY) continue;
    const float m_new = fmaxf(m, m_tile);
    const float corr = expf(m - m_new);  // m = -inf -> 0
    const float pl = valid ? expf(s - m_new) : 0.f;
    l = __fmaf_rn(l, corr, warp_sum(pl));
#pragma unroll
    for (int c = 0; c < kMaxChunks; ++c) acc[c] *= corr;
    const int count = min(32, p - t0 + 1);
    // the values of kAhead keys are asked for before the first is used (each lane holds its own key's page)
    constexpr int kAhead = kMaxChunks <= 4 ? 8 : (kMaxChunks <= 8 ? 4 : 2);
    for (int j0 = 0; j0 < count; j0 += kAhead) {
      float pj[kAhead], vj[kAhead][kMaxChunks];
#pragma unroll
      for (int e = 0; e < kAhead; ++e) {
        pj[e] = __shfl_sync(0xffffffffu, pl, (j0 + e) & 31);
        const int pg = __shfl_sync(0xffffffffu, page, (j0 + e) & 31);
        if (j0 + e >= count) pj[e] = 0.f;
        if (pj[e] == 0.f) continue;          // masked, or too small to count: its value is not read
        const T* vrow = v_pool + ((static_cast<size_t>(pg) * nkv + kvh) * page_size + (t0 + j0 + e) % page_size) * v_row;
#pragma unroll
        for (int c = 0; c < kMaxChunks; ++c) {
          const int i = lane + 32 * c;
          vj[e][c] = i < dv ? to_float(vrow[i]) : 0.f;
        }
      }
#pragma unroll
      for (int e = 0; e < kAhead; ++e) {
        if (pj[e] == 0.f) continue;
#pragma unroll
        for (int c = 0; c < kMaxChunks; ++c) acc[c] = fmaf(pj[e], vj[e][c], acc[c]);
      }
    }
    m = m_new;
  }
  T* orow = out + (static_cast<size_t>(token) * nq + head) * dv;
  const float inv = l > 0.f ? 1.f / l : 0.f;   // a row without any visible key (padding) gives zeros
#pragma unroll
  for (int c = 0; c < kMaxChunks; ++c) {
    const int i = lane + 32 * c;
    if (i < dv) orow[i] = from_float<T>(acc[c] * inv);
  }
}

// Prompt portions in float32: 128 threads hold 32 rows (32 / group consecutive tokens of one request times the query heads
// that share a key head) and walk the keys in the tiles of 32 that the kernel above takes them in; keys and values pass
// through shared memory once for all rows, the next tile's on their way while this one is worked on.  A thread owns four
// rows and, of a tile, the keys c and c + 16: the sum of its two weights and four shuffles are then the sum that 32 lanes
// form by xor shuffles, and every other sum is one chain, so the results are the same bits.  A weight of zero reads no
// value here either (a later token's value may be anything): only a warp that has one takes the loop that asks.
// One warp per token and head reads every key for every row from the L2: 509 tokens, 16 heads of 128 over 8: 574 us; so: 77
// (64 rows of keys and values at once 161; two rows a thread and twice the threads 87, 2,000 tokens in a window of 300 244 against 198).
// A tile of keys takes 32 rows about 5 us, mostly latency: of the softmax (its steps are taken for all rows at once: 10 us less of 88)
// and of reads of shared memory (lanes i and i ^ 1 read the same key: half the passes, 4 % at 1,021 keys).  So the time is that of the
// SM with most tiles of keys.  More row tiles than SMs go in pairs, a CTA with two sets of threads that share nothing: the tile with most
// keys beside that with fewest, the next beside the next; the CTAs take the shared memory that leaves room for no more than an even
// share an SM.  Within a prompt's layers, where CTAs start while the kernel before still holds some SMs: 133 us one by one, 90 in pairs, 78 with
// the softmax's steps taken together.
constexpr int kTileRows = 32, kTileKeys = 32, kRowsOf = 4, kTileThreads = kTileRows / kRowsOf * 16, kPPitch = kTileKeys + 4;
constexpr size_t kMostTileSmem = 227 * 1024;
constexpr size_t attention_tile_smem(int dmax) {
  return sizeof(float) * (static_cast<size_t>(kTileRows + 2 * kTileKeys) * (dmax + 4) + kTileRows * kPPitch);
}

struct TileParams {
  const float* q; const float* k_pool; const float* v_pool; float* out;
  const int* positions; const int* q_start; const int* block_table;
  int entries, table_stride, page_size, nq, nkv, d, dv, per_tile, tiles, window, chunk, sink;
  float scale, softcap;
  const float* slopes; const float* log_r1; const float* log_r2; const float* sinks;
};

template <int DMAX>
__global__ void __launch_bounds__(2 * kTileThreads) paged_attention_tile_kernel(const TileParams p) {
  constexpr int PITCH = DMAX + 4, CG = DMAX > 64 ? 2 : 1;   // CG: groups of four value columns a thread owns
  constexpr size_t SET = attention_tile_smem(DMAX) / sizeof(float);
  extern __shared__ __align__(16) float smem[];
  float* qs = smem + threadIdx.x / kTileThreads * SET;   // [32][PITCH]
  float* ks = qs + kTileRows * PITCH;                   // [32][PITCH]
  float* vs = ks + kTileKeys * PITCH;                   // [32][PITCH]
  float* ps = vs + kTileKeys * PITCH;                   // [32][kPPitch]
  pdl_trigger();
  pdl_wait();
  // the tile's request: every request has its own tiles, the last one (with most keys) first, for all key heads
  const int half = threadIdx.x / kTileThreads, order = half ? p.tiles - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
  if (half && 2 * static_cast<int>(blockIdx.x) + 1 == p.tiles) return;   // of an odd number the one in the middle has no partner
  auto meet = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + half), "n"(kTileThreads) : "memory"); };
  int entry = 0, tile = order / p.nkv, first = 0, tokens = 0;
  for (;; ++entry) {
    if (entry == p.entries) return;
    first = p.q_start[entry];
    tokens = p.q_start[entry + 1] - first;
    const int tiles = (tokens + p.per_tile - 1) / p.per_tile;
    if (tile < tiles) {
      tile = tiles - 1 - tile;
      break;
    }
    tile -= tiles;
  }
  first += tile * p.per_tile;
  tokens = min(p.per_tile, tokens - tile * p.per_tile);
  const int tid = threadIdx.x % kTileThreads, c = tid % 32 / 2, rg = tid / 32 * 2 + tid % 2;
  const int group = p.nq / p.nkv, kvh = order % p.nkv;
  const int* table = p.block_table + static_cast<size_t>(entry) * p.table_stride;
  const int d = p.d, dv = p.dv, quads = d / 4, vquads = dv / 4;

  for (int idx = tid; idx < kTileRows * quads; idx += kTileThreads) {
    const int row = idx / quads, i = idx % quads * 4, t = row / group;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < tokens) v = *reinterpret_cast<const float4*>(p.q + (static_cast<size_t>(first + t) * p.nq + kvh * group + row % group) * d + i);
    *reinterpret_cast<float4*>(qs + row * PITCH + i) = v;
  }
  const float inv_cap = p.softcap > 0.f ? 1.f / p.softcap : 0.f;
  float slope[kRowsOf], r1[kRowsOf], r2[kRowsOf];
  int pos[kRowsOf], w0[kRowsOf];
  float m[kRowsOf], l[kRowsOf];
  float2 acc[kRowsOf][2 * CG];
#pragma unroll
  for (int r = 0; r < kRowsOf; ++r) {
    const int row = rg * kRowsOf + r, t = row / group, head = kvh * group + row % group;
    pos[r] = t < tokens ? p.positions[first + t] : -1;   // -1: no such row; it sees no key
    w0[r] = p.window > 0 ? max(0, pos[r] - p.window + 1) : 0;
    if (p.chunk > 0) w0[r] = max(w0[r], pos[r] / p.chunk * p.chunk);
    slope[r] = p.slopes ? p.slopes[head] : 0.f;
    r1[r] = p.log_r1 ? p.log_r1[head] : 0.f;
    r2[r] = p.log_r2 ? p.log_r2[head] : 0.f;
    m[r] = p.sinks ? p.sinks[head] : (p.sink ? 0.f : -INFINITY);
    l[r] = p.sink || p.sinks ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 2 * CG; ++j) acc[r][j] = make_float2(0.f, 0.f);
  }
  const int p_first = p.positions[first], p_last = p.positions[first + tokens - 1];    // positions ascend within a request
  int lowest = p.window > 0 ? max(0, p_first - p.window + 1) : 0;
  if (p.chunk > 0) lowest = max(lowest, p_first / p.chunk * p.chunk);

  // Four threads copy a row of a tile, 16 bytes at a time, zeros where there is no page; the row's page is looked up a
  // tile ahead of its keys and serves its values too.
  const int crow = tid / (kTileThreads / kTileKeys), cquad = tid % (kTileThreads / kTileKeys);
  auto page_of = [&](int t) { return t <= p_last ? table[t / p.page_size] : -1; };
  auto ask = [&](const float* pool, float* to, int page, int t, int width, int nquads) {
    const float* src = pool + ((static_cast<size_t>(max(page, 0)) * p.nkv + kvh) * p.page_size + t % p.page_size) * width;
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(to + crow * PITCH));
    const int bytes = page >= 0 ? 16 : 0;
    for (int i = cquad; i < nquads; i += kTileThreads / kTileKeys)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + i * 16), "l"(src + i * 4), "r"(bytes) : "memory");
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  int t0 = lowest / kTileKeys * kTileKeys;
  int page = page_of(t0 + crow), next_page = page_of(t0 + kTileKeys + crow);
  ask(p.k_pool, ks, page, t0 + crow, d, quads);
  ask(p.v_pool, vs, page, t0 + crow, dv, vquads);
  for (; t0 <= p_last; t0 += kTileKeys) {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");            // the keys; the values may still be on their way
    meet();
    const int ahead_page = page_of(t0 + 2 * kTileKeys + crow);
    int key_page[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) key_page[n] = page_of(t0 + c + 16 * n);
    float s[kRowsOf][2];
#pragma unroll
    for (int r = 0; r < kRowsOf; ++r) s[r][0] = s[r][1] = 0.f;
    const float* qrow = qs + rg * kRowsOf * PITCH;
    const float* krow = ks + c * PITCH;
#pragma unroll 4
    for (int i = 0; i < d; i += 4) {
      float4 qv[kRowsOf], kv[2];
#pragma unroll
      for (int r = 0; r < kRowsOf; ++r) qv[r] = *reinterpret_cast<const float4*>(qrow + r * PITCH + i);
#pragma unroll
      for (int n = 0; n < 2; ++n) kv[n] = *reinterpret_cast<const float4*>(krow + n * 16 * PITCH + i);
#pragma unroll
      for (int r = 0; r < kRowsOf; ++r)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          s[r][n] = fmaf(qv[r].x, kv[n].x, s[r][n]);
          s[r][n] = fmaf(qv[r].y, kv[n].y, s[r][n]);
          s[r][n] = fmaf(qv[r].z, kv[n].z, s[r][n]);
          s[r][n] = fmaf(qv[r].w, kv[n].w, s[r][n]);
        }
    }
    // every step for all rows before the next one: their shuffles and exponentials then run side by side
    bool valid[kRowsOf][2];
    float top[kRowsOf], sum[kRowsOf], corr[kRowsOf];
#pragma unroll
    for (int r = 0; r < kRowsOf; ++r) {
      const ScoreRules rules{p.scale, p.softcap, inv_cap, slope[r], r1[r], r2[r], p.log_r1 != nullptr};
      top[r] = -INFINITY;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int t = t0 + c + 16 * n;
        valid[r][n] = key_page[n] >= 0 && t <= pos[r] && t >= w0[r];
        s[r][n] = valid[r][n] ? rules(s[r][n], pos[r] - t) : -INFINITY;
        top[r] = fmaxf(top[r], s[r][n]);
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < kRowsOf; ++r) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2 * o));
    bool full = true;                                                 // no weight of this thread's is zero
#pragma unroll
    for (int r = 0; r < kRowsOf; ++r) {
      const bool any = top[r] != -INFINITY;                           // otherwise the row keeps what it has: a factor of one, weights of zero
      const float m_new = any ? fmaxf(m[r], top[r]) : 0.f;
      const float scaled = expf(m[r] - m_new);
      corr[r] = any ? scaled : 1.f;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float w = expf(s[r][n] - m_new);
        s[r][n] = any && valid[r][n] ? w : 0.f;
        full = full && s[r][n] != 0.f;
      }
      sum[r] = __fadd_rn(s[r][0], s[r][1]);
      m[r] = any ? m_new : m[r];
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < kRowsOf; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2 * o);
#pragma unroll
    for (int r = 0; r < kRowsOf; ++r) {
      l[r] = __fmaf_rn(l[r], corr[r], sum[r]);
#pragma unroll
      for (int j = 0; j < 2 * CG; ++j) { acc[r][j].x *= corr[r]; acc[r][j].y *= corr[r]; }
#pragma unroll
      for (int n = 0; n < 2; ++n) ps[(rg * kRowsOf + r) * kPPitch + c + 16 * n] = s[r][n];
    }
    full = __all_sync(0xffffffffu, full);                             // then all 32 keys exist, for all rows of the warp
    meet();                                                  // the keys have been read, all weights are written
    const bool more = t0 + kTileKeys <= p_last;
    if (more) {
      ask(p.k_pool, ks, next_page, t0 + kTileKeys + crow, d, quads);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");          // the values
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    meet();
    auto add_values = [&](auto ask_first, int count) {
      for (int j = 0; j < count; j += 4) {
        float4 pw[kRowsOf];
#pragma unroll
        for (int r = 0; r < kRowsOf; ++r) pw[r] = *reinterpret_cast<const float4*>(ps + (rg * kRowsOf + r) * kPPitch + j);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float4 vv[CG];
#pragma unroll
          for (int g = 0; g < CG; ++g) vv[g] = *reinterpret_cast<const float4*>(vs + (j + e) * PITCH + (g * 64 + c * 4) % DMAX);
#pragma unroll
          for (int r = 0; r < kRowsOf; ++r) {
            const float w = e == 0 ? pw[r].x : e == 1 ? pw[r].y : e == 2 ? pw[r].z : pw[r].w;
            if (decltype(ask_first)::value && w == 0.f) continue;
#pragma unroll
            for (int g = 0; g < CG; ++g) {
              acc[r][2 * g] = __ffma2_rn(make_float2(w, w), make_float2(vv[g].x, vv[g].y), acc[r][2 * g]);
              acc[r][2 * g + 1] = __ffma2_rn(make_float2(w, w), make_float2(vv[g].z, vv[g].w), acc[r][2 * g + 1]);
            }
          }
        }
      }
    };
    if (full) add_values(std::false_type(), kTileKeys);
    else add_values(std::true_type(), min(kTileKeys, p_last - t0 + 1));
    meet();                                                  // the values and the weights have been read
    if (more) ask(p.v_pool, vs, next_page, t0 + kTileKeys + crow, dv, vquads);
    next_page = ahead_page;
  }
#pragma unroll
  for (int r = 0; r < kRowsOf; ++r) {
    const int row = rg * kRowsOf + r, t = row / group;
    if (t >= tokens) continue;
    const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
    float* orow = p.out + (static_cast<size_t>(first + t) * p.nq + kvh * group + row % group) * dv;
#pragma unroll
    for (int g = 0; g < CG; ++g) {
      const int i = g * 64 + c * 4;
      if (i < dv)
        *reinterpret_cast<float4*>(orow + i) = make_float4(acc[r][2 * g].x * inv, acc[r][2 * g].y * inv, acc[r][2 * g + 1].x * inv, acc[r][2 * g + 1].y * inv);
    }
  }
}

template <int DMAX>
int launch_attention_tiles(const TileParams& p, cudaStream_t stream) {
  static DeviceOnce once;
  int sms = 0;
  const int status = configure_once(once, paged_attention_tile_kernel<DMAX>, kMostTileSmem, &sms);
  if (status) return status;
  if (p.tiles <= sms) {                                                // an SM for each: no pairs
    launch(paged_attention_tile_kernel<DMAX>, dim3(p.tiles), dim3(kTileThreads), attention_tile_smem(DMAX), stream, p);
    return launch_status();
  }
  const long long ctas = (p.tiles + 1LL) / 2, share = (ctas + sms - 1) / sms;
  const size_t even = share <= 4 ? ((kMostTileSmem + 1024) / share - 1024) / 128 * 128 : 0, needed = 2 * attention_tile_smem(DMAX);
  launch(paged_attention_tile_kernel<DMAX>, dim3(static_cast<unsigned>(ctas)), dim3(2 * kTileThreads), even > needed ? even : needed, stream, p);
  return launch_status();
}

}  // namespace b200

// q [n, nq, d], keys [pages, nkv, page_size, d], values [pages, nkv, page_size, v_row] of which the first dv columns are read
// (v_row = dv: a pool of its own; v_row = d with v_pool = k_pool: the values are the leading columns of the keys),
// out [n, nq, dv].  softcap <= 0: no cap; slopes (nq floats) may be null; sink 0 or 1.
extern "C" int b200_paged_attention_simt_strided(
    const void* q, const void* k_pool, const void* v_pool, void* out, const int* positions,
    const int* token_entry, const int* block_table, int table_stride, int page_size, int n,
    int nq, int nkv, int d, int dv, int v_row, float scale, int window, float softcap, const float* slopes, int sink,
    int dtype, cudaStream_t stream);

// The same with the mask in blocks (chunk <= 0: none) and the bias by the logarithm of the distance (log_r1, log_r2:
// [nq] floats each, or both null), and a sink of a score per query head (sinks, [nq] floats, or null).
extern "C" int b200_paged_attention_simt_masked(
    const void* q, const void* k_pool, const void* v_pool, void* out, const int* positions,
    const int* token_entry, const int* block_table, int table_stride, int page_size, int n,
    int nq, int nkv, int d, int dv, int v_row, float scale, int window, float softcap, const float* slopes, int sink,
    int chunk, const float* log_r1, const float* log_r2, const float* sinks, int dtype, cudaStream_t stream) {
  using namespace b200;
  if (n <= 0) return 0;
  if (d <= 0 || dv <= 0 || nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 || v_row < dv ||
      (log_r1 == nullptr) != (log_r2 == nullptr))
    return B200_ERR_BAD_SIZE;
  if (dv > 32 * 20 || d > 2048) return B200_ERR_TOO_LARGE;
  dim3 grid(n, (nq + 3) / 4);
  if (grid.y > 65535) return B200_ERR_TOO_LARGE;
  const size_t smem = static_cast<size_t>(4) * d * sizeof(float);
#define B200_SIMT_ATTENTION(CH)                                                                             \
  B200_DISPATCH_DTYPE(dtype, T,                                                                             \
      launch(paged_attention_simt_kernel<T, CH>, dim3(grid), dim3(128), smem, stream,                       \
          static_cast<const T*>(q), static_cast<const T*>(k_pool), static_cast<const T*>(v_pool),          \
          static_cast<T*>(out), positions, token_entry, block_table, table_stride, page_size, nq,           \
          nkv, d, scale, window, dv, softcap, slopes, sink, v_row, chunk, log_r1, log_r2, sinks))
  if (dv <= 64) { B200_SIMT_ATTENTION(2); }
  else if (dv <= 128) { B200_SIMT_ATTENTION(4); }
  else if (dv <= 256) { B200_SIMT_ATTENTION(8); }
  else { B200_SIMT_ATTENTION(20); }
#undef B200_SIMT_ATTENTION
  return launch_status();
}

extern "C" int b200_paged_attention_simt_strided(
    const void* q, const void* k_pool, const void* v_pool, void* out, const int* positions,
    const int* token_entry, const int* block_table, int table_stride, int page_size, int n,
    int nq, int nkv, int d, int dv, int v_row, float scale, int window, float softcap, const float* slopes, int sink,
    int dtype, cudaStream_t stream) {
  return b200_paged_attention_simt_masked(q, k_pool, v_pool, out, positions, token_entry, block_table, table_stride, page_size,
                                          n, nq, nkv, d, dv, v_row, scale, window, softcap, slopes, sink, 0, nullptr, nullptr,
                                          nullptr, dtype, stream);
}

extern "C" int b200_paged_attention_simt_rules(
    const void* q, const void* k_pool, const void* v_pool, void* out, const int* positions,
    const int* token_entry, const int* block_table, int table_stride, int page_size, int n,
    int nq, int nkv, int d, int dv, float scale, int window, float softcap, const float* slopes, int sink,
    int dtype, cudaStream_t stream) {
  if (d > 256 || dv > 256) return B200_ERR_TOO_LARGE;
  return b200_paged_attention_simt_strided(q, k_pool, v_pool, out, positions, token_entry, block_table, table_stride, page_size,
                                           n, nq, nkv, d, dv, dv, scale, window, softcap, slopes, sink, dtype, stream);
}

extern "C" int b200_paged_attention_simt(
    const void* q, const void* k_pool, const void* v_pool, void* out, const int* positions,
    const int* token_entry, const int* block_table, int table_stride, int page_size, int n,
    int nq, int nkv, int d, float scale, int window, int dtype, cudaStream_t stream) {
  return b200_paged_attention_simt_rules(q, k_pool, v_pool, out, positions, token_entry, block_table, table_stride,
                                         page_size, n, nq, nkv, d, d, scale, window, 0.f, nullptr, 0, dtype, stream);
}

// float32, rows of 16-byte multiples, head sizes up to 128, at most 32 query heads a key head: the tiles of a prompt portion.  The
// same results, bit for bit, as the entry points above give.  q_start [entries + 1]: the tokens of entry e are q_start[e] ..
// q_start[e + 1] - 1, at consecutive positions; block_table [entries, table_stride].
extern "C" int b200_paged_attention_tiles(
    const float* q, const float* k_pool, const float* v_pool, float* out, const int* positions, const int* q_start,
    const int* block_table, int entries, int table_stride, int page_size, int n, int nq, int nkv, int d, int dv, float scale,
    int window, float softcap, const float* slopes, int sink, int chunk, const float* log_r1, const float* log_r2,
    const float* sinks, cudaStream_t stream) {
  using namespace b200;
  if (n <= 0 || entries <= 0) return 0;
  if (d <= 0 || dv <= 0 || d % 4 || dv % 4 || nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 ||
      (log_r1 == nullptr) != (log_r2 == nullptr))
    return B200_ERR_BAD_SIZE;
  if (d > 128 || dv > 128 || nq / nkv > kTileRows) return B200_ERR_TOO_LARGE;
  const int per_tile = kTileRows / (nq / nkv);
  const long long tiles = (static_cast<long long>(n) / per_tile + entries) * nkv;      // at least as many as there are; the others return
  if (nkv > 65535 || tiles > 0x7fffffff) return B200_ERR_TOO_LARGE;
  const TileParams p{q, k_pool, v_pool, out, positions, q_start, block_table, entries, table_stride, page_size, nq, nkv, d, dv,
                     per_tile, static_cast<int>(tiles), window, chunk, sink, scale, softcap, slopes, log_r1, log_r2, sinks};
  const int widest = d > dv ? d : dv;
  if (widest <= 32) return launch_attention_tiles<32>(p, stream);
  if (widest <= 64) return launch_attention_tiles<64>(p, stream);
  return launch_attention_tiles<128>(p, stream);
}
