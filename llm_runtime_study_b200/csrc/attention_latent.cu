// bfloat16 tensor-core attention of many query heads over ONE shared row per token whose leading columns are also
// the value (latent attention with the up-projections moved to the query's side), built once per pair of sizes
// (-DLATENT_RANK=<value columns> -DLATENT_ROT=<further key columns>, both multiples of 16).
//
// A CTA takes up to BM = 64 rows: consecutive query tokens of one request times the heads of one group of at most 64
// heads.  Keys are streamed in tiles of 32 rows through shared memory (cp.async, two stages) from the request's pages.
// Eight warps: warp w owns rows 16 (w & 3) .. + 15 and the value columns of half (w >> 2); the two warps of a row group
// each form the scores S = Q K^T (mma.sync m16n8k16, float accumulation) of half of the tile's keys and exchange them through
// shared memory, run the same online softmax in float32, round P to bfloat16 and multiply it with their half of the value
// columns, read transposed out of the key tile.  Both forming all scores made that 70 % of a warp's products.  Rows of more than 868
// columns leave no room for the exchange and still do; so do rows of less than 80, whose few products cost less than it.
// Before the exchange and with it: 32 heads over rows of 576 columns, one prompt of 1,733 tokens 633 and 541 us, of 300 tokens 49.3
// and 43.0, single tokens of 100 requests over 2,049 rows 264 and 213; 4 heads over rows of 32 columns, a prompt of 300 tokens beside
// 24 single tokens over 1,500 rows 38.7 and 47.2.
// Key t is visible to a query at position p iff t <= p and (window == 0 or t > p - window).  With a sink every head's sum has
// one more term exp(sink[head]), which belongs to no key.
#include "common.cuh"
#include "mma.cuh"

#if !defined(LATENT_RANK) || !defined(LATENT_ROT)
#error "compile with -DLATENT_RANK=<value columns> -DLATENT_ROT=<further key columns>"
#endif
static_assert(LATENT_RANK % 16 == 0 && LATENT_RANK >= 16 && LATENT_RANK <= 512, "the value width must be 16..512 in steps of 16");
static_assert(LATENT_ROT % 16 == 0 && LATENT_ROT >= 0, "the further key columns come in steps of 16");

namespace b200 {

using bf16 = __nv_bfloat16;
constexpr int DV = LATENT_RANK, DK = LATENT_RANK + LATENT_ROT;
constexpr int BM = 64, BN = 32, NT = 256;
constexpr int LDS = DK + 8;                 // padded row: ldmatrix rows fall into different banks
constexpr int KSTEPS = DK / 16;
constexpr int DVH = DV / 2;                 // value columns of one warp
constexpr int OTILES = DVH / 8;
constexpr int kTileBytes = (BM + 2 * BN) * LDS * 2, kExchangeBytes = NT * 32;    // eight scores a thread
// else both warps form all scores: there is no room, or a warp's few products cost less than the exchange
constexpr bool kShareScores = DK >= 80 && kTileBytes + kExchangeBytes <= 227 * 1024;
constexpr int kSmemBytes = kTileBytes + (kShareScores ? kExchangeBytes : 0);
// CTAs that a multiprocessor holds: what the cut of single tokens' keys into parts counts on (two_fit in ops/attention_latent.py)
constexpr int kResident = DV <= 144 && 2 * (kSmemBytes + 1024) <= 228 * 1024 ? 2 : 1;

struct LatentParams {
  const bf16* q;            // [n, heads, DK]
  const bf16* pool;         // [pages, page_size, DK]
  bf16* out;                // [n, heads, DV]
  const int* positions;     // [n]
  const int* block_table;   // [entries, table_stride]
  const int* tile_entry;    // per tile: entry, first token (index into the batch's rows), tokens
  const int* tile_start;
  const int* tile_count;
  int table_stride, page_size, heads, group_heads, tokens_per_tile, window;
  float scale_log2;
  const float* sink;        // [heads] or null
  // a tile's keys cut into `splits` parts (single tokens only): CTA z takes its share of the key tiles and leaves
  // (maximum, sum) and the unnormalised output of row token * heads + head in scratch memory for the merge kernel
  int splits;
  float* part_o;    // [rows][splits][DV]
  float* part_ml;   // [rows][splits][2]
};

// Several threads copy a key row: its page is looked up once for all of them, a tile ahead of the copies (three prompts of 1,733 tokens in
// all, 32 heads over rows of 576 columns: 323 us with a lookup before every 16-byte copy, so 247; single tokens of 8 requests 40.7
// and 32.9 us).  Rows of less than 64 columns have fewer copies than a row has threads: the others look up nothing.
constexpr int kRowThreads = DK >= 64 ? NT / BN : (DK >= 32 ? 4 : 2);
__device__ __forceinline__ const bf16* key_row(const LatentParams& p, const int* table, int t, int lo, int hi) {
  if (t < lo || t > hi || threadIdx.x >= BN * kRowThreads) return nullptr;
  const int page = table[t / p.page_size];
  return page >= 0 ? p.pool + (static_cast<size_t>(page) * p.page_size + t % p.page_size) * DK : nullptr;
}
__device__ __forceinline__ void load_key_tile(bf16* ks, const LatentParams& p, const bf16* row) {
  if (kRowThreads * BN < NT && threadIdx.x >= BN * kRowThreads) return;
  const bf16* src = row != nullptr ? row : p.pool;
  const int bytes = row != nullptr ? 16 : 0;
  ks += threadIdx.x / kRowThreads * LDS;
#pragma unroll
  for (int ch = threadIdx.x % kRowThreads; ch < DK / 8; ch += kRowThreads) cp_async_16(ks + ch * 8, src + ch * 8, bytes);
}

__global__ void __launch_bounds__(NT, kResident)
latent_attention_kernel(const LatentParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* qs = reinterpret_cast<bf16*>(smem_raw);
  bf16* ks = qs + BM * LDS;
  float4* exchange = reinterpret_cast<float4*>(smem_raw + kTileBytes);      // [row group][half][2][lane]
  pdl_trigger();
  pdl_wait();
  const int tile = blockIdx.x, hgroup = blockIdx.y;
  const int entry = p.tile_entry[tile], start = p.tile_start[tile], count = p.tile_count[tile];
  const int hg = min(p.group_heads, p.heads - hgroup * p.group_heads);
  const int* table = p.block_table + static_cast<size_t>(entry) * p.table_stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rg = warp & 3, half = warp >> 2;

  // the rows of this thread: r0 = 16 rg + lane / 4 and r0 + 8; row r is token r / hg, head r % hg of the tile
  int pos[2], row_token[2], row_head[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = rg * 16 + (lane >> 2) + i * 8;
    const int tl = r / hg, hl = r - tl * hg;
    const bool valid = tl < count && tl < p.tokens_per_tile;
    row_token[i] = valid ? start + tl : -1;
    row_head[i] = hgroup * p.group_heads + hl;
    pos[i] = valid ? p.positions[start + tl] : -1;
  }
  const int p_first = p.positions[start], p_last = p.positions[start + count - 1];
  const int lo = p.window > 0 ? max(0, p_first - p.window + 1) : 0, hi = p_last;

  // Q tile
  {
    constexpr int CH = DK / 8;
    for (int c = threadIdx.x; c < BM * CH; c += NT) {
      const int r = c / CH, ch = c - r * CH;
      const int tl = r / hg, hl = r - tl * hg;
      const bool valid = tl < count && tl < p.tokens_per_tile;
      const bf16* src = valid ? p.q + (static_cast<size_t>(start + tl) * p.heads + hgroup * p.group_heads + hl) * DK + ch * 8 : p.q;
      cp_async_16(qs + r * LDS + ch * 8, src, valid ? 16 : 0);
    }
  }
  int t_begin = (lo / BN) * BN;
  int tiles = hi >= t_begin ? (hi - t_begin) / BN + 1 : 0;
  if (p.splits > 1) {          // this CTA's share of the key tiles
    const int per = (tiles + p.splits - 1) / p.splits;
    const int first_tile = min(tiles, static_cast<int>(blockIdx.z) * per);
    tiles = min(tiles - first_tile, per);
    t_begin += first_tile * BN;
  }
  const int in_tile = threadIdx.x / kRowThreads;             // which of a tile's rows this thread copies
  if (tiles > 0) load_key_tile(ks, p, key_row(p, table, t_begin + in_tile, lo, hi));
  const bf16* next_row = tiles > 1 ? key_row(p, table, t_begin + BN + in_tile, lo, hi) : nullptr;
  cp_async_commit();

  float o[OTILES][4];
#pragma unroll
  for (int j = 0; j < OTILES; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  if (p.sink != nullptr && blockIdx.z == 0) {       // the first part of a token's keys holds the sink: it starts the maximum and sum
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (row_head[i] < p.heads) {
        m[i] = p.sink[row_head[i]] * 1.4426950408889634f;
        l[i] = 1.f;
      }
  }

  for (int kt = 0; kt < tiles; ++kt) {
    const int t0 = t_begin + kt * BN;
    bf16* kcur = ks + (kt & 1) * BN * LDS;
    if (kt + 1 < tiles) load_key_tile(ks + ((kt + 1) & 1) * BN * LDS, p, next_row);
    next_row = kt + 2 < tiles ? key_row(p, table, t0 + 2 * BN + in_tile, lo, hi) : nullptr;
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    // S = Q K^T for this warp's 16 rows and the tile's 32 keys
    float s[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
    if constexpr (kShareScores) {
#pragma unroll 4
      for (int kk = 0; kk < KSTEPS; ++kk) {          // s[0], s[1]: this warp's sixteen keys
        uint32_t a[4], b[4];
        ldmatrix_x4(a, qs + (rg * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDS + kk * 16 + (lane >> 4) * 8);
        ldmatrix_x4(b, kcur + (half * 16 + (lane & 7) + (lane >> 4) * 8) * LDS + kk * 16 + ((lane >> 3) & 1) * 8);
        mma_bf16(s[0], a, b[0], b[1]);
        mma_bf16(s[1], a, b[2], b[3]);
      }
      float4* mine = exchange + (rg * 2 + half) * 64 + lane;
      mine[0] = make_float4(s[0][0], s[0][1], s[0][2], s[0][3]);
      mine[32] = make_float4(s[1][0], s[1][1], s[1][2], s[1][3]);
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + rg) : "memory");       // the two warps of the row group
      const float4* theirs = exchange + (rg * 2 + (half ^ 1)) * 64 + lane;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float4 t = theirs[32 * j];
        const float other[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[2 + j][e] = half ? s[j][e] : other[e];
          s[j][e] = half ? other[e] : s[j][e];
        }
      }
    } else {
#pragma unroll 4
      for (int kk = 0; kk < KSTEPS; ++kk) {
        uint32_t a[4], b[2][4];
        ldmatrix_x4(a, qs + (rg * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDS + kk * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int j = 0; j < 2; ++j)
          ldmatrix_x4(b[j], kcur + (j * 16 + (lane & 7) + (lane >> 4) * 8) * LDS + kk * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(s[j], a, b[j >> 1][(j & 1) * 2], b[j >> 1][(j & 1) * 2 + 1]);
      }
    }
    // mask, online softmax (base 2)
    float m_new[2] = {m[0], m[1]};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = e >> 1;
        const int t = t0 + j * 8 + (lane & 3) * 2 + (e & 1);
        const bool seen = pos[i] >= 0 && t <= pos[i] && (p.window == 0 || t > pos[i] - p.window);
        s[j][e] = seen ? s[j][e] * p.scale_log2 : -INFINITY;
        m_new[i] = fmaxf(m_new[i], s[j][e]);
      }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      m_new[i] = fmaxf(m_new[i], __shfl_xor_sync(0xffffffffu, m_new[i], 1));
      m_new[i] = fmaxf(m_new[i], __shfl_xor_sync(0xffffffffu, m_new[i], 2));
    }
    float corr[2], sum[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float base = m_new[i] == -INFINITY ? 0.f : m_new[i];
      corr[i] = exp2f(m[i] - base);        // m = -inf: 0
      m[i] = m_new[i];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float pv = exp2f(s[j][i * 2 + e] - base);
          s[j][i * 2 + e] = pv;
          sum[i] += pv;
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 1);
      sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 2);
      l[i] = l[i] * corr[i] + sum[i];
    }
#pragma unroll
    for (int j = 0; j < OTILES; ++j) {
      o[j][0] *= corr[0]; o[j][1] *= corr[0];
      o[j][2] *= corr[1]; o[j][3] *= corr[1];
    }
    // O += P V, V = this warp's half of the leading columns of the key rows
#pragma unroll
    for (int kk = 0; kk < BN / 16; ++kk) {
      uint32_t a[4];
      a[0] = pack_bf16(s[2 * kk][0], s[2 * kk][1]);
      a[1] = pack_bf16(s[2 * kk][2], s[2 * kk][3]);
      a[2] = pack_bf16(s[2 * kk + 1][0], s[2 * kk + 1][1]);
      a[3] = pack_bf16(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
      for (int j = 0; j < OTILES; j += 2) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, kcur + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDS + half * DVH + j * 8 + (lane >> 4) * 8);
        mma_bf16(o[j], a, b[0], b[1]);
        if (j + 1 < OTILES) mma_bf16(o[j + 1], a, b[2], b[3]);
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  if (p.splits > 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (row_token[i] < 0 || row_head[i] >= p.heads) continue;
      const size_t slot = (static_cast<size_t>(row_token[i]) * p.heads + row_head[i]) * p.splits + blockIdx.z;
      if (half == 0 && (lane & 3) == 0) {
        p.part_ml[slot * 2] = m[i];
        p.part_ml[slot * 2 + 1] = l[i];
      }
      float* dst = p.part_o + slot * DV + half * DVH + (lane & 3) * 2;
#pragma unroll
      for (int j = 0; j < OTILES; ++j) *reinterpret_cast<float2*>(dst + j * 8) = make_float2(o[j][i * 2], o[j][i * 2 + 1]);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (row_token[i] < 0 || row_head[i] >= p.heads || (rg * 16 + (lane >> 2) + i * 8) / hg >= p.tokens_per_tile) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    bf16* dst = p.out + (static_cast<size_t>(row_token[i]) * p.heads + row_head[i]) * DV + half * DVH + (lane & 3) * 2;
#pragma unroll
    for (int j = 0; j < OTILES; ++j)
      *reinterpret_cast<__nv_bfloat162*>(dst + j * 8) = __floats2bfloat162_rn(o[j][i * 2] * inv, o[j][i * 2 + 1] * inv);
  }
}

// out[row] = sum_z 2^(m_z - M) o_z / sum_z 2^(m_z - M) l_z over the parts of a row's keys, M the largest maximum.
// The parts' factors are formed once, a lane a part (at most 64 parts), and a thread owns four columns: 4.5 us for 256 rows of 512
// columns in 16 parts (13.4 with every factor formed by every thread behind its loads).
__global__ void __launch_bounds__(128)
latent_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, bf16* __restrict__ out, int splits) {
  __shared__ float factor[64];
  pdl_trigger();
  pdl_wait();
  const size_t row = blockIdx.x;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    const float2* ml = reinterpret_cast<const float2*>(part_ml) + row * splits;
    float2 mine[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) mine[i] = lane + 32 * i < splits ? ml[lane + 32 * i] : make_float2(-INFINITY, 0.f);
    const float top = warp_max(fmaxf(mine[0].x, mine[1].x));
    float f[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) f[i] = mine[i].x == -INFINITY ? 0.f : exp2f(mine[i].x - top);
    const float total = warp_sum(f[0] * mine[0].y + f[1] * mine[1].y);
    const float inv = total > 0.f ? 1.f / total : 0.f;
    factor[lane] = f[0] * inv;
    factor[lane + 32] = f[1] * inv;
  }
  __syncthreads();
  for (int c = threadIdx.x * 4; c < DV; c += 512) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* src = part_o + row * splits * DV + c;
#pragma unroll 8
    for (int z = 0; z < splits; ++z) {
      const float f = factor[z];
      if (f == 0.f) continue;            // a part without a visible key holds no output
      const float4 v = *reinterpret_cast<const float4*>(src + static_cast<size_t>(z) * DV);
      acc.x = fmaf(f, v.x, acc.x);
      acc.y = fmaf(f, v.y, acc.y);
      acc.z = fmaf(f, v.z, acc.z);
      acc.w = fmaf(f, v.w, acc.w);
    }
    __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(out + row * DV + c);
    dst[0] = __floats2bfloat162_rn(acc.x, acc.y);
    dst[1] = __floats2bfloat162_rn(acc.z, acc.w);
  }
}

DeviceOnce latent_once;

}  // namespace b200

extern "C" int b200_attention_latent_rank() { return b200::DV; }
extern "C" int b200_attention_latent_rot() { return LATENT_ROT; }

// q [n, heads, DK], pool [pages, page_size, DK], out [n, heads, DV]; tiles: (entry, first row, rows) of consecutive
// tokens of one entry, at most tokens_per_tile = max(1, 64 / heads) each.  splits > 1 (every tile is token t alone, tile t):
// the keys of a token are cut into that many parts, merged by a second launch; scratch holds splits * (DV + 2) floats a row.
extern "C" int b200_attention_latent_bf16(const void* q, const void* pool, void* out, const int* positions, const int* block_table,
                                          int table_stride, int page_size, int heads, float scale, int window, const float* sink, const int* tile_entry,
                                          const int* tile_start, const int* tile_count, int num_tiles, int splits, float* scratch,
                                          long scratch_floats, cudaStream_t stream) {
  using namespace b200;
  if (num_tiles <= 0) return 0;
  if (heads <= 0 || page_size <= 0 || window < 0 || splits < 1 || splits > 64) return B200_ERR_BAD_SIZE;
  // parts only for single tokens (one tile a token): the scratch rows are token * heads + head
  if (splits > 1 && (scratch == nullptr || scratch_floats < static_cast<long>(num_tiles) * heads * splits * (DV + 2))) return 10004;
  const int status = configure_once(latent_once, latent_attention_kernel, kSmemBytes);
  if (status != 0) return status;
  LatentParams p{};
  p.q = static_cast<const bf16*>(q);
  p.pool = static_cast<const bf16*>(pool);
  p.out = static_cast<bf16*>(out);
  p.positions = positions;
  p.block_table = block_table;
  p.tile_entry = tile_entry;
  p.tile_start = tile_start;
  p.tile_count = tile_count;
  p.table_stride = table_stride;
  p.page_size = page_size;
  p.heads = heads;
  p.group_heads = heads < BM ? heads : BM;
  p.tokens_per_tile = BM / p.group_heads;
  p.window = window;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.sink = sink;
  p.splits = splits;
  if (splits > 1) {
    p.tokens_per_tile = 1;
    p.part_o = scratch;
    p.part_ml = scratch + static_cast<size_t>(num_tiles) * heads * splits * DV;
  }
  dim3 grid(num_tiles, (heads + p.group_heads - 1) / p.group_heads, splits);
  if (grid.y > 65535) return B200_ERR_TOO_LARGE;
  launch(latent_attention_kernel, grid, dim3(NT), kSmemBytes, stream, p);
  if (splits > 1) launch(latent_merge_kernel, dim3(num_tiles * heads), dim3(128), 0, stream, p.part_o, p.part_ml, p.out, splits);
  return launch_status();
}
