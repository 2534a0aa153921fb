// bfloat16 matrix product C[M,N] = A[M,K] * W[N,K]^T (+ bias) with the weight as the tensor cores' row operand, for some hundred
// rows of A: they are the columns of the accumulator, padded to 32 instead of 128 or 256, and up to 512 of them meet a weight
// tile while it is in shared memory.  A pair of CTAs (cta_group::2) computes 256 features x (n1 + n2) tokens as one or two products
// of up to 256 columns each; a tile's K range can be shared by 2 or 4 pairs (one cluster), which hand each other their shares of
// the partial sums through distributed shared memory.
//   warp 0   producer: TMA loads of 64-wide K blocks, the first ring of weights that are at rest ahead of the wait for the kernel before;
//   warp 1   tensor-core issue (in the pair's leader);
//   warps 2-17  epilogue: a lane has a feature, a warp's stores are 32 neighbouring features of a row of C (64 or 128 bytes),
//            where the kernels of gemm_tcgen05.cu write 16 bytes of 32 rows at a time.
// What bounds it: up to 256 tokens a tile the copies into shared memory (an SM takes 105 bytes a ns, 56 a clock, from a TMA ring
// whose source is in the L2: 175 ns a K block and 0.7 ns a token), beyond that the tensor pipe; with few K blocks the fixed costs, of which
// 0.8 us lie between two kernels, 1.5 before the first product, 1.2 in the exchange of a shared tile.
// Microseconds, float32 sum into C, against the kernels that these products went to before (from cold caches, back to back in a graph):
// 320 x 4,096 x 4,096 17.3 (30.6), 405 x 4,096 x 4,096 19.0 (25.2), 405 x 4,096 x 12,288 40.3 (52.9), 512 x 2,048 x 8,192
// 23.7 (37.6), 768 x 1,024 x 3,072 13.1 (19.4), 1,024 x 4,096 x 4,096 29.7 (35.1); bfloat16: 160 x 4,096 x 1,024 9.0 (12.5).
// Tried and not kept: the SwiGLU epilogue here (gate and up lie in different lanes: 8 us for 416 tokens, none of it under products); clusters of
// 8 CTAs for every size (15 of them find room at once, 33 of four, 74 of two).
//
// Every wait on an mbarrier is bounded: after its limit of polls the kernel records an error code, stops issuing work, frees
// its TMEM and returns.
#include <cuda.h>

#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

namespace b200 {

constexpr int kFeatBM = 128;            // weight rows per CTA = TMEM lanes; a pair has 256
constexpr int kFeatBK = 64;             // 64 bf16 = 128 bytes = one swizzle row
constexpr int kFeatWarps = 16;          // epilogue warps, four for each quarter of the lanes
constexpr int kFeatCols = 16;           // tokens that an epilogue warp finishes at a time
constexpr int kFeatThreads = 64 + 32 * kFeatWarps;

__device__ int g_features_error = 0;

struct FeatureParams {
  void* c;
  const float* bias;
  int M, N, K, ldc;
  int n1, n2;          // tokens a tile: columns of the first and of the second product, multiples of 32, at most 256 each
  int splits;          // pairs (one cluster) that share a tile's K range
  int share;           // splits > 1: columns of the tile that a pair finishes, a multiple of 16
  int wide;            // splits == 1: tiles that are computed whole; of those behind them the two products are items of their own
  int stages, accumulate;
  int weight_ahead;    // no kernel that may still be running writes the weight
};

// What a cluster computes at a time: `count` tokens from `token` on of the 256 features from `feature` on, as the product with the first
// (`first`) and the second (`second`) group of a tile's tokens.
struct FeatureItem {
  int feature, token, count;
  bool first, second;
};
__device__ __forceinline__ FeatureItem feature_item(const FeatureParams& p, int m_tiles, int item) {
  const int behind = item - p.wide, tile = behind < 0 ? item : p.wide + (behind >> 1);
  const int m0 = (tile % m_tiles) * (p.n1 + p.n2), feature = (tile / m_tiles) * 256;
  if (behind < 0) return {feature, m0, p.n1 + p.n2, true, p.n2 > 0};
  if (behind & 1) return {feature, m0 + p.n1, p.n2, false, true};
  return {feature, m0, p.n1, true, false};
}

__device__ __forceinline__ void feat_store(float* p, float v) { *p = v; }
__device__ __forceinline__ void feat_store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// What C holds for the tokens from `token` on of this lane's feature n (the sum that the product is added to).
__device__ __forceinline__ void held_tokens(float (&have)[kFeatCols], const FeatureParams& p, int n, int token) {
  const float* c = static_cast<const float*>(p.c) + static_cast<size_t>(token) * p.ldc + n;
#pragma unroll
  for (int j = 0; j < kFeatCols; ++j) have[j] = n < p.N && token + j < p.M ? c[static_cast<size_t>(j) * p.ldc] : 0.f;
}

// The tokens from `token` on of this lane's feature n: a warp's lanes are 32 neighbouring features of a row of C.
template <typename OutT>
__device__ __forceinline__ void finish_tokens(const float (&v)[kFeatCols], const FeatureParams& p, int n, int token) {
  if (n >= p.N) return;
  OutT* c = static_cast<OutT*>(p.c) + static_cast<size_t>(token) * p.ldc + n;
  const int count = min(kFeatCols, p.M - token);
  if (count == kFeatCols) {
#pragma unroll
    for (int j = 0; j < kFeatCols; ++j) feat_store(c + static_cast<size_t>(j) * p.ldc, v[j]);
  } else {
#pragma unroll
    for (int j = 0; j < kFeatCols; ++j)
      if (j < count) feat_store(c + static_cast<size_t>(j) * p.ldc, v[j]);
  }
}

template <typename OutT>
__global__ void __launch_bounds__(kFeatThreads, 1)
gemm_features_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a1,
                     const __grid_constant__ CUtensorMap map_a2, FeatureParams p) {
  constexpr uint32_t W_BYTES = kFeatBM * kFeatBK * 2, TMEM_COLS = 512;
  const int n1 = p.n1, n2 = p.n2, width = n1 + n2, stages = p.stages, splits = p.splits, share = p.share;
  const uint32_t a1_bytes = static_cast<uint32_t>(n1) * kFeatBK, a2_bytes = static_cast<uint32_t>(n2) * kFeatBK;   // half the rows, 2 bytes
  const uint32_t stage_bytes = W_BYTES + a1_bytes + a2_bytes;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  unsigned char* handed = smem + stages * stage_bytes;            // splits > 1: the other pairs' sums for this pair's share
  uint64_t* full = reinterpret_cast<uint64_t*>(handed + (splits - 1) * share * kFeatBM * 4);
  uint64_t* empty = full + stages;
  uint64_t* acc_full = empty + stages;    // [2]
  uint64_t* acc_empty = acc_full + 2;     // [2], used in the leader
  uint64_t* received = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(received + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank(), rank = crank & 1, leader_rank = crank & ~1u;
  const bool leader = rank == 0;
  const int part = static_cast<int>(crank >> 1);
  const int cluster = blockIdx.x / (2 * splits), clusters = gridDim.x / (2 * splits);
  const int m_tiles = (p.M + width - 1) / width, n_tiles = (p.N + 255) / 256;
  const int tiles = m_tiles * n_tiles, items = splits > 1 ? tiles : p.wide + 2 * (tiles - p.wide);
  const int num_kb = (p.K + kFeatBK - 1) / kFeatBK;
  const int kb0 = static_cast<int>(static_cast<long long>(num_kb) * part / splits);
  const int kb1 = static_cast<int>(static_cast<long long>(num_kb) * (part + 1) / splits);
  const int buffers = width <= 256 ? 2 : 1;           // accumulators in tensor memory, 256 columns apart

  if (warp == 0) {
    mbar_init_warp(full, 2 * stages + 4, 2, 2 * kFeatWarps);
    if (lane == 0) mbar_init(received, splits > 1 ? kFeatWarps * (splits - 1) : 1);
    fence_barrier_init();
    __syncwarp();
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    tcgen05_fence_before();
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");   // every CTA's barriers exist before anything arrives on them
  const uint32_t pair_full = map_to_cta(smem_addr(full), leader_rank);
  int ahead = 0;
  if (warp == 0 && cluster < items && p.weight_ahead) {
    // weights that do not depend on the kernel before this one: the first ring of them is asked for ahead of the wait
    const FeatureItem it = feature_item(p, m_tiles, cluster);
    const uint32_t bytes = 2 * (W_BYTES + (it.first ? a1_bytes : 0) + (it.second ? a2_bytes : 0));
    const int y = it.feature + static_cast<int>(rank) * kFeatBM;
    ahead = min(stages, kb1 - kb0);
    if (elect_one()) {
      for (int i = 0; i < ahead; ++i) {
        if (leader) mbar_expect_tx(full + i, bytes);
        tma_load_2d_pair(smem + i * stage_bytes, &map_w, pair_full + i * 8, (kb0 + i) * kFeatBK, y);
      }
    }
    __syncwarp();
  }
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int quarter = warp & 3, row = quarter * 32 + lane;
  pdl_wait();

  if (warp == 0) {
    // ---------------------------------------------------------------- producer (both CTAs)
    int s = 0, seen = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int item = cluster; item < items && ok; item += clusters) {
      const FeatureItem it = feature_item(p, m_tiles, item);
      const uint32_t bytes = 2 * (W_BYTES + (it.first ? a1_bytes : 0) + (it.second ? a2_bytes : 0));
      const int y = it.feature + static_cast<int>(rank) * kFeatBM;
      const int y1 = it.token + static_cast<int>(rank) * (n1 >> 1);
      const int y2 = it.token + (it.first ? n1 : 0) + static_cast<int>(rank) * (n2 >> 1);
      for (int kb = kb0; kb < kb1; ++kb, ++seen) {
        unsigned char* stage = smem + s * stage_bytes;
        if (seen >= ahead && !mbar_wait_warp(empty + s, phase ^ 1)) { atomicExch(&g_features_error, 1); ok = false; break; }
        if (elect_one()) {
          if (seen >= ahead) {
            if (leader) mbar_expect_tx(full + s, bytes);
            tma_load_2d_pair(stage, &map_w, pair_full + s * 8, kb * kFeatBK, y);
          }
          if (it.first) tma_load_2d_pair(stage + W_BYTES, &map_a1, pair_full + s * 8, kb * kFeatBK, y1);
          if (it.second) tma_load_2d_pair(stage + W_BYTES + a1_bytes, &map_a2, pair_full + s * 8, kb * kFeatBK, y2);
        }
        __syncwarp();
        if (++s == stages) { s = 0; phase ^= 1; }
      }
    }
    if (ok && !stages_returned(empty, stages, s, phase)) atomicExch(&g_features_error, 1);
  } else if (warp == 1) {
    // ---------------------------------------------------------------- tensor-core issue (leader)
    if (leader) {
      const uint32_t idesc1 = umma_idesc_pair(n1), idesc2 = umma_idesc_pair(n2);
      const uint16_t both = static_cast<uint16_t>(3u << leader_rank);
      int s = 0, local = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = cluster; item < items && ok; item += clusters, ++local) {
        const FeatureItem it = feature_item(p, m_tiles, item);
        const int buf = local % buffers;
        const uint32_t acc_phase = (local / buffers) & 1;
        if (!mbar_wait_warp(acc_empty + buf, acc_phase ^ 1)) { atomicExch(&g_features_error, 4); ok = false; break; }
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + buf * 256, tmem_d2 = tmem_d + (it.first ? n1 : 0);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(full + s, phase)) { atomicExch(&g_features_error, 2); ok = false; break; }
          tcgen05_fence_after();
          const uint32_t w_addr = smem_addr(smem + s * stage_bytes), a_addr = w_addr + W_BYTES;
          if (elect_one()) {
            if (it.first) {
#pragma unroll
              for (int k = 0; k < kFeatBK / 16; ++k)
                umma_bf16_pair(tmem_d, umma_desc_sw128(w_addr + k * 32, 16, 1024), umma_desc_sw128(a_addr + k * 32, 16, 1024), idesc1,
                               ((kb - kb0) | k) != 0);
            }
            if (it.second) {
#pragma unroll
              for (int k = 0; k < kFeatBK / 16; ++k)
                umma_bf16_pair(tmem_d2, umma_desc_sw128(w_addr + k * 32, 16, 1024),
                               umma_desc_sw128(a_addr + a1_bytes + k * 32, 16, 1024), idesc2, ((kb - kb0) | k) != 0);
            }
            umma_commit_pair(empty + s, both);
          }
          __syncwarp();
          if (++s == stages) { s = 0; phase ^= 1; }
        }
        if (elect_one()) umma_commit_pair(acc_full + buf, both);
        __syncwarp();
      }
    }
  } else if (splits == 1) {
    // -------------------------------------------------------------------- epilogue (both CTAs)
    const int first = ((warp - 2) >> 2) * kFeatCols, step = kFeatWarps / 4 * kFeatCols;
    int local = 0;
    for (int item = cluster; item < items; item += clusters, ++local) {
      const FeatureItem it = feature_item(p, m_tiles, item);
      const int buf = local % buffers;
      const int n = it.feature + static_cast<int>(rank) * kFeatBM + row;
      const float bias = p.bias != nullptr && n < p.N ? p.bias[n] : 0.f;
      const bool add = sizeof(OutT) == 4 && p.accumulate;
      float next[kFeatCols];              // asked for a chunk ahead: its latency is a chunk's whole time otherwise
      if (add) held_tokens(next, p, n, it.token + first);
      if (!mbar_wait_warp(acc_full + buf, (local / buffers) & 1)) { atomicExch(&g_features_error, 3); break; }
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * 256;
#pragma unroll 1
      for (int c = first; c < it.count; c += step) {
        uint32_t r[kFeatCols];
        tmem_ld_16(taddr + c, r);
        float v[kFeatCols];
#pragma unroll
        for (int j = 0; j < kFeatCols; ++j) v[j] = __uint_as_float(r[j]) + bias + (add ? next[j] : 0.f);
        if (add && c + step < it.count) held_tokens(next, p, n, it.token + c + step);
        finish_tokens<OutT>(v, p, n, it.token + c);
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0 && accumulator_reused(item, clusters, buffers, items)) mbar_arrive_cluster(map_to_cta(smem_addr(acc_empty + buf), leader_rank));
    }
  } else {
    // ------------------------------------ epilogue of a shared tile: every pair hands the others their shares of its partial sums,
    // 16-byte groups of four tokens, the 128 features of a group side by side, and finishes its own share
    const int first = ((warp - 2) >> 2) * kFeatCols, step = kFeatWarps / 4 * kFeatCols;
    const FeatureItem it = feature_item(p, m_tiles, cluster);
    const int n = it.feature + static_cast<int>(rank) * kFeatBM + row;
    const int mine = part * share, end_mine = min(width, mine + share);
    const float bias = p.bias != nullptr && n < p.N ? p.bias[n] : 0.f;
    const bool add = sizeof(OutT) == 4 && p.accumulate;
    float next[kFeatCols];
    if (add) held_tokens(next, p, n, it.token + mine + first);
    bool ok = mbar_wait_warp(acc_full, 0);
    if (!ok) atomicExch(&g_features_error, 3);
    tcgen05_fence_after();
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
#pragma unroll 1
    for (int other = 1; other < splits; ++other) {
      const int to = (part + other) % splits, begin = to * share, end = min(width, begin + share);
      const int slot = part < to ? part : part - 1;
      const uint32_t base = map_to_cta(smem_addr(handed), static_cast<uint32_t>(2 * to) + rank) + static_cast<uint32_t>((slot * (share / 4) * kFeatBM + row) * 16);
#pragma unroll 1
      for (int c = begin + first; c < end; c += step) {
        uint32_t r[kFeatCols];
        tmem_ld_16(taddr + c, r);
#pragma unroll
        for (int j = 0; j < kFeatCols; j += 4)
          asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(base + static_cast<uint32_t>(((c - begin + j) >> 2) * kFeatBM * 16)),
                       "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3])
                       : "memory");
      }
    }
    __syncwarp();
    // one lane for each pair that was handed something: an arrival waits for the stores before it, so they are all issued first
    if (lane < splits && lane != part) mbar_arrive_cluster(map_to_cta(smem_addr(received), static_cast<uint32_t>(2 * lane) + rank));
    __syncwarp();
    if (ok && !mbar_wait_cluster_warp(received, 0)) { atomicExch(&g_features_error, 5); ok = false; }
    const float4* got = reinterpret_cast<const float4*>(handed) + row;
#pragma unroll 1
    for (int c = mine + first; c < end_mine; c += step) {
      uint32_t r[kFeatCols];
      tmem_ld_16(taddr + c, r);
      float v[kFeatCols];
#pragma unroll
      for (int j = 0; j < kFeatCols; ++j) v[j] = 0.f;
#pragma unroll 1
      for (int q = 0; q < splits; ++q) {          // in the order of the K ranges
        if (q == part) {
#pragma unroll
          for (int j = 0; j < kFeatCols; ++j) v[j] += __uint_as_float(r[j]);
        } else {
          const int slot = q < part ? q : q - 1;
#pragma unroll
          for (int j = 0; j < kFeatCols; j += 4) {
            const float4 t = got[(slot * (share / 4) + ((c - mine + j) >> 2)) * kFeatBM];
            v[j] += t.x; v[j + 1] += t.y; v[j + 2] += t.z; v[j + 3] += t.w;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kFeatCols; ++j) v[j] = v[j] + bias + (add ? next[j] : 0.f);
      if (add && c + step < end_mine) held_tokens(next, p, n, it.token + c + step);
      if (ok) finish_tokens<OutT>(v, p, n, it.token + c);
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_relaxed();                 // nobody leaves while the tensor cores of its pair still read its shared memory
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// 2-D bf16 row-major [rows, cols] matrix, box = [box_rows, 64 columns], 128-byte swizzle
static int features_map(CUtensorMap* map, const void* base, int rows, int cols, int box_rows) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return 10005;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
  const cuuint32_t box[2] = {kFeatBK, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 10006;
}

// The tokens of a tile and the pairs that share its K range: what a model of the time says is fastest, in ns, fitted to 1,500
// measured products.  A K block takes the longer of its copies and its products; a launch 5.9 us beside them, 5.0 and 5.7 with two
// and four pairs a tile and their exchange; no product is faster than its weights arrive.  It picks within 3 % of the best
// form measured in the mean.  Shared tiles only where all clusters are resident at once.
static void features_shape(int M, int N, int K, int sm_count, int* n1, int* n2, int* splits) {
  const int kb = (K + kFeatBK - 1) / kFeatBK, n_tiles = (N + 255) / 256;
  const float arrive = 2.f * N * static_cast<float>(K) / 4100.f;
  auto block = [](int columns) { return fmaxf(1.4f * columns, 173.f + 0.68f * columns); };
  float best = 1e30f;
  int before = 0;
  for (int parts = (M + 511) / 512; parts <= 64; ++parts) {
    const int width = ((M + parts - 1) / parts + 31) / 32 * 32;
    if (width > 512) continue;
    if (width == before || (width < 64 && parts > 1)) break;
    before = width;
    const long tiles = static_cast<long>((M + width - 1) / width) * n_tiles;
    const int half = (width / 2 + 31) / 32 * 32, pairs = sm_count / 2 > 0 ? sm_count / 2 : 1;
    auto take = [&](float time, int a, int b, int s) {
      if (time < best) { best = time; *n1 = a; *n2 = b; *splits = s; }
    };
    const long full = tiles / pairs, rest = tiles % pairs;
    if (width <= 256) {
      take(5900.f + fmaxf(arrive, kb * (full + (rest > 0)) * block(width)), width, 0, 1);
      for (const int s : {2, 4}) {
        const long resident = static_cast<long>(sm_count) * (s == 2 ? 33 : 15) / 148;
        if (s <= kb && tiles <= resident)
          take((s == 2 ? 5000.f : 5700.f) + fmaxf(arrive, (kb + s - 1) / s * block(width)) + 26.f * width / s, width, 0, s);
      }
    }
    if (width >= 128 && 2 * rest <= pairs)
      take(5900.f + fmaxf(arrive, kb * (full * block(width) + (rest > 0 ? block(half) : 0.f))) + 8.f * width, half, width - half, 1);
    else if (width > 256)
      take(5900.f + fmaxf(arrive, kb * (full + 1) * block(width)) + 8.f * width, half, width - half, 1);
  }
}

constexpr size_t kFeatRing = 224 * 1024, kFeatTail = 1024 + 512;

template <typename OutT>
static int launch_features(const CUtensorMap& w, const CUtensorMap& a1, const CUtensorMap& a2, FeatureParams p, cudaStream_t stream) {
  auto kernel = gemm_features_kernel<OutT>;
  static DeviceOnce once;
  int sm_count = 0;
  if (int e = configure_once(once, kernel, kFeatRing + kFeatTail, &sm_count)) return e;
  const int width = p.n1 + p.n2;
  const size_t stage = kFeatBM * kFeatBK * 2 + static_cast<size_t>(width) * kFeatBK;
  p.share = p.splits > 1 ? ((width + p.splits - 1) / p.splits + 15) / 16 * 16 : 0;
  const size_t handed = static_cast<size_t>(p.splits - 1) * p.share * kFeatBM * 4;
  if (handed + 2 * stage > kFeatRing) return B200_ERR_BAD_SIZE;
  p.stages = static_cast<int>((kFeatRing - handed) / stage);
  if (p.stages > 12) p.stages = 12;
  const int tiles = ((p.M + width - 1) / width) * ((p.N + 255) / 256);
  const int resident = sm_count / (2 * p.splits);
  p.wide = tiles;
  if (p.splits == 1 && p.n2 > 0) {
    // tiles beyond the last full round of pairs: their two products on a pair each where all of them then fit one round
    const int rest = tiles % resident;
    if (2 * rest <= resident) p.wide = tiles - rest;
  }
  const int items = p.wide + 2 * (tiles - p.wide);
  const int clusters = p.splits > 1 || items < resident ? items : resident;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(clusters * 2 * p.splits);
  config.blockDim = dim3(kFeatThreads);
  config.dynamicSmemBytes = kFeatRing + kFeatTail;       // one CTA an SM: all of its tensor memory is taken
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * p.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&config, kernel, w, a1, a2, p);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

}  // namespace b200

using namespace b200;

// Read and clear the error flag set by a bounded wait that ran out.  Synchronises the device.
extern "C" int b200_gemm_features_error() {
  int v = 0, zero = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  cudaMemcpyFromSymbol(&v, g_features_error, sizeof(int));
  cudaMemcpyToSymbol(g_features_error, &zero, sizeof(int));
  return v;
}

// The tile and the number of pairs to its K range that are chosen for a product on a GPU with `sm_count` SMs (callable without a GPU).
extern "C" int b200_gemm_features_shape(int M, int N, int K, int sm_count, int* n1, int* n2, int* splits) {
  if (M <= 0 || M > 16384 || N <= 0 || K <= 0 || sm_count <= 0 || !n1 || !n2 || !splits) return B200_ERR_BAD_SIZE;
  features_shape(M, N, K, sm_count, n1, n2, splits);
  return 0;
}

// C[M,N] (ldc) = A[M,K] * W[N,K]^T + bias, or (accumulate, float output) C += that.
// n1, n2: tokens of a tile in its first and second product; splits: pairs of CTAs that share a tile's K range (1, 2, 4); all 0:
// chosen by size.  M up to 16,384.  weight_ahead: no kernel that may still be running on the stream writes W, which is then read ahead of
// the wait for it.
extern "C" int b200_gemm_features(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, int ldc, int out_f32,
                                  int accumulate, int n1, int n2, int splits, int weight_ahead, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 8 != 0 || ldc < N) return B200_ERR_BAD_SIZE;
  if (accumulate && !out_f32) return B200_ERR_BAD_SIZE;
  if (M > 16384) return B200_ERR_TOO_LARGE;
  if (n1 == 0 && n2 == 0 && splits == 0) {
    int device = 0, sm_count = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device);
    features_shape(M, N, K, sm_count, &n1, &n2, &splits);
  }
  if (n1 < 32 || n1 > 256 || n1 % 32 || n2 < 0 || n2 > 256 || n2 % 32 || (splits != 1 && splits != 2 && splits != 4) || splits > (K + kFeatBK - 1) / kFeatBK)
    return B200_ERR_BAD_SIZE;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) return B200_ERR_BAD_SIZE;
  FeatureParams p{C, bias, M, N, K, ldc, n1, n2, splits, 0, 0, 0, accumulate, weight_ahead};
  CUtensorMap w, a1, a2;
  if (int e = features_map(&w, W, N, K, kFeatBM)) return e;
  if (int e = features_map(&a1, A, M, K, n1 / 2)) return e;
  if (int e = features_map(&a2, A, M, K, (n2 > 0 ? n2 : n1) / 2)) return e;
  return out_f32 ? launch_features<float>(w, a1, a2, p, stream) : launch_features<__nv_bfloat16>(w, a1, a2, p, stream);
}
