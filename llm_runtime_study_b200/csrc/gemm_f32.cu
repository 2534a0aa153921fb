// True 32-bit matrix product for the verification path: C[M,N] = A[M,K] * W[N,K]^T (+ bias).
// Plain FFMA on CUDA cores: no tensor-core instruction is issued, so no operand is
// ever rounded to TF32 or bfloat16 (nn.Linear layout, mini_llm/nn/attention.py:102-111).
//
// The order of an output's sum is a function of K alone: k is cut into segments of kSegment and segments into at most
// eight blocks (block_length).  A segment is accumulated in ascending k by fused multiply-adds from zero, a block is the
// sum of its segments in ascending order, the output the sum of its blocks in ascending order.  Every kernel below keeps
// that order, so a row's bits do not depend on how many other rows are in the batch or on which kernel took it.
#include <cooperative_groups.h>

#include "common.cuh"

namespace b200 {

namespace cg = cooperative_groups;

constexpr int kSegment = 128;
// Blocks of 1,024, longer ones where K is longer than eight of those: whole segments.
inline int block_length(int K) {
  const int eighth = ((K + 7) / 8 + kSegment - 1) / kSegment * kSegment;
  return eighth > 8 * kSegment ? eighth : 8 * kSegment;
}

// ------------------------------------------------------------------------------------------ tiles
// A cluster per BM x BN tile, one CTA for each block of K, (BM / TM) x (BN / TN) threads with TM x TN outputs each (rows
// ty * 4 + g BM / (TM / 4), columns likewise: every fragment is one 16-byte read that neighbouring threads share or lay
// side by side).  Two buffers of BK columns in shared memory and AHEAD more in registers.  AHEAD is two for tiles of 64 x 64, of which
// an SM often holds only one or two CTAs (one step ahead: 509 x 1024 x 3072 80 us against 78), and one for tiles of 128 x 64, whose
// registers are better spent on a third CTA an SM (509 x 6144 x 1024: 147 us with two steps and 170 registers, 140 with one and 168).
// A wide read of shared memory takes two passes instead of four if lanes i and i ^ 1, or i and i ^ 2, read the same address: the
// lowest bit of a lane is tx's, the next one ty's.  Transposed stores of four columns fall on four times the same bank; rows are
// therefore kept at row ^ 2 k for the four-column group that starts at k.  The two took 509 x 1024 x 3072 from 89.6 to 77.7 us, 509 x 1024
// x 2048 from 63.2 to 54.8, 509 x 4096 x 1024 from 108 to 97.
// The sums of finished segments wait in shared memory, one private 16-byte column per thread, so that registers hold one
// accumulator an output and two or three CTAs fit an SM; at the end the CTAs of a cluster share out the outputs and add the
// blocks' sums up through distributed shared memory.  Bound by the FMA pipe, the reads of shared memory beside it and the last
// wave: 509 x 6144 x 1024 140 us (46 TFLOP/s of the 74 that the pipe could do; 53 in the SMs that get three tiles of the 2.6 on
// average).
// GATED: the columns are two factors in blocks of eight and act(g) * u leaves instead; a kernel less per feed-forward part (a step of few rows
// through a small model is bound by its launches) and its pass over memory: 509 x 6144 x 1024 146 and 4.3 us in two kernels, 148 in
// one (154 while only the half of the threads that own gate columns worked).
// VEC: rows of A and W start on 16-byte boundaries and K is a multiple of 4; otherwise elements are loaded one by one.
constexpr int kBK = 16;
constexpr size_t kMostSmem = 227 * 1024;
// A cluster's CTAs lie in one GPC, whose last SMs may not hold another cluster.
inline int usable_sms(int blocks, int sms) { return sms > 8 * (blocks - 1) ? sms - 4 * (blocks - 1) : (sms + 1) / 2; }
constexpr size_t tile_smem(int bm, int bn) { return sizeof(float) * (static_cast<size_t>(bm) * bn + 2 * kBK * (bm + 4 + bn + 4)); }

template <int BM, int BN, int TM, int TN, bool VEC, bool GATED>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), BM == 128 ? 3 : 4)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K, int lda, int ldc, int block, int act) {
  constexpr int THREADS = (BM / TM) * (BN / TN), BK = kBK, PA = BM + 4, PW = BN + 4;
  constexpr int RPP = THREADS / 4;                                  // rows a pass of 16-byte loads covers
  constexpr int LA = BM / RPP, LW = BN / RPP;
  constexpr int SM_ = BM / (TM / 4), SN_ = BN / (TN / 4);           // distance of a thread's groups of four rows, columns
  constexpr int TX = BN / TN, AHEAD = BM == 128 ? 1 : 2;
  static_assert((TX == 8 || TX == 16) && THREADS == 128 && SM_ % 32 == 0 && SN_ % 32 == 0, "lanes of a warp");
  static_assert(TM % 4 == 0 && TN % 4 == 0 && kSegment % BK == 0 && BM % RPP == 0 && BN % RPP == 0, "tile shape");
  extern __shared__ __align__(16) float smem[];
  float* As = smem;                                                 // [2][BK][PA]
  float* Ws = As + 2 * BK * PA;                                     // [2][BK][PW]
  float4* sums = reinterpret_cast<float4*>(Ws + 2 * BK * PW);       // [TM * TN / 4][THREADS]
  pdl_trigger();
  pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  const int blocks = cluster.num_blocks(), rank = cluster.block_rank();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x / blocks * BN;
  const int k_begin = rank * block, k_end = min(K, k_begin + block);
  // lane bits 0 .. 4: tx, ty, tx, tx, ty with eight columns of threads; tx, ty, tx, tx, tx with sixteen
  const int tx = TX == 8 ? (tid & 1) | (tid >> 1 & 6) : (tid & 1) | (tid >> 1 & 2) | (tid >> 1 & 12);
  const int ty = TX == 8 ? (tid >> 1 & 1) | (tid >> 3 & 2) | (tid >> 5) * 4 : (tid >> 1 & 1) | (tid >> 5) * 2;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;
  struct Rows { float4 a[LA], w[LW]; };

  auto load4 = [&](const float* base, int row, int rows, int ld, int k) -> float4 {
    if (row >= rows || k >= k_end) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float* p = base + static_cast<size_t>(row) * ld + k;
    if (VEC) return *reinterpret_cast<const float4*>(p);
    return make_float4(p[0], k + 1 < k_end ? p[1] : 0.f, k + 2 < k_end ? p[2] : 0.f, k + 3 < k_end ? p[3] : 0.f);
  };
  auto fetch = [&](Rows& r, int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) r.a[i] = load4(A, m0 + lrow + RPP * i, M, lda, k0 + lk);
#pragma unroll
    for (int i = 0; i < LW; ++i) r.w[i] = load4(W, n0 + lrow + RPP * i, N, K, k0 + lk);
  };
  auto stash = [&](const Rows& r, int buf) {
    float* as = As + (buf * BK + lk) * PA + (lrow ^ 2 * lk);
    float* ws = Ws + (buf * BK + lk) * PW + (lrow ^ 2 * lk);
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      as[RPP * i] = r.a[i].x; as[PA + RPP * i] = r.a[i].y; as[2 * PA + RPP * i] = r.a[i].z; as[3 * PA + RPP * i] = r.a[i].w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      ws[RPP * i] = r.w[i].x; ws[PW + RPP * i] = r.w[i].y; ws[2 * PW + RPP * i] = r.w[i].z; ws[3 * PW + RPP * i] = r.w[i].w;
    }
  };

  // two neighbouring columns share a register pair: one packed instruction does two fused multiply-adds, each
  // rounded as by itself
  float2 acc[TM][TN / 2];
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
  };
  clear();
  // `spent` goes on its way to hold the rows AHEAD steps on; with two, `next` was asked for a step ago
  auto step = [&](int k0, int buf, Rows& spent, const Rows& next) {
    const bool more = k0 + BK < k_end;
    fetch(spent, k0 + AHEAD * BK);
    const float* as = As + buf * BK * PA;
    const float* ws = Ws + buf * BK * PW;
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM];
      float2 w[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(as + (ty * 4 ^ k / 4 * 8) + k * PA + i / 4 * SM_);
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(ws + (tx * 4 ^ k / 4 * 8) + k * PW + j / 4 * SN_);
        w[j / 2] = make_float2(v.x, v.y);
        w[j / 2 + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i], a[i]), w[j], acc[i][j]);
    }
    if ((k0 + BK - k_begin) % kSegment == 0 || !more) {             // the segment is complete
      const bool first = k0 - k_begin < kSegment;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
          float4* s = sums + (i * (TN / 4) + j) * THREADS + tid;
          const float4 t = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *s;
          *s = make_float4(t.x + acc[i][2 * j].x, t.y + acc[i][2 * j].y, t.z + acc[i][2 * j + 1].x, t.w + acc[i][2 * j + 1].y);
        }
      clear();
    }
    if (more) stash(AHEAD == 2 ? next : spent, buf ^ 1);
    __syncthreads();
  };
  Rows even, odd;
  fetch(even, k_begin);
  if (AHEAD == 2) fetch(odd, k_begin + BK);
  stash(even, 0);
  __syncthreads();
  for (int k0 = k_begin; k0 < k_end; k0 += 2 * BK) {
    step(k0, 0, even, odd);
    if (k0 + BK < k_end) step(k0 + BK, 1, AHEAD == 2 ? odd : even, even);
  }
  if (blocks > 1) cluster.sync();                                   // every block's sums are in its CTA's shared memory
  const bool wide = VEC && ldc % 4 == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0;
  auto total = [&](int q, int thread) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b = 0; b < blocks; ++b) {
      const float4 t = (blocks > 1 ? cluster.map_shared_rank(sums, b) : sums)[q * THREADS + thread];
      v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
    }
    return v;
  };
  if (GATED) {
    // A thread's columns and those of the thread four behind it (tx + 2: eight columns on) are each other's factors: the two take turns.
    const int upper = tid >> 2 & 1, gate = tid & ~4, n0_ = n0 + (tx & ~2) * 4;
    for (int q = rank + blocks * upper; q < TM * TN / 4; q += 2 * blocks) {
      const int i = q / (TN / 4), j = q % (TN / 4);
      const int m = m0 + ty * 4 + i / 4 * SM_ + i % 4, n = n0_ + j * SN_;
      if (m >= M || n >= N) continue;
      const float4 v = total(q, gate), u = total(q, gate + 4);
      float out[4] = {v.x, v.y, v.z, v.w};
      const float other[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        out[e] = gate_act(bias ? out[e] + bias[n + e] : out[e], act) * (bias ? other[e] + bias[n + 8 + e] : other[e]);
      float* c = C + static_cast<size_t>(m) * ldc + n / 16 * 8 + n % 8;
      if (wide) *reinterpret_cast<float4*>(c) = make_float4(out[0], out[1], out[2], out[3]);
      else
#pragma unroll
        for (int e = 0; e < 4; ++e) c[e] = out[e];
    }
  } else for (int q = rank; q < TM * TN / 4; q += blocks) {
    const int i = q / (TN / 4), j = q % (TN / 4);
    const int m = m0 + ty * 4 + i / 4 * SM_ + i % 4, n = n0 + tx * 4 + j * SN_;
    const float4 v = total(q, tid);
    if (m >= M || n >= N) continue;
    float* c = C + static_cast<size_t>(m) * ldc + n;
    const float out[4] = {v.x, v.y, v.z, v.w};
    if (bias == nullptr && wide && n + 4 <= N) {
      *reinterpret_cast<float4*>(c) = v;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n + e < N) c[e] = out[e] + (bias ? bias[n + e] : 0.f);
    }
  }
  if (blocks > 1) cluster.sync();                                   // nobody leaves while its sums are being read
}

// ------------------------------------------------------------------------------------------ few rows
// Up to eight rows of A per CTA beside kRowsW rows of W: the time is that of streaming W.  A thread forms the sums of one
// segment of one weight row against every row of A (1 x 151,936 x 1024: 93 us = 6.7 TB/s, where tiles took 708); kSegments segments of all the CTA's weight rows are in shared memory
// at a time, copied there 16 bytes at a time without passing through registers, two or three CTAs an SM so that one's copies
// run under the other's arithmetic.  Rows are padded by 16 bytes: the eight threads of a 128-byte phase then read from
// different banks.  GATED is a kernel of its own: chosen at run time, its rows cost every product 3 to 25 % (8 x 1024 x 3072 21.5 us, 18.0; 24 x 512
// x 512 9.3, 7.7).
constexpr int kRowsW = 8, kSegments = 16, kPass = kSegments * kSegment;
constexpr size_t few_smem(int pitch) { return sizeof(float) * kRowsW * pitch; }

template <int MB, bool GATED>
__global__ void __launch_bounds__(kRowsW * kSegments)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                    float* __restrict__ C, int M, int N, int K, int lda, int ldc, int pitch, int block, int act) {
  extern __shared__ __align__(16) float ws[];                    // [kRowsW][pitch]
  __shared__ float sums[kSegments][MB][kRowsW];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * kRowsW, m0 = blockIdx.y * MB;
  const int n = tid % kRowsW, seg = tid / kRowsW;
  // a gated product takes four rows of one factor and the four of the other eight rows on
  auto row_of = [&](int r) {
    if constexpr (GATED) return static_cast<int>(blockIdx.x) / 2 * 16 + blockIdx.x % 2 * 4 + r / 4 * 8 + r % 4;
    else return n0 + r;
  };
  const int rows = min(MB, M - m0);
  const float* a0 = A + static_cast<size_t>(m0) * lda;
  float total = 0.f, part = 0.f;                                 // of output (tid / kRowsW, tid % kRowsW), for tid < MB * kRowsW
  for (int k0 = 0; k0 < K; k0 += kPass) {
    const int span = min(kPass, K - k0), quads = span / 4;       // K is a multiple of 4 here
    for (int r = tid / 32; r < kRowsW; r += kRowsW * kSegments / 32) {
      if (row_of(r) >= N) continue;                              // never read: that row's outputs are not stored
      const float* src = W + static_cast<size_t>(row_of(r)) * K + k0;
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(ws + r * pitch));
      for (int q = tid % 32; q < quads; q += 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + q * 16), "l"(src + q * 4) : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    float acc[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) acc[m] = 0.f;
    const int first = seg * kSegment, last = min(first + kSegment, span);
    if (n0 + n < N) {                                            // (as many of a gated product's rows are there: all)
      const float* wrow = ws + n * pitch;
#pragma unroll 4
      for (int k = first; k < last; k += 4) {
        const float4 w = *reinterpret_cast<const float4*>(wrow + k);
#pragma unroll
        for (int m = 0; m < MB; ++m) {
          const float4 a = *reinterpret_cast<const float4*>(a0 + static_cast<size_t>(m < rows ? m : 0) * lda + k0 + k);
          acc[m] = fmaf(a.x, w.x, acc[m]);
          acc[m] = fmaf(a.y, w.y, acc[m]);
          acc[m] = fmaf(a.z, w.z, acc[m]);
          acc[m] = fmaf(a.w, w.w, acc[m]);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) sums[seg][m][n] = acc[m];
    __syncthreads();
    if (tid < MB * kRowsW) {
      const int used = (span + kSegment - 1) / kSegment;
      for (int s = 0; s < used; ++s) {
        part += sums[s][tid / kRowsW][tid % kRowsW];
        if ((k0 + (s + 1) * kSegment) % block == 0) {             // the block is complete
          total += part;
          part = 0.f;
        }
      }
    }
    __syncthreads();                                             // the sums and the rows have been read
  }
  if constexpr (GATED) {
    const int m = m0 + tid / kRowsW, nn = row_of(n);
    const bool stored = tid < MB * kRowsW && m < M && nn < N;
    const float out = (K % block ? total + part : total) + (stored && bias ? bias[nn] : 0.f);
    const float other = __shfl_down_sync(0xffffffffu, out, 4);
    if (stored && n < 4) C[static_cast<size_t>(m) * ldc + blockIdx.x * 4 + n] = gate_act(out, act) * other;
  } else if (tid < MB * kRowsW) {
    const int m = m0 + tid / kRowsW, nn = n0 + tid % kRowsW;
    if (m < M && nn < N) C[static_cast<size_t>(m) * ldc + nn] = (K % block ? total + part : total) + (bias ? bias[nn] : 0.f);
  }
}

// ------------------------------------------------------------------------------------------ short rows
// K of at most one segment: 64 x 64 tiles, 4 x 4 outputs a thread, one buffer.  The tiles above prepare for long K (two steps of
// loads ahead, sums of segments in shared memory), which costs more than it saves in a few steps of kBK columns: 24 x 39 x 19 3.1 us
// against 4.8, 509 x 753 x 35 4.9 against 6.1, 8 x 1441 x 95 6.8 against 7.3.
__global__ void __launch_bounds__(256)
gemm_f32_short_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                      float* __restrict__ C, int M, int N, int K, int lda, int ldc) {
  constexpr int BM = 64, BN = 64, BK = kBK;
  __shared__ float As[BK][BM + 4], Ws[BK][BN + 4];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid & 15, ty = tid >> 4, lrow = tid >> 2, lk = (tid & 3) * 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + lk + i, am = m0 + lrow, wn = n0 + lrow;
      As[lk + i][lrow] = am < M && k < K ? A[static_cast<size_t>(am) * lda + k] : 0.f;
      Ws[lk + i][lrow] = wn < N && k < K ? W[static_cast<size_t>(wn) * K + k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[static_cast<size_t>(m) * ldc + n] = acc[i][j] + (bias ? bias[n] : 0.f);
    }
  }
}

// The kernel for a product by its size (vec: rows are 16-byte vectors) and the GPU's number of SMs.
inline int choose_kernel(int M, int N, int K, bool vec, bool gated, int sms) {
  const int blocks = (K + block_length(K) - 1) / block_length(K);
  const long long small = static_cast<long long>((M + 63) / 64) * ((N + 63) / 64) * blocks;
  const long long large = static_cast<long long>((M + 127) / 128) * ((N + 63) / 64) * blocks;
  // Up to 8 rows the weights cross once and that is the time (1 x 1024 x 3072: 7.9 us against 37.6 with tiles; 8 x 151,936 x
  // 1024: 285 against 495).  Every further eight rows read them again, from the L2 while the product is small: 24 x 6144
  // x 1024 37.5 against 39.0, 24 x 1024 x 3072 25.6 against 37.8, 64 x 6144 x 1024 83 against 40.
  // Tiles of 128 rows do a third more arithmetic per byte of shared memory read, tiles of 64 leave less of the last wave empty.  A
  // product takes 9 us and 22.9 for each 64 x 64 x 1024 that the busiest SM gets, or 11 and 43.2 for each 128 x 64 x 1024 (509 x
  // 6144 x 1024: 140 us with 128 rows, 146 with 64; 700 x 4096 x 1024: 140, 123; 130 x 6144 x 1024: 96, 54; 2048 x 4096 x 1024:
  // 313, 329).  One CTA of 128 rows an SM has nobody to work under its loads (509 x 1024 x 2048, the weights in HBM: 68 us, 57 with
  // 64 rows).  Clusters cannot use every SM to the last slot (700 x 1024 x 3072, 96 clusters of three: 140, 100).
  // Few rows: up to about seven CTAs an SM at once (ten up to four rows), 8 us a round of them from K of 128 on (K beyond 512: as the weights
  // stream), where tiles take 3 us and 0.034 a column.  So beyond one round a short K goes to tiles (9 x 6400 x 256: 15.6 us against
  // 12.2, 24 x 9400 x 1024: 48 against 38), and so does K up to 160 beyond four rows (8 x 6400 x 64: 6.1 against 5.6, 20 x 2880 x 64: 9.0 against 5.4)
  // except K up to 64 in a third of a round (8 x 64 x 64: 4.9 against 5.4, 24 x 512 x 64: 5.4 both).
  // Short rows: up to 112 columns that are not whole 16-byte vectors and up to 32 that are, while the tiles are few.
  const long long ctas = static_cast<long long>((N + kRowsW - 1) / kRowsW) * ((M + 7) / 8), rounds = (ctas + 7 * sms - 1) / (7 * sms);
  const float few_us = rounds * (8.f + (K > 512 ? (K - 512) / 128.f : 0.f)), tiles_us = 3.f + 0.034f * (K < 1024 ? K : 1024);
  const bool few = M <= 2 || (M <= 24 && K <= 64 && ctas <= 400) || (M <= 4 && (K > 160 || ctas <= 10 * sms)) || (M <= 8 && K >= 512) ||
                   (K > 160 && (M <= 8 || (M <= 24 && small < sms)) && few_us <= tiles_us);
  if (vec && few) return 1;
  if (K <= (vec ? 32 : 112) && small <= 512 && !gated) return 4;
  const int block = block_length(K), usable = usable_sms(blocks, sms);
  const float depth = (K < block ? K : block) / 1024.f;
  const float small_us = 9.f + 22.9f * depth * ((small + usable - 1) / usable), large_us = 11.f + 43.2f * depth * ((large + usable - 1) / usable);
  return large > usable && large_us < small_us ? 3 : 2;
}

template <int BM, int BN, int TM, int TN, bool VEC, bool GATED>
int launch_tiles(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldc, int act, cudaStream_t stream) {
  static DeviceOnce once;
  int sms = 0;
  const int status = configure_once(once, gemm_f32_tile_kernel<BM, BN, TM, TN, VEC, GATED>, kMostSmem, &sms);
  if (status) return status;
  const int block = block_length(K), blocks = (K + block - 1) / block;
  // Launched while the kernel before still holds some SMs, the CTAs would crowd on the others, three where two suffice (509 x 4096 x
  // 1024 in a prompt's layers: 144 us against 97 with two an SM): each takes as much shared memory as leaves no room for one more than an even
  // share, and no more than that: what is left caches the loads (64 x 1024 x 3072, one CTA an SM: 45.5 us with all of it, 40.0; 509 x 1024 x
  // 3072, two: 80.6, 79.3).
  const int usable = usable_sms(blocks, sms);
  const long long share = (static_cast<long long>((N + BN - 1) / BN) * blocks * ((M + BM - 1) / BM) + usable - 1) / usable;
  const size_t even = share <= (BM == 128 ? 2 : 3) ? ((kMostSmem + 1024) / (share + 1) / 128 + 1) * 128 - 1024 : 0;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3((N + BN - 1) / BN * blocks, (M + BM - 1) / BM);
  config.blockDim = dim3((BM / TM) * (BN / TN));
  config.dynamicSmemBytes = even > tile_smem(BM, BN) ? even : tile_smem(BM, BN);
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = blocks;
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&config, gemm_f32_tile_kernel<BM, BN, TM, TN, VEC, GATED>, A, W, bias, C, M, N, K, lda, ldc, block, act);
  return launch_status();
}

template <int MB, bool GATED>
int launch_few(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldc, int act, cudaStream_t stream) {
  static DeviceOnce once;
  const int status = configure_once(once, gemm_f32_few_kernel<MB, GATED>, few_smem(kPass + 4));
  if (status) return status;
  const dim3 grid((N + kRowsW - 1) / kRowsW, (M + MB - 1) / MB);
  const int pitch = (K < kPass ? K : kPass) + 4;      // a short K takes less shared memory: more CTAs an SM
  launch(gemm_f32_few_kernel<MB, GATED>, grid, dim3(kRowsW * kSegments), few_smem(pitch), stream, A, W, bias, C, M, N, K, lda, ldc, pitch,
         block_length(K), act);
  return launch_status();
}

}  // namespace b200

// `kernel`: 0 chooses by size; 1: few rows, 2: tiles of 64 x 64, 3: tiles of 128 x 64, 4: short rows (for tests and measurements).
// `act` (ACT_SILU, ACT_GELU_TANH): the rows of W are two factors in blocks of eight, [g0..g7 | u0..u7 | ...], and C [M, N / 2] is act(g) * u,
// each product rounded as it would be stored; otherwise 0.
extern "C" int b200_gemm_f32_gated(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda,
                                   int ldc, int kernel, int act, cudaStream_t stream) {
  using namespace b200;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldc < (act ? N / 2 : N)) return B200_ERR_BAD_SIZE;
  if (act && (N % 16 || M > 65535 || (act != ACT_SILU && act != ACT_GELU_TANH))) return B200_ERR_BAD_SIZE;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(W) % 16 == 0;
  if (kernel == 0) {
    static DeviceOnce once;
    int sms = 0;
    if (const int status = configure_once(once, gemm_f32_short_kernel, 0, &sms)) return status;
    kernel = choose_kernel(M, N, K, vec, act != 0, sms);
  }
  if ((M + 63) / 64 > 65535) return B200_ERR_TOO_LARGE;
  if (kernel == 1) {
    if (!vec) return B200_ERR_BAD_SIZE;
#define B200_F32_FEW(MB)                                                                   \
  (act ? launch_few<MB, true>(A, W, bias, C, M, N, K, lda, ldc, act, stream)                \
       : launch_few<MB, false>(A, W, bias, C, M, N, K, lda, ldc, act, stream))
    if (M == 1) return B200_F32_FEW(1);
    if (M == 2) return B200_F32_FEW(2);
    return M <= 4 ? B200_F32_FEW(4) : B200_F32_FEW(8);
#undef B200_F32_FEW
  }
  if (kernel == 4) {
    if (K > kSegment || act) return B200_ERR_BAD_SIZE;
    launch(gemm_f32_short_kernel, dim3((N + 63) / 64, (M + 63) / 64), dim3(256), 0, stream, A, W, bias, C, M, N, K, lda, ldc);
    return launch_status();
  }
#define B200_F32_TILES(BM, TN, VEC)                                                                                 \
  (act ? launch_tiles<BM, 64, 8, TN, VEC, true>(A, W, bias, C, M, N, K, lda, ldc, act, stream)                       \
       : launch_tiles<BM, 64, 8, TN, VEC, false>(A, W, bias, C, M, N, K, lda, ldc, act, stream))
  if (kernel == 3) return vec ? B200_F32_TILES(128, 8, true) : B200_F32_TILES(128, 8, false);
  return vec ? B200_F32_TILES(64, 4, true) : B200_F32_TILES(64, 4, false);
#undef B200_F32_TILES
}

// The kernel that is chosen for rows of 16-byte vectors on a GPU with `sm_count` SMs (callable without a GPU).
extern "C" int b200_gemm_f32_choice(int M, int N, int K, int gated, int sm_count) {
  return M > 0 && N > 0 && K > 0 && sm_count > 0 ? b200::choose_kernel(M, N, K, K % 4 == 0, gated != 0, sm_count) : 0;
}

extern "C" int b200_gemm_f32_variant(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda,
                                     int ldc, int kernel, cudaStream_t stream) {
  return b200_gemm_f32_gated(A, W, bias, C, M, N, K, lda, ldc, kernel, 0, stream);
}

extern "C" int b200_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M,
                             int N, int K, int lda, int ldc, cudaStream_t stream) {
  return b200_gemm_f32_variant(A, W, bias, C, M, N, K, lda, ldc, 0, stream);
}
