// Gated GQA attention over the paged fp16 K/V pool.
//
// attention_prepare_kernel <- attention_prepare (attention.metal:14-50) + the cache append that the
//                             reference does inside attention_scan (:126-133)
// attention_scan_kernel    <- attention_scan   (attention.metal:103-183), row by row: queries of one row, and passes whose
//                             queries have few rows on average
// attention_tile_kernel    <- the same, for the queries of several rows of the other passes
// attention_group_kernel   <- the same, where the contexts of those passes are short
// attention_reduce_kernel  <- attention_reduce (attention.metal:185-216)
//
// K/V pool of one layer: [physical block][4 kv heads][blockTokens][256] fp16, so the 16 tokens of a tile of
// one kv head are 8 KB contiguous. A per-slot block table maps logical to physical blocks (the reference
// reaches the same effect through Metal sparse-buffer page mappings, device.cpp:147-198).
//
// Split-K: the reference uses max(1, 8/rows) splits (forward.cpp:92), which leaves a 148-SM part idle on a
// long single-row context and makes the reduction order depend on the batch. Here the number of splits of a decode
// row depends only on how many tokens that row attends to, so a sequence that decodes gets the same arithmetic whether
// it runs alone, batched or beside a prompt (the rows of a prompt or a draft do not: see attention_launch). One CTA
// serves the four query heads that share a kv head, so K and V are read once per group.
#include <algorithm>
#include <mutex>
#include "act_image.cuh"
#include "ops.h"
#include "tcgen05.cuh"

namespace infdev {
namespace {

constexpr int kQHeads = 16, kKvHeads = 4, kDim = 256, kGroup = kQHeads / kKvHeads, kTile = 16;
constexpr int kPartialStride = kDim + 4;  // 260 floats keeps every record 16-byte aligned for the float4 stores

// Row -> query. In a decode pass every query is one row, so query `row` is the answer; probing it first saves a chain
// of dependent loads at the head of every CTA (queryCount bounds the probe).
__device__ __forceinline__ const infdev_query& query_of_row(const infdev_query* queries, int queryCount, uint32_t row) {
  const infdev_query& guess = queries[min(row, uint32_t(queryCount - 1))];
  if (row >= guess.start && row < guess.start + guess.count)
    return guess;
  while (row >= queries->start + queries->count)
    ++queries;
  return *queries;
}

// Splits of a row that attends to `attended` tokens: 64-token pieces, at most maxSplits, each a multiple of
// the 16-token tile. The piece length trades the fixed cost of a CTA (query load, first tile fetch, partial store)
// against the number of CTAs in flight; it depends only on the row's own context, never on the batch.
__device__ __forceinline__ void split_range(uint32_t attended, uint32_t maxSplits, uint32_t split, uint32_t& begin, uint32_t& end, uint32_t& count) {
  count = min(maxSplits, (attended + 63u) / 64u);
  const uint32_t per = (((attended + count - 1) / count) + kTile - 1) / kTile * kTile;
  begin = min(attended, split * per);
  end = min(attended, begin + per);
}

// One warp per (row, head), eight consecutive dims a lane: heads 0..15 are queries, 16..19 keys (which also store the value head). A CTA
// of 256 threads per head spent its time on two barriers and a chain of single loads: 128 rows 5.6 us, 3.5 now. ALIGNED: all
// operands lie on 16-byte boundaries (a caller's views may start at any element).
template <bool ALIGNED> __device__ __forceinline__ void load_eight(float (&to)[8], const float* from) {
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    const float4 v = ALIGNED ? *reinterpret_cast<const float4*>(from + i) : make_float4(from[i], from[i + 1], from[i + 2], from[i + 3]);
    to[i] = v.x, to[i + 1] = v.y, to[i + 2] = v.z, to[i + 3] = v.w;
  }
}
// Sum of the squares of a head's 256 dims, eight a lane, in the order in which a warp for every 32 dims adds them: partners 16, 8, 4, 2
// and 1 dims apart, then the eight warps in turn. What a key is stored as, and with it a sequence's tokens, hangs on that order.
__device__ __forceinline__ float head_square_sum(const float (&v)[8], int lane) {
  const bool upper = lane & 2, odd = lane & 1;  // bits 4 and 3 of the lane's dims
  float part[4], half[2];  // each step halves the dims that a lane still sums for
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float own = upper ? v[4 + j] : v[j], other = __shfl_xor_sync(0xffffffffu, upper ? v[j] : v[4 + j], 2);
    part[j] = __fadd_rn(__fmul_rn(own, own), __fmul_rn(other, other));
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    half[j] = (odd ? part[2 + j] : part[j]) + __shfl_xor_sync(0xffffffffu, odd ? part[j] : part[2 + j], 1);
  float sum = (upper ? half[1] : half[0]) + __shfl_xor_sync(0xffffffffu, upper ? half[0] : half[1], 2);
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  float total = __shfl_sync(0xffffffffu, sum, 0);
#pragma unroll
  for (int i = 4; i < 32; i += 4)
    total += __shfl_sync(0xffffffffu, sum, i);
  return total;
}
__device__ __forceinline__ uint4 pack_eight(const float (&v)[8]) {
  return make_uint4(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]), pack_half2(v[4], v[5]), pack_half2(v[6], v[7]));
}
template <bool ALIGNED>
__global__ void __launch_bounds__(256) attention_prepare_kernel(const float* qg, const float* rawK, const float* rawV, const float* qNorm,
                                                                const float* kNorm, const float* rope, const infdev_query* queries, int queryCount,
                                                                const int32_t* table, int tableStride, int blockTokens, int heads, float* q, __half* cacheK,
                                                                __half* cacheV) {
  pdl_launch_dependents();
  pdl_wait();
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), row = item / 20, head = item % 20, lane = threadIdx.x & 31;
  const bool query = head < kQHeads;
  if (item >= heads || (query && !qg))  // K/V store only (mtp_store_kv, attention.metal:53-100)
    return;
  const int local = query ? head : head - kQHeads;
  float v[8], weight[8], values[8];
  load_eight<ALIGNED>(v, (query ? qg + (size_t(row) * kQHeads + local) * kDim * 2 : rawK + (size_t(row) * kKvHeads + local) * kDim) + lane * 8);
  load_eight<ALIGNED>(weight, (query ? qNorm : kNorm) + lane * 8);
  if (!query)
    load_eight<ALIGNED>(values, rawV + (size_t(row) * kKvHeads + local) * kDim + lane * 8);
  const infdev_query& info = query_of_row(queries, queryCount, row);
  const uint32_t position = info.position + row - info.start;
  // what hangs on the position is under way while the squares are added
  float angle[2][8];  // lanes 0..7: cos, sin of pairs 8 (lane % 4) .. + 3, then of the next four
  if (lane < 8) {
    const float* entry = rope + (size_t(position) * 32 + (lane & 3) * 8) * 2;
    load_eight<ALIGNED>(angle[0], entry);
    load_eight<ALIGNED>(angle[1], entry + 8);
  }
  const size_t block = query ? 0 : table[size_t(info.slot) * tableStride + position / blockTokens];
  const float scale = rsqrtf(head_square_sum(v, lane) / float(kDim) + 1.0e-6f);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    v[i] = v[i] * scale * weight[i];
  // dims d and d + 32 of the first 64 turn together: lanes 0..3 and 4..7
  float other[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    other[i] = __shfl_xor_sync(0xffffffffu, v[i], 4);
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = v[i] * angle[i >> 2][2 * (i & 3)] + (lane < 4 ? -other[i] : other[i]) * angle[i >> 2][2 * (i & 3) + 1];
  }
  if (query) {
    float* to = q + (size_t(row) * kQHeads + local) * kDim + lane * 8;
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      if (ALIGNED)
        *reinterpret_cast<float4*>(to + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      else
        to[i] = v[i], to[i + 1] = v[i + 1], to[i + 2] = v[i + 2], to[i + 3] = v[i + 3];
    }
    return;
  }
  const size_t at = ((block * kKvHeads + local) * blockTokens + position % blockTokens) * kDim + lane * 8;
  if (ALIGNED) {
    *reinterpret_cast<uint4*>(cacheK + at) = pack_eight(v);
    *reinterpret_cast<uint4*>(cacheV + at) = pack_eight(values);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      cacheK[at + i] = __float2half_rn(v[i]), cacheV[at + i] = __float2half_rn(values[i]);
  }
}

// 16-byte asynchronous copy global -> shared; `bytes` = 0 writes zeros instead (a token past the end of the piece).
__device__ __forceinline__ void copy_async16(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// grid (maxSplits, 4 kv heads, rows), 128 threads. The 16-token K and V tiles of the piece are copied into a
// double buffer in shared memory with cp.async one tile ahead of the arithmetic, so the walk over the piece is not a
// chain of load latencies. Both contractions run on the tensor cores as m16n8k16 with fp16 operands split hi + lo where
// they are not fp16 already: warp 0 scores the tile's 16 tokens for the four query heads of the group, then warp w
// accumulates the weighted values of dims 64w .. 64w+63 for all four heads.
// SINGLES: grid (maxSplits + 1, 4 kv heads, queries), for the queries of one row of a pass whose other queries the tile kernel
// takes, beside that kernel: launched after it and early, it reads nothing that kernel writes and does not wait for it. The
// tile kernel lets it start only after its own wait, so what the kernels before both wrote is there; the fence keeps this
// CTA's reads behind. One CTA does wait, so that the end of this kernel still means the end of all before it.
template <bool SINGLES>
__global__ void __launch_bounds__(128, 6) attention_scan_kernel(const float* q, const __half* cacheK, const __half* cacheV,
                                                                const infdev_query* queries, int queryCount, const int32_t* table, int tableStride,
                                                                int blockTokens, uint32_t maxSplits, float* partials) {
  pdl_launch_dependents();
  const uint32_t split = blockIdx.x, kvHead = blockIdx.y;
  if (!SINGLES) {
    pdl_wait();
  } else {
    if (split == maxSplits) {
      if (!kvHead && !blockIdx.z)
        pdl_wait();
      return;
    }
    __threadfence();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const infdev_query& info = SINGLES ? queries[blockIdx.z] : query_of_row(queries, queryCount, blockIdx.z);
  if (SINGLES && info.count != 1)
    return;
  const uint32_t row = SINGLES ? info.start : blockIdx.z;
  const uint32_t attended = info.position + (row - info.start) + 1;
  uint32_t begin, end, count;
  split_range(attended, maxSplits, split, begin, end, count);
  if (split >= count)
    return;
  __shared__ float scores[kGroup][kTile];
  // [buffer][K, V][token][dim]; rows padded by 16 bytes so that the eight token rows one ldmatrix phase reads hit different banks
  __shared__ __align__(16) __half tiles[2][2][kTile][kDim + 8];
  const int32_t* slotTable = table + size_t(info.slot) * tableStride;
  auto fetch = [&](uint32_t tile, int buffer) {
    const size_t block = slotTable[tile / blockTokens];
    const size_t base = ((block * kKvHeads + kvHead) * blockTokens + tile % blockTokens) * kDim;
    // 16 tokens x 512 bytes per tensor = 512 chunks of 16 bytes, four per thread
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int chunk = c * 128 + threadIdx.x, token = chunk >> 5, offset = (chunk & 31) * 8;
      const uint32_t bytes = tile + token < end ? 16u : 0u;
      copy_async16(&tiles[buffer][0][token][offset], cacheK + base + token * kDim + offset, bytes);
      copy_async16(&tiles[buffer][1][token][offset], cacheV + base + token * kDim + offset, bytes);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(begin, 0);
  // Scores on the tensor cores too (warp 0): A = the K tile (16 tokens x 256 dims, 16 dims per MMA), B = q of the four
  // heads as 8 columns, columns 0..3 the fp16 high halves, columns 4..7 the low halves (q - hi). Lane (g, t) keeps column
  // g of B for all 16 dim steps: 32 registers.
  const int g = lane >> 2, t = lane & 3, myHead = g & 3;
  uint32_t qFragment[16][2];
  if (warp == 0) {
    const float* src = q + (size_t(row) * kQHeads + kvHead * kGroup + myHead) * kDim;
#pragma unroll
    for (int step = 0; step < 16; ++step) {
      const float2 a = *reinterpret_cast<const float2*>(src + 16 * step + 2 * t), b = *reinterpret_cast<const float2*>(src + 16 * step + 2 * t + 8);
      __half2 h0 = __floats2half2_rn(a.x, a.y), h1 = __floats2half2_rn(b.x, b.y);
      if (g >= 4) {
        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
        h0 = __floats2half2_rn(a.x - f0.x, a.y - f0.y), h1 = __floats2half2_rn(b.x - f1.x, b.y - f1.y);
      }
      qFragment[step][0] = *reinterpret_cast<const uint32_t*>(&h0), qFragment[step][1] = *reinterpret_cast<const uint32_t*>(&h1);
    }
  }
  // Value accumulation on the tensor cores (m16n8k16, fp16 operands, fp32 accumulate): warp w owns value dims 64w .. 64w+63
  // in four 16-dim chunks; A = V^T of the tile (dims x tokens, read transposed by ldmatrix), B = the tile's softmax weights
  // (tokens x 8 columns: columns 0..3 the fp16 high halves for the four heads, columns 4..7 the low halves, so the result is
  // accurate to fp32 rounding of the weights). Lane (g, t) builds column g of B, i.e. head g % 4, and tracks that head's
  // running maximum and, over its four tokens of every tile, its share of the norm.
  float runningMax = -1.0e30f, runningNorm = 0.f, acc[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
    acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
  int buffer = 0;
  for (uint32_t tile = begin; tile < end; tile += kTile, buffer ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // this tile is complete for every thread, and every thread is done with the previous tile and its scores
    if (tile + kTile < end)
      fetch(tile + kTile, buffer ^ 1);  // lands while this tile is worked on
    if (warp == 0) {
      // scores of the tile's 16 tokens for the four heads: two accumulator chains over the 16 dim steps
      float score[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      const int matrix = lane >> 3, tokenRow = (lane & 7) + 8 * (matrix & 1), dimOffset = 8 * (matrix >> 1);
#pragma unroll
      for (int step = 0; step < 16; ++step) {
        uint32_t a[4];
        const uint32_t address = smem_u32(&tiles[buffer][0][tokenRow][16 * step + dimOffset]);
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(address));
        mma_16816(score[step & 1], a, qFragment[step][0], qFragment[step][1]);
      }
      // columns 4..7 (lanes t = 2, 3) carry the low-half products of heads 0..3
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        score[0][i] += score[1][i];
        score[0][i] += __shfl_xor_sync(0xffffffffu, score[0][i], 2);
      }
      if (t < 2) {
        scores[2 * t][g] = tile + g < end ? score[0][0] * (1.0f / 16.0f) : -INFINITY;
        scores[2 * t + 1][g] = tile + g < end ? score[0][1] * (1.0f / 16.0f) : -INFINITY;
        scores[2 * t][g + 8] = tile + g + 8 < end ? score[0][2] * (1.0f / 16.0f) : -INFINITY;
        scores[2 * t + 1][g + 8] = tile + g + 8 < end ? score[0][3] * (1.0f / 16.0f) : -INFINITY;
      }
    }
    __syncthreads();
    // online softmax. A token past the end has score -inf: weight 0 against a zero-filled value row.
    float tileMax = -INFINITY;
#pragma unroll
    for (int i = 0; i < kTile; i += 4) {
      const float4 four = *reinterpret_cast<const float4*>(&scores[myHead][i]);
      tileMax = fmaxf(fmaxf(tileMax, fmaxf(four.x, four.y)), fmaxf(four.z, four.w));
    }
    const float nextMax = fmaxf(runningMax, tileMax), rescale = expf(runningMax - nextMax);
    runningMax = nextMax;
    // weights of this lane's four tokens (the summation slots 2t, 2t+1, 2t+8, 2t+9 of the B fragment)
    const float w0 = expf(scores[myHead][2 * t] - nextMax), w1 = expf(scores[myHead][2 * t + 1] - nextMax);
    const float w2 = expf(scores[myHead][2 * t + 8] - nextMax), w3 = expf(scores[myHead][2 * t + 9] - nextMax);
    runningNorm = runningNorm * rescale + ((w0 + w1) + (w2 + w3));
    __half2 b0 = __floats2half2_rn(w0, w1), b1 = __floats2half2_rn(w2, w3);
    if (g >= 4) {  // the low halves
      const float2 f0 = __half22float2(b0), f1 = __half22float2(b1);
      b0 = __floats2half2_rn(w0 - f0.x, w1 - f0.y), b1 = __floats2half2_rn(w2 - f1.x, w3 - f1.y);
    }
    // this lane's accumulators are columns 2t and 2t+1: heads (2t) % 4 and (2t+1) % 4
    const float r0 = __shfl_sync(0xffffffffu, rescale, ((2 * t) & 3) * 4), r1 = __shfl_sync(0xffffffffu, rescale, ((2 * t + 1) & 3) * 4);
    const int matrix = lane >> 3, tokenRow = (lane & 7) + 8 * (matrix >> 1), dimOffset = 8 * (matrix & 1);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t a[4];
      const uint32_t address = smem_u32(&tiles[buffer][1][tokenRow][64 * warp + 16 * c + dimOffset]);
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(address));
      acc[c][0] *= r0, acc[c][1] *= r1, acc[c][2] *= r0, acc[c][3] *= r1;
      mma_16816(acc[c], a, *reinterpret_cast<const uint32_t*>(&b0), *reinterpret_cast<const uint32_t*>(&b1));
    }
  }
  // columns 4..7 (lanes t = 2, 3) hold the low-half products of heads 0..3: add them to columns 0..3 (lanes t = 0, 1)
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      acc[c][i] += __shfl_xor_sync(0xffffffffu, acc[c][i], 2);
  runningNorm += __shfl_xor_sync(0xffffffffu, runningNorm, 1);
  runningNorm += __shfl_xor_sync(0xffffffffu, runningNorm, 2);
  float* base = partials + ((size_t(row) * kQHeads + kvHead * kGroup) * maxSplits + split) * kPartialStride;
  const size_t headStride = size_t(maxSplits) * kPartialStride;
  if (t < 2) {
    float *first = base + (2 * t) * headStride, *second = base + (2 * t + 1) * headStride;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int dim = 64 * warp + 16 * c + g;
      first[dim] = acc[c][0], second[dim] = acc[c][1];
      first[dim + 8] = acc[c][2], second[dim + 8] = acc[c][3];
    }
  }
  if (warp == 0 && g < 4 && t == 0) {
    base[g * headStride + kDim] = runningMax;
    base[g * headStride + kDim + 1] = runningNorm;
  }
}

// ---- rows of one query together: prompt chunks and speculative rows --------------------------------------------------
// The scan above reads K and V once per row: 128 prompt rows behind 2000 tokens pull 1 GB through the L2 (170 us, and
// 18 us to merge 32 splits of every row). Here up to 32 consecutive rows of a query share every K/V tile: the 32 rows x 4 query
// heads of one kv head are the 128 rows of two tcgen05 contractions. A CTA takes its piece of the context in rounds of up to four
// tiles of 64 tokens:
//   * loader warps copy the tiles of K, then those of V, with cp.async into a ring of three 32 KB slots, as 16-byte chunks
//     [8 dims][token], which is the no-swizzle layout of K as a K-major operand and of V as an MN-major one at once;
//   * scores of the round: q hi and q lo (fp16, 128 KB of shared memory, laid out once per item) x K into 64 columns of tensor
//     memory a tile;
//   * worker warps (a thread has one row, and every second tile) take maximum and weights of the whole round, so there is no
//     rescaling between tiles, and write the weights as fp16 hi and lo over the scores. Their loops are kept short: most of this code
//     runs once or a few times in a launch, with thirteen warps at work on different parts of it at once, so instruction fetch counts;
//   * values: the weights in tensor memory x V into 256 columns. Between rounds the workers rescale them.
// Operands as in the scan: fp16 keys and values, query and softmax weights as fp16 hi + lo, fp32 accumulation. A tile of 64 tokens is
// 1.6 k cycles of MMAs for the scores (bounded by shared memory: A and B both come from there) and 1 k for the values; mma.sync,
// with 16 rows x 4 heads, was 8 k for half the rows.
// Measured, with the merge, and before, with mma.sync: 128 rows behind 1920 tokens 51.0 -> 32.0 us, four times 30 rows behind up to 1970 49.3 -> 33.5 (33.8
// with every tile masked), 2048 rows behind 2048 1070 -> 443 (455 with every tile masked); by its own clocks the first of these spent, with weights by
// ex2.approx, 5000 of 38000 on its start, 6500 on q, 10000 on scores, which wait for their copies, 4300 on weights, 4000 on the last values and 5300 on the
// store of its results; 64 rows of 64 tokens 13.0 -> 16.1: a fixed start of laying out q and an end of
// reading tensor memory, which little work has to pay for, so short contexts stay with attention_group_kernel below.
// Left out: weights as ex2.approx.ftz of a product rounded once, 31.3, 32.7 and 419 us, but weights between 1/4 and 1/2 then are off by 8.1e-8 rms and
// -3.7e-8 on average instead of 7.3e-8 and 1.1e-8.
// Errors against fp64 (rms, of the result's): 128 rows behind 1920 tokens 1.4e-6 and 1.9e-6 before, 300 behind 8700 7.6e-6 and 2.1e-5,
// 32 behind 29968 2.9e-6 and 4.6e-6: fewer roundings between tiles.
//
// Work items (tile of rows, piece of context, kv head) are dealt to one CTA per SM; which exist only the device knows, so
// a CTA finds its next item by a scan over the queries. The pieces of a tile follow from its context and from `most`, which
// the host sets so that the items of the pass fill the SMs about once; a tile of few rows (speculative rows that share a pass
// with a prompt) is cut as finely as the caller's scratch allows. Queries of one row are no items: the arithmetic of a whole tile
// for one row made them the longest part of a pass (seven decode rows of 4000 tokens beside a prompt of 121 rows 97 us, 47 with
// the scan beside this kernel, 63 with all rows in the scan; seven of 32000 tokens 518, 194 and 198).
constexpr int kGroupRows = 32, kGroupTokens = 64, kRoundTiles = 4;
constexpr int kWorkers = 8, kMmaWarp = kWorkers, kLoaders = 4, kTileThreads = (kWorkers + 1 + kLoaders) * kWarp;  // warps
constexpr int kSlots = 3, kSlotBytes = kGroupTokens * kDim * 2;
constexpr int kQueryGroup = kGroup * kGroupRows * 16 + 16, kQueryBytes = kDim / 8 * kQueryGroup;  // 16 bytes more, so that the lanes of a row of q write to different banks
constexpr int kStagePitch = 36;  // floats of a row of 32 staged results

struct TileShared {
  uint64_t full[kSlots], slotFree[kSlots], queryReady, scoresReady[kRoundTiles], weightsReady[kRoundTiles], valuesReady, valuesFree, drained;
  uint32_t tmemBase;
  int abort;
  int broken[2];  // by item parity: a value was not finite of a token that some rows do not attend to
  float exchange[2][kGroup * kGroupRows];
};
constexpr int kTileControlBytes = 2048;
static_assert(sizeof(TileShared) <= kTileControlBytes, "control block too large");
constexpr size_t kTileSharedBytes = kTileControlBytes + 2 * kQueryBytes + kSlots * kSlotBytes;
static_assert(kTileSharedBytes <= 227 * 1024 && kWorkers * 32 * kStagePitch * 4 <= 2 * kQueryBytes, "shared memory");
constexpr uint32_t kColScores = 0, kColValues = 256;  // tensor memory: four tiles of 64 score columns, 256 value columns

struct RowTile {
  uint32_t start, rows, first, attended, slot;  // first: position of its first row; attended: context of its last row
};

template <uint32_t ROWS> __device__ __forceinline__ uint32_t tiles_of(const infdev_query& query) { return query.count > 1 ? (query.count + ROWS - 1) / ROWS : 0u; }

template <uint32_t ROWS> __device__ __forceinline__ RowTile tile_of(const infdev_query& query, uint32_t index) {
  RowTile tile;
  tile.start = query.start + index * ROWS;
  tile.rows = min(ROWS, query.count - index * ROWS);
  tile.first = query.position + index * ROWS;
  tile.attended = tile.first + tile.rows;
  tile.slot = query.slot;
  return tile;
}

// Pieces of a tile's context: whole 64-token tiles.
__device__ __forceinline__ uint32_t piece_tokens(uint32_t attended, uint32_t rows, uint32_t most, uint32_t maxSplits) {
  const uint32_t wanted = max(1u, min((attended + kGroupTokens - 1) / kGroupTokens, rows <= 4 ? maxSplits : most));
  return ((attended + wanted - 1) / wanted + kGroupTokens - 1) / kGroupTokens * kGroupTokens;
}
__device__ __forceinline__ uint32_t piece_count(uint32_t attended, uint32_t piece) { return (attended + piece - 1) / piece; }

// Work item `item` of the pass, found by one warp together; false when there are fewer. `items`: how many there are, where one
// round tells. A lane has one tile of rows at a time, whichever query it is of: with a lane per query, which counted its tiles one
// after the other, this took 2.2 us of the 128 rows of one prompt, most of it the divisions of four tiles in a row.
template <uint32_t ROWS>
__device__ __forceinline__ bool find_item(const infdev_query* queries, int queryCount, uint32_t most, uint32_t maxSplits, uint32_t item, RowTile& tile,
                                          uint32_t& split, uint32_t& piece, uint32_t& items) {
  const uint32_t lane = threadIdx.x & 31;
  auto running_sum = [&](uint32_t value) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t other = __shfl_up_sync(0xffffffffu, value, o);
      if (int(lane) >= o)
        value += other;
    }
    return value;
  };
  items = 0xffffffffu;
  for (int base = 0; base < queryCount; base += 32) {
    infdev_query query = {};
    if (base + int(lane) < queryCount)
      query = queries[base + lane];
    const uint32_t own = tiles_of<ROWS>(query);
    const bool single = !__any_sync(0xffffffffu, own > 1);  // a lane's tile is its query's then, and there is nothing to look for
    const uint32_t tilesUpTo = single ? 0u : running_sum(own), tiles = single ? 32u : __shfl_sync(0xffffffffu, tilesUpTo, 31);
    for (uint32_t first = 0; first < tiles; first += 32) {
      infdev_query whose = query;
      uint32_t index = 0;
      bool live = own > 0;
      if (!single) {  // the query of this lane's tile: how many queries end at or before it
        const uint32_t mine = first + lane;
        uint32_t owner = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
          if (__shfl_sync(0xffffffffu, tilesUpTo, owner + step - 1) <= mine)
            owner += step;
        }
        whose.start = __shfl_sync(0xffffffffu, query.start, owner), whose.count = __shfl_sync(0xffffffffu, query.count, owner);
        whose.position = __shfl_sync(0xffffffffu, query.position, owner), whose.slot = __shfl_sync(0xffffffffu, query.slot, owner);
        index = mine - __shfl_sync(0xffffffffu, tilesUpTo - own, owner);
        live = mine < tiles;
      }
      RowTile each = {};
      uint32_t tokens = 0, count = 0;
      if (live) {
        each = tile_of<ROWS>(whose, index);
        tokens = piece_tokens(each.attended, each.rows, most, maxSplits), count = piece_count(each.attended, tokens);
      }
      const uint32_t inclusive = running_sum(count), total = __shfl_sync(0xffffffffu, inclusive, 31);
      if (queryCount <= 32 && tiles <= 32)
        items = total;
      if (item >= total) {
        item -= total;
        continue;
      }
      const int holder = __ffs(__ballot_sync(0xffffffffu, inclusive > item)) - 1;
      tile = {__shfl_sync(0xffffffffu, each.start, holder), __shfl_sync(0xffffffffu, each.rows, holder), __shfl_sync(0xffffffffu, each.first, holder),
              __shfl_sync(0xffffffffu, each.attended, holder), __shfl_sync(0xffffffffu, each.slot, holder)};
      split = item - __shfl_sync(0xffffffffu, inclusive - count, holder), piece = __shfl_sync(0xffffffffu, tokens, holder);
      return true;
    }
  }
  return false;
}

// {a, b} as fp16 hi and lo pairs
__device__ __forceinline__ uint2 split_pair(float a, float b) {
  const uint32_t hi = pack_half2(a, b);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  return make_uint2(hi, pack_half2(a - f.x, b - f.y));
}

// 0x8000 in each half of `pair` that is an infinity or a NaN.
__device__ __forceinline__ uint32_t not_finite(uint32_t pair) { return ((pair & 0x7c007c00u) + 0x04000400u) & 0x80008000u; }

__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Scores of tokens first .. first + 15 of a tile that a row with `live` of its tokens does not attend to.
__device__ __forceinline__ void mask_scores(uint32_t (&score)[16], uint32_t first, uint32_t live) {
#pragma unroll
  for (int i = 0; i < 16; ++i)
    score[i] = first + i < live ? score[i] : __float_as_uint(-INFINITY);
}

__global__ void __launch_bounds__(kTileThreads, 1)
    attention_tile_kernel(const float* q, const __half* cacheK, const __half* cacheV, const infdev_query* queries, int queryCount, const int32_t* table,
                          int tableStride, int blockTokens, uint32_t most, uint32_t maxSplits, float* partials, int* status) {
  pdl_wait();  // first: the scan of the queries of one row starts beside this kernel and relies on it
  pdl_launch_dependents();
  extern __shared__ __align__(128) uint8_t tileRaw[];
  TileShared& sh = *reinterpret_cast<TileShared*>(tileRaw);
  uint8_t* const query = tileRaw + kTileControlBytes;  // [hi, lo][8 dims][row] of 16 bytes, row = 32 * head + r, 8 dims kQueryGroup apart
  uint8_t* const ring = query + 2 * kQueryBytes;       // [slot][8 dims][token] of 16 bytes
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  volatile int* abortFlag = &sh.abort;
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&sh.full[s], kLoaders * kWarp);
      mbar_init(&sh.slotFree[s], 1);
    }
    mbar_init(&sh.queryReady, kWorkers);
    for (int j = 0; j < kRoundTiles; ++j) {
      mbar_init(&sh.scoresReady[j], 1);
      mbar_init(&sh.weightsReady[j], kWorkers);
    }
    mbar_init(&sh.valuesReady, 1);
    mbar_init(&sh.valuesFree, kWorkers);
    mbar_init(&sh.drained, 1);
    sh.abort = sh.broken[0] = sh.broken[1] = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp)
    tmem_alloc(&sh.tmemBase, 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sh.tmemBase;
  bool ok = true;
  RowTile tile;
  uint32_t split, piece, items = 0xffffffffu, itemCount = 0, roundCount = 0;
  auto next_item = [&](uint32_t item) {
    return item / kKvHeads < items && find_item<kGroupRows>(queries, queryCount, most, maxSplits, item / kKvHeads, tile, split, piece, items);
  };
  auto tiles_in_round = [](uint32_t from, uint32_t end) { return min(uint32_t(kRoundTiles), (end - from + kGroupTokens - 1) / kGroupTokens); };
  constexpr uint32_t kRoundTokens = kRoundTiles * kGroupTokens;

  if (warp > kMmaWarp) {
    // ---------------- loaders: the K tiles of a round, then its V tiles ----------------
    const int loader = warp - kMmaWarp - 1;
    uint32_t count = 0;    // tiles asked for
    bool pending = false;  // the last of them has not been handed over yet
    uint32_t pendingMasked = 0, pendingPast = 0, pendingParity = 0;  // V: its tokens [masked, past) are masked for some rows
    const uint32_t blockShift = blockTokens & (blockTokens - 1) ? 32u : uint32_t(__ffs(blockTokens) - 1);  // 32: not a power of two
    const uint32_t chunkOffset = (4 * loader + (lane >> 3)) * (kGroupTokens * 16) + (lane & 7) * 16;
    auto hand_over = [&] {  // this thread's part of the pending tile has landed
      uint8_t* slot = ring + (count - 1) % kSlots * kSlotBytes + chunkOffset;
      if (pendingMasked < pendingPast) {
        // A value that is not finite, of a token that some rows of the tile do not attend to, times their weights of zero would
        // reach them: it stands as zero, and the rows that do attend to it get NaN at the end.
        bool bad = false;
        for (int c = 0; c < 16; ++c) {
          const uint32_t token = (c & 7) * 8 + (lane & 7);
          if (token < pendingMasked || token >= pendingPast)
            continue;
          uint4* at = reinterpret_cast<uint4*>(slot + (c >> 3) * (16 * kGroupTokens * 16) + (c & 7) * 128);
          const uint4 v = *at;
          uint32_t words[4] = {v.x, v.y, v.z, v.w}, found = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t mask = not_finite(words[i]);
            found |= mask;
            words[i] &= ~((mask >> 15) * 0xffffu);
          }
          if (found)
            *at = make_uint4(words[0], words[1], words[2], words[3]), bad = true;
        }
        if (bad)
          *reinterpret_cast<volatile int*>(&sh.broken[pendingParity]) = 1;
      }
      fence_async_proxy();
      mbar_arrive(&sh.full[(count - 1) % kSlots]);
      pending = false;
    };
    for (uint32_t item = blockIdx.x; ok && next_item(item); item += gridDim.x, ++itemCount) {
      const uint32_t kvHead = item % kKvHeads, begin = split * piece, end = min(tile.attended, begin + piece);
      const int32_t* slotTable = table + size_t(tile.slot) * tableStride;
      for (uint32_t from = begin; ok && from < end; from += kRoundTokens) {
        const uint32_t tiles = tiles_in_round(from, end);
        for (uint32_t j = 0; ok && j < 2 * tiles; ++j) {
          const bool values = j >= tiles;
          const uint32_t first = from + (values ? j - tiles : j) * kGroupTokens, slot = count % kSlots;
          if (count >= uint32_t(kSlots)) {
            const uint32_t parity = (count / kSlots - 1) & 1;
            if (pending && !__all_sync(0xffffffffu, mbar_test_wait(&sh.slotFree[slot], parity))) {  // not while what may free it is held back
              asm volatile("cp.async.wait_group 0;" ::: "memory");
              hand_over();
            }
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&sh.slotFree[slot], parity, abortFlag));
            if (!ok)
              break;
          }
          const __half* cache = (values ? cacheV : cacheK) + (lane >> 3) * 8 + loader * 32;
          uint8_t* to = ring + slot * kSlotBytes + chunkOffset;
#pragma unroll 4
          for (int c = 0; c < 8; ++c) {  // eight tokens x four groups of eight dims, twice
            const uint32_t token = first + c * 8 + (lane & 7), at = min(token, end - 1);
            const uint32_t bytes = token < end ? 16u : 0u;  // zeros past the end
            const uint32_t block = blockShift < 32 ? at >> blockShift : at / blockTokens;
            const __half* source = cache + ((size_t(slotTable[block]) * kKvHeads + kvHead) * blockTokens + (at - block * blockTokens)) * kDim;
            copy_async16(to + c * 128, source, bytes);
            copy_async16(to + 16 * kGroupTokens * 16 + c * 128, source + 128, bytes);
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
          if (pending) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            hand_over();
          }
          ++count;
          pending = true;
          pendingMasked = values && tile.first + 1 > first ? tile.first + 1 - first : 0u;
          pendingPast = values ? min(uint32_t(kGroupTokens), end - first) : 0u;
          pendingParity = itemCount & 1;
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (pending)
      hand_over();
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issuer ----------------
    constexpr uint32_t kScores = (1u << 4) | (uint32_t(kGroupTokens >> 3) << 17) | (8u << 24);       // fp16 x fp16 -> fp32, M 128, N 64, both K-major
    constexpr uint32_t kValues = (1u << 4) | (1u << 16) | (uint32_t(kDim >> 3) << 17) | (8u << 24);  // N 256, B MN-major
    constexpr uint32_t kQueryStep = 2 * kQueryGroup, kTokenStep = 2 * kGroupTokens * 16;  // 16 dims of q and of K
    const uint32_t queryBase = smem_u32(query);
    uint32_t count = 0, weightPhases = 0;
    for (uint32_t item = blockIdx.x; ok && next_item(item); item += gridDim.x, ++itemCount) {
      const uint32_t begin = split * piece, end = min(tile.attended, begin + piece);
      for (uint32_t from = begin; ok && from < end; from += kRoundTokens, ++roundCount) {
        const uint32_t tiles = tiles_in_round(from, end);
        if (elect_one()) {
          if (from == begin)
            ok = mbar_wait_bounded(&sh.queryReady, itemCount & 1, abortFlag);
          else  // the round before has read its weights, whose columns the scores take now
            ok = mbar_wait_bounded(&sh.valuesReady, (roundCount - 1) & 1, abortFlag);
          for (uint32_t j = 0; ok && j < tiles; ++j) {
            const uint32_t n = count + j, slot = n % kSlots, base = smem_u32(ring + slot * kSlotBytes);
            ok = mbar_wait_bounded(&sh.full[slot], (n / kSlots) & 1, abortFlag);
            if (!ok)
              break;
            fence_after_sync();
#pragma unroll 2
            for (uint32_t step = 0; step < kDim / 16; ++step) {
              const uint64_t keys = smem_descriptor(base + step * kTokenStep, kTokenStep / 2, 128);
              umma_ss(tmem + kColScores + j * 64, smem_descriptor(queryBase + step * kQueryStep, kQueryStep / 2, 128), keys, kScores, step != 0);
              umma_ss(tmem + kColScores + j * 64, smem_descriptor(queryBase + kQueryBytes + step * kQueryStep, kQueryStep / 2, 128), keys, kScores, 1);
            }
            umma_commit(&sh.slotFree[slot]);
            umma_commit(&sh.scoresReady[j]);
          }
          if (ok && from == begin && itemCount > 0)  // the workers have read the values of the item before
            ok = mbar_wait_bounded(&sh.valuesFree, (itemCount - 1) & 1, abortFlag);
          for (uint32_t j = 0; ok && j < tiles; ++j) {
            const uint32_t n = count + tiles + j, slot = n % kSlots, base = smem_u32(ring + slot * kSlotBytes);
            ok = mbar_wait_bounded(&sh.full[slot], (n / kSlots) & 1, abortFlag) &&
                 mbar_wait_bounded(&sh.weightsReady[j], (weightPhases >> j) & 1, abortFlag);
            if (!ok)
              break;
            fence_after_sync();
#pragma unroll 2
            for (uint32_t step = 0; step < kGroupTokens / 16; ++step) {
              const uint64_t values = smem_descriptor(base + step * 256, 128, kGroupTokens * 16);
              umma_ts(tmem + kColValues, tmem + kColScores + j * 64 + step * 16, values, kValues, from != begin || j != 0 || step != 0);
              umma_ts(tmem + kColValues, tmem + kColScores + j * 64 + step * 16 + 8, values, kValues, 1);
            }
            umma_commit(&sh.slotFree[slot]);
          }
          if (ok)
            umma_commit(&sh.valuesReady);
        }
        ok = __all_sync(0xffffffffu, ok);
        count += 2 * tiles;
        weightPhases ^= (1u << tiles) - 1;
      }
    }
    if (elect_one()) {  // no product may be under way when the CTA ends, whoever gave up
      umma_commit(&sh.drained);
      mbar_wait_bounded(&sh.drained, 0, abortFlag);
    }
  } else {
    // ---------------- workers: rows of q, softmax, results ----------------
    const int quadrant = warp & 3, side = warp >> 2;  // head; the tiles side, side + 2 and value columns 128 side .. 128 side + 127
    const int row = quadrant * 32 + lane;
    const uint32_t laneBase = tmem + (uint32_t(quadrant * 32) << 16);
    uint32_t scorePhases = 0;
    // Nobody leaves a loop early: the named barriers have no time limit, so who gave up goes on without waiting for the others.
    auto wait = [&](uint64_t* bar, uint32_t parity) { ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(bar, parity, abortFlag)); };
    for (uint32_t item = blockIdx.x; next_item(item); item += gridDim.x, ++itemCount) {
      const uint32_t kvHead = item % kKvHeads, begin = split * piece, end = min(tile.attended, begin + piece);
      named_barrier(5, kWorkers * kWarp);  // the item before is done with the shared memory of q, which its results were staged in
      if (tid == 0)
        sh.broken[(itemCount + 1) & 1] = 0;  // of the item before; the next one of that parity has no V tile yet
      // A warp takes half of a head's 32 rows, eight at a time, a lane eight dims of each: whole rows of 1 KB. Rows past the tile's are zero.
#pragma unroll 1
      for (int r0 = (warp & 1) * 16; r0 < (warp & 1) * 16 + 16; r0 += 8) {
        const int head = warp >> 1;
        const float* from = q + ((size_t(tile.start) + r0) * kQHeads + kvHead * kGroup + head) * kDim + lane * 8;
        float4 value[8][2];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          value[r][0] = value[r][1] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r0 + r < int(tile.rows)) {
            const float4* src = reinterpret_cast<const float4*>(from + size_t(r) * kQHeads * kDim);
            value[r][0] = src[0], value[r][1] = src[1];
          }
        }
        uint8_t* const to = query + lane * kQueryGroup + (head * kGroupRows + r0) * 16;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float4 a = value[r][0], b = value[r][1];
          const uint2 s0 = split_pair(a.x, a.y), s1 = split_pair(a.z, a.w), s2 = split_pair(b.x, b.y), s3 = split_pair(b.z, b.w);
          *reinterpret_cast<uint4*>(to + r * 16) = make_uint4(s0.x, s1.x, s2.x, s3.x);
          *reinterpret_cast<uint4*>(to + r * 16 + kQueryBytes) = make_uint4(s0.y, s1.y, s2.y, s3.y);
        }
      }
      fence_async_proxy();
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&sh.queryReady);
      float maximum = -1.0e30f, norm = 0.f;
      const uint32_t limit = min(end, tile.first + lane + 1);  // this row's scores from here on are masked
      for (uint32_t from = begin; from < end; from += kRoundTokens, ++roundCount) {
        const uint32_t tiles = tiles_in_round(from, end);
        float best = -INFINITY;
        for (uint32_t j = side; j < tiles; j += 2) {
          wait(&sh.scoresReady[j], (scorePhases >> j) & 1);
          fence_after_sync();
          const uint32_t first = from + j * kGroupTokens, live = limit > first ? limit - first : 0u;
          const bool whole = __all_sync(0xffffffffu, live >= kGroupTokens);
#pragma unroll 1
          for (uint32_t c = 0; c < kGroupTokens; c += 16) {
            uint32_t score[16];
            tmem_load16(laneBase + kColScores + j * 64 + c, score);
            tmem_wait_load();
            if (!whole)
              mask_scores(score, c, live);
#pragma unroll
            for (int i = 0; i < 16; ++i)
              best = fmaxf(best, __uint_as_float(score[i]));
          }
        }
        best *= 1.0f / 16.0f;
        sh.exchange[side][row] = best;
        named_barrier(1 + quadrant, 64);
        const float next = fmaxf(maximum, fmaxf(best, sh.exchange[side ^ 1][row])), rescale = expf(maximum - next);
        maximum = next, norm *= rescale;
        if (from != begin) {  // the values so far are of the maximum so far
          wait(&sh.valuesReady, (roundCount - 1) & 1);
          fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < 8; ++c) {
            uint32_t v[16];
            tmem_load16(laneBase + kColValues + side * 128 + c * 16, v);
            tmem_wait_load();
#pragma unroll
            for (int i = 0; i < 16; ++i)
              v[i] = __float_as_uint(__uint_as_float(v[i]) * rescale);
            tmem_store16(laneBase + kColValues + side * 128 + c * 16, v);
          }
          tmem_wait_store();
        }
        for (uint32_t j = 0; j < tiles; ++j) {
          if (int(j & 1) == side) {
            const uint32_t first = from + j * kGroupTokens, live = limit > first ? limit - first : 0u;
            const bool whole = __all_sync(0xffffffffu, live >= kGroupTokens);
#pragma unroll 1
            for (uint32_t c = 0; c < kGroupTokens; c += 16) {  // the halves of 16 weights take the columns of their scores
              uint32_t score[16], halves[16];
              tmem_load16(laneBase + kColScores + j * 64 + c, score);
              tmem_wait_load();
              if (!whole)
                mask_scores(score, c, live);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float w0 = expf(__uint_as_float(score[2 * i]) * (1.0f / 16.0f) - maximum), w1 = expf(__uint_as_float(score[2 * i + 1]) * (1.0f / 16.0f) - maximum);
                norm += w0 + w1;
                const uint2 w = split_pair(w0, w1);
                halves[i] = w.x, halves[8 + i] = w.y;
              }
              tmem_store16(laneBase + kColScores + j * 64 + c, halves);
            }
            tmem_wait_store();
          }
          fence_before_sync();
          __syncwarp();
          if (lane == 0)
            mbar_arrive(&sh.weightsReady[j]);
        }
        scorePhases ^= (1u << tiles) - 1;
        named_barrier(1 + quadrant, 64);  // both sides have read the exchange
      }
      // the norm over both sides' tiles, then this piece's record of every live row
      sh.exchange[side][row] = norm;
      named_barrier(1 + quadrant, 64);
      norm = sh.exchange[0][row] + sh.exchange[1][row];
      wait(&sh.valuesReady, (roundCount - 1) & 1);
      fence_after_sync();
      const bool broken = *reinterpret_cast<volatile int*>(&sh.broken[itemCount & 1]) != 0;
      const size_t headPitch = size_t(maxSplits) * kPartialStride;
      float* const records = partials + ((size_t(tile.start) * kQHeads + kvHead * kGroup + quadrant) * maxSplits + split) * kPartialStride;
      float* const stage = reinterpret_cast<float*>(query) + warp * 32 * kStagePitch;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const int column = side * 128 + c * 32;
#pragma unroll 1
        for (int half = 0; half < 32; half += 16) {
          uint32_t v[16];
          tmem_load16(laneBase + kColValues + column + half, v);
          tmem_wait_load();
          if (broken) {
            const int32_t* slotTable = table + size_t(tile.slot) * tableStride;
            for (uint32_t token = max(begin, tile.first + 1); token < limit; ++token) {
              const __half* source =
                  cacheV + ((size_t(slotTable[token / blockTokens]) * kKvHeads + kvHead) * blockTokens + token % blockTokens) * kDim + column + half;
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (not_finite(uint32_t(__half_as_ushort(source[i]))) & 0x8000u)
                  v[i] = __float_as_uint(NAN);
            }
          }
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            *reinterpret_cast<uint4*>(stage + lane * kStagePitch + half + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        __syncwarp();
#pragma unroll 4
        for (int step = 0; step < 8; ++step) {  // four rows x 128 bytes a store
          const int r = step * 4 + (lane >> 3);
          if (r < int(tile.rows))
            *reinterpret_cast<float4*>(records + size_t(r) * kQHeads * headPitch + column + (lane & 7) * 4) =
                *reinterpret_cast<const float4*>(stage + r * kStagePitch + (lane & 7) * 4);
        }
        __syncwarp();
      }
      if (side == 0 && lane < int(tile.rows))
        *reinterpret_cast<float2*>(records + size_t(lane) * kQHeads * headPitch + kDim) = make_float2(maximum, norm);
      fence_before_sync();
      named_barrier(1 + quadrant, 64);  // both sides have read the exchange
      if (lane == 0)
        mbar_arrive(&sh.valuesFree);
    }
  }
  if (!ok && lane == 0) {
    *abortFlag = 1;
    atomicExch(status, kStatusBarrierTimeout);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp)
    tmem_dealloc(tmem, 512);
}

// The same for passes of short contexts, with mma.sync: 16 rows a tile and a warp, two warps a scheduler. K and V tiles come through
// a cp.async double buffer; warp = (head, half), a half takes 32 of a tile's 64 tokens for the scores and 128 of the 256 value
// dims, and the halves exchange maxima, weights and norms. Each tile of tokens is a chain of all of that, 8 k cycles of MMAs in it, which
// long contexts cannot afford, but there is next to nothing before the first one: 64 rows of 64 tokens 13.0 us with the merge (13.7 before
// items were found a lane per tile), 16.1 with attention_tile_kernel, and row by row 17.8; attention_launch has the line between the two.
constexpr int kShortRows = 16, kGroupThreads = 256, kGroupPitch = kDim + 8, kWeightPitch = kGroupTokens + 8;

struct GroupShared {
  __half q[2][kGroup * kShortRows][kGroupPitch];                         // hi, lo; row 16 * head + r
  __half k[2][kGroupTokens][kGroupPitch], v[2][kGroupTokens][kGroupPitch];  // two buffers
  __half p[2][kGroup * kShortRows][kWeightPitch];                        // hi, lo
  float exchange[2][kGroup * kShortRows];
};

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __half* address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(address)));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], const __half* address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(address)));
}
__global__ void __launch_bounds__(kGroupThreads, 1)
    attention_group_kernel(const float* q, const __half* cacheK, const __half* cacheV, const infdev_query* queries, int queryCount, const int32_t* table,
                           int tableStride, int blockTokens, uint32_t most, uint32_t maxSplits, float* partials) {
  pdl_wait();  // first: the scan of the queries of one row starts beside this kernel and relies on it
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t groupRaw[];
  GroupShared& sh = *reinterpret_cast<GroupShared*>(groupRaw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = warp & 3, half = warp >> 2, g = lane >> 2, t = lane & 3;
  const int rowBase = head * kShortRows;  // this warp's 16 rows of q, p and exchange
  RowTile tile;
  uint32_t split, piece, items = 0xffffffffu;
  for (uint32_t item = blockIdx.x;
       item / kKvHeads < items && find_item<kShortRows>(queries, queryCount, most, maxSplits, item / kKvHeads, tile, split, piece, items); item += gridDim.x) {
    const uint32_t kvHead = item % kKvHeads, begin = split * piece, end = min(tile.attended, begin + piece);
    const int32_t* slotTable = table + size_t(tile.slot) * tableStride;
    auto fetch = [&](uint32_t from, int buffer) {  // a warp copies one token's 512 bytes at a time
#pragma unroll
      for (int c = 0; c < kGroupTokens / 8; ++c) {
        const uint32_t token = c * 8 + warp, at = min(from + token, end - 1);
        const uint32_t bytes = from + token < end ? 16u : 0u;  // zeros past the end
        const size_t base = ((size_t(slotTable[at / blockTokens]) * kKvHeads + kvHead) * blockTokens + at % blockTokens) * kDim + lane * 8;
        copy_async16(&sh.k[buffer][token][lane * 8], cacheK + base, bytes);
        copy_async16(&sh.v[buffer][token][lane * 8], cacheV + base, bytes);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncthreads();  // the item before this one is finished with the shared arrays
    // the 16 rows x 4 heads of q, hi and lo; rows past the tile's are zero. All loads are in flight before the first is used.
    constexpr int kQuads = kGroup * kShortRows * (kDim / 4) / kGroupThreads;
    float4 value[kQuads];
#pragma unroll
    for (int i = 0; i < kQuads; ++i) {
      const int at = i * kGroupThreads + threadIdx.x, row = at / (kDim / 4), d = at % (kDim / 4) * 4, r = row % kShortRows, h = row / kShortRows;
      value[i] = r < int(tile.rows) ? *reinterpret_cast<const float4*>(q + (size_t(tile.start + r) * kQHeads + kvHead * kGroup + h) * kDim + d)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    fetch(begin, 0);
#pragma unroll
    for (int i = 0; i < kQuads; ++i) {
      const int at = i * kGroupThreads + threadIdx.x, row = at / (kDim / 4), d = at % (kDim / 4) * 4;
      const uint2 a = split_pair(value[i].x, value[i].y), b = split_pair(value[i].z, value[i].w);
      *reinterpret_cast<uint2*>(&sh.q[0][row][d]) = make_uint2(a.x, b.x);
      *reinterpret_cast<uint2*>(&sh.q[1][row][d]) = make_uint2(a.y, b.y);
    }
    float maximum[2] = {-1.0e30f, -1.0e30f}, norm[2] = {0.f, 0.f}, acc[16][4];  // rows g and g + 8
#pragma unroll
    for (int j = 0; j < 16; ++j)
      acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    int buffer = 0;
    for (uint32_t from = begin; from < end; from += kGroupTokens, buffer ^= 1) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // the tile has landed, and everybody is done with the one before
      if (from + kGroupTokens < end)
        fetch(from + kGroupTokens, buffer ^ 1);
      float score[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        score[j][0] = score[j][1] = score[j][2] = score[j][3] = 0.f;
#pragma unroll
      for (int step = 0; step < kDim / 16; ++step) {
        uint32_t hi[4], lo[4];
        ldmatrix4(hi, &sh.q[0][rowBase + (lane & 15)][16 * step + 8 * (lane >> 4)]);
        ldmatrix4(lo, &sh.q[1][rowBase + (lane & 15)][16 * step + 8 * (lane >> 4)]);
#pragma unroll
        for (int pair = 0; pair < 2; ++pair) {
          if (from + 32 * half + 16 * pair >= end)  // past the piece: these scores are masked below
            continue;
          uint32_t b[4];
          ldmatrix4(b, &sh.k[buffer][32 * half + 16 * pair + 8 * (lane >> 4) + (lane & 7)][16 * step + 8 * ((lane >> 3) & 1)]);
          mma_16816(score[2 * pair], hi, b[0], b[1]);
          mma_16816(score[2 * pair + 1], hi, b[2], b[3]);
          mma_16816(score[2 * pair], lo, b[0], b[1]);
          mma_16816(score[2 * pair + 1], lo, b[2], b[3]);
        }
      }
      // scale, causal mask, row maxima over both halves of the tile
      float best[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t token = from + 32 * half + 8 * j + 2 * t + (i & 1), limit = min(end, tile.first + g + 8 * (i >> 1) + 1);
          score[j][i] = token < limit ? score[j][i] * (1.0f / 16.0f) : -INFINITY;
          best[i >> 1] = fmaxf(best[i >> 1], score[j][i]);
        }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        best[r] = fmaxf(best[r], __shfl_xor_sync(0xffffffffu, best[r], 1));
        best[r] = fmaxf(best[r], __shfl_xor_sync(0xffffffffu, best[r], 2));
        if (t == 0)
          sh.exchange[half][rowBase + g + 8 * r] = best[r];
      }
      named_barrier(1 + head, 64);
      float rescale[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float next = fmaxf(maximum[r], fmaxf(best[r], sh.exchange[half ^ 1][rowBase + g + 8 * r]));
        rescale[r] = expf(maximum[r] - next);
        maximum[r] = next;
        norm[r] *= rescale[r];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float w0 = expf(score[j][2 * r] - maximum[r]), w1 = expf(score[j][2 * r + 1] - maximum[r]);
          norm[r] += w0 + w1;
          const uint2 w = split_pair(w0, w1);
          *reinterpret_cast<uint32_t*>(&sh.p[0][rowBase + g + 8 * r][32 * half + 8 * j + 2 * t]) = w.x;
          *reinterpret_cast<uint32_t*>(&sh.p[1][rowBase + g + 8 * r][32 * half + 8 * j + 2 * t]) = w.y;
        }
      // A value that is not finite, of a token that some rows of the tile do not attend to, times their weights of zero would
      // reach them: in such a tile it stands as zero, and the rows that do attend to it get NaN afterwards. (128 rows behind 1920
      // tokens 55.4 -> 56.3 us with the test; a test within the loop of products 58.)
      const uint32_t masked = max(from, tile.first + 1), past = min(from + kGroupTokens, end);
      uint32_t broken = 0;
      for (uint32_t token = masked; token < past; ++token) {
        const uint2 four = *reinterpret_cast<const uint2*>(&sh.v[buffer][token - from][128 * half + 4 * lane]);
        broken |= not_finite(four.x) | not_finite(four.y);
      }
      broken = __any_sync(0xffffffffu, broken != 0);
      named_barrier(1 + head, 64);  // both halves of the weights are there
#pragma unroll
      for (int j = 0; j < 16; ++j)
        acc[j][0] *= rescale[0], acc[j][1] *= rescale[0], acc[j][2] *= rescale[1], acc[j][3] *= rescale[1];
      auto add_values = [&](int step, bool clean) {
        uint32_t hi[4], lo[4];
        ldmatrix4(hi, &sh.p[0][rowBase + (lane & 15)][16 * step + 8 * (lane >> 4)]);
        ldmatrix4(lo, &sh.p[1][rowBase + (lane & 15)][16 * step + 8 * (lane >> 4)]);
#pragma unroll
        for (int pair = 0; pair < 8; ++pair) {
          uint32_t b[4];
          ldmatrix4_trans(b, &sh.v[buffer][16 * step + (lane & 15)][128 * half + 16 * pair + 8 * (lane >> 4)]);
          if (clean) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              b[i] &= ~((not_finite(b[i]) >> 15) * 0xffffu);
          }
          mma_16816(acc[2 * pair], hi, b[0], b[1]);
          mma_16816(acc[2 * pair + 1], hi, b[2], b[3]);
          mma_16816(acc[2 * pair], lo, b[0], b[1]);
          mma_16816(acc[2 * pair + 1], lo, b[2], b[3]);
        }
      };
      if (!broken) {
#pragma unroll
        for (int step = 0; step < kGroupTokens / 16; ++step) {
          if (from + 16 * step >= end)  // weights of zero
            break;
          add_values(step, false);
        }
      } else {
#pragma unroll 1
        for (int step = 0; step < kGroupTokens / 16; ++step)
          add_values(step, true);
#pragma unroll 1
        for (uint32_t token = from; token < past; ++token)
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const uint32_t bad = not_finite(*reinterpret_cast<const uint32_t*>(&sh.v[buffer][token - from][128 * half + 8 * j + 2 * t]));
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if ((bad & (i & 1 ? 0x80000000u : 0x8000u)) && token <= tile.first + g + 8 * (i >> 1))
                acc[j][i] = NAN;
          }
      }
    }
    // the norm over both halves, then this piece's record of every live row
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      norm[r] += __shfl_xor_sync(0xffffffffu, norm[r], 1);
      norm[r] += __shfl_xor_sync(0xffffffffu, norm[r], 2);
      if (t == 0)
        sh.exchange[half][rowBase + g + 8 * r] = norm[r];
    }
    named_barrier(1 + head, 64);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t row = g + 8 * r;
      if (row >= tile.rows)
        continue;
      float* record = partials + ((size_t(tile.start + row) * kQHeads + kvHead * kGroup + head) * maxSplits + split) * kPartialStride;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        *reinterpret_cast<float2*>(record + 128 * half + 8 * j + 2 * t) = make_float2(acc[j][2 * r], acc[j][2 * r + 1]);
      if (half == 0 && t == 0)
        *reinterpret_cast<float2*>(record + kDim) = make_float2(maximum[r], sh.exchange[0][rowBase + row] + sh.exchange[1][rowBase + row]);
    }
  }
}

// grid (rows * 16), 256 threads: merge the splits, normalise, multiply by sigmoid(gate).
// `image`, when not null, also receives the activation image of the output rows: a head is one 256-value block.
// ROWS: the splits of a row whose query has several are those of the kernel with tiles of so many rows; 0: of the scan.
template <uint32_t ROWS>
__global__ void __launch_bounds__(256) attention_reduce_kernel(const float* partials, const float* qg, const infdev_query* queries, int queryCount,
                                                               uint32_t most, uint32_t maxSplits, float* out, uint8_t* image) {
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t headRow = blockIdx.x, row = headRow / kQHeads, dim = threadIdx.x;
  const infdev_query& info = query_of_row(queries, queryCount, row);
  uint32_t count;
  if (ROWS > 0 && info.count > 1) {
    const RowTile tile = tile_of<ROWS>(info, (row - info.start) / max(ROWS, 1u));
    count = piece_count(tile.attended, piece_tokens(tile.attended, tile.rows, most, maxSplits));
  } else {
    uint32_t begin, end;
    split_range(info.position + (row - info.start) + 1, maxSplits, 0, begin, end, count);
  }
  const float* src = partials + size_t(headRow) * maxSplits * kPartialStride;
  // Lane s of every warp fetches the running maximum and norm of split s (at most 32 splits) in one trip to the L2; the
  // weights of the splits then travel by shuffle, and the loop below has only independent loads, taken in split order
  // so the sums are those of a sequential merge.
  const uint32_t lane = dim & 31;
  float splitMaximum = -1.0e30f, splitNorm = 0.f;
  if (lane < count) {
    const float2 pair = *reinterpret_cast<const float2*>(src + lane * kPartialStride + kDim);
    splitMaximum = pair.x, splitNorm = pair.y;
  }
  const float maximum = warp_max(splitMaximum);
  const float splitWeight = lane < count ? expf(splitMaximum - maximum) : 0.f;
  float norm = 0.f, numerator = 0.f;
#pragma unroll 8
  for (uint32_t s = 0; s < count; ++s) {
    const float w = __shfl_sync(0xffffffffu, splitWeight, int(s));
    norm += __shfl_sync(0xffffffffu, splitNorm, int(s)) * w;
    numerator += src[s * kPartialStride + dim] * w;
  }
  const float gate = qg[size_t(headRow) * kDim * 2 + kDim + dim];
  const float value = (numerator / norm) / (1.0f + expf(-gate));
  out[size_t(headRow) * kDim + dim] = value;
  if (image) {
    __shared__ __align__(16) float staged[kDim];
    staged[dim] = value;
    __syncthreads();
    if (dim < 32) {
      const float4 a = *reinterpret_cast<const float4*>(&staged[dim * 8]), b = *reinterpret_cast<const float4*>(&staged[dim * 8 + 4]);
      const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      image_store_block(image + (size_t(row >> 3) * kQHeads + headRow % kQHeads) * kImageBlockBytes, row & 7, dim, v);
    }
  }
}

}  // namespace

cudaError_t attention_prepare_launch(const float* qg, const float* rawK, const float* rawV, const float* qNorm, const float* kNorm, const float* rope,
                                     const infdev_query* queries, int queryCount, const int32_t* table, int tableStride, int blockTokens, int64_t rows, float* q,
                                     void* cacheK, void* cacheV, cudaStream_t stream) {
  if (rows <= 0)
    return cudaSuccess;
  uintptr_t addresses = reinterpret_cast<uintptr_t>(cacheK) | reinterpret_cast<uintptr_t>(cacheV);
  for (const float* p : {qg, rawK, rawV, qNorm, kNorm, rope, static_cast<const float*>(q)})
    addresses |= reinterpret_cast<uintptr_t>(p);
  auto launch = [&](auto kernel) {
    launch_kernel<2>(kernel, unsigned((rows * 20 + 7) / 8), 256, 0, stream, qg, rawK, rawV, qNorm, kNorm, rope, queries, queryCount, table, tableStride, blockTokens,
                     int(rows * 20), q, static_cast<__half*>(cacheK), static_cast<__half*>(cacheV));
  };
  launch(addresses & 15 ? attention_prepare_kernel<false> : attention_prepare_kernel<true>);
  return cudaGetLastError();
}

cudaError_t attention_launch(const float* q, const float* qg, const void* cacheK, const void* cacheV, const infdev_query* queries,
                             int queryCount, const int32_t* table, int tableStride, int blockTokens, int64_t rows, int64_t longest, uint32_t maxSplits,
                             float* partials, float* out, uint8_t* image, bool rowwise, int sms, int* status, cudaStream_t stream, int* launches) {
  *launches = 0;
  if (rows <= 0)
    return cudaSuccess;
  *launches = 2;
  const uint32_t splits = std::min<uint32_t>(maxSplits, 32);  // the merge keeps one split per lane
  // Tiles take passes whose queries have five rows or more on average, unless no context of the pass can be long (the table has no
  // room for it): with r rows a query, their longer chain costs 2 us where r x context is below about 4096 (8 rows of 128 tokens
  // 18.7 against 16.7 us for preparation and attention), from there on it is level or faster (8 rows of 2008 tokens 20.8 against
  // 29.1, 64 of 64 13.0 against 17.8 for the attention alone, 64 of 256 15.1 against 22.4, 128 of 128 15.8 against 29.0).
  const int64_t capacity = int64_t(tableStride) * blockTokens;
  const bool grouped = rows >= 32 * int64_t(queryCount) || (rows >= 5 * int64_t(queryCount) && rows * capacity >= 4096 * int64_t(queryCount));
  // The tile kernels copy q in pieces of 16 bytes, that of 32 rows the partial results too, the scan in pieces of 8 and less.
  if (grouped && !rowwise && reinterpret_cast<uintptr_t>(q) % 16 == 0) {
    // The tiles of 16 rows have the shorter chain, those of 32 the higher rate: the line is drawn by the work of the whole pass, its rows times
    // its longest context, which is what its caller says or else what a table row holds. us with tiles of 16 / 32, by queries x rows at
    // tokens: 1x64 at 64 13.0 / 16.5, 8x5 at 100 12.4 / 15.5, 1x128 at 256 17.4 / 20.6, 4x32 at 256 18.5 / 21.6, 1x128 at 512 22.3 / 22.6,
    // 4x32 at 512 23.3 / 23.5; at the line 1x128 at 768 26.7 / 25.4, 1x96 at 1024 26.7 / 22.6, 4x16 at 1536 26.2 / 25.5, 8x12 at 1024 33.6 / 33.1;
    // above 1x128 at 2048 49.1 / 32.2, 8x32 at 1024 56.5 / 43.0. One query of few rows gains later: 1x8 at 8192 28.1 / 30.9, at 12288 37.2 / 40.2, at
    // 16384 46.0 / 46.6, at 24000 63.7 / 61.4. Several queries of 17 to 31 rows on average gain earlier, because their tiles of 16 are reckoned
    // too few (below): 2x24 at 1536 32.9 / 22.6, 4x24 at 768 36.9 / 24.7.
    // They also take partial results that are on 8 bytes only.
    const int64_t context = longest > 0 ? std::min(longest, capacity) : capacity;
    const int64_t line = rows < 10 ? 131072 : queryCount > 1 && rows > 16 * int64_t(queryCount) && rows < 32 * int64_t(queryCount) ? 73728 : 98304;
    const bool shortPass = rows * context < line || reinterpret_cast<uintptr_t>(partials) % 16 != 0;
    const int tileRows = shortPass ? kShortRows : kGroupRows;
    static PerDeviceOnce configured, shortConfigured;
    if (const cudaError_t e = shortPass ? configure_shared_memory(attention_group_kernel, sizeof(GroupShared), shortConfigured)
                                        : configure_shared_memory(attention_tile_kernel, kTileSharedBytes, configured))
      return e;
    // How many rows each query has only the device knows. Queries of 33 to 63 rows on average are taken to have two tiles of 32 each: too few
    // reckoned with is a second turn of items for some CTAs (4x48 at 1024 tokens with six tiles 51.6 us, with eight 37).
    const int64_t perQuery = !shortPass && rows > 32 * int64_t(queryCount) && rows < 64 * int64_t(queryCount) ? 2 : 1;
    const int64_t tiles = std::max<int64_t>((rows + tileRows - 1) / tileRows, perQuery * queryCount);
    const uint32_t most = uint32_t(std::clamp<int64_t>(sms / (kKvHeads * tiles), 1, splits));
    const int64_t items = (rows + queryCount) * kKvHeads * splits;  // no more than these
    const unsigned grid = unsigned(std::min<int64_t>(items, sms));
    if (shortPass)
      launch_kernel<2>(attention_group_kernel, grid, kGroupThreads, sizeof(GroupShared), stream, q, static_cast<const __half*>(cacheK),
                       static_cast<const __half*>(cacheV), queries, queryCount, table, tableStride, blockTokens, most, splits, partials);
    else
      launch_kernel<2>(attention_tile_kernel, grid, kTileThreads, kTileSharedBytes, stream, q, static_cast<const __half*>(cacheK),
                       static_cast<const __half*>(cacheV), queries, queryCount, table, tableStride, blockTokens, most, splits, partials, status);
    // Queries of one row stay with the scan, which is faster there: no query rows to share a tile with, and six small CTAs per
    // SM hide the copies that the tile kernel's single CTA waits for. Which queries they are only the device knows; with a
    // single query there are none.
    if (queryCount > 1) {
      *launches = 3;
      // Its CTAs start on the SMs that the tile kernel leaves first: shared memory that nobody uses spreads the few of a pass with
      // few queries over all SMs (one row of 32000 tokens beside a prompt: six on an SM 124 us, one 89).
      constexpr size_t kSmShared = 228 * 1024, kScanShared = sizeof(float) * kGroup * kTile + sizeof(__half) * 2 * 2 * kTile * (kDim + 8) + 1024;
      static PerDeviceOnce scanConfigured;
      if (const cudaError_t e = configure_shared_memory(attention_scan_kernel<true>, kSmShared / 2 - kScanShared + 256, scanConfigured))
        return e;
      const size_t perSm = std::clamp<size_t>((splits * kKvHeads * size_t(queryCount - 1) + sms - 1) / sms, 1, 6);
      const size_t spread = perSm < 6 ? kSmShared / (perSm + 1) - kScanShared + 256 : 0;
      launch_kernel<2>(attention_scan_kernel<true>, dim3(splits + 1, kKvHeads, unsigned(queryCount)), 128, spread, stream, q, static_cast<const __half*>(cacheK),
                       static_cast<const __half*>(cacheV), queries, queryCount, table, tableStride, blockTokens, splits, partials);
    }
    launch_kernel<2>(shortPass ? attention_reduce_kernel<kShortRows> : attention_reduce_kernel<kGroupRows>, unsigned(rows * kQHeads), 256, 0, stream, partials, qg, queries, queryCount, most, splits, out, image);
    return cudaGetLastError();
  }
  launch_kernel(attention_scan_kernel<false>, dim3(splits, kKvHeads, unsigned(rows)), 128, 0, stream, q, static_cast<const __half*>(cacheK),
                                                                                       static_cast<const __half*>(cacheV), queries, queryCount, table,
                                                                                       tableStride, blockTokens, splits, partials);
  launch_kernel(attention_reduce_kernel<0>, unsigned(rows * kQHeads), 256, 0, stream, partials, qg, queries, queryCount, 0u, splits, out, image);
  return cudaGetLastError();
}

// ---- attention without any allocation -------------------------------------------------------------
// Some users of this library cannot give the attention call a scratch buffer: a serving process that sized its
// K/V pool to whatever device memory was free at start-up has nothing left for a later cudaMalloc, and a
// latency-critical decode loop cannot afford an allocation call that synchronises the whole device. For them the
// split-K partials of up to kStaticRows packed rows live in this file-scope array (about 2 MiB), which every GPU
// that loads the library keeps until the process exits.
constexpr int kStaticRows = 8, kStaticSplits = 16;
static __device__ __align__(256) float staticPartials[size_t(kStaticRows) * kQHeads * kStaticSplits * kPartialStride];

cudaError_t attention_static_launch(const float* q, const float* qg, const void* cacheK, const void* cacheV, const infdev_query* queries,
                                    int queryCount, const int32_t* table, int tableStride, int blockTokens, int64_t rows, int device, float* out,
                                    cudaStream_t stream) {
  // In host code `staticPartials` is only a handle; the kernels need the device address, looked up once per
  // device (with that device current, which the caller guarantees) and remembered.
  static std::mutex guard;
  static float* address[64] = {nullptr};
  if (device < 0 || device >= 64 || rows > kStaticRows)
    return cudaErrorInvalidValue;
  if (rows <= 0)
    return cudaSuccess;
  float* partials;
  {
    std::lock_guard<std::mutex> lock(guard);
    if (!address[device]) {
      void* found = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&found, staticPartials);
      if (e != cudaSuccess)
        return e;
      address[device] = static_cast<float*>(found);
    }
    partials = address[device];
  }
  // Nothing has to start at zero: the reduction reads exactly the (row, head, split) records that the scan of the
  // same call wrote; whatever an earlier call left in the array is never read.
  launch_kernel(attention_scan_kernel<false>, dim3(kStaticSplits, kKvHeads, unsigned(rows)), 128, 0, stream, q, static_cast<const __half*>(cacheK),
                                                                                          static_cast<const __half*>(cacheV), queries, queryCount, table,
                                                                                          tableStride, blockTokens, kStaticSplits, partials);
  launch_kernel(attention_reduce_kernel<0>, unsigned(rows * kQHeads), 256, 0, stream, partials, qg, queries, queryCount, 0u, uint32_t(kStaticSplits), out, nullptr);
  return cudaGetLastError();
}

int attention_static_max_rows() { return kStaticRows; }

}  // namespace infdev
