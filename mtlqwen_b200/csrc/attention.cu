// Gated GQA attention over the paged fp16 K/V pool.
//
// attention_prepare_kernel <- attention_prepare (attention.metal:14-50) + the cache append that the
//                             reference does inside attention_scan (:126-133)
// attention_scan_kernel    <- attention_scan   (attention.metal:103-183), row by row: queries of one row, and passes whose
//                             queries have few rows on average
// attention_group_kernel   <- the same, for the queries of several rows of the other passes
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

// grid (rows * 20), 256 threads: heads 0..15 are queries, 16..19 keys (which also store the value head).
__global__ void __launch_bounds__(256) attention_prepare_kernel(const float* qg, const float* rawK, const float* rawV, const float* qNorm,
                                                                const float* kNorm, const float* rope, const infdev_query* queries, int queryCount,
                                                                const int32_t* table, int tableStride, int blockTokens, float* q, __half* cacheK,
                                                                __half* cacheV) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x / 20, head = blockIdx.x % 20, lane = threadIdx.x;
  const bool query = head < kQHeads;
  if (query && !qg)  // K/V store only (mtp_store_kv, attention.metal:53-100)
    return;
  const int local = query ? head : head - kQHeads;
  const float* source = query ? qg + (size_t(row) * kQHeads + local) * kDim * 2 : rawK + (size_t(row) * kKvHeads + local) * kDim;
  const float* weight = query ? qNorm : kNorm;
  const float value = source[lane];
  __shared__ float partial[8], scale;
  const float sum = warp_sum(value * value);
  if ((lane & 31) == 0)
    partial[lane >> 5] = sum;
  __syncthreads();
  if (lane == 0) {
    float total = 0.f;
    for (int i = 0; i < 8; ++i)
      total += partial[i];
    scale = rsqrtf(total / float(kDim) + 1.0e-6f);
  }
  __syncthreads();
  const infdev_query& info = query_of_row(queries, queryCount, row);
  const uint32_t position = info.position + row - info.start;
  float result = value * scale * weight[lane];
  if (lane < 64) {
    const int other = lane < 32 ? lane + 32 : lane - 32, pair = lane & 31;
    const float paired = source[other] * scale * weight[other];
    const float2 cs = *reinterpret_cast<const float2*>(rope + (size_t(position) * 32 + pair) * 2);
    result = result * cs.x + (lane < 32 ? -paired : paired) * cs.y;
  }
  if (query) {
    q[(size_t(row) * kQHeads + local) * kDim + lane] = result;
  } else {
    const size_t block = table[size_t(info.slot) * tableStride + position / blockTokens];
    const size_t at = ((block * kKvHeads + local) * blockTokens + position % blockTokens) * kDim + lane;
    cacheK[at] = __float2half_rn(result);
    cacheV[at] = __float2half_rn(rawV[(size_t(row) * kKvHeads + local) * kDim + lane]);
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
// SINGLES: grid (maxSplits + 1, 4 kv heads, queries), for the queries of one row of a pass whose other queries the group kernel
// takes, beside that kernel: launched after it and early, it reads nothing that kernel writes and does not wait for it. The
// group kernel lets it start only after its own wait, so what the kernels before both wrote is there; the fence keeps this
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
// 18 us to merge 32 splits of every row). Here up to 16 consecutive rows of a query share every K/V tile: a CTA holds the
// 16 rows x 4 query heads of one kv head as 64 rows of the two contractions, and walks its piece of the context in tiles
// of 64 tokens, softmax online. 8 warps = 4 heads x 2 halves: a warp scores 32 tokens of the tile, hands its weights to
// its partner through shared memory and accumulates 128 of the 256 value dims for all 64. Operands as in the scan: fp16
// keys and values, query and softmax weights as fp16 hi + lo, fp32 accumulation.
// 128 rows behind 1920 tokens are 4.2 G multiply-adds with both halves of q and p, 14 us at the 1016 per clock and SM of
// mma.sync; the kernel takes about 38, because with two warps a scheduler the products, the fragment reads and the exchange
// between the halves wait for each other (tensor pipe 42 % of the active cycles, 0.29 issued per cycle and scheduler). In an
// earlier form sixteen warps instead of eight measured 66 instead of 61 us for the whole call, and two groups of four warps
// with tiles and softmax of their own, nothing exchanged, the same 61.
//
// Work items (tile of rows, piece of context, kv head) are dealt to one CTA per SM; which exist only the device knows, so
// a CTA finds its next item by a scan over the queries. The pieces of a tile follow from its context and from `most`, which
// the host sets so that the items of the pass fill the SMs about once; a tile of few rows (speculative rows that share a pass
// with a prompt) is cut as finely as the caller's scratch allows. Queries of one row are no items: the arithmetic of 16 rows
// for one made them the longest part of a pass (seven decode rows of 4000 tokens beside a prompt of 121 rows 97 us, 47 with
// the scan beside this kernel, 63 with all rows in the scan; seven of 32000 tokens 518, 194 and 198).
constexpr int kGroupRows = 16, kGroupTokens = 64, kGroupThreads = 256, kGroupPitch = kDim + 8, kWeightPitch = kGroupTokens + 8;

struct GroupShared {
  __half q[2][kGroup * kGroupRows][kGroupPitch];                         // hi, lo; row 16 * head + r
  __half k[2][kGroupTokens][kGroupPitch], v[2][kGroupTokens][kGroupPitch];  // two buffers
  __half p[2][kGroup * kGroupRows][kWeightPitch];                        // hi, lo
  float exchange[2][kGroup * kGroupRows];
};

struct RowTile {
  uint32_t start, rows, first, attended, slot;  // first: position of its first row; attended: context of its last row
};

__device__ __forceinline__ uint32_t tiles_of(const infdev_query& query) { return query.count > 1 ? (query.count + kGroupRows - 1) / kGroupRows : 0u; }

__device__ __forceinline__ RowTile tile_of(const infdev_query& query, uint32_t index) {
  RowTile tile;
  tile.start = query.start + index * kGroupRows;
  tile.rows = min(uint32_t(kGroupRows), query.count - index * kGroupRows);
  tile.first = query.position + index * kGroupRows;
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
// round over the queries tells.
__device__ __forceinline__ bool find_item(const infdev_query* queries, int queryCount, uint32_t most, uint32_t maxSplits, uint32_t item, RowTile& tile,
                                          uint32_t& split, uint32_t& piece, uint32_t& items) {
  const uint32_t lane = threadIdx.x & 31;
  for (int base = 0; base < queryCount; base += 32) {
    uint32_t mine = 0, tiles = 0;
    infdev_query query = {};
    if (base + int(lane) < queryCount) {
      query = queries[base + lane];
      tiles = tiles_of(query);
      for (uint32_t t = 0; t < tiles; ++t) {
        const RowTile each = tile_of(query, t);
        mine += piece_count(each.attended, piece_tokens(each.attended, each.rows, most, maxSplits));
      }
    }
    uint32_t inclusive = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t other = __shfl_up_sync(0xffffffffu, inclusive, o);
      if (int(lane) >= o)
        inclusive += other;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inclusive, 31);
    items = queryCount <= 32 ? total : 0xffffffffu;
    if (item >= total) {
      item -= total;
      continue;
    }
    const int owner = __ffs(__ballot_sync(0xffffffffu, inclusive > item)) - 1;
    uint32_t found[7] = {};
    if (int(lane) == owner) {
      uint32_t local = item - (inclusive - mine);
      for (uint32_t t = 0; t < tiles; ++t) {
        const RowTile each = tile_of(query, t);
        const uint32_t tokens = piece_tokens(each.attended, each.rows, most, maxSplits), count = piece_count(each.attended, tokens);
        if (local < count) {
          found[0] = each.start, found[1] = each.rows, found[2] = each.first, found[3] = each.attended, found[4] = each.slot, found[5] = local,
          found[6] = tokens;
          break;
        }
        local -= count;
      }
    }
#pragma unroll
    for (int i = 0; i < 7; ++i)
      found[i] = __shfl_sync(0xffffffffu, found[i], owner);
    tile = {found[0], found[1], found[2], found[3], found[4]};
    split = found[5], piece = found[6];
    return true;
  }
  return false;
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __half* address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(address)));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], const __half* address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(address)));
}
// {a, b} as fp16 hi and lo pairs
__device__ __forceinline__ uint2 split_pair(float a, float b) {
  const uint32_t hi = pack_half2(a, b);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  return make_uint2(hi, pack_half2(a - f.x, b - f.y));
}

// 0x8000 in each half of `pair` that is an infinity or a NaN.
__device__ __forceinline__ uint32_t not_finite(uint32_t pair) { return ((pair & 0x7c007c00u) + 0x04000400u) & 0x80008000u; }

__global__ void __launch_bounds__(kGroupThreads, 1)
    attention_group_kernel(const float* q, const __half* cacheK, const __half* cacheV, const infdev_query* queries, int queryCount, const int32_t* table,
                           int tableStride, int blockTokens, uint32_t most, uint32_t maxSplits, float* partials) {
  pdl_wait();  // first: the scan of the queries of one row starts beside this kernel and relies on it
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t groupRaw[];
  GroupShared& sh = *reinterpret_cast<GroupShared*>(groupRaw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = warp & 3, half = warp >> 2, g = lane >> 2, t = lane & 3;
  const int rowBase = head * kGroupRows;  // this warp's 16 rows of q, p and exchange
  RowTile tile;
  uint32_t split, piece, items = 0xffffffffu;
  for (uint32_t item = blockIdx.x;
       item / kKvHeads < items && find_item(queries, queryCount, most, maxSplits, item / kKvHeads, tile, split, piece, items); item += gridDim.x) {
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
    constexpr int kQuads = kGroup * kGroupRows * (kDim / 4) / kGroupThreads;
    float4 value[kQuads];
#pragma unroll
    for (int i = 0; i < kQuads; ++i) {
      const int at = i * kGroupThreads + threadIdx.x, row = at / (kDim / 4), d = at % (kDim / 4) * 4, r = row % kGroupRows, h = row / kGroupRows;
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
// GROUPED: the splits of a row whose query has several are those of attention_group_kernel.
template <bool GROUPED>
__global__ void __launch_bounds__(256) attention_reduce_kernel(const float* partials, const float* qg, const infdev_query* queries, int queryCount,
                                                               uint32_t most, uint32_t maxSplits, float* out, uint8_t* image) {
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t headRow = blockIdx.x, row = headRow / kQHeads, dim = threadIdx.x;
  const infdev_query& info = query_of_row(queries, queryCount, row);
  uint32_t count;
  if (GROUPED && info.count > 1) {
    const RowTile tile = tile_of(info, (row - info.start) / kGroupRows);
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
  launch_kernel<2>(attention_prepare_kernel, unsigned(rows * 20), 256, 0, stream, qg, rawK, rawV, qNorm, kNorm, rope, queries, queryCount, table, tableStride, blockTokens, q,
                                                                     static_cast<__half*>(cacheK), static_cast<__half*>(cacheV));
  return cudaGetLastError();
}

cudaError_t attention_launch(const float* q, const float* qg, const void* cacheK, const void* cacheV, const infdev_query* queries,
                             int queryCount, const int32_t* table, int tableStride, int blockTokens, int64_t rows, uint32_t maxSplits, float* partials, float* out,
                             uint8_t* image, bool rowwise, int sms, cudaStream_t stream, int* launches) {
  *launches = 0;
  if (rows <= 0)
    return cudaSuccess;
  *launches = 2;
  const uint32_t splits = std::min<uint32_t>(maxSplits, 32);  // the merge keeps one split per lane
  // The group kernel takes passes whose queries have five rows or more on average, unless no context of the pass can be long
  // (the table has no room for it): with r rows a query, its longer chain costs 2 us where r x context is below about 4096 (8
  // rows of 128 tokens 18.7 against 16.7 us for prepare and attention), from there on it is level or faster (8 rows of 2008
  // tokens 20.8 against 29.1, 16 of 616 22.8 against 23.6, 16 of 2016 22.8 against 39.4, 64 of 128 24.0 against 28.0).
  const int64_t capacity = int64_t(tableStride) * blockTokens;
  const bool grouped = rows >= 32 * int64_t(queryCount) || (rows >= 5 * int64_t(queryCount) && rows * capacity >= 4096 * int64_t(queryCount));
  // The group kernel copies q in pieces of 16 bytes, the scan in pieces of 8.
  if (grouped && !rowwise && reinterpret_cast<uintptr_t>(q) % 16 == 0) {
    static PerDeviceOnce configured;
    if (const cudaError_t e = configure_shared_memory(attention_group_kernel, sizeof(GroupShared), configured))
      return e;
    const int64_t tiles = std::max<int64_t>((rows + kGroupRows - 1) / kGroupRows, queryCount);
    const uint32_t most = uint32_t(std::clamp<int64_t>(sms / (kKvHeads * tiles), 1, splits));
    const int64_t items = (rows + queryCount) * kKvHeads * splits;  // no more than these
    launch_kernel<2>(attention_group_kernel, unsigned(std::min<int64_t>(items, sms)), kGroupThreads, sizeof(GroupShared), stream, q,
                  static_cast<const __half*>(cacheK), static_cast<const __half*>(cacheV), queries, queryCount, table, tableStride, blockTokens, most, splits,
                  partials);
    // Queries of one row stay with the scan, which is faster there: no query rows to share a tile with, and six small CTAs per
    // SM hide the copies that the group kernel's single CTA waits for. Which queries they are only the device knows; with a
    // single query there are none.
    if (queryCount > 1) {
      *launches = 3;
      // Its CTAs start on the SMs that the group kernel leaves first: shared memory that nobody uses spreads the few of a pass with
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
    launch_kernel<2>(attention_reduce_kernel<true>, unsigned(rows * kQHeads), 256, 0, stream, partials, qg, queries, queryCount, most, splits, out, image);
    return cudaGetLastError();
  }
  launch_kernel(attention_scan_kernel<false>, dim3(splits, kKvHeads, unsigned(rows)), 128, 0, stream, q, static_cast<const __half*>(cacheK),
                                                                                       static_cast<const __half*>(cacheV), queries, queryCount, table,
                                                                                       tableStride, blockTokens, splits, partials);
  launch_kernel(attention_reduce_kernel<false>, unsigned(rows * kQHeads), 256, 0, stream, partials, qg, queries, queryCount, 0u, splits, out, image);
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
  launch_kernel(attention_reduce_kernel<false>, unsigned(rows * kQHeads), 256, 0, stream, partials, qg, queries, queryCount, 0u, uint32_t(kStaticSplits), out, nullptr);
  return cudaGetLastError();
}

int attention_static_max_rows() { return kStaticRows; }

}  // namespace infdev
