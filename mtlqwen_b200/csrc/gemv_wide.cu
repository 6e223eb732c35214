// Fused-dequantisation tensor-core GEMM for 9 to 128 activation rows over GGUF Q5_K / Q6_K / Q8_0 / IQ4_XS weights, with the
// precision of the fp16 GEMV (gemv.cu): exact integer quants as the A operand, activations split x = hi + lo into two fp16
// fragments, sub-block scales applied to fp32 accumulators.
//
// Replaces linear_prefill[_small] of those types (quant_linear.metal:151-233) and the output head of passes with several
// sampled rows per sequence. The GEMV in slices of eight rows decodes every weight once per slice; decoding a fragment of 16 k
// costs about 30 instructions, multiplying it with a tile of eight rows about 8, so here up to five tiles share one decode.
// The scales of 16 or 32 k have to reach the accumulators between MMAs, which needs them in registers: mma.sync, not tcgen05
// (whose accumulators live in tensor memory; weights with their scales multiplied in need three fp16 products to keep 22 bits).
//
//  * wide_prepare_kernel writes the activations once, in fragment order, as one contiguous image per super-block and group of
//    NT tiles, so that a CTA fetches them with bulk copies.
//  * A CTA keeps the image of up to 20 / NT super-blocks in shared memory and streams weights past it, one 16-row x 1
//    super-block slab per stage. Each of the eight consumer warps owns 16-row tiles of its own: no reduction, no barrier
//    between warps while a chunk of K lasts. Between chunks the sums rest in the result (which the L2 holds).
//  * CTAs are spread over (group of up to 40 rows, slice of K) pairs; slices are added up by wide_reduce_kernel in a fixed
//    order. More slices are taken only where the tiles alone leave the SMs short of work (see slices()).
//
// What bounds it: shared memory and the tensor pipe together. A group of 16 k x 16 weights x 8 rows is 16 cycles of MMA and 16
// cycles of a scheduler's share of the fragment reads; with four tiles a unit (16 rows x 256 k) takes a scheduler 1.0 to 1.3
// us of which the MMAs are 0.57. Slices of eight rows against this kernel: Q6_K output head 248320 x 4096, 16 rows 481 -> 304
// us, 40 rows 1180 -> 650 us; projections of a layer of mixed types, 16 rows 176 -> 126 us, 40 rows 440 -> 216 us, 128 rows
// 1410 -> 544 us. At nine rows 176 -> 119 us for the layer, which is why it starts there. A chunk's sum is added to what
// rests in the result at the chunk's end: fetching that first and adding on top hid the latency (530 us at 128 rows) but lost
// accuracy (Q6_K, K = 12288: 2.0e-7 against fp64; 1.3e-7 now, 1.4e-7 for the slices). The warp index is made warp-uniform for
// the compiler (__shfl_sync): without it the roles' addresses take registers of every lane and five tiles spilled (40 rows of
// the head 790 us).
#include <algorithm>
#include <type_traits>
#include "gemv_units.cuh"
#include "kernels.h"

namespace infdev {
namespace {

constexpr int kConsumerWarps = 8;
constexpr int kThreads = (kConsumerWarps + 2) * kWarp;  // + weight producer, + activation producer
constexpr int kTileRows = kGemvTileRows;
constexpr int kMaxSlices = 8;  // of K
constexpr int kMaxDepth = 4;  // ring slots of a consumer warp
constexpr int kMaxTiles = 5;  // a group's tiles of eight rows: the MMAs of four take longer than the decode, more tiles spill registers
constexpr int kSharedBytes = 227 * 1024, kControlBytes = 1024;
constexpr int kFragmentBytes = 16 * 32 * 16, kSumBytes = 32 * 8, kScaleBytes = 8 * 4;
static_assert(kFragmentBytes + kSumBytes + kScaleBytes == kWideTileBytes, "image layout");

// Bytes of a super-block and of the box row that holds it: blocks start at any even byte (Q6_K) or at 8 mod 16 (IQ4_XS),
// a copy at the 16-byte boundary before it. All pitches are odd multiples of 16, which puts the eight rows of a warp-wide
// load into different banks. kResidentTiles: tiles x super-blocks of activations that leave every consumer warp two ring slots.
struct Q5K {
  static constexpr int kBlockBytes = 176, kPitch = 176, kResidentTiles = 20;
};
struct Q6K {
  static constexpr int kBlockBytes = 210, kPitch = 240, kResidentTiles = 20;
};
struct Q8 {
  static constexpr int kBlockBytes = 272, kPitch = 272, kResidentTiles = 19;
};
struct IQ4 {
  static constexpr int kBlockBytes = 136, kPitch = 144, kResidentTiles = 20;
};

struct Control {
  uint64_t full[kMaxDepth][kConsumerWarps], empty[kMaxDepth][kConsumerWarps], imageFull, imageFree;
  int abort;
};
static_assert(sizeof(Control) <= kControlBytes, "control block too large");

template <class Q> constexpr int stage_bytes() { return kTileRows * Q::kPitch; }
template <class Q, int NT> constexpr int resident_blocks() { return Q::kResidentTiles / NT; }
template <class Q, int NT> constexpr int resident_bytes() {  // tiled copies land on 128-byte boundaries
  return (resident_blocks<Q, NT>() * NT * kWideTileBytes + 127) / 128 * 128;
}
// Slots of a consumer warp. They are its own: with slots that change hands, a warp that runs ahead could find the parity of
// the phase before last, whose copy has not landed, and take it for its own.
template <class Q, int NT> constexpr int depth() {
  return std::min(kMaxDepth, (kSharedBytes - kControlBytes - resident_bytes<Q, NT>()) / (kConsumerWarps * stage_bytes<Q>()));
}
template <class Q, int NT> constexpr int shared_bytes() {
  return kControlBytes + resident_bytes<Q, NT>() + depth<Q, NT>() * kConsumerWarps * stage_bytes<Q>();
}

// The image of one super-block: per tile the fragments hi.xy lo.xy of a lane, then the sums and the scales of all tiles.
template <int NT> struct ImageRows {
  const uint4* fragments;  // this lane's entry of fragment 0, tile 0
  const uint2* minSums;    // this lane's entry of tile 0
  const float* powers;     // rows 2t and 2t + 1 of tile 0
  static constexpr bool kSplit = true;
  __device__ __forceinline__ uint4 fragment(int i, int tile) const { return fragments[(i * NT + tile) * 32]; }
  __device__ __forceinline__ float2 scales(int tile) const { return *reinterpret_cast<const float2*>(powers + tile * 8); }
  __device__ __forceinline__ uint2 sums(int tile) const { return minSums[tile * 32]; }
};

// One warp per (super-block, tile of eight rows): row = lane / 4, jj = lane % 4 loads four float4 of a 64-value span at
// 16 e + 4 jj. Scaled by a power of two per row and super-block so that the largest value lies in [512, 1024), as in gemv.cu.
__global__ void __launch_bounds__(128) wide_prepare_kernel(const float* x, int ldx, int m, int tiles, int groupTiles, int blocks, uint8_t* image) {
  pdl_launch_dependents();
  pdl_wait();
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= blocks * tiles)
    return;
  const int sb = item / tiles, group = item % tiles / groupTiles, tile = item % tiles % groupTiles;
  const int row = lane >> 2, jj = lane & 3, source = (item % tiles) * 8 + row;
  uint8_t* out = image + size_t(group * blocks + sb) * groupTiles * kWideTileBytes;
  uint4* fragments = reinterpret_cast<uint4*>(out) + tile * 32 + lane;
  uint2* sums = reinterpret_cast<uint2*>(out + groupTiles * kFragmentBytes) + tile * 32;
  float* powers = reinterpret_cast<float*>(out + groupTiles * (kFragmentBytes + kSumBytes)) + tile * 8;
  float4 v[4][4];
  float largest = 0.f;
#pragma unroll
  for (int tq = 0; tq < 4; ++tq)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[tq][e] = source < m ? *reinterpret_cast<const float4*>(x + size_t(source) * ldx + 256 * sb + 64 * tq + 16 * e + 4 * jj)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
      largest = fmaxf(fmaxf(fmaxf(largest, fabsf(v[tq][e].x)), fmaxf(fabsf(v[tq][e].y), fabsf(v[tq][e].z))), fabsf(v[tq][e].w));
    }
  largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
  largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 2));
  const float2 power = activation_power(largest);
  if (jj == 0)
    powers[row] = largest != INFINITY ? power.y : INFINITY;
  auto store = [&](int tq, const float4 (&span)[4]) {  // four scaled float4 of a 64-value span
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 w = span[e];
      uint4 b;
      b.x = pack_half2(w.x, w.y), b.y = pack_half2(w.z, w.w);
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&b.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&b.y));
      b.z = pack_half2(w.x - f0.x, w.y - f0.y), b.w = pack_half2(w.z - f1.x, w.w - f1.y);
      fragments[(tq * 4 + e) * groupTiles * 32] = b;
      s[e] = (w.x + w.y) + (w.z + w.w);
      s[e] += __shfl_xor_sync(0xffffffffu, s[e], 1);
      s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
    }
    if (jj == 0) {  // sums of the two 32-value sub-blocks of the span, hi and lo
      const float s0 = s[0] + s[1], s1 = s[2] + s[3];
      const uint32_t hi = pack_half2(s0, s1);
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
      sums[row * 4 + tq] = make_uint2(hi, pack_half2(s0 - f.x, s1 - f.y));
    }
  };
#pragma unroll
  for (int tq = 0; tq < 4; ++tq) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      v[tq][e].x *= power.x, v[tq][e].y *= power.x, v[tq][e].z *= power.x, v[tq][e].w *= power.x;
    store(tq, v[tq]);
  }
  if (__any_sync(0xffffffffu, largest == INFINITY)) {  // once more, from memory: out of the way of the ordinary case
#pragma unroll 1
    for (int tq = 0; tq < 4; ++tq) {
      float4 span[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        span[e] = scaled_with_infinities(source < m ? *reinterpret_cast<const float4*>(x + size_t(source) * ldx + 256 * sb + 64 * tq + 16 * e + 4 * jj)
                                                    : make_float4(0.f, 0.f, 0.f, 0.f),
                                         largest, power.x);
      store(tq, span);
    }
  }
}

__device__ __forceinline__ int find_segment(const WideParams& p, int tile) {
  int s = 0;
  while (s + 1 < p.nseg && tile >= p.seg[s + 1].tile0)
    ++s;
  return s;
}

// A CTA's part of the work: row group, slice [first, last) of the super-blocks, and the tiles index, index + ctas, ...
struct Part {
  int group, slice, first, last, index, ctas, tiles;
  __device__ explicit Part(const WideParams& p) {
    const int parts = p.groups * p.slices, part = int(blockIdx.x) % parts;
    index = int(blockIdx.x) / parts, ctas = int(gridDim.x) / parts;
    group = part % p.groups, slice = part / p.groups;
    first = p.blocks * slice / p.slices, last = p.blocks * (slice + 1) / p.slices;
    tiles = index < p.tiles ? (p.tiles - 1 - index) / ctas + 1 : 0;
  }
};

template <class Q, int NT> __global__ void __launch_bounds__(kThreads, 1) wide_kernel(const __grid_constant__ WideParams p) {
  constexpr int kDepth = depth<Q, NT>(), kResident = resident_blocks<Q, NT>();
  constexpr uint32_t kImageBytes = NT * kWideTileBytes;
  extern __shared__ __align__(128) uint8_t smem[];
  static_assert(kDepth >= 2 && stage_bytes<Q>() % 128 == 0 && kControlBytes % 128 == 0, "ring geometry");
  Control& ctl = *reinterpret_cast<Control*>(smem);
  uint8_t* image = smem + kControlBytes;
  uint8_t* ring = image + resident_bytes<Q, NT>();  // [kDepth][warp]

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kDepth * kConsumerWarps; ++s) {
      mbar_init(&ctl.full[s / kConsumerWarps][s % kConsumerWarps], 1);
      mbar_init(&ctl.empty[s / kConsumerWarps][s % kConsumerWarps], 1);
    }
    mbar_init(&ctl.imageFull, 1);
    mbar_init(&ctl.imageFree, kConsumerWarps);
    ctl.abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();
  volatile int* abortFlag = &ctl.abort;
  const Part part(p);
  const int chunks = (part.last - part.first + kResident - 1) / kResident, perChunk = (part.last - part.first + chunks - 1) / chunks;
  auto give_up = [&] {
    *abortFlag = 1;
    atomicExch(p.status, kStatusBarrierTimeout);
  };

  if (warp == kConsumerWarps) {
    // ---- weights: do not depend on the kernels before this one. Lane w serves consumer warp w: a copy is small, and one lane
    // that waits, looks up and issues for all eight warps in turn (about 500 cycles a copy) was what bounded the kernel.
    uint32_t used = 0;  // slots that this lane has filled
    bool ok = true;
    for (int chunk = 0; chunk < chunks && ok; ++chunk) {
      const int b0 = part.first + chunk * perChunk, b1 = min(part.last, b0 + perChunk);
      for (int round = 0; round < part.tiles && ok; round += kConsumerWarps) {
        const int live = min(kConsumerWarps, part.tiles - round);
        const bool mine = lane < live;
        const int tile = part.index + (round + lane) * part.ctas, segment = mine ? find_segment(p, tile) : 0;
        const int row = mine ? (tile - p.seg[segment].tile0) * kTileRows : 0;
        const CUtensorMap* const map = &p.map[segment];
        for (int sb = b0; sb < b1 && ok; ++sb) {
          if (mine) {
            const uint32_t slot = used % kDepth, lap = used / kDepth;
            if (lap > 0)
              ok = mbar_wait_bounded(&ctl.empty[slot][lane], (lap - 1) & 1, abortFlag);
            if (ok) {
              mbar_arrive_expect_tx(&ctl.full[slot][lane], uint32_t(stage_bytes<Q>()));
              tma_load_2d(ring + (slot * kConsumerWarps + lane) * stage_bytes<Q>(), map, (sb * Q::kBlockBytes & ~15) / 8, row, &ctl.full[slot][lane]);
              ++used;
            }
          }
          ok = __all_sync(0xffffffffu, ok);
        }
      }
    }
    if (!ok)
      give_up();
    // no copy may be in flight when the CTA ends, whoever gave up
    for (uint32_t i = used > uint32_t(kDepth) ? used - kDepth : 0; i < used; ++i)
      mbar_wait_bounded(&ctl.full[i % kDepth][lane], (i / kDepth) & 1, abortFlag);
    __syncwarp();
    pdl_wait();  // every thread of every kernel waits, so completion stays transitive along the stream
    return;
  }
  pdl_wait();  // activations, residuals and partial sums belong to the kernels before this one
  if (warp == kConsumerWarps + 1) {
    // ---- activations: the super-blocks of a chunk ----
    if (lane == 0) {
      bool ok = true;
      for (int chunk = 0; chunk < chunks; ++chunk) {
        if (chunk > 0)
          ok = mbar_wait_bounded(&ctl.imageFree, (chunk - 1) & 1, abortFlag);
        if (!ok)
          break;
        const int b0 = part.first + chunk * perChunk, count = min(part.last - b0, perChunk);
        mbar_arrive_expect_tx(&ctl.imageFull, uint32_t(count) * kImageBytes);
        for (int i = 0; i < count; ++i)
          bulk_load(image + i * kImageBytes, p.image + size_t(part.group * p.blocks + b0 + i) * kImageBytes, kImageBytes, &ctl.imageFull);
        ok = mbar_wait_bounded(&ctl.imageFull, chunk & 1, abortFlag);  // no copy may be in flight when the CTA ends
      }
      if (!ok)
        give_up();
    }
    return;
  }

  // ---- consumers ----
  const int g = lane >> 2, t = lane & 3, row0 = part.group * NT * 8 + 2 * t, m = p.m;
  const bool parked = p.pair || p.slices > 1;
  uint32_t used = 0;  // slots that this warp has read
  bool ok = true;
  for (int chunk = 0; chunk < chunks && ok; ++chunk) {
    const int b0 = part.first + chunk * perChunk, count = min(part.last - b0, perChunk);
    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&ctl.imageFull, chunk & 1, abortFlag));
    for (int round = 0; round < part.tiles && ok; round += kConsumerWarps) {
      const int live = min(kConsumerWarps, part.tiles - round);
      if (warp < live) {
        // Where the sums rest: the result, or the partial results that wide_reduce_kernel finishes. Copied out of the parameter
        // block, which is reached through a generic address and would be read again after every store.
        const int tile = part.index + (round + warp) * part.ctas;
        const GemvSeg& seg = p.seg[find_segment(p, tile)];
        const int ldy = parked ? p.pitch : seg.ldy, column = (tile - (parked ? 0 : seg.tile0)) * kTileRows + g;
        float* const y = parked ? p.partial + size_t(part.slice) * m * ldy : seg.y;
        const float* const before = chunk > 0 ? y : parked ? nullptr : seg.res;
        float total[NT][4];
        clear(total);
#pragma unroll 1
        for (int j = 0; j < count; ++j, ++used) {
          const uint32_t slot = used % kDepth;
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&ctl.full[slot][warp], (used / kDepth) & 1, abortFlag));
          if (!ok)
            break;
          const uint8_t* pA = ring + (slot * kConsumerWarps + warp) * stage_bytes<Q>() + ((b0 + j) * Q::kBlockBytes & 15) + g * Q::kPitch;
          const uint8_t* pB = pA + 8 * Q::kPitch;
          const uint8_t* block = image + j * kImageBytes;
          const ImageRows<NT> rows{reinterpret_cast<const uint4*>(block) + lane, reinterpret_cast<const uint2*>(block + NT * kFragmentBytes) + lane,
                                   reinterpret_cast<const float*>(block + NT * (kFragmentBytes + kSumBytes)) + 2 * t};
          if constexpr (std::is_same_v<Q, Q5K>) {
            q5k_unit(pA, pB, lane, rows, total);
          } else if constexpr (std::is_same_v<Q, Q8>) {
            q8_unit(pA, pB, lane, rows, total);
          } else if constexpr (std::is_same_v<Q, IQ4>) {
            iq4_unit(pA, pB, lane, rows, total);
          } else {
            q6k_unit<false>(pA, pB, lane, rows, total);
          }
          __syncwarp();
          if (lane == 0)
            mbar_arrive(&ctl.empty[slot][warp]);
        }
        if (ok) {
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // added here, not at the start: a chunk's own sum is rounded on a finer grid
              const int row = row0 + 8 * n + (i & 1);
              if (before && row < m)
                total[n][i] += before[size_t(row) * ldy + column + 8 * (i >> 1)];
            }
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int row = row0 + 8 * n + (i & 1);
              if (row < m)
                y[size_t(row) * ldy + column + 8 * (i >> 1)] = total[n][i];
            }
        }
      }
    }
    __syncwarp();
    if (lane == 0)
      mbar_arrive(&ctl.imageFree);
  }
  if (!ok && lane == 0)
    give_up();
}

// Adds up the slices, four values per thread, and finishes: y = sum (+ residual), or silu(gate) * up for a pair. The columns of
// all matrices lie side by side in a row of the partial results. AT_ONCE: a thread asks for all slices before it adds; with many rows it is the
// number of resident blocks that counts, which takes few registers. Projections of a layer of mixed types with 9, 16, 32, 48, 64, 80, 96 and 128 rows,
// one after the other / at once: 102.5 / 102.6, 104.5 / 101.0, 150.5 / 148.2, 218.8 / 223.0, 267.3 / 262.9, 315.6 / 315.7, 366.2 / 368.5 and 491.8 / 498.4 us.
template <bool AT_ONCE> __global__ void __launch_bounds__(256) wide_reduce_kernel(const __grid_constant__ WideParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int width = p.pair ? p.pitch / 2 : p.pitch;
  const size_t at = (size_t(blockIdx.x) * 256 + threadIdx.x) * 4, count = size_t(p.m) * p.pitch;
  if (at >= size_t(p.m) * width)
    return;
  const int row = int(at / width), column = int(at % width), slices = p.slices;
  auto total = [&](int from) {
    const float* partial = p.partial + size_t(row) * p.pitch + from;
    auto add = [](float4& sum, const float4& v) { sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w; };
    float4 sum = *reinterpret_cast<const float4*>(partial);
    if (AT_ONCE) {
      float4 v[kMaxSlices];
#pragma unroll
      for (int s = 1; s < kMaxSlices; ++s)
        if (s < slices)
          v[s] = *reinterpret_cast<const float4*>(partial + s * count);
#pragma unroll
      for (int s = 1; s < kMaxSlices; ++s)
        if (s < slices)
          add(sum, v[s]);
    } else {
      for (int s = 1; s < slices; ++s)
        add(sum, *reinterpret_cast<const float4*>(partial + s * count));
    }
    return sum;
  };
  float4 sum = total(column);
  const GemvSeg& seg = p.seg[find_segment(p, column / kTileRows)];
  const size_t to = size_t(row) * seg.ldy + (column - seg.tile0 * kTileRows);
  float* const y = seg.y + to;
  if (p.pair) {
    const float4 up = total(column + width);
    sum.x = silu_f(sum.x) * up.x, sum.y = silu_f(sum.y) * up.y, sum.z = silu_f(sum.z) * up.z, sum.w = silu_f(sum.w) * up.w;
  } else if (const float* residual = seg.res) {
    residual += to;
    sum.x += residual[0], sum.y += residual[1], sum.z += residual[2], sum.w += residual[3];
  }
  y[0] = sum.x, y[1] = sum.y, y[2] = sum.z, y[3] = sum.w;
}

// Slices of K, and CTAs: what the fullest CTA has to do, plus what a reduction of the slices costs (every partial result written
// and read). A round of up to four tiles puts one warp on a scheduler, which then waits for its own copies and products; a round
// of eight takes two such warps' issue slots. Fitted to every slice count of 616 shapes (four types, 16 to 20480 weight rows,
// K 2048 to 12288, 9 to 128 rows): 1.2 % above the best count on average, where a model without the idle schedulers' share
// lost 10.5 % (Q6_K 4096 x 4096 with 16 rows in one slice 19.5 us, in four 13.5; the slices of eight rows 16.5).
int slices(const WideParams& p, int tilesPerGroup, int sms) {
  int best = 1;
  double least = 0;
  for (int s = 1; s <= kMaxSlices && s <= p.blocks; ++s) {
    const int ctas = sms / (p.groups * s);
    if (ctas < 1 || ((s > 1 || p.pair) && size_t(s) * p.m * p.pitch > kWidePartialFloats))
      break;
    const int perCta = (p.tiles + ctas - 1) / ctas, rest = perCta % kConsumerWarps;
    const double busy = 0.15 + 0.1 * tilesPerGroup, lone = 0.2 + 0.1 * tilesPerGroup;  // microseconds for 16 weight rows x 256 k
    const double block = perCta / kConsumerWarps * 2 * busy + (rest == 0 ? 0.0 : rest <= kConsumerWarps / 2 ? lone : 2 * busy);
    const double cost = block * ((p.blocks + s - 1) / s) + (s > 1 ? s * double(p.m) * p.pitch * 8 / 2e7 : 0.0);
    if (s == 1 || cost < least)
      least = cost, best = s;
  }
  return best;
}

template <class Q, int NT> cudaError_t launch_tiles(const WideParams& p, int sms, cudaStream_t stream) {
  static PerDeviceOnce configured;
  constexpr size_t bytes = shared_bytes<Q, NT>();
  if (cudaError_t e = configure_shared_memory(wide_kernel<Q, NT>, bytes, configured))
    return e;
  const int parts = p.groups * p.slices;
  launch_kernel<1>(wide_kernel<Q, NT>, std::min(p.tiles, sms / parts) * parts, kThreads, bytes, stream, p);
  return cudaGetLastError();
}

template <class Q> cudaError_t launch(const WideParams& params, const float* x, int ldx, int sms, cudaStream_t stream, int* launches) {
  WideParams p = params;
  const int tiles = (p.m + 7) / 8;
  p.groups = (tiles + kMaxTiles - 1) / kMaxTiles;
  const int groupTiles = (tiles + p.groups - 1) / p.groups;
  p.slices = slices(p, groupTiles, sms);
  const int warps = p.groups * groupTiles * p.blocks;
  launch_kernel<1>(wide_prepare_kernel, (warps + 3) / 4, 128, 0, stream, x, ldx, p.m, p.groups * groupTiles, groupTiles, p.blocks,
                const_cast<uint8_t*>(p.image));
  cudaError_t e = cudaErrorInvalidValue;
  switch (groupTiles) {
    case 2: e = launch_tiles<Q, 2>(p, sms, stream); break;
    case 3: e = launch_tiles<Q, 3>(p, sms, stream); break;
    case 4: e = launch_tiles<Q, 4>(p, sms, stream); break;
    case 5: e = launch_tiles<Q, 5>(p, sms, stream); break;
  }
  *launches = 2;
  if (e == cudaSuccess && (p.pair || p.slices > 1)) {
    launch_kernel<1>(p.m <= 64 ? wide_reduce_kernel<true> : wide_reduce_kernel<false>, unsigned((size_t(p.m) * p.pitch / (p.pair ? 8 : 4) + 255) / 256), 256, 0, stream, p);
    *launches = 3;
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace

GemvBox wide_box(int type) {
  switch (type) {
    case 8: return {Q8::kBlockBytes, 1, Q8::kPitch - Q8::kBlockBytes};
    case 13: return {Q5K::kBlockBytes, 1, Q5K::kPitch - Q5K::kBlockBytes};
    case 14: return {Q6K::kBlockBytes, 1, Q6K::kPitch - Q6K::kBlockBytes};
    case 23: return {IQ4::kBlockBytes, 1, IQ4::kPitch - IQ4::kBlockBytes};
    default: return {0, 0, 0};
  }
}

cudaError_t wide_launch(int type, const WideParams& p, const float* x, int ldx, int sms, cudaStream_t stream, int* launches) {
  switch (type) {
    case 8: return launch<Q8>(p, x, ldx, sms, stream, launches);
    case 13: return launch<Q5K>(p, x, ldx, sms, stream, launches);
    case 14: return launch<Q6K>(p, x, ldx, sms, stream, launches);
    case 23: return launch<IQ4>(p, x, ldx, sms, stream, launches);
  }
  return cudaErrorInvalidValue;
}

}  // namespace infdev
