// Dequant-fused fp16 tensor-core GEMV for decode (M <= 8 activation rows) over GGUF Q4_K / Q5_K / Q6_K / Q8_0 / IQ4_XS
// weights. It serves every Q6_K matrix (lm_head), the Q5_K, Q8_0 and IQ4_XS ones whose shape it takes (formats.cu has the
// rest) and, when the integer kernel of q4k_decode.cu is switched off, the Q4_K ones.
//
// Replaces linear_decode_q4_k[_add] (quant_linear.metal:245-327), linear_decode_q5_k / q6_k / q8_0[_add] (:329-570) and
// mlp_gate_up of Q4_K, Q5_K and IQ4_XS (fused_kernels.metal:11-200). The reference re-reads the weights once per
// activation row (grid.y = rows); here up to 8 rows share one pass over the weights.
//
// Design (one persistent CTA per SM: 16 consumer warps, or 8 where K is one slab, 2 finisher warps (1 where a pair's ring would be too
// short) and 1 producer warp):
//  * The weight matrix is a contiguous byte stream (row n = K/256 super-blocks). The producer warp moves
//    16-row x 8-super-block slabs into a shared-memory ring with one tiled TMA copy each (a tensor map over
//    the packed rows as 8-byte elements) that completes on an mbarrier; nothing else touches HBM for the weights.
//  * At 8 rows the fp32 FMA pipe cannot keep up with HBM (8 FMAs per 4-bit weight), so the products run
//    on the tensor cores as m16n8k16: A = 16 weight rows x 16 k, B = 16 k x 8 activation rows.
//    The summation index of an MMA is a dummy, so k is permuted freely to suit the packed layout; the
//    activations come in the same permutation.
//  * A consumer warp works on the same super-block of every tile of a K chunk. It loads and splits that super-block's activations
//    itself, once per chunk, and keeps the high halves in registers and the low ones in shared memory where only it reads them.
//  * The partial sums of a tile go to a finisher warp (gemv_ring.cuh), so consumers never wait for each other.
//    With eight consumer warps that took two super-blocks a tile, all activations in shared memory and a barrier after every tile:
//    output head 248320 x 4096 Q6_K, eight rows 232 -> 211 us, 12288 x 4096 Q5_K 17.7 -> 16.0, Q8_0 16.7 -> 14.4, IQ4_XS 19.9 -> 18.2,
//    4096 x 12288 (three chunks) Q6_K 24.8 -> 21.2, Q8_0 23.7 -> 19.9. Eight warps that held all their activations in registers,
//    216 of them by setmaxnreg, measured 250 on the head: two warps a scheduler leave it idle while one waits for a product.
//    (Sixteen leave a thread 96 registers: Q5_K spills five of them, which 12288 x 4096 does not show.)
//  * Q4_K: A holds the exact integers sc*q (<= 945, exact in fp16); the super-block scale d is applied to
//    the fp32 accumulator after each super-block, and the -dmin*m term is one more MMA against the
//    per-sub-block activation sums. Q6_K: A holds q-32 exactly, the per-16 scale sc is applied to the
//    accumulator after each MMA (one MMA = one scale group) and d once per super-block.
//  * Activations are split x = hi + lo into two fp16 fragments (XSPLIT = 2) so the result keeps fp32
//    accuracy; XSPLIT = 1 drops lo (relative error ~3e-4, still inside the 1e-3 contract).
//  * Every mbarrier wait is bounded; on a timeout the kernel raises an abort flag, records a status code
//    and all roles leave their loops.
#include <type_traits>
#include "gemv_ring.cuh"
#include "gemv_units.cuh"

namespace infdev {
namespace {

constexpr int kStageBlocks = kGemvStageBlocks;  // super-blocks per ring stage: one per warp of a half
constexpr int kStageWarps = kStageBlocks;

constexpr int kTileRows = kGemvTileRows;

// How a block type lies in a ring stage: kBoxes tiled copies of 16 rows x kStageBlocks / kBoxes super-blocks (a box is at
// most 256 elements of 8 bytes wide, which eight super-blocks of Q8_0 exceed), each row kPad bytes wider than its
// super-blocks where the pitch would otherwise put the eight rows of a warp-wide load into the same banks.
struct Q4K {
  static constexpr int kBlockBytes = 144, kBoxes = 1, kPad = 0;
  static constexpr bool kMinTerm = true;
};
struct Q5K {
  static constexpr int kBlockBytes = 176, kBoxes = 1, kPad = 16;  // pitch 1424 = 16 mod 128
  static constexpr bool kMinTerm = true;
};
struct Q6K {
  static constexpr int kBlockBytes = 210, kBoxes = 1, kPad = 0;  // pitch 1680 = 16 mod 128
  static constexpr bool kMinTerm = false;
};
struct Q8 {
  static constexpr int kBlockBytes = 272, kBoxes = 2, kPad = 16;  // eight Q8_0 blocks; pitch 1104 = 80 mod 128
  static constexpr bool kMinTerm = false;
};
struct IQ4 {
  static constexpr int kBlockBytes = 136, kBoxes = 1, kPad = 16;  // pitch 1104
  static constexpr bool kMinTerm = false;
};
template <class Q> constexpr int box_blocks() { return kStageBlocks / Q::kBoxes; }
template <class Q> constexpr int row_pitch() { return box_blocks<Q>() * Q::kBlockBytes + Q::kPad; }
template <class Q> constexpr int box_bytes() { return kTileRows * row_pitch<Q>(); }
template <class Q> constexpr int stage_bytes() { return Q::kBoxes * box_bytes<Q>(); }

// Roles and shared memory of a CTA. HALVES: groups of eight consumer warps; with two, consecutive ring stages alternate between them.
template <class Q, int NMAT, int XSPLIT, int HALVES> struct Layout {
  static constexpr int kConsumers = kStageWarps * HALVES;
  static constexpr int kChunkBlocks = kStageBlocks * HALVES;  // super-blocks of K per pass over the tiles: a slab per half
  static constexpr int kLowBytes = XSPLIT == 2 ? kConsumers * 16 * 32 * 8 : 0;  // low halves of the activations: [warp][fragment][lane]
  static constexpr size_t fixed_bytes(int finishers) { return kRingControlBytes + kLowBytes + size_t(finishers) * NMAT * kConsumers * 128 * 4; }
  // As many ring stages as fit beside that in the 227 KB a CTA may use; with two halves an even number, so that a slot always belongs to
  // the same one (a half that ran ahead in a slot of the other one could find the parity of the phase before last).
  static constexpr int stages(int finishers) {
    const int fit = int((size_t(227) * 1024 - fixed_bytes(finishers)) / stage_bytes<Q>());
    return (fit > kMaxStages ? kMaxStages : fit) / HALVES * HALVES;
  }
  // A second finisher's buffer may not cost a half its second stage, without which it computes and copies in turn: a pair of Q8_0
  // (12288 x 4096, eight rows) 36.8 us with two finishers and two stages, 25.8 with one and four; IQ4_XS and Q5_K, which have four and six
  // with two finishers, 32.6 and 27.1 against 33.4 and 27.5.
  static constexpr int kFinishers = stages(2) < 2 * HALVES ? 1 : 2;
  static constexpr int kStages = stages(kFinishers);
  static constexpr size_t kBytes = fixed_bytes(kFinishers) + size_t(kStages) * stage_bytes<Q>();
  static constexpr int kProducer = kConsumers + kFinishers;  // warps: consumers, finishers, producer
  static constexpr int kThreads = (kProducer + 1) * kWarp;
  static_assert(kStages >= 2 && kStages >= HALVES, "a slot for each half");
};

// ---- Q4_K: one 16-row x 256-k unit -------------------------------------------------------------
// Lane (g = lane/4, t = lane%4) owns weight rows g and g+8 and, in each, the 16-byte quant chunks t and
// t+4 of the super-block (chunk c = bytes [16c,16c+16) of qs: low nibbles are elements 64*(c/2) +
// 16*(c%2) + [0,16) , high nibbles the same + 32; GGUF layout as read by dequant_tile,
// quant_linear.metal:39-46). MMA i = (chunk select, word j, nibble h) consumes bytes 0..3 of word j.
__device__ __forceinline__ uint4 lds128(uint32_t address) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(address));
  return v;
}
// The activations of one super-block as a lane (g, t) of its consumer warp has them: of row g the four values of quarter t of every
// 16-value group, as B fragments, scaled by a power of two per row.
template <int XSPLIT> struct OwnRows {
  uint2 high[16];
  uint2* low;     // this lane's entry of fragment 0; XSPLIT 2
  uint2 minSums;  // Q4_K, Q5_K: fragment of the sums of the sub-blocks 2t and 2t + 1 of row g, hi and lo
  float2 powers;  // inverse powers of the rows 2t and 2t + 1
  static constexpr bool kSplit = XSPLIT == 2;
  __device__ __forceinline__ uint4 fragment(int i, int) const {
    const uint2 l = kSplit ? low[i * 32] : make_uint2(0u, 0u);
    return make_uint4(high[i].x, high[i].y, l.x, l.y);
  }
  __device__ __forceinline__ float2 scales(int) const { return powers; }
  __device__ __forceinline__ uint2 sums(int) const { return minSums; }
};

// Loads them for the super-block at x.
template <class Q, int XSPLIT> __device__ __forceinline__ void load_rows(OwnRows<XSPLIT>& to, const float* x, int ldx, int m, int lane) {
  constexpr bool kQ4 = std::is_same_v<Q, Q4K>;
  const int g = lane >> 2, t = lane & 3;
  const float* src = x + size_t(g) * ldx;
  float4 v[16];
  float largest = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    // Q4_K: MMA i = (chunk select, word, nibble) multiplies the bytes of word (i / 2) % 4 of chunk t + 4 (i / 8)
    const int chunk = t + 4 * (i >> 3), at = kQ4 ? 64 * (chunk >> 1) + 16 * (chunk & 1) + 32 * (i & 1) + 4 * ((i >> 1) & 3) : 16 * i + 4 * t;
    v[i] = g < m ? *reinterpret_cast<const float4*>(src + at) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i)
    largest = fmaxf(fmaxf(fmaxf(largest, fabsf(v[i].x)), fmaxf(fabsf(v[i].y), fabsf(v[i].z))), fabsf(v[i].w));
  largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
  largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 2));
  const float2 power = activation_power(largest);
  if (__any_sync(0xffffffffu, largest == INFINITY)) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      v[i] = scaled_with_infinities(v[i], largest, power.x);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      v[i].x *= power.x, v[i].y *= power.x, v[i].z *= power.x, v[i].w *= power.x;
  }
  const float inverse = largest != INFINITY ? power.y : INFINITY;
  to.powers.x = __shfl_sync(0xffffffffu, inverse, 8 * t), to.powers.y = __shfl_sync(0xffffffffu, inverse, 8 * t + 4);
  if (Q::kMinTerm) {
    float even, odds;  // the sums of the sub-blocks 2t and 2t + 1
    if (kQ4) {
      float part[4];  // [chunk select][nibble]; two lanes share a sub-block
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        part[c] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 w = v[(c >> 1) * 8 + 2 * j + (c & 1)];
          part[c] += (w.x + w.y) + (w.z + w.w);
        }
        part[c] += __shfl_xor_sync(0xffffffffu, part[c], 1);
        part[c] = __shfl_sync(0xffffffffu, part[c], (lane & ~3) | 2 * (t & 1));
      }
      even = t < 2 ? part[0] : part[2], odds = t < 2 ? part[1] : part[3];
    } else {
      float part[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 a = v[2 * j], b = v[2 * j + 1];
        part[j] = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
      }
      // over the four lanes of a row; each step halves the sub-blocks that a lane still sums for
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, t & 2 ? part[j] : part[4 + j], 2);
        part[j] = (t & 2 ? part[4 + j] : part[j]) + other;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, t & 1 ? part[j] : part[2 + j], 1);
        part[j] = (t & 1 ? part[2 + j] : part[j]) + other;
      }
      even = part[0], odds = part[1];
    }
    to.minSums.x = pack_half2(even, odds);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&to.minSums.x));
    to.minSums.y = pack_half2(even - f.x, odds - f.y);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float4 w = kQ4 ? make_float4(v[i].x, v[i].z, v[i].y, v[i].w) : v[i];  // Q4_K: A pairs bytes (0,2) and (1,3) of a quant word
    uint2 h = make_uint2(pack_half2(w.x, w.y), pack_half2(w.z, w.w)), l = make_uint2(0u, 0u);
    if (XSPLIT == 2) {
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&h.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
      l = make_uint2(pack_half2(w.x - f0.x, w.y - f0.y), pack_half2(w.z - f1.x, w.w - f1.y));
    }
    to.high[i] = h;
    if (XSPLIT == 2)
      to.low[i * 32] = l;
  }
}

// pA / pB: shared-memory addresses of the super-block of rows g and g+8.
template <int XSPLIT>
__device__ __forceinline__ void q4k_unit(uint32_t pA, uint32_t pB, int t, const OwnRows<XSPLIT>& x, float (&total)[4]) {
  const uint4 hA = lds128(pA), hB = lds128(pB);
  // 6-bit scales / mins of the 8 sub-blocks, four per word (scale_min_k4, quant_linear.metal:12-20).
  const uint32_t scA[2] = {hA.y & 0x3f3f3f3fu, (hA.w & 0x0f0f0f0fu) | ((hA.y >> 2) & 0x30303030u)};
  const uint32_t mnA[2] = {hA.z & 0x3f3f3f3fu, ((hA.w >> 4) & 0x0f0f0f0fu) | ((hA.z >> 2) & 0x30303030u)};
  const uint32_t scB[2] = {hB.y & 0x3f3f3f3fu, (hB.w & 0x0f0f0f0fu) | ((hB.y >> 2) & 0x30303030u)};
  const uint32_t mnB[2] = {hB.z & 0x3f3f3f3fu, ((hB.w >> 4) & 0x0f0f0f0fu) | ((hB.z >> 2) & 0x30303030u)};
  const int shift = (t >> 1) * 16;
  constexpr uint32_t k1024 = 0x64006400u, kNeg1024 = 0xE400E400u, kSixteenth = 0x2C002C00u, kNeg64 = 0xD400D400u;
  // Four independent accumulator chains: consecutive MMAs never wait on each other's results.
  float acc[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
    acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
#pragma unroll
  for (int cs = 0; cs < 2; ++cs) {
    // This lane's quant chunk t + 4*cs of both rows. Its low nibbles belong to sub-block 2*(c/2), the high ones to
    // 2*(c/2)+1; their scales are bytes 2*(t/2), 2*(t/2)+1 of the cs-th scale word.
    const uint4 qA = lds128(pA + 16 + 64 * cs + 16 * t), qB = lds128(pB + 16 + 64 * cs + 16 * t);
    const uint32_t pairA = (scA[cs] >> shift) & 0xffffu, pairB = (scB[cs] >> shift) & 0xffffu;
    const uint32_t sLA = hsub2_u32(__byte_perm(pairA, 0x64u, 0x4040), k1024), sHA = hsub2_u32(__byte_perm(pairA, 0x64u, 0x4141), k1024);
    const uint32_t sLB = hsub2_u32(__byte_perm(pairB, 0x64u, 0x4040), k1024), sHB = hsub2_u32(__byte_perm(pairB, 0x64u, 0x4141), k1024);
    const uint32_t nLA = hmul2_u32(sLA, kNeg1024), nLB = hmul2_u32(sLB, kNeg1024);
    const uint32_t mHA = hmul2_u32(sHA, kSixteenth), mHB = hmul2_u32(sHB, kSixteenth);
    const uint32_t nHA = hmul2_u32(sHA, kNeg64), nHB = hmul2_u32(sHB, kNeg64);
    const uint32_t wordsA[4] = {qA.x, qA.y, qA.z, qA.w}, wordsB[4] = {qB.x, qB.y, qB.z, qB.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t wA = wordsA[j], wB = wordsB[j], vA = wA >> 8, vB = wB >> 8;
      const int i = (cs * 4 + j) * 2;          // MMA index of the low-nibble step; i + 1 is the high-nibble step
      uint32_t a[4];
      // low nibbles: (1024 + q) * sc - 1024 * sc, exact in fp16
      a[0] = hfma2_u32((wA & 0x000f000fu) | k1024, sLA, nLA);
      a[1] = hfma2_u32((wB & 0x000f000fu) | k1024, sLB, nLB);
      a[2] = hfma2_u32((vA & 0x000f000fu) | k1024, sLA, nLA);
      a[3] = hfma2_u32((vB & 0x000f000fu) | k1024, sLB, nLB);
      uint4 b = x.fragment(i, 0);
      mma_16816(acc[j & 1], a, b.x, b.y);
      if (XSPLIT == 2)
        mma_16816(acc[j & 1], a, b.z, b.w);
      // high nibbles in place: (1024 + 16 q) * sc/16 - 64 * sc
      a[0] = hfma2_u32((wA & 0x00f000f0u) | k1024, mHA, nHA);
      a[1] = hfma2_u32((wB & 0x00f000f0u) | k1024, mHB, nHB);
      a[2] = hfma2_u32((vA & 0x00f000f0u) | k1024, mHA, nHA);
      a[3] = hfma2_u32((vB & 0x00f000f0u) | k1024, mHB, nHB);
      b = x.fragment(i + 1, 0);
      mma_16816(acc[2 + (j & 1)], a, b.x, b.y);
      if (XSPLIT == 2)
        mma_16816(acc[2 + (j & 1)], a, b.z, b.w);
    }
  }
  // min term: sum_j m_j * (sum of the activations of sub-block j); k 0..7 carry the hi half of the sums,
  // k 8..15 the lo half, against the same mins.
  float accm[4] = {0.f, 0.f, 0.f, 0.f};
  {
    const uint32_t wordA = (t & 2) ? mnA[1] : mnA[0], wordB = (t & 2) ? mnB[1] : mnB[0];
    const uint32_t pA2 = (wordA >> ((t & 1) * 16)) & 0xffffu, pB2 = (wordB >> ((t & 1) * 16)) & 0xffffu;
    uint32_t a[4];
    a[0] = a[2] = hsub2_u32(__byte_perm(pA2, 0x64u, 0x4140), k1024);
    a[1] = a[3] = hsub2_u32(__byte_perm(pB2, 0x64u, 0x4140), k1024);
    mma_16816(accm, a, x.minSums.x, x.minSums.y);
  }
  const float2 xs = x.powers;
  const float2 dA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x)), dB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
  total[0] += xs.x * (dA.x * ((acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0])) - dA.y * accm[0]);
  total[1] += xs.y * (dA.x * ((acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1])) - dA.y * accm[1]);
  total[2] += xs.x * (dB.x * ((acc[0][2] + acc[1][2]) + (acc[2][2] + acc[3][2])) - dB.y * accm[2]);
  total[3] += xs.y * (dB.x * ((acc[0][3] + acc[1][3]) + (acc[2][3] + acc[3][3])) - dB.y * accm[3]);
}

template <class Q, int NMAT, int XSPLIT, int HALVES>
__global__ void __launch_bounds__(Layout<Q, NMAT, XSPLIT, HALVES>::kThreads, 1) gemv_kernel(const __grid_constant__ GemvParams p) {
  using L = Layout<Q, NMAT, XSPLIT, HALVES>;
  constexpr int kConsumerWarps = L::kConsumers, kFinisherWarps = L::kFinishers, kProducerWarp = L::kProducer, kChunkBlocks = L::kChunkBlocks, kStages = L::kStages;
  extern __shared__ __align__(128) uint8_t smemRaw[];
  RingControl& ctl = *reinterpret_cast<RingControl*>(smemRaw);
  uint2* low = reinterpret_cast<uint2*>(smemRaw + kRingControlBytes);
  float* partial = reinterpret_cast<float*>(smemRaw + kRingControlBytes + L::kLowBytes);
  uint8_t* ring = reinterpret_cast<uint8_t*>(partial + kFinisherWarps * NMAT * kConsumerWarps * 128);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int blocksPerRow = p.k / 256;
  const int chunks = (blocksPerRow + kChunkBlocks - 1) / kChunkBlocks;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], kStageWarps);
    }
    for (int b = 0; b < kFinisherWarps; ++b) {
      mbar_init(&ctl.partialReady[b], kConsumerWarps);
      mbar_init(&ctl.partialFree[b], 1);
    }
    ctl.abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();
  volatile int* abortFlag = &ctl.abort;
  auto give_up = [&] {
    *abortFlag = 1;
    atomicExch(p.status, kStatusBarrierTimeout);
  };

  if (warp == kProducerWarp) {
    // ---- producer: stream weight slabs into the ring (they do not depend on the kernels before this one) ----
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int chunk = 0; chunk < chunks && ok; ++chunk) {
        const int chunkBlocks = min(kChunkBlocks, blocksPerRow - chunk * kChunkBlocks);
        const int groups = (chunkBlocks + kStageBlocks - 1) / kStageBlocks;
        for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
          const int segment = find_segment(p, tile);
          const int row0 = (tile - p.seg[segment].tile0) * kTileRows;
          for (int mat = 0; mat < NMAT && ok; ++mat)
            for (int grp = 0; grp < groups; ++grp, ++it) {
              const uint32_t slot = it % kStages, round = it / kStages;
              if (round > 0 && !mbar_wait_bounded(&ctl.empty[slot], (round - 1) & 1, abortFlag)) {
                give_up();
                ok = false;
                break;
              }
              // One tiled copy moves the whole 16-row x 8-super-block slab; columns past the end of a row are zero-filled
              // and still counted, so the transaction size is always the full box.
              mbar_arrive_expect_tx(&ctl.full[slot], uint32_t(stage_bytes<Q>()));
#pragma unroll
              for (int box = 0; box < Q::kBoxes; ++box)
                tma_load_2d(ring + size_t(slot) * stage_bytes<Q>() + box * box_bytes<Q>(), &p.map[segment][mat],
                            ((chunk * (kChunkBlocks / kStageBlocks) + grp) * Q::kBoxes + box) * (box_blocks<Q>() * Q::kBlockBytes / 8), row0, &ctl.full[slot]);
            }
        }
      }
      // no copy may be in flight when the CTA ends, whoever gave up
      for (uint32_t i = it > uint32_t(kStages) ? it - kStages : 0; i < it; ++i)
        mbar_wait_bounded(&ctl.full[i % kStages], (i / kStages) & 1, abortFlag);
    }
    __syncwarp();
    pdl_wait();  // every thread of every kernel waits, so completion stays transitive along the stream
    return;
  }
  pdl_wait();  // the activations come from the kernels before this one
  if (warp >= kConsumerWarps) {
    finish_tiles<NMAT, kConsumerWarps, kFinisherWarps>(p, ctl, partial, warp - kConsumerWarps, chunks, lane);
    return;
  }

  // ---- consumers ----
  // The super-block of a warp in its half's slabs: of Q6_K each scheduler has as many of one parity as of the other.
  const int g = lane >> 2, t = lane & 3, half = warp / kStageWarps, unit = std::is_same_v<Q, Q6K> ? (warp % kStageWarps) ^ (warp >> 2 & 1) : warp % kStageWarps;
  static_assert(row_pitch<Q>() % 4 == 0 && Q::kBlockBytes * 2 % 4 == 0 && box_blocks<Q>() % 2 == 0, "blocks of even number lie at words");
  const uint8_t* const blocks = ring + (unit / box_blocks<Q>()) * box_bytes<Q>() + (unit % box_blocks<Q>()) * Q::kBlockBytes + g * row_pitch<Q>();
  uint32_t it = 0, mine = half, slot = half, phase = 0;
  uint32_t bufferState = 0;  // bit b: parity of the next use of partial-sum buffer b; bit 4 + b: it has been used before
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int chunkBlocks = min(kChunkBlocks, blocksPerRow - chunk * kChunkBlocks);
    const int groups = (chunkBlocks + kStageBlocks - 1) / kStageBlocks;
    // With two slabs per tile the stages of a tile alternate between the halves (a chunk starts at an even stage, only the last
    // chunk of a row can be a single slab), with one slab every stage is slab 0: this warp meets the same super-block in every tile.
    const int myBlock = (groups == 2 ? half * kStageBlocks : 0) + unit;
    const bool live = myBlock < chunkBlocks;
    OwnRows<XSPLIT> rows;
    rows.low = low + warp * 16 * 32 + lane;
    if (live)
      load_rows<Q, XSPLIT>(rows, p.x + size_t(chunk * kChunkBlocks + myBlock) * 256, p.ldx, p.m, lane);
    int buffer = 0;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, buffer = buffer == kFinisherWarps - 1 ? 0 : buffer + 1) {
      float total[NMAT][1][4];
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat)
        clear(total[mat]);
      // `mine` is the next stage of this half (they are the stages congruent to `half` modulo HALVES), `slot` and `phase`
      // its place in the ring.
      const int perTile = NMAT * groups;
      for (; mine < it + perTile; mine += HALVES, slot += HALVES) {
        if (slot >= kStages) {
          slot -= kStages;
          phase ^= 1;
        }
        if (!mbar_wait_bounded(&ctl.full[slot], phase, abortFlag)) {  // also leaves when another role raised the abort flag
          give_up();
          break;
        }
        if (live) {
          const uint8_t *pA = blocks + slot * stage_bytes<Q>(), *pB = pA + 8 * row_pitch<Q>();
          float sum[1][4];
          clear(sum);
          if constexpr (std::is_same_v<Q, Q4K>) {
            q4k_unit<XSPLIT>(smem_u32(pA), smem_u32(pB), t, rows, sum[0]);
          } else if constexpr (std::is_same_v<Q, Q5K>) {
            q5k_unit(pA, pB, lane, rows, sum);
          } else if constexpr (std::is_same_v<Q, Q8>) {
            q8_unit(pA, pB, lane, rows, sum);
          } else if constexpr (std::is_same_v<Q, IQ4>) {
            iq4_unit(pA, pB, lane, rows, sum);
          } else {
            // Every second super-block of a row lies at a multiple of four bytes and is read by whole words: 48 of 634 instructions less (output head
            // 203.5 -> 192.7 us). The others by words that are put together from two: 225 us.
            if (unit & 1)
              q6k_unit<false>(pA, pB, lane, rows, sum);
            else
              q6k_unit<true>(pA, pB, lane, rows, sum);
          }
          // a branch: chosen by a run-time index the sums would live in local memory
          if (NMAT == 2 && int(mine - it) >= groups) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              total[NMAT - 1][0][i] += sum[0][i];
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              total[0][0][i] += sum[0][i];
          }
        }
        __syncwarp();
        if (lane == 0)
          mbar_arrive(&ctl.empty[slot]);
      }
      it += perTile;
      // Hand the partial sums of the K split to the buffer's finisher, which adds them in the order of the super-blocks, and go on with the next tile.
      const uint32_t parity = (bufferState >> buffer) & 1u;
      if (((bufferState >> (4 + buffer)) & 1u) && !mbar_wait_bounded(&ctl.partialFree[buffer], parity ^ 1u, abortFlag))
        give_up();
      bufferState = (bufferState ^ (1u << buffer)) | (16u << buffer);
      float* sums = partial + size_t(buffer) * NMAT * kConsumerWarps * 128;
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat)
        reinterpret_cast<float4*>(sums + (mat * kConsumerWarps + half * kStageWarps + unit) * 128)[lane] = make_float4(total[mat][0][0], total[mat][0][1], total[mat][0][2], total[mat][0][3]);
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&ctl.partialReady[buffer]);
    }
  }
}

template <class Q, int NMAT, int XSPLIT, int HALVES> cudaError_t launch_halves(const GemvParams& p, int sms, cudaStream_t stream) {
  using L = Layout<Q, NMAT, XSPLIT, HALVES>;
  static PerDeviceOnce configured;
  if (cudaError_t e = configure_shared_memory(gemv_kernel<Q, NMAT, XSPLIT, HALVES>, L::kBytes, configured))
    return e;
  const int grid = p.tiles < sms ? p.tiles : sms;
  launch_kernel<1>(gemv_kernel<Q, NMAT, XSPLIT, HALVES>, grid, L::kThreads, L::kBytes, stream, p);
  return cudaGetLastError();
}
// Rows of one slab leave the second half nothing but a second conversion of the same activations, which holds the first one up: 2048 x 2048 with
// one row, one half / two: Q5_K 3.0 / 4.1 us, Q6_K 2.9 / 3.8, Q8_0 2.9 / 3.6, IQ4_XS 3.3 / 4.0; 8192 x 2048 with eight 7.0 / 8.2, 7.3 / 8.2, 7.1 / 8.1, 8.0 / 8.6.
template <class Q, int NMAT, int XSPLIT> cudaError_t launch(const GemvParams& p, int sms, cudaStream_t stream) {
  return p.k <= kStageBlocks * 256 ? launch_halves<Q, NMAT, XSPLIT, 1>(p, sms, stream) : launch_halves<Q, NMAT, XSPLIT, 2>(p, sms, stream);
}

}  // namespace

GemvBox gemv_box(int type) {
  switch (type) {
    case 8: return {Q8::kBlockBytes, box_blocks<Q8>(), Q8::kPad};
    case 12: return {Q4K::kBlockBytes, box_blocks<Q4K>(), Q4K::kPad};
    case 13: return {Q5K::kBlockBytes, box_blocks<Q5K>(), Q5K::kPad};
    case 14: return {Q6K::kBlockBytes, box_blocks<Q6K>(), Q6K::kPad};
    case 23: return {IQ4::kBlockBytes, box_blocks<IQ4>(), IQ4::kPad};
    default: return {0, 0, 0};
  }
}

// type: ggml type id; pair: gate/up fusion (two matrices, silu(a)*b epilogue). Only Q4_K and Q6_K may drop the low half of
// the activations (xsplit 1).
cudaError_t gemv_launch(int type, bool pair, int xsplit, const GemvParams& p, int sms, cudaStream_t stream) {
  switch (type) {
    case 8: return pair ? launch<Q8, 2, 2>(p, sms, stream) : launch<Q8, 1, 2>(p, sms, stream);
    case 12:
      if (pair)
        return xsplit == 2 ? launch<Q4K, 2, 2>(p, sms, stream) : launch<Q4K, 2, 1>(p, sms, stream);
      return xsplit == 2 ? launch<Q4K, 1, 2>(p, sms, stream) : launch<Q4K, 1, 1>(p, sms, stream);
    case 13: return pair ? launch<Q5K, 2, 2>(p, sms, stream) : launch<Q5K, 1, 2>(p, sms, stream);
    case 14:
      if (pair)
        break;
      return xsplit == 2 ? launch<Q6K, 1, 2>(p, sms, stream) : launch<Q6K, 1, 1>(p, sms, stream);
    case 23: return pair ? launch<IQ4, 2, 2>(p, sms, stream) : launch<IQ4, 1, 2>(p, sms, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace infdev
