// Dequant-fused fp16 tensor-core GEMV for decode (M <= 8 activation rows) over GGUF Q4_K / Q5_K / Q6_K / Q8_0 / IQ4_XS
// weights. It serves every Q6_K matrix (lm_head), the Q5_K, Q8_0 and IQ4_XS ones whose shape it takes (formats.cu has the
// rest) and, when the integer kernel of q4k_decode.cu is switched off, the Q4_K ones.
//
// Replaces linear_decode_q4_k[_add] (quant_linear.metal:245-327), linear_decode_q5_k / q6_k / q8_0[_add] (:329-570) and
// mlp_gate_up of Q4_K, Q5_K and IQ4_XS (fused_kernels.metal:11-200). The reference re-reads the weights once per
// activation row (grid.y = rows); here up to 8 rows share one pass over the weights.
//
// Design (one persistent CTA per SM, 8 consumer warps + 1 producer warp):
//  * The weight matrix is a contiguous byte stream (row n = K/256 super-blocks). The producer warp moves
//    16-row x 8-super-block slabs into a shared-memory ring with one tiled TMA copy each (a tensor map over
//    the packed rows as 8-byte elements) that completes on an mbarrier; nothing else touches HBM for the weights.
//  * At 8 rows the fp32 FMA pipe cannot keep up with HBM (8 FMAs per 4-bit weight), so the products run
//    on the tensor cores as m16n8k16: A = 16 weight rows x 16 k, B = 16 k x 8 activation rows.
//    The summation index of an MMA is a dummy, so k is permuted freely to suit the packed layout; the
//    activations are staged once per CTA in shared memory already in B-fragment order under the same
//    permutation.
//  * Q4_K: A holds the exact integers sc*q (<= 945, exact in fp16); the super-block scale d is applied to
//    the fp32 accumulator after each super-block, and the -dmin*m term is one more MMA against the
//    per-sub-block activation sums. Q6_K: A holds q-32 exactly and the per-16 scale d*sc is applied to
//    the accumulator after each MMA (one MMA = one scale group).
//  * Activations are split x = hi + lo into two fp16 fragments (XSPLIT = 2) so the result keeps fp32
//    accuracy; XSPLIT = 1 drops lo (relative error ~3e-4, still inside the 1e-3 contract).
//  * Every mbarrier wait is bounded; on a timeout the kernel raises an abort flag, records a status code
//    and all roles leave their loops.
#include <type_traits>
#include "gemv_units.cuh"
#include "kernels.h"

namespace infdev {
namespace {

constexpr int kConsumerWarps = 8;   // one warp per super-block of a stage
constexpr int kThreads = (kConsumerWarps + 1) * kWarp;
constexpr int kChunkBlocks = 16;   // super-blocks of K staged per pass (4096 values)
constexpr int kStageBlocks = kGemvStageBlocks;  // super-blocks per ring stage (one per consumer warp)
constexpr int kMaxStages = 8;
constexpr int kTileRows = kGemvTileRows;

// How a block type lies in a ring stage: kBoxes tiled copies of 16 rows x kStageBlocks / kBoxes super-blocks (a box is at
// most 256 elements of 8 bytes wide, which eight super-blocks of Q8_0 exceed), each row kPad bytes wider than its
// super-blocks where the pitch would otherwise put the eight rows of a warp-wide load into the same banks.
struct Q4K {
  static constexpr int kBlockBytes = 144, kBoxes = 1, kPad = 0;
  static constexpr bool kMinTerm = true, kRotated = true;
};
struct Q5K {
  static constexpr int kBlockBytes = 176, kBoxes = 1, kPad = 16;  // pitch 1424 = 16 mod 128
  static constexpr bool kMinTerm = true, kRotated = false;
};
struct Q6K {
  static constexpr int kBlockBytes = 210, kBoxes = 1, kPad = 0;  // pitch 1680 = 16 mod 128
  static constexpr bool kMinTerm = false, kRotated = false;
};
struct Q8 {
  static constexpr int kBlockBytes = 272, kBoxes = 2, kPad = 16;  // eight Q8_0 blocks; pitch 1104 = 80 mod 128
  static constexpr bool kMinTerm = false, kRotated = false;
};
struct IQ4 {
  static constexpr int kBlockBytes = 136, kBoxes = 1, kPad = 16;  // pitch 1104
  static constexpr bool kMinTerm = false, kRotated = false;
};
template <class Q> constexpr int box_blocks() { return kStageBlocks / Q::kBoxes; }
template <class Q> constexpr int row_pitch() { return box_blocks<Q>() * Q::kBlockBytes + Q::kPad; }
template <class Q> constexpr int box_bytes() { return kTileRows * row_pitch<Q>(); }
template <class Q> constexpr int stage_bytes() { return Q::kBoxes * box_bytes<Q>(); }

struct Smem {
  uint64_t full[kMaxStages], empty[kMaxStages];
  int abort;
};
constexpr int kControlBytes = 256;
static_assert(sizeof(Smem) <= kControlBytes, "control block overlaps the activation fragments");

template <class Q, int NMAT, int XSPLIT> constexpr size_t fixed_bytes() {
  size_t frag = size_t(kChunkBlocks) * 16 * 32 * 8 * XSPLIT;
  size_t sums = Q::kMinTerm ? size_t(kChunkBlocks) * 32 * 8 : 0;
  size_t scales = size_t(kChunkBlocks) * 8 * 4;
  size_t partial = size_t(2) * NMAT * kConsumerWarps * 128 * 4;
  return kControlBytes + frag + sums + scales + partial;
}

// As many ring stages as fit beside the fragments in the 227 KB a CTA may use.
template <class Q, int NMAT, int XSPLIT> constexpr int stage_count() {
  int stages = int((size_t(227) * 1024 - fixed_bytes<Q, NMAT, XSPLIT>()) / stage_bytes<Q>());
  return stages > kMaxStages ? kMaxStages : stages;
}

template <class Q, int NMAT, int XSPLIT> constexpr size_t smem_bytes() {
  return fixed_bytes<Q, NMAT, XSPLIT>() + size_t(stage_count<Q, NMAT, XSPLIT>()) * stage_bytes<Q>();
}

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
__device__ __forceinline__ uint2 lds64(uint32_t address) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(address));
  return v;
}

// All operands are 32-bit shared-memory addresses: pA / pB the super-block of rows g and g+8, xhi / xlo the B
// fragments of this super-block already offset by the lane's rotated slot for j = 0 (slots for j = 1..3 follow from
// `rot`, the byte offsets of the other three rotations), xsum the lane's min-term fragment.
template <int XSPLIT>
__device__ __forceinline__ void q4k_unit(uint32_t pA, uint32_t pB, int t, uint32_t xhi, uint32_t xlo, const int (&rot)[4], uint32_t xsum,
                                         float2 xs, float (&total)[4]) {
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
      const int at = i * 256 + rot[j];         // byte offset of fragment (i, rotated slot): 32 slots x 8 bytes per MMA
      uint32_t a[4];
      // low nibbles: (1024 + q) * sc - 1024 * sc, exact in fp16
      a[0] = hfma2_u32((wA & 0x000f000fu) | k1024, sLA, nLA);
      a[1] = hfma2_u32((wB & 0x000f000fu) | k1024, sLB, nLB);
      a[2] = hfma2_u32((vA & 0x000f000fu) | k1024, sLA, nLA);
      a[3] = hfma2_u32((vB & 0x000f000fu) | k1024, sLB, nLB);
      uint2 b = lds64(xhi + at);
      mma_16816(acc[j & 1], a, b.x, b.y);
      if (XSPLIT == 2) {
        b = lds64(xlo + at);
        mma_16816(acc[j & 1], a, b.x, b.y);
      }
      // high nibbles in place: (1024 + 16 q) * sc/16 - 64 * sc
      a[0] = hfma2_u32((wA & 0x00f000f0u) | k1024, mHA, nHA);
      a[1] = hfma2_u32((wB & 0x00f000f0u) | k1024, mHB, nHB);
      a[2] = hfma2_u32((vA & 0x00f000f0u) | k1024, mHA, nHA);
      a[3] = hfma2_u32((vB & 0x00f000f0u) | k1024, mHB, nHB);
      b = lds64(xhi + at + 256);
      mma_16816(acc[2 + (j & 1)], a, b.x, b.y);
      if (XSPLIT == 2) {
        b = lds64(xlo + at + 256);
        mma_16816(acc[2 + (j & 1)], a, b.x, b.y);
      }
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
    const uint2 b = lds64(xsum);
    mma_16816(accm, a, b.x, b.y);
  }
  const float2 dA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x)), dB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
  total[0] += xs.x * (dA.x * ((acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0])) - dA.y * accm[0]);
  total[1] += xs.y * (dA.x * ((acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1])) - dA.y * accm[1]);
  total[2] += xs.x * (dB.x * ((acc[0][2] + acc[1][2]) + (acc[2][2] + acc[3][2])) - dB.y * accm[2]);
  total[3] += xs.y * (dB.x * ((acc[0][3] + acc[1][3]) + (acc[2][3] + acc[3][3])) - dB.y * accm[3]);
}

// The activations of one super-block as the units of gemv_units.cuh read them: one tile of eight rows, hi and lo fragments apart.
template <int XSPLIT> struct StagedRows {
  const uint2 *hi, *lo;  // fragment 0, this lane's slot
  uint2 minSums;
  float2 powers;
  static constexpr bool kSplit = XSPLIT == 2;
  __device__ __forceinline__ uint4 fragment(int i, int) const {
    const uint2 h = hi[i * 32], l = XSPLIT == 2 ? lo[i * 32] : make_uint2(0u, 0u);
    return make_uint4(h.x, h.y, l.x, l.y);
  }
  __device__ __forceinline__ float2 scales(int) const { return powers; }
  __device__ __forceinline__ uint2 sums(int) const { return minSums; }
};

__device__ __forceinline__ int find_segment(const GemvParams& p, int tile) {
  int s = 0;
  while (s + 1 < p.nseg && tile >= p.seg[s + 1].tile0)
    ++s;
  return s;
}

template <class Q, int NMAT, int XSPLIT> __global__ void __launch_bounds__(kThreads, 1) gemv_kernel(const __grid_constant__ GemvParams p) {
  constexpr int kStages = stage_count<Q, NMAT, XSPLIT>();
  extern __shared__ __align__(128) uint8_t smemRaw[];
  Smem& ctl = *reinterpret_cast<Smem*>(smemRaw);
  uint2* fragHi = reinterpret_cast<uint2*>(smemRaw + kControlBytes);
  uint2* fragLo = fragHi + (XSPLIT == 2 ? kChunkBlocks * 16 * 32 : 0);
  uint2* fragSum = fragHi + kChunkBlocks * 16 * 32 * XSPLIT;
  float* xScale = reinterpret_cast<float*>(fragSum + (Q::kMinTerm ? kChunkBlocks * 32 : 0));  // [super-block][activation row]
  float* partial = xScale + kChunkBlocks * 8;
  uint8_t* ring = reinterpret_cast<uint8_t*>(partial + 2 * NMAT * kConsumerWarps * 128);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blocksPerRow = p.k / 256;
  const size_t rowBytes = size_t(blocksPerRow) * Q::kBlockBytes;
  const int chunks = (blocksPerRow + kChunkBlocks - 1) / kChunkBlocks;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], kConsumerWarps);
    }
    ctl.abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();
  volatile int* abortFlag = &ctl.abort;

  if (warp == kConsumerWarps) {
    // ---- producer: stream weight slabs into the ring (they do not depend on the kernels before this one) ----
    uint32_t it = 0;
    for (int chunk = 0; chunk < chunks && !*abortFlag; ++chunk) {
      const int chunkBlocks = min(kChunkBlocks, blocksPerRow - chunk * kChunkBlocks);
      const int groups = (chunkBlocks + kStageBlocks - 1) / kStageBlocks;
      for (int tile = blockIdx.x; tile < p.tiles && !*abortFlag; tile += gridDim.x) {
        const int segment = find_segment(p, tile);
        const size_t row0 = size_t(tile - p.seg[segment].tile0) * kTileRows;
        for (int mat = 0; mat < NMAT; ++mat) {
          for (int grp = 0; grp < groups; ++grp, ++it) {
            const uint32_t slot = it % kStages, round = it / kStages;
            bool ok = true;
            if (lane == 0 && round > 0)
              ok = mbar_wait_bounded(&ctl.empty[slot], (round - 1) & 1, abortFlag);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) {
              if (lane == 0) {
                *abortFlag = 1;
                atomicExch(p.status, kStatusBarrierTimeout);
              }
              break;
            }
            // One tiled copy moves the whole 16-row x 8-super-block slab; columns past the end of a row are zero-filled
            // and still counted, so the transaction size is always the full box.
            if (lane == 0) {
              mbar_arrive_expect_tx(&ctl.full[slot], uint32_t(stage_bytes<Q>()));
#pragma unroll
              for (int box = 0; box < Q::kBoxes; ++box)
                tma_load_2d(ring + size_t(slot) * stage_bytes<Q>() + box * box_bytes<Q>(), &p.map[segment][mat],
                            ((chunk * (kChunkBlocks / kStageBlocks) + grp) * Q::kBoxes + box) * (box_blocks<Q>() * Q::kBlockBytes / 8), int(row0),
                            &ctl.full[slot]);
            }
            __syncwarp();
          }
        }
      }
    }
    if (lane == 0)  // no copy may be in flight when the CTA ends, whoever gave up
      for (uint32_t i = it > uint32_t(kStages) ? it - kStages : 0; i < it; ++i)
        mbar_wait_bounded(&ctl.full[i % kStages], (i / kStages) & 1, abortFlag);
    __syncwarp();
    pdl_wait();  // every thread of every kernel waits, so completion stays transitive along the stream
    return;
  }

  // ---- consumers ----
  pdl_wait();  // the activations come from the kernels before this one
  const int g = lane >> 2, t = lane & 3;
  // Shared-memory byte addresses of this lane's B fragments: slot rotated by j inside each 32-entry line.
  const int rotation[4] = {0, (((lane + 1) & 31) - lane) * 8, (((lane + 2) & 31) - lane) * 8, (((lane + 3) & 31) - lane) * 8};
  const uint32_t fragHiAddress = smem_u32(fragHi) + lane * 8, fragLoAddress = smem_u32(fragLo) + lane * 8, fragSumAddress = smem_u32(fragSum) + lane * 8;
  uint32_t it = 0;
  int tileCounter = 0;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int chunkBlocks = min(kChunkBlocks, blocksPerRow - chunk * kChunkBlocks);
    const int groups = (chunkBlocks + kStageBlocks - 1) / kStageBlocks;
    const int k0 = chunk * kChunkBlocks * 256;
    // Stage the activations of this K chunk in B-fragment order (hi / lo fp16 split). A warp takes one super-block of all
    // 8 rows at a time, in 64-value spans: lane (row = lane/4, jj = lane%4) loads four float4 of a span at 16*e + 4*jj,
    // so each row contributes whole 64-byte pieces. Q4_K fragments are stored rotated by jj inside their 32-entry line,
    // which makes both these writes and the MMA-time reads conflict-free.
    const int row = lane >> 2, jj = lane & 3;
    // The warp's next super-block is under way while it works on one (Q6_K 4096 x 4096, eight rows: 10.0 -> 9.5 us; volatile, or
    // the compiler moves the loads to where they are used).
    float4 next[4][4];
    auto fetch = [&](int sb) {
      const bool live = row < p.m && sb < chunkBlocks;
      const float* from = p.x + size_t(row) * p.ldx + k0 + 256 * sb + 4 * jj;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float4& to = next[i >> 2][i & 3];
        to = make_float4(0.f, 0.f, 0.f, 0.f);
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t@p ld.global.v4.f32 {%0, %1, %2, %3}, [%5];\n\t}"
                     : "+f"(to.x), "+f"(to.y), "+f"(to.z), "+f"(to.w)
                     : "r"(uint32_t(live)), "l"(from + 16 * i));
      }
    };
    fetch(warp);
    for (int sb = warp; sb < chunkBlocks; sb += kConsumerWarps) {
      float4 v[4][4];
      float largest = 0.f;
#pragma unroll
      for (int tq = 0; tq < 4; ++tq)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[tq][e] = next[tq][e];
          largest = fmaxf(fmaxf(fmaxf(largest, fabsf(v[tq][e].x)), fmaxf(fabsf(v[tq][e].y), fabsf(v[tq][e].z))), fabsf(v[tq][e].w));
        }
      fetch(sb + kConsumerWarps);
      largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
      largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 2));
      const float2 power = activation_power(largest);
      if (jj == 0)
        xScale[sb * 8 + row] = largest != INFINITY ? power.y : INFINITY;
      auto store = [&](int tq, const float4 (&span)[4]) {  // four scaled float4 of a 64-value span
        float s[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 w = span[e];
          uint2 hi;
          float4 r;
          int slot;
          if (Q::kRotated) {  // A pairs bytes (0,2) and (1,3) of a quant word
            const int c = 2 * tq + (e & 1), i = ((c >> 2) * 4 + jj) * 2 + (e >> 1);
            slot = (sb * 16 + i) * 32 + ((row * 4 + (c & 3) + jj) & 31);
            hi.x = pack_half2(w.x, w.z);
            hi.y = pack_half2(w.y, w.w);
            const float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&hi.x)), f1 = __half22float2(*reinterpret_cast<__half2*>(&hi.y));
            r = make_float4(w.x - f0.x, w.z - f0.y, w.y - f1.x, w.w - f1.y);
          } else {
            slot = (sb * 16 + tq * 4 + e) * 32 + lane;
            hi.x = pack_half2(w.x, w.y);
            hi.y = pack_half2(w.z, w.w);
            const float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&hi.x)), f1 = __half22float2(*reinterpret_cast<__half2*>(&hi.y));
            r = make_float4(w.x - f0.x, w.y - f0.y, w.z - f1.x, w.w - f1.y);
          }
          fragHi[slot] = hi;
          if (XSPLIT == 2)
            fragLo[slot] = make_uint2(pack_half2(r.x, r.y), pack_half2(r.z, r.w));
          if (Q::kMinTerm)  // sums of the two 32-value sub-blocks of this span, for the min term
            s[e] = (w.x + w.y) + (w.z + w.w);
        }
        if (Q::kMinTerm) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[e] += __shfl_xor_sync(0xffffffffu, s[e], 1);
            s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
          }
          const float s0 = s[0] + s[1], s1 = s[2] + s[3];
          if (jj == 0) {
            const uint32_t hi = pack_half2(s0, s1);
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
            fragSum[sb * 32 + row * 4 + tq] = make_uint2(hi, pack_half2(s0 - f.x, s1 - f.y));
          }
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
            span[e] = scaled_with_infinities(row < p.m ? *reinterpret_cast<const float4*>(p.x + size_t(row) * p.ldx + k0 + 256 * sb + 64 * tq + 16 * e + 4 * jj)
                                                       : make_float4(0.f, 0.f, 0.f, 0.f),
                                             largest, power.x);
          store(tq, span);
        }
      }
    }
    named_barrier(1, kConsumerWarps * kWarp);

    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, ++tileCounter) {
      // Where this thread's element of the tile goes and what is added to it (the residual, or the sum over the earlier
      // K chunks), looked up and fetched before the arithmetic: the parameter block is reached through a generic address
      // (the segment is a run-time index), and a chain of such reads after the reduction would delay every tile.
      float* destination = nullptr;
      float addend = 0.f;
      if (tid < 128 && (tid >> 4) < p.m) {
        const GemvSeg& seg = p.nseg == 1 ? p.seg[0] : p.seg[find_segment(p, tile)];
        const size_t at = size_t(tid >> 4) * seg.ldy + size_t(tile - seg.tile0) * kTileRows + (tid & 15);
        destination = seg.y + at;
        if (NMAT == 1 && chunk > 0)
          addend = *destination;
        else if (NMAT == 1 && seg.res)
          addend = seg.res[at];
      }
      float total[NMAT][1][4];
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat)
        clear(total[mat]);
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat)
        for (int grp = 0; grp < groups; ++grp, ++it) {
          const uint32_t slot = it % kStages, round = it / kStages;
          if (*abortFlag)
            continue;
          if (!mbar_wait_bounded(&ctl.full[slot], round & 1, abortFlag)) {
            *abortFlag = 1;
            atomicExch(p.status, kStatusBarrierTimeout);
            continue;
          }
          const int count = min(kStageBlocks, chunkBlocks - grp * kStageBlocks);
          if (warp < count) {
            const uint8_t* base = ring + size_t(slot) * stage_bytes<Q>() + (warp / box_blocks<Q>()) * box_bytes<Q>() + (warp % box_blocks<Q>()) * Q::kBlockBytes;
            const uint8_t *pA = base + g * row_pitch<Q>(), *pB = base + (g + 8) * row_pitch<Q>();
            const int sb = grp * kStageBlocks + warp;
            const float2 xs = *reinterpret_cast<const float2*>(xScale + sb * 8 + 2 * t);
            StagedRows<XSPLIT> rows{fragHi + sb * 512 + lane, fragLo + sb * 512 + lane, make_uint2(0u, 0u), xs};
            if constexpr (std::is_same_v<Q, Q4K>) {
              q4k_unit<XSPLIT>(smem_u32(pA), smem_u32(pB), t, fragHiAddress + sb * 4096, fragLoAddress + sb * 4096, rotation, fragSumAddress + sb * 256, xs,
                               total[mat][0]);
            } else if constexpr (std::is_same_v<Q, Q5K>) {
              rows.minSums = fragSum[sb * 32 + lane];
              q5k_unit(pA, pB, lane, rows, total[mat]);
            } else if constexpr (std::is_same_v<Q, Q8>) {
              q8_unit(pA, pB, lane, rows, total[mat]);
            } else if constexpr (std::is_same_v<Q, IQ4>) {
              iq4_unit(pA, pB, lane, rows, total[mat]);
            } else {
              q6k_unit(pA, pB, lane, rows, total[mat]);
            }
          }
          __syncwarp();
          if (lane == 0)
            mbar_arrive(&ctl.empty[slot]);
        }
      // Cross-warp reduction of the K split, then the epilogue.
      float* mine = partial + size_t(tileCounter & 1) * NMAT * kConsumerWarps * 128;
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat) {
        float* dst = mine + (mat * kConsumerWarps + warp) * 128;
        dst[(2 * t) * 16 + g] = total[mat][0][0];
        dst[(2 * t + 1) * 16 + g] = total[mat][0][1];
        dst[(2 * t) * 16 + g + 8] = total[mat][0][2];
        dst[(2 * t + 1) * 16 + g + 8] = total[mat][0][3];
      }
      named_barrier(1, kConsumerWarps * kWarp);
      if (tid < 128) {
        float sum[NMAT];
#pragma unroll
        for (int mat = 0; mat < NMAT; ++mat) {
          sum[mat] = 0.f;
#pragma unroll
          for (int w = 0; w < kConsumerWarps; ++w)
            sum[mat] += mine[(mat * kConsumerWarps + w) * 128 + tid];
        }
        if (destination)
          *destination = NMAT == 2 ? silu_f(sum[0]) * sum[NMAT - 1] : sum[0] + addend;
      }
    }
  }
}

template <class Q, int NMAT, int XSPLIT> cudaError_t launch(const GemvParams& p, int sms, cudaStream_t stream) {
  static PerDeviceOnce configured;
  constexpr size_t bytes = smem_bytes<Q, NMAT, XSPLIT>();
  if (cudaError_t e = configure_shared_memory(gemv_kernel<Q, NMAT, XSPLIT>, bytes, configured))
    return e;
  const int grid = p.tiles < sms ? p.tiles : sms;
  launch_kernel<1>(gemv_kernel<Q, NMAT, XSPLIT>, grid, kThreads, bytes, stream, p);
  return cudaGetLastError();
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
