// What the integer Q4_K kernels share: the operand fragments of the activations and the arithmetic of one 16-row x 256-k unit, which
// q4k_decode.cu describes.
#pragma once
#include "act_image.cuh"
#include "kernels.h"

namespace infdev {

constexpr int kQ4BlockBytes = 144;
constexpr int kQ4RowPitch = kGemvStageBlocks * kQ4BlockBytes + kDecodePadBytes;  // 1184
constexpr int kQ4StageBytes = kGemvTileRows * kQ4RowPitch;                       // 18,944

// Ordinary loads (not volatile asm): the compiler may hoist and interleave them with the MMAs, but not move them
// above the mbarrier wait, which clobbers memory.
__device__ __forceinline__ uint4 lds128(const uint8_t* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint2 lds64(const uint8_t* p) { return *reinterpret_cast<const uint2*>(p); }

// D(16x8,s32) += A(16x32,u8,row) * B(32x8,s8 or u8,col)
__device__ __forceinline__ void imma_u8s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma_u8u8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// What one lane keeps of the image of one super-block (act_image.cuh) while its warp walks the tiles. With eight activation
// rows the eight columns of an MMA are the rows. With ROWS = 1 or 2 they are (row, sub-block) pairs: column c stands for
// row c % ROWS and, of every 8 / ROWS consecutive sub-blocks, for sub-block c / ROWS, and the B operand of a sub-block is zero
// in the other columns. The MMAs of 8 / ROWS sub-blocks then share one accumulator, and a sub-block scale multiplies
// every result once instead of leaving columns empty.
// Lane (g = lane/4, t = lane%4) holds, per sub-block j, the B fragments of column g, quarter t: registers b0, b1 of the
// high-byte MMA in x, y and of the low-byte MMA in z, w.
struct Fragments {
  uint4 quant[8];
  uint2 sums;    // min-term fragment: fp16 pairs of S_j / 32, high halves in x, low halves in y
  uint2 scales;  // fp32 bits of the activation scales of the rows of columns 2t and 2t+1
};

template <int ROWS> __device__ __forceinline__ Fragments load_fragments(const uint8_t* block, int lane) {
  constexpr int kShare = 8 / ROWS;
  Fragments f;
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    f.quant[j] = g / ROWS == j % kShare ? *reinterpret_cast<const uint4*>(block + j * 512 + (g % ROWS) * 64 + t * 16) : make_uint4(0, 0, 0, 0);
  f.sums = *reinterpret_cast<const uint2*>(block + kImageSumOffset + lane * 8);
  f.scales = *reinterpret_cast<const uint2*>(block + kImageScaleOffset + (2 * t % ROWS) * 4);
  return f;
}

// rint(v * inv), |v * inv| <= 32768, in the low bits of the result: the sum with 1.5 x 2^23 has an ulp of one.
__device__ __forceinline__ uint32_t level_bits(float v, float inv) { return __float_as_uint(__fadd_rn(__fmul_rn(v, inv), 12582912.f)); }

// The same from fp32 activations: what image_store_block writes of this super-block and load_fragments reads, bit for bit, without the
// launch between. A lane owns row g % ROWS and, of it, the eight values of quarter t of every sub-block that its column stands for.
//
// With norm.weight the activations are the RMS norm of the row, bit for bit as rms_norm_4096_kernel computes it, for 16 warps that hold
// a row of 4096 between them: a block's squares are summed over the lanes of that kernel's warp, in its order whatever ROWS.
struct RowNorm {
  const float* weight;  // the row's 4096 weights; null: x as it is
  float* normalised;    // [m][4096], where this warp's super-block of the result goes; null: nowhere
  float* squares;       // shared [super-block][row]
  int block;            // the warp's super-block
};

template <int ROWS> __device__ __forceinline__ Fragments quantize_fragments(const float* x, int ldx, int m, int lane, const RowNorm& norm) {
  constexpr int kShare = 8 / ROWS;
  const int g = lane >> 2, t = lane & 3, row = g % ROWS;
  const float* src = x + size_t(row) * ldx + (g / ROWS) * 32 + t * 8;
  float v[ROWS][8];  // of sub-blocks kShare * i + g / ROWS
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (row < m)
      a = *reinterpret_cast<const float4*>(src + i * kShare * 32), b = *reinterpret_cast<const float4*>(src + i * kShare * 32 + 4);
    v[i][0] = a.x, v[i][1] = a.y, v[i][2] = a.z, v[i][3] = a.w, v[i][4] = b.x, v[i][5] = b.y, v[i][6] = b.z, v[i][7] = b.w;
  }
  if (norm.weight) {
    constexpr int kBlocks = kGemvNormK / 256;
    float sum[ROWS];  // of sub-block j, quarter t: lane 4 j + t of the other kernel
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
      sum[i] = square_sum(make_float4(v[i][0], v[i][1], v[i][2], v[i][3]), make_float4(v[i][4], v[i][5], v[i][6], v[i][7]));
    // j = kShare * i + g / ROWS: the bits of i are the upper ones of j
#pragma unroll
    for (int step = ROWS / 2; step; step /= 2)
#pragma unroll
      for (int i = 0; i < step; ++i)
        sum[i] += sum[i + step];
#pragma unroll
    for (int lanes = 16; lanes; lanes /= 2)
      if (lanes < 4 || lanes >= 4 * ROWS)
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], lanes);
    if (t == 0 && g < ROWS)
      norm.squares[norm.block * kImageRows + g] = sum[0];
    named_barrier(1, kBlocks * kWarp);
    float total = 0.f;
#pragma unroll
    for (int b = 0; b < kBlocks; ++b)
      total += norm.squares[b * kImageRows + row];
    const float scale = rsqrtf(total / float(kGemvNormK) + 1.0e-6f);
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int at = norm.block * 256 + (kShare * i + g / ROWS) * 32 + t * 8;
      const float4 a = *reinterpret_cast<const float4*>(norm.weight + at), b = *reinterpret_cast<const float4*>(norm.weight + at + 4);
      v[i][0] = v[i][0] * scale * a.x, v[i][1] = v[i][1] * scale * a.y, v[i][2] = v[i][2] * scale * a.z, v[i][3] = v[i][3] * scale * a.w;
      v[i][4] = v[i][4] * scale * b.x, v[i][5] = v[i][5] * scale * b.y, v[i][6] = v[i][6] * scale * b.z, v[i][7] = v[i][7] * scale * b.w;
      if (norm.normalised && row < m) {
        float4* to = reinterpret_cast<float4*>(norm.normalised + size_t(row) * kGemvNormK + at);
        to[0] = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]), to[1] = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
      }
    }
  }
  float amax = 0.f, finite = 0.f;
#pragma unroll
  for (int i = 0; i < ROWS; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e)
      amax = fmaxf(amax, fabsf(v[i][e])), finite = fmaf(v[i][e], 0.f, finite);
#pragma unroll
  for (int lanes = 1; lanes < 32; lanes *= 2)
    if (lanes < 4 || lanes >= 4 * ROWS)
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, lanes));
  const float xs = amax / kImageLevels;
  float inv = amax > 0.f ? kImageLevels / amax : 0.f;
  if (__any_sync(0xffffffffu, !(finite == 0.f) || inv == INFINITY)) {  // the levels themselves; of NaN, or infinity times zero, zero
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float level = __fmul_rn(v[i][e], inv);
        v[i][e] = level == level ? fminf(fmaxf(level, -kImageLevels), kImageLevels) : 0.f;
      }
    inv = 1.f;
  }
  uint4 quant[ROWS];
  int sum[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    uint32_t q[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
      q[e] = level_bits(v[i][e], inv);
    const uint32_t low01 = __byte_perm(q[0], q[1], 0x5140), low23 = __byte_perm(q[2], q[3], 0x5140);  // lo, lo, hi, hi of two values
    const uint32_t low45 = __byte_perm(q[4], q[5], 0x5140), low67 = __byte_perm(q[6], q[7], 0x5140);
    quant[i].x = __byte_perm(low01, low23, 0x7632), quant[i].y = __byte_perm(low45, low67, 0x7632);
    quant[i].z = __byte_perm(low01, low23, 0x5410), quant[i].w = __byte_perm(low45, low67, 0x5410);
    sum[i] = 256 * __dp4a(int(quant[i].x), 0x01010101, __dp4a(int(quant[i].y), 0x01010101, 0)) +
             int(__dp4a(quant[i].z, 0x01010101u, __dp4a(quant[i].w, 0x01010101u, 0u)));
  }
  Fragments f;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    f.quant[j] = g / ROWS == j % kShare ? quant[j / kShare] : make_uint4(0, 0, 0, 0);
  // S_2t and S_2t+1 of row g for lane (g, t); with fewer than eight rows the columns from ROWS on are not used
  int even, odd;
  if (ROWS == 8) {  // each step halves the sub-blocks a lane still sums for
    int part[4], half[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int other = __shfl_xor_sync(0xffffffffu, t & 2 ? sum[i] : sum[(4 + i) % ROWS], 2);
      part[i] = (t & 2 ? sum[(4 + i) % ROWS] : sum[i]) + other;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int other = __shfl_xor_sync(0xffffffffu, t & 1 ? part[i] : part[2 + i], 1);
      half[i] = (t & 1 ? part[2 + i] : part[i]) + other;
    }
    even = half[0], odd = half[1];
  } else {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 1);
      sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 2);  // of sub-block kShare * i + g / ROWS of row g % ROWS
    }
    const int from = 2 * t % kShare * ROWS + row;  // the g that holds sub-block 2t; ROWS further on the one with 2t + 1
    const int low[2] = {__shfl_sync(0xffffffffu, sum[0], from * 4), __shfl_sync(0xffffffffu, sum[0], (from + ROWS) * 4)};
    const int high[2] = {__shfl_sync(0xffffffffu, sum[ROWS - 1], from * 4), __shfl_sync(0xffffffffu, sum[ROWS - 1], (from + ROWS) * 4)};
    const bool second = 2 * t >= kShare;
    even = second ? high[0] : low[0], odd = second ? high[1] : low[1];
  }
  const float s0 = float(even) * 0.03125f, s1 = float(odd) * 0.03125f;
  f.sums.x = pack_half2(s0, s1);
  const float2 rounded = __half22float2(*reinterpret_cast<const __half2*>(&f.sums.x));
  f.sums.y = pack_half2(s0 - rounded.x, s1 - rounded.y);
  f.scales.x = __float_as_uint(__shfl_sync(0xffffffffu, xs, (2 * t % ROWS) * 4));
  f.scales.y = __float_as_uint(__shfl_sync(0xffffffffu, xs, ((2 * t + 1) % ROWS) * 4));
  return f;
}

// One 16-row x 256-k unit. Lane (g, t) owns weight rows g and g+8 (shared-memory addresses pA, pB) and, in each
// 32-byte quant chunk c, bytes 8t .. 8t+7: their low nibbles are values 8t .. 8t+7 of sub-block 2c, their high
// nibbles the same values of sub-block 2c+1 (GGUF layout as read by dequant_tile, quant_linear.metal:39-46). The four
// bytes of a word fill four consecutive summation slots of the MMA, which is the order the image stores the
// activations in.
// The integer sums are exact, and with fewer than eight rows they are completed over the lanes of a row before they are
// rounded to fp32, so that a row has the same bits whatever ROWS. Only lanes with 2t < ROWS then hold results.
template <int ROWS> __device__ __forceinline__ void q4k_unit(const uint8_t* pA, const uint8_t* pB, int t, const Fragments& f, float (&total)[4]) {
  static_assert(ROWS == 1 || ROWS == 2 || ROWS == 8, "scale selection");
  constexpr int kShare = 8 / ROWS;
  const uint4 hA = lds128(pA), hB = lds128(pB);
  // 6-bit scales / mins of the 8 sub-blocks, four per word (scale_min_k4, quant_linear.metal:12-20).
  const uint32_t scA[2] = {hA.y & 0x3f3f3f3fu, (hA.w & 0x0f0f0f0fu) | ((hA.y >> 2) & 0x30303030u)};
  const uint32_t mnA[2] = {hA.z & 0x3f3f3f3fu, ((hA.w >> 4) & 0x0f0f0f0fu) | ((hA.z >> 2) & 0x30303030u)};
  const uint32_t scB[2] = {hB.y & 0x3f3f3f3fu, (hB.w & 0x0f0f0f0fu) | ((hB.y >> 2) & 0x30303030u)};
  const uint32_t mnB[2] = {hB.z & 0x3f3f3f3fu, ((hB.w >> 4) & 0x0f0f0f0fu) | ((hB.z >> 2) & 0x30303030u)};
  // 16 x the sum over the 8 sub-blocks of scale * (integer dot product), separately for the low and the high activation
  // byte: |low| <= 16 * 8 * 63 * 15 * 32 * 255 < 2^30 and |high| <= 16 * 8 * 63 * 15 * 32 * 128 both stay inside int32.
  int sumLow[4] = {0, 0, 0, 0}, sumHigh[4] = {0, 0, 0, 0};
  int high[4], low[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint2 qA = lds64(pA + 16 + 32 * c + 8 * t), qB = lds64(pB + 16 + 32 * c + 8 * t);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 2 * c + h, set = ROWS == 2 ? j / kShare : 0;
      uint32_t a[4];
      // Low nibbles as they are, high nibbles in place as 16 q (still a byte); the sub-block scale of the low ones is
      // taken 16-fold instead, and the common factor leaves with d at the end.
      const uint32_t mask = h == 0 ? 0x0f0f0f0fu : 0xf0f0f0f0u;
      a[0] = qA.x & mask, a[1] = qB.x & mask, a[2] = qA.y & mask, a[3] = qB.y & mask;
      const uint4 b = f.quant[j];
      if (j % kShare == 0)
        high[0] = high[1] = high[2] = high[3] = low[0] = low[1] = low[2] = low[3] = 0;
      imma_u8s8(high, a, b.x, b.y);
      imma_u8u8(low, a, b.z, b.w);
      if (j % kShare != kShare - 1)
        continue;
      if (ROWS == 1) {  // columns 2t and 2t + 1 are the sub-blocks of those numbers
        const uint32_t pairA = (t & 2 ? scA[1] : scA[0]) >> (16 * (t & 1)), pairB = (t & 2 ? scB[1] : scB[0]) >> (16 * (t & 1));
        const int evenA = int(pairA & 0xffu) * 16, oddA = int(pairA >> 8 & 0xffu), evenB = int(pairB & 0xffu) * 16, oddB = int(pairB >> 8 & 0xffu);
        sumLow[0] = evenA * low[0] + oddA * low[1], sumHigh[0] = evenA * high[0] + oddA * high[1];
        sumLow[2] = evenB * low[2] + oddB * low[3], sumHigh[2] = evenB * high[2] + oddB * high[3];
        continue;
      }
      int sA, sB;
      if (ROWS == 8) {
        const int byteA = int(__byte_perm(scA[j >> 2], 0u, 0x4440 + (j & 3))), byteB = int(__byte_perm(scB[j >> 2], 0u, 0x4440 + (j & 3)));
        sA = h == 0 ? byteA * 16 : byteA, sB = h == 0 ? byteB * 16 : byteB;
      } else {  // sub-block 4 * set + t; even ones hold low nibbles
        const int fold = t & 1 ? 0 : 4;
        sA = int(scA[set] >> (8 * t) & 0xffu) << fold, sB = int(scB[set] >> (8 * t) & 0xffu) << fold;
      }
      sumLow[0] += sA * low[0], sumHigh[0] += sA * high[0];
      sumLow[1] += sA * low[1], sumHigh[1] += sA * high[1];
      sumLow[2] += sB * low[2], sumHigh[2] += sB * high[2];
      sumLow[3] += sB * low[3], sumHigh[3] += sB * high[3];
    }
  }
#pragma unroll
  for (int lanes = 1; ROWS < 8 && lanes < 4; lanes *= 2)
#pragma unroll
    for (int i = 0; i < 4; i += ROWS == 1 ? 2 : 1) {
      sumLow[i] += __shfl_xor_sync(0xffffffffu, sumLow[i], lanes);
      sumHigh[i] += __shfl_xor_sync(0xffffffffu, sumHigh[i], lanes);
    }
  // min term: sum_j m_j * S_j / 32; summation slots 0..7 carry the fp16 high halves of the sums, 8..15 the low halves.
  float accm[4] = {0.f, 0.f, 0.f, 0.f};
  {
    constexpr uint32_t k1024 = 0x64006400u;
    const uint32_t wordA = (t & 2) ? mnA[1] : mnA[0], wordB = (t & 2) ? mnB[1] : mnB[0];
    const uint32_t pairA = (wordA >> ((t & 1) * 16)) & 0xffffu, pairB = (wordB >> ((t & 1) * 16)) & 0xffffu;
    uint32_t a[4];
    a[0] = a[2] = hsub2_u32(__byte_perm(pairA, 0x64u, 0x4140), k1024);
    a[1] = a[3] = hsub2_u32(__byte_perm(pairB, 0x64u, 0x4140), k1024);
    mma_16816(accm, a, f.sums.x, f.sums.y);
  }
  const float xs0 = __uint_as_float(f.scales.x), xs1 = __uint_as_float(f.scales.y);
  const float2 dA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x)), dB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
  const float mA = 32.f * dA.y, mB = 32.f * dB.y, sixteenthA = 0.0625f * dA.x, sixteenthB = 0.0625f * dB.x;
  total[0] += xs0 * (sixteenthA * fmaf(float(sumHigh[0]), 256.f, float(sumLow[0])) - mA * accm[0]);
  if (ROWS > 1)
    total[1] += xs1 * (sixteenthA * fmaf(float(sumHigh[1]), 256.f, float(sumLow[1])) - mA * accm[1]);
  total[2] += xs0 * (sixteenthB * fmaf(float(sumHigh[2]), 256.f, float(sumLow[2])) - mB * accm[2]);
  if (ROWS > 1)
    total[3] += xs1 * (sixteenthB * fmaf(float(sumHigh[3]), 256.f, float(sumLow[3])) - mB * accm[3]);
}

}  // namespace infdev
