// One unit (16 weight rows x 256 k) of the block formats whose quants enter the tensor cores as exact fp16 integers and whose
// sub-block scales multiply the fp32 accumulators of an m16n8k16 chain: Q5_K, Q6_K, Q8_0, IQ4_XS. Lane (g = lane / 4,
// t = lane % 4) owns weight rows g and g + 8; pA and pB are their super-blocks in shared memory. `b` holds the activations:
// b.fragment(i, tile) is a lane's B operand of 16 k and tile `tile` (eight rows), the hi half in x and y, the lo half (if
// kSplit) in z and w; b.scales(tile) are the powers of two of the rows 2t and 2t + 1; b.sums(tile) is the fragment of the
// sub-block sums (Q5_K). NT tiles share a decoded fragment. From three tiles on the loops over sub-blocks are unrolled less:
// loads hoisted over a whole unit push registers to local memory, which these kernels' shared-memory carve-out leaves no L1
// for (9 % of the time of Q6_K with 40 rows).
#pragma once
#include "common.cuh"

namespace infdev {

// The power of two that brings a row's largest activation of a super-block into [512, 1024) (exponent field 136; sub-block sums
// then stay below 2^15), and its inverse. Both are normal numbers, whatever the magnitude is: the fields lie in 1 .. 253.
__device__ __forceinline__ float2 activation_power(float largest) {
  const int field = min(253, max(1, 263 - int(__float_as_uint(largest) >> 23)));
  return make_float2(__uint_as_float(uint32_t(field) << 23), __uint_as_float(uint32_t(254 - field) << 23));
}
// Four activations scaled, for a super-block in which some row has an infinite one: in such a row infinite values stand as +-512
// and finite ones as zero, and infinity takes the place of the power's inverse, so that products come out as +-infinity with the
// sign of the weight (the hi + lo halves of an infinity would be infinity - infinity). NaN stays NaN.
__device__ __forceinline__ float4 scaled_with_infinities(const float4& v, float largest, float power) {
  auto scaled = [&](float x) { return largest != INFINITY ? x * power : fabsf(x) == INFINITY ? copysignf(512.f, x) : x * 0.f; };
  return make_float4(scaled(v.x), scaled(v.y), scaled(v.z), scaled(v.w));
}

__device__ __forceinline__ uint32_t lds_u32_unaligned(const uint8_t* p) {
  return uint32_t(*reinterpret_cast<const uint16_t*>(p)) | (uint32_t(*reinterpret_cast<const uint16_t*>(p + 2)) << 16);
}

// Fragment of one MMA from four quant bytes of the rows g and g+8: (base + byte) - base in fp16, base = 1024 + bias, exact.
__device__ __forceinline__ void byte_fragment(uint32_t (&a)[4], uint32_t bytesA, uint32_t bytesB, uint32_t bias2) {
  a[0] = hsub2_u32(__byte_perm(bytesA, 0x64u, 0x4140), bias2);
  a[1] = hsub2_u32(__byte_perm(bytesB, 0x64u, 0x4140), bias2);
  a[2] = hsub2_u32(__byte_perm(bytesA, 0x64u, 0x4342), bias2);
  a[3] = hsub2_u32(__byte_perm(bytesB, 0x64u, 0x4342), bias2);
}
__device__ __forceinline__ void add_scaled(float (&sum)[4], float sA, float sB, const float (&acc)[4]) {
  sum[0] = fmaf(sA, acc[0], sum[0]), sum[1] = fmaf(sA, acc[1], sum[1]), sum[2] = fmaf(sB, acc[2], sum[2]), sum[3] = fmaf(sB, acc[3], sum[3]);
}
// total[tile] += (the powers of two of the tile's activation rows) * sum[tile]
template <int NT, class B> __device__ __forceinline__ void add_totals(float (&total)[NT][4], const B& b, const float (&sum)[NT][4]) {
#pragma unroll
  for (int tile = 0; tile < NT; ++tile) {
    const float2 xs = b.scales(tile);
    total[tile][0] = fmaf(xs.x, sum[tile][0], total[tile][0]), total[tile][1] = fmaf(xs.y, sum[tile][1], total[tile][1]);
    total[tile][2] = fmaf(xs.x, sum[tile][2], total[tile][2]), total[tile][3] = fmaf(xs.y, sum[tile][3], total[tile][3]);
  }
}
template <int NT> __device__ __forceinline__ void clear(float (&sum)[NT][4]) {
#pragma unroll
  for (int tile = 0; tile < NT; ++tile)
    sum[tile][0] = sum[tile][1] = sum[tile][2] = sum[tile][3] = 0.f;
}
// sum[tile] += scale * (the fragments a[0 .. F) times the activations of fragments first .. first + F). The MMAs of one half
// over all tiles come before those of the other, so that no two neighbours depend on each other. LOW_FIRST: the low halves of
// all fragments before the high ones. An accumulator cuts off at its own magnitude with every product that is added, and that
// of the low halves is 2^-11 of the others': half as many cuts. Q5_K needs it, whose values have not been centred yet (K =
// 2048, against fp64: 1.4e-7 with it, 1.85e-7 without, 1.5e-7 for the plain fp32 kernel); the other types are at 1.2e-7 to
// 1.5e-7 without, and it costs 3 to 8 % at 9 to 24 rows.
template <bool LOW_FIRST, int F, int NT, class B>
__device__ __forceinline__ void scaled_products(float (&sum)[NT][4], const uint32_t (&a)[F][4], const B& b, int first, float sA, float sB) {
  float acc[NT][4];
  clear(acc);
  if (LOW_FIRST) {
    uint2 high[F][NT];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int tile = 0; tile < NT; ++tile) {
        const uint4 x = b.fragment(first + f, tile);
        high[f][tile] = make_uint2(x.x, x.y);
        if (B::kSplit)
          mma_16816(acc[tile], a[f], x.z, x.w);
      }
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int tile = 0; tile < NT; ++tile)
        mma_16816(acc[tile], a[f], high[f][tile].x, high[f][tile].y);
  }
#pragma unroll
  for (int f = 0; f < (LOW_FIRST ? 0 : F); ++f) {
    uint4 x[NT];
#pragma unroll
    for (int tile = 0; tile < NT; ++tile)
      x[tile] = b.fragment(first + f, tile);
#pragma unroll
    for (int tile = 0; tile < NT; ++tile)
      mma_16816(acc[tile], a[f], x[tile].x, x[tile].y);
    if (B::kSplit) {
#pragma unroll
      for (int tile = 0; tile < NT; ++tile)
        mma_16816(acc[tile], a[f], x[tile].z, x[tile].w);
    }
  }
#pragma unroll
  for (int tile = 0; tile < NT; ++tile)
    add_scaled(sum[tile], sA, sB, acc[tile]);
}
__device__ __forceinline__ uint32_t lds_u32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ float byte_of(uint32_t word, int i) { return float(__byte_perm(word, 0u, 0x4440 + i)); }

// Q5_K (quant_linear.metal:50-67): fp16 d, dmin | 6-bit scales and mins | qh[32] | qs[128]. Element l of sub-block j has its
// low nibble in qs[32 (j / 2) + l] (high half of the byte when j is odd) and its fifth bit in bit j of qh[l].
template <int NT, class B> __device__ __forceinline__ void q5k_unit(const uint8_t* pA, const uint8_t* pB, int lane, const B& b, float (&total)[NT][4]) {
  const int t = lane & 3;
  const uint4 hA = *reinterpret_cast<const uint4*>(pA), hB = *reinterpret_cast<const uint4*>(pB);
  const uint32_t scA[2] = {hA.y & 0x3f3f3f3fu, (hA.w & 0x0f0f0f0fu) | ((hA.y >> 2) & 0x30303030u)};
  const uint32_t mnA[2] = {hA.z & 0x3f3f3f3fu, ((hA.w >> 4) & 0x0f0f0f0fu) | ((hA.z >> 2) & 0x30303030u)};
  const uint32_t scB[2] = {hB.y & 0x3f3f3f3fu, (hB.w & 0x0f0f0f0fu) | ((hB.y >> 2) & 0x30303030u)};
  const uint32_t mnB[2] = {hB.z & 0x3f3f3f3fu, ((hB.w >> 4) & 0x0f0f0f0fu) | ((hB.z >> 2) & 0x30303030u)};
  constexpr uint32_t k1024 = 0x64006400u;
  uint32_t highA[2], highB[2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
    highA[u] = lds_u32(pA + 16 + 16 * u + 4 * t), highB[u] = lds_u32(pB + 16 + 16 * u + 4 * t);
  float sum[NT][4];
  clear(sum);
#pragma unroll(NT > 2 ? 2 : 4)
  for (int c = 0; c < 4; ++c) {
    uint32_t lowA[2], lowB[2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
      lowA[u] = lds_u32(pA + 48 + 32 * c + 16 * u + 4 * t), lowB[u] = lds_u32(pB + 48 + 32 * c + 16 * u + 4 * t);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 2 * c + h;
      uint32_t a[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t fifthA = (j < 4 ? highA[u] << (4 - j) : highA[u] >> (j - 4)) & 0x10101010u;
        const uint32_t fifthB = (j < 4 ? highB[u] << (4 - j) : highB[u] >> (j - 4)) & 0x10101010u;
        byte_fragment(a[u], ((h ? lowA[u] >> 4 : lowA[u]) & 0x0f0f0f0fu) | fifthA, ((h ? lowB[u] >> 4 : lowB[u]) & 0x0f0f0f0fu) | fifthB, k1024);
      }
      const uint32_t wordA = (c < 2 ? scA[0] : scA[1]) >> (16 * (c & 1)), wordB = (c < 2 ? scB[0] : scB[1]) >> (16 * (c & 1));
      scaled_products<true>(sum, a, b, 2 * j, byte_of(wordA, h), byte_of(wordB, h));
    }
  }
  const float2 dA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x)), dB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
  const uint32_t wordA = (t & 2) ? mnA[1] : mnA[0], wordB = (t & 2) ? mnB[1] : mnB[0];
  const uint32_t pairA = (wordA >> ((t & 1) * 16)) & 0xffffu, pairB = (wordB >> ((t & 1) * 16)) & 0xffffu;
  uint32_t a[4];
  a[0] = a[2] = hsub2_u32(__byte_perm(pairA, 0x64u, 0x4140), k1024);
  a[1] = a[3] = hsub2_u32(__byte_perm(pairB, 0x64u, 0x4140), k1024);
#pragma unroll
  for (int tile = 0; tile < NT; ++tile) {
    float accm[4] = {0.f, 0.f, 0.f, 0.f};
    const uint2 xsum = b.sums(tile);
    mma_16816(accm, a, xsum.x, xsum.y);
    sum[tile][0] = dA.x * sum[tile][0] - dA.y * accm[0], sum[tile][1] = dA.x * sum[tile][1] - dA.y * accm[1];
    sum[tile][2] = dB.x * sum[tile][2] - dB.y * accm[2], sum[tile][3] = dB.x * sum[tile][3] - dB.y * accm[3];
  }
  add_totals(total, b, sum);
}

// Q8_0 (quant_linear.metal:87-97): eight blocks of fp16 d | int8[32] stand for one super-block.
template <int NT, class B> __device__ __forceinline__ void q8_unit(const uint8_t* pA, const uint8_t* pB, int lane, const B& b, float (&total)[NT][4]) {
  const int t = lane & 3;
  constexpr uint32_t k1152 = 0x64806480u;
  float sum[NT][4];
  clear(sum);
#pragma unroll(NT > 4 ? 2 : NT > 2 ? 4 : 8)
  for (int j = 0; j < 8; ++j) {
    uint32_t a[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int at = 34 * j + 2 + 16 * u + 4 * t;  // word-aligned in odd blocks only
      const uint32_t bytesA = (j & 1 ? lds_u32(pA + at) : lds_u32_unaligned(pA + at)) ^ 0x80808080u;
      const uint32_t bytesB = (j & 1 ? lds_u32(pB + at) : lds_u32_unaligned(pB + at)) ^ 0x80808080u;
      byte_fragment(a[u], bytesA, bytesB, k1152);
    }
    scaled_products<false>(sum, a, b, 2 * j, load_half_bits(pA + 34 * j), load_half_bits(pB + 34 * j));
  }
  add_totals(total, b, sum);
}

// IQ4_XS (quant_linear.metal:99-115): fp16 d | scales_h u16 | scales_l[4] | qs[128]. Element l of sub-block j is the grid
// value at the low (l < 16) or high nibble of qs[16 j + l % 16], times ls_j - 32.
// Eight grid values of a word by byte permutes: `low` = grid values + 128 of the low nibbles of bytes 0..3 and of the high
// ones, as the pairs (byte 0 low, byte 0 high, byte 1 low, byte 1 high) in x and those of bytes 2 and 3 in y.
__device__ __forceinline__ uint2 iq4_lookup(uint32_t word) {
  constexpr uint32_t k0 = 0x3f2d1801u, k1 = 0x766a5d4fu, k2 = 0xa6998d81u, k3 = 0xf1d9c5b5u;  // grid + 128, four per word
  const uint32_t index = word & 0x77777777u, half = ((word >> 1) & 0x44444444u) | 0x32103210u;
  uint2 out;
  out.x = __byte_perm(__byte_perm(k0, k1, index), __byte_perm(k2, k3, index), half);
  out.y = __byte_perm(__byte_perm(k0, k1, index >> 16), __byte_perm(k2, k3, index >> 16), half >> 16);
  return out;
}
template <int NT, class B> __device__ __forceinline__ void iq4_unit(const uint8_t* pA, const uint8_t* pB, int lane, const B& b, float (&total)[NT][4]) {
  const int t = lane & 3;
  constexpr uint32_t k1152 = 0x64806480u;
  const uint2 hA = *reinterpret_cast<const uint2*>(pA), hB = *reinterpret_cast<const uint2*>(pB);
  float sum[NT][4];
  clear(sum);
#pragma unroll(NT > 4 ? 2 : NT > 2 ? 4 : 8)
  for (int j = 0; j < 8; ++j) {
    const uint2 qA = iq4_lookup(lds_u32(pA + 8 + 16 * j + 4 * t)), qB = iq4_lookup(lds_u32(pB + 8 + 16 * j + 4 * t));
    uint32_t a[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      a[u][0] = hsub2_u32(__byte_perm(qA.x, 0x64u, u ? 0x4341 : 0x4240), k1152);
      a[u][1] = hsub2_u32(__byte_perm(qB.x, 0x64u, u ? 0x4341 : 0x4240), k1152);
      a[u][2] = hsub2_u32(__byte_perm(qA.y, 0x64u, u ? 0x4341 : 0x4240), k1152);
      a[u][3] = hsub2_u32(__byte_perm(qB.y, 0x64u, u ? 0x4341 : 0x4240), k1152);
    }
    const int lsA = int((hA.y >> (4 * j)) & 15u) | int(((hA.x >> (16 + 2 * j)) & 3u) << 4);
    const int lsB = int((hB.y >> (4 * j)) & 15u) | int(((hB.x >> (16 + 2 * j)) & 3u) << 4);
    scaled_products<false>(sum, a, b, 2 * j, float(lsA - 32), float(lsB - 32));
  }
  const float dA = load_half_bits(pA), dB = load_half_bits(pB);
#pragma unroll
  for (int tile = 0; tile < NT; ++tile)
    sum[tile][0] *= dA, sum[tile][1] *= dA, sum[tile][2] *= dB, sum[tile][3] *= dB;
  add_totals(total, b, sum);
}

// ---- Q6_K: one 16-row x 256-k unit -------------------------------------------------------------
// Block layout (quant_linear.metal:69-85): ql[128] | qh[64] | int8 sc[16] | fp16 d. Element r = 128*hh + 32*s
// + l has its low nibble in ql[64*hh + 32*(s&1) + l] (high half of the byte when s >= 2), its top two bits
// in qh[32*hh + l] >> 2s, and scale sc[r/16]. MMA gi covers elements [16gi, 16gi+16); lane t supplies
// elements 16gi + 4t + {0,1,2,3}. Blocks are only 2-byte aligned, so words are fetched as two halves; WORDS: as they are, of a block that is
// known to lie at a multiple of four bytes.
template <bool WORDS, int NT, class B>
__device__ __forceinline__ void q6k_unit(const uint8_t* pA, const uint8_t* pB, int lane, const B& b, float (&total)[NT][4]) {
  const int t = lane & 3;
  auto load = [](const uint8_t* p) { return WORDS ? lds_u32(p) : lds_u32_unaligned(p); };
  float sum[NT][4];
  clear(sum);
  const float dA = load_half_bits(pA + 208), dB = load_half_bits(pB + 208);
  constexpr uint32_t k1056 = 0x64206420u;
#pragma unroll(NT > 2 ? 1 : 2)
  for (int hh = 0; hh < 2; ++hh) {
#pragma unroll(NT > 3 ? 1 : 2)
    for (int u = 0; u < 2; ++u) {
      const uint32_t hiA = load(pA + 128 + 32 * hh + 16 * u + 4 * t), hiB = load(pB + 128 + 32 * hh + 16 * u + 4 * t);
#pragma unroll
      for (int sl = 0; sl < 2; ++sl) {
        const uint32_t loA = load(pA + 64 * hh + 32 * sl + 16 * u + 4 * t), loB = load(pB + 64 * hh + 32 * sl + 16 * u + 4 * t);
#pragma unroll
        for (int sh = 0; sh < 2; ++sh) {
          const int s = sl + 2 * sh, gi = hh * 8 + s * 2 + u;
          const uint32_t bytesA = ((sh ? loA >> 4 : loA) & 0x0f0f0f0fu) | ((s < 3 ? hiA << (4 - 2 * s) : hiA >> 2) & 0x30303030u);
          const uint32_t bytesB = ((sh ? loB >> 4 : loB) & 0x0f0f0f0fu) | ((s < 3 ? hiB << (4 - 2 * s) : hiB >> 2) & 0x30303030u);
          uint32_t a[1][4];
          byte_fragment(a[0], bytesA, bytesB, k1056);
          scaled_products<false>(sum, a, b, gi, float(int(reinterpret_cast<const int8_t*>(pA + 192)[gi])), float(int(reinterpret_cast<const int8_t*>(pB + 192)[gi])));
        }
      }
    }
  }
#pragma unroll
  for (int tile = 0; tile < NT; ++tile)
    sum[tile][0] *= dA, sum[tile][1] *= dA, sum[tile][2] *= dB, sum[tile][3] *= dB;
  add_totals(total, b, sum);
}

}  // namespace infdev
