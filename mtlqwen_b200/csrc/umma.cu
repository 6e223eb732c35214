// Q4_K prefill GEMM on the 5th-generation tensor cores (tcgen05) with the weight operand in tensor memory.
//
// Replaces linear_prefill / linear_prefill_small (quant_linear.metal:151-233, epilogues 0 / 1 / 2) for weight matrices
// whose row count is a multiple of 128 and whose K is a multiple of 2048, for 9 to 128 activation rows per launch:
//   * one thread owns one weight row of a 128-row tile: it reads the row's 144-byte super-block from a TMA-filled slab,
//     dequantises it to fp16 (d*sc*q - dmin*m, d*sc and dmin*m rounded once, one fused multiply-add per two weights) and
//     writes it to tensor memory with tcgen05.st;
//   * tcgen05.mma (kind::f16, M = 128 weight rows, N = 128 activation rows, K = 16) takes A from TMEM and B, the
//     activations, from shared memory through a matrix descriptor. The activations were rounded to fp16 beforehand
//     (umma_prepare_rows_kernel), already laid out as canonical no-swizzle K-major core matrices under the same K
//     permutation that the nibble extraction produces;
//   * two fp32 accumulators of 128 columns: the halves of every super-block, added up at the end, or a gate / up pair, whose matrices
//     share every copy of the activations and whose silu(gate) * up is formed from the two.
// Warp roles: 0 = weight slabs, 1 = activations (one thread each issues the copies), 2 and 3 = MMA issuers (warp 2 owns the TMEM
// allocation), 4..19 = four dequant groups of four warps (one TMEM lane quadrant each), which also store the results. Every mbarrier wait is
// bounded; on a timeout the kernel raises an abort flag, records a status code, and every role leaves its loops.
// Weight slabs (a super-block of 128 rows, 18 KB) and activations (half a super-block, 4 to 32 KB by the rows of the launch) travel through
// rings of their own. The operand A has four places in tensor memory, half a super-block each, one per dequant group; the accumulators are two, one
// per issuer. An issuer spends 430 to 700 clocks on the waits, eight MMAs and two commits of a half, whatever N; one issuer of both
// halves was what set the pace of a pair (12288 x 4096, 128 rows 35.3 us, 29.1 with two; 9 rows 28.8 and 23.3).
// Bulk prefetches of whole tiles into the L2 got in the way of the copies (18944 x 16384 with 9 rows 71.9 -> 64.6 us without them).
// The kernel is launched programmatically dependent on the kernel that lays out the activations: set-up and the first
// weight slabs run while that one is still at work, and only the activation copies and the epilogue wait for it.
// What bounds it, by its own clocks: a super-block of 128 rows takes a CTA about 850 clocks with few rows (the dequant groups, 500 warp
// instructions a scheduler) and 1250 with 128 (of which the MMAs are 1024). What is left is not in the loop: 4 to 5 us
// from the end of the kernel before to the first MMA, through the layout kernel and two launches, and 1.5 us (a pair with 128 rows 3.3 us: silu)
// of stores. 96 tiles (n = 12288) occupy 96 of 148 SMs. All projections of a layer, before the two issuers, the cheaper dequantisation and the
// rings by row count, and now, back to back in a graph: 9 rows 78.0 -> 55.1 us, 40 rows 82.6 -> 59.0, 128 rows 100.8 -> 79.7.
// Tried and left out: fp32 activations converted by four warps of the kernel itself instead of the layout kernel (12288 x 4096, 9 rows 16.0 us
// against 14.1, 40 rows 20.5 against 14.9: copies of twice the bytes, and a proxy fence between every conversion and its MMAs); K slices as
// clusters that add up over distributed shared memory instead of umma_reduce_kernel (4096 x 4096, 9 rows 8.8 against 8.6 us, 40 rows 10.1 against 9.5);
// equal parts of all tiles' super-blocks for all SMs, the last CTA of a shared tile adding up what the others left in global memory
// (12288 x 4096, 9 rows 18.7 against 14.3, 128 rows 32.6 against 18.4: every CTA then ends two tiles, not one).
#include "kernels.h"
#include "tcgen05.cuh"

namespace infdev {
namespace {

constexpr int kRows = kUmmaTileRows;      // weight rows per tile = TMEM lanes
constexpr int kActs = 128;                // most activation rows per launch; the MMA N is the live rows rounded up to 16
constexpr int kSlabBytes = kRows * 144;   // 18,432
constexpr int kGroups = 4;                // dequant groups of four warps
constexpr int kWeightWarp = 0, kActWarp = 1, kIssueWarp = 2, kFirstDequantWarp = 4;  // two issuers: warps 2 and 3
constexpr int kThreads = (kFirstDequantWarp + 4 * kGroups) * kWarp;
constexpr int kMaxStages = 10, kMaxActStages = 8;
// kind::f16 instruction descriptor: fp32 accumulate, fp16 A and B, both K-major, M = 128
__device__ __forceinline__ uint32_t instruction_descriptor(int n) { return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(kRows >> 4) << 24); }
constexpr int kTmemCols = 512;
constexpr uint32_t kColA = 0, kColD = 256;  // A: 64 columns (half a super-block) per dequant group; D: 128 columns per issuer

struct Control {
  uint64_t full[kMaxStages], slotFree[kMaxStages], actFull[kMaxActStages], actFree[kMaxActStages], aReady[kGroups], aFree[kGroups], dReady, dFree;
  uint32_t tmemBase;
  int abort;
};
constexpr int kControlBytes = 512;
static_assert(sizeof(Control) <= kControlBytes, "control block too large");
// 222 KB, and registers for 768 threads, leave an SM room for a block of the small kernels before and after, which start early: with all of the
// shared memory (a block without any takes 1 KB) they waited for SMs that have no CTA of this kernel (4096 x 4096, 24 rows 10.2 -> 8.9 us).
constexpr int kBoundThreads = 768;
constexpr size_t kSharedBytes = 222 * 1024, kRingBytes = kSharedBytes - 1024 - kControlBytes;

__device__ __forceinline__ void tmem_load8(uint32_t address, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(address)
               : "memory");
}

__device__ __forceinline__ int find_segment(const UmmaParams& p, int tile) {
  int segment = 0;
  while (segment + 1 < p.nseg && tile >= p.seg[segment + 1].tile0)
    ++segment;
  return segment;
}

// Where the 32 TMEM lanes (= weight rows = output columns) of the calling warp go. Everything the store loop needs is copied out of the
// parameter block: the segment is a run-time index, so the block is reached through a generic address, and the compiler must assume that
// the stores change it and would read pointer and pitch again after every one of them (measured: 110 ns per store instead of 10).
struct Destination {
  float* y;
  const float* residual;
  size_t pitch;
};
template <bool PAIR> __device__ __forceinline__ Destination destination(const UmmaParams& p, int item, int row) {
  const int tile = item % p.tiles, slice = item / p.tiles, segment = find_segment(p, tile);
  Destination d;
  d.pitch = size_t(p.seg[segment].ldy);
  const size_t column = size_t(tile - p.seg[segment].tile0) * kRows + row;
  // a K slice: the partial sums are added up, with the residual, by umma_reduce_kernel
  const bool parts = !PAIR && p.splits > 1;
  d.y = (parts ? p.partial + size_t(slice) * p.m * d.pitch : p.seg[segment].y) + column;
  d.residual = PAIR || parts || !p.seg[segment].res ? nullptr : p.seg[segment].res + column;
  return d;
}
// Eight activation rows of an item from `first` on.
template <bool PAIR> __device__ __forceinline__ void store_rows(const Destination& d, int m, uint32_t accumulator, int first, const float (&residual)[8]) {
  uint32_t v[8], w[8];
  tmem_load8(accumulator + first, v);
  tmem_load8(accumulator + kActs + first, w);
  float* y = d.y + size_t(first) * d.pitch;
  tmem_wait_load();
#pragma unroll
  for (int i = 0; i < 8; ++i, y += d.pitch) {
    const float a = __uint_as_float(v[i]), b = __uint_as_float(w[i]);  // of a pair gate and up (post == 2 epilogue, quant_linear.metal:224-232)
    if (first + i < m)
      *y = PAIR ? silu_f(a) * b : a + b + residual[i];
  }
}
template <bool PAIR> __device__ __forceinline__ void load_residual(const Destination& d, int m, int first, float (&residual)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    residual[i] = !PAIR && d.residual && first + i < m ? d.residual[size_t(first + i) * d.pitch] : 0.f;
}

// Whether one of two scales is not below 2^-6 (or not a number).
__device__ __forceinline__ bool reaches_64th(const __half2& scales) {
  return (((*reinterpret_cast<const uint32_t*>(&scales) & 0x7fff7fffu) + 0x5c005c00u) & 0x80008000u) != 0;
}

// 64 weights scale * q + low of two sub-blocks, in the order of the operand's columns: the low nibbles of eight words belong to the first, the
// high ones to the second. SMALL: scales below 2^-6. The nibbles in bits 2..5 or 6..9 of a 16-bit group are fp16 numbers as they are, q x 2^-22
// and q x 2^-18, and one multiply-add with the scale times 2^22 or 2^18, which is exact, gives the bits that the general form has: there q is
// brought to an exponent of its own and made exact first (13 instructions for eight weights; 10 here, of which five on the
// half-rate ALU pipe: projections of a layer with 9, 40 and 128 rows 64.1 -> 56.6, 67.2 -> 59.7 and 83.3 -> 80.3 us).
template <bool SMALL> __device__ __forceinline__ void dequantise(const uint4& q0, const uint4& q1, const __half2& scale, const __half2& low, uint32_t (&v)[32]) {
  constexpr uint32_t k1024 = 0x64006400u, kSixteenth = 0x2c002c00u, kMinus64 = 0xd400d400u, k2048 = 0x68006800u, k512 = 0x60006000u;
  const __half2 scaleLow = __low2half2(scale), scaleHigh = __high2half2(scale), lowLow = __low2half2(low), lowHigh = __high2half2(low);
  uint32_t sL = *reinterpret_cast<const uint32_t*>(&scaleLow), sH = *reinterpret_cast<const uint32_t*>(&scaleHigh);
  const uint32_t nL = *reinterpret_cast<const uint32_t*>(&lowLow), nH = *reinterpret_cast<const uint32_t*>(&lowHigh);
  if (SMALL)
    sL = hmul2_u32(hmul2_u32(sL, k2048), k2048), sH = hmul2_u32(hmul2_u32(sH, k512), k512);
  const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (SMALL) {
      const uint32_t a = words[w] << 2, b = words[w] >> 6;
      v[2 * w] = hfma2_u32(a & 0x003c003cu, sL, nL);
      v[2 * w + 1] = hfma2_u32(b & 0x003c003cu, sL, nL);
      v[16 + 2 * w] = hfma2_u32(a & 0x03c003c0u, sH, nH);
      v[16 + 2 * w + 1] = hfma2_u32(b & 0x03c003c0u, sH, nH);
    } else {
      const uint32_t a = words[w], b = a >> 8;
      v[2 * w] = hfma2_u32(hsub2_u32((a & 0x000f000fu) | k1024, k1024), sL, nL);
      v[2 * w + 1] = hfma2_u32(hsub2_u32((b & 0x000f000fu) | k1024, k1024), sL, nL);
      v[16 + 2 * w] = hfma2_u32(hfma2_u32((a & 0x00f000f0u) | k1024, kSixteenth, kMinus64), sH, nH);
      v[16 + 2 * w + 1] = hfma2_u32(hfma2_u32((b & 0x00f000f0u) | k1024, kSixteenth, kMinus64), sH, nH);
    }
  }
}

template <bool PAIR> __global__ void __launch_bounds__(kBoundThreads, 1) umma_linear_kernel(const __grid_constant__ UmmaParams p) {
  constexpr int kMats = PAIR ? 2 : 1;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
  Control& ctl = *reinterpret_cast<Control*>(smem);
  uint8_t* ring = smem + kControlBytes;
  uint8_t* actRing = ring + size_t(p.stages) * kSlabBytes;

  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // With p.splits > 1 (one matrix) the work items are (tile, K slice) pairs, so that a matrix of few 128-row tiles still
  // fills the GPU; `blocksPerRow` is then the super-blocks of one slice.
  const int blocksPerRow = p.k / 256 / p.splits, items = p.tiles * p.splits;
  const uint32_t stages = uint32_t(p.stages), actStages = uint32_t(p.actStages);
  const uint32_t actBytes = uint32_t(p.actRows) * 256;  // half a super-block: 8 k-steps x [actRows x 16] fp16
  volatile int* abortFlag = &ctl.abort;
  auto give_up = [&] {
    *abortFlag = 1;
    atomicExch(p.status, kStatusBarrierTimeout);
  };

  if (tid == 0) {
    for (uint32_t s = 0; s < stages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.slotFree[s], 8);  // the warps of the two groups that share a super-block
    }
    for (uint32_t s = 0; s < actStages; ++s) {
      mbar_init(&ctl.actFull[s], 1);
      mbar_init(&ctl.actFree[s], kMats);  // the issuers that read it
    }
    for (int g = 0; g < kGroups; ++g) {
      mbar_init(&ctl.aReady[g], 4);  // the warps of the group
      mbar_init(&ctl.aFree[g], 1);
    }
    mbar_init(&ctl.dReady, 2);
    mbar_init(&ctl.dFree, 4 * kGroups);
    ctl.abort = 0;
    mbar_fence_init();
  }
  if (warp == kIssueWarp)
    tmem_alloc(&ctl.tmemBase, kTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = ctl.tmemBase;

  if (warp == kWeightWarp) {
    // ---------------- weight slabs: do not depend on the kernels before this one ----------------
    if (elect_one()) {
      uint32_t slot = 0, lap = 0, slabs = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int tile = item % p.tiles, firstBlock = (item / p.tiles) * blocksPerRow;
        const int segment = find_segment(p, tile);
        const int row0 = (tile - p.seg[segment].tile0) * kRows;
        for (int sb = firstBlock; sb < firstBlock + blocksPerRow && ok; ++sb)
          for (int mat = 0; mat < kMats && ok; ++mat) {
            if (lap > 0)
              ok = mbar_wait_bounded(&ctl.slotFree[slot], (lap - 1) & 1, abortFlag);
            if (ok) {
              mbar_arrive_expect_tx(&ctl.full[slot], kSlabBytes);
              tma_load_2d(ring + size_t(slot) * kSlabBytes, &p.map[segment][mat], sb * 18, row0, &ctl.full[slot]);
              ++slabs;
              if (++slot == stages)
                slot = 0, ++lap;
            }
          }
      }
      if (!ok)
        give_up();
      // no copy may be in flight when the CTA ends, whoever gave up
      for (uint32_t i = slabs > stages ? slabs - stages : 0; i < slabs; ++i)
        mbar_wait_bounded(&ctl.full[i % stages], (i / stages) & 1, abortFlag);
    }
  } else if (warp == kActWarp) {
    // ---------------- activations, by halves of a super-block: the preceding kernel's output ----------------
    pdl_wait();
    if (elect_one()) {
      uint32_t slot = 0, lap = 0, copies = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int firstHalf = (item / p.tiles) * blocksPerRow * 2;
        for (int half = firstHalf; half < firstHalf + blocksPerRow * 2 && ok; ++half) {
          if (lap > 0)
            ok = mbar_wait_bounded(&ctl.actFree[slot], (lap - 1) & 1, abortFlag);
          if (ok) {
            mbar_arrive_expect_tx(&ctl.actFull[slot], actBytes);
            bulk_load(actRing + size_t(slot) * actBytes, p.acts + size_t(half) * actBytes, actBytes, &ctl.actFull[slot]);
            ++copies;
            if (++slot == actStages)
              slot = 0, ++lap;
          }
        }
      }
      if (!ok)
        give_up();
      for (uint32_t i = copies > actStages ? copies - actStages : 0; i < copies; ++i)
        mbar_wait_bounded(&ctl.actFull[i % actStages], (i / actStages) & 1, abortFlag);
    }
  } else if (warp < kFirstDequantWarp) {
    // ---------------- MMA issuers: of a pair one matrix each, otherwise one half of every super-block ----------------
    if (elect_one()) {
      const uint32_t issuer = uint32_t(warp - kIssueWarp);
      uint32_t slot = PAIR ? 0 : issuer, parity = 0, count = 0, unit = 0;  // count: super-blocks
      bool ok = true;
      const uint32_t instruction = instruction_descriptor(p.actRows), stepBytes = uint32_t(p.actRows) * 32;
      const uint32_t dColumn = tmem + kColD + issuer * kActs;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++unit) {
        if (unit > 0)
          ok = mbar_wait_bounded(&ctl.dFree, (unit - 1) & 1, abortFlag);
        for (int j = 0; j < blocksPerRow && ok; ++j, ++count) {
#pragma unroll
          for (int turn = 0; turn < kMats; ++turn) {
            // the dequant group that fills this operand, and how often it has
            const uint32_t half = PAIR ? uint32_t(turn) : issuer, group = PAIR ? 2 * issuer + half : 2 * (count & 1) + half, fill = PAIR ? count : count >> 1;
            ok = ok && mbar_wait_bounded(&ctl.actFull[slot], parity, abortFlag) && mbar_wait_bounded(&ctl.aReady[group], fill & 1, abortFlag);
            if (!ok)
              break;
            const uint64_t act = smem_descriptor(smem_u32(actRing + size_t(slot) * actBytes), 128, 256);
            fence_after_sync();
#pragma unroll
            for (uint32_t step = 0; step < 8; ++step)
              umma_ts(dColumn, tmem + kColA + group * 64 + step * 8, act + (step * stepBytes >> 4), instruction, uint32_t(j | turn) | step);
            umma_commit(&ctl.aFree[group]);
            umma_commit(&ctl.actFree[slot]);
            if ((slot += PAIR ? 1 : 2) >= actStages)
              slot -= actStages, parity ^= 1;
          }
        }
        if (ok)
          umma_commit(&ctl.dReady);
      }
      if (!ok)
        give_up();
    }
  } else {
    // ---------------- dequant: thread = weight row; a group takes one half of every second slab and has a place of its own in tensor
    // memory for it, so that a group fills its operand while the MMAs of the others run ----------------
    const uint32_t group = uint32_t(warp - kFirstDequantWarp) >> 2, side = group & 1;
    const int quadrant = warp & 3, row = quadrant * 32 + lane;
    const uint32_t laneBase = tmem + (uint32_t(quadrant * 32) << 16), aAddress = laneBase + kColA + group * 64;
    constexpr uint32_t k1024 = 0x64006400u;
    // of the whole warp, which reads and writes tensor memory together: a lane whose limit runs out takes the others with it
    auto wait = [&](uint64_t* bar, uint32_t parity) { return bool(__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abortFlag))); };
    uint32_t slot = group >> 1, parity = 0, fills = 0, unit = 0, slab = group >> 1;  // slab: the next of this group, counted over all items
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++unit) {
      const uint32_t end = (unit + 1) * uint32_t(blocksPerRow * kMats);
      for (; slab < end && ok; slab += 2, ++fills) {
        ok = wait(&ctl.full[slot], parity);
        if (!ok)
          break;
        const uint8_t* block = ring + size_t(slot) * kSlabBytes + row * 144;
        const uint4 header = *reinterpret_cast<const uint4*>(block);
        uint4 quads[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          quads[i] = *reinterpret_cast<const uint4*>(block + 16 + 64 * side + 16 * i);
        // 6-bit scales / mins of this half's four sub-blocks (scale_min_k4, quant_linear.metal:12-20)
        const uint32_t scales = side == 0 ? header.y & 0x3f3f3f3fu : (header.w & 0x0f0f0f0fu) | ((header.y >> 2) & 0x30303030u);
        const uint32_t mins = side == 0 ? header.z & 0x3f3f3f3fu : ((header.w >> 4) & 0x0f0f0f0fu) | ((header.z >> 2) & 0x30303030u);
        const __half2 dm = *reinterpret_cast<const __half2*>(&header.x), d = __low2half2(dm), dmin = __hneg2(__high2half2(dm));
        // dequantised weight d*sc*q - dmin*m, in fp16: sc and m are made exact first, then the products d*sc and dmin*m are rounded once
        __half2 scale[2], low[2];  // of sub-blocks 2t and 2t + 1
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t scalePair = hsub2_u32(__byte_perm(scales, 0x64u, t == 0 ? 0x4140 : 0x4342), k1024);
          const uint32_t minPair = hsub2_u32(__byte_perm(mins, 0x64u, t == 0 ? 0x4140 : 0x4342), k1024);
          scale[t] = __hmul2(d, *reinterpret_cast<const __half2*>(&scalePair)), low[t] = __hmul2(dmin, *reinterpret_cast<const __half2*>(&minPair));
        }
        // the slab is in registers by now; the MMAs that read this group's operand before may run until the first store
        auto store = [&](int t, const uint32_t (&v)[32]) {
          if (t == 0) {
            __syncwarp();
            if (lane == 0)
              mbar_arrive(&ctl.slotFree[slot]);
            if (fills > 0)
              ok = wait(&ctl.aFree[group], (fills - 1) & 1);
            fence_after_sync();
          }
          if (ok)
            tmem_store32(aAddress + 32 * t, v);
        };
        if (__any_sync(0xffffffffu, reaches_64th(scale[0]) || reaches_64th(scale[1]))) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            uint32_t v[32];
            dequantise<false>(quads[2 * t], quads[2 * t + 1], scale[t], low[t], v);
            store(t, v);
          }
        } else {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            uint32_t v[32];
            dequantise<true>(quads[2 * t], quads[2 * t + 1], scale[t], low[t], v);
            store(t, v);
          }
        }
        if (!ok)
          break;
        tmem_wait_store();
        fence_before_sync();
        __syncwarp();
        if (lane == 0)
          mbar_arrive(&ctl.aReady[group]);
        if ((slot += 2) >= stages)
          slot -= stages, parity ^= 1;
      }
      // ---- epilogue: thread = weight row ----
      pdl_wait();  // residuals, results and the partial-sum buffer belong to earlier kernels
      const Destination to = destination<PAIR>(p, item, row);
      const int m = p.m;
      float residual[8];
      load_residual<PAIR>(to, m, int(group) * 8, residual);
      ok = ok && wait(&ctl.dReady, unit & 1);
      if (!ok)
        break;
      fence_after_sync();
      for (int first = int(group) * 8; first < m; first += kGroups * 8) {
        float next[8];
        load_residual<PAIR>(to, m, first + kGroups * 8, next);
        store_rows<PAIR>(to, m, laneBase + kColD, first, residual);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          residual[i] = next[i];
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&ctl.dFree);
    }
    if (!ok && lane == 0)
      give_up();
  }
  fence_before_sync();
  __syncthreads();
  if (warp == kIssueWarp)
    tmem_dealloc(tmem, kTmemCols);
}

// Lays the activations out as the B operand, per 256-wide super-block: [16 k-steps][16 row groups][2 K halves][8 rows]
// [8 values] fp16, rows rounded to fp16, rows from m up zero. K inside a step follows the order in which the
// dequantiser emits weights: step s covers the quant bytes of 64-group t = s / 4, nibble side (s / 2) % 2, words
// 4 * (s % 2) .. +3; TMEM column c of a step holds the nibbles of bytes (c % 2, c % 2 + 2) of word c / 2. Eight
// consecutive k of a super-block are thus one 16-byte core-matrix row of a k-step (in the order 0,2,1,3,4,6,5,7), and a
// thread turns two float4 loads into one 16-byte store.
__device__ __forceinline__ void store_operand(__half* acts, int actRows, int sb, int n, int group, const float4& a, const float4& b) {
  const __half2 h0 = __floats2half2_rn(a.x, a.z), h1 = __floats2half2_rn(a.y, a.w), h2 = __floats2half2_rn(b.x, b.z), h3 = __floats2half2_rn(b.y, b.w);
  uint4 packed;
  packed.x = *reinterpret_cast<const uint32_t*>(&h0), packed.y = *reinterpret_cast<const uint32_t*>(&h1);
  packed.z = *reinterpret_cast<const uint32_t*>(&h2), packed.w = *reinterpret_cast<const uint32_t*>(&h3);
  __half* out = acts + size_t(sb) * (actRows * 256);
  *reinterpret_cast<uint4*>(out + size_t(group >> 1) * (actRows * 16) + (n >> 3) * 128 + (group & 1) * 64 + (n & 7) * 8) = packed;
}

// grid (k / 256, actRows / 8), 256 threads: actRows x 32 groups of eight per super-block, one per thread; a warp reads
// one activation row's 256 values.
__global__ void __launch_bounds__(256) umma_prepare_rows_kernel(const float* x, int ldx, int m, int actRows, __half* acts) {
  pdl_launch_dependents();
  pdl_wait();
  const int sb = blockIdx.x, item = blockIdx.y * 256 + threadIdx.x, n = item >> 5, group = item & 31;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  if (n < m) {
    const float4* src = reinterpret_cast<const float4*>(x + size_t(n) * ldx + size_t(sb) * 256 + group * 8);
    a = src[0], b = src[1];
  }
  store_operand(acts, actRows, sb, n, group, a, b);
}

// The same of the RMS norm of x (k = 4096), with the bits of rms_norm_4096_kernel, whose launch it saves; `normalised`, when not null, receives the
// rows themselves. grid actRows, 512 threads: a warp has one super-block of a row. Norm and projections of 9, 40 and 128 rows, 8192 and 4096 x 4096
// 14.4 -> 13.6, 14.9 -> 14.4, 20.2 -> 19.6 us, gate and up of 12288 x 4096 20.1 -> 18.9, 21.5 -> 20.5, 31.2 -> 29.4.
__global__ void __launch_bounds__(512) umma_norm_rows_kernel(const float* x, const float* w, int m, int actRows, float* normalised, __half* acts) {
  pdl_launch_dependents();
  pdl_wait();
  const int n = blockIdx.x, d = threadIdx.x * 8;
  float v[8] = {};
  if (n < m) {
    const float4* src = reinterpret_cast<const float4*>(x + size_t(n) * 4096 + d);
    const float4* weights = reinterpret_cast<const float4*>(w + d);
    normalise_4096(src[0], src[1], weights[0], weights[1], v);
  }
  const float4 a = make_float4(v[0], v[1], v[2], v[3]), b = make_float4(v[4], v[5], v[6], v[7]);
  store_operand(acts, actRows, threadIdx.x / kWarp, n, threadIdx.x % kWarp, a, b);
  if (normalised && n < m) {
    float4* to = reinterpret_cast<float4*>(normalised + size_t(n) * 4096 + d);
    to[0] = a, to[1] = b;
  }
}

// y = partial[0] + partial[1] + ... (+ residual), four values per thread. AT_ONCE: a thread asks for all of them before it adds, one trip to
// the L2 instead of one for each slice. With more than 64 rows the blocks are so many that what counts is how many of them fit beside the GEMM's
// CTAs and are there when it ends, which takes few registers. One after the other / at once, 4096 x 4096 with 9, 32, 48, 64, 80, 96 and 128 rows 8.1 / 7.7,
// 8.6 / 8.0, 9.3 / 8.4, 9.3 / 9.0, 10.2 / 10.5, 10.0 / 11.3 and 11.5 / 12.7 us; 4096 x 12288 with 48, 64 and 80 rows 14.5 / 14.9, 15.4 / 15.2, 15.8 / 15.9.
template <bool AT_ONCE> __global__ void __launch_bounds__(256) umma_reduce_kernel(const float* partial, int splits, size_t count, const float* residual, float* y) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t at = (size_t(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (at >= count)
    return;
  auto add = [](float4& sum, const float4& v) { sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w; };
  float4 sum = *reinterpret_cast<const float4*>(partial + at);
  if (AT_ONCE) {
    float4 slice[kUmmaMaxSplits], more = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 1; s < kUmmaMaxSplits; ++s)
      if (s < splits)
        slice[s] = *reinterpret_cast<const float4*>(partial + s * count + at);
    if (residual)
      more = *reinterpret_cast<const float4*>(residual + at);
#pragma unroll
    for (int s = 1; s < kUmmaMaxSplits; ++s)
      if (s < splits)
        add(sum, slice[s]);
    if (residual)
      add(sum, more);
  } else {
    for (int s = 1; s < splits; ++s)
      add(sum, *reinterpret_cast<const float4*>(partial + s * count + at));
    if (residual)
      add(sum, *reinterpret_cast<const float4*>(residual + at));
  }
  *reinterpret_cast<float4*>(y + at) = sum;
}

template <bool PAIR>
cudaError_t launch_tiles(const UmmaParams& params, const float* x, int ldx, const float* norm, float* normalised, int sms, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (const cudaError_t e = configure_shared_memory(umma_linear_kernel<PAIR>, kSharedBytes, configured))
    return e;
  // The MMA is as wide as the launch has rows, in steps of 16: a speculative pass of 40 rows moves 24 KB of activations
  // per super-block instead of 64 KB and spends a third of the tensor time.
  UmmaParams p = params;
  p.actRows = (p.m + 15) / 16 * 16;
  const int actBytes = p.actRows * 256;
  p.actStages = int((kRingBytes - 4 * kSlabBytes) / actBytes) / 2 * 2;
  p.actStages = p.actStages > kMaxActStages ? kMaxActStages : p.actStages;
  // An even number of slab slots: a slot then always belongs to the same dequant groups (they take the slabs in pairs by turns). Otherwise
  // a group could find the parity of the phase before last in a slot whose slab for another group had not landed yet, and read it
  // ahead of its own copy.
  p.stages = int((kRingBytes - size_t(p.actStages) * actBytes) / kSlabBytes) / 2 * 2;
  p.stages = p.stages > kMaxStages ? kMaxStages : p.stages;
  __half* const acts = reinterpret_cast<__half*>(const_cast<uint8_t*>(p.acts));
  if (norm)
    launch_kernel<1>(umma_norm_rows_kernel, unsigned(p.actRows), 512, 0, stream, x, norm, p.m, p.actRows, normalised, acts);
  else
    launch_kernel<1>(umma_prepare_rows_kernel, dim3(p.k / 256, p.actRows / 8), 256, 0, stream, x, ldx, p.m, p.actRows, acts);
  const int items = p.tiles * p.splits, grid = items < sms ? items : sms;
  launch_kernel<1>(umma_linear_kernel<PAIR>, grid, kThreads, kSharedBytes, stream, p);
  if (p.splits > 1) {
    const size_t count = size_t(p.m) * p.seg[0].ldy;
    launch_kernel<1>(p.m <= 64 ? umma_reduce_kernel<true> : umma_reduce_kernel<false>, unsigned((count / 4 + 255) / 256), 256, 0, stream, p.partial, p.splits, count,
                     p.seg[0].res, p.seg[0].y);
  }
  return cudaGetLastError();
}

}  // namespace

// 9 to 128 activation rows (p.m), rows of x `ldx` floats apart (a multiple of 4). norm: the activations are the RMS norm of x with these weights
// (k = ldx = 4096), and go to `normalised` too where that is not null.
cudaError_t umma_launch(bool pair, const UmmaParams& p, const float* x, int ldx, const float* norm, float* normalised, int sms, cudaStream_t stream) {
  return pair ? launch_tiles<true>(p, x, ldx, norm, normalised, sms, stream) : launch_tiles<false>(p, x, ldx, norm, normalised, sms, stream);
}

}  // namespace infdev
