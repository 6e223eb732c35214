// Q4_K prefill GEMM on the 5th-generation tensor cores (tcgen05) with the weight operand in tensor memory.
//
// Replaces linear_prefill / linear_prefill_small (quant_linear.metal:151-233, epilogues 0 / 1 / 2) for weight matrices
// whose row count is a multiple of 128 and whose K is a multiple of 2048, for 9 to 128 activation rows per launch:
//   * one thread owns one weight row of a 128-row tile: it reads the row's 144-byte super-block from a TMA-filled slab,
//     dequantises it to fp16 (d*sc*q - dmin*m, q made exact first, then one fused multiply-add per two weights) and
//     writes it to tensor memory with tcgen05.st;
//   * tcgen05.mma (kind::f16, M = 128 weight rows, N = 128 activation rows, K = 16) takes A from TMEM and B, the
//     activations, from shared memory through a matrix descriptor. The activations were rounded to fp16 beforehand
//     (umma_prepare_rows_kernel), already laid out as canonical no-swizzle K-major core matrices under the same K
//     permutation that the nibble extraction produces;
//   * one 128-column fp32 accumulator per tile, double-buffered, so the epilogue of one overlaps the MMAs of the next. A gate /
//     up pair takes both: every super-block of the activations is copied once and multiplied with both matrices (one after the other,
//     with 96 CTAs on the activations twice, the copies were what the tensor cores waited for: 47.5 us for 12288 x 4096 with 128
//     rows, 35.0 now), and silu(gate) * up is formed from the two accumulators.
// Warp roles: 0 = TMA producer, 1 = MMA issuer (owns the TMEM allocation), 4..11 (4..19) = dequant (two or four groups of
// four, one TMEM lane quadrant each), the last four = epilogue. Every mbarrier wait is bounded; on a timeout the kernel raises an abort
// flag, records a status code, and every role leaves its loops.
// The fp16 activations of a super-block are 64 KB, so weight slabs and activations travel through separate rings, the
// activations in two halves of eight k-steps each: 4 slab stages + 4 half stages. Bulk prefetches of whole tiles into the L2, which
// the producer once began with, got in the way of the copies (18944 x 16384 with 9 rows 71.9 -> 64.6 us without them, with 128 rows
// 92.0 -> 84.3; all projections of a layer 88.3 -> 82.1 and 121.7 -> 112.9).
// The kernel is launched programmatically dependent on the kernel that lays out the activations: set-up and the first
// weight slab run while that one is still at work, and only the activation copies and the epilogue wait for it.
// What bounds it, by its own clocks (18944 x 8192, every SM at work): with 128 rows the copies, 82 KB a super-block of which 64 are
// activations, at 45 bytes a clock and SM (0.95 us; the 16 MMAs are 0.55); with few rows a dequant group's 1200 clocks a half. 96 tiles
// (n = 12288) occupy 96 of 148 SMs.
#include "kernels.h"
#include "tcgen05.cuh"

namespace infdev {
namespace {

constexpr int kRows = kUmmaTileRows;      // weight rows per tile = TMEM lanes
constexpr int kActs = 128;                // most activation rows per launch; the MMA N is the live rows rounded up to 16
constexpr int kSlabBytes = kRows * 144;   // 18,432
template <int GROUPS> constexpr int kThreads = (8 + 4 * GROUPS) * kWarp;  // GROUPS: dequant groups of four warps, 2 or 4
// An even number of slab slots: a slot then always belongs to the same dequant groups (four groups take the super-blocks in
// pairs by turns). Otherwise a group could find the parity of the phase before last in a slot whose slab for another group
// had not landed yet, and read it ahead of its own copy.
constexpr int kStages = 4, kActStages = 4;
static_assert(kStages % 2 == 0, "a slot serves the same dequant groups throughout");
constexpr int kActHalfBytes = 8 * kActs * 16 * 2;  // ring stage: 8 k-steps x [128 x 16] fp16; a launch of N rows uses N x 256 of it
// kind::f16 instruction descriptor: fp32 accumulate, fp16 A and B, both K-major, M = 128
__device__ __forceinline__ uint32_t instruction_descriptor(int n) { return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(kRows >> 4) << 24); }
constexpr int kTmemCols = 512;
constexpr uint32_t kColA = 0, kColD = 256;  // A: ring of 4 x 64 columns, half a super-block each; D: 2 x 128 columns
constexpr uint32_t kABuffers = 4;

struct Control {
  uint64_t full[8], slotFree[8], actFull[8], actFree[8], aReady[kABuffers], aFree[kABuffers], dReady[2], dFree[2];
  uint32_t tmemBase;
  int abort;
};
constexpr int kControlBytes = 512;
static_assert(sizeof(Control) <= kControlBytes, "control block too large");
constexpr size_t kSharedBytes = 1024 + kControlBytes + size_t(kStages) * kSlabBytes + size_t(kActStages) * kActHalfBytes;

__device__ __forceinline__ void tmem_load8(uint32_t address, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(address)
               : "memory");
  tmem_wait_load();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    v[i] = __uint_as_float(r[i]);
}

// The epilogue of one item for the 32 TMEM lanes (= weight rows = output columns) of the calling
// warp: groups of eight activation rows `first`, `first + stride`, ... of the 16. Everything the store loop needs is
// copied out of the parameter block first: the segment is a run-time index, so the block is reached through a generic
// address, and the compiler must assume that the stores change it and would read pointer and pitch again after every
// one of them (measured: 110 ns per store instead of 10).
template <int NMAT> __device__ __forceinline__ void store_accumulator(const UmmaParams& p, int item, uint32_t accumulator, int row, int first, int stride) {
  const int tile = item % p.tiles, slice = item / p.tiles;
  int segment = 0;
  while (segment + 1 < p.nseg && tile >= p.seg[segment + 1].tile0)
    ++segment;
  const size_t pitch = size_t(p.seg[segment].ldy), column = size_t(tile - p.seg[segment].tile0) * kRows + row;
  const int liveRows = p.m;
  // a K slice: the partial sums are added up, with the residual, by umma_reduce_kernel
  const bool parts = NMAT == 1 && p.splits > 1;
  float* const y = parts ? p.partial + size_t(slice) * p.m * pitch : p.seg[segment].y;
  const float* const residual = NMAT == 2 || parts ? nullptr : p.seg[segment].res;
  for (int c = first; c < kActs / 8 && c * 8 < liveRows; c += stride) {
    float v[8], up[8];
    tmem_load8(accumulator + c * 8, v);
    if (NMAT == 2)  // post == 2 epilogue, quant_linear.metal:224-232
      tmem_load8(accumulator + kActs + c * 8, up);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = c * 8 + i;
      if (m < liveRows) {
        const size_t at = size_t(m) * pitch + column;
        y[at] = NMAT == 2 ? silu_f(v[i]) * up[i] : residual ? v[i] + residual[at] : v[i];
      }
    }
  }
}

template <int NMAT, int GROUPS> __global__ void __launch_bounds__(kThreads<GROUPS>, 1) umma_linear_kernel(const __grid_constant__ UmmaParams p) {
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
  Control& ctl = *reinterpret_cast<Control*>(smem);
  uint8_t* ring = smem + kControlBytes;
  uint8_t* actRing = ring + size_t(kStages) * kSlabBytes;  // halves of a super-block's activations

  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // With p.splits > 1 (one matrix) the work items are (tile, K slice) pairs, so that a matrix of few 128-row tiles still
  // fills the GPU; `blocksPerRow` is then the super-blocks of one slice.
  const int blocksPerRow = p.k / 256 / p.splits, items = p.tiles * p.splits;
  const uint32_t units = int(blockIdx.x) < items ? uint32_t((items - 1 - int(blockIdx.x)) / int(gridDim.x) + 1) : 0u;  // items of this CTA
  constexpr uint32_t kDBuffers = 2 / NMAT;  // a pair's accumulators take both
  volatile int* abortFlag = &ctl.abort;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.slotFree[s], 8);  // the warps of the two groups that share a super-block
    }
    for (int s = 0; s < kActStages; ++s) {
      mbar_init(&ctl.actFull[s], 1);
      mbar_init(&ctl.actFree[s], 1);
    }
    for (uint32_t b = 0; b < kABuffers; ++b) {
      mbar_init(&ctl.aReady[b], 4);  // the warps of one dequant group
      mbar_init(&ctl.aFree[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl.dReady[b], 1);
      mbar_init(&ctl.dFree[b], 4);
    }
    ctl.abort = 0;
    mbar_fence_init();
  }
  if (warp == 1)
    tmem_alloc(&ctl.tmemBase, kTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = ctl.tmemBase;

  if (warp == 0) {
    // ---------------- producer: one weight slab and two activation halves per super-block ----------------
    const uint32_t halfBytes = uint32_t(p.actRows) * 256;  // 8 k-steps x [actRows x 16] fp16
    uint32_t it = 0, slabs = 0, halves = 0;  // slabs, halves: copies issued
    bool ok = true, waited = false;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const int tile = item % p.tiles, firstBlock = (item / p.tiles) * blocksPerRow;
      int segment = 0;
      while (segment + 1 < p.nseg && tile >= p.seg[segment + 1].tile0)
        ++segment;
      const int row0 = (tile - p.seg[segment].tile0) * kRows;
      if (elect_one())  // the same lane every time: it keeps the counters
        for (int sb = firstBlock; sb < firstBlock + blocksPerRow && ok; ++sb, ++it) {
          for (int mat = 0; mat < NMAT && ok; ++mat) {
            const uint32_t slab = it * NMAT + mat, slot = slab % kStages, round = slab / kStages;
            if (round > 0)
              ok = mbar_wait_bounded(&ctl.slotFree[slot], (round - 1) & 1, abortFlag);
            if (ok) {
              mbar_arrive_expect_tx(&ctl.full[slot], kSlabBytes);
              tma_load_2d(ring + size_t(slot) * kSlabBytes, &p.map[segment][mat], sb * 18, row0, &ctl.full[slot]);
              ++slabs;
            }
          }
          if (!waited) {  // the activations are the preceding kernel's output
            pdl_wait();
            waited = true;
          }
          for (int h = 0; h < 2 && ok; ++h) {  // the two activation halves of this super-block
            const uint32_t half = 2 * it + h, actSlot = half % kActStages, actRound = half / kActStages;
            if (actRound > 0)
              ok = mbar_wait_bounded(&ctl.actFree[actSlot], (actRound - 1) & 1, abortFlag);
            if (ok) {
              mbar_arrive_expect_tx(&ctl.actFull[actSlot], halfBytes);
              bulk_load(actRing + size_t(actSlot) * kActHalfBytes, p.acts + (size_t(sb) * 2 + h) * halfBytes, halfBytes, &ctl.actFull[actSlot]);
              ++halves;
            }
          }
          if (!ok) {
            *abortFlag = 1;
            atomicExch(p.status, kStatusBarrierTimeout);
          }
        }
      ok = __all_sync(0xffffffffu, ok);
    }
    // no copy may be in flight when the CTA ends, whoever gave up
    if (elect_one()) {
      for (uint32_t i = slabs > uint32_t(kStages) ? slabs - kStages : 0; i < slabs; ++i)
        mbar_wait_bounded(&ctl.full[i % kStages], (i / kStages) & 1, abortFlag);
      for (uint32_t i = halves > uint32_t(kActStages) ? halves - kActStages : 0; i < halves; ++i)
        mbar_wait_bounded(&ctl.actFull[i % kActStages], (i / kActStages) & 1, abortFlag);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (one lane) ----------------
    if (elect_one()) {
      uint32_t it = 0, unit = 0;
      bool ok = true;
      const uint32_t instruction = instruction_descriptor(p.actRows), stepBytes = uint32_t(p.actRows) * 32;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++unit) {
        const uint32_t buffer = unit % kDBuffers;
        if (unit >= kDBuffers)
          ok = mbar_wait_bounded(&ctl.dFree[buffer], (unit / kDBuffers - 1) & 1, abortFlag);
        for (int j = 0; j < blocksPerRow && ok; ++j, ++it) {
          for (int turn = 0; turn < 2 * NMAT && ok; ++turn) {  // eight k-steps per half of a super-block, of one matrix and the other
            const uint32_t mat = turn >> 1, h = turn & 1, act = 2 * it + h, half = 2 * (it * NMAT + mat) + h, actSlot = act % kActStages, aBuffer = half % kABuffers;
            const uint32_t dColumn = tmem + kColD + (NMAT == 2 ? mat : buffer) * 128;
            ok = mbar_wait_bounded(&ctl.aReady[aBuffer], (half / kABuffers) & 1, abortFlag) &&
                 mbar_wait_bounded(&ctl.actFull[actSlot], (act / kActStages) & 1, abortFlag);
            if (!ok)
              break;
            fence_after_sync();
            const uint32_t actBase = smem_u32(actRing + size_t(actSlot) * kActHalfBytes);
#pragma unroll
            for (int step = 0; step < 8; ++step)
              umma_ts(dColumn, tmem + kColA + aBuffer * 64 + step * 8, smem_descriptor(actBase + step * stepBytes, 128, 256), instruction,
                      (j | h | step) != 0);
            if (mat == NMAT - 1)
              umma_commit(&ctl.actFree[actSlot]);
            umma_commit(&ctl.aFree[aBuffer]);
          }
          if (!ok)
            break;
          if (j == blocksPerRow - 1)
            umma_commit(&ctl.dReady[buffer]);
        }
      }
      if (!ok) {
        *abortFlag = 1;
        atomicExch(p.status, kStatusBarrierTimeout);
      }
    }
  } else if (warp >= 4 && warp < 4 + 4 * GROUPS) {
    // ---------------- dequant: thread = weight row; a group takes one half of every super-block (two groups) or of every
    // second one (four). A lies in tensor memory as a ring of four halves, so a group fills one while the MMAs of another run.
    // See umma_launch for which.
    const int group = (warp - 4) >> 2, side = group & 1, quadrant = warp & 3, row = quadrant * 32 + lane;
    constexpr uint32_t k1024 = 0x64006400u;
    uint32_t it = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x)
      for (int j = 0; j < blocksPerRow * NMAT && ok; ++j, ++it) {  // of a pair, the matrices in turn
        if (GROUPS == 4 && (it & 1) != uint32_t(group >> 1))
          continue;
        const uint32_t slot = it % kStages, round = it / kStages, half = 2 * it + side, aBuffer = half % kABuffers;
        ok = mbar_wait_bounded(&ctl.full[slot], round & 1, abortFlag);
        if (ok && half >= kABuffers)
          ok = mbar_wait_bounded(&ctl.aFree[aBuffer], (half / kABuffers - 1) & 1, abortFlag);
        if (!ok)
          break;
        fence_after_sync();
        const uint8_t* block = ring + size_t(slot) * kSlabBytes + row * 144;
        const uint4 header = *reinterpret_cast<const uint4*>(block);
        const uint4* const quants = reinterpret_cast<const uint4*>(block + 16 + 64 * side);
        uint4 quads[4];  // read ahead where other warps wait for the same pipe (a pair with 128 rows 37.3 -> 35.0 us; with two groups 1 % slower)
        if (GROUPS == 4)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            quads[i] = quants[i];
        const float2 dm = __half22float2(*reinterpret_cast<const __half2*>(&header.x));
        // 6-bit scales / mins of this half's four sub-blocks (scale_min_k4, quant_linear.metal:12-20)
        const uint32_t scales = side == 0 ? header.y & 0x3f3f3f3fu : (header.w & 0x0f0f0f0fu) | ((header.y >> 2) & 0x30303030u);
        const uint32_t mins = side == 0 ? header.z & 0x3f3f3f3fu : ((header.w >> 4) & 0x0f0f0f0fu) | ((header.z >> 2) & 0x30303030u);
        const uint32_t aAddress = tmem + (uint32_t(quadrant * 32) << 16) + kColA + aBuffer * 64;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t pair = (scales >> (16 * t)) & 0xffffu, minPair = (mins >> (16 * t)) & 0xffffu;
          const uint4 q0 = GROUPS == 4 ? quads[2 * t] : quants[2 * t], q1 = GROUPS == 4 ? quads[2 * t + 1] : quants[2 * t + 1];
          const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
          // dequantised weight d*sc*q - dmin*m, in fp16: q is made exact first, then one fused multiply-add
          const uint32_t sL = pack_half2(dm.x * float(pair & 0xffu), dm.x * float(pair & 0xffu));
          const uint32_t sH = pack_half2(dm.x * float(pair >> 8), dm.x * float(pair >> 8));
          const uint32_t nL = pack_half2(-dm.y * float(minPair & 0xffu), -dm.y * float(minPair & 0xffu));
          const uint32_t nH = pack_half2(-dm.y * float(minPair >> 8), -dm.y * float(minPair >> 8));
          uint32_t v[32];
#pragma unroll
          for (int w = 0; w < 8; ++w) {
            const uint32_t a = words[w];
            v[2 * w] = hfma2_u32(hsub2_u32((a & 0x000f000fu) | k1024, k1024), sL, nL);
            v[2 * w + 1] = hfma2_u32(hsub2_u32(((a >> 8) & 0x000f000fu) | k1024, k1024), sL, nL);
            v[16 + 2 * w] = hfma2_u32(hsub2_u32(((a >> 4) & 0x000f000fu) | k1024, k1024), sH, nH);
            v[16 + 2 * w + 1] = hfma2_u32(hsub2_u32(((a >> 12) & 0x000f000fu) | k1024, k1024), sH, nH);
          }
          tmem_store32(aAddress + 32 * t, v);
        }
          tmem_wait_store();
        fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&ctl.aReady[aBuffer]);
          mbar_arrive(&ctl.slotFree[slot]);
        }
      }
    if (ok && units > 0) {
      // their share of the CTA's last accumulator (see the epilogue warps): groups of eight activation rows 1 + group,
      // 2 + GROUPS + group, ...; the accumulator has no later user, so nobody waits for these reads
      const uint32_t unit = units - 1, buffer = unit % kDBuffers;
      pdl_wait();
      ok = mbar_wait_bounded(&ctl.dReady[buffer], (unit / kDBuffers) & 1, abortFlag);
      if (ok) {
        fence_after_sync();
        const int lastItem = int(blockIdx.x) + int(units - 1) * int(gridDim.x);
        store_accumulator<NMAT>(p, lastItem, tmem + (uint32_t(quadrant * 32) << 16) + kColD + buffer * 128, row, 1 + group, 1 + GROUPS);
      }
    }
    if (!ok && lane == 0) {
      *abortFlag = 1;
      atomicExch(p.status, kStatusBarrierTimeout);
    }
  } else if (warp >= 4 + 4 * GROUPS) {
    // ---------------- epilogue: thread = weight row ----------------
    pdl_wait();  // residuals, results and the partial-sum buffer belong to earlier kernels
    const int quadrant = warp & 3, row = quadrant * 32 + lane;
    const uint32_t laneBase = tmem + (uint32_t(quadrant * 32) << 16) + kColD;
    uint32_t unit = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++unit) {
      const uint32_t buffer = unit % kDBuffers;
      ok = mbar_wait_bounded(&ctl.dReady[buffer], (unit / kDBuffers) & 1, abortFlag);
      if (!ok)
        break;
      fence_after_sync();
      // the CTA's last accumulator: the dequant warps, idle by then, take most of it
      store_accumulator<NMAT>(p, item, laneBase + buffer * 128, row, 0, unit + 1 == units ? 1 + GROUPS : 1);
      fence_before_sync();
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&ctl.dFree[buffer]);
    }
    if (!ok && lane == 0) {
      *abortFlag = 1;
      atomicExch(p.status, kStatusBarrierTimeout);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 1)
    tmem_dealloc(tmem, kTmemCols);
}

// Lays the activations out as the B operand, per 256-wide super-block: [16 k-steps][16 row groups][2 K halves][8 rows]
// [8 values] fp16, rows rounded to fp16, rows from m up zero. K inside a step follows the order in which the
// dequantiser emits weights: step s covers the quant bytes of 64-group t = s / 4, nibble side (s / 2) % 2, words
// 4 * (s % 2) .. +3; TMEM column c of a step holds the nibbles of bytes (c % 2, c % 2 + 2) of word c / 2. Eight
// consecutive k of a super-block are thus one 16-byte core-matrix row of a k-step (in the order 0,2,1,3,4,6,5,7), and a
// thread turns two float4 loads into one 16-byte store.
// grid (k / 256, actRows / 8), 256 threads: actRows x 32 groups of eight per super-block, one per thread; a warp reads
// one activation row's 256 values.
__global__ void __launch_bounds__(256) umma_prepare_rows_kernel(const float* x, int ldx, int m, int actRows, __half* acts) {
  pdl_launch_dependents();
  pdl_wait();
  const int sb = blockIdx.x;
  __half* out = acts + size_t(sb) * (actRows * 256);
  {
    const int item = blockIdx.y * 256 + threadIdx.x, n = item >> 5, group = item & 31;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (n < m) {
      const float4* src = reinterpret_cast<const float4*>(x + size_t(n) * ldx + size_t(sb) * 256 + group * 8);
      a = src[0], b = src[1];
    }
    const __half2 h0 = __floats2half2_rn(a.x, a.z), h1 = __floats2half2_rn(a.y, a.w), h2 = __floats2half2_rn(b.x, b.z), h3 = __floats2half2_rn(b.y, b.w);
    uint4 packed;
    packed.x = *reinterpret_cast<const uint32_t*>(&h0), packed.y = *reinterpret_cast<const uint32_t*>(&h1);
    packed.z = *reinterpret_cast<const uint32_t*>(&h2), packed.w = *reinterpret_cast<const uint32_t*>(&h3);
    *reinterpret_cast<uint4*>(out + size_t(group >> 1) * (actRows * 16) + (n >> 3) * 128 + (group & 1) * 64 + (n & 7) * 8) = packed;
  }
}

// y = partial[0] + partial[1] + ... (+ residual), four values per thread.
__global__ void __launch_bounds__(256) umma_reduce_kernel(const float* partial, int splits, size_t count, const float* residual, float* y) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t at = (size_t(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (at >= count)
    return;
  float4 sum = *reinterpret_cast<const float4*>(partial + at);
  for (int s = 1; s < splits; ++s) {
    const float4 v = *reinterpret_cast<const float4*>(partial + s * count + at);
    sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
  }
  if (residual) {
    const float4 v = *reinterpret_cast<const float4*>(residual + at);
    sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
  }
  *reinterpret_cast<float4*>(y + at) = sum;
}

template <int NMAT, int GROUPS> cudaError_t launch_tiles(const UmmaParams& params, const float* x, int ldx, int sms, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (const cudaError_t e = configure_shared_memory(umma_linear_kernel<NMAT, GROUPS>, kSharedBytes, configured))
    return e;
  // The MMA is as wide as the launch has rows, in steps of 16: a speculative pass of 40 rows moves 24 KB of activations
  // per super-block instead of 64 KB and spends a third of the tensor time.
  UmmaParams p = params;
  p.actRows = (p.m + 15) / 16 * 16;
  launch_kernel<1>(umma_prepare_rows_kernel, dim3(p.k / 256, p.actRows / 8), 256, 0, stream, x, ldx, p.m, p.actRows,
                reinterpret_cast<__half*>(const_cast<uint8_t*>(p.acts)));
  const int items = p.tiles * p.splits, grid = items < sms ? items : sms;
  launch_kernel<1>(umma_linear_kernel<NMAT, GROUPS>, grid, kThreads<GROUPS>, kSharedBytes, stream, p);
  if (p.splits > 1) {
    const size_t count = size_t(p.m) * p.seg[0].ldy;
    launch_kernel<1>(umma_reduce_kernel, unsigned((count / 4 + 255) / 256), 256, 0, stream, p.partial, p.splits, count, p.seg[0].res, p.seg[0].y);
  }
  return cudaGetLastError();
}

}  // namespace

// 9 to 128 activation rows (p.m), rows of x `ldx` floats apart (a multiple of 4).
cudaError_t umma_launch(bool pair, const UmmaParams& p, const float* x, int ldx, int sms, cudaStream_t stream) {
  // Two dequant groups take a half of every super-block each, four of every second one. A pair wants four (12288 x 4096 with 9, 40 and
  // 64 rows 28.8, 30.1 and 32.0 us, with two 32.4, 33.9 and 35.6): its activations come once for two super-blocks, so the dequantisation is what
  // the MMAs wait for. One matrix with few rows wants two, which start and drain faster (4096 x 12288 with 9 and 64 rows 17.6 and 20.5,
  // with four 18.7 and 21.1); with 128 rows four keep up with the MMAs (projections of a layer 124.6 us, with two 128.6).
  if (pair)
    return launch_tiles<2, 4>(p, x, ldx, sms, stream);
  return p.m > 96 ? launch_tiles<1, 4>(p, x, ldx, sms, stream) : launch_tiles<1, 2>(p, x, ldx, sms, stream);
}

}  // namespace infdev
