// What the persistent GEMV kernels (gemv.cu, q4k_decode.cu) share: the control block of the ring of weight slabs, and the warps
// that add up the partial sums of a tile.
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace infdev {

constexpr int kMaxStages = 12, kMaxFinishers = 3;

struct RingControl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t partialReady[kMaxFinishers], partialFree[kMaxFinishers];  // per partial-sum buffer: consumers -> its finisher and back
  int abort;
};
constexpr int kRingControlBytes = 256;
static_assert(sizeof(RingControl) <= kRingControlBytes, "control block overlaps what follows it");

__device__ __forceinline__ int find_segment(const GemvParams& p, int tile) {
  int s = 0;
  while (s + 1 < p.nseg && tile >= p.seg[s + 1].tile0)
    ++s;
  return s;
}

// The partial sums of a tile go through one of FINISHERS buffers, taken in turn within a K chunk, and each buffer has
// its own finisher warp and two mbarriers: partialReady[b] "every consumer warp has stored its partial sums" and
// partialFree[b] "the finisher has read them", which a consumer tests before it stores into the buffer again.
// Nobody waits for a warp of its own role, each barrier is watched phase by phase by the same warps, and a tile of
// the result has the same finisher in every K chunk, so the sum over the earlier chunks it adds is its own store.
// `partial`: [buffer][matrix][consumer warp][lane] float4.
template <int NMAT, int CONSUMERS, int FINISHERS>
__device__ __forceinline__ void finish_tiles(const GemvParams& p, RingControl& ctl, const float* partial, int buffer, int chunks, int lane) {
  volatile int* abortFlag = &ctl.abort;
  uint32_t uses = 0;
  for (int chunk = 0; chunk < chunks; ++chunk)
    for (int tile = blockIdx.x + buffer * gridDim.x; tile < p.tiles; tile += FINISHERS * gridDim.x, ++uses) {
      // Lane (g = lane/4, t = lane%4) sums what the same lane of every consumer warp holds: weight rows g and g+8 for
      // activation rows 2t and 2t+1. What is added to them (the residual, or the sum over the earlier K chunks) is
      // fetched before the wait.
      const GemvSeg& seg = p.nseg == 1 ? p.seg[0] : p.seg[find_segment(p, tile)];
      const int g = lane >> 2, t = lane & 3;
      float* destination[2] = {nullptr, nullptr};  // activation rows 2t, 2t+1 at weight row g; g + 8 is 8 floats on
      float addend[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (2 * t + r < p.m) {
          const size_t at = size_t(2 * t + r) * seg.ldy + size_t(tile - seg.tile0) * kGemvTileRows + g;
          destination[r] = seg.y + at;
          if (NMAT == 1 && chunk > 0)
            addend[r] = destination[r][0], addend[2 + r] = destination[r][8];
          else if (NMAT == 1 && seg.res)
            addend[r] = seg.res[at], addend[2 + r] = seg.res[at + 8];
        }
      const float4* sums = reinterpret_cast<const float4*>(partial + size_t(buffer) * NMAT * CONSUMERS * 128) + lane;
      if (!mbar_wait_bounded(&ctl.partialReady[buffer], uses & 1, abortFlag)) {
        *abortFlag = 1;
        atomicExch(p.status, kStatusBarrierTimeout);
        return;
      }
      float4 sum[NMAT];
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;  // two chains in a fixed order: the result does not depend on timing
#pragma unroll
        for (int w = 0; w < CONSUMERS; w += 2) {
          const float4 u = sums[(mat * CONSUMERS + w) * 32], v = sums[(mat * CONSUMERS + w + 1) * 32];
          a.x += u.x, a.y += u.y, a.z += u.z, a.w += u.w;
          b.x += v.x, b.y += v.y, b.z += v.z, b.w += v.w;
        }
        sum[mat] = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
      }
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&ctl.partialFree[buffer]);
      const float4 first = sum[0], second = sum[NMAT - 1];
      const float lowRows[2] = {NMAT == 2 ? silu_f(first.x) * second.x : first.x + addend[0], NMAT == 2 ? silu_f(first.y) * second.y : first.y + addend[1]};
      const float highRows[2] = {NMAT == 2 ? silu_f(first.z) * second.z : first.z + addend[2], NMAT == 2 ? silu_f(first.w) * second.w : first.w + addend[3]};
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (destination[r])
          destination[r][0] = lowRows[r], destination[r][8] = highRows[r];
    }
}

}  // namespace infdev
