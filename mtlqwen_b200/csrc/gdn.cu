// Gated delta-rule (GDN) layer kernels.
//
// gdn_prepare_kernel <- gdn_ba_prepare_4096x32 (native_ops.metal:89-113) and gdn_causal_conv_silu
//                      (fused_kernels.metal:202-232) in one launch
// delta_rule_kernel <- delta_rule_decode (delta_rule.metal:256-363) for every query length, fused with
//                      gated_rms_norm_128 (fused_kernels.metal:234-254).
//
// The recurrence keeps the whole 128x128 fp32 state of one (sequence, value head) in the registers of one
// CTA (256 threads x 64 values): it is read from HBM once, updated for every token of the query, and
// written once (or once per token for speculative queries, whose every row must stay selectable). The
// reference makes two passes over the state in device memory per token (delta_rule.metal:320-333, 351-360).
#include <cuda_bf16.h>
#include <algorithm>
#include "act_image.cuh"
#include "kernels.h"
#include "ops.h"

namespace infdev {
namespace {

constexpr int kChannels = 8192, kHeadDim = 128, kValueHeads = 32, kKeyHeads = 16;
constexpr uint32_t kUnbound = 0xffffffffu;

// The four products of a gate dot-product step with the roundings spelled out: the preparation kernel and the fused
// decode kernel must agree bit for bit (a token's result may not depend on which kind of pass computed it), and the
// compiler is otherwise free to contract a.x*b.x + a.y*b.y + ... differently in the two.
__device__ __forceinline__ float dot4(const float4& a, const float4& b) {
  return __fmaf_rn(a.w, b.w, __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x))));
}

__device__ __forceinline__ const infdev_query& query_of_row(const infdev_query* queries, uint32_t row) {
  while (row >= queries->start + queries->count)
    ++queries;
  return *queries;
}

// warp_sum of COUNT sums, in its order, but a lane goes on with one half of them and leaves the other to its partner: 62 exchanges instead of 320 for
// 64 sums (preparation of 2411 rows 106.7 -> 101.2 us). Lane l is left with the sums from l x COUNT / 32 on: two of 64, otherwise one.
template <int COUNT, int PARTNER, int SIZE> __device__ __forceinline__ void share_sums(float (&sum)[SIZE], int lane) {
  if constexpr (PARTNER > 0) {
    constexpr int kLeft = COUNT > 1 ? COUNT / 2 : 1;
    const bool upper = lane & PARTNER;
#pragma unroll
    for (int o = 0; o < kLeft; ++o) {
      if constexpr (COUNT > 1) {
        const float other = __shfl_xor_sync(0xffffffffu, upper ? sum[o] : sum[o + kLeft], PARTNER);
        sum[o] = (upper ? sum[o + kLeft] : sum[o]) + other;
      } else {
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], PARTNER);
      }
    }
    share_sums<kLeft, PARTNER / 2>(sum, lane);
  }
}

// gdn_prepare_kernel: both preparation steps of a GDN layer in one launch of 256-thread CTAs.
//  * CTAs [0, gateBlocks): beta / g of eight rows and GATE_HEADS of the 32 value heads. Warps 0..3 share the 4096-long dot
//    products with wBeta (a quarter each), warps 4..7 those with wAlpha; a warp keeps a tile of rows x heads of partial
//    sums in registers, so a row fetched once meets eight weight rows and the other way round. With one head per CTA the
//    kernel pulled 2.5 GB through the L2 for 2411 rows.
//  * the others: causal conv + SiLU of CONV_ROWS packed rows and 1024 channels, four channels per thread. A thread walks
//    the rows with the last three inputs of its channels in registers: every input is loaded once (a thread per output
//    element loaded each four times and searched the query table for each: together with the gates 339 us for 2411 rows,
//    where reading and writing everything once takes 30). State layout: conv taps fp32 [8192][4] at record + stateOffset.
// CONV_ROWS rows per thread and GATE_HEADS heads per CTA (the sums are the same whatever they are): the rows of short prompt pieces are spread
// thinly, so that no thread has a long chain of them; with more rows an SM, which holds two CTAs, would take them in several turns.
// 1 and 1, 2 and 2, 4 and 4, 8 and 8: 24 rows 5.7 / 5.8 / 6.7 / 9.8 us, 32 rows 7.6 / 5.7 / 5.7 / 8.7, 48 rows 8.8 / 5.7 / 6.2 / 8.8, 64 rows 10.3 / 7.7 /
// 6.7 / 8.8, 128 rows 15.9 / 10.9 / 8.8 / 9.8, 160 rows 18.5 / 12.4 / 10.3 / 10.8, 192 rows 21.6 / 13.9 / 11.4 / 10.8, 512 rows 50 / 31 / 23.2 / 21.1.
// What bounds the last is instructions: the parts of 2411 rows, each alone, issue 2.8 a cycle in 46 and 39 us, 45 for a value of the convolution
// (its division and exponential are most of them). The gates' operands through shared memory by cp.async 103.9 us, the convolution as a launch of
// more and smaller blocks 102.1, gates and convolution side by side on an SM 121, as below 93.5.
// ALIGNED: mixed, convWeight, q, k and v lie on 16-byte boundaries; without, they are read and written value by value.
constexpr int kGateRows = 8, kPrepareRows1 = 24, kPrepareRows2 = 48, kPrepareRows4 = 176;  // most rows of each spread
constexpr int kConvChannels = 4 * 256;  // per CTA

template <bool ALIGNED> __device__ __forceinline__ float4 load_four(const float* p) {
  return ALIGNED ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

template <int CONV_ROWS, int GATE_HEADS, bool ALIGNED>
__global__ void __launch_bounds__(256, 2) gdn_prepare_kernel(const float* x, const float* wBeta, const float* wAlpha, const float* A, const float* dt,
                                                          const float* mixed, const float* w, const infdev_query* queries, int rows, int gateBlocks,
                                                          uint64_t stateOffset, uint64_t stateBytes, float* q, float* k, float* v, float* beta,
                                                          float* g) {
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  if (int(blockIdx.x) < gateBlocks) {
    constexpr int kHeadGroups = kValueHeads / GATE_HEADS;
    const int row0 = (blockIdx.x / kHeadGroups) * kGateRows, head0 = (blockIdx.x % kHeadGroups) * GATE_HEADS;
    const int live = min(kGateRows, rows - row0);
    const int warp = tid >> 5, lane = tid & 31, which = warp >> 2, quarter = warp & 3;
    const float* weights = (which ? wAlpha : wBeta) + size_t(head0) * 4096 + quarter * 1024 + lane * 4;
    const float* src = x + size_t(row0) * 4096 + quarter * 1024 + lane * 4;
    constexpr int kSums = kGateRows * GATE_HEADS;
    float sum[kSums];
#pragma unroll
    for (int o = 0; o < kSums; ++o)
      sum[o] = 0.f;
#pragma unroll 2
    for (int i = 0; i < 8; ++i) {
      float4 a[kGateRows];
#pragma unroll
      for (int r = 0; r < kGateRows; ++r)
        a[r] = r < live ? *reinterpret_cast<const float4*>(src + size_t(r) * 4096 + i * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int h = 0; h < GATE_HEADS; ++h) {
        const float4 b = *reinterpret_cast<const float4*>(weights + size_t(h) * 4096 + i * 128);
#pragma unroll
        for (int r = 0; r < kGateRows; ++r)
          sum[r * GATE_HEADS + h] += dot4(a[r], b);
      }
    }
    share_sums<kSums, 16>(sum, lane);
    __shared__ float parts[kSums][8];
#pragma unroll
    for (int o = 0; o < (kSums + 31) / 32; ++o)
      parts[lane * kSums / 32 + o][warp] = sum[o];  // fewer than 32: several lanes have the same one
    __syncthreads();
    if (tid < 2 * kSums) {
      const int r = (tid / GATE_HEADS) % kGateRows, head = head0 + tid % GATE_HEADS;
      if (r < live) {
        const float* p = parts[tid % kSums] + (tid < kSums ? 0 : 4);
        const float dot = (p[0] + p[1]) + (p[2] + p[3]);
        if (tid < kSums)
          beta[(row0 + r) * kValueHeads + head] = 1.0f / (1.0f + expf(-dot));
        else
          g[(row0 + r) * kValueHeads + head] = A[head] * logf(1.0f + expf(dot + dt[head]));
      }
    }
    return;
  }
  const int item = blockIdx.x - gateBlocks, row0 = (item / (kChannels / kConvChannels)) * CONV_ROWS, last = min(rows, row0 + CONV_ROWS);
  const int c = (item % (kChannels / kConvChannels)) * kConvChannels + 4 * tid;
  float4 input[CONV_ROWS];
#pragma unroll
  for (int i = 0; i < CONV_ROWS; ++i)
    if (row0 + i < last)
      input[i] = load_four<ALIGNED>(mixed + size_t(row0 + i) * kChannels + c);
  // The three inputs before this one, oldest first: asked for before it is known whether they are of the same query (101.2 -> 98.4 us).
  float4 window[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
    window[r] = row0 - 3 + r >= 0 ? load_four<ALIGNED>(mixed + size_t(row0 - 3 + r) * kChannels + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 weight[4];  // of the thread's four channels, oldest tap first
#pragma unroll
  for (int j = 0; j < 4; ++j)
    weight[j] = load_four<ALIGNED>(w + size_t(c + j) * 4);
  float* const out = c < 2048 ? q + c : c < 4096 ? k + (c - 2048) : v + (c - 4096);
  const size_t pitch = c < 4096 ? 2048 : 4096;
  const infdev_query* info = &query_of_row(queries, uint32_t(row0));
  // Kept: the stores below would have them read again for every row (98.4 -> 93.5 us).
  int start = int(info->start), end = start + int(info->count);
  bool enter = row0 - 3 < start, speculative = info->state != kUnbound;
#pragma unroll
  for (int i = 0; i < CONV_ROWS; ++i) {
    const int row = row0 + i;
    if (row >= last)
      break;
    if (row >= end) {
      info = &query_of_row(info, uint32_t(row));
      start = int(info->start), end = start + int(info->count), speculative = info->state != kUnbound;
      enter = true;
    }
    const int p = row - start;
    if (enter) {
      // the window at position p of this query: earlier rows of the query, before them the taps of the state record
      const float* prev = reinterpret_cast<const float*>(info->previous + stateOffset) + size_t(c) * 4;
      float4 taps[4];
      if (p < 3)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          taps[j] = info->previous ? load_four<ALIGNED>(prev + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int position = p - 3 + r;  // tap position + 4 of the record (1 .. 3) when negative
        if (position >= 0)
          window[r] = load_four<ALIGNED>(mixed + size_t(start + position) * kChannels + c);
        else if (position == -3)
          window[r] = make_float4(taps[0].y, taps[1].y, taps[2].y, taps[3].y);
        else if (position == -2)
          window[r] = make_float4(taps[0].z, taps[1].z, taps[2].z, taps[3].z);
        else
          window[r] = make_float4(taps[0].w, taps[1].w, taps[2].w, taps[3].w);
      }
      enter = false;
    }
    const float4 now = input[i];
    auto tap = [](const float4& weights, float a, float b, float d, float e) {
      return silu_f(fmaf(e, weights.w, fmaf(d, weights.z, fmaf(b, weights.y, fmaf(a, weights.x, 0.f)))));
    };
    const float4 result =
        make_float4(tap(weight[0], window[0].x, window[1].x, window[2].x, now.x), tap(weight[1], window[0].y, window[1].y, window[2].y, now.y),
                    tap(weight[2], window[0].z, window[1].z, window[2].z, now.z), tap(weight[3], window[0].w, window[1].w, window[2].w, now.w));
    float* const to = out + size_t(row) * pitch;
    if (ALIGNED)
      *reinterpret_cast<float4*>(to) = result;
    else
      to[0] = result.x, to[1] = result.y, to[2] = result.z, to[3] = result.w;
    if (speculative || row + 1 == end) {
      float4* state = reinterpret_cast<float4*>(info->next + stateOffset + (speculative ? uint64_t(p) * stateBytes : 0)) + c;
      state[0] = make_float4(window[0].x, window[1].x, window[2].x, now.x);
      state[1] = make_float4(window[0].y, window[1].y, window[2].y, now.y);
      state[2] = make_float4(window[0].z, window[1].z, window[2].z, now.z);
      state[3] = make_float4(window[0].w, window[1].w, window[2].w, now.w);
    }
    window[0] = window[1], window[1] = window[2], window[2] = now;
  }
}

// The queries that the chunked kernel takes.
__device__ __forceinline__ bool chunked(const infdev_query& info, uint32_t chunkedFrom) { return chunkedFrom && info.state == kUnbound && info.count >= chunkedFrom; }
// How many they are among up to 32; more count as 32. Every lane of a warp calls.
__device__ __forceinline__ uint32_t chunked_queries(const infdev_query* queries, uint32_t count, uint32_t chunkedFrom) {
  const uint32_t lane = threadIdx.x & 31;
  return count > 32 ? 32 : __popc(__ballot_sync(0xffffffffu, lane < count && chunked(queries[lane], chunkedFrom)));
}

// gated_rms_norm_128 of one head of a query's rows, in place: eight warps, eight rows each at a time, in turn with the CTAs of the grid's third dimension.
// Not inlined: delta_rule_kernel<false>, whose launch this is, would keep fewer registers for its own queries (68 bytes of spills instead of 24; 12 rows
// 24.7 us instead of 23.9, 215 instead of 211.6 for 128).
// The squares are added in the order in which the chunked kernel with the norm in its chain has them, columns c and c + 8 first, then the eight pairs of
// 16 columns by halves, then the eight 16s one after the other, so the bits do not depend on which of the two norms a call takes. Rows are halved between
// lanes as in share_sums: 41 exchanges for eight rows, where warp_sum takes 40 in its own order.
__device__ __noinline__ void gated_norm_rows(float* out, const float* z, const float* normWeight, uint32_t start, uint32_t count, int head) {
  constexpr uint32_t kRows = 8;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr size_t kPitch = size_t(kValueHeads) * kHeadDim;
  float weight[4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
    weight[c] = normWeight[lane + 32 * c];
  for (uint32_t first = (blockIdx.z * 8 + warp) * kRows; first < count; first += gridDim.z * 8 * kRows) {
    float o[kRows][4], gate[kRows][4];
    const size_t at = size_t(start + first) * kPitch + size_t(head) * kHeadDim + lane;
#pragma unroll
    for (uint32_t r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        o[r][c] = first + r < count ? out[at + r * kPitch + 32 * c] : 0.f;
        gate[r][c] = first + r < count ? z[at + r * kPitch + 32 * c] : 0.f;
      }
    // lanes with bit 3 go on with columns 64 .. 127 and leave the others to their partners, eight columns off
    const bool high = lane & 8;
    float pairs[kRows][2];
#pragma unroll
    for (uint32_t r = 0; r < kRows; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float other = __shfl_xor_sync(0xffffffffu, high ? o[r][e] : o[r][e + 2], 8), own = high ? o[r][e + 2] : o[r][e];
        const float low8 = high ? other : own, high8 = high ? own : other;
        pairs[r][e] = __fmaf_rn(high8, high8, __fmul_rn(low8, low8));
      }
#pragma unroll
    for (uint32_t partner = 1; partner < 8; partner *= 2) {
      const uint32_t left = kRows / 2 / partner;
      const bool upper = lane & partner;
#pragma unroll
      for (uint32_t r = 0; r < left; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float other = __shfl_xor_sync(0xffffffffu, upper ? pairs[r][e] : pairs[r + left][e], partner);
          pairs[r][e] = (upper ? pairs[r + left][e] : pairs[r][e]) + other;
        }
    }
    // 16 columns each: 32 c + 16 (bit 4) of the row that bits 0, 1 and 2 name, c = e or, with bit 3, e + 2
    float even[2], odd[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float other = __shfl_xor_sync(0xffffffffu, pairs[0][e], 16);
      even[e] = lane & 16 ? other : pairs[0][e], odd[e] = lane & 16 ? pairs[0][e] : other;
    }
    const float below = __shfl_xor_sync(0xffffffffu, ((even[0] + odd[0]) + even[1]) + odd[1], 8);
    const float total = (((below + even[0]) + odd[0]) + even[1]) + odd[1];  // of lanes with bit 3
    const float scales = rsqrtf(total / float(kHeadDim) + 1.0e-6f);
#pragma unroll
    for (uint32_t r = 0; r < kRows; ++r) {
      const float scale = __shfl_sync(0xffffffffu, scales, 8 | (r >> 2 & 1) | (r >> 1 & 1) << 1 | (r & 1) << 2);
      if (first + r < count)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          out[at + r * kPitch + 32 * c] = o[r][c] * scale * weight[c] * silu_f(gate[r][c]);
    }
  }
}

// grid (32 value heads, queries), 256 threads. Thread (part = tid/32, lane) owns S[k][4*lane .. 4*lane+3]
// for k = part + 8*i, i < 16.
// `image`, when not null, also receives the activation image of `out`. A 256-value block holds two heads, which two
// CTAs produce: each adds one to the block's entry in `counters` (zero between launches) after its stores, and the
// second to arrive reads both halves back and writes the block's image, then clears the entry.
// FUSED: the preparation of gdn_prepare_kernel happens here as well, for this CTA's channels only: the conv + SiLU of
// its 128 q, k and v channels (the taps of the q / k channels are written by the first of the two value heads that
// share a key head) and its beta / g dot products, with the same arithmetic and summation order; q, k, v, g, beta
// are then not read. One launch less per layer for passes without prefill chunks.
//
// What bounds a decode launch is latency, not bytes: all 256 CTAs are resident at once, so the time is the longest
// dependent chain of one CTA. The kernel therefore asks for everything up front and keeps block-wide barriers to two per
// token:
//  * before griddepcontrol.wait, like the weights of every kernel here, the gate-projection rows of the head go to shared
//    memory with cp.async (no registers held while in flight). So do the conv weights and taps, and the 64 KB state goes
//    to registers: before the wait too where the caller vouches that the preceding kernel writes neither table nor records
//    (`ahead`), else right after it (one call after the other, 4.3 MB a sequence in the L2: one sequence 5.1 us with and 6.1
//    without, four 6.9 and 7.4, eight 8.6 and 9.7; 6.4, 9.1 and 10.3 with the gate rows behind the wait as well). The
//    token's input row follows after the wait. The small operands, which hit the L2, arrive and are consumed while the
//    state is still on its way from HBM.
//  * after the first barrier every thread derives the q / k norms and the two gates itself from the partial sums
//    (redundantly; a second barrier to broadcast them costs more than 256 threads repeating a few instructions);
//  * after the second barrier (partial products with the state) every warp sums the eight partials of its own four
//    columns, so each has delta and the output for them without another barrier; warp 0 alone normalises, gates and
//    stores the 128 outputs and runs the image protocol while the others update and store the state.
struct GdnInputs {
  const float *x, *wBeta, *wAlpha, *A, *dt, *mixed, *convWeight;
  uint64_t convStateOffset;
  bool ahead;  // the query table and the state records may be read before griddepcontrol.wait (see the kernel)
};

struct GdnStage {                      // dynamic shared memory of the fused form
  float4 x[1024];                      // the token's input row (4096 values)
  float4 wBeta[1024], wAlpha[1024];    // this head's rows of the two gate projections
  float4 window[3][kHeadDim];          // conv taps of this CTA's q, k and v channels, rolled forward token by token
  float4 convWeight[3][kHeadDim];
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <bool FUSED>
__global__ void __launch_bounds__(256, 2) delta_rule_kernel(const float* q, const float* k, const float* v, const float* g, const float* beta,
                                                         const float* z, const float* normWeight, const infdev_query* queries,
                                                         uint64_t stateOffset, uint64_t stateBytes, float* out, uint8_t* image, int* counters,
                                                         uint32_t chunkedFrom, GdnInputs in) {
  pdl_launch_dependents();
  // A kernel that is launched early lets its successor go before its own wait, so with a few small ones in a row this one can
  // start while the kernel three or four before it, say the step that writes these records, still runs. The caller knows
  // whether one of the kernels between is not launched early and so bounds how far ahead this one gets.
  extern __shared__ float4 stageRaw[];
  GdnStage& stage = *reinterpret_cast<GdnStage*>(stageRaw);
  if (FUSED) {
    const float4* wb = reinterpret_cast<const float4*>(in.wBeta + size_t(blockIdx.x) * 4096);
    const float4* wa = reinterpret_cast<const float4*>(in.wAlpha + size_t(blockIdx.x) * 4096);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      cp_async16(&stage.wBeta[threadIdx.x + 256 * i], wb + threadIdx.x + 256 * i);
      cp_async16(&stage.wAlpha[threadIdx.x + 256 * i], wa + threadIdx.x + 256 * i);
    }
  }
  if (!in.ahead)
    pdl_wait();
  const infdev_query info = queries[blockIdx.y];
  const int head = blockIdx.x, keyHead = head % kKeyHeads, tid = threadIdx.x, part = tid >> 5, lane = tid & 31;
  const bool speculative = info.state != kUnbound;
  if (!FUSED && chunked(info, chunkedFrom)) {  // delta_rule_chunked_kernel had this query, all but its norm
    if (z && z != out)
      gated_norm_rows(out, z, normWeight, info.start, info.count, head);
    return;
  }
  if (!FUSED && blockIdx.z > 0)
    return;
  __shared__ float qraw[kHeadDim], kraw[kHeadDim], vraw[kHeadDim], red[12], dots[8];
  __shared__ float4 partialPred[8][32], partialQ[8][32];
  const int channels[3] = {keyHead * kHeadDim + (tid & 127), 2048 + keyHead * kHeadDim + (tid & 127), 4096 + head * kHeadDim + (tid & 127)};
  float headA = 0.f, headDt = 0.f;

  if (FUSED) {
    if (tid < kHeadDim) {
      const float4* taps = reinterpret_cast<const float4*>(info.previous + in.convStateOffset);
#pragma unroll
      for (int which = 0; which < 3; ++which) {
        cp_async16(&stage.convWeight[which][tid], reinterpret_cast<const float4*>(in.convWeight) + channels[which]);
        if (info.previous)
          cp_async16(&stage.window[which][tid], taps + channels[which]);
        else
          stage.window[which][tid] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    cp_async_commit();
    headA = in.A[head], headDt = in.dt[head];
  }

  float4 S[16];
  if (info.previous) {
    const float4* src = reinterpret_cast<const float4*>(info.previous + stateOffset) + size_t(head) * kHeadDim * 32;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      S[i] = src[(part + 8 * i) * 32 + lane];
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      S[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (in.ahead)
    pdl_wait();

  for (uint32_t t = 0; t < info.count; ++t) {
    const size_t row = info.start + t;
    const size_t at = (row * kValueHeads + head) * kHeadDim + 4 * lane;  // warp 0: this lane's four outputs
    float qv = 0.f, kv = 0.f, vv = 0.f, decay = 0.f, betaValue = 0.f;
    if (FUSED) {
      float mixedNow[3] = {0.f, 0.f, 0.f};
      if (tid < kHeadDim) {
#pragma unroll
        for (int which = 0; which < 3; ++which)
          mixedNow[which] = in.mixed[row * kChannels + channels[which]];
      }
      const float4* xrow = reinterpret_cast<const float4*>(in.x + row * 4096);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        cp_async16(&stage.x[tid + 256 * i], xrow + tid + 256 * i);
      cp_async_commit();
      cp_async_wait_all();
      __syncthreads();
      // beta / g: warps 0..3 share the dot product with wBeta, warps 4..7 the one with wAlpha (as gdn_prepare_kernel)
      const float4* weights = ((part >> 2) ? stage.wAlpha : stage.wBeta) + (part & 3) * 256;
      const float4* src = stage.x + (part & 3) * 256;
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = src[i * 32 + lane], b = weights[i * 32 + lane];
        sum += dot4(a, b);
      }
      sum = warp_sum(sum);
      if (lane == 0)
        dots[part] = sum;
      if (tid < kHeadDim) {
        // causal conv + SiLU of this head's q, k and v channel `tid` (gdn_causal_conv_silu, fused_kernels.metal:202-232):
        // the window holds the three tokens before this one, oldest first in .y (.x is the tap that falls out)
        float values[3];
#pragma unroll
        for (int which = 0; which < 3; ++which) {
          const float4 taps = stage.window[which][tid], w4 = stage.convWeight[which][tid];
          const float4 context = make_float4(taps.y, taps.z, taps.w, mixedNow[which]);
          float acc = fmaf(context.x, w4.x, 0.f);
          acc = fmaf(context.y, w4.y, acc), acc = fmaf(context.z, w4.z, acc), acc = fmaf(context.w, w4.w, acc);
          values[which] = silu_f(acc);
          stage.window[which][tid] = context;
          if ((speculative || t + 1 == info.count) && (which == 2 || head < kKeyHeads)) {
            float* state = reinterpret_cast<float*>(info.next + in.convStateOffset + (speculative ? uint64_t(t) * stateBytes : 0)) + channels[which] * 4;
            *reinterpret_cast<float4*>(state) = context;
          }
        }
        qv = values[0], kv = values[1], vv = values[2];
      }
    } else {
      if (tid < kHeadDim) {
        qv = q[(row * kKeyHeads + keyHead) * kHeadDim + tid];
        kv = k[(row * kKeyHeads + keyHead) * kHeadDim + tid];
        vv = v[(row * kValueHeads + head) * kHeadDim + tid];
      }
      decay = expf(g[row * kValueHeads + head]);
      betaValue = beta[row * kValueHeads + head];
    }
    // L2-normalise q (scaled by 1/sqrt(128)) and k; q.k of the normalised vectors (delta_rule.metal:281-311).
    if (tid < kHeadDim) {
      qraw[tid] = qv, kraw[tid] = kv, vraw[tid] = vv;
      const float a = warp_sum(qv * qv), b = warp_sum(kv * kv), c = warp_sum(qv * kv);
      if (lane == 0) {
        red[part] = a;
        red[4 + part] = b;
        red[8 + part] = c;
      }
    }
    __syncthreads();
    float4 gate = make_float4(0.f, 0.f, 0.f, 0.f), weight = gate;
    if (part == 0 && z)  // needed after the next barrier; asked for here
      gate = *reinterpret_cast<const float4*>(z + at), weight = *reinterpret_cast<const float4*>(normWeight + 4 * lane);
    const float qn = rsqrtf(red[0] + red[1] + red[2] + red[3] + 1.0e-6f) * 0.08838834764831845f;
    const float kn = rsqrtf(red[4] + red[5] + red[6] + red[7] + 1.0e-6f);
    const float qk = (red[8] + red[9] + red[10] + red[11]) * qn * kn;
    if (FUSED) {
      const float dotBeta = (dots[0] + dots[1]) + (dots[2] + dots[3]), dotAlpha = (dots[4] + dots[5]) + (dots[6] + dots[7]);
      decay = expf(headA * logf(1.0f + expf(dotAlpha + headDt)));
      betaValue = 1.0f / (1.0f + expf(-dotBeta));
    }
    float4 pred = make_float4(0.f, 0.f, 0.f, 0.f), qstate = pred;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float kk = kraw[part + 8 * i] * kn, qq = qraw[part + 8 * i] * qn;
      S[i].x *= decay, S[i].y *= decay, S[i].z *= decay, S[i].w *= decay;
      pred.x = fmaf(S[i].x, kk, pred.x), pred.y = fmaf(S[i].y, kk, pred.y), pred.z = fmaf(S[i].z, kk, pred.z), pred.w = fmaf(S[i].w, kk, pred.w);
      qstate.x = fmaf(S[i].x, qq, qstate.x), qstate.y = fmaf(S[i].y, qq, qstate.y), qstate.z = fmaf(S[i].z, qq, qstate.z),
      qstate.w = fmaf(S[i].w, qq, qstate.w);
    }
    partialPred[part][lane] = pred;
    partialQ[part][lane] = qstate;
    __syncthreads();
    // every warp: the sums of the eight partials for its lanes' four columns, delta and the output there
    float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f), s4 = p4;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float4 a = partialPred[w][lane], b = partialQ[w][lane];
      p4.x += a.x, p4.y += a.y, p4.z += a.z, p4.w += a.w;
      s4.x += b.x, s4.y += b.y, s4.z += b.z, s4.w += b.w;
    }
    const float4 v4 = *reinterpret_cast<const float4*>(&vraw[4 * lane]);
    const float4 d4 = make_float4((v4.x - p4.x) * betaValue, (v4.y - p4.y) * betaValue, (v4.z - p4.z) * betaValue, (v4.w - p4.w) * betaValue);
    if (part == 0) {
      float4 o = make_float4(s4.x + d4.x * qk, s4.y + d4.y * qk, s4.z + d4.z * qk, s4.w + d4.w * qk);
      if (z) {  // gated_rms_norm_128
        const float scale = rsqrtf(warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w) / float(kHeadDim) + 1.0e-6f);
        o = make_float4(o.x * scale * weight.x * silu_f(gate.x), o.y * scale * weight.y * silu_f(gate.y), o.z * scale * weight.z * silu_f(gate.z),
                        o.w * scale * weight.w * silu_f(gate.w));
      }
      *reinterpret_cast<float4*>(out + at) = o;
      if (image && row < kImageCounters / (kValueHeads / 2)) {  // later rows have no counter and get no image
        const int entry = int(row) * (kValueHeads / 2) + (head >> 1);
        __syncwarp();
        int arrivals = 0;
        if (lane == 0) {
          __threadfence();
          arrivals = atomicAdd(&counters[entry], 1);
        }
        if (__shfl_sync(0xffffffffu, arrivals, 0) == 1) {
          __threadfence();
          const float* src = out + (row * kValueHeads + (head & ~1)) * kHeadDim + lane * 8;
          const float4 a = __ldcg(reinterpret_cast<const float4*>(src)), b = __ldcg(reinterpret_cast<const float4*>(src + 4));
          const float values[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
          image_store_block(image + (size_t(row >> 3) * (kValueHeads / 2) + (head >> 1)) * kImageBlockBytes, int(row & 7), lane, values);
          if (lane == 0)
            counters[entry] = 0;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float kk = kraw[part + 8 * i] * kn;
      S[i].x = fmaf(kk, d4.x, S[i].x), S[i].y = fmaf(kk, d4.y, S[i].y), S[i].z = fmaf(kk, d4.z, S[i].z), S[i].w = fmaf(kk, d4.w, S[i].w);
    }
    if (speculative || t + 1 == info.count) {
      float4* dst = reinterpret_cast<float4*>(info.next + stateOffset + (speculative ? uint64_t(t) * stateBytes : 0)) + size_t(head) * kHeadDim * 32;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        dst[(part + 8 * i) * 32 + lane] = S[i];
    }
    if (t + 1 < info.count)
      __syncthreads();  // the shared arrays are rewritten for the next token
  }
}

// ---- chunked form for long prefill queries -----------------------------------------------------------
// Replaces delta_rule_prefill (delta_rule.metal:19-253): 16 tokens per step instead of one. With S the state before the
// chunk, G_t = d_0 ... d_t the cumulated decay, R[t][i] = G_t / G_i and the unit lower-triangular
// A[t][i] = beta_t R[t][i] (k_t . k_i) for i < t, the recurrence of delta_rule_kernel unrolls to
//   delta  = A^-1 rhs,   rhs_t = beta_t * (v_t - G_t * S^T k_t)
//   o_t    = G_t * S^T q_t + sum_{i<=t} R[t][i] (q_t . k_i) delta_i
//   S      = G_15 * S + sum_i (G_15 / G_i) k_i delta_i^T
// grid (32 value heads, queries, or more where so few are split), 12 warps; serves the non-speculative queries of at least `chunkedFrom` tokens, all
// but the norm of their outputs, which is delta_rule_kernel's launch (gated_norm_rows): here it stood in the chain, 2000 of 8200 clocks a chunk. A last
// chunk of fewer than 16 tokens is padded with tokens of beta = 0, k = q = v = 0 and decay 1, which change nothing.
//
// A query is a chain of chunks per head, so what counts is the time of one chunk. Everything that does not depend on S - the
// normalised keys and queries, the gates, A^-1 and the weights of the second sum - is prepared by four warps of their own,
// a chunk or two ahead, in two shared-memory buffers. The eight others hold S^T in registers, 16 value columns each: a warp
// needs nothing from its neighbours, because a value column's recurrence is its own. All
// products run on the tensor cores; a warp's accumulators (value column x key dim, or x token) are at the same time, as they
// lie in its registers, the A operand of the next product.
// Where no more than two queries are chunked (64 CTAs of 148 SMs), a head's columns go to two CTAs: four computing warps then have the tensor
// cores of an SM to themselves, and the four that are left over prepare every second chunk.
//
// Precision. Keys, queries, S and the update of S are split into fp16 hi + lo after scaling by a power of two (fixed for keys
// and queries, whose norm is at most 1; by the largest value of each value column for the others), and the three products that
// matter (lo hi, hi lo, hi hi) are formed. A^-1, the weights of the second sum, rhs and delta span whatever the decays and the
// values span, so they are split into three bf16 parts (24 bits and the exponents of fp32) and six products. The tensor cores
// cut off what does not fit their accumulator instead of rounding it, so no sum is carried through them: every product of 16
// terms starts from zero and is added with a rounded fp32 addition. Decays are cumulated in double precision, because their
// logarithms reach hundreds while differences of neighbours matter to the last bit. Against fp64, with gates, values and states
// as a model has them, 512 tokens: outputs 1.8e-7, state 1.4e-7 (2-norms); the fp32 chunk form before it 2.1e-7 and 4.7e-7,
// token by token 1.1e-7 and 0.7e-7. One scale for the 16 columns of a warp, fp16 parts throughout and sums carried in the
// accumulators gave 4.1e-7 and 5.4e-7, and lost value columns far below their neighbours; they took 278 us for eight queries
// of 59 to 493 rows when this form, with its preparation, took 311 us.
// By its own clocks a chunk takes 5000 with half of the columns (KS and QS 1900, A^-1 rhs 550, the second sum 500, the update 1000, the rest
// stores, scales and barriers) and 6900 with all (2800, 700, 700, 1400), where the preparing warps are as slow as that; 8200 when the norm was part of
// the chain and one preparing warp had gates, decays and the inverse. With the norms, before and now: eight queries of 59 to 493 rows 199.9 -> 176.9 us,
// of 128 rows 88.8 -> 80.4, one of 493 rows 143.4 -> 88.3, of 128 rows 42.1 -> 30.8, of 64 rows 24.7 -> 20.6. Tried and left out: the outputs by
// warps of their own that are handed S through shared memory (eight queries 200 -> 244 us), two of the preparing warps a stage behind the two others
// (187 -> 222, without spread norms), 16 warps of 128 registers (237).
constexpr int kChunk = 16, kComputeWarps = 8, kPrepareWarps = 4;
constexpr int kChunkThreads = (kComputeWarps + kPrepareWarps) * kWarp;
constexpr int kSplitWarps = kComputeWarps / 2;  // computing warps of a CTA that has half of a head's value columns
constexpr float kKeyUnit = 256.f;  // fixed scale of the normalised keys and queries
using TokenMatrix = __nv_bfloat16[3][kChunk][kChunk + 8];  // lower triangular, [part][token][token]
struct ChunkBuffer {
  __half k[2][kChunk][kHeadDim + 8], q[2][kChunk][kHeadDim + 8];  // hi, lo of kKeyUnit x the normalised rows
  TokenMatrix solve, mix;  // three parts of A^-1 and R (q . k)
  float decay[kChunk], tail[kChunk], beta[kChunk];                // G_t, G_15 / G_t, beta_t
};
struct ChunkShared {
  ChunkBuffer buffer[2];
  // of the chunk being prepared, two sets in turn: warp 1 reads one while warp 3 may already write the next chunk's, and a set
  // comes up again only behind the barrier that frees its buffer
  double cumulative[2][kChunk];
  float gateBeta[2][kChunk];
  float system[2][kChunk][kChunk + 1], ratio[2][kChunk][kChunk + 1];  // of each preparing group: the triangular system; R
  float squares[2][kComputeWarps][kChunk];                            // of the outputs, where they are normalised here
};
// named barriers: 1, 2 buffer filled; 3, 4 buffer free; 5, 6 a preparing group
__device__ __forceinline__ void chunk_ldmatrix(uint32_t (&r)[4], const void* address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(address)) : "memory");
}
__device__ __forceinline__ void chunk_ldmatrix_trans(uint32_t (&r)[4], const __half* address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(address))
               : "memory");
}
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_half2(a, b);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  lo = pack_half2(a - f.x, b - f.y);
}
// a, b as three bf16 pairs, largest first
__device__ __forceinline__ void split_three(float a, float b, uint32_t (&part)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(a, b);
    part[i] = *reinterpret_cast<const uint32_t*>(&pair);
    a -= __low2float(pair), b -= __high2float(pair);
  }
}
// 2^n that brings a value column's largest magnitude into [512, 1024), and 2^-n; the column's values lie in the four lanes of a
// quad. Both are normal numbers, whatever the magnitude is: the exponent fields lie in 1 .. 253 (all zero: 2^126 and 2^-126).
__device__ __forceinline__ float2 column_unit(float largest) {
  largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
  largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 2));
  const int field = min(253, max(1, 263 - int(__float_as_uint(largest) >> 23)));
  return make_float2(__uint_as_float(uint32_t(field) << 23), __uint_as_float(uint32_t(254 - field) << 23));
}
// The two 16 x 8 accumulators of 16 x 16 values (C fragments) x their columns' units as the A operand, hi and lo.
__device__ __forceinline__ void split_tile(const float (&c0)[4], const float (&c1)[4], float unit, float unit8, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  split_pair(c0[0] * unit, c0[1] * unit, hi[0], lo[0]);
  split_pair(c0[2] * unit8, c0[3] * unit8, hi[1], lo[1]);
  split_pair(c1[0] * unit, c1[1] * unit, hi[2], lo[2]);
  split_pair(c1[2] * unit8, c1[3] * unit8, hi[3], lo[3]);
}
// d = A x B for the two n-tiles of B fragments bHi, bLo, as lo hi + hi lo + hi hi.
__device__ __forceinline__ void mma_three(float (&d)[2][4], const uint32_t (&hi)[4], const uint32_t (&lo)[4], const uint32_t (&bHi)[4],
                                          const uint32_t (&bLo)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e)
    d[0][e] = d[1][e] = 0.f;
  mma_16816(d[0], lo, bHi[0], bHi[1]), mma_16816(d[1], lo, bHi[2], bHi[3]);
  mma_16816(d[0], hi, bLo[0], bLo[1]), mma_16816(d[1], hi, bLo[2], bLo[3]);
  mma_16816(d[0], hi, bHi[0], bHi[1]), mma_16816(d[1], hi, bHi[2], bHi[3]);
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// token_product without the products with the matrix's zeros; values: this lane's eight of c (element 4n + e), then of d.
__device__ __forceinline__ void token_sums(const TokenMatrix& b, float (&values)[8]) {
  const int lane = threadIdx.x & 31, t2 = 2 * (lane & 3);
  float sum[8] = {};
#pragma unroll 1
  for (int from = 0; from < kChunk; ++from) {
    const int source = (lane & ~3) + ((from & 7) >> 1), element = 4 * (from >> 3) + (from & 1);
    const float value[2] = {__shfl_sync(0xffffffffu, values[element], source), __shfl_sync(0xffffffffu, values[element + 2], source)};
    for (int i = 0; i < 8; ++i) {
      const int token = 8 * (i >> 2) + t2 + (i & 1);
      if (from <= token)
        sum[i] = fmaf((__bfloat162float(b[2][token][from]) + __bfloat162float(b[1][token][from])) + __bfloat162float(b[0][token][from]), value[(i >> 1) & 1],
                      sum[i]);
    }
  }
  for (int i = 0; i < 8; ++i)
    values[i] = sum[i];
}
// d = the 16 x 16 values c (C fragments, 16 value columns x 16 tokens) x B^T; all the products of three parts by three that
// reach 24 bits, summed by their order of magnitude.
__device__ __forceinline__ void token_product(float (&d)[2][4], const float (&c)[2][4], const TokenMatrix& b, int row, int column) {
  float finite = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    finite = fmaf(c[i >> 2][i & 3], 0.f, finite);
  if (__any_sync(0xffffffffu, !(finite == 0.f))) {  // times the zeros it would reach the tokens before it
    float values[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      values[i] = c[i >> 2][i & 3];
    token_sums(b, values);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      d[i >> 2][i & 3] = values[i];
    return;
  }
  uint32_t a[3][4], fragment[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t part[3];
    split_three(c[i >> 1][2 * (i & 1)], c[i >> 1][2 * (i & 1) + 1], part);
    a[0][i] = part[0], a[1][i] = part[1], a[2][i] = part[2];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
    chunk_ldmatrix(fragment[i], &b[i][row][column]);
  float sum[3][2][4] = {};  // by order of magnitude
#pragma unroll
  for (int order = 2; order >= 0; --order)
#pragma unroll
    for (int i = 0; i <= order; ++i)
#pragma unroll
      for (int n = 0; n < 2; ++n)
        mma_bf16(sum[order][n], a[i], fragment[order - i][2 * n], fragment[order - i][2 * n + 1]);
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      d[n][e] = sum[0][n][e] + (sum[1][n][e] + sum[2][n][e]);
}
// e^x rounded from more digits than a float x has: cumulated log decays of hundreds would lose all but a few of e^x.
__device__ __forceinline__ float exp_of(double x) {
  const float hi = float(x), lo = x == double(hi) ? 0.f : float(x - double(hi)), e = expf(hi);
  return e < INFINITY ? fmaf(e, lo, e) : e;
}

__device__ __forceinline__ void store_three(TokenMatrix& to, int t, int i, float value) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    to[p][t][i] = __float2bfloat16_rn(value);
    value -= __bfloat162float(to[p][t][i]);
  }
}

// The four preparing warps: chunk after chunk into the two buffers. All normalise four tokens each; then warps 0 and 1 have the products
// k . k and q . k while 2 and 3 form the decays between the tokens, and warp 3 cumulates the gates of the next chunk while warp 0 inverts.
__device__ __forceinline__ void chunk_prepare(ChunkShared& sh, const infdev_query& info, const float* q, const float* k, const float* g, const float* beta,
                                              int head, int group, int groups, int threads) {
  const int warp = (threadIdx.x >> 5) % kPrepareWarps, lane = threadIdx.x & 31, keyHead = head % kKeyHeads;
  const int tokenOfB = (lane & 7) + 8 * (lane >> 4), dimOfB = 8 * ((lane >> 3) & 1);  // ldmatrix rows of a B operand stored [n][k]
  float4 nextQ[4], nextK[4];
  float nextG = 0.f, nextBeta = 0.f;
  double cumulative = 0.0;  // warp 3: of the next chunk's tokens
  auto load = [&](uint32_t first) {  // warp w: tokens 4w .. 4w + 3
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t token = first + 4 * warp + j;
      nextQ[j] = nextK[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (token < info.count) {
        const size_t at = (size_t(info.start + token) * kKeyHeads + keyHead) * kHeadDim + 4 * lane;
        nextQ[j] = *reinterpret_cast<const float4*>(q + at), nextK[j] = *reinterpret_cast<const float4*>(k + at);
      }
    }
    if (warp == 3) {
      const bool live = lane < kChunk && first + lane < info.count;
      nextG = live ? g[size_t(info.start + first + lane) * kValueHeads + head] : 0.f;
      nextBeta = live ? beta[size_t(info.start + first + lane) * kValueHeads + head] : 0.f;
    }
  };
  auto cumulate = [&] {  // lanes 16 .. 31: the sum over all 16 tokens
    cumulative = double(nextG);
#pragma unroll
    for (int step = 1; step < kChunk; step *= 2) {
      const double other = __shfl_up_sync(0xffffffffu, cumulative, step);
      if (lane >= step)
        cumulative += other;
    }
    const double all = __shfl_sync(0xffffffffu, cumulative, kChunk - 1);
    cumulative = lane < kChunk ? cumulative : all;
  };
  load(group * kChunk);
  if (warp == 3)
    cumulate();
  uint32_t step = group;
  for (uint32_t first = group * kChunk; first < info.count; first += groups * kChunk, step += groups) {
    ChunkBuffer& out = sh.buffer[step & 1];
    if (step >= 2)
      named_barrier(3 + (step & 1), threads);
    const float gateBeta = nextBeta;
    if (warp == 3 && lane < kChunk)
      sh.cumulative[step & 1][lane] = cumulative, sh.gateBeta[step & 1][lane] = gateBeta;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 a = nextQ[j], b = nextK[j];
      const float qq = warp_sum(a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w), kk = warp_sum(b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w);
      const float qn = rsqrtf(qq + 1.0e-6f) * 0.08838834764831845f * kKeyUnit, kn = rsqrtf(kk + 1.0e-6f) * kKeyUnit;
      uint2 hi, lo;
      split_pair(a.x * qn, a.y * qn, hi.x, lo.x), split_pair(a.z * qn, a.w * qn, hi.y, lo.y);
      *reinterpret_cast<uint2*>(&out.q[0][4 * warp + j][4 * lane]) = hi, *reinterpret_cast<uint2*>(&out.q[1][4 * warp + j][4 * lane]) = lo;
      split_pair(b.x * kn, b.y * kn, hi.x, lo.x), split_pair(b.z * kn, b.w * kn, hi.y, lo.y);
      *reinterpret_cast<uint2*>(&out.k[0][4 * warp + j][4 * lane]) = hi, *reinterpret_cast<uint2*>(&out.k[1][4 * warp + j][4 * lane]) = lo;
    }
    load(first + groups * kChunk);  // past the end: zeros
    named_barrier(5 + group, kPrepareWarps * kWarp);
    float dot[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    if (warp < 2) {
      const auto& left = warp == 0 ? out.k : out.q;
#pragma unroll
      for (int s = 0; s < kHeadDim / 16; ++s) {
        uint32_t hi[4], lo[4], bHi[4], bLo[4];
        chunk_ldmatrix(hi, &left[0][lane & 15][16 * s + 8 * (lane >> 4)]);
        chunk_ldmatrix(lo, &left[1][lane & 15][16 * s + 8 * (lane >> 4)]);
        chunk_ldmatrix(bHi, &out.k[0][tokenOfB][16 * s + dimOfB]);
        chunk_ldmatrix(bLo, &out.k[1][tokenOfB][16 * s + dimOfB]);
        float part[2][4];
        mma_three(part, hi, lo, bHi, bLo);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          dot[0][e] += part[0][e], dot[1][e] += part[1][e];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = 8 * (warp - 2) + 2 * j + (lane >> 4), i = lane & 15;
        sh.ratio[group][t][i] = i <= t ? exp_of(sh.cumulative[step & 1][t] - sh.cumulative[step & 1][i]) : 0.f;
      }
    }
    named_barrier(5 + group, kPrepareWarps * kWarp);
    if (warp < 2) {
      // warp 0: the triangular system and its inverse; warp 1: the weights of the second sum
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = (lane >> 2) + 8 * (e >> 1), i = 8 * n + 2 * (lane & 3) + (e & 1);
          const float value = dot[n][e] * (1.0f / (kKeyUnit * kKeyUnit)) * sh.ratio[group][t][i];
          if (warp == 0) {
            sh.system[group][t][i] = i < t ? value * sh.gateBeta[step & 1][t] : 0.f;
          } else {
            store_three(out.mix, t, i, i <= t ? value : 0.f);
          }
        }
      if (warp == 0) {
        __syncwarp();
        // column `lane` of the inverse by forward substitution (lanes 16 .. 31 repeat columns 0 .. 15)
        const int column = lane & 15;
        float x[kChunk];
#pragma unroll
        for (int t = 0; t < kChunk; ++t)
          x[t] = t == column ? 1.f : 0.f;
#pragma unroll
        for (int i = 0; i < kChunk; ++i)
#pragma unroll
          for (int t = i + 1; t < kChunk; ++t)
            x[t] = fmaf(-sh.system[group][t][i], x[i], x[t]);
        if (lane < kChunk)
#pragma unroll
          for (int t = 0; t < kChunk; ++t) {
            store_three(out.solve, t, column, x[t]);
          }
      }
    } else if (warp == 3) {
      const double all = __shfl_sync(0xffffffffu, cumulative, kChunk);
      if (lane < kChunk)
        out.decay[lane] = exp_of(cumulative), out.tail[lane] = exp_of(all - cumulative), out.beta[lane] = gateBeta;
      cumulate();
    }
    named_barrier_arrive(1 + (step & 1), threads);
  }
}

// Which query the CTAs of row `rank` of the grid take: of those that this kernel takes the one with the rank-th largest count, so that the longest
// chains start first and the short ones fill the SMs that are left over (eight queries of 59 to 493 rows, 256 CTAs on 148 SMs, with an
// earlier form of the chunk and its preparation: 323 us in the order of the pass, 281 us sorted). Every lane of a warp calls; beyond 32 queries the order of the pass stays.
__device__ __forceinline__ uint32_t query_by_length(const infdev_query* queries, uint32_t count, uint32_t chunkedFrom, uint32_t rank) {
  if (count > 32)
    return rank;
  const uint32_t lane = threadIdx.x & 31, mine = lane < count && chunked(queries[lane], chunkedFrom) ? queries[lane].count : 0u;
  uint32_t before = 0;
  for (uint32_t j = 0; j < count; ++j) {
    const uint32_t other = __shfl_sync(0xffffffffu, mine, j);
    before += other > mine || (other == mine && j < lane) ? 1u : 0u;
  }
  return uint32_t(__ffs(__ballot_sync(0xffffffffu, lane < count && before == rank)) - 1);
}

// NORM: the outputs go over the gates z, which would be gone before the norm's launch reads them, so they are normalised in the chain, by one CTA a head.
// Over the gates / apart: eight queries of 59 to 493 rows 195.6 / 176.9 us, one of 493 rows 140.1 / 88.3.
template <bool NORM>
__global__ void __launch_bounds__(kChunkThreads, 1)
    delta_rule_chunked_kernel(const float* q, const float* k, const float* v, const float* g, const float* beta, const float* normWeight,
                              const infdev_query* queries, uint64_t stateOffset, float* out, uint32_t chunkedFrom, uint32_t queryCount, uint32_t sms) {
  pdl_launch_dependents();
  pdl_wait();
  // Two CTAs have half of a head's columns each: rows of the grid from the number of chunked queries on, which else have nothing to do, take the second halves.
  const uint32_t taken = chunked_queries(queries, queryCount, chunkedFrom);
  const bool split = !NORM && 2 * kValueHeads * taken <= sms;
  const uint32_t part = split && blockIdx.y >= taken ? 1 : 0, rank = blockIdx.y - part * taken;
  if (rank >= (split ? taken : queryCount))
    return;
  const infdev_query info = queries[query_by_length(queries, queryCount, chunkedFrom, rank)];
  if (!chunked(info, chunkedFrom))  // delta_rule_kernel takes this query
    return;
  extern __shared__ __align__(16) uint8_t chunkRaw[];
  ChunkShared& sh = *reinterpret_cast<ChunkShared*>(chunkRaw);
  const int head = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int threads = split ? (kSplitWarps + kPrepareWarps) * kWarp : kChunkThreads;  // at the barriers of a buffer
  // The computing warps hold more than a third of the registers each: 2 x 192 + 120 = 3 x 168 a thread, of the 168 that the launch
  // bounds give all three groups of four warps.
  if (warp >= (split ? kSplitWarps : kComputeWarps)) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 120;");
    chunk_prepare(sh, info, q, k, g, beta, head, split ? warp / kPrepareWarps - 1 : 0, split ? 2 : 1, threads);
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
  const int row = lane >> 2, t2 = 2 * (lane & 3), column = 16 * (warp + int(part) * kSplitWarps) + row;  // value columns `column` and `column` + 8
  const int tokenOfB = (lane & 7) + 8 * (lane >> 4), dimOfB = 8 * ((lane >> 3) & 1);
  float S[kHeadDim / 8][4];  // S^T: tile j holds key dims 8j + t2, + 1 of the two value columns
  const size_t state = size_t(head) * kHeadDim * kHeadDim + column;
#pragma unroll
  for (int j = 0; j < kHeadDim / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      S[j][e] = info.previous ? reinterpret_cast<const float*>(info.previous + stateOffset)[state + (8 * j + t2 + (e & 1)) * kHeadDim + 8 * (e >> 1)] : 0.f;
  // element (n, e) of a token tile: token 8n + t2 + e % 2, value column + 8 (e / 2)
  float value[2][4];
  auto load = [&](float (&into)[2][4], const float* from, uint32_t first) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t token = first + 8 * n + t2 + (e & 1);
        into[n][e] = token < info.count ? from[(size_t(info.start + token) * kValueHeads + head) * kHeadDim + column + 8 * (e >> 1)] : 0.f;
      }
  };
  load(value, v, 0);
  [[maybe_unused]] float gate[2][4], weight[2];
  if constexpr (NORM)
    weight[0] = normWeight[column], weight[1] = normWeight[column + 8];
  uint32_t step = 0;
  for (uint32_t first = 0; first < info.count; first += kChunk, ++step) {
    const ChunkBuffer& in = sh.buffer[step & 1];
    if constexpr (NORM)
      load(gate, out, first);
    float largest[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < kHeadDim / 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        largest[e >> 1] = fmaxf(largest[e >> 1], fabsf(S[j][e]));
    const float2 unit = column_unit(largest[0]), unit8 = column_unit(largest[1]);
    named_barrier(1 + (step & 1), threads);
    // S^T k and S^T q of the 16 tokens
    float ks[2][4], qs[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        ks[n][e] = qs[n][e] = 0.f;
#pragma unroll
    for (int s = 0; s < kHeadDim / 16; ++s) {
      uint32_t hi[4], lo[4], bHi[4], bLo[4];
      float part[2][4];
      split_tile(S[2 * s], S[2 * s + 1], unit.x, unit8.x, hi, lo);
      chunk_ldmatrix(bHi, &in.k[0][tokenOfB][16 * s + dimOfB]);
      chunk_ldmatrix(bLo, &in.k[1][tokenOfB][16 * s + dimOfB]);
      mma_three(part, hi, lo, bHi, bLo);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        ks[0][e] += part[0][e], ks[1][e] += part[1][e];
      chunk_ldmatrix(bHi, &in.q[0][tokenOfB][16 * s + dimOfB]);
      chunk_ldmatrix(bLo, &in.q[1][tokenOfB][16 * s + dimOfB]);
      mma_three(part, hi, lo, bHi, bLo);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        qs[0][e] += part[0][e], qs[1][e] += part[1][e];
    }
    const float productUnit[2] = {unit.y * (1.0f / kKeyUnit), unit8.y * (1.0f / kKeyUnit)};
    float decay[2][2];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        decay[n][e] = in.decay[8 * n + t2 + e];
    // rhs, delta = A^-1 rhs
    float rhs[2][4], delta[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        rhs[n][e] = in.beta[8 * n + t2 + (e & 1)] * (value[n][e] - decay[n][e & 1] * (ks[n][e] * productUnit[e >> 1]));
    load(value, v, first + kChunk);  // of the next chunk
    token_product(delta, rhs, in.solve, tokenOfB, dimOfB);
    // outputs, and the state's update with (G_15 / G_i) delta_i
    float mixed[2][4];
    token_product(mixed, delta, in.mix, tokenOfB, dimOfB);
    largest[0] = largest[1] = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        delta[n][e] *= in.tail[8 * n + t2 + (e & 1)];
        largest[e >> 1] = fmaxf(largest[e >> 1], fabsf(delta[n][e]));
      }
    const float2 scale = column_unit(largest[0]), scale8 = column_unit(largest[1]);
    uint32_t hi[4], lo[4];
    split_tile(delta[0], delta[1], scale.x, scale8.x, hi, lo);
    // The sum over the tokens starts from zero and is scaled before it meets the state, which stays in units of its own: deltas
    // may be zero or any number of powers of two smaller than the state (beta = 0, value columns without weights).
    const float stateDecay = in.decay[kChunk - 1], updateUnit[2] = {scale.y * (1.0f / kKeyUnit), scale8.y * (1.0f / kKeyUnit)};
#pragma unroll
    for (int s = 0; s < kHeadDim / 16; ++s) {
      uint32_t bHi[4], bLo[4];
      float added[2][4];
      chunk_ldmatrix_trans(bHi, &in.k[0][lane & 15][16 * s + 8 * (lane >> 4)]);
      chunk_ldmatrix_trans(bLo, &in.k[1][lane & 15][16 * s + 8 * (lane >> 4)]);
      mma_three(added, hi, lo, bHi, bLo);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          S[2 * s + n][e] = fmaf(added[n][e], updateUnit[e >> 1], S[2 * s + n][e] * stateDecay);
    }
    named_barrier_arrive(3 + (step & 1), threads);  // the buffer may be refilled
    auto output = [&](int n, int e) { return decay[n][e & 1] * (qs[n][e] * productUnit[e >> 1]) + mixed[n][e]; };
    if constexpr (NORM) {  // gated_rms_norm_128 over the columns of all computing warps
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          mixed[n][e] = output(n, e);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float sum = __fmaf_rn(mixed[n][e + 2], mixed[n][e + 2], __fmul_rn(mixed[n][e], mixed[n][e]));
#pragma unroll
          for (int m = 4; m < 32; m <<= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, m);
          if (row == 0)
            sh.squares[step & 1][warp][8 * n + t2 + e] = sum;
        }
      named_barrier(7, kComputeWarps * kWarp);  // two sets of sums in turn: nobody is two chunks behind
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float sum = 0.f;
#pragma unroll
          for (int w = 0; w < kComputeWarps; ++w)
            sum += sh.squares[step & 1][w][8 * n + t2 + e];
          const float scale = rsqrtf(sum / float(kHeadDim) + 1.0e-6f);
          mixed[n][e] = mixed[n][e] * scale * weight[0] * silu_f(gate[n][e]);
          mixed[n][e + 2] = mixed[n][e + 2] * scale * weight[1] * silu_f(gate[n][e + 2]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t token = first + 8 * n + t2 + (e & 1);
        if (token < info.count)
          out[(size_t(info.start + token) * kValueHeads + head) * kHeadDim + column + 8 * (e >> 1)] = NORM ? mixed[n][e] : output(n, e);
      }
  }
#pragma unroll
  for (int j = 0; j < kHeadDim / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      reinterpret_cast<float*>(info.next + stateOffset)[state + (8 * j + t2 + (e & 1)) * kHeadDim + 8 * (e >> 1)] = S[j][e];
}

}  // namespace

cudaError_t gdn_prepare_launch(const float* x, const float* mixed, const float* wBeta, const float* wAlpha, const float* A, const float* dt,
                               const float* convWeight, const infdev_query* queries, int64_t rows, uint64_t stateOffset, uint64_t stateBytes,
                               float* q, float* k, float* v, float* beta, float* g, cudaStream_t stream) {
  if (rows <= 0)
    return cudaSuccess;
  auto launch = [&](auto kernel, int convRows, int gateHeads) {
    const int gateBlocks = int((rows + kGateRows - 1) / kGateRows) * (kValueHeads / gateHeads);
    const int convBlocks = int((rows + convRows - 1) / convRows) * (kChannels / kConvChannels);
    launch_kernel<2>(kernel, unsigned(gateBlocks + convBlocks), 256, 0, stream, x, wBeta, wAlpha, A, dt, mixed, convWeight, queries, int(rows), gateBlocks,
                     stateOffset, stateBytes, q, k, v, beta, g);
  };
  // A caller's views may start at any float.
  uintptr_t addresses = 0;
  for (const float* p : {mixed, convWeight, static_cast<const float*>(q), static_cast<const float*>(k), static_cast<const float*>(v)})
    addresses |= reinterpret_cast<uintptr_t>(p);
  if (addresses & 15)
    launch(gdn_prepare_kernel<1, 1, false>, 1, 1);
  else if (rows <= kPrepareRows1)
    launch(gdn_prepare_kernel<1, 1, true>, 1, 1);
  else if (rows <= kPrepareRows2)
    launch(gdn_prepare_kernel<2, 2, true>, 2, 2);
  else if (rows <= kPrepareRows4)
    launch(gdn_prepare_kernel<4, 4, true>, 4, 4);
  else
    launch(gdn_prepare_kernel<8, 8, true>, 8, 8);
  return cudaGetLastError();
}

cudaError_t delta_rule_launch(const float* q, const float* k, const float* v, const float* g, const float* beta, const float* z,
                              const float* normWeight, const infdev_query* queries, int queryCount, uint64_t stateOffset, uint64_t stateBytes,
                              float* out, uint8_t* image, int* counters, uint32_t chunkedFrom, int sms, cudaStream_t stream) {
  if (queryCount <= 0)
    return cudaSuccess;
  if (chunkedFrom) {
    static PerDeviceOnce configured[2];
    const bool norm = z == out;
    const auto kernel = norm ? delta_rule_chunked_kernel<true> : delta_rule_chunked_kernel<false>;
    if (cudaError_t e = configure_shared_memory(kernel, sizeof(ChunkShared), configured[norm]))
      return e;
    // rows for the halves of as many queries as may be split. Rows of their own beside those of all queries made three turns of CTAs out of two where
    // eight queries are all short (5 rows each 18.6 -> 19.6 us), and a grid too large out of 65535 queries.
    const int rows = norm ? queryCount : std::max(queryCount, 2 * std::min(queryCount, sms / (2 * kValueHeads)));
    launch_kernel<2>(kernel, dim3(kValueHeads, unsigned(rows)), kChunkThreads, sizeof(ChunkShared), stream, q, k, v, g, beta, normWeight, queries,
                     stateOffset, out, chunkedFrom, uint32_t(queryCount), uint32_t(sms));
  }
  // The norms of long queries are spread over several CTAs a head, which else were a chain of loads and stores after the last chunk: one query of 493
  // rows 111 -> 96.5 us, six of 17 to 700 rows 202 -> 179, eight of 59 to 493 rows 187 -> 179, as they were measured then. Few enough of them that those without rows do not
  // tell (eight queries of 128 rows 81.0, with four CTAs a head 81.7, with eight 83.4).
  const int spread = chunkedFrom && z && z != out ? std::clamp(6 * sms / (kValueHeads * queryCount), 1, 8) : 1;
  // Not launched early: its CTAs would be placed around those of the kernels before it, two on an SM, and the token-by-token chain
  // of short queries runs slower for it (12 rows: 37.5 against 31.0 us; passes that the chunked kernel takes lose 1 us).
  launch_kernel(delta_rule_kernel<false>, dim3(kValueHeads, unsigned(queryCount), unsigned(spread)), 256, 0, stream, q, k, v, g, beta, z, normWeight, queries, stateOffset,
                stateBytes, out, image, counters, chunkedFrom, GdnInputs{});
  return cudaGetLastError();
}

cudaError_t gdn_decode_launch(const float* x, const float* mixed, const float* wBeta, const float* wAlpha, const float* A, const float* dt,
                              const float* convWeight, const float* z, const float* normWeight, const infdev_query* queries, int queryCount,
                              uint64_t convStateOffset, uint64_t stateOffset, uint64_t stateBytes, float* out, uint8_t* image, int* counters,
                              bool ahead, cudaStream_t stream) {
  if (queryCount <= 0)
    return cudaSuccess;
  static PerDeviceOnce configured;
  if (cudaError_t e = configure_shared_memory(delta_rule_kernel<true>, sizeof(GdnStage), configured))
    return e;
  launch_kernel<1>(delta_rule_kernel<true>, dim3(kValueHeads, unsigned(queryCount)), 256, sizeof(GdnStage), stream, nullptr, nullptr, nullptr, nullptr, nullptr, z, normWeight,
                   queries, stateOffset, stateBytes, out, image, counters, 0u, GdnInputs{x, wBeta, wAlpha, A, dt, mixed, convWeight, convStateOffset, ahead && pdl_mode() != 1});
  return cudaGetLastError();
}

}  // namespace infdev
