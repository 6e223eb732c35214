// Integer tensor-core GEMV for decode (M <= 8 activation rows) over GGUF Q4_K weights.
//
// Replaces linear_decode_q4_k[_add] (quant_linear.metal:245-327) and mlp_gate_up_q4_k_decode
// (fused_kernels.metal:11-78) like gemv.cu, with a cheaper inner loop: the 4-bit quants feed the tensor cores
// as unsigned bytes (one AND per four weights) against activations quantised to 16-bit integers per
// (row, 256-value block) and split into a signed high and an unsigned low byte (act_image.cuh). One m16n8k32
// integer MMA covers exactly one 32-weight sub-block of 16 weight rows, so the 6-bit sub-block scale is applied
// to the int32 result with one integer multiply-add per accumulator; the super-block scale d, the activation
// scale and the -dmin * m term (one fp16 MMA against the sub-block sums) are applied once per super-block.
// The only approximation is the 16-bit activation grid: absolute error at most 1.6e-5 of the block maximum.
//
// One persistent CTA per SM: 16 consumer warps, 3 finisher warps and 1 producer warp (five warps per scheduler). The producer streams 16-row x
// 8-super-block weight slabs with one tiled TMA copy each into a shared-memory ring. A consumer warp works on the
// same super-block of every tile (warp w of a half takes super-block w of the half's slab), so it keeps the activation
// fragments of that super-block in registers for a whole K chunk, loaded straight from the image in global memory:
// shared memory is read for the weights only, which is what bounds the rate of this kernel (the activation fragments
// of a unit are 4 KB against 2.3 KB of weights). Every wait on an mbarrier is bounded and ends in an abort flag plus a
// device status code.
#include "gemv_ring.cuh"
#include "q4k_units.cuh"

namespace infdev {
namespace {

constexpr int kConsumerWarps = 16;  // two halves of 8; consecutive ring stages alternate between the halves
constexpr int kStageWarps = 8;       // one warp per super-block of a stage
constexpr int kFinisherWarps = 3;  // each sums the consumers' partial results of every third tile and stores it
constexpr int kProducerWarp = kConsumerWarps + kFinisherWarps;  // 16 + 3 + 1 warps: five on each scheduler
constexpr int kThreads = (kProducerWarp + 1) * kWarp;
constexpr int kChunkBlocks = 16;  // super-blocks of K per pass over the tiles: two slabs, one per half
static_assert(kChunkBlocks == 2 * kGemvStageBlocks, "a consumer warp's super-block within a chunk is fixed by its half");

constexpr int kSquaresBytes = kConsumerWarps * kImageRows * 4;

template <int NMAT> constexpr size_t fixed_bytes() { return kRingControlBytes + kSquaresBytes + size_t(kFinisherWarps) * NMAT * kConsumerWarps * 128 * 4; }
template <int NMAT> constexpr int stage_count() {
  int stages = int((size_t(227) * 1024 - fixed_bytes<NMAT>()) / kQ4StageBytes);
  // Even, so that a slot always belongs to the same half of the consumers: a half that ran ahead in a slot of the other one could
  // find the parity of the phase before last and read the slot ahead of its own copy.
  return (stages > kMaxStages ? kMaxStages : stages) / 2 * 2;
}
template <int NMAT> constexpr size_t smem_bytes() { return fixed_bytes<NMAT>() + size_t(stage_count<NMAT>()) * kQ4StageBytes; }

// IMAGE: the activations come from an image; otherwise from p.image or, where that is null, from fp32.
template <int NMAT, int ROWS, bool IMAGE> __global__ void __launch_bounds__(kThreads, 1) q4k_decode_kernel(const __grid_constant__ GemvParams p) {
  constexpr int kStages = stage_count<NMAT>();
  extern __shared__ __align__(128) uint8_t smemRaw[];
  RingControl& ctl = *reinterpret_cast<RingControl*>(smemRaw);
  float* squaresOfBlock = reinterpret_cast<float*>(smemRaw + kRingControlBytes);  // [super-block][row]
  float* partial = reinterpret_cast<float*>(smemRaw + kRingControlBytes + kSquaresBytes);
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

  if (warp == kProducerWarp) {
    // ---- producer (one thread): weight slabs into the ring. The weights do not depend on the kernels before this
    // one, so the ring fills while they finish.
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int chunk = 0; chunk < chunks && ok; ++chunk) {
        const int chunkBlocks = min(kChunkBlocks, blocksPerRow - chunk * kChunkBlocks);
        const int groups = (chunkBlocks + kGemvStageBlocks - 1) / kGemvStageBlocks;
        for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
          const int segment = find_segment(p, tile);
          const int row0 = (tile - p.seg[segment].tile0) * kGemvTileRows;
          for (int mat = 0; mat < NMAT && ok; ++mat) {
            for (int grp = 0; grp < groups; ++grp, ++it) {
              const uint32_t slot = it % kStages, round = it / kStages;
              if (round > 0 && !mbar_wait_bounded(&ctl.empty[slot], (round - 1) & 1, abortFlag)) {
                *abortFlag = 1;
                atomicExch(p.status, kStatusBarrierTimeout);
                ok = false;
                break;
              }
              // One tiled copy moves the whole slab; bytes past the end of a row are zero-filled and still counted, so
              // the transaction size is always the full box.
              mbar_arrive_expect_tx(&ctl.full[slot], uint32_t(kQ4StageBytes));
              tma_load_2d(ring + size_t(slot) * kQ4StageBytes, &p.map[segment][mat], (chunk * (kChunkBlocks / kGemvStageBlocks) + grp) * (kGemvStageBlocks * kQ4BlockBytes / 8),
                          row0, &ctl.full[slot]);
            }
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

  if (warp >= kConsumerWarps) {
    // ---- finishers ----
    pdl_wait();
    finish_tiles<NMAT, kConsumerWarps, kFinisherWarps>(p, ctl, partial, warp - kConsumerWarps, chunks, lane);
    return;
  }

  // ---- consumers ----
  pdl_wait();  // the activations come from the kernels before this one
  const int g = lane >> 2, t = lane & 3, half = warp / kStageWarps, unit = warp % kStageWarps;
  const int laneRow = g * kQ4RowPitch + unit * kQ4BlockBytes;
  uint32_t it = 0, mine = half, slot = half, phase = 0;
  uint32_t bufferState = 0;  // bit b: parity of the next use of partial-sum buffer b; bit 4 + b: it has been used before
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int chunkBlocks = min(kChunkBlocks, blocksPerRow - chunk * kChunkBlocks);
    const int groups = (chunkBlocks + kGemvStageBlocks - 1) / kGemvStageBlocks;
    // With two slabs per tile the stages of a tile alternate between the halves (a chunk starts at an even stage,
    // only the last chunk of a row can be a single slab), with one slab every stage is slab 0: either way this warp
    // meets the same super-block in every tile of the chunk.
    const int myBlock = (groups == 2 ? half * kGemvStageBlocks : 0) + unit;
    const bool live = myBlock < chunkBlocks;
    Fragments fragments;
    if (live)  // with a norm every warp: the row is one chunk of 16 super-blocks; one of the CTAs stores what a warp normalises
      fragments = IMAGE || p.image
                      ? load_fragments<ROWS>(p.image + size_t(chunk * kChunkBlocks + myBlock) * kImageBlockBytes, lane)
                      : quantize_fragments<ROWS>(p.x + size_t(chunk * kChunkBlocks + myBlock) * 256, p.ldx, p.m, lane,
                                                 {p.norm, myBlock % int(gridDim.x) == int(blockIdx.x) ? p.normalised : nullptr, squaresOfBlock, myBlock});
    int buffer = 0;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, buffer = buffer == kFinisherWarps - 1 ? 0 : buffer + 1) {
      float total[NMAT][4];
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat)
        total[mat][0] = total[mat][1] = total[mat][2] = total[mat][3] = 0.f;
      // `mine` is the next stage of this half (they are the stages congruent to `half` modulo 2), `slot` and `phase`
      // its place in the ring.
      const int perTile = NMAT * groups;
      for (; mine < it + perTile; mine += 2, slot += 2) {
        if (slot >= kStages) {
          slot -= kStages;
          phase ^= 1;
        }
        const int mat = NMAT == 2 && int(mine - it) >= groups;
        if (!mbar_wait_bounded(&ctl.full[slot], phase, abortFlag)) {  // also leaves when another role raised the abort flag
          *abortFlag = 1;
          atomicExch(p.status, kStatusBarrierTimeout);
          break;
        }
        if (live) {
          const uint8_t* rows = ring + slot * kQ4StageBytes + laneRow;
          if (NMAT == 2 && mat)
            q4k_unit<ROWS>(rows, rows + 8 * kQ4RowPitch, t, fragments, total[NMAT - 1]);
          else
            q4k_unit<ROWS>(rows, rows + 8 * kQ4RowPitch, t, fragments, total[0]);
        }
        __syncwarp();
        if (lane == 0)
          mbar_arrive(&ctl.empty[slot]);
      }
      it += perTile;
      // Hand the partial sums of the K split to the buffer's finisher and go on with the next tile.
      const uint32_t parity = (bufferState >> buffer) & 1u;
      if (((bufferState >> (4 + buffer)) & 1u) && !mbar_wait_bounded(&ctl.partialFree[buffer], parity ^ 1u, abortFlag)) {
        *abortFlag = 1;
        atomicExch(p.status, kStatusBarrierTimeout);
      }
      bufferState = (bufferState ^ (1u << buffer)) | (16u << buffer);
      float* sums = partial + size_t(buffer) * NMAT * kConsumerWarps * 128;
#pragma unroll
      for (int mat = 0; mat < NMAT; ++mat) {
        reinterpret_cast<float4*>(sums + (mat * kConsumerWarps + warp) * 128)[lane] = make_float4(total[mat][0], total[mat][1], total[mat][2], total[mat][3]);
      }
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&ctl.partialReady[buffer]);
    }
  }
}

// One warp per (row, 256-value block).
__global__ void __launch_bounds__(256) activation_image_kernel(const float* x, int ldx, int m, int blocks, uint8_t* image) {
  pdl_launch_dependents();
  pdl_wait();
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= blocks * kImageRows)
    return;
  const int block = item >> 3, row = item & 7;
  uint8_t* out = image + size_t(block) * kImageBlockBytes;
  if (row >= m) {
    image_zero_block(out, row, lane);
    return;
  }
  const float4* src = reinterpret_cast<const float4*>(x + size_t(row) * ldx + size_t(block) * 256 + lane * 8);
  const float4 lo = src[0], hi = src[1];
  const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  image_store_block(out, row, lane, v);
}

template <int NMAT, int ROWS, bool IMAGE> cudaError_t launch_kind(const GemvParams& p, int sms, cudaStream_t stream) {
  static PerDeviceOnce configured;
  constexpr size_t bytes = smem_bytes<NMAT>();
  if (cudaError_t e = configure_shared_memory(q4k_decode_kernel<NMAT, ROWS, IMAGE>, bytes, configured))
    return e;
  const int grid = p.tiles < sms ? p.tiles : sms;
  launch_kernel<1>(q4k_decode_kernel<NMAT, ROWS, IMAGE>, grid, kThreads, bytes, stream, p);
  return cudaGetLastError();
}
// A launch that is a start and an end only feels the code that it carries and does not run: with its image launch 512 x 8192 with eight
// rows 5.3 us, 5.1 in a kernel without, a pair of 1024 x 4096 5.3 and 5.1. With more tiles than SMs one kernel for both kinds of activations
// is no slower, and projections that follow each other share its instructions (those of a layer with eight rows, the last of them from
// an image of its own, 44.1 us; 44.7 with a kernel for that).
template <int NMAT, int ROWS> cudaError_t launch(const GemvParams& p, int sms, cudaStream_t stream) {
  return p.image && p.tiles <= sms ? launch_kind<NMAT, ROWS, true>(p, sms, stream) : launch_kind<NMAT, ROWS, false>(p, sms, stream);
}

// One or two rows pay for their own columns only: 12288 x 4096 with its image launch 12.5 -> 11.0 us at one row, 11.5 at two;
// all projections of a layer 54.4 -> 48.8 and 52.7 us. Four rows in two sub-blocks a column set measured 56.4 us against 55.0
// (the fragments and eight sums of two sets spill at 96 registers), so three rows and more take the plain columns.
template <int NMAT> cudaError_t launch_rows(const GemvParams& p, int sms, cudaStream_t stream) {
  return p.m <= 1   ? launch<NMAT, 1>(p, sms, stream)
         : p.m == 2 ? launch<NMAT, 2>(p, sms, stream)
                    : launch<NMAT, 8>(p, sms, stream);
}

}  // namespace

cudaError_t q4k_decode_launch(bool pair, const GemvParams& p, int sms, cudaStream_t stream) {
  return pair ? launch_rows<2>(p, sms, stream) : launch_rows<1>(p, sms, stream);
}

cudaError_t activation_image_launch(const float* x, int ldx, int m, int k, uint8_t* image, cudaStream_t stream) {
  const int blocks = k / 256;
  launch_kernel<1>(activation_image_kernel, (blocks * kImageRows + 7) / 8, 256, 0, stream, x, ldx, m, blocks, image);
  return cudaGetLastError();
}

}  // namespace infdev
