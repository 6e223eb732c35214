// On-GPU sampling, query packing and draft verification.
//
// sample_kernel <- sample_logits (native_ops.metal:122-224). The reference runs the temperature path on one
// thread (a serial insertion sort over 248,320 logits); here a cluster of CTAs finds the top-k set, and only the
// final <= 64-step softmax / top-p / inverse-CDF walk is serial, in exactly the reference's order.
// RNG: Philox4x32-10 keyed by the slot seed, counter = absolute index of the sampled token in its sequence,
// so a sequence draws the same variates whether it runs alone, batched or speculatively (the reference
// advances an xorshift64 state per sample and commits it on the host, engine.cpp:210-211).
#include <cooperative_groups.h>
#include "common.cuh"
#include "ops.h"

namespace infdev {
namespace {

constexpr uint32_t kUnbound = 0xffffffffu;

__device__ __forceinline__ const infdev_query& query_of_logit(const infdev_query* queries, uint32_t row) {
  while (!queries->samples || row >= queries->logit + queries->samples)
    ++queries;
  return *queries;
}

__device__ __forceinline__ float philox_uniform(uint64_t key, uint64_t counter) {
  uint32_t c0 = uint32_t(counter), c1 = uint32_t(counter >> 32), c2 = 0, c3 = 0, k0 = uint32_t(key), k1 = uint32_t(key >> 32);
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint32_t h0 = __umulhi(0xD2511F53u, c0), l0 = 0xD2511F53u * c0, h1 = __umulhi(0xCD9E8D57u, c2), l1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = h1 ^ c1 ^ k0, n2 = h0 ^ c3 ^ k1;
    c0 = n0, c1 = l1, c2 = n2, c3 = l0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return float(c0 >> 8) * (1.0f / 16777216.0f);
}

// Order-preserving map float -> uint32 (larger float = larger key).
__device__ __forceinline__ uint32_t sortable(float v) {
  const uint32_t bits = __float_as_uint(v);
  return bits ^ ((bits & 0x80000000u) ? 0xffffffffu : 0x80000000u);
}

// ---- one row of logits, a cluster of up to eight CTAs -----------------------------------------------------------------
// grid (C, count), clusters of C = 1, 2, 4 or 8 CTAs of 512 threads: a cluster samples one row, each CTA looks at a C-th of the
// vocabulary and the results meet in the shared memory of the cluster's first CTA. A row is 1 MB that the output head
// has just left in the L2, so what bounds it is how many SMs ask for it and how often; one CTA per row needed 20 us for
// the argmax of eight rows of 248320 logits and 361 us for their top-40 (five walks over the row, and a histogram whose
// shared-memory atomics nearly all hit the few bins that hold the exponents of ordinary logits). C: see sample_launch.
//
// Top-k without a histogram: the cluster's threads fall into 128 groups that hold 128 disjoint parts of the row, so the
// wanted-th largest of their 128 maxima has at least `wanted` logits at or above it and can serve as a threshold; a second walk
// collects what reaches it (about 50 logits for a top-40 of random ones), and the exact order among those, value then index, is
// found by counting. Divisions by the temperature are left to the few logits near the threshold. Equal logits can make that
// collection arbitrarily large: a row whose mask leaves few logits has its threshold among the masked ones. The first walk
// therefore counts the logits that equal their part's maximum; where too many equal the threshold, only what lies above it is
// collected, each warp looks for the first equal ones of a contiguous piece of the row, and the earliest of them fill the set up
// (ten logits of 248320 left by a mask, eight rows: 32 us; 548 with one CTA and a radix select). Where the collection does
// not fit all the same, the first CTA walks the row by itself with that select (radix_candidates below).
constexpr int kMaxClusterCtas = 8, kClusterThreads = 512, kClusterWarps = kClusterThreads / kWarp;
constexpr int kParts = 128;         // disjoint parts whose maxima the threshold is taken from
constexpr int kCandidates = 2048;   // collected logits that fit
constexpr int kMostTied = 256;      // more at the threshold than these stay out of the collection (ranking all of 1003 took 40 us)
constexpr int kMostWanted = 64;
constexpr int kChunks = 128;        // plain temperature sampling sums the row in this many contiguous pieces per CTA
static_assert(kChunks % (2 * kClusterWarps) == 0, "a warp takes two pieces at a time, all of them of its own CTA");

struct SampleShared {
  float maxima[kParts];  // of the parts; of the warps for the argmax
  int indices[kParts];
  float value[kCandidates];
  int index[kCandidates];
  float sortedValue[2 * kMostWanted], weight[kMostWanted];
  int sortedIndex[2 * kMostWanted];
  int tie[kClusterWarps][kMostWanted], tieCount[kClusterWarps];  // the first logits equal to the threshold in this warp's piece
  double chunkSum[kMaxClusterCtas * kChunks];
  uint32_t histogram[256];
  uint32_t equals[kParts];  // logits of the part that equal its maximum
  uint32_t count, prefix, remaining, tied;
  float threshold;
  int owner;
  double before;
};

// Calls f(logit, index) for this thread's logits of the CTA's part of the row, in ascending order of the index.
template <class F> __device__ __forceinline__ void for_part(const float* row, int vocab, uint32_t part, uint32_t ctas, F f) {
  if (vocab % 4 == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int quads = vocab / 4, per = (quads + int(ctas) - 1) / int(ctas), last = min(quads, int(part + 1) * per);
#pragma unroll 4
    for (int j = int(part) * per + int(threadIdx.x); j < last; j += kClusterThreads) {
      const float4 v = row4[j];
      f(v.x, 4 * j), f(v.y, 4 * j + 1), f(v.z, 4 * j + 2), f(v.w, 4 * j + 3);
    }
    return;
  }
  const int per = (vocab + int(ctas) - 1) / int(ctas), last = min(vocab, int(part + 1) * per);
  for (int j = int(part) * per + int(threadIdx.x); j < last; j += kClusterThreads)
    f(row[j], j);
}

__device__ __forceinline__ bool ahead(float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); }

// The wanted largest of logit / temperature, ties by the earliest index, by a radix select over the order-preserving
// integer image, for rows with too many equal logits for the cluster's collection. One CTA; leaves the (unsorted) set in
// sh.value / sh.index and returns its size. A logit that is not a number belongs to no set, as in the cluster's collection.
__device__ uint32_t radix_candidates(SampleShared& sh, const float* row, int vocab, float temperature, uint32_t wanted) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (tid == 0)
    sh.prefix = 0, sh.remaining = wanted, sh.count = 0;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    if (tid < 256)
      sh.histogram[tid] = 0;
    __syncthreads();
    const uint32_t prefix = sh.prefix, prefixMask = pass ? (0xffffffffu << (shift + 8)) : 0u;
    for (int j = tid; j < vocab; j += kClusterThreads) {
      const float value = row[j] / temperature;
      const uint32_t key = sortable(value);
      if (value == value && (key & prefixMask) == prefix)
        atomicAdd(&sh.histogram[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t remaining = sh.remaining;
      int bin = 255;
      for (; bin > 0; --bin) {
        if (sh.histogram[bin] >= remaining)
          break;
        remaining -= sh.histogram[bin];
      }
      sh.prefix = prefix | (uint32_t(bin) << shift);
      sh.remaining = remaining;
    }
    __syncthreads();
  }
  // sh.prefix is now the key of the wanted-th largest value; sh.remaining of the elements equal to it belong to the set
  // (the ones with the smallest indices, as the reference's stable insertion keeps the earliest).
  const uint32_t threshold = sh.prefix;
  for (int j = tid; j < vocab; j += kClusterThreads) {
    const float value = row[j] / temperature;
    if (value == value && sortable(value) > threshold) {
      const uint32_t at = atomicAdd(&sh.count, 1u);
      if (at < uint32_t(kMostWanted))
        sh.value[at] = value, sh.index[at] = j;
    }
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t count = min(sh.count, uint32_t(kMostWanted)), need = sh.remaining;
    for (int j = 0; j < vocab && need && count < uint32_t(kMostWanted); ++j) {  // serial scan in index order
      const float value = row[j] / temperature;
      if (value == value && sortable(value) == threshold) {
        sh.value[count] = value, sh.index[count] = j;
        ++count;
        --need;
      }
    }
    sh.count = count;
  }
  __syncthreads();
  return sh.count;
}

// mode 0: target sampling; mode 1: MTP drafting (always argmax, and bumps the drafter query's position,
// native_ops.metal:128-129).
__global__ void __launch_bounds__(kClusterThreads, 1)
    sample_kernel(const float* logits, int vocab, infdev_query* queries, uint32_t mode, int32_t* tokens) {
  __shared__ SampleShared sh;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  pdl_launch_dependents();
  const uint32_t i = blockIdx.y, part = cluster.block_rank(), ctas = cluster.num_blocks();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  SampleShared& first = *cluster.map_shared_rank(&sh, 0);
  if (tid == 0)
    sh.count = 0, sh.tied = 0;
  cluster.sync();  // every CTA of the cluster runs, and the first one's counter is zero
  pdl_wait();
  const infdev_query info = query_of_logit(queries, i);
  const float* row = logits + size_t(i) * vocab;

  if (mode || info.temperature <= 0.f) {
    // first-index argmax (native_ops.metal:137-158)
    float best = -INFINITY;
    int index = 0;
    for_part(row, vocab, part, ctas, [&](float v, int j) {
      if (v > best)
        best = v, index = j;
    });
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, index, o);
      if (ahead(ov, oi, best, index))
        best = ov, index = oi;
    }
    if (lane == 0)
      first.maxima[part * kClusterWarps + warp] = best, first.indices[part * kClusterWarps + warp] = index;
    cluster.sync();
    if (part || warp)
      return;
    best = -INFINITY, index = 0;
    for (int w = lane; w < int(ctas) * kClusterWarps; w += 32)
      if (ahead(sh.maxima[w], sh.indices[w], best, index))
        best = sh.maxima[w], index = sh.indices[w];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, index, o);
      if (ahead(ov, oi, best, index))
        best = ov, index = oi;
    }
    if (lane == 0) {
      tokens[i] = index;
      if (mode == 1) {
        infdev_query* q = queries;
        while (!q->samples || i >= q->logit + q->samples)
          ++q;
        ++q->position;
      }
    }
    return;
  }

  const float temperature = info.temperature;
  const float random = philox_uniform(info.seed, uint64_t(info.position) + info.count - info.samples + (i - info.logit) + 1);
  // the maximum of every part (4 x ctas lanes) and how many logits equal it, for every CTA of the cluster
  float maximum = -INFINITY;
  uint32_t equals = 0;
  for_part(row, vocab, part, ctas, [&](float v, int) {
    equals = v > maximum ? 1u : equals + (v == maximum ? 1u : 0u);
    maximum = fmaxf(maximum, v);
  });
  const uint32_t lanes = 4 * ctas, mine = (part * kClusterThreads + tid) / lanes;
  const float own = maximum;
  for (uint32_t o = lanes / 2; o; o >>= 1)
    maximum = fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, o));
  equals = own == maximum ? equals : 0u;
  for (uint32_t o = lanes / 2; o; o >>= 1)
    equals += __shfl_xor_sync(0xffffffffu, equals, o);
  if (lane % lanes < ctas) {
    SampleShared& to = *cluster.map_shared_rank(&sh, lane % lanes);
    to.maxima[mine] = maximum, to.equals[mine] = equals;
  }
  cluster.sync();

  if (info.topK == 0) {
    // plain temperature sampling over the vocabulary, top-p ignored (native_ops.metal:172-188). The row is summed in
    // double precision in contiguous chunks, 128 of them per CTA and two at a time per warp; the first CTA finds the chunk
    // in which the cumulative sum passes the target and walks that one in vocabulary order. What bounds it is latency, so everything is
    // asked for eight values at a time: one and eight rows of 248320 logits 33.4 -> 17.0 and 37.5 -> 20.5 us, in the order of addition as before.
    maximum = fmaxf(fmaxf(sh.maxima[lane], sh.maxima[lane + 32]), fmaxf(sh.maxima[lane + 64], sh.maxima[lane + 96]));
    maximum = warp_max(maximum) / temperature;
    const int chunks = int(ctas) * kChunks, chunk = (vocab + chunks - 1) / chunks;
    for (int c = int(part) * kChunks + warp; c < int(part + 1) * kChunks; c += 2 * kClusterWarps) {
      double sum[2] = {0.0, 0.0};  // of two chunks at a time
      int from[2], end[2];
#pragma unroll
      for (int s = 0; s < 2; ++s)
        from[s] = (c + s * kClusterWarps) * chunk, end[s] = min(vocab, from[s] + chunk);
      for (int at = lane; at < chunk; at += 8 * kWarp) {
        float value[2][8];
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int e = 0; e < 8; ++e)
            value[s][e] = from[s] + at + kWarp * e < end[s] ? row[from[s] + at + kWarp * e] : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
          for (int s = 0; s < 2; ++s)
            if (from[s] + at + kWarp * e < end[s])
              sum[s] += double(expf(value[s][e] / temperature - maximum));
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
#pragma unroll
        for (int o = 16; o; o >>= 1)
          sum[s] += __shfl_xor_sync(0xffffffffu, sum[s], o);
        if (lane == 0)
          first.chunkSum[c + s * kClusterWarps] = sum[s];
      }
    }
    cluster.sync();
    if (part || warp)
      return;
    // lane l holds the sum of its consecutive chunks; exclusive scan over the lanes
    const int perLane = chunks / 32;
    double lanes32 = 0.0;
#pragma unroll 4
    for (int c = 0; c < perLane; ++c)
      lanes32 += sh.chunkSum[lane * perLane + c];
    double inclusive = lanes32;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double other = __shfl_up_sync(0xffffffffu, inclusive, o);
      if (lane >= o)
        inclusive += other;
    }
    const double target = double(random) * __shfl_sync(0xffffffffu, inclusive, 31);
    const uint32_t reached = __ballot_sync(0xffffffffu, inclusive >= target);
    const int ownerLane = reached ? __ffs(reached) - 1 : 31;
    if (lane == ownerLane) {
      double cumulative = inclusive - lanes32;
      int owner = lane * perLane;
      const int end = owner + perLane - 1;
      for (bool before = true; before;) {  // the sums of eight chunks are asked for at once
        double sums[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
          sums[e] = owner + e < end ? sh.chunkSum[owner + e] : 0.0;
        const int at = owner;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          before = before && at + e < end && cumulative + sums[e] < target;
          if (before)
            cumulative += sums[e], ++owner;
        }
      }
      sh.owner = owner, sh.before = cumulative;
    }
    __syncwarp();
    double cumulative = sh.before;
    const int a = sh.owner * chunk, b = min(vocab, a + chunk);
    int token = vocab - 1;
    float value[8];
    for (int base = a, e = 0; base < b; base += 32, ++e) {
      const int j = base + lane;
      if (e % 8 == 0)
#pragma unroll
        for (int ahead = 0; ahead < 8; ++ahead)
          value[ahead] = j + 32 * ahead < b ? row[j + 32 * ahead] : 0.f;
      double running = j < b ? double(expf(value[0] / temperature - maximum)) : 0.0;
#pragma unroll
      for (int ahead = 0; ahead < 7; ++ahead)
        value[ahead] = value[ahead + 1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, running, o);
        if (lane >= o)
          running += other;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, j < b && cumulative + running >= target);
      if (hit) {
        token = base + __ffs(hit) - 1;
        break;
      }
      cumulative += __shfl_sync(0xffffffffu, running, 31);
    }
    if (lane == 0)
      tokens[i] = token;
    return;
  }

  // ---- top-k (<= 64) ----
  const uint32_t wanted = min(uint32_t(info.topK), uint32_t(kMostWanted));
  if (tid < kParts) {
    const float limit = sh.maxima[tid];
    uint32_t above = 0, level = 0;
#pragma unroll 8
    for (int w = 0; w < kParts; ++w) {
      above += sh.maxima[w] > limit ? 1u : 0u;
      level += sh.maxima[w] >= limit ? 1u : 0u;
    }
    if (above < wanted && wanted <= level)  // the parts whose maximum is the threshold, which all write it
      sh.threshold = limit, atomicAdd(&sh.tied, sh.equals[tid]);
  }
  __syncthreads();
  const float threshold = sh.threshold / temperature;
  // A quotient reaches the threshold's only if its logit comes within rounding of it (or if the quotients overflow).
  const float slack = fmaxf(fmaxf(fabsf(sh.threshold) * 1.0e-6f, 1.0e-36f), temperature * 1.0e-44f), near = fabsf(threshold) < INFINITY ? sh.threshold - slack : -INFINITY;
  const bool ties = sh.tied <= uint32_t(kMostTied);  // the collection holds what equals the threshold too
  for_part(row, vocab, part, ctas, [&](float v, int j) {
    if (!(v >= near))
      return;
    const float value = v / temperature;
    if (ties ? value >= threshold : value > threshold) {
      const uint32_t at = atomicAdd(&first.count, 1u);
      if (at < uint32_t(kCandidates))
        first.value[at] = value, first.index[at] = j;
    }
  });
  cluster.sync();
  if (ties && part)
    return;
  uint32_t count = first.count;
  if (!ties && count < wanted) {
    // every warp: the first logits of its contiguous piece that equal the threshold, no more than are missing
    const uint32_t missing = wanted - count;
    const int pieces = int(ctas) * kClusterWarps, per = (vocab + pieces - 1) / pieces, from = (int(part) * kClusterWarps + warp) * per, to = min(vocab, from + per);
    uint32_t have = 0;
    for (int base = from; base < to && have < missing; base += 4 * kWarp) {
      float value[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = base + kWarp * e + lane;
        value[e] = j < to ? row[j] / temperature : NAN;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t equal = __ballot_sync(0xffffffffu, value[e] == threshold), before = have + __popc(equal & ((1u << lane) - 1u));
        if (value[e] == threshold && before < missing)
          sh.tie[warp][before] = base + kWarp * e + lane;
        have += __popc(equal);
      }
    }
    if (lane == 0)
      sh.tieCount[warp] = int(min(have, missing));
    cluster.sync();
    if (part == 0 && warp == 0) {
      // the pieces in the order of the vocabulary
      uint32_t filled = 0;
      for (uint32_t rank = 0; rank < ctas && filled < missing; ++rank) {
        const SampleShared& other = *cluster.map_shared_rank(&sh, rank);
        for (int w = 0; w < kClusterWarps && filled < missing; ++w) {
          const uint32_t take = min(uint32_t(other.tieCount[w]), missing - filled);
          for (uint32_t e = lane; e < take; e += kWarp)
            sh.value[count + filled + e] = threshold, sh.index[count + filled + e] = other.tie[w][e];
          filled += take;
        }
      }
      if (lane == 0)
        sh.count = count + filled;
    }
    cluster.sync();  // the others' lists have been read
    count = sh.count;  // of use in the first CTA
  } else if (!ties) {
    cluster.sync();  // all have read the first CTA's count
  }
  if (part)
    return;
  if (count > uint32_t(kCandidates))
    count = radix_candidates(sh, row, vocab, temperature, wanted);
  // the exact order: value descending, index ascending
  for (uint32_t a = tid; a < count; a += kClusterThreads) {
    const float v = sh.value[a];
    const int x = sh.index[a];
    uint32_t rank = 0;
    for (uint32_t b = 0; b < count; ++b)
      rank += ahead(sh.value[b], sh.index[b], v, x) ? 1u : 0u;
    if (rank < wanted)
      sh.sortedValue[rank] = v, sh.sortedIndex[rank] = x;
  }
  __syncthreads();
  const uint32_t kept = min(count, wanted);
  if (tid < int(kept))
    sh.weight[tid] = expf(sh.sortedValue[tid] - sh.sortedValue[0]);
  __syncthreads();
  if (tid == 0 && !kept)  // not one comparable logit
    tokens[i] = 0;
  if (tid == 0 && kept) {
    // softmax over the set, top-p cut, inverse CDF, summed in the reference's order (native_ops.metal:208-223)
    float total = 0.f;
#pragma unroll 8
    for (uint32_t j = 0; j < kept; ++j)
      total += sh.weight[j];
    const float limit = info.topP * total;
    // eight weights at a time: one by one every step waits for the shared memory (16.6 -> 16.0 us for the top-40 of eight rows of 248320 logits)
    auto walk = [&](uint32_t end, float limit, float& sum) {  // adds up weights until they are no longer below the limit; how many they are
      uint32_t taken = 0;
      for (bool more = true; more;) {
        float weight[8];
        const uint32_t at = taken;
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e)
          weight[e] = at + e < end ? sh.weight[at + e] : 0.f;
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e)
          if (more)
            sum += weight[e], ++taken, more = taken < end && sum < limit;
      }
      return taken;
    };
    float nucleus = 0.f, cumulative = 0.f;
    const uint32_t keep = walk(kept, limit, nucleus);
    tokens[i] = sh.sortedIndex[walk(keep, random * nucleus, cumulative) - 1];
  }
}

// Finishes the per-query records of one pass on the device: forward()'s packing loop (forward.cpp:171-191).
// in[i] carries slot, count, position, state, sampling parameters, seed and (in `samples`) the slot's
// requested-token count; out gets start, samples, logit offsets and the state addresses.
// meta[0] = rows, meta[1] = logit rows, meta[2] = flags (1 sequential, 2 prefill).
__global__ void pack_queries_kernel(const infdev_query* in, int count, int drafting, uint32_t draftWidth, const uint64_t* statePrevious,
                                    const uint64_t* stateNext, uint64_t candidateBase, uint64_t stateBytes, infdev_query* out, uint32_t* meta) {
  pdl_launch_dependents();
  pdl_wait();
  // One lane per query (at most 32): the records and the state addresses live in host-visible memory, so every read is
  // a trip over PCIe; the lanes make theirs at the same time and the running totals come from a warp scan.
  const uint32_t lane = threadIdx.x;
  if (blockIdx.x || lane >= 32)
    return;
  infdev_query query = {};
  bool keep = false, speculative = false;
  if (int(lane) < count) {
    query = in[lane];
    speculative = query.state != kUnbound;
    keep = !(drafting && !speculative);
  }
  uint32_t flags = 0;
  if (keep) {
    const uint32_t requested = query.samples;
    if (drafting)
      query.count = 1;
    query.samples = drafting ? 1 : speculative ? query.count : (query.position + query.count == requested ? 1u : 0u);
    flags = ((speculative || query.count == 1) ? 1u : 0u) | ((!speculative && query.count > 1) ? 2u : 0u);
    query.previous = query.position ? statePrevious[query.slot] : 0;
    query.next = speculative ? candidateBase + uint64_t(query.state) * stateBytes : stateNext[query.slot];
  }
  // inclusive scans of rows, logit rows and kept queries over the lanes
  uint32_t rows = keep ? query.count : 0u, logits = keep ? query.samples : 0u, packed = keep ? 1u : 0u;
#pragma unroll
  for (int step = 1; step < 32; step <<= 1) {
    const uint32_t r = __shfl_up_sync(0xffffffffu, rows, step), l = __shfl_up_sync(0xffffffffu, logits, step), k = __shfl_up_sync(0xffffffffu, packed, step);
    if (int(lane) >= step)
      rows += r, logits += l, packed += k;
  }
  flags = __reduce_or_sync(0xffffffffu, flags);
  if (keep) {
    query.start = rows - query.count;
    query.logit = logits - query.samples;
    out[packed - 1] = query;
  }
  (void)draftWidth;
  if (lane == 31) {
    meta[0] = rows;
    meta[1] = logits;
    meta[2] = flags;
    meta[3] = packed;
  }
}

// The acceptance loop of Engine::schedule (engine.cpp:205-216) on the device, one thread per query. For query i it
// walks the sampled rows exactly as the host loop does: a sampled token is emitted; a stop token ends the walk after
// this token; a speculative query goes on to the next row only while the sampled token equals the drafter's proposal
// for that row and fewer than draftWidth proposals have been accepted. verdict[3 i .. 3 i + 2] = accepted proposals,
// emitted tokens, stopped (0 / 1). stops: [slot][stopStride] token ids, stopCounts[slot] of them valid.
__global__ void verify_drafts_kernel(const infdev_query* queries, int count, const int32_t* sampled, const int32_t* proposed, uint32_t draftWidth,
                                     const int32_t* stops, uint32_t stopStride, const uint32_t* stopCounts, uint32_t* verdict) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count)
    return;
  const infdev_query& query = queries[i];
  const bool speculative = query.state != kUnbound;
  const uint32_t column = speculative ? query.state / query.count : 0;
  uint32_t accepted = 0, emitted = 0, stopped = 0;
  for (uint32_t s = 0; s < query.samples && !stopped; ++s) {
    const int32_t token = sampled[query.logit + s];
    ++emitted;
    for (uint32_t k = 0; k < stopCounts[query.slot]; ++k)
      stopped |= stops[size_t(query.slot) * stopStride + k] == token ? 1u : 0u;
    if (!speculative || s == draftWidth || token != proposed[(s + 1) * 8 + column])
      break;
    ++accepted;
  }
  verdict[3 * i] = accepted;
  verdict[3 * i + 1] = emitted;
  verdict[3 * i + 2] = stopped;
}

// Copies the accepted candidate state row of each speculative query to the slot's next state buffer
// (engine.cpp:217-218), driven by the verdicts of verify_drafts_kernel. grid (chunks, queries).
__global__ void __launch_bounds__(256) commit_states_kernel(const infdev_query* queries, const uint32_t* verdict, const uint64_t* stateNext,
                                                            uint64_t candidateBase, uint64_t stateBytes) {
  pdl_launch_dependents();
  pdl_wait();
  const infdev_query& query = queries[blockIdx.y];
  if (query.state == kUnbound)
    return;
  const uint4* src = reinterpret_cast<const uint4*>(candidateBase + uint64_t(query.state + verdict[3 * blockIdx.y]) * stateBytes);
  uint4* dst = reinterpret_cast<uint4*>(stateNext[query.slot]);
  const size_t total = stateBytes / 16;
  for (size_t at = size_t(blockIdx.x) * blockDim.x + threadIdx.x; at < total; at += size_t(gridDim.x) * blockDim.x)
    dst[at] = src[at];
}

}  // namespace

cudaError_t sample_launch(const float* logits, int vocab, infdev_query* queries, int64_t count, uint32_t mode, int32_t* tokens, int sms,
                          cudaStream_t stream) {
  if (count <= 0)
    return cudaSuccess;
  // As many CTAs for a row as leave every one an SM of its own and a float4 per thread: 40 rows of 248320 logits with eight CTAs
  // each 24.5 us (argmax) and 66.8 (top-40), with two 14.8 and 38.6; eight rows with eight CTAs each 5.9 and 17.5, 1003 logits a
  // row 53 us with eight (most warps had none, and the threshold let everything through), 9 with one.
  unsigned ctas = kMaxClusterCtas;
  while (ctas > 1 && (count * int64_t(ctas) > sms || vocab < int(ctas) * kClusterThreads * 4))
    ctas /= 2;
  return launch_clusters<2>(ctas, sample_kernel, dim3(ctas, unsigned(count)), kClusterThreads, 0, stream, logits, vocab, queries, mode, tokens);
}

cudaError_t pack_queries_launch(const infdev_query* in, int count, int drafting, uint32_t draftWidth, const uint64_t* statePrevious,
                                const uint64_t* stateNext, uint64_t candidateBase, uint64_t stateBytes, infdev_query* out, uint32_t* meta,
                                cudaStream_t stream) {
  launch_kernel(pack_queries_kernel, 1, 32, 0, stream, in, count, drafting, draftWidth, statePrevious, stateNext, candidateBase, stateBytes, out, meta);
  return cudaGetLastError();
}

cudaError_t verify_drafts_launch(const infdev_query* queries, int count, const int32_t* sampled, const int32_t* proposed, uint32_t draftWidth,
                                 const int32_t* stops, uint32_t stopStride, const uint32_t* stopCounts, uint32_t* verdict, cudaStream_t stream) {
  if (count <= 0)
    return cudaSuccess;
  launch_kernel(verify_drafts_kernel, 1, 32, 0, stream, queries, count, sampled, proposed, draftWidth, stops, stopStride, stopCounts, verdict);
  return cudaGetLastError();
}

cudaError_t commit_states_launch(const infdev_query* queries, int count, const uint32_t* verdict, const uint64_t* stateNext,
                                 uint64_t candidateBase, uint64_t stateBytes, cudaStream_t stream) {
  if (count <= 0)
    return cudaSuccess;
  launch_kernel(commit_states_kernel, dim3(64, unsigned(count)), 256, 0, stream, queries, verdict, stateNext, candidateBase, stateBytes);
  return cudaGetLastError();
}

}  // namespace infdev
