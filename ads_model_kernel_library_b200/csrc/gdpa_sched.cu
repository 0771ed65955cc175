// Device-side builder of the longest-first work list walked by the persistent GDPA kernels.
//
// Forward items are (sequence, head, 256-row Q block) weighted by the number of KV tiles of the
// sequence; backward items are (sequence, head, 128-row KV tile) weighted by the number of Q tiles.
// The list is a counting sort by weight, heaviest first, built by one thread block without any
// host synchronisation.  Buffer layout: int32 header {count, mode, 0, 0}, then one int4
// {sequence, head, block, weight} per item.
#include "gdpa_common.cuh"
#include "gdpa_launch.h"

namespace gdpa {

namespace {

constexpr int kSchedThreads = 1024;
constexpr int kBins = 4096;

__device__ __forceinline__ void seq_geometry(const SchedArgs& a, int b, int& nblk, int& weight) {
  long long s0, e0;
  seq_bounds(a.q_off, b, a.off64, s0, e0);
  long long lq = e0 - s0;
  int kb = b;
  if (a.kv_index != nullptr) {  // an entry beyond the KV batch is clamped, as the kernels do
    kb = static_cast<int>(load_offset(a.kv_index, b, a.off64));
    kb = kb < 0 ? 0 : (kb >= a.kv_batch ? a.kv_batch - 1 : kb);
  }
  seq_bounds(a.kv_off, kb, a.off64, s0, e0);
  long long lkv = e0 - s0;
  lq = lq < 0 ? 0 : (lq < a.max_q ? lq : a.max_q);
  lkv = lkv < 0 ? 0 : (lkv < a.max_kv ? lkv : a.max_kv);
  const int nq = static_cast<int>((lq + kTile - 1) / kTile);
  const int nkv = static_cast<int>((lkv + kTile - 1) / kTile);
  if (a.mode == 0) {
    nblk = static_cast<int>((lq + kFwdQBlock - 1) / kFwdQBlock);
    weight = nkv;
  } else {
    nblk = nkv;
    weight = nq;
  }
  if (weight > kBins - 1) weight = kBins - 1;
}

// Latency-bound: one block, a few thousand items, and the forward or backward kernel waits for it.  What it costs is the
// chain of dependent steps, so: only the bins that a sequence of the given maximum length can have are cleared and
// scanned (17 of 4096 for 2048 tokens), the scan gives each thread its own run of neighbouring bins (a warp reads
// consecutive words, no bank conflicts) instead of one warp walking all of them, and the items of a chunk of 1024
// sequences are written by all warps together, 32 consecutive items (512 bytes) per store, instead of each thread
// writing the items of one sequence one after another (13 us for 8 sequences, 26 us for 1024, a call of 256 short
// sequences 86.7 -> 81.8 us in all).
__global__ void __launch_bounds__(kSchedThreads, 1) gdpa_build_schedule_kernel(const SchedArgs a) {
  __shared__ int hist[kBins];
  __shared__ int warp_sum[kSchedThreads / 32];
  __shared__ int4 seq[kSchedThreads];  // of the sequences of one chunk: first slot, blocks, weight, -
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int longest = a.mode == 0 ? a.max_kv : a.max_q;
  const int bins = min(kBins, (longest > 0 ? (longest - 1) / kTile + 1 : 0) + 1);  // weights 0 .. bins - 1
  const long long cap = a.capacity_items;
  for (int i = t; i < bins; i += kSchedThreads) hist[i] = 0;
  __syncthreads();
  int nblk = 0, w = 0;  // of this thread's sequence of the last chunk: the only one unless the batch is large
  for (int b = t; b < a.batch; b += kSchedThreads) {
    seq_geometry(a, b, nblk, w);
    if (nblk > 0) atomicAdd(&hist[w], nblk * a.heads);
  }
  __syncthreads();
  // Exclusive prefix over bins from the heaviest down: hist[w] becomes the first slot of weight w.  Thread t owns the
  // `per` bins from bins - 1 - t * per down.
  const int per = (bins + kSchedThreads - 1) / kSchedThreads;
  const int hi = bins - 1 - t * per;
  int sum = 0;
  for (int i = 0; i < per; ++i) sum += hi - i >= 0 ? hist[hi - i] : 0;
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += n;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  // every warp scans the 32 warp totals for itself
  int before = warp_sum[lane];
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, before, d);
    if (lane >= d) before += n;
  }
  const int total = __shfl_sync(0xffffffffu, before, 31);
  before = __shfl_sync(0xffffffffu, before, warp > 0 ? warp - 1 : 0);
  int run = incl - sum + (warp > 0 ? before : 0);
  for (int i = 0; i < per; ++i) {
    if (hi - i < 0) break;
    const int c = hist[hi - i];
    hist[hi - i] = run;
    run += c;
  }
  __syncthreads();
  int4* items = reinterpret_cast<int4*>(a.sched + kSchedHeaderInts);
  for (int b0 = 0; b0 < a.batch; b0 += kSchedThreads) {
    const int n = min(kSchedThreads, a.batch - b0);
    if (t < n) {
      if (a.batch > kSchedThreads) seq_geometry(a, b0 + t, nblk, w);
      const int count = nblk * a.heads;
      seq[t] = make_int4(count > 0 ? atomicAdd(&hist[w], count) : 0, nblk, w, 0);
    }
    __syncthreads();
    for (int i = warp; i < n; i += kSchedThreads / 32) {
      const int4 sq = seq[i];
      const int count = sq.y * a.heads;
      for (int k = lane; k < count; k += 32) {
        const long long slot = static_cast<long long>(sq.x) + k;
        const int h = k / sq.y;
        if (slot < cap) items[slot] = make_int4(b0 + i, h, k - h * sq.y, sq.z);
      }
    }
    __syncthreads();
  }
  if (t == 0) {
    a.sched[0] = static_cast<int>(total < cap ? total : cap);
    a.sched[1] = a.mode;
    a.sched[2] = total;  // items the batch needs; larger than [0] only if the buffer was too small
    a.sched[3] = 0;
  }
}

}  // namespace

int launch_build_schedule(const SchedArgs& a, cudaStream_t stream) {
  gdpa_build_schedule_kernel<<<1, kSchedThreads, 0, stream>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : GDPA_ERR_LAUNCH_;
}

}  // namespace gdpa
