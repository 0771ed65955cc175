// Device-side builder of the longest-first work list walked by the persistent GDPA kernels.
//
// Forward items are (sequence, head, 256-row Q block) weighted by the number of KV tiles of the
// sequence; backward items are (sequence, head, 128-row KV tile) weighted by the number of Q tiles.
// The list is a counting sort by weight, heaviest first, built by one thread block without any
// host synchronisation.  Buffer layout: int32 header {count, mode, 0, 0}, then one int4
// {sequence, head, block, weight} per item ({first sequence, head, first row, row past the last} with kSchedFwdShared,
// where neighbouring Q sequences of one KV sequence are taken together).
#include "gdpa_common.cuh"
#include "gdpa_launch.h"

namespace gdpa {

namespace {

constexpr int kSchedThreads = 1024;
constexpr int kBins = 4096;
constexpr int kSms = 148;  // CTAs of the persistent kernels

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
  if (a.mode != kSchedBwd) {
    nblk = static_cast<int>((lq + kFwdQBlock - 1) / kFwdQBlock);
    weight = nkv;
  } else {
    nblk = nkv;
    weight = nq;
  }
  if (weight > kBins - 1) weight = kBins - 1;
}

// The same for kSchedFwdShared, for the 1024 sequences from b0: sequences that follow one another, read the same KV
// sequence and are not cut by max_q form a run, one long sequence as far as the forward is concerned (their rows are
// neighbours in the packed tensors).  The first sequence of a run gets all its blocks, the others none; runs end at the
// end of a chunk.  (4 requests of 64 candidates of 1 to 32 rows, 4 heads: 1 024 items of one mostly empty Q tile became 140
// full ones, the forward kernel 75 -> 23 us.)  Called by the whole block; `first_head[w]` is the first run head among warp w's sequences.
__device__ __forceinline__ void run_geometry(const SchedArgs& a, int b0, int n, int piece, int* first_head, int& nblk, int& weight,
                                             int& rows) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int b = b0 + t;
  auto kv_of = [&](int i) {
    const int kb = static_cast<int>(load_offset(a.kv_index, i, a.off64));
    return kb < 0 ? 0 : (kb >= a.kv_batch ? a.kv_batch - 1 : kb);
  };
  auto whole = [&](int i) {
    const long long len = load_offset(a.q_off, i + 1, a.off64) - load_offset(a.q_off, i, a.off64);
    return len >= 0 && len <= a.max_q;
  };
  const bool joins = t < n && whole(b);
  const bool head = t < n && (t == 0 || !joins || !whole(b - 1) || kv_of(b) != kv_of(b - 1));
  const unsigned heads = __ballot_sync(0xffffffffu, head);
  if (lane == 0) first_head[warp] = heads != 0u ? warp * 32 + __ffs(heads) - 1 : -1;
  __syncthreads();
  nblk = 0, weight = 0, rows = 0;
  if (head) {
    seq_geometry(a, b, nblk, weight);  // the weight; the blocks follow from the rows of the run
    long long s0, e0;
    seq_bounds(a.q_off, b, a.off64, s0, e0);
    long long len = e0 - s0;
    if (joins) {
      int end = n;  // of the run, within the chunk
      const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
      if (later != 0u) {
        end = t + __ffs(later);
      } else {
        for (int w = warp + 1; w < kSchedThreads / 32; ++w)
          if (first_head[w] >= 0) {
            end = first_head[w];
            break;
          }
      }
      len = load_offset(a.q_off, b0 + end, a.off64) - s0;
    } else {
      len = len < 0 ? 0 : a.max_q;
    }
    rows = static_cast<int>(len);
    nblk = (rows + piece - 1) / piece;
  }
  __syncthreads();  // first_head is written again by the next call
}

// Latency-bound: one block, a few thousand items, and the forward or backward kernel waits for it.  What it costs is the
// chain of dependent steps, so: only the bins that a sequence of the given maximum length can have are cleared and
// scanned (17 of 4096 for 2048 tokens), and the scan gives each thread its own run of neighbouring bins (a warp reads
// consecutive words, no bank conflicts) instead of one warp walking all of them.  With many sequences it is the number of
// instructions: without runs no warp waits for another between two sequences, and a warp writes the items of its sequences
//  - each lane its own sequence's, if none has more than four (100 000 sequences of one head: 168 us);
//  - one sequence after another, 32 items (512 bytes) a store, if they have 64 and more on average;
//  - otherwise 32 items at a time across its sequences (100 000 sequences of 8 heads: 458 us, 642 us with a lane for each
//    sequence, 1216 us with a warp for each).
// Launch and kernel of a build, back to back: 8 sequences 15 -> 10 us; 1152 of up to 100 tokens and 8 heads 21 -> 11 us, of
// up to 2000 tokens 42 -> 21 us (from a warp that walks all bins and a lane for each sequence).
__global__ void __launch_bounds__(kSchedThreads, 1) gdpa_build_schedule_kernel(const SchedArgs a) {
  __shared__ int hist[kBins];
  __shared__ int warp_sum[kSchedThreads / 32];
  __shared__ int4 seq[kSchedThreads + kSchedThreads / 32];  // first slot, blocks, weight, rows of a run; a gap after every 32
  __shared__ int first_head[kSchedThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool shared = a.mode == kSchedFwdShared;
  const int longest = a.mode == kSchedBwd ? a.max_q : a.max_kv;
  const int bins = min(kBins, (longest > 0 ? (longest - 1) / kTile + 1 : 0) + 1);  // weights 0 .. bins - 1
  const long long cap = a.capacity_items;
  for (int i = t; i < bins; i += kSchedThreads) hist[i] = 0;
  __syncthreads();
  // Runs are cut into blocks of two Q tiles when that gives every CTA one, else of one tile: with idle CTAs the longest
  // block is what the call takes, and one tile is done sooner than two.
  int piece = kFwdQBlock;
  if (shared && a.batch > 0 &&
      (load_offset(a.q_off, a.batch, a.off64) - load_offset(a.q_off, 0, a.off64)) / kFwdQBlock * a.heads < kSms)
    piece = kTile;
  // Chunks of up to 1024 sequences, a sequence per thread, dealt out evenly to the warps (runs: in the order of the threads).
  int nblk = 0, w = 0, rows = 0;  // of this thread's sequence of the last chunk: the only one unless the batch is large
  auto geometry = [&](int b0, int n, int each) {
    const int mine = warp * each + lane;
    if (shared) run_geometry(a, b0, n, piece, first_head, nblk, w, rows);
    else if (lane < each && mine < n) seq_geometry(a, b0 + mine, nblk, w);
    else nblk = 0;
  };
  for (int b0 = 0; b0 < a.batch; b0 += kSchedThreads) {
    const int n = min(kSchedThreads, a.batch - b0);
    geometry(b0, n, shared ? 32 : (n + 31) / 32);
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
  auto put = [&](long long slot, int b, int h, int blk, int last) {  // last: the weight, or the rows of a run
    if (slot < cap)
      items[slot] = shared ? make_int4(b, h, blk * piece, min(last, (blk + 1) * piece)) : make_int4(b, h, blk, last);
  };
  // k / blocks: (k + 0.5) / blocks is at least 0.5 / blocks away from a whole number, further than it is rounded for k < 2^21
  auto head_of = [&](int k, int blocks, float inv) {
    return k < (1 << 21) ? static_cast<int>((static_cast<float>(k) + 0.5f) * inv) : k / blocks;
  };
  // The items of a warp's sequences: lane `src` holds sequence first_b + src * step_b, its first slot, blocks, weight and rows.
  auto put_items = [&](const int4& sq, int first_b, int step_b) {
    const int count = sq.y * a.heads, my_last = shared ? sq.w : sq.z;
    if (!__any_sync(0xffffffffu, count > 4)) {
      for (int k = 0, h = 0, blk = 0; k < count; ++k) {
        put(static_cast<long long>(sq.x) + k, first_b + lane * step_b, h, blk, my_last);
        if (++blk == sq.y) blk = 0, ++h;
      }
      return;
    }
    int end = count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, end, d);
      if (lane >= d) end += n;
    }
    const int begin = end - count, all = __shfl_sync(0xffffffffu, end, 31);
    const float my_inv = 1.f / static_cast<float>(sq.y);
    unsigned left = __ballot_sync(0xffffffffu, count > 0);
    if (all >= 64 * __popc(left)) {
      for (; left != 0u; left &= left - 1u) {
        const int src = __ffs(left) - 1;
        const int slot = __shfl_sync(0xffffffffu, sq.x, src), nb = __shfl_sync(0xffffffffu, sq.y, src);
        const int last = __shfl_sync(0xffffffffu, my_last, src), n = __shfl_sync(0xffffffffu, count, src);
        const float inv = __shfl_sync(0xffffffffu, my_inv, src);
        for (int k = lane; k < n; k += 32) {
          const int h = head_of(k, nb, inv);
          put(static_cast<long long>(slot) + k, first_b + src * step_b, h, k - h * nb, last);
        }
      }
      return;
    }
    for (int i0 = 0; i0 < all; i0 += 32) {
      const int i = i0 + lane;
      int src = 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
        if (__shfl_sync(0xffffffffu, end, src + d - 1) <= i) src += d;
      const int k = i - __shfl_sync(0xffffffffu, begin, src), slot = __shfl_sync(0xffffffffu, sq.x, src);
      const int nb = __shfl_sync(0xffffffffu, sq.y, src), last = __shfl_sync(0xffffffffu, my_last, src);
      const int h = head_of(k, nb, __shfl_sync(0xffffffffu, my_inv, src));
      if (i < all) put(static_cast<long long>(slot) + k, first_b + src * step_b, h, k - h * nb, last);
    }
  };
  const bool one_chunk = a.batch <= kSchedThreads;
  for (int b0 = 0; b0 < a.batch; b0 += kSchedThreads) {
    const int n = min(kSchedThreads, a.batch - b0);
    const int each = shared ? 32 : (n + 31) / 32;
    if (!one_chunk) geometry(b0, n, each);
    const int count = nblk * a.heads;
    const int4 sq = make_int4(count > 0 ? atomicAdd(&hist[w], count) : 0, nblk, w, rows);
    if (shared && one_chunk) {  // the few first sequences of runs: dealt out to the warps one by one
      seq[t + warp] = sq;
      __syncthreads();
      put_items(seq[lane * 33 + warp], warp, 32);
    } else {
      put_items(sq, b0 + warp * each, 1);
    }
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
