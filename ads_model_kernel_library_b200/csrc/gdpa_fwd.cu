// GDPA forward for sm_100a:  O = cast(act(Q K^T) * scale) V  over a jagged batch.
//
// One persistent CTA per SM walks a longest-first list of work items (sequence, head, 256-row
// Q block).  A work item keeps two 128-row Q tiles resident in shared memory and streams the
// sequence's K and V tiles through a shared-memory ring.  Roles (20 warps, 96 registers each):
//
//   warps 0-7   activation of Q tile 0: S0 (TMEM) -> registers -> act * scale -> bf16 P0 (TMEM); two
//               warps per TMEM lane quarter, each owning 64 of the 128 S columns.  At the end of a work
//               item the same warps drain their half of O0 (TMEM -> bf16 -> a staging slab in shared memory ->
//               TMA store).
//   warps 8-15  the same for Q tile 1
//   warp  16    MMA issuer (one elected thread): S_s = Q_s K^T (tcgen05.mma, operands in shared memory),
//               O_s += P_s V (A operand P read from TMEM)
//   warp  17    TMA loader (lane 0 issues the copies, the warp zeroes the tails of ragged tiles);  warps 18-19 idle
//
// TMEM (512 columns): S0 [0,128)  S1 [128,256)  O0 [256,256+D)  O1 [384,384+D).  P_s (bf16, two
// values per column) of column half h overwrites the first 32 columns of that half's own S columns.
// While the warps of one Q tile run their activation the tensor cores run the other tile's P V and
// next Q K^T, so activation and MMA overlap.
//
// Variants of the same kernel: softmax with online rescaling (the two column halves exchange their row
// maxima through shared memory, keep partial row sums and write the log-sum-exp for the backward), and
// FP8 e4m3 operands with per-128-token-block scales.
//
// Tiles reach their consumers zero-padded (the loader zeroes the tail of a ragged tile in shared memory): rows of a
// tile beyond the end of its sequence are zeros, not the next sequence's tokens, as with the reference's per-sequence block loads
// (gdpa/triton/triton_generalized_dot_product_attention.py:270, :317).  So S columns beyond the KV length are
// exactly 0 and act(0) = 0 for every supported element-wise activation: no masking, and nothing a neighbouring
// sequence holds (Inf and NaN included) reaches this one.  Only the softmax (where a padded column must not count)
// and the band (window_size) test columns.  Q rows beyond the Q length are computed and never stored.
#include "gdpa_common.cuh"
#include "gdpa_launch.h"

namespace gdpa {

namespace {

// 20 warps: warps 0-7 / 8-15 activation of Q tile 0 / 1 (two warps per TMEM lane quarter, each owning 64
// of the 128 S columns; they also drain their half of O at the end of a work item), 16 MMA, 17 TMA,
// 18-19 idle.  A single warp cannot overlap its MUFU instructions with its FMA-pipe instructions, so two
// activation warps per SM sub-partition and Q tile halve the activation time.
constexpr int kFwdThreads = 20 * 32;
constexpr int kKvStages = 4;
constexpr int kWorkSlots = 4;

// Barrier indices inside the shared barrier array.
enum FwdBar : int {
  B_Q_FULL = 0,                        // [2] TMA -> MMA
  B_Q_EMPTY = 2,                       // [2] MMA commit -> TMA
  B_KV_FULL = 4,                       // [kKvStages]
  B_KV_EMPTY = 4 + kKvStages,          // [kKvStages]
  B_S_FULL = 4 + 2 * kKvStages,        // [2] MMA commit -> activation group
  B_P_FULL = 6 + 2 * kKvStages,        // [2] activation group (256 arrivals) -> MMA
  B_O_FULL = 8 + 2 * kKvStages,        // [2] MMA commit -> epilogue
  B_O_EMPTY = 10 + 2 * kKvStages,      // [2] epilogue (256 arrivals) -> MMA
  B_L_FULL = 12 + 2 * kKvStages,       // [2] softmax: activation group -> epilogue (row sums)
  B_M_FULL = 14 + 2 * kKvStages,       // [2] softmax, wide layout: both column halves have published their row maxima
  B_LD_TMP = 16 + 2 * kKvStages,       // [4] the loader's own: a ragged tile has landed and can have its padding rows zeroed
  B_WORK_FULL = 20 + 2 * kKvStages,               // [kWorkSlots] the loader has published a work item
  B_WORK_EMPTY = 20 + 2 * kKvStages + kWorkSlots, // [kWorkSlots] the MMA warp and the 16 activation warps have read it
  B_COUNT = 20 + 2 * kKvStages + 2 * kWorkSlots
};

template <int D, int EB>
struct FwdSmem {
  static constexpr int kTileBytes = kTile * D * EB;      // one 128 x D tile of EB-byte elements
  static constexpr int kHalfBytes = kTile * 128;         // one swizzled box: 128 rows x 128 bytes
  static constexpr int kBoxes = D * EB / 128;            // boxes per tile
  static constexpr int kBoxCols = 128 / EB;              // elements per box row
  static constexpr int kQOff = 0;
  static constexpr int kKvOff = 2 * kTileBytes;
  static constexpr int kRowSumOff = kKvOff + kKvStages * kTileBytes;  // softmax: float[2 Q tiles][2 halves][128]
  static constexpr int kRowMaxOff = kRowSumOff + 4 * kTile * 4;       // softmax, wide: float[2 parity][2][2][128]
  // Output staging: one slab of 32 rows x 32 bf16 per activation warp, 64-byte swizzled, from which that warp's O
  // rows leave by TMA store.  Where shared memory has room the slabs follow the softmax arrays (kSeparate); with
  // 32 KB bf16 tiles (head_dim 128) it has not, the slabs lie over those arrays, and the softmax kernels of that
  // shape store O from registers instead.
  static constexpr int kOutSlabBytes = 32 * 64;
  static constexpr int kStatBytes = 12 * kTile * 4;
  static constexpr bool kSeparate = kRowSumOff + kStatBytes + 16 * kOutSlabBytes + 2048 <= 227 * 1024;
  static constexpr int kOutOff = kSeparate ? kRowSumOff + kStatBytes : kRowSumOff;
  // ... and there the softmax kernel has narrow slabs of its own behind its arrays: 32 rows x 16 bf16 (32-byte swizzle)
  static constexpr int kNarrowSlabBytes = 32 * 32;
  static constexpr int kNarrowOff = kRowSumOff + kStatBytes;
  static_assert(kStatBytes + 16 * kNarrowSlabBytes <= 16 * kOutSlabBytes, "the narrow slabs fit in the staging region");
  static constexpr int kBarOff = kOutOff + 16 * kOutSlabBytes;
  static_assert(16 * kOutSlabBytes >= kStatBytes, "the softmax arrays fit in the staging region");
  static constexpr int kWorkOff = (kBarOff + B_COUNT * 8 + 15) / 16 * 16;  // WorkSlot[kWorkSlots]: the work items in flight
  static constexpr int kTmemPtrOff = kWorkOff + kWorkSlots * 48;
  static constexpr int kAbortOff = kTmemPtrOff + 4;
  static constexpr int kBytes = kAbortOff + 4;
  static constexpr int kDynBytes = kBytes + 1024;        // slack to align the base to 1024 bytes
};

// Every role waits as a whole warp: the decision to leave is the warp's, so no lane runs ahead into a collective instruction
// (tcgen05.ld / st, the vote for the thread that issues the MMAs).
#define GDPA_WAIT_WARP(bar_idx, parity, role)                                                                       \
  {                                                                                                                 \
    const bool ok_ = mbar_wait(bar_base + 8u * (bar_idx), (parity), abort_flag, a.status, ((bar_idx) << 8) | (role)); \
    if (!__all_sync(0xffffffffu, ok_)) goto role_done;                                                              \
  }

// Sum of squares of eight bf16 values packed in a uint4.
__device__ __forceinline__ float sumsq_bf16x8(const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xffff0000u);
    s = fmaf(lo, lo, fmaf(hi, hi, s));
  }
  return s;
}

// FUSE = the epilogue of the norm pipeline (residual add, row sums of squares) compiled in: a template parameter
// rather than a run-time branch, so that the plain forward carries none of it.
template <int D, int ACT, bool FP8, bool FUSE>
__global__ void __launch_bounds__(kFwdThreads, 1)
gdpa_fwd_kernel(const __grid_constant__ TmapSet tm_q, const __grid_constant__ TmapSet tm_k,
                const __grid_constant__ TmapSet tm_v, const __grid_constant__ OutTmap tm_o, const FwdArgs a) {
  constexpr int EB = FP8 ? 1 : 2;
  constexpr bool kSoftmax = (ACT == ACT_SOFTMAX);
  // O leaves through shared memory and TMA stores (whole 64-byte row pieces per transaction); the bf16 softmax
  // kernel at head_dim 128 (its row statistics hold that shared memory) has narrower slabs of its own (32-byte row
  // pieces); the norm-pipeline epilogue has its own path through the wide slabs
  constexpr bool kNarrowOut = !FUSE && kSoftmax && !FwdSmem<D, FP8 ? 1 : 2>::kSeparate;
  constexpr bool kTmaOut = !FUSE && !kNarrowOut;
  constexpr int kActWarps = 16;
  constexpr int kMmaWarp = 16;
  constexpr int kLoadWarp = 17;
  constexpr uint32_t kStageThreads = 256u;  // threads that work on one Q tile's S / O
  using L = FwdSmem<D, EB>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_base + L::kBarOff;
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(smem + L::kTmemPtrOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kAbortOff);

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      const bool by_threads = (i >= B_P_FULL && i < B_P_FULL + 2) || (i >= B_O_EMPTY && i < B_O_EMPTY + 2) ||
                            (i >= B_L_FULL && i < B_L_FULL + 2) || (i >= B_M_FULL && i < B_M_FULL + 2);
      const bool by_readers = i >= B_WORK_EMPTY && i < B_WORK_EMPTY + kWorkSlots;
      mbar_init(bar_base + 8u * i, by_threads ? kStageThreads : by_readers ? 1u + kActWarps : 1u);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_base + L::kTmemPtrOff, 512);
    tmem_relinquish();
  }
  if (warp == kLoadWarp && lane == 0) {
    tma_prefetch_desc(&tm_q.m[0]);
    tma_prefetch_desc(&tm_k.m[0]);
    tma_prefetch_desc(&tm_v.m[0]);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_ptr);
  const SeqLimits lim = {a.total_q, a.total_kv, a.kv_batch};

  // The loader warp walks the list, reads an item and its sequence's offsets (two dependent trips to memory, with FP8
  // a third for the rows of the block scales) and publishes what they say through a small ring in shared memory, an item
  // ahead of its use; the MMA warp and the activation warps start on an item with two or three shared-memory loads
  // instead of making those trips each.  FP8 forward 4.96 -> 4.83 ms, the norm pipeline's step unchanged within its spread.
  // Slot: {head, row offset q0 of the Q block, first Q row, first KV row}, {lq, lkv, first KV tile, KV tiles}, {Q scale row of Q tile 0, KV
  // scale row of KV tile 0 (FP8), -, -}; head -1 ends the walk.
  int4* const work_ring = reinterpret_cast<int4*>(smem + L::kWorkOff);
  uint32_t work_pos = 0;  // items this role has taken: ring slot = work_pos % kWorkSlots, parity = (work_pos / kWorkSlots) & 1
  struct Item {
    int h, q0, q_start, kv_start, lq, lkv, j0, nkv, q_scale0, kv_scale0;  // the block takes rows [q0, min(lq, q0 + 256))
  };
  // Consumer side: this role's next work item; h = -1 at the end of the list, -2 if the wait ran out.
  // Called by a whole warp, whose lane 0 releases the slot.
  auto take_work_item = [&](int role) -> Item {
    const uint32_t slot = work_pos % kWorkSlots, parity = (work_pos / kWorkSlots) & 1u;
    ++work_pos;
    bool ok = mbar_wait(bar_base + 8u * (B_WORK_FULL + slot), parity, abort_flag, a.status, ((B_WORK_FULL + slot) << 8) | role);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) return Item{-2, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int4 u = work_ring[3 * slot], v = work_ring[3 * slot + 1];
    int4 x = make_int4(0, 0, 0, 0);
    if (FP8) x = work_ring[3 * slot + 2];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_base + 8u * (B_WORK_EMPTY + slot));
    return Item{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w, x.x, x.y};
  };

  // Operand format code: 1 = bf16 for kind::f16, 0 = e4m3 for kind::f8f6f4.
  constexpr uint32_t kFmt = FP8 ? 0u : 1u;
  // QK: A = Q tile (K-major), B = K tile (K-major), M = 128, N = 128.
  constexpr uint32_t kIdescQK = umma_idesc(kFmt, kFmt, 0, 0, kTile, kTile);
  // PV: A = P in TMEM, B = V tile (MN-major: head dim contiguous), M = 128, N = D.
  constexpr uint32_t kIdescPV = umma_idesc(kFmt, kFmt, 0, 1, kTile, D);

  if (warp >= kMmaWarp) {
   if (warp == kLoadWarp) {
    // ------------------------------------------------------------------ TMA loader
    // The whole warp walks the items; lane 0 issues the copies.  A full tile goes straight to its consumers' barrier.
    // A ragged tile (the last of its sequence) is fetched as the same full boxes onto the loader's own barrier -- its
    // rows past the sequence end are the next sequence's, or, past the tensor's end, the TMA unit's zero fill -- then
    // the warp overwrites those rows with zeros in shared memory and only then releases the tile: the consumers see a
    // zero-padded tile and nothing of the neighbour reaches them.
    {
      uint32_t kv_pos = 0;  // K / V tiles of the items before this one; tile number p sits in ring slot p % kKvStages
      uint32_t q_phase = 0, tmp_phase = 0;  // bit s = parity of Q stage s, of B_LD_TMP + s
      [[maybe_unused]] int ltr = 0;  // KV tiles before this item (trace rows)
      // asks for one tile = L::kBoxes boxes of 128 rows x 128 bytes; a ragged one (valid < 128) on B_LD_TMP + tmp
      auto load_tile = [&](uint32_t dst_off, const CUtensorMap* tm, int full_bar, int tmp, int y, int row0, int valid) {
        if (lane == 0) {
          const uint32_t bar = bar_base + 8u * (valid < kTile ? B_LD_TMP + tmp : full_bar);
          mbar_arrive_expect_tx(bar, L::kTileBytes);
#pragma unroll
          for (int hf = 0; hf < L::kBoxes; ++hf)
            tma_load_3d(smem_base + dst_off + hf * L::kHalfBytes, tm, bar, hf * L::kBoxCols, y, row0);
        }
      };
      // a ragged tile: once it has landed, zero its rows >= valid and release it on its consumers' barrier
      auto release = [&](uint32_t dst_off, int full_bar, int tmp, int valid) -> bool {
        if (valid >= kTile) return true;
        const bool ok = mbar_wait(bar_base + 8u * (B_LD_TMP + tmp), (tmp_phase >> tmp) & 1u, abort_flag, a.status,
                                  ((B_LD_TMP + tmp) << 8) | ST_ROLE_LOAD);
        if (!__all_sync(0xffffffffu, ok)) return false;
        tmp_phase ^= 1u << tmp;
        for (int bx = 0; bx < L::kBoxes; ++bx)
          for (int off = max(valid, 0) * 128 + lane * 16; off < L::kHalfBytes; off += 512)
            *reinterpret_cast<uint4*>(smem + dst_off + bx * L::kHalfBytes + off) = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_base + 8u * full_bar);
        return true;
      };
      // runs of sequences have no block scales of their own (FP8), no positions in a sequence (a window), and need the
      // KV sequence's index
      const bool shared_runs = !FP8 && a.sched[1] == kSchedFwdShared && a.window < 0 && a.kv_index != nullptr;
      WorkWalker walker(schedule_items(a.sched, shared_runs || a.sched[1] == kSchedFwd, a.status));
      // producer side of the work ring: the slot must have been read by every consumer of its previous use
      auto next_item = [&](Item& it) -> bool {
        const uint32_t slot = work_pos % kWorkSlots, parity = (work_pos / kWorkSlots) & 1u;
        it = Item{-1, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        int i;
        if (walker.next(i)) {
          Work w = load_work(a.sched, i, a.q_off, a.kv_off, a.off64, a.max_q, a.max_kv, lim, a.kv_index);
          it.h = w.h;
          it.q_start = static_cast<int>(w.q_start), it.kv_start = static_cast<int>(w.kv_start);
          if (shared_runs) {
            // rows of a run of sequences instead of a block of one, still clamped to the tensor
            const int4 run = reinterpret_cast<const int4*>(a.sched + kSchedHeaderInts)[i];
            w.blk = 0;
            w.lq = static_cast<int>(min(static_cast<long long>(run.w), a.total_q - w.q_start));
            it.q0 = run.z;
          }
          it.q0 += w.blk * kFwdQBlock;
          it.lq = w.lq, it.lkv = w.lkv;
          fwd_kv_range(w, a.window, it.j0, it.nkv);
          if constexpr (FP8) {
            it.q_scale0 = static_cast<int>(load_offset(a.q_blk_off, w.b, a.off64)) + w.blk * 2;
            it.kv_scale0 = static_cast<int>(load_offset(a.kv_blk_off, w.kb, a.off64));
          }
        }
        const bool ok = mbar_wait(bar_base + 8u * (B_WORK_EMPTY + slot), parity ^ 1u, abort_flag, a.status,
                                  ((B_WORK_EMPTY + slot) << 8) | ST_ROLE_LOAD);
        if (!__all_sync(0xffffffffu, ok)) return false;
        if (lane == 0) {
          work_ring[3 * slot] = make_int4(it.h, it.q0, it.q_start, it.kv_start);
          work_ring[3 * slot + 1] = make_int4(it.lq, it.lkv, it.j0, it.nkv);
          if (FP8) work_ring[3 * slot + 2] = make_int4(it.q_scale0, it.kv_scale0, 0, 0);
          mbar_arrive(bar_base + 8u * (B_WORK_FULL + slot));
        }
        ++work_pos;
        return true;
      };
      Item w, w_next;
      if (!next_item(w)) goto role_done;
      for (; w.h >= 0; w = w_next) {
        if (!next_item(w_next)) goto role_done;
        const int j0 = w.j0, nkv = w.nkv;  // first KV tile and number of KV tiles this item visits
        if (nkv == 0) continue;
        const int q0 = w.q0;
        const int nst = (w.lq - q0 > kTile) ? 2 : 1;
        const int q_row = w.q_start + q0;
        const int kv_row = w.kv_start + j0 * kTile;
        // Issue order Q0, K0, Q1, V0, K1, V1, ...  In an item of one or two KV tiles (all its tiles fit in the ring) none of
        // the copies of a group (the first four, then K1 and V1) waits for another to land: ragged tiles are zeroed and
        // released when the whole group has been asked for.  There the round trips to memory are what the item takes
        // (lengths up to 256: the forward kernel 204 -> 162 us); with more KV tiles the loader is
        // ahead of the MMAs, and a ragged K that waits for the ring slot of its V would come later than it could (log-normal
        // forward 1.215 -> 1.232 ms with groups everywhere).  The softmax kernels' items are bound by their element-wise
        // work: FP8 4.82 -> 4.86 ms with groups, so they have none.
        const bool group = !kSoftmax && nkv <= 2;
        const int head_kv = w.h / a.kv_group;
        const int q_valid0 = w.lq - q0, q_valid1 = w.lq - q0 - kTile;
        for (int j = 0; j < nkv; ++j) {
          const int kv_valid = w.lkv - (j0 + j) * kTile;
          const uint32_t k_stage = kv_pos % kKvStages, v_stage = (kv_pos + 1) % kKvStages;
          const uint32_t k_off = L::kKvOff + k_stage * L::kTileBytes, v_off = L::kKvOff + v_stage * L::kTileBytes;
          if (j == 0) {
            if (lane == 0) GDPA_TRACE(a, ltr * 32 + 24);
            GDPA_WAIT_WARP(B_Q_EMPTY, (q_phase & 1u) ^ 1u, ST_ROLE_LOAD);
            q_phase ^= 1u;
            load_tile(L::kQOff, &tm_q.m[0], B_Q_FULL, 0, w.h, q_row, q_valid0);
            if (!group && !release(L::kQOff, B_Q_FULL, 0, q_valid0)) goto role_done;
          }
          GDPA_WAIT_WARP(B_KV_EMPTY + k_stage, ((kv_pos / kKvStages) & 1u) ^ 1u, ST_ROLE_LOAD);
          load_tile(k_off, &tm_k.m[0], B_KV_FULL + k_stage, 2, head_kv, kv_row + j * kTile, kv_valid);
          if (!group && !release(k_off, B_KV_FULL + k_stage, 2, kv_valid)) goto role_done;
          if (j == 0 && nst == 2) {
            GDPA_WAIT_WARP(B_Q_EMPTY + 1, ((q_phase >> 1) & 1u) ^ 1u, ST_ROLE_LOAD);
            q_phase ^= 2u;
            load_tile(L::kQOff + L::kTileBytes, &tm_q.m[0], B_Q_FULL + 1, 1, w.h, q_row + kTile, q_valid1);
            if (!group && !release(L::kQOff + L::kTileBytes, B_Q_FULL + 1, 1, q_valid1)) goto role_done;
          }
          GDPA_WAIT_WARP(B_KV_EMPTY + v_stage, (((kv_pos + 1) / kKvStages) & 1u) ^ 1u, ST_ROLE_LOAD);
          load_tile(v_off, &tm_v.m[0], B_KV_FULL + v_stage, 3, head_kv, kv_row + j * kTile, kv_valid);
          if (group) {
            if (j == 0 && !release(L::kQOff, B_Q_FULL, 0, q_valid0)) goto role_done;
            if (!release(k_off, B_KV_FULL + k_stage, 2, kv_valid)) goto role_done;
            if (j == 0 && nst == 2 && !release(L::kQOff + L::kTileBytes, B_Q_FULL + 1, 1, q_valid1)) goto role_done;
          }
          if (!release(v_off, B_KV_FULL + v_stage, 3, kv_valid)) goto role_done;
          kv_pos += 2;
        }
        ltr += nkv;
      }
    }
   } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer
    // The tensor pipe's queue is short, so how fast this warp issues is how fast it runs.  The whole warp walks the loop,
    // with bounds and stages that are the same for its lanes, and one elected thread issues: operands stay in uniform
    // registers.  As one lane's code under a branch: log-normal forward 1002 -> 966 us, FP8 3.79 -> 3.66 ms, head_dim 64 with a
    // band 430 -> 380 us, 14.0 -> 13.0 ms on 512 sequences of 512 to 4096 tokens of 8 heads.  (In that form a rolled loop of
    // the slices cost 19 %.  Two issuing warps, one for each Q tile, cost 25 %: the Q tiles fall into step, both in the
    // activation and then both on the tensor pipe, where one warp keeps them alternating.)
    {
      uint32_t kv_stage = 0, kv_phase = 0;
      // bit s of q_phase / p_phase / o_phase = parity of that barrier of Q tile s (registers, not arrays indexed by s)
      uint32_t q_phase = 0, p_phase = 0, o_phase = 0;
      int tr = 0;
      // Descriptors of stage 0 / ring slot 0, built once; per MMA only the low word moves.
      const uint64_t dq0 = umma_smem_desc_sw128(smem_base + L::kQOff, 16, 1024);
      const uint64_t dk0 = umma_smem_desc_sw128(smem_base + L::kKvOff, 16, 1024);
      const uint64_t dv0 = umma_smem_desc_sw128(smem_base + L::kKvOff, L::kHalfBytes, 1024);
      auto issue_qk = [&](int s, uint32_t k_stage) {
        const uint64_t da = umma_desc_advance(dq0, s * L::kTileBytes);
        const uint64_t db = umma_desc_advance(dk0, k_stage * L::kTileBytes);
        const uint32_t d_tmem = tmem_base + s * kTile;
        // one K slice = 32 bytes of the head dim (16 bf16 or 32 e4m3), four slices per 128-byte box
#pragma unroll
        for (int kk = 0; kk < D * EB / 32; ++kk) {
          const uint32_t off = (kk >> 2) * L::kHalfBytes + (kk & 3) * 32;
          if constexpr (FP8) umma_ss_f8(d_tmem, umma_desc_advance(da, off), umma_desc_advance(db, off), kIdescQK, kk > 0 ? 1u : 0u);
          else umma_ss_f16(d_tmem, umma_desc_advance(da, off), umma_desc_advance(db, off), kIdescQK, kk > 0 ? 1u : 0u);
        }
      };
      auto issue_pv = [&](int s, uint32_t v_stage, bool accumulate) {
        const uint64_t db = umma_desc_advance(dv0, v_stage * L::kTileBytes);
        const uint32_t d_tmem = tmem_base + 256 + s * kTile, a_tmem = tmem_base + s * kTile;
        // one K slice = 16 (bf16) or 32 (e4m3) KV rows of 128 bytes; P holds it in 8 TMEM columns
        constexpr int kRowsPerSlice = 32 / EB;
#pragma unroll
        for (int kk = 0; kk < kTile / kRowsPerSlice; ++kk) {
          const uint32_t acc = (accumulate || kk > 0) ? 1u : 0u;
          // the P slices of column half h sit at the start of that half's own S columns
          const uint32_t a_col = FP8 ? (kk >> 1) * 64 + (kk & 1) * 8 : (kk >> 2) * 64 + (kk & 3) * 8;
          if constexpr (FP8) umma_ts_f8(d_tmem, a_tmem + a_col, umma_desc_advance(db, kk * kRowsPerSlice * 128), kIdescPV, acc);
          else umma_ts_f16(d_tmem, a_tmem + a_col, umma_desc_advance(db, kk * kRowsPerSlice * 128), kIdescPV, acc);
        }
      };
      while (true) {
        Item w = take_work_item(ST_ROLE_MMA);
        w.h = warp_uniform(w.h), w.nkv = warp_uniform(w.nkv), w.lq = warp_uniform(w.lq), w.q0 = warp_uniform(w.q0);
        if (w.h < 0) {
          if (w.h == -2) goto role_done;
          break;
        }
        const int nkv = w.nkv;
        if (nkv == 0) continue;
        const int nst = (w.lq - w.q0 > kTile) ? 2 : 1;
        // First S tiles: S_s = Q_s K_0^T.
        {
          const uint32_t k_stage = kv_stage;
          for (int s = 0; s < nst; ++s) {
            GDPA_WAIT_WARP(B_Q_FULL + s, (q_phase >> s) & 1u, ST_ROLE_MMA);
            q_phase ^= 1u << s;
            if (s == 0) GDPA_WAIT_WARP(B_KV_FULL + k_stage, kv_phase, ST_ROLE_MMA);
            tc_fence_after();
            issue_qk(s, k_stage);
            tc_commit(bar_base + 8u * (B_S_FULL + s));
            if (nkv == 1) tc_commit(bar_base + 8u * (B_Q_EMPTY + s));
          }
          tc_commit(bar_base + 8u * (B_KV_EMPTY + k_stage));
          if (++kv_stage == kKvStages) { kv_stage = 0; kv_phase ^= 1u; }
        }
        for (int j = 0; j < nkv; ++j) {
          const bool more = (j + 1 < nkv);
          const uint32_t v_stage = kv_stage, v_phase = kv_phase;
          if (++kv_stage == kKvStages) { kv_stage = 0; kv_phase ^= 1u; }
          const uint32_t k_stage = kv_stage, k_phase = kv_phase;  // K_{j+1}, valid if more
          if (more) { if (++kv_stage == kKvStages) { kv_stage = 0; kv_phase ^= 1u; } }
          GDPA_WAIT_WARP(B_KV_FULL + v_stage, v_phase, ST_ROLE_MMA);
          for (int s = 0; s < nst; ++s) {
            GDPA_TRACE(a, tr * 32 + 16 + s * 4 + 0);
            GDPA_WAIT_WARP(B_P_FULL + s, (p_phase >> s) & 1u, ST_ROLE_MMA);
            GDPA_TRACE(a, tr * 32 + 16 + s * 4 + 1);
            p_phase ^= 1u << s;
            if (j == 0) {
              GDPA_WAIT_WARP(B_O_EMPTY + s, ((o_phase >> s) & 1u) ^ 1u, ST_ROLE_MMA);
              o_phase ^= 1u << s;
            }
            tc_fence_after();
            issue_pv(s, v_stage, j > 0);
            if (more) {
              if (s == 0) {
                GDPA_WAIT_WARP(B_KV_FULL + k_stage, k_phase, ST_ROLE_MMA);
                tc_fence_after();
              }
              issue_qk(s, k_stage);
              tc_commit(bar_base + 8u * (B_S_FULL + s));
              if (j + 2 == nkv) tc_commit(bar_base + 8u * (B_Q_EMPTY + s));
            } else {
              tc_commit(bar_base + 8u * (B_O_FULL + s));
            }
            GDPA_TRACE(a, tr * 32 + 16 + s * 4 + 2);
          }
          ++tr;
          tc_commit(bar_base + 8u * (B_KV_EMPTY + v_stage));
          if (more) tc_commit(bar_base + 8u * (B_KV_EMPTY + k_stage));
        }
      }
    }
   }
  } else if (warp < kActWarps) {
    // ------------------------------------------------------------------ activation + epilogue
    const int s = warp >> 3;           // Q tile
    const int half = (warp >> 2) & 1;  // which 64 of the 128 S columns
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_tmem = tmem_base + lane_base + s * kTile + half * 64;
    const uint32_t o_tmem = tmem_base + lane_base + 256 + s * kTile + half * (D / 2);
    const float scale = a.scale, hscale = 0.5f * a.scale;
    uint32_t s_phase = 0, o_phase = 0;
    int tr = 0;
    while (true) {
      const Item w = take_work_item(ST_ROLE_ACT);
      if (w.h < 0) {
        if (w.h == -2) goto role_done;
        break;
      }
      const int j0 = w.j0, nkv = w.nkv;
      const int q0 = w.q0;
      const int nst = (w.lq - q0 > kTile) ? 2 : 1;
      if (s >= nst) continue;
      const int qr = q0 + s * kTile + row;
      const bool row_valid = qr < w.lq;
      const long long o_elem = (static_cast<long long>(w.q_start + qr) * a.heads + w.h) * D + half * (D / 2);
      uint4* dst = reinterpret_cast<uint4*>(a.o + o_elem);
      // fused epilogue of the norm pipeline: x = O + residual, and the sum of x^2 over this thread's half row is
      // added to the row's entry of row_sumsq (the RMS norm over all heads is finished by a second kernel)
      const uint4* res = (FUSE && a.residual != nullptr) ? reinterpret_cast<const uint4*>(a.residual + o_elem) : nullptr;
      float* const row_sumsq = FUSE ? a.row_sumsq : nullptr;
      float ssq = 0.f;
      if (nkv == 0) {
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < D / 16; ++i) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (res != nullptr) {
              v = res[i];
              ssq += sumsq_bf16x8(v);
            }
            dst[i] = v;
          }
          if (row_sumsq != nullptr) atomicAdd(row_sumsq + w.q_start + qr, ssq);
        }
        continue;
      }
      float inv_l = 1.f;
      if constexpr (kSoftmax) {
        // ---- softmax, one row split over two warps (64 columns each): the halves publish their partial
        // row maxima through shared memory and an mbarrier, take the common maximum, and keep partial row
        // sums that the epilogue adds.  P = exp2(c S + bias - m); the O accumulator is rescaled only when
        // the running maximum m grew by more than kThr.  FP8: c carries the Q- and K-block scales and
        // bias = log2(V-block scale), so P contains the V scale and uses the whole e4m3 range; the row
        // sum divides it out again.
        constexpr float kThr = FP8 ? 1.f : 8.f;
        constexpr float kPScale = FP8 ? 128.f : 1.f;
        constexpr float kLog2e = 1.4426950408889634f;
        float* rowmax = reinterpret_cast<float*>(smem + L::kRowMaxOff);
        float* rowsum = reinterpret_cast<float*>(smem + L::kRowSumOff);
        float m_used = -INFINITY, row_sum = 0.f;
        float sq = 1.f, sk_next = 1.f, sv_next = 1.f;
        const float *k_scale = nullptr, *v_scale = nullptr;
        if constexpr (FP8) {
          sq = a.q_scales[static_cast<long long>(w.q_scale0 + s) * a.heads + w.h];
          if (nkv > 0) {  // the row of an empty KV sequence at the end of the batch is past the end of the scales
            const long long at = static_cast<long long>(w.kv_scale0 + j0) * a.kv_heads + w.h / a.kv_group;
            k_scale = a.k_scales + at, v_scale = a.v_scales + at;
            sk_next = *k_scale, sv_next = *v_scale;
          }
        }
        for (int j = 0; j < nkv; ++j) {
          // columns [clo, chi) of this warp's 64 take part: inside the KV length and inside the band
          const int kbase = (j0 + j) * kTile + half * 64;
          int clo = 0, chi = min(kTile, w.lkv - (j0 + j) * kTile) - half * 64;
          if (a.window >= 0) {
            clo = max(clo, qr - a.window - kbase);
            chi = min(chi, qr + a.window - kbase + 1);
          }
          float c = a.scale * kLog2e, bias = 0.f, inv_sv = 1.f;
          if constexpr (FP8) {
            // this tile's scales were asked for a tile ago
            c *= sq * sk_next;
            bias = log2f(sv_next);
            inv_sv = 1.f / sv_next;
            if (j + 1 < nkv) {
              k_scale += a.kv_heads, v_scale += a.kv_heads;
              sk_next = *k_scale, sv_next = *v_scale;
            }
          }
          GDPA_WAIT_WARP(B_S_FULL + s, s_phase, ST_ROLE_ACT);
          tc_fence_after();
          uint32_t ra[32], rb[32];
          // pass 1: partial row maximum of c * S over this warp's valid columns (chunk 1 in flight
          // while chunk 0 is scanned)
          float pmax = -INFINITY;
          tmem_ld32(s_tmem, ra);
#pragma unroll
          for (int ch = 0; ch < 2; ++ch) {
            uint32_t(&cur)[32] = ch ? rb : ra;
            tmem_wait_ld();
            tmem_regs_ready(cur);
            if (ch == 0) tmem_ld32(s_tmem + 32, rb);
            // a chunk wholly inside [clo, chi) for every row of the warp needs no predicates; without a band
            // the lower bound is 0
            // (c >= 0: the largest c * S is c times the largest S, one three-way maximum per two columns; with the
            // packed arithmetic of pass 2 about 190 instead of 350 issue slots per warp and tile: bf16 training step
            // 1.96 -> 1.94 ms)
            if (c >= 0.f && __all_sync(0xffffffffu, clo <= ch * 32 && chi >= (ch + 1) * 32)) {
              float m0 = __uint_as_float(cur[0]), m1 = __uint_as_float(cur[1]);
#pragma unroll
              for (int i = 2; i < 32; i += 4) {
                m0 = max3(m0, __uint_as_float(cur[i]), __uint_as_float(cur[i + 1]));
                if (i + 2 < 32) m1 = max3(m1, __uint_as_float(cur[i + 2]), __uint_as_float(cur[i + 3]));
              }
              pmax = fmaxf(pmax, fmaxf(m0, m1) * c);
            } else if (a.window < 0) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float t = __uint_as_float(cur[i]) * c;
                pmax = (ch * 32 + i < chi) ? fmaxf(pmax, t) : pmax;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float t = __uint_as_float(cur[i]) * c;
                pmax = (ch * 32 + i >= clo && ch * 32 + i < chi) ? fmaxf(pmax, t) : pmax;
              }
            }
          }
          float* slot = rowmax + (((s_phase * 2 + s) * 2) * kTile);
          slot[half * kTile + row] = pmax;
          mbar_arrive(bar_base + 8u * (B_M_FULL + s));
          GDPA_WAIT_WARP(B_M_FULL + s, s_phase, ST_ROLE_ACT);
          const float rmax = fmaxf(pmax, reinterpret_cast<volatile float*>(slot)[(half ^ 1) * kTile + row]);
          s_phase ^= 1u;
          const float m_new = fmaxf(m_used, rmax + bias);
          if (j == 0) {
            m_used = m_new;
          } else if (__any_sync(0xffffffffu, m_new > m_used + kThr)) {
            // The rows of a warp move their maxima together.  In a run of sequences each row moves its own, so that no row's
            // rounding depends on another sequence.  A row that has not seen a key yet (both maxima -inf) keeps its zeros.
            const bool stays = !FP8 && m_new <= m_used + kThr && a.sched[1] == kSchedFwdShared;
            const float alpha = (m_new == -INFINITY || stays) ? 1.f : ex2_approx(m_used - m_new);
            row_sum *= alpha;
            if (!stays) m_used = m_new;
#pragma unroll
            for (int ch = 0; ch < D / 64; ++ch) {
              uint32_t ro[32];
              tmem_ld32(o_tmem + ch * 32, ro);
              tmem_wait_ld();
              tmem_regs_ready(ro);
#pragma unroll
              for (int i = 0; i < 32; ++i) ro[i] = __float_as_uint(__uint_as_float(ro[i]) * alpha);
              tmem_st32(o_tmem + ch * 32, ro);
            }
          }
          // pass 2: reload the scores, P = exp2(c S + bias - m), partial row sum, quantise, store over
          // columns of this half that have been read
          // (FP8: P is stored times 2^7, a multiplication after the exponential.  As a term of the exponent the factor
          // moves the place where the argument is rounded, and a P beside a midpoint of e4m3 falls to the other side, 6 to
          // 12 % of its value.  The sums of P are taken column after column, so that they do not depend on the packing
          // either.  FP8 forward 4.80 -> 4.97 ms.)
          const float off = (m_used == -INFINITY) ? 0.f : bias - m_used;  // a row may have seen no column yet
          const uint64_t c2 = pack_f32x2(c, c), off2 = pack_f32x2(off, off);
          float psum = 0.f;                     // partial row sum
          [[maybe_unused]] uint64_t psum2 = 0;  // bf16: those of the even and the odd columns
          tmem_ld32(s_tmem, ra);
#pragma unroll
          for (int ch = 0; ch < 2; ++ch) {
            uint32_t(&cur)[32] = ch ? rb : ra;
            tmem_wait_ld();
            tmem_regs_ready(cur);
            if (ch == 0) tmem_ld32(s_tmem + 32, rb);
            // P of this chunk with the column test `inside`; three instantiations so that the common case (the
            // chunk wholly inside [clo, chi) for every row of the warp) carries no predicates at all
            auto emit = [&](auto inside) {
              auto prob2 = [&](int i, float& p0, float& p1) {  // columns 2i and 2i + 1 of the chunk
                float e0, e1;
                unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(cur[2 * i]), __uint_as_float(cur[2 * i + 1])), c2, off2), e0, e1);
                e0 = ex2_approx(e0);
                e1 = ex2_approx(e1);
                p0 = inside(2 * i) ? e0 : 0.f;
                p1 = inside(2 * i + 1) ? e1 : 0.f;
                if constexpr (FP8) {
                  psum += p0;
                  psum += p1;
                  unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), pack_f32x2(kPScale, kPScale)), p0, p1);
                } else {
                  psum2 = add_f32x2(psum2, pack_f32x2(p0, p1));
                }
              };
              if constexpr (FP8) {
                uint32_t pk[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  float p0, p1, p2, p3;
                  prob2(2 * i, p0, p1);
                  prob2(2 * i + 1, p2, p3);
                  pk[i] = pack_e4m3x4(p0, p1, p2, p3);
                }
                tmem_st8(s_tmem + ch * 8, pk);
              } else {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  float p0, p1;
                  prob2(i, p0, p1);
                  pk[i] = pack_bf16x2(p0, p1);
                }
                tmem_st16(s_tmem + ch * 16, pk);
              }
            };
            if (__all_sync(0xffffffffu, clo <= ch * 32 && chi >= (ch + 1) * 32)) emit([](int) { return true; });
            else if (a.window < 0) emit([&](int i) { return ch * 32 + i < chi; });  // without a band the lower bound is 0
            else emit([&](int i) { return ch * 32 + i >= clo && ch * 32 + i < chi; });
          }
          if constexpr (!FP8) {
            float psum_odd;
            unpack_f32x2(psum2, psum, psum_odd);
            psum += psum_odd;
          }
          row_sum = fmaf(psum, inv_sv, row_sum);
          tmem_wait_st();
          tc_fence_before();
          mbar_arrive(bar_base + 8u * (B_P_FULL + s));
        }
        // both halves publish their partial row sums; each then divides its half of O by the total
        rowsum[(s * 2 + half) * kTile + row] = row_sum * kPScale;
        mbar_arrive(bar_base + 8u * (B_L_FULL + s));
        GDPA_WAIT_WARP(B_L_FULL + s, o_phase, ST_ROLE_EPI);
        const float l_total = row_sum * kPScale + reinterpret_cast<volatile float*>(rowsum)[(s * 2 + (half ^ 1)) * kTile + row];
        inv_l = l_total > 0.f ? 1.f / l_total : 0.f;  // a row whose band holds no key gives zeros
        if constexpr (!FP8) {
          // log-sum-exp of the scaled scores in base 2, for the softmax backward (+inf for a row without
          // keys, which makes every P of that row zero there)
          if (half == 0 && row_valid && a.lse != nullptr)
            a.lse[static_cast<long long>(w.h) * a.total_q + w.q_start + qr] = l_total > 0.f ? m_used + log2f(l_total) : INFINITY;
        }
      }
      // FP8 with an element-wise activation: S = sq sk (Q8 K8^T) per tile, and P is stored as
      // e4m3(act(S) sv_j / sv_max) with sv_max the largest V-block scale the item visits, so that every KV tile
      // adds into the same accumulator; O = qk_scale sv_max sum_j P_j V8_j (the factor goes into the epilogue).
      float fp8_sq = 1.f, fp8_inv_svmax = 1.f;
      long long fp8_kv_blk0 = 0;
      if constexpr (FP8 && !kSoftmax) {
        const int hkv = w.h / a.kv_group;
        fp8_sq = a.q_scales[static_cast<long long>(w.q_scale0 + s) * a.heads + w.h];
        fp8_kv_blk0 = w.kv_scale0;
        float sv_max = 0.f;
        for (int j = 0; j < nkv; ++j) sv_max = fmaxf(sv_max, a.v_scales[(fp8_kv_blk0 + j0 + j) * a.kv_heads + hkv]);
        fp8_inv_svmax = sv_max > 0.f ? 1.f / sv_max : 0.f;
        inv_l = a.scale * sv_max;
      }
      for (int j = 0; !kSoftmax && j < nkv; ++j) {
        // columns [clo, chi) of this warp's 64 take part: inside the KV length and inside the band
        const int kbase = (j0 + j) * kTile + half * 64;
        int clo = 0, chi = min(kTile, w.lkv - (j0 + j) * kTile) - half * 64;
        if (a.window >= 0) {
          clo = max(clo, qr - a.window - kbase);
          chi = min(chi, qr + a.window - kbase + 1);
        }
        float fp8_xs = 1.f, fp8_g = 1.f;
        if constexpr (FP8 && !kSoftmax) {
          const int hkv = w.h / a.kv_group;
          fp8_xs = fp8_sq * a.k_scales[(fp8_kv_blk0 + j0 + j) * a.kv_heads + hkv];
          fp8_g = a.v_scales[(fp8_kv_blk0 + j0 + j) * a.kv_heads + hkv] * fp8_inv_svmax;
        }
        if ((threadIdx.x & 255) == 0) GDPA_TRACE(a, tr * 32 + s * 8 + 0);
        GDPA_WAIT_WARP(B_S_FULL + s, s_phase, ST_ROLE_ACT);
        s_phase ^= 1u;
        tc_fence_after();
        if ((threadIdx.x & 255) == 0) GDPA_TRACE(a, tr * 32 + s * 8 + 1);
        uint32_t ra[32], rb[32];
        tmem_ld32(s_tmem, ra);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t(&cur)[32] = c ? rb : ra;
          uint32_t pk[16];
          tmem_wait_ld();
          tmem_regs_ready(cur);
          if (c == 0) tmem_ld32(s_tmem + 32, rb);
          if constexpr (FP8) {
            // 32 values -> 32 e4m3 in 8 registers, over the first columns of this half
            uint32_t p8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float pv[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int c0 = c * 32 + 4 * i + e;
                const float x = (c0 >= clo && c0 < chi) ? __uint_as_float(cur[4 * i + e]) * fp8_xs : 0.f;
                pv[e] = act_scaled<ACT>(x, fp8_g, 0.5f * fp8_g);
              }
              p8[i] = pack_e4m3x4(pv[0], pv[1], pv[2], pv[3]);
            }
            tmem_st8(s_tmem + c * 8, p8);
            continue;
          }
          // without a band nothing is masked (the tile's padding is zero, act(0) = 0); with one, the unmasked path
          // is taken by the warp as a whole
          if (a.window < 0 || __all_sync(0xffffffffu, clo <= c * 32 && chi >= (c + 1) * 32)) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              pk[i] = act_scaled_pair_bf16<ACT>(__uint_as_float(cur[2 * i]), __uint_as_float(cur[2 * i + 1]), scale, hscale);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int c0 = c * 32 + 2 * i;
              const float x0 = (c0 >= clo && c0 < chi) ? __uint_as_float(cur[2 * i]) : 0.f;
              const float x1 = (c0 + 1 >= clo && c0 + 1 < chi) ? __uint_as_float(cur[2 * i + 1]) : 0.f;
              pk[i] = act_scaled_pair_bf16<ACT>(x0, x1, scale, hscale);
            }
          }
          tmem_st16(s_tmem + c * 16, pk);  // over columns of this half that have been read
        }
        if ((threadIdx.x & 255) == 0) GDPA_TRACE(a, tr * 32 + s * 8 + 2);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(bar_base + 8u * (B_P_FULL + s));
        if ((threadIdx.x & 255) == 0) GDPA_TRACE(a, tr * 32 + s * 8 + 3);
        ++tr;
      }
      // Norm pipeline, a warp whose 32 rows all belong to the sequence: its residual rows are fetched now, under the
      // wait for the last P V, as whole 64-byte row pieces (four neighbouring lanes per piece), and turned into one row
      // per thread through the staging slab below.  Piece p = i * 32 + lane: row p / 4, 16-byte chunk p % 4.
      [[maybe_unused]] uint4 rres[D / 64][4];
      [[maybe_unused]] const bool fuse_staged = FUSE && (w.lq - (qr - lane) >= 32);
      if constexpr (FUSE) {
        if (fuse_staged && a.residual != nullptr) {
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int p = i * 32 + lane;
              rres[c][i] = *reinterpret_cast<const uint4*>(
                  a.residual + (static_cast<long long>(w.q_start + (qr - lane) + (p >> 2)) * a.heads + w.h) * D + half * (D / 2) +
                  c * 32 + (p & 3) * 8);
            }
        }
      }
      // epilogue: this warp's half of the O tile, TMEM -> bf16 -> global
      GDPA_WAIT_WARP(B_O_FULL + s, o_phase, ST_ROLE_EPI);
      o_phase ^= 1u;
      tc_fence_after();
      if ((threadIdx.x & 255) == 0) GDPA_TRACE(a, (tr - 1) * 32 + s * 8 + 4);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint32_t r[32];
        tmem_ld32(o_tmem + c * 32, r);
        tmem_wait_ld();
        tmem_regs_ready(r);
        if (c == D / 64 - 1) {
          tc_fence_before();
          mbar_arrive(bar_base + 8u * (B_O_EMPTY + s));
        }
        // rows of this warp's 32 inside the sequence (the same for every lane)
        const int slab_rows = w.lq - (qr - lane);
        if (kTmaOut && slab_rows >= 32) {
          // this warp's 32 rows x 32 columns: registers -> its slab (row = 64 bytes, 16-byte pieces XORed with bits 1-2
          // of the row, the 64-byte swizzle of the tensor map) -> one TMA store.  (A slab that the sequence ends in is
          // stored from registers below.)
          const uint32_t slab = smem_base + L::kOutOff + warp * L::kOutSlabBytes;
          uint8_t* const slab_row = smem + L::kOutOff + warp * L::kOutSlabBytes + lane * 64;
          if (lane == 0) tma_store_wait_read<0>();  // the store that read this slab last has finished reading it
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(r[8 * i + 0]) * inv_l, __uint_as_float(r[8 * i + 1]) * inv_l);
            v.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv_l, __uint_as_float(r[8 * i + 3]) * inv_l);
            v.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv_l, __uint_as_float(r[8 * i + 5]) * inv_l);
            v.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv_l, __uint_as_float(r[8 * i + 7]) * inv_l);
            *reinterpret_cast<uint4*>(slab_row + ((i ^ ((lane >> 1) & 3)) << 4)) = v;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tm_o.m, slab, half * (D / 2) + c * 32, w.h, w.q_start + qr);
            tma_store_commit();
          }
        } else if (kNarrowOut && slab_rows >= 32) {
          // the same with this variant's narrow slab: 16 columns at a time, 32-byte rows whose two 16-byte pieces swap
          // places in every other group of four rows (the tensor map's 32-byte swizzle)
          const uint32_t slab = smem_base + L::kNarrowOff + warp * L::kNarrowSlabBytes;
          uint8_t* const slab_row = smem + L::kNarrowOff + warp * L::kNarrowSlabBytes + lane * 32;
#pragma unroll
          for (int h2 = 0; h2 < 2; ++h2) {
            if (lane == 0) tma_store_wait_read<0>();
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int e = 16 * h2 + 8 * i;
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[e + 0]) * inv_l, __uint_as_float(r[e + 1]) * inv_l);
              v.y = pack_bf16x2(__uint_as_float(r[e + 2]) * inv_l, __uint_as_float(r[e + 3]) * inv_l);
              v.z = pack_bf16x2(__uint_as_float(r[e + 4]) * inv_l, __uint_as_float(r[e + 5]) * inv_l);
              v.w = pack_bf16x2(__uint_as_float(r[e + 6]) * inv_l, __uint_as_float(r[e + 7]) * inv_l);
              *reinterpret_cast<uint4*>(slab_row + ((i ^ ((lane >> 2) & 1)) << 4)) = v;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_3d(&tm_o.m, slab, half * (D / 2) + c * 32 + h2 * 16, w.h, w.q_start + qr);
              tma_store_commit();
            }
          }
        } else if (FUSE && fuse_staged) {
          // the norm pipeline's epilogue through the same slab: residual pieces in, one row per thread out, x = O + residual
          // and its bf16 back in, one TMA store
          const uint32_t slab = smem_base + L::kOutOff + warp * L::kOutSlabBytes;
          uint8_t* const slab_base = smem + L::kOutOff + warp * L::kOutSlabBytes;
          uint8_t* const slab_row = slab_base + lane * 64;
          if (lane == 0) tma_store_wait_read<0>();
          __syncwarp();
          uint4 own[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
          if (a.residual != nullptr) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int p = i * 32 + lane, prow = p >> 2;
              *reinterpret_cast<uint4*>(slab_base + prow * 64 + (((p & 3) ^ ((prow >> 1) & 3)) << 4)) = rres[c][i];
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) own[i] = *reinterpret_cast<const uint4*>(slab_row + ((i ^ ((lane >> 1) & 3)) << 4));
            __syncwarp();
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t rw[4] = {own[i].x, own[i].y, own[i].z, own[i].w};
            uint32_t ow[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float x0 = fmaf(__uint_as_float(r[8 * i + 2 * j]), inv_l, __uint_as_float(rw[j] << 16));
              const float x1 = fmaf(__uint_as_float(r[8 * i + 2 * j + 1]), inv_l, __uint_as_float(rw[j] & 0xffff0000u));
              ssq = fmaf(x0, x0, fmaf(x1, x1, ssq));
              ow[j] = pack_bf16x2(x0, x1);
            }
            *reinterpret_cast<uint4*>(slab_row + ((i ^ ((lane >> 1) & 3)) << 4)) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tm_o.m, slab, half * (D / 2) + c * 32, w.h, w.q_start + qr);
            tma_store_commit();
          }
        } else if (row_valid) {
          if (!FUSE || (res == nullptr && row_sumsq == nullptr)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[8 * i + 0]) * inv_l, __uint_as_float(r[8 * i + 1]) * inv_l);
              v.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv_l, __uint_as_float(r[8 * i + 3]) * inv_l);
              v.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv_l, __uint_as_float(r[8 * i + 5]) * inv_l);
              v.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv_l, __uint_as_float(r[8 * i + 7]) * inv_l);
              dst[c * 4 + i] = v;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 rv = make_uint4(0, 0, 0, 0);
              if (res != nullptr) rv = res[c * 4 + i];
              const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
              uint32_t ow[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float x0 = fmaf(__uint_as_float(r[8 * i + 2 * j]), inv_l, __uint_as_float(rw[j] << 16));
                const float x1 = fmaf(__uint_as_float(r[8 * i + 2 * j + 1]), inv_l, __uint_as_float(rw[j] & 0xffff0000u));
                ssq = fmaf(x0, x0, fmaf(x1, x1, ssq));
                ow[j] = pack_bf16x2(x0, x1);
              }
              dst[c * 4 + i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
            }
          }
        }
      }
      if (row_sumsq != nullptr && row_valid) atomicAdd(row_sumsq + w.q_start + qr, ssq);
      if ((threadIdx.x & 255) == 0) GDPA_TRACE(a, (tr - 1) * 32 + s * 8 + 5);
    }
  }

role_done:
  // Teardown: everyone meets here (also after a wait ran out), then the allocating warp frees TMEM.
  __syncwarp();
  if (*abort_flag != 0) {
    // a wait ran out: give this CTA's TMA copies and MMAs in flight a bounded time (1 ms) to finish
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 1000000ull) {}
  }
  if ((kTmaOut || kNarrowOut || FUSE) && warp < kActWarps && lane == 0) tma_store_wait_all<0>();  // this warp's stores have left shared memory
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

#undef GDPA_WAIT_WARP

template <int D, int ACT, bool FP8, bool FUSE>
int launch_fwd_fuse(const FwdLaunch& l) {
  using L = FwdSmem<D, FP8 ? 1 : 2>;
  auto kernel = gdpa_fwd_kernel<D, ACT, FP8, FUSE>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynBytes);
  if (e != cudaSuccess) return GDPA_ERR_LAUNCH_;
  kernel<<<l.grid, kFwdThreads, L::kDynBytes, l.stream>>>(l.tm_q, l.tm_k, l.tm_v, l.tm_o, l.args);
  return cudaGetLastError() == cudaSuccess ? 0 : GDPA_ERR_LAUNCH_;
}

template <int D, int ACT, bool FP8>
int launch_fwd_inst(const FwdLaunch& l) {
  // the fused epilogue exists for bf16 operands and the element-wise activations (the entry point refuses the rest)
  if constexpr (!FP8 && ACT != ACT_SOFTMAX) {
    if (l.args.residual != nullptr || l.args.row_sumsq != nullptr) return launch_fwd_fuse<D, ACT, FP8, true>(l);
  }
  return launch_fwd_fuse<D, ACT, FP8, false>(l);
}

template <int D>
int launch_fwd_d(const FwdLaunch& l, int act_class) {
  switch (act_class) {
    case ACT_RAW: return launch_fwd_inst<D, ACT_RAW, false>(l);
    case ACT_GELU_ERF: return launch_fwd_inst<D, ACT_GELU_ERF, false>(l);
    case ACT_GELU_TANH: return launch_fwd_inst<D, ACT_GELU_TANH, false>(l);
    case ACT_LEAKY_RELU: return launch_fwd_inst<D, ACT_LEAKY_RELU, false>(l);
    case ACT_RELU: return launch_fwd_inst<D, ACT_RELU, false>(l);
    case ACT_SILU: return launch_fwd_inst<D, ACT_SILU, false>(l);
    case ACT_HARDSWISH: return launch_fwd_inst<D, ACT_HARDSWISH, false>(l);
    case ACT_RELU_SQUARE: return launch_fwd_inst<D, ACT_RELU_SQUARE, false>(l);
    case ACT_SOFTMAX: return launch_fwd_inst<D, ACT_SOFTMAX, false>(l);
    default: return GDPA_ERR_UNSUPPORTED_ACT_;
  }
}

}  // namespace

int launch_fwd_bf16(const FwdLaunch& l, int head_dim, int act_class) {
  if (head_dim == 128) return launch_fwd_d<128>(l, act_class);
  if (head_dim == 64) return launch_fwd_d<64>(l, act_class);
  return GDPA_ERR_UNSUPPORTED_DIM_;
}

int launch_fwd_softmax_bf16(const FwdLaunch& l, int head_dim) { return launch_fwd_bf16(l, head_dim, ACT_SOFTMAX); }

// FP8 e4m3 operands: head_dim 128 only (a 64-byte row would need the 64-byte swizzle).
int launch_fwd_fp8(const FwdLaunch& l, int head_dim, int act_class) {
  if (head_dim != 128) return GDPA_ERR_UNSUPPORTED_DIM_;
  switch (act_class) {
    case ACT_RAW: return launch_fwd_inst<128, ACT_RAW, true>(l);
    case ACT_GELU_ERF: return launch_fwd_inst<128, ACT_GELU_ERF, true>(l);
    case ACT_GELU_TANH: return launch_fwd_inst<128, ACT_GELU_TANH, true>(l);
    case ACT_LEAKY_RELU: return launch_fwd_inst<128, ACT_LEAKY_RELU, true>(l);
    case ACT_RELU: return launch_fwd_inst<128, ACT_RELU, true>(l);
    case ACT_SILU: return launch_fwd_inst<128, ACT_SILU, true>(l);
    case ACT_HARDSWISH: return launch_fwd_inst<128, ACT_HARDSWISH, true>(l);
    case ACT_RELU_SQUARE: return launch_fwd_inst<128, ACT_RELU_SQUARE, true>(l);
    case ACT_SOFTMAX: return launch_fwd_inst<128, ACT_SOFTMAX, true>(l);
    default: return GDPA_ERR_UNSUPPORTED_ACT_;
  }
}

}  // namespace gdpa
