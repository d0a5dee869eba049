// Backward attention for sm_100a: dQ, dK, dV from dO, O and LSE.  Three kernels on one stream, each started under the one
// before (see launch_bwd):
//
//   1. preprocess   -delta[b,h,i] = -sum_d dO*O (fp32) and -lse2 = -LSE*log2(e) (stored negated so that
//                   the consumers need only fused multiply-adds), both padded to a multiple of 128 rows
//                   per (b, h); padded rows get -lse2 = -inf so that they produce P = 0.
//   2. dQ kernel    items = 128-row Q tiles; loops over K/V blocks:
//                     S  = Q K_j^T, dP = dO V_j^T            (tcgen05 SS, fp32 in TMEM)
//                     P  = exp2(S*c - lse2), dS = P o (dP - delta) -> fp16, written to TMEM columns of its own
//                     dQ += dS K_j                            (tcgen05 TS, K_j as MN-major B operand)
//   3. dK/dV kernel items = 128-key tiles of one KV head (packed batches with groups at D = 128: a CTA each); loops over
//                   the query heads of the GQA group and their Q tiles, accumulating in TMEM (fp32) so that
//                   dK/dV are written once per KV head:
//                     S^T = K Q_i^T, dP^T = V dO_i^T          (SS)
//                     P^T, dS^T -> fp16 in TMEM columns of their own
//                     dV += P^T dO_i, dK += dS^T Q_i          (TS, dO_i / Q_i as MN-major B operands)
// Warp roles in kernels 2 and 3 (640 threads): warps 0-15 elementwise math (four threads per TMEM lane,
// each owning 32 of the 128 columns of a tile), warp 16 TMA producer, warp 17 issues the SS products
// that feed the elementwise warps, warp 18 the accumulating TS products, warp 19 claims the work items (the
// kernel with a CTA per key tile does without it: 608 threads).
// TMEM columns.  dQ kernel: S [0,128), dP [128,256), dQ [256,256+D), packed dS double-buffered in
// [384,448) / [448,512).  dK/dV kernel: one 128-column accumulator region A [0,128) that holds S^T and
// then dP^T of the same Q tile in turn, packed P^T [128,192) and dS^T [192,256), dV [256,256+D),
// dK [256+D,256+2D) (at D = 64 columns 384-511 are left over and dP^T gets them as a region of its own).
// A region is handed back to the MMA warp as soon as its values sit in registers, so the next S / dP /
// S^T is computed while the elementwise warps are still busy with the current tile.
//
// Replaces flash_bwd_dot_do_o_kernel (csrc/flash_attn/src/flash_bwd_preprocess_kernel.h:23-96),
// compute_dq_1rowblock and compute_dk_dv_1colblock (src/flash_bwd_kernel.h:25-609, 613-1344) and
// the GQA group sum torch::sum_out (csrc/flash_attn/flash_api.cpp:338-348) of the reference.
#include "bwd_common.cuh"

#include <algorithm>

#include "packed_rows.cuh"
#include "work_order.cuh"

namespace fa {
namespace {

// =============================================================================================
// 1. preprocess
// =============================================================================================
struct PreParams {
  const __half* o;
  const __half* dout;
  const float* lse;
  float* delta;
  float* lse2;
  int64_t o_batch_stride, o_row_stride, o_head_stride;
  int64_t do_batch_stride, do_row_stride, do_head_stride;
  int64_t lse_row_stride;
  int h, seqlen_q, sq_pad, d;
  const int* cu_seqlens_q;
  PackedRows clear[3];  // FA_BWD_ZERO_UNUSED_ROWS: dq, dk, dv
  const int* status;
  int keys_written;     // keys per sequence that the dK/dV kernel writes: max_seqlen_k rounded up to whole tiles
};

// Work item = (group of kPreRows consecutive rows, head), heads fastest, d/8 threads per item (16-byte loads):
// the threads of a block read neighbouring heads of the same rows, i.e. contiguous memory when the heads of a
// row are adjacent, every thread has 2 * kPreRows loads in flight, and an item writes one full 32-byte sector
// of each statistic.  grid (ceil(items / items_per_block), 1, b).
// Bound by memory, with three blocks per SM: 80 registers, which the clearing code of packed calls is held to as well (one spill; left
// to itself it takes 100, two blocks).  That and the padding of short sequences left out: 16 documents of 256-4096 tokens (Hq32 D128)
// 142 -> 112 us, 64 texts of 130-640 (H16 D64) 23.2 -> 21.1, (D128) 43.6 -> 39.5.
constexpr int kPreRows = 8;
static_assert(kClearThreads == 256, "the clearing threads are those of the preprocess kernel");
template <bool kClear>
__global__ void __launch_bounds__(256, 3) bwd_preprocess_kernel(const __grid_constant__ PreParams p) {
  grid_launch_dependents();
  const bool stopped = kClear && wait_timed_out(p.status);  // read here, under the row loads
  const int tpr = p.d / 8;  // threads per item: 8 or 16
  const int item = blockIdx.x * (256 / tpr) + threadIdx.x / tpr;
  const int sub = threadIdx.x % tpr;
  const int head = item % p.h, row0 = (item / p.h) * kPreRows;
  const int batch = blockIdx.z;
  // items past the end take part in the shuffles and touch no memory (every access below is bounded)
  const int q_off = p.cu_seqlens_q ? p.cu_seqlens_q[batch] : 0;
  const int sq = min(p.cu_seqlens_q ? p.cu_seqlens_q[batch + 1] - q_off : p.seqlen_q, p.sq_pad);
  const int64_t o_base = (p.cu_seqlens_q ? static_cast<int64_t>(q_off) * p.o_row_stride : batch * p.o_batch_stride) +
                         head * p.o_head_stride + sub * 8;
  const int64_t do_base = (p.cu_seqlens_q ? static_cast<int64_t>(q_off) * p.do_row_stride : batch * p.do_batch_stride) +
                          head * p.do_head_stride + sub * 8;
  // the padding of a sequence much shorter than the longest: nothing reads statistics past its last 128-row tile
  if (__any_sync(0xffffffffu, row0 < (sq + kBlock - 1) / kBlock * kBlock)) {
    uint4 a[kPreRows], b[kPreRows];
#pragma unroll
    for (int i = 0; i < kPreRows; ++i) {
      a[i] = make_uint4(0, 0, 0, 0);
      b[i] = make_uint4(0, 0, 0, 0);
      if (row0 + i < sq) {
        a[i] = *reinterpret_cast<const uint4*>(p.o + o_base + static_cast<int64_t>(row0 + i) * p.o_row_stride);
        b[i] = *reinterpret_cast<const uint4*>(p.dout + do_base + static_cast<int64_t>(row0 + i) * p.do_row_stride);
      }
    }
    // lane `sub` of the item keeps the statistics of row `sub` (sub < kPreRows <= tpr)
    const int64_t bh = static_cast<int64_t>(batch) * p.h + head;
    float my_lse = 0.f;
    if (sub < kPreRows && row0 + sub < sq) my_lse = p.lse[bh * p.lse_row_stride + row0 + sub];
    float mine = 0.f;
#pragma unroll
    for (int i = 0; i < kPreRows; ++i) {
      const __half2* ah = reinterpret_cast<const __half2*>(&a[i]);
      const __half2* bh2 = reinterpret_cast<const __half2*>(&b[i]);
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 x = __half22float2(ah[k]), y = __half22float2(bh2[k]);
        acc = fmaf(x.x, y.x, acc);
        acc = fmaf(x.y, y.y, acc);
      }
      // sum over the tpr (8 or 16) consecutive lanes of the item; every lane ends up with the total
      for (int off = tpr / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (sub == i) mine = acc;
    }
    if (sub < kPreRows && row0 + sub < p.sq_pad) {
      const int64_t idx = bh * p.sq_pad + row0 + sub;
      const bool valid = row0 + sub < sq;
      p.delta[idx] = valid ? -mine : 0.f;
      p.lse2[idx] = valid ? -my_lse * kLog2e : -INFINITY;
    }
  }
  if constexpr (kClear) {  // the other kernels write all other rows of dq, dk, dv
    // The blocks of all sequences share the unused rows: those of one sequence are too few when the buffer is much larger than
    // what it holds.  Backward of 64 texts of 64 tokens, H16 D64, in 32768 rows: 1270 us with one sequence's blocks and a
    // division per store, 115 now; 79 in 4096 rows, and clearing the three whole tensors takes 62.
    const int64_t block = static_cast<int64_t>(blockIdx.z) * gridDim.x + blockIdx.x;
    const int64_t blocks = min(static_cast<int64_t>(gridDim.x) * gridDim.z, static_cast<int64_t>(kMaxClearBlocks));
    if (block < blocks) {
      const uint32_t worker = static_cast<uint32_t>(block) * kClearThreads + threadIdx.x;
#pragma unroll 1
      for (int i = 0; i < 3; ++i) clear_unused_rows(p.clear[i], stopped, worker, static_cast<uint32_t>(blocks) * kClearThreads);
    }
    // keys past max_seqlen_k: the first blocks of the sequence
    const int* cu_k = p.clear[1].cu_seqlens;
    const int64_t first = static_cast<int64_t>(cu_k[batch]) + p.keys_written;
    const int64_t last = min(static_cast<int64_t>(cu_k[batch + 1]), p.clear[1].total);
    const uint32_t workers = min(gridDim.x, static_cast<unsigned>(kMaxClearBlocks)) * kClearThreads;
    if (first < last && blockIdx.x < kMaxClearBlocks) {
#pragma unroll 1
      for (int i = 1; i < 3; ++i) clear_rows(p.clear[i], first, last, blockIdx.x * kClearThreads + threadIdx.x, workers);
    }
  }
}

// =============================================================================================
// 2. dQ kernel
// =============================================================================================
// A work item is one 128-row Q tile of one (sequence, query head): S = Q K^T and dP = dO V^T per key block (SS),
// P and dS in the elementwise warps, dQ += dS K (TS, A = packed dS in TMEM, two alternating buffers).  The kernel
// is persistent: one CTA per SM takes items from a global counter (heaviest causal tiles first, see section_item()) and
// keeps its barriers, its TMEM allocation and the K / V rings across items: every barrier phase is derived from
// the cumulative block count G (or the item count), the Q / dO tiles and the row statistics of the next item are
// loaded as soon as the current item has read its own for the last time, and the first S product of the next
// item is issued under the last elementwise block and the epilogue of the current one.  An item is claimed two blocks
// before the current one ends; the scheduler thread derives everything the roles need from it once and leaves it in
// shared memory (decoding it in five roles was code the instruction cache had to hold).
//
// Bound by its products (1536 clocks a block at the tensor peak) and, above S = 4096, by the power cap.  Under elect_one() against
// lane == 0 the issuing loops took B4 S4096 H32 D128 792 -> 728 us, S8192 2835 -> 2614, 64 texts H16 D64 110 -> 103.  S and dP of a block are issued back
// to back, fetched into registers together and handed back together, so that the whole arithmetic of the block runs
// under the next S / dP: ONE wait and one hand-back per block where waiting for S and dP in turn took two of each, at
// 150-300 clocks apiece for warps in lock-step.  The hand-back has to leave before the arithmetic starts (see
// schedule_barrier: without it 40 % slower, 267 against 188 us at B2 S4096 H16 D128 causal).  Measured (loops under lane == 0) per 128 x 128 block at B4 S8192 H32 D128 causal: 2511 -> 2226 clocks;
// launch, SM clocks: D128 S8192 4520 -> 4005 k, D128 S1024 462 -> 436 k, D64 S16384 3417 -> 3189 k.
constexpr int kDqThreads = 640;
constexpr int kDqSchedWarp = 19;
constexpr int kDqReaders = kComputeWarps + 3;  // elementwise warps, producer warp, two MMA threads
static_assert((kDqThreads / 32 + 3) / 4 * 32 * 96 <= 16384, "register file of one SM sub-partition");

// dQ of an item is stored at the end of the first block of the next one: its last product ends 900 to 2500 clocks after its last dS, and
// the elementwise warps, who have the next S and dP waiting, do not stand by.  The accumulator is written again only behind that
// (acc_free).  Three items are in shared memory then: the one to be stored, the current one, and the next, whose tiles are being fetched.
// dQ kernel, medians of 11 alternations: 64 texts H16 D64 99.4 -> 95.9 us, D128 135.8 -> 131.4, B16 S1024 H32 D128 243.9 -> 238.1; B4 S4096 H32
// D128 683 -> 680 and B1 S16384 H16 D64 892 -> 908, inside the spread (power-capped).  The dK/dV kernel got slower by as much in the same form (B16 S1024 347 -> 372: more code, spills in packed batches).
constexpr int kItemSlots = 3;

// A work item with everything the roles derive from it, filled in once by the scheduler thread.
struct __align__(16) DqItem {
  int nb;  // key blocks to visit; < 0: no more work
  int sk, shift, row0;
  int q_off, k_off, sq, bq;
  int batch, head, head_k, fix_k_tail;  // fix_k_tail: rows of the last K tile belong to the next sequence
};
struct DqBarriers {
  BBarriers b;
  uint64_t q_free;          // the Q / dO tiles (last dP products) and the statistics (elementwise warps) have been read
  // dS(g) is whole in packed buffer g & 1.  Two barriers in turn: a warp may be at the end of block g + 1 while another is still in
  // the arithmetic of block g (S and dP are handed back before it), and on one barrier its second arrival would stand for the other
  // warp's first: dQ(g) on half a dS.  For block g + 2, the next on the same barrier, dP(g+2) has waited for dQ(g).
  uint64_t ds_full[2];
  uint64_t acc_free;        // the accumulator of the item before has been read (see kItemSlots)
  uint64_t sched_full[kItemSlots], sched_empty[kItemSlots], sched_go;
  DqItem items[kItemSlots];
};
static_assert(sizeof(DqBarriers) <= 1024, "barrier block");

__device__ __forceinline__ void dq_make_item(const BwdKernelParams& p, int batch, int head, int mblk, DqItem& w) {
  const bool varlen = p.cu_seqlens_q != nullptr;
  w.batch = batch, w.head = head;
  w.q_off = varlen ? p.cu_seqlens_q[batch] : 0;
  w.sq = varlen ? p.cu_seqlens_q[batch + 1] - w.q_off : p.seqlen_q;
  w.k_off = varlen ? p.cu_seqlens_k[batch] : 0;
  w.sk = varlen ? p.cu_seqlens_k[batch + 1] - w.k_off : p.seqlen_k;
  w.row0 = mblk * kBlock;
  w.bq = varlen ? 0 : batch;
  w.head_k = head / p.group;
  const int nkb = (w.sk + kBlock - 1) / kBlock;
  w.shift = (p.is_causal == 2) ? p.causal_shift : w.sk - w.sq;
  w.nb = nkb;
  if (p.is_causal) {
    const int x = w.row0 + kBlock + w.shift;
    w.nb = x <= 0 ? 0 : min(nkb, (x + kBlock - 1) / kBlock);
  }
  w.fix_k_tail = varlen && (w.sk % kBlock) != 0 && w.nb == nkb && w.nb > 0;
}

template <int D>
__global__ void __launch_bounds__(kDqThreads, 1)
bwd_dq_kernel(const __grid_constant__ BwdKernelParams p) {
  using C = BCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  const int stop_probe = stop_probe_begin(p.status);

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + C::kTileBytes;
  uint8_t* sK = sdO + C::kTileBytes;
  uint8_t* sV = sK + C::kStagesK * C::kTileBytes;
  float* sStats = reinterpret_cast<float*>(sV + C::kStagesV * C::kTileBytes);  // lse2[128] | delta[128]
  DqBarriers* xb = reinterpret_cast<DqBarriers*>(reinterpret_cast<uint8_t*>(sStats) + 1024);
  BBarriers* bars = &xb->b;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == kProducerWarp && lane == 0) {
    init_barriers(bars, C::kStagesK, 2, 1);
    mbar_init(&xb->q_free, 1 + kComputeWarps);
    mbar_init(&xb->acc_free, kComputeWarps);
    for (int i = 0; i < 2; ++i) mbar_init(&xb->ds_full[i], kComputeWarps);
    for (int i = 0; i < kItemSlots; ++i) {
      mbar_init(&xb->sched_full[i], 1);
      mbar_init(&xb->sched_empty[i], kDqReaders);
    }
    mbar_init(&xb->sched_go, 1);
    fence_mbar_init();
    grid_dependency_wait();  // the row statistics; everything behind the synchronisation below may read them
    fence_acq_rel_gpu();     // ... and so may the dK/dV kernel, which starts behind the next line without a wait of its own
    grid_launch_dependents();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  const bool stop = __syncthreads_or(stop_probe) != 0;
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  WaitCtx ctx{&bars->abort_flag, p.status};

  auto wait_item = [&](int n) -> bool { return mbar_wait(&xb->sched_full[n % kItemSlots], (n / kItemSlots) & 1, ctx); };
  auto release_item = [&](int n) { mbar_arrive(&xb->sched_empty[n % kItemSlots]); };

  if (stop) {
  } else if (warp == kDqSchedWarp) {
    if (lane == 0) {
      bool finished = false;
      int seq = 0;
      for (int n = 0;; ++n) {
        int next = blockIdx.x;
        if (n > 0) {
          if (!mbar_wait(&xb->sched_go, (n - 1) & 1, ctx)) break;
          next = gridDim.x + atomicAdd(p.sched, 1);
        }
        DqItem it;
        it.nb = -1;
        while (next < p.total_items) {
          int batch, head, mblk, sq;
          if (p.cu_seqlens_q == nullptr) {
            const HeadPlace at = section_item(next, p.h * p.b, p.items_x, p.group, p.seqlen_k, p.section_rows);
            batch = at.head / p.h, head = at.head - batch * p.h, mblk = p.items_x - 1 - at.place, sq = p.seqlen_q;
          } else {  // slots per sequence from cu_seqlens_q / 128 (at most one spare slot per sequence and head)
            while (seq + 1 < p.b && p.h * ((p.cu_seqlens_q[seq + 1] >> 7) + seq + 1) <= next) ++seq;
            const int v0 = (p.cu_seqlens_q[seq] >> 7) + seq, v1 = (p.cu_seqlens_q[seq + 1] >> 7) + seq + 1;
            const int rel = next - p.h * v0, cnt = v1 - v0;
            sq = p.cu_seqlens_q[seq + 1] - p.cu_seqlens_q[seq];
            batch = seq, head = 0, mblk = -1;
            if (rel >= 0 && rel < p.h * cnt) {  // else before the first sequence (cu_seqlens_q[0] >= 128) or past the last one
              const HeadPlace at = section_item(rel, p.h, cnt, p.group, p.cu_seqlens_k[seq + 1] - p.cu_seqlens_k[seq], p.section_rows);
              head = at.head, mblk = (sq + kBlock - 1) / kBlock - 1 - at.place;
            }
          }
          if (mblk >= 0 && mblk * kBlock < sq) {
            dq_make_item(p, batch, head, mblk, it);
            break;
          }
          next = gridDim.x + atomicAdd(p.sched, 1);
        }
        if (!mbar_wait(&xb->sched_empty[n % kItemSlots], ((n / kItemSlots) & 1) ^ 1, ctx)) break;
        xb->items[n % kItemSlots] = it;
        mbar_arrive(&xb->sched_full[n % kItemSlots]);
        if (it.nb < 0) {
          finished = true;
          break;
        }
      }
      if (finished) {
        __threadfence();
        if (atomicAdd(p.sched + 1, 1) == static_cast<int>(gridDim.x) - 1) {
          atomicExch(p.sched, 0);
          atomicExch(p.sched + 1, 0);
        }
      }
    }
  } else if (warp == kProducerWarp) {
    int G = 0, ni = 0, nf = 0;
    for (int n = 0;; ++n) {
      bool ok = wait_item(n);
      if (!__all_sync(0xffffffffu, ok)) break;
      const DqItem w = xb->items[n % kItemSlots];
      __syncwarp();
      if (lane == 0) release_item(n);
      if (w.nb < 0) break;
      if (w.nb == 0) continue;
      if (lane == 0) {
        ok = mbar_wait(&xb->q_free, (ni & 1) ^ 1, ctx);
        if (ok) {
          mbar_arrive_expect_tx(&bars->fixed_full, 2 * C::kTileBytes + 1024);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c) {
            tma_load_4d(sQ + c * C::kChunkBytes, &p.tm_q, &bars->fixed_full, c * 64, w.head, w.q_off + w.row0, w.bq);
            tma_load_4d(sdO + c * C::kChunkBytes, &p.tm_do, &bars->fixed_full, c * 64, w.head, w.q_off + w.row0, w.bq);
          }
          const int64_t st = (static_cast<int64_t>(w.batch) * p.h + w.head) * p.sq_pad + w.row0;
          bulk_load_1d(sStats, p.lse2 + st, 512, &bars->fixed_full);
          bulk_load_1d(sStats + 128, p.delta + st, 512, &bars->fixed_full);
        }
        for (int j = 0; ok && j < w.nb; ++j) {
          const int g = G + j;
          const int s = g % C::kStagesK, sv = g % C::kStagesV;
          const int krow = w.k_off + j * kBlock;
          if (!(ok = mbar_wait(&bars->a_empty[s], ((g / C::kStagesK) & 1) ^ 1, ctx))) break;
          mbar_arrive_expect_tx(&bars->a_full[s], C::kTileBytes);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c)
            tma_load_4d(sK + s * C::kTileBytes + c * C::kChunkBytes, &p.tm_k, &bars->a_full[s], c * 64, w.head_k, krow, w.bq);
          if (!(ok = mbar_wait(&bars->b_empty[sv], ((g / C::kStagesV) & 1) ^ 1, ctx))) break;
          mbar_arrive_expect_tx(&bars->b_full[sv], C::kTileBytes);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c)
            tma_load_4d(sV + sv * C::kTileBytes + c * C::kChunkBytes, &p.tm_v, &bars->b_full[sv], c * 64, w.head_k, krow, w.bq);
        }
      }
      if (!__all_sync(0xffffffffu, ok)) break;
      if (w.fix_k_tail) {
        const int g = G + w.nb - 1, s = g % C::kStagesK;
        if (!mbar_wait_warp(&bars->a_full[s], (g / C::kStagesK) & 1, ctx)) break;
        zero_tile_rows_from<D>(sK + s * C::kTileBytes, w.sk - (w.nb - 1) * kBlock, lane);
        // Barriers in turn: with short items this warp can be ahead of the accumulating thread, and on one barrier that thread
        // would then wait for a phase that is over and comes round only after it has moved on.  It cannot be kItemSlots items
        // ahead: that item is published when dQ of this one has been stored.
        if (lane == 0) mbar_arrive(&bars->tail_fixed[nf % kItemSlots]);
        ++nf;
      }
      G += w.nb;
      ++ni;
    }
  } else if (warp == kMmaWarp) {
    if (elect_one()) {
      constexpr uint32_t idesc_nn = make_idesc_f16(128, kBlock, false, false);
      const uint32_t q_addr = smem_u32(sQ), do_addr = smem_u32(sdO);
      auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity, ctx); };
      int G = 0, ni = 0;
      bool ok = true;
      for (int n = 0; ok; ++n) {
        if (!(ok = wait_item(n))) break;
        const int nb = xb->items[n % kItemSlots].nb;
        release_item(n);
        if (nb < 0) break;
        if (nb <= 2) mbar_arrive(&xb->sched_go);  // short item: claim the next one right away
        if (nb == 0) continue;
        ok = wait(&bars->fixed_full, ni & 1);
        for (int j = 0; ok && j < nb; ++j) {
          const int g = G + j, s = g % C::kStagesK, sv = g % C::kStagesV;
          // the loads are polled before the hand-back of S and dP, while nothing could be issued anyway
          if (!(ok = wait(&bars->a_full[s], (g / C::kStagesK) & 1))) break;
          if (!(ok = wait(&bars->b_full[sv], (g / C::kStagesV) & 1))) break;
          if (g > 0 && !(ok = wait(&bars->s_loaded, (g - 1) & 1))) break;
          tc_fence_after_sync();
          gemm_ss<D>(tmem_base + kColS, q_addr, smem_u32(sK + s * C::kTileBytes), idesc_nn);
          // dP(g) complete tells the elementwise warps that packed-dS buffer g & 1 is free again (dQ(g-2) ends about
          // when S(g) starts)
          ok = gemm_ss<D>(tmem_base + kColDP, do_addr, smem_u32(sV + sv * C::kTileBytes), idesc_nn,
                          [&] { return g < 2 || wait(&bars->ds_free[g & 1], ((g >> 1) - 1) & 1); });
          if (!ok) break;
          tc_commit(&bars->dp_full);
          tc_commit(&bars->a_empty[s]);  // second reader: the dQ MMAs of this block
          tc_commit(&bars->b_empty[sv]);
          if (j + 1 == nb) tc_commit(&xb->q_free);  // Q and dO may be replaced
          if (nb > 2 && j + 3 == nb) mbar_arrive(&xb->sched_go);
        }
        G += nb;
        ++ni;
      }
    }
  } else if (warp == kAccMmaWarp) {
    if (elect_one()) {
      constexpr uint32_t idesc_acc = make_idesc_f16(128, D, false, true);
      int G = 0, nf = 0, na = 0;
      bool ok = true;
      for (int n = 0; ok; ++n) {
        if (!(ok = wait_item(n))) break;
        const int nb = xb->items[n % kItemSlots].nb, fix_k_tail = xb->items[n % kItemSlots].fix_k_tail;
        release_item(n);
        if (nb < 0) break;
        if (nb == 0) continue;
        for (int j = 0; ok && j < nb; ++j) {
          const int g = G + j, s = g % C::kStagesK;
          // dS(g) written implies that K(g) has landed: S(g) read it, and the elementwise warps have seen S(g)
          if (!(ok = mbar_wait(&xb->ds_full[g & 1], (g >> 1) & 1, ctx))) break;
          if (fix_k_tail && j == nb - 1) {
            if (!(ok = mbar_wait(&bars->tail_fixed[nf % kItemSlots], (nf / kItemSlots) & 1, ctx))) break;
            ++nf;
          }
          if (j == 0 && na++ > 0 && !(ok = mbar_wait(&xb->acc_free, na & 1, ctx))) break;  // phase na - 2 of the items before
          tc_fence_after_sync();
          gemm_ts<D>(tmem_base + kColAcc, tmem_base + kColPacked + (g & 1) * 64, smem_u32(sK + s * C::kTileBytes),
                     idesc_acc, j == 0);
          tc_commit(&bars->a_empty[s]);
          tc_commit(&bars->ds_free[g & 1]);
        }
        if (ok) tc_commit(&bars->acc_full);
        G += nb;
      }
    }
  } else if (warp < kComputeWarps) {
    // ---- elementwise warps: thread = (row, 32-column quarter) ----
    const int cq = warp >> 2, quarter = warp & 3;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tS = tmem_base + lane_base + kColS + cq * 32;
    const uint32_t tDP = tmem_base + lane_base + kColDP + cq * 32;
    const float c = p.scale_log2;
    const float2 c2 = make_float2(c, c);
    int G = 0, ni = 0, pending = -1;  // pending: the item whose dQ is still to be stored
    bool ok = true;
    for (int n = 0; ok; ++n) {
      ok = wait_item(n);
      if (!(ok = __all_sync(0xffffffffu, ok))) break;
      const DqItem* it = &xb->items[n % kItemSlots];  // stays in its slot until this warp has stored its dQ
      const int nb = it->nb, sk = it->sk, shift = it->shift, row = it->row0 + row_in_tile;
      float2 nl2 = make_float2(0.f, 0.f), nd2 = make_float2(0.f, 0.f);
      int j = 0;
      do {
        if (j < nb) {
          const int g = G + j;
          // dP(g) complete: S and dP are there and packed-dS buffer g & 1 is free.  S and dP are fetched at once and handed back together, then the arithmetic of the block runs under the next products.
          if (!(ok = mbar_wait_warp(&bars->dp_full, g & 1, ctx)))
            break;
          tc_fence_after_sync();
          uint32_t sr[32], dr[32];
          tmem_ld32(tS, sr);
          tmem_ld32(tDP, dr);
          if (j == 0) {  // S(0) of the item was issued after its statistics had landed
            const float l = sStats[row_in_tile], dl = sStats[128 + row_in_tile];
            nl2 = make_float2(l, l), nd2 = make_float2(dl, dl);
          }
          tmem_wait_ld();
          warp_arrive_loaded(&bars->s_loaded, lane);
          if (j == 0 && lane == 0) mbar_arrive(&xb->q_free);  // the statistics are in registers
          schedule_barrier(lane);
          const int col0 = j * kBlock + cq * 32;
          int limit = sk - 1 - col0;
          if (p.is_causal) limit = min(limit, row + shift - col0);
          float2 pr[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = ffma2(make_float2(__uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1])), c2, nl2);
            pr[i] = exp2_pair(x);
          }
          if (limit < 31) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (2 * i > limit) pr[i].x = 0.f;
              if (2 * i + 1 > limit) pr[i].y = 0.f;
            }
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 d = fmul2(pr[i], fadd2(make_float2(__uint_as_float(dr[2 * i]), __uint_as_float(dr[2 * i + 1])), nd2));
            pk[i] = pack_half2(d.x, d.y);
          }
          if (limit < 31) {  // by selection: dP of a masked column may be NaN/Inf (rows of the next sequence in V)
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (2 * i > limit) pk[i] &= 0xffff0000u;
              if (2 * i + 1 > limit) pk[i] &= 0x0000ffffu;
            }
          }
          tmem_st16(tmem_base + lane_base + kColPacked + (g & 1) * 64 + cq * 16, pk);
          warp_arrive(&xb->ds_full[g & 1], lane);
        }
        // ---- epilogue of the item before: dQ = scale * acc ----
        if (j == 0 && pending >= 0) {
          if (!(ok = mbar_wait_warp(&bars->acc_full, ni & 1, ctx))) break;
          ++ni;
          tc_fence_after_sync();
          if (cq < D / 32) {
            const DqItem* done = &xb->items[pending % kItemSlots];
            const int first = done->row0 + quarter * 32;
            uint32_t r[32];
            tmem_ld32(tmem_base + lane_base + kColAcc + cq * 32, r);
            tmem_wait_ld();
            store_scaled_rows(p.dq + done->bq * p.dq_batch_stride + static_cast<int64_t>(done->q_off + first) * p.dq_row_stride +
                                  done->head * p.dq_head_stride + cq * 32,
                              p.dq_row_stride, done->sq - first, r, p.scale, lane);
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&xb->acc_free);
          if (lane == 0) release_item(pending);
          pending = -1;
        }
      } while (++j < nb);
      if (!ok || nb < 0) break;
      if (nb > 0) {
        pending = n;
        G += nb;
      } else {  // no key is visible to any row
        if (cq < D / 32 && row < it->sq) {
          __half* to = p.dq + it->bq * p.dq_batch_stride + static_cast<int64_t>(it->q_off + row) * p.dq_row_stride +
                       it->head * p.dq_head_stride + cq * 32;
#pragma unroll
          for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(to + i * 8) = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
        if (lane == 0) release_item(n);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (bars->abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// =============================================================================================
// 3. dK/dV kernel
// =============================================================================================
// A work item is one 128-key tile of one (sequence, KV head): the CTA loops over the query heads of the GQA group
// and their Q tiles (iterations), S^T = K Q^T and dP^T = V dO^T per iteration (SS), P^T and dS^T in the elementwise
// warps, dV += P^T dO and dK += dS^T Q (TS) accumulated in TMEM over the whole group.  Persistent like the dQ
// kernel: one CTA per SM takes items from the work counter (heaviest causal key tiles first), every barrier phase
// is derived from the cumulative iteration count T (or the item count), the K / V tiles of the next item are
// loaded as soon as the last dP^T product of the current item has read them, and its first S^T product is issued
// under the last elementwise iteration and the epilogue of the current one.  Bound by the chain of a tile through the sixteen
// elementwise warps (about 3250 clocks a tile at D = 128, of 2048 at the tensor peak; 2250 at D = 64).
//   D = 64: the row statistics of a tile arrive on the barrier of its Q tile (there is shared memory for as many stages of them),
// which the thread that issues S^T waits for anyway: the elementwise warps, which have seen S^T, need no wait and no release of
// their own.  2600 -> 2510 us at B2 S16384 H16 causal, 377 -> 364 at B4 S4096, 49.2 -> 47.1 at B4 Sq333 Sk2047.
//   kVarlen: packed sequences.  A Q tile can hold rows of the neighbouring sequence; this form carries the code that guards
// against them.  D = 64, and D = 128 without grouped heads; the rest goes to bwd_dkdv_packed_kernel (see there).
constexpr int kDkvThreads = 640;  // + one scheduler warp: 20 warps, five on one sub-partition -> 96 registers
constexpr int kDkvSchedWarp = 19;
constexpr int kDkvReaders = kComputeWarps + 3;  // elementwise warps, producer warp, two MMA threads
static_assert((kDkvThreads / 32 + 3) / 4 * 32 * 96 <= 16384, "register file of one SM sub-partition");
struct __align__(16) DkvItem {
  int batch, head_k, nblk, q_off;  // nblk < 0: no more work
  int k_off, sq, sk, pad;          // the extents of the sequence: from cu_seqlens_* for packed batches
};
struct DkvBarriers {
  BBarriers b;
  uint64_t kv_free;         // the K / V tiles of the item have been read for the last time
  uint64_t sched_full[2], sched_empty[2], sched_go;
  DkvItem items[2];
};
static_assert(sizeof(DkvBarriers) <= 512, "barrier block");

struct DkvWork {
  int batch, head_k, q_off, k_off, sq, sk, key0, group, nq, i_min, shift, per_head, n_it;
};
template <bool kVarlen>
__device__ __forceinline__ DkvWork dkv_decode(const BwdKernelParams& p, const DkvItem& it) {
  DkvWork w;
  w.batch = it.batch, w.head_k = it.head_k;
  w.q_off = kVarlen ? it.q_off : 0, w.k_off = kVarlen ? it.k_off : 0;
  w.sq = kVarlen ? it.sq : p.seqlen_q;
  w.sk = kVarlen ? it.sk : p.seqlen_k;
  w.key0 = it.nblk * kBlock;
  w.group = p.group;
  w.nq = (w.sq + kBlock - 1) / kBlock;
  w.i_min = 0;
  w.shift = (p.is_causal == 2) ? p.causal_shift : w.sk - w.sq;  // key j visible to query i iff j <= i + shift
  if (p.is_causal) {
    const int first_row = w.key0 - w.shift;  // first query row that can see key0
    w.i_min = first_row <= 0 ? 0 : first_row / kBlock;
  }
  w.per_head = max(0, w.nq - w.i_min);
  w.n_it = w.per_head * w.group;
  return w;
}

template <int D, bool kVarlen>
__global__ void __launch_bounds__(kDkvThreads, 1)
bwd_dkdv_kernel(const __grid_constant__ BwdKernelParams p) {
  using C = BCfg<D>;
  // P^T and dS^T are handed back together, by the dK product, which is long over when the next P^T is written: one wait less per
  // tile.  D64 2524 -> 2431 us at B2 S16384 H16 causal, 369 -> 354 at B4 S4096, 47.1 -> 46.0 at B4 Sq333 Sk2047; at D = 128 +1 to -1 %, in
  // packed batches +2 to +5 % with one or two tiles an item (spills).
  constexpr bool kOneRelease = D == 64 && !kVarlen;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int stop_probe = stop_probe_begin(p.status);

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::kTileBytes;
  uint8_t* sQ = sV + C::kTileBytes;
  uint8_t* sdO = sQ + C::kStagesQ * C::kTileBytes;
  float* sStats = reinterpret_cast<float*>(sdO + C::kStagesDO * C::kTileBytes);  // [kStatsStages][lse2 128 | delta 128]
  DkvBarriers* xb = reinterpret_cast<DkvBarriers*>(reinterpret_cast<uint8_t*>(sStats) + C::kStatsStages * 1024);
  BBarriers* bars = &xb->b;
  if (smem - smem_raw > C::kAlignPadDkdv) {  // uniform over the CTA: nothing has been set up yet
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, kStatusSmemLayout);
    grid_dependency_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == kProducerWarp && lane == 0) {
    init_barriers(bars, C::kStagesQ, 2, 2);
    mbar_init(&xb->kv_free, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&xb->sched_full[i], 1);
      mbar_init(&xb->sched_empty[i], kDkvReaders);
    }
    mbar_init(&xb->sched_go, 1);
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  const bool stop = __syncthreads_or(stop_probe) != 0;  // sticky time-out bit set: the CTA does no work
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  WaitCtx ctx{&bars->abort_flag, p.status};

  auto read_item = [&](int n, DkvItem& it) -> bool {
    if (!mbar_wait(&xb->sched_full[n & 1], (n >> 1) & 1, ctx)) return false;
    it = xb->items[n & 1];
    return true;
  };
  auto release_item = [&](int n) { mbar_arrive(&xb->sched_empty[n & 1]); };

  if (stop) {
  } else if (warp == kDkvSchedWarp) {
    if (lane == 0) {
      bool finished = false;
      int seq = 0;  // packed sequences: the sequence of the last claimed index
      for (int n = 0;; ++n) {
        int next = blockIdx.x;
        if (n > 0) {
          if (!mbar_wait(&xb->sched_go, (n - 1) & 1, ctx)) break;
          next = gridDim.x + atomicAdd(p.sched, 1);
        }
        DkvItem it;
        it.batch = 0, it.head_k = 0, it.nblk = -1, it.pad = 0, it.q_off = 0, it.k_off = 0;
        it.sq = p.seqlen_q, it.sk = p.seqlen_k;
        if constexpr (!kVarlen) {
          if (next < p.total_items) {  // every index is a live item: key tile 0 of a head is the heaviest
            const HeadPlace at = section_item(next, p.h_k * p.b, p.items_x, 1, p.seqlen_q, p.section_rows);
            it.batch = at.head / p.h_k, it.head_k = at.head - it.batch * p.h_k, it.nblk = at.place;
          }
        } else {
          while (next < p.total_items) {  // slots per sequence from cu_seqlens_k / 128 (see the forward kernel)
            while (seq + 1 < p.b && p.h_k * ((p.cu_seqlens_k[seq + 1] >> 7) + seq + 1) <= next) ++seq;
            const int k0 = p.cu_seqlens_k[seq], k1 = p.cu_seqlens_k[seq + 1];
            const int v0 = (k0 >> 7) + seq, v1 = (k1 >> 7) + seq + 1;
            const int rel = next - p.h_k * v0, cnt = v1 - v0;
            if (rel >= 0 && rel < p.h_k * cnt) {
              it.q_off = p.cu_seqlens_q[seq], it.sq = p.cu_seqlens_q[seq + 1] - it.q_off;
              const HeadPlace at = section_item(rel, p.h_k, cnt, 1, it.sq, p.section_rows);
              // items_x: key tiles up to the maximum the caller gave; later ones are not computed
              if (at.place < p.items_x && at.place * kBlock < k1 - k0) {
                it.batch = seq, it.head_k = at.head, it.nblk = at.place;
                it.k_off = k0, it.sk = k1 - k0;
                break;
              }
            }
            next = gridDim.x + atomicAdd(p.sched, 1);
          }
        }
        if (!mbar_wait(&xb->sched_empty[n & 1], ((n >> 1) & 1) ^ 1, ctx)) break;
        xb->items[n & 1] = it;
        mbar_arrive(&xb->sched_full[n & 1]);
        if (it.nblk < 0) {
          finished = true;
          break;
        }
      }
      if (finished) {
        __threadfence();
        if (atomicAdd(p.sched + 1, 1) == static_cast<int>(gridDim.x) - 1) {
          atomicExch(p.sched, 0);
          atomicExch(p.sched + 1, 0);
        }
      }
    }
  } else if (warp == kProducerWarp) {
    int T0 = 0, ni = 0;
    for (int n = 0;; ++n) {
      DkvItem item;
      bool ok = read_item(n, item);
      if (!__all_sync(0xffffffffu, ok)) break;
      __syncwarp();
      if (lane == 0) release_item(n);
      if (item.nblk < 0) break;
      const DkvWork w = dkv_decode<kVarlen>(p, item);
      if (w.n_it == 0) continue;
      // Q tile, row statistics and dO tile of iteration `it` of the item into the rings at position T0 + it
      auto load_q_do = [&](int it) -> bool {
        const int T = T0 + it;
        const int sq_ = T % C::kStagesQ, sd = T % C::kStagesDO, ss = T & 1;
        const uint32_t phq = (T / C::kStagesQ) & 1, phd = (T / C::kStagesDO) & 1, phs = (T >> 1) & 1;
        const int head = w.head_k * w.group + it / w.per_head;
        const int i = w.i_min + it % w.per_head;
        const int qrow = w.q_off + i * kBlock;
        const int64_t stat = (static_cast<int64_t>(w.batch) * p.h + head) * p.sq_pad + i * kBlock;
        if (!mbar_wait(&bars->a_empty[sq_], phq ^ 1, ctx)) return false;
        mbar_arrive_expect_tx(&bars->a_full[sq_], C::kTileBytes + (C::kStatsWithQ ? 1024 : 0));
        if constexpr (C::kStatsWithQ) {
          bulk_load_1d(sStats + sq_ * 256, p.lse2 + stat, 512, &bars->a_full[sq_]);
          bulk_load_1d(sStats + sq_ * 256 + 128, p.delta + stat, 512, &bars->a_full[sq_]);
        }
#pragma unroll
        for (int c = 0; c < C::kChunks; ++c)
          tma_load_4d(sQ + sq_ * C::kTileBytes + c * C::kChunkBytes, &p.tm_q, &bars->a_full[sq_], c * 64, head, qrow, kVarlen ? 0 : w.batch);
        if constexpr (!C::kStatsWithQ) {
          if (!mbar_wait(&bars->st_empty[ss], phs ^ 1, ctx)) return false;
          mbar_arrive_expect_tx(&bars->st_full[ss], 1024);
          bulk_load_1d(sStats + ss * 256, p.lse2 + stat, 512, &bars->st_full[ss]);
          bulk_load_1d(sStats + ss * 256 + 128, p.delta + stat, 512, &bars->st_full[ss]);
        }
        if (!mbar_wait(&bars->b_empty[sd], phd ^ 1, ctx)) return false;
        mbar_arrive_expect_tx(&bars->b_full[sd], C::kTileBytes);
#pragma unroll
        for (int c = 0; c < C::kChunks; ++c)
          tma_load_4d(sdO + sd * C::kTileBytes + c * C::kChunkBytes, &p.tm_do, &bars->b_full[sd], c * 64, head, qrow, kVarlen ? 0 : w.batch);
        return true;
      };
      if (lane == 0) {
        ok = mbar_wait(&xb->kv_free, (ni & 1) ^ 1, ctx);
        if (ok) {
          mbar_arrive_expect_tx(&bars->fixed_full, 2 * C::kTileBytes);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c) {
            tma_load_4d(sK + c * C::kChunkBytes, &p.tm_k, &bars->fixed_full, c * 64, w.head_k, w.k_off + w.key0, kVarlen ? 0 : w.batch);
            tma_load_4d(sV + c * C::kChunkBytes, &p.tm_v, &bars->fixed_full, c * 64, w.head_k, w.k_off + w.key0, kVarlen ? 0 : w.batch);
          }
        }
      }
      if (!kVarlen || (w.sq % kBlock) == 0) {
        if (lane == 0) {
          for (int it = 0; ok && it < w.n_it; ++it) ok = load_q_do(it);
        }
      } else {
        // the whole warp walks the tiles: lane 0 issues the loads, all lanes zero the rows of the next sequence
        ok = __all_sync(0xffffffffu, ok);
        for (int it = 0; ok && it < w.n_it; ++it) {
          if (lane == 0) ok = load_q_do(it);
          if (!(ok = __all_sync(0xffffffffu, ok))) break;
          if (it % w.per_head == w.per_head - 1) {  // the last Q tile of this head
            const int T = T0 + it, sq_ = T % C::kStagesQ, sd = T % C::kStagesDO;
            if (!(ok = mbar_wait_warp(&bars->a_full[sq_], (T / C::kStagesQ) & 1, ctx))) break;
            if (!(ok = mbar_wait_warp(&bars->b_full[sd], (T / C::kStagesDO) & 1, ctx))) break;
            const int q_tail_rows = w.sq - (w.nq - 1) * kBlock;
            zero_tile_rows_from<D>(sQ + sq_ * C::kTileBytes, q_tail_rows, lane);
            zero_tile_rows_from<D>(sdO + sd * C::kTileBytes, q_tail_rows, lane);
            if (lane == 0) mbar_arrive(&bars->tail_fixed[sd]);
          }
        }
      }
      if (!__all_sync(0xffffffffu, ok)) break;
      T0 += w.n_it;
      ++ni;
    }
  } else if (warp == kMmaWarp) {
    if (elect_one()) {
      constexpr uint32_t idesc_nn = make_idesc_f16(128, kBlock, false, false);
      const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV);
      // One accumulator region A holds S^T(T) and then dP^T(T): dP^T(T) is issued as soon as S^T(T)
      // sits in registers, S^T(T+1) as soon as dP^T(T) does.  The hooks wait for the TMA load the next
      // product reads.
      auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity, ctx); };
      auto q_tile = [&](int T) { return smem_u32(sQ + (T % C::kStagesQ) * C::kTileBytes); };
      auto do_tile = [&](int T) { return smem_u32(sdO + (T % C::kStagesDO) * C::kTileBytes); };
      auto q_full = [&](int T) { return wait(&bars->a_full[T % C::kStagesQ], (T / C::kStagesQ) & 1); };
      auto do_full = [&](int T) { return wait(&bars->b_full[T % C::kStagesDO], (T / C::kStagesDO) & 1); };
      const uint32_t tA = tmem_base + kColS, tA2 = tmem_base + kColDPT<D>;
      constexpr bool kSharedRegion = kColDPT<D> == kColS;
      int T0 = 0, ni = 0;
      bool ok = true;
      for (int n = 0; ok; ++n) {
        DkvItem item;
        if (!(ok = read_item(n, item))) break;
        release_item(n);
        if (item.nblk < 0) break;
        const DkvWork w = dkv_decode<kVarlen>(p, item);
        // the next item is claimed kGoAhead iterations before this one ends; a shorter item: right away
        constexpr int kGoAhead = 2;
        if (w.n_it <= kGoAhead) mbar_arrive(&xb->sched_go);
        if (w.n_it == 0) continue;
        ok = wait(&bars->fixed_full, ni & 1) && q_full(T0);
        for (int it = 0; ok && it < w.n_it; ++it) {
          const int T = T0 + it;
          // region A is free once its last content was read: dP^T(T-1) when the region is shared, S^T(T-1) otherwise
          if (T > 0 && !(ok = wait(kSharedRegion ? &bars->dp_loaded : &bars->s_loaded, (T - 1) & 1))) break;
          tc_fence_after_sync();
          ok = gemm_ss<D>(tA, k_addr, q_tile(T), idesc_nn, [&] { return do_full(T); });  // S^T = K Q^T
          if (!ok) break;
          tc_commit(&bars->s_full);
          tc_commit(&bars->a_empty[T % C::kStagesQ]);  // second reader: the dK MMAs of this tile
          // the region of dP^T is free once S^T(T) (shared) or dP^T(T-1) (own region) was read
          if (kSharedRegion) {
            if (!(ok = wait(&bars->s_loaded, T & 1))) break;
          } else if (T > 0) {
            if (!(ok = wait(&bars->dp_loaded, (T - 1) & 1))) break;
          }
          tc_fence_after_sync();
          ok = gemm_ss<D>(tA2, v_addr, do_tile(T), idesc_nn,  // dP^T = V dO^T
                          [&] { return it + 1 >= w.n_it || q_full(T + 1); });
          if (!ok) break;
          tc_commit(&bars->dp_full);
          tc_commit(&bars->b_empty[T % C::kStagesDO]);  // second reader: the dV MMAs of this tile
          if (it + 1 == w.n_it) tc_commit(&xb->kv_free);  // K and V may be replaced
          if (w.n_it > kGoAhead && it + kGoAhead + 1 == w.n_it) mbar_arrive(&xb->sched_go);
        }
        T0 += w.n_it;
        ++ni;
      }
    }
  } else if (warp == kAccMmaWarp) {
    if (elect_one()) {
      // dV += P^T dO as soon as the packed P^T is written, dK += dS^T Q likewise.
      constexpr uint32_t idesc_acc = make_idesc_f16(128, D, false, true);
      const uint32_t tP = tmem_base + kColDP, tDS = tmem_base + kColDP + 64;
      const uint32_t tDV = tmem_base + kColAcc, tDK = tmem_base + kColAcc + D;
      bool ok = true;
      int T0 = 0;
      uint32_t tail_phase = 0;  // bit sd: parity of the next tail_fixed[sd] phase to wait for
      for (int n = 0; ok; ++n) {
        DkvItem item;
        if (!(ok = read_item(n, item))) break;
        release_item(n);
        if (item.nblk < 0) break;
        const DkvWork w = dkv_decode<kVarlen>(p, item);
        if (w.n_it == 0) continue;
        for (int it = 0; ok && it < w.n_it; ++it) {
          const int T = T0 + it;
          const int sq_ = T % C::kStagesQ, sd = T % C::kStagesDO;
          if (!(ok = mbar_wait(&bars->b_full[sd], (T / C::kStagesDO) & 1, ctx))) break;
          if (!(ok = mbar_wait(&bars->p_full, T & 1, ctx))) break;
          if (kVarlen && (w.sq % kBlock) != 0 && it % w.per_head == w.per_head - 1) {
            if (!(ok = mbar_wait(&bars->tail_fixed[sd], (tail_phase >> sd) & 1, ctx))) break;
            tail_phase ^= 1u << sd;
          }
          tc_fence_after_sync();
          gemm_ts<D>(tDV, tP, smem_u32(sdO + sd * C::kTileBytes), idesc_acc, it == 0);
          tc_commit(&bars->b_empty[sd]);
          if constexpr (!kOneRelease) tc_commit(&bars->p_free);
          if (!(ok = mbar_wait(&bars->a_full[sq_], (T / C::kStagesQ) & 1, ctx))) break;
          if (!(ok = mbar_wait(&bars->ds_full, T & 1, ctx))) break;
          tc_fence_after_sync();
          gemm_ts<D>(tDK, tDS, smem_u32(sQ + sq_ * C::kTileBytes), idesc_acc, it == 0);
          tc_commit(&bars->a_empty[sq_]);
          tc_commit(&bars->ds_free[0]);
        }
        if (ok) tc_commit(&bars->acc_full);
        T0 += w.n_it;
      }
    }
  } else if (warp < kComputeWarps) {
    // ---- elementwise warps: thread = (key row, 32-query-column quarter) ----
    const int cq = warp >> 2, quarter = warp & 3;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tA = tmem_base + lane_base + kColS + cq * 32;         // S^T, then dP^T
    const uint32_t tP = tmem_base + lane_base + kColDP + cq * 16;        // packed P^T
    const float c = p.scale_log2;
    const float2 c2 = make_float2(c, c);
    const float* stats = sStats + cq * 32;
    int T0 = 0, ni = 0;
    bool ok = true;
    for (int n = 0; ok; ++n) {
      int n_it, per_head, cmin0, cmax_last;
      {
        DkvItem item;
        ok = read_item(n, item);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        if (item.nblk < 0) break;
        const DkvWork w = dkv_decode<kVarlen>(p, item);
        n_it = w.n_it, per_head = w.per_head;
        // valid columns in the last Q tile
        cmax_last = kVarlen ? max(0, min(32, w.sq - (w.nq - 1) * kBlock - cq * 32)) : 32;
        // causal: query column q of tile i is masked for this key when key > q + shift, i.e. the columns of
        // this thread's quarter below  key - shift - (i * 128 + cq * 32)  are masked
        cmin0 = p.is_causal ? (w.key0 + row_in_tile) - w.shift - (w.i_min * kBlock + cq * 32) : 0;
      }
      int i_rel = 0;  // Q tile within the current head
      for (int it = 0; it < n_it; ++it) {
        const int T = T0 + it;
        const int ss = C::kStatsWithQ ? T % C::kStagesQ : T & 1;
        if constexpr (!C::kStatsWithQ) {
          if (!(ok = mbar_wait_warp(&bars->st_full[ss], (T >> 1) & 1, ctx))) break;
        }
        // D = 128: the LSE of this thread's 32 query columns is fetched while the warp waits for S^T anyway.
        // Read after the wait, these shared-memory loads compete with the operand fetches of the dP^T MMAs, which
        // take the whole shared-memory bandwidth (measured: 4.5-7 % of the kernel; at D = 64 the MMAs are half as
        // long and the early loads cost 2 % instead).
        const float4* st_lse = reinterpret_cast<const float4*>(stats + ss * 256);
        const float4* st_delta = reinterpret_cast<const float4*>(stats + ss * 256 + 128);
        constexpr bool kEarlyLse = (D == 128);
        float4 lse_q[8];
        if constexpr (kEarlyLse) {
#pragma unroll
          for (int e = 0; e < 8; ++e) lse_q[e] = st_lse[e];
        }
        if (!(ok = mbar_wait_warp(&bars->s_full, T & 1, ctx))) break;
        tc_fence_after_sync();
        uint32_t sr[32];
        tmem_ld32(tA, sr);
        tmem_wait_ld();
        warp_arrive_loaded(&bars->s_loaded, lane);  // region A may now receive dP^T
        // whole backward, best of five without it against with: 64 texts of 130-640 tokens H16 443 : 438 us, 16 documents H8
        // 644 : 633, 8 of 520-3000 H4 not causal 144 : 142 (medians inside the spread); dense batches: nothing
        if constexpr (kVarlen && D == 128) schedule_barrier(lane);
        // columns below cmin are masked by causality (clamped to [0, 32])
        const int cmask = max(0, min(32, cmin0 - i_rel * kBlock)) | (((kVarlen && i_rel == per_head - 1) ? cmax_last : 32) << 8);
        const bool col_masked = cmask != (32 << 8);
        if (++i_rel == per_head) i_rel = 0;
        float2 pr[16];
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float4 l = kEarlyLse ? lse_q[e] : st_lse[e];
          pr[2 * e] = exp2_pair(ffma2(make_float2(__uint_as_float(sr[4 * e]), __uint_as_float(sr[4 * e + 1])), c2,
                                      make_float2(l.x, l.y)));
          pr[2 * e + 1] = exp2_pair(ffma2(make_float2(__uint_as_float(sr[4 * e + 2]), __uint_as_float(sr[4 * e + 3])),
                                          c2, make_float2(l.z, l.w)));
        }
        if (col_masked) {
          const int cmin = cmask & 0xff, cmax = kVarlen ? cmask >> 8 : 32;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            if (2 * e < cmin || 2 * e >= cmax) pr[e].x = 0.f;
            if (2 * e + 1 < cmin || 2 * e + 1 >= cmax) pr[e].y = 0.f;
          }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack_half2(pr[e].x, pr[e].y);
        // the dV MMAs of the previous tile must have consumed the old P^T before it is overwritten; kOneRelease: the dK MMAs
        // behind them the old dS^T too
        if (T > 0 && !(ok = mbar_wait_warp(kOneRelease ? &bars->ds_free[0] : &bars->p_free, (T - 1) & 1, ctx))) break;
        tmem_st16(tP, pk);
        warp_arrive(&bars->p_full, lane);

        if (!(ok = mbar_wait_warp(&bars->dp_full, T & 1, ctx))) break;
        tc_fence_after_sync();
        tmem_ld32(tA + (kColDPT<D> - kColS), sr);
        tmem_wait_ld();
        warp_arrive_loaded(&bars->dp_loaded, lane);  // region A may now receive the next S^T
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float4 dl = st_delta[e];
          const float2 d0 = fmul2(pr[2 * e], fadd2(make_float2(__uint_as_float(sr[4 * e]), __uint_as_float(sr[4 * e + 1])),
                                                   make_float2(dl.x, dl.y)));
          const float2 d1 = fmul2(pr[2 * e + 1], fadd2(make_float2(__uint_as_float(sr[4 * e + 2]), __uint_as_float(sr[4 * e + 3])),
                                                       make_float2(dl.z, dl.w)));
          pk[2 * e] = pack_half2(d0.x, d0.y);
          pk[2 * e + 1] = pack_half2(d1.x, d1.y);
        }
        if (col_masked) {  // by selection: dP of a masked column may be NaN/Inf (dO rows of the next sequence)
          const int cmin = cmask & 0xff, cmax = kVarlen ? cmask >> 8 : 32;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            if (2 * e < cmin || 2 * e >= cmax) pk[e] &= 0xffff0000u;
            if (2 * e + 1 < cmin || 2 * e + 1 >= cmax) pk[e] &= 0x0000ffffu;
          }
        }
        if constexpr (!C::kStatsWithQ) {  // the statistics of this tile are in use no longer
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->st_empty[ss]);
        }
        if (!kOneRelease && T > 0 && !(ok = mbar_wait_warp(&bars->ds_free[0], (T - 1) & 1, ctx))) break;
        tmem_st16(tP + 64, pk);  // packed dS^T
        warp_arrive(&bars->ds_full, lane);
      }
      if (!ok) break;
      // ---- epilogue: column quarters 0,1 store the halves of dV, quarters 2,3 the halves of dK * scale; what it
      // needs of the item is derived again from the ring slot ----
      DkvItem item;
      {
        const volatile int* src = reinterpret_cast<const volatile int*>(&xb->items[n & 1]);
        item.batch = src[0], item.head_k = src[1], item.nblk = src[2], item.q_off = src[3];
        item.k_off = src[4], item.sq = src[5], item.sk = src[6], item.pad = 0;
      }
      const DkvWork w = dkv_decode<kVarlen>(p, item);
      const int key = w.key0 + row_in_tile;
      const int which = cq >> 1;        // 0 = dV, 1 = dK
      const int col_half = cq & 1;      // which D/2 columns
      __half* dst_base = (which == 0) ? p.dv : p.dk;
      const int64_t bs = (which == 0) ? p.dv_batch_stride : p.dk_batch_stride;
      const int64_t rs = (which == 0) ? p.dv_row_stride : p.dk_row_stride;
      const int64_t hs = (which == 0) ? p.dv_head_stride : p.dk_head_stride;
      __half* dst = dst_base + (kVarlen ? 0 : w.batch * bs) + static_cast<int64_t>(w.k_off + key) * rs + w.head_k * hs + col_half * (D / 2);
      const float mul = (which == 0) ? 1.f : p.scale;
      if (n_it > 0) {
        if (!(ok = mbar_wait_warp(&bars->acc_full, ni & 1, ctx))) break;
        ++ni;
        tc_fence_after_sync();
#pragma unroll
        for (int q = 0; q < D / 64; ++q) {
          uint32_t r[32];
          tmem_ld32(tmem_base + lane_base + kColAcc + which * D + col_half * (D / 2) + q * 32, r);
          tmem_wait_ld();
          store_scaled_rows(dst - lane * rs + q * 32, rs, w.sk - (key - lane), r, mul, lane);
        }
        tc_fence_before_sync();
      } else if (key < w.sk) {
        const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i3 = 0; i3 < D / 16; ++i3) *reinterpret_cast<uint4*>(dst + i3 * 8) = z;
      }
      T0 += n_it;
      __syncwarp();
      if (lane == 0) release_item(n);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (bars->abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
  // the dQ kernel may still be running: this launch must not complete before it (see launch_bwd)
  if (blockIdx.x == 0 && threadIdx.x == 0) grid_dependency_wait();
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// =============================================================================================
// 4. dK/dV kernel for packed sequences, one CTA per (sequence, KV head, key tile)
// =============================================================================================
// The same products and hand-offs as bwd_dkdv_kernel, but launched as a grid of max_seqlen_k / 128 x h_k x b CTAs
// that each set up, process one key tile and exit.  Kept for packed batches with grouped heads at D = 128, whose items are several
// times as long and gain little from running into one another: this kernel against the persistent one, 16 documents of 256-4096 tokens
// Hq32 Hkv8 1556 : 1650 us, 24 of 700-1700 Hq16 Hkv4 430 : 456, 4 of 4096-8192 1066 : 1126.  Whole backward, Hq16, groups of
// 2 / 4 / 8 / 16: 16 documents 1263 : 1251, 1268 : 1353, 1252 : 1447, 1455 : 1632 us, 64 texts of 130-640 tokens 415 : 407, 394 : 409,
// -, 439 : 482; with groups of 2 the two are within what runs of one differ.  The other way round without
// groups (64 texts of 130-640 tokens H16 308 : 254, 24 of 700-1700 not causal 812 : 782) and at D = 64 (64 texts of 130-640 H16
// 227 : 168, 16 documents 609 : 528, 32 of 500-1500 Hq16 Hkv4 457 : 438; groups of 16 there 331 : 333).
// A Q tile of a packed batch can hold rows of the neighbouring sequence; this kernel carries the code that guards
// against them.

// The z-th largest sequence by the pairs of a head, for up to 32 of them; otherwise the z-th.  Called by whole warps.
// Blocks start in the order of the grid, and an item of the longest sequence can take a tenth of the launch: begun last, it runs on
// alone: 16 documents of 256-4096 tokens Hq32 Hkv8 1557 -> 1538 us, 4 of 4096-8192 Hq16 Hkv4 1034 -> 995, 24 of 700-1700 the same.
// (32: one lane of a warp each.  The forward gained nothing from the same order over the sequences of a cache.)
__device__ __forceinline__ int sequence_by_size(const int* cu_q, const int* cu_k, int b, int z) {
  if (b > 32) return z;
  const int lane = threadIdx.x & 31;
  float size = -1.f;
  if (lane < b) size = static_cast<float>(cu_q[lane + 1] - cu_q[lane]) * static_cast<float>(cu_k[lane + 1] - cu_k[lane]);
  int rank = 0;
  for (int j = 0; j < b; ++j) {
    const float other = __shfl_sync(0xffffffffu, size, j);
    rank += other > size || (other == size && j < lane);
  }
  return __ffs(__ballot_sync(0xffffffffu, lane < b && rank == z)) - 1;
}

__global__ void __launch_bounds__(kNumThreads, 1)
bwd_dkdv_packed_kernel(const __grid_constant__ BwdKernelParams p) {
  constexpr int D = 128;
  using C = BCfg<D>;
  static_assert(kColDPT<D> == kColS && !C::kStatsWithQ, "S^T and dP^T share a region, the statistics have a ring of their own");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int batch = sequence_by_size(p.cu_seqlens_q, p.cu_seqlens_k, p.b, blockIdx.z);
  const int q_off = p.cu_seqlens_q[batch];
  const int sq = p.cu_seqlens_q[batch + 1] - q_off;
  const int k_off = p.cu_seqlens_k[batch];
  const int sk = p.cu_seqlens_k[batch + 1] - k_off;
  const bool first_cta = (blockIdx.x | blockIdx.z) == 0;
  int nblk = blockIdx.x / p.h_k, head_k = blockIdx.x - nblk * p.h_k;  // the heaviest key tiles of all heads first
  if (nblk * kBlock >= sk) {
    if (first_cta) grid_dependency_wait();
    return;
  }
  if (static_cast<int64_t>(sq) * p.h_k > p.section_rows) {  // section by section
    const HeadPlace at = section_item(blockIdx.x, p.h_k, min((sk + kBlock - 1) / kBlock, static_cast<int>(gridDim.x) / p.h_k), 1, sq, p.section_rows);
    nblk = at.place, head_k = at.head;
  }
  const int key0 = nblk * kBlock;
  const int stop_probe = stop_probe_begin(p.status);
  const int group = p.group;
  const int nq = (sq + kBlock - 1) / kBlock;
  int i_min = 0;
  const int shift = sk - sq;  // key j visible to query i iff j <= i + shift (FA_CAUSAL_SHIFT is for dense batches)
  if (p.is_causal) {
    const int first_row = key0 - shift;  // first query row that can see key0
    i_min = first_row <= 0 ? 0 : first_row / kBlock;
  }
  const int per_head = max(0, nq - i_min);
  const int n_it = per_head * group;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::kTileBytes;
  uint8_t* sQ = sV + C::kTileBytes;
  uint8_t* sdO = sQ + C::kStagesQ * C::kTileBytes;
  float* sStats = reinterpret_cast<float*>(sdO + C::kStagesDO * C::kTileBytes);  // [kStatsStages][lse2 128 | delta 128]
  BBarriers* bars = reinterpret_cast<BBarriers*>(reinterpret_cast<uint8_t*>(sStats) + C::kStatsStages * 1024);
  static_assert(sizeof(BBarriers) <= 512, "barrier block");
  if (smem - smem_raw > C::kAlignPadDkdv) {  // uniform over the CTA: nothing has been set up yet
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, kStatusSmemLayout);
    if (first_cta) grid_dependency_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // The TMA producer thread initialises the barriers itself and issues the loads of K, V and of the first
  // Q / statistics / dO tiles BEFORE the CTA-wide synchronisation, so that their latency overlaps the TMEM
  // allocation.
  WaitCtx ctx{&bars->abort_flag, p.status};
  auto load_q_do = [&](int it) -> bool {
    const int sq_ = it % C::kStagesQ, sd = it % C::kStagesDO, ss = it & 1;
    const uint32_t phq = (it / C::kStagesQ) & 1, phd = (it / C::kStagesDO) & 1, phs = (it >> 1) & 1;
    const int head = head_k * group + it / per_head;
    const int i = i_min + it % per_head;
    const int qrow = q_off + i * kBlock;
    const int64_t stat = (static_cast<int64_t>(batch) * p.h + head) * p.sq_pad + i * kBlock;
    if (!mbar_wait(&bars->a_empty[sq_], phq ^ 1, ctx)) return false;
    mbar_arrive_expect_tx(&bars->a_full[sq_], C::kTileBytes);
#pragma unroll
    for (int c = 0; c < C::kChunks; ++c)
      tma_load_4d(sQ + sq_ * C::kTileBytes + c * C::kChunkBytes, &p.tm_q, &bars->a_full[sq_], c * 64, head, qrow, 0);
    if (!mbar_wait(&bars->st_empty[ss], phs ^ 1, ctx)) return false;
    mbar_arrive_expect_tx(&bars->st_full[ss], 1024);
    bulk_load_1d(sStats + ss * 256, p.lse2 + stat, 512, &bars->st_full[ss]);
    bulk_load_1d(sStats + ss * 256 + 128, p.delta + stat, 512, &bars->st_full[ss]);
    if (!mbar_wait(&bars->b_empty[sd], phd ^ 1, ctx)) return false;
    mbar_arrive_expect_tx(&bars->b_full[sd], C::kTileBytes);
#pragma unroll
    for (int c = 0; c < C::kChunks; ++c)
      tma_load_4d(sdO + sd * C::kTileBytes + c * C::kChunkBytes, &p.tm_do, &bars->b_full[sd], c * 64, head, qrow, 0);
    return true;
  };
  const int n_early = min(n_it, 2);  // stages that are free from the start: no wait blocks
  if (warp == kProducerWarp && lane == 0) {
    init_barriers(bars, C::kStagesQ, 2, 2);
    if (n_it > 0) {
      mbar_arrive_expect_tx(&bars->fixed_full, 2 * C::kTileBytes);
#pragma unroll
      for (int c = 0; c < C::kChunks; ++c) {
        tma_load_4d(sK + c * C::kChunkBytes, &p.tm_k, &bars->fixed_full, c * 64, head_k, k_off + key0, 0);
        tma_load_4d(sV + c * C::kChunkBytes, &p.tm_v, &bars->fixed_full, c * 64, head_k, k_off + key0, 0);
      }
      for (int it = 0; it < n_early; ++it) load_q_do(it);
    }
  }
  if (warp == kMmaWarp) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  const bool stop = __syncthreads_or(stop_probe) != 0;  // sticky time-out bit set: the CTA does no work
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  if (stop && threadIdx.x == 0) bars->abort_flag = 1;  // the common exit then lets the loads issued above land

  // the last Q / dO tile of a packed sequence holds rows of the next sequence (see zero_tile_rows_from)
  const bool fix_q_tail = (sq % kBlock) != 0 && n_it > 0;
  const int q_tail_rows = sq - (nq - 1) * kBlock;  // valid rows of the last Q tile
  if (stop) {
  } else if (warp == kProducerWarp) {
    if (!fix_q_tail) {
      if (lane == 0) {
        for (int it = n_early; it < n_it; ++it)
          if (!load_q_do(it)) break;
      }
    } else {
      // the whole warp walks the tiles: lane 0 issues the loads, all lanes zero the tails
      for (int it = 0; it < n_it; ++it) {
        bool loaded = true;
        if (lane == 0 && it >= n_early) loaded = load_q_do(it);
        if (!__shfl_sync(0xffffffffu, loaded, 0)) break;
        if (it % per_head == per_head - 1) {  // the last Q tile of this head
          const int sq_ = it % C::kStagesQ, sd = it % C::kStagesDO;
          if (!mbar_wait_warp(&bars->a_full[sq_], (it / C::kStagesQ) & 1, ctx)) break;
          if (!mbar_wait_warp(&bars->b_full[sd], (it / C::kStagesDO) & 1, ctx)) break;
          zero_tile_rows_from<D>(sQ + sq_ * C::kTileBytes, q_tail_rows, lane);
          zero_tile_rows_from<D>(sdO + sd * C::kTileBytes, q_tail_rows, lane);
          if (lane == 0) mbar_arrive(&bars->tail_fixed[sd]);
        }
      }
    }
  } else if (warp == kMmaWarp) {
    if (elect_one() && n_it > 0) {
      constexpr uint32_t idesc_nn = make_idesc_f16(128, kBlock, false, false);
      const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV);
      // One accumulator region A holds S^T(it) and then dP^T(it): dP^T(it) is issued as soon as S^T(it)
      // sits in registers, S^T(it+1) as soon as dP^T(it) does.  The hooks wait for the TMA load the next
      // product reads.
      auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity, ctx); };
      auto q_tile = [&](int it) { return smem_u32(sQ + (it % C::kStagesQ) * C::kTileBytes); };
      auto do_tile = [&](int it) { return smem_u32(sdO + (it % C::kStagesDO) * C::kTileBytes); };
      auto q_full = [&](int it) { return wait(&bars->a_full[it % C::kStagesQ], (it / C::kStagesQ) & 1); };
      auto do_full = [&](int it) { return wait(&bars->b_full[it % C::kStagesDO], (it / C::kStagesDO) & 1); };
      const uint32_t tA = tmem_base + kColS;
      bool ok = wait(&bars->fixed_full, 0) && q_full(0);
      for (int it = 0; ok && it < n_it; ++it) {
        // region A is free once its last content, dP^T(it-1), was read
        if (it > 0 && !(ok = wait(&bars->dp_loaded, (it - 1) & 1))) break;
        tc_fence_after_sync();
        ok = gemm_ss<D>(tA, k_addr, q_tile(it), idesc_nn, [&] { return do_full(it); });  // S^T(it) = K Q^T
        if (!ok) break;
        tc_commit(&bars->s_full);
        tc_commit(&bars->a_empty[it % C::kStagesQ]);  // second reader: the dK MMAs of this tile
        if (!(ok = wait(&bars->s_loaded, it & 1))) break;  // ... and for dP^T(it) once S^T(it) was
        tc_fence_after_sync();
        ok = gemm_ss<D>(tA, v_addr, do_tile(it), idesc_nn,  // dP^T(it) = V dO^T
                        [&] { return it + 1 >= n_it || q_full(it + 1); });
        if (!ok) break;
        tc_commit(&bars->dp_full);
        tc_commit(&bars->b_empty[it % C::kStagesDO]);  // second reader: the dV MMAs of this tile
      }
    }
  } else if (warp == kAccMmaWarp) {
    if (elect_one() && n_it > 0) {
      // dV += P^T(it) dO(it) as soon as the packed P^T is written, dK += dS^T(it) Q(it) likewise.
      constexpr uint32_t idesc_acc = make_idesc_f16(128, D, false, true);
      const uint32_t tP = tmem_base + kColDP, tDS = tmem_base + kColDP + 64;
      const uint32_t tDV = tmem_base + kColAcc, tDK = tmem_base + kColAcc + D;
      bool ok = true;
      uint32_t tail_phase = 0;  // bit sd: parity of the next tail_fixed[sd] phase to wait for
      for (int it = 0; ok && it < n_it; ++it) {
        const int sq_ = it % C::kStagesQ, sd = it % C::kStagesDO;
        if (!(ok = mbar_wait(&bars->b_full[sd], (it / C::kStagesDO) & 1, ctx))) break;
        if (!(ok = mbar_wait(&bars->p_full, it & 1, ctx))) break;
        if (fix_q_tail && it % per_head == per_head - 1) {
          if (!(ok = mbar_wait(&bars->tail_fixed[sd], (tail_phase >> sd) & 1, ctx))) break;
          tail_phase ^= 1u << sd;
        }
        tc_fence_after_sync();
        gemm_ts<D>(tDV, tP, smem_u32(sdO + sd * C::kTileBytes), idesc_acc, it == 0);
        tc_commit(&bars->b_empty[sd]);
        tc_commit(&bars->p_free);
        if (!(ok = mbar_wait(&bars->a_full[sq_], (it / C::kStagesQ) & 1, ctx))) break;
        if (!(ok = mbar_wait(&bars->ds_full, it & 1, ctx))) break;
        tc_fence_after_sync();
        gemm_ts<D>(tDK, tDS, smem_u32(sQ + sq_ * C::kTileBytes), idesc_acc, it == 0);
        tc_commit(&bars->a_empty[sq_]);
        tc_commit(&bars->ds_free[0]);
      }
      if (ok) tc_commit(&bars->acc_full);
    }
  } else {
    // ---- elementwise warps: thread = (key row, 32-query-column quarter) ----
    const int cq = warp >> 2, quarter = warp & 3;
    const int row_in_tile = quarter * 32 + lane;
    const int key = key0 + row_in_tile;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tA = tmem_base + lane_base + kColS + cq * 32;         // S^T, then dP^T
    const uint32_t tP = tmem_base + lane_base + kColDP + cq * 16;        // packed P^T
    const float c = p.scale_log2;
    const float2 c2 = make_float2(c, c);
    // causal: query column q of tile i is masked for this key when key > q + sk - sq, i.e. the columns of
    // this thread's quarter below  key - (sk - sq) - (i * 128 + cq * 32)  are masked
    const int cmin0 = p.is_causal ? key - shift - (i_min * kBlock + cq * 32) : 0;
    const float* stats = sStats + cq * 32;
    const int cmax_last = fix_q_tail ? max(0, min(32, q_tail_rows - cq * 32)) : 32;  // valid columns in the last Q tile
    int i_rel = 0;  // Q tile within the current head
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int ss = it & 1;
      if (!(ok = mbar_wait_warp(&bars->st_full[ss], (it >> 1) & 1, ctx))) break;
      // The LSE of this thread's 32 query columns is fetched while the warp waits for S^T anyway.  Read after the wait,
      // these shared-memory loads compete with the operand fetches of the dP^T MMAs, which take the whole shared-memory
      // bandwidth (measured: 4.5-7 % of the kernel).
      const float4* st_lse = reinterpret_cast<const float4*>(stats + ss * 256);
      const float4* st_delta = reinterpret_cast<const float4*>(stats + ss * 256 + 128);
      float4 lse_q[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) lse_q[e] = st_lse[e];
      if (!(ok = mbar_wait_warp(&bars->s_full, it & 1, ctx))) break;
      tc_fence_after_sync();
      uint32_t sr[32];
      tmem_ld32(tA, sr);
      tmem_wait_ld();
      warp_arrive_loaded(&bars->s_loaded, lane);  // region A may now receive dP^T
      // 1650 -> 1600 us for 16 packed documents (Hq32 Hkv8); nothing in the dense kernel, where the other products of the
      // pipe are in the way of the earlier dP^T
      schedule_barrier(lane);
      // columns below cmin are masked by causality; columns from cmax on are query rows past the end of the
      // sequence (last Q tile of a packed sequence).  Both clamped to [0, 32] and packed into one register.
      const int cmask = max(0, min(32, cmin0 - i_rel * kBlock)) |
                        ((i_rel == per_head - 1 ? cmax_last : 32) << 8);
      const bool col_masked = cmask != (32 << 8);
      if (++i_rel == per_head) i_rel = 0;
      float2 pr[16];
      uint32_t pk[16];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 l = lse_q[e];
        pr[2 * e] = exp2_pair(ffma2(make_float2(__uint_as_float(sr[4 * e]), __uint_as_float(sr[4 * e + 1])), c2,
                                    make_float2(l.x, l.y)));
        pr[2 * e + 1] = exp2_pair(ffma2(make_float2(__uint_as_float(sr[4 * e + 2]), __uint_as_float(sr[4 * e + 3])),
                                        c2, make_float2(l.z, l.w)));
      }
      if (col_masked) {
        const int cmin = cmask & 0xff, cmax = cmask >> 8;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (2 * e < cmin || 2 * e >= cmax) pr[e].x = 0.f;
          if (2 * e + 1 < cmin || 2 * e + 1 >= cmax) pr[e].y = 0.f;
        }
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) pk[e] = pack_half2(pr[e].x, pr[e].y);
      // the dV MMAs of the previous tile must have consumed the old P^T before it is overwritten
      if (it > 0 && !(ok = mbar_wait_warp(&bars->p_free, (it - 1) & 1, ctx))) break;
      tmem_st16(tP, pk);
      warp_arrive(&bars->p_full, lane);

      if (!(ok = mbar_wait_warp(&bars->dp_full, it & 1, ctx))) break;
      tc_fence_after_sync();
      tmem_ld32(tA, sr);
      tmem_wait_ld();
      warp_arrive_loaded(&bars->dp_loaded, lane);  // region A may now receive the next S^T
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 dl = st_delta[e];
        const float2 d0 = fmul2(pr[2 * e], fadd2(make_float2(__uint_as_float(sr[4 * e]), __uint_as_float(sr[4 * e + 1])),
                                                 make_float2(dl.x, dl.y)));
        const float2 d1 = fmul2(pr[2 * e + 1], fadd2(make_float2(__uint_as_float(sr[4 * e + 2]), __uint_as_float(sr[4 * e + 3])),
                                                     make_float2(dl.z, dl.w)));
        pk[2 * e] = pack_half2(d0.x, d0.y);
        pk[2 * e + 1] = pack_half2(d1.x, d1.y);
      }
      if (col_masked) {  // by selection: dP^T of a masked column may be NaN/Inf (dO rows of the next sequence)
        const int cmin = cmask & 0xff, cmax = cmask >> 8;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (2 * e < cmin || 2 * e >= cmax) pk[e] &= 0xffff0000u;
          if (2 * e + 1 < cmin || 2 * e + 1 >= cmax) pk[e] &= 0x0000ffffu;
        }
      }
      // the statistics of this tile are in use no longer
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->st_empty[ss]);
      if (it > 0 && !(ok = mbar_wait_warp(&bars->ds_free[0], (it - 1) & 1, ctx))) break;
      tmem_st16(tP + 64, pk);  // packed dS^T
      warp_arrive(&bars->ds_full, lane);
    }
    // ---- epilogue: column quarters 0,1 store the halves of dV, quarters 2,3 the halves of dK * scale ----
    const int which = cq >> 1;        // 0 = dV, 1 = dK
    const int col_half = cq & 1;      // which D/2 columns
    __half* dst_base = (which == 0) ? p.dv : p.dk;
    const int64_t rs = (which == 0) ? p.dv_row_stride : p.dk_row_stride;
    const int64_t hs = (which == 0) ? p.dv_head_stride : p.dk_head_stride;
    __half* dst = dst_base + static_cast<int64_t>(k_off + key) * rs + head_k * hs + col_half * (D / 2);
    const float mul = (which == 0) ? 1.f : p.scale;
    if (ok && n_it > 0) ok = mbar_wait_warp(&bars->acc_full, 0, ctx);
    if (ok) {
      if (n_it > 0) {
        tc_fence_after_sync();
#pragma unroll
        for (int q = 0; q < D / 64; ++q) {
          uint32_t r[32];
          tmem_ld32(tmem_base + lane_base + kColAcc + which * D + col_half * (D / 2) + q * 32, r);
          tmem_wait_ld();
          store_scaled_rows(dst - lane * rs + q * 32, rs, sk - (key - lane), r, mul, lane);
        }
      } else if (key < sk) {
        const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i3 = 0; i3 < D / 16; ++i3) *reinterpret_cast<uint4*>(dst + i3 * 8) = z;
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (bars->abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
  if (first_cta && threadIdx.x == 0) grid_dependency_wait();  // as in bwd_dkdv_kernel
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

int round_up(int x, int m) { return (x + m - 1) / m * m; }

size_t stats_floats(const FaBwdParams* p) {
  return static_cast<size_t>(p->b) * p->h * round_up(p->seqlen_q, kBlock);
}

// Whether dK or dV lies over K or V, by the first and last bytes of the tensors (so interleaved tensors count as well).
bool gradients_over_keys(const FaBwdParams* p) {
  const bool varlen = p->cu_seqlens_q != nullptr;
  const int64_t rows = varlen ? p->total_k : p->seqlen_k, batches = varlen ? 1 : p->b;
  struct Span {
    intptr_t first, last;
  };
  auto span = [&](const void* base, int64_t batch_stride, int64_t row_stride, int64_t head_stride) {
    const int64_t ends[] = {(batches - 1) * batch_stride, (rows - 1) * row_stride, (p->h_k - 1) * head_stride};
    int64_t low = 0, high = p->d;
    for (int64_t e : ends) low += std::min<int64_t>(e, 0), high += std::max<int64_t>(e, 0);
    const intptr_t b = reinterpret_cast<intptr_t>(base);
    return Span{b + 2 * low, b + 2 * high};
  };
  const Span in[] = {span(p->k, p->k_batch_stride, p->k_row_stride, p->k_head_stride),
                     span(p->v, p->v_batch_stride, p->v_row_stride, p->v_head_stride)};
  const Span out[] = {span(p->dk, p->dk_batch_stride, p->dk_row_stride, p->dk_head_stride),
                      span(p->dv, p->dv_batch_stride, p->dv_row_stride, p->dv_head_stride)};
  for (const Span& x : in)
    for (const Span& y : out)
      if (x.first < y.last && y.first < x.last) return true;
  return false;
}

template <int D>
int launch_bwd(const BwdKernelParams& kp, const FaBwdParams* p, int stage_mask, cudaStream_t stream) {
  using C = BCfg<D>;
  static bool configured[64] = {};
  int dev = 0;
  FA_CHECK_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    FA_CHECK_CUDA(cudaFuncSetAttribute(bwd_dkdv_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytesDkdv));
    FA_CHECK_CUDA(cudaFuncSetAttribute(bwd_dkdv_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytesDkdv));
    if constexpr (D == 128)
      FA_CHECK_CUDA(cudaFuncSetAttribute(bwd_dkdv_packed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytesDkdv));
    configured[dev & 63] = true;
  }
  if (stage_mask & 2) {
    static bool configured_p[64] = {};
    if (!configured_p[dev & 63]) {
      FA_CHECK_CUDA(cudaFuncSetAttribute(bwd_dq_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         C::kSmemBytesDq + 1024));
      configured_p[dev & 63] = true;
    }
    BwdKernelParams kq = kp;
    const int sms = device_sm_count();
    kq.sched = next_sched_slot(stream);
    if (sms <= 0 || kq.sched == nullptr) return set_error(FA_ERR_CUDA, "fa_bwd: device attributes not available");
    kq.items_x = (p->seqlen_q + kBlock - 1) / kBlock;
    kq.b = p->b;
    const int64_t total = kq.cu_seqlens_q ? static_cast<int64_t>(p->h) * (p->total_q / kBlock + p->b)
                                          : static_cast<int64_t>(kq.items_x) * p->h * p->b;
    FA_CHECK_ARG(total < (1ll << 30), "fa_bwd: too many work items");
    kq.total_items = static_cast<int>(total);
    kq.section_rows = section_rows(p->is_causal != 0, p->seqlen_q, p->seqlen_k, 4 * D);
    const int grid = kq.total_items < sms ? kq.total_items : sms;
    if (stage_mask & 1) {
      FA_CHECK_CUDA(launch_overlapped(bwd_dq_kernel<D>, dim3(grid), kDqThreads, C::kSmemBytesDq + 1024, stream, kq));
    } else {
      bwd_dq_kernel<D><<<grid, kDqThreads, C::kSmemBytesDq + 1024, stream>>>(kq);
      FA_CHECK_CUDA(cudaGetLastError());
    }
  }
  if (stage_mask & 4) {
    // The dK/dV kernel reads nothing that the dQ kernel writes.  It starts on the SMs that the dQ kernel leaves idle (fewer
    // items than SMs, the last wave) and ends after it: every CTA of the dQ kernel lets it go only when the preprocess
    // kernel has finished, and its CTA 0 waits for the dQ kernel before it exits.  Whole backward, three launches in turn
    // against overlapped: B3 S197 H12 D64 28.3 -> 17.0 us, B2 S512 H8 D64 32.4 -> 17.7, B1 S1000 H16 D128 causal
    // 49.5 -> 43.6, B2 S2047 Hq16 Hkv4 D128 causal 195 -> 182, B16 S1024 H32 805 -> 786, B4 S8192 H32 7317 -> 7135.
    // dK and dV may be written over K and V (a CTA reads its own tile before it writes it): then the dQ kernel, which reads
    // K and V too, has to be over first.
    const bool overlap = (stage_mask & 2) != 0 && !gradients_over_keys(p);
    const int rows = section_rows(p->is_causal != 0, p->seqlen_q, p->seqlen_k, static_cast<int64_t>(4 * D) * kp.group);
    if (D == 128 && kp.cu_seqlens_q != nullptr && p->h != p->h_k) {  // one CTA per key tile: see bwd_dkdv_packed_kernel
      if constexpr (D == 128) {
        BwdKernelParams kk = kp;
        // Sections as elsewhere, but of eight heads at least: 18 CTAs to a head still read its rows together, and fewer heads leave the
        // heaviest items of the last ones for the end.  All heads of a sequence at once, sections of the common rule, these (us, causal): 4 x
        // 8000-16384 Hkv4 (group 4) 4567 : 4770 : 4576; 30000 Hkv16 13528 : 13067 : 13254; without the mask all heads at once read from
        // memory what a head by itself reads from L2: 30000 Hkv16 29832 : 25804, 2 x 8192 Hkv32 8690 : 7835.
        kk.section_rows = rows == 0 ? 0 : std::max(rows, 8 * p->seqlen_q);
        dim3 grid_k((p->seqlen_k + kBlock - 1) / kBlock * p->h_k, 1, p->b);
        if (overlap) {
          FA_CHECK_CUDA(launch_overlapped(bwd_dkdv_packed_kernel, grid_k, kNumThreads, C::kSmemBytesDkdv, stream, kk));
        } else {
          bwd_dkdv_packed_kernel<<<grid_k, kNumThreads, C::kSmemBytesDkdv, stream>>>(kk);
        }
      }
    } else {
      BwdKernelParams kk = kp;
      const int sms = device_sm_count();
      kk.sched = next_sched_slot(stream);
      if (sms <= 0 || kk.sched == nullptr) return set_error(FA_ERR_CUDA, "fa_bwd: device attributes not available");
      kk.items_x = (p->seqlen_k + kBlock - 1) / kBlock;
      kk.b = p->b;
      const int64_t total = kk.cu_seqlens_k ? static_cast<int64_t>(p->h_k) * (p->total_k / kBlock + p->b)
                                            : static_cast<int64_t>(kk.items_x) * p->h_k * p->b;
      FA_CHECK_ARG(total < (1ll << 30), "fa_bwd: too many work items");
      kk.total_items = static_cast<int>(total);
      kk.section_rows = rows;
      const int grid = kk.total_items < sms ? kk.total_items : sms;
      const auto kernel = kk.cu_seqlens_q ? bwd_dkdv_kernel<D, true> : bwd_dkdv_kernel<D, false>;
      if (overlap) {
        FA_CHECK_CUDA(launch_overlapped(kernel, dim3(grid), kDkvThreads, C::kSmemBytesDkdv, stream, kk));
      } else {
        kernel<<<grid, kDkvThreads, C::kSmemBytesDkdv, stream>>>(kk);
      }
    }
    FA_CHECK_CUDA(cudaGetLastError());
  }
  return FA_OK;
}

}  // namespace
}  // namespace fa

namespace fa {
namespace {
// rows per head of the fp32 dQ accumulator of the single-kernel path (whole 128-row tiles per sequence)
int64_t dq_acc_rows(const FaBwdParams* p) {
  if (p->cu_seqlens_q != nullptr) return ((static_cast<int64_t>(p->total_q) + kBlock - 1) / kBlock + p->b) * kBlock;
  return static_cast<int64_t>(p->b) * round_up(p->seqlen_q, kBlock);
}
size_t stats_bytes(const FaBwdParams* p) { return (2 * stats_floats(p) * sizeof(float) + 255) / 256 * 256; }
}  // namespace
}  // namespace fa

extern "C" size_t fa_bwd_workspace_bytes(const FaBwdParams* p) {
  if (p == nullptr || p->b < 1 || p->h < 1 || p->seqlen_q < 1) return 0;
  if ((p->flags & FA_BWD_SINGLE_KERNEL) == 0) return 2 * fa::stats_floats(p) * sizeof(float);
  return fa::stats_bytes(p) + static_cast<size_t>(fa::dq_acc_rows(p)) * p->h * p->d * sizeof(float);
}

extern "C" int fa_bwd(const FaBwdParams* p, fa_stream_t stream) { return fa_bwd_stages(p, 7, stream); }

extern "C" int fa_bwd_stages(const FaBwdParams* p, int stage_mask, fa_stream_t stream_) {
  using namespace fa;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  FA_CHECK_ARG(p != nullptr, "fa_bwd: params is NULL");
  FA_CHECK_ARG(p->q && p->k && p->v && p->o && p->dout && p->lse && p->dq && p->dk && p->dv,
               "fa_bwd: q, k, v, o, dout, lse, dq, dk, dv must be non-NULL");
  if (p->d != 64 && p->d != 128) return set_error(FA_ERR_UNSUPPORTED, "fa_bwd: head_dim must be 64 or 128");
  FA_CHECK_ARG(p->b >= 1 && p->h >= 1 && p->h_k >= 1 && p->h % p->h_k == 0, "fa_bwd: bad b / h / h_k");
  FA_CHECK_ARG(p->seqlen_q >= 1 && p->seqlen_k >= 1, "fa_bwd: bad sequence lengths");
  FA_CHECK_ARG((p->cu_seqlens_q == nullptr) == (p->cu_seqlens_k == nullptr),
               "fa_bwd: cu_seqlens_q and cu_seqlens_k go together");
  FA_CHECK_ARG(p->lse_row_stride >= p->seqlen_q, "fa_bwd: lse_row_stride is smaller than seqlen_q");
  FA_CHECK_ARG(p->is_causal >= 0 && p->is_causal <= 2, "fa_bwd: is_causal must be 0, 1 or FA_CAUSAL_SHIFT");
  FA_CHECK_ARG(p->is_causal != 2 || p->cu_seqlens_q == nullptr, "fa_bwd: FA_CAUSAL_SHIFT is for dense q / k / v only");
  const bool varlen = p->cu_seqlens_q != nullptr;
  {
    const void* ptrs[] = {p->o, p->dout, p->dq, p->dk, p->dv};
    for (const void* x : ptrs) FA_CHECK_ARG(aligned16(x), "fa_bwd: o, dout, dq, dk, dv must be 16-byte aligned");
    const int64_t strides[] = {p->o_row_stride,  p->o_head_stride,  p->do_row_stride, p->do_head_stride,
                               p->dq_row_stride, p->dq_head_stride, p->dk_row_stride, p->dk_head_stride,
                               p->dv_row_stride, p->dv_head_stride};
    for (int64_t s : strides) FA_CHECK_ARG(s % 8 == 0, "fa_bwd: strides must be multiples of 8 elements");
    if (!varlen) {
      const int64_t bs[] = {p->o_batch_stride, p->do_batch_stride, p->dq_batch_stride, p->dk_batch_stride,
                            p->dv_batch_stride};
      for (int64_t s : bs) FA_CHECK_ARG(s % 8 == 0, "fa_bwd: batch strides must be multiples of 8 elements");
    }
  }
  const size_t need = fa_bwd_workspace_bytes(p);
  if (p->workspace == nullptr || p->workspace_bytes < need)
    return set_error(FA_ERR_WORKSPACE, "fa_bwd: workspace smaller than fa_bwd_workspace_bytes()");
  FA_CHECK_ARG((reinterpret_cast<uintptr_t>(p->workspace) & 255) == 0, "fa_bwd: workspace must be 256-byte aligned");
  int rc = check_device_sm100();
  if (rc != FA_OK) return rc;

  const int sq_pad = round_up(p->seqlen_q, kBlock);
  float* delta = static_cast<float*>(p->workspace);
  float* lse2 = delta + stats_floats(p);

  PreParams pp;
  pp.o = static_cast<const __half*>(p->o);
  pp.dout = static_cast<const __half*>(p->dout);
  pp.lse = p->lse;
  pp.delta = delta;
  pp.lse2 = lse2;
  pp.o_batch_stride = p->o_batch_stride; pp.o_row_stride = p->o_row_stride; pp.o_head_stride = p->o_head_stride;
  pp.do_batch_stride = p->do_batch_stride; pp.do_row_stride = p->do_row_stride; pp.do_head_stride = p->do_head_stride;
  pp.lse_row_stride = p->lse_row_stride;
  pp.h = p->h; pp.seqlen_q = p->seqlen_q; pp.sq_pad = sq_pad; pp.d = p->d;
  pp.cu_seqlens_q = p->cu_seqlens_q;
  const bool clears = varlen && (p->flags & FA_BWD_ZERO_UNUSED_ROWS) != 0;
  pp.clear[0] = PackedRows{clears ? static_cast<__half*>(p->dq) : nullptr, p->dq_row_stride, p->dq_head_stride, p->total_q,
                           p->h, p->d, p->cu_seqlens_q, p->b};
  pp.clear[1] = PackedRows{static_cast<__half*>(p->dk), p->dk_row_stride, p->dk_head_stride, p->total_k,
                           p->h_k, p->d, p->cu_seqlens_k, p->b};
  pp.clear[2] = PackedRows{static_cast<__half*>(p->dv), p->dv_row_stride, p->dv_head_stride, p->total_k,
                           p->h_k, p->d, p->cu_seqlens_k, p->b};
  pp.keys_written = round_up(p->seqlen_k, kBlock);
  pp.status = device_status_ptr();
  const int64_t pre_items = static_cast<int64_t>((sq_pad + kPreRows - 1) / kPreRows) * p->h;
  const int items_per_block = 256 / (p->d / 8);
  int64_t pre_blocks = (pre_items + items_per_block - 1) / items_per_block;
  if (clears) {  // at least a block per SM for the unused rows; blocks past the last item do nothing else
    const int sms = device_sm_count();
    if (sms <= 0) return set_error(FA_ERR_CUDA, "fa_bwd: device attributes not available");
    pre_blocks = std::max<int64_t>(pre_blocks, (sms + p->b - 1) / p->b);
  }
  dim3 grid_pre(static_cast<unsigned>(pre_blocks), 1, p->b);
  if (stage_mask & 1) {
    const auto preprocess = clears ? bwd_preprocess_kernel<true> : bwd_preprocess_kernel<false>;
    preprocess<<<grid_pre, 256, 0, stream>>>(pp);
    FA_CHECK_CUDA(cudaGetLastError());
  }
  const bool fused = (p->flags & FA_BWD_SINGLE_KERNEL) != 0;
  float* dq_acc = fused ? reinterpret_cast<float*>(static_cast<uint8_t*>(p->workspace) + stats_bytes(p)) : nullptr;
  if (fused && (stage_mask & 1)) {
    // the accumulator starts at zero; the pairs of the single kernel add their dQ partials into it
    FA_CHECK_CUDA(cudaMemsetAsync(dq_acc, 0, static_cast<size_t>(dq_acc_rows(p)) * p->h * p->d * sizeof(float), stream));
  }

  BwdKernelParams kp;
  const int64_t q_rows = varlen ? p->total_q : p->seqlen_q;
  const int64_t k_rows = varlen ? p->total_k : p->seqlen_k;
  const int64_t nb = varlen ? 1 : p->b;
  FA_CHECK_ARG(q_rows >= 1 && k_rows >= 1, "fa_bwd: empty q or k");
  rc = make_tensor_map_4d(&kp.tm_q, p->q, p->d, p->h, q_rows, nb, p->q_head_stride, p->q_row_stride,
                          p->q_batch_stride, kBlock, "fa_bwd: q");
  if (rc != FA_OK) return rc;
  rc = make_tensor_map_4d(&kp.tm_do, p->dout, p->d, p->h, q_rows, nb, p->do_head_stride, p->do_row_stride,
                          p->do_batch_stride, kBlock, "fa_bwd: dout");
  if (rc != FA_OK) return rc;
  rc = make_tensor_map_4d(&kp.tm_k, p->k, p->d, p->h_k, k_rows, nb, p->k_head_stride, p->k_row_stride,
                          p->k_batch_stride, kBlock, "fa_bwd: k");
  if (rc != FA_OK) return rc;
  rc = make_tensor_map_4d(&kp.tm_v, p->v, p->d, p->h_k, k_rows, nb, p->v_head_stride, p->v_row_stride,
                          p->v_batch_stride, kBlock, "fa_bwd: v");
  if (rc != FA_OK) return rc;
  kp.dq = static_cast<__half*>(p->dq);
  kp.dk = static_cast<__half*>(p->dk);
  kp.dv = static_cast<__half*>(p->dv);
  kp.dq_batch_stride = p->dq_batch_stride; kp.dq_row_stride = p->dq_row_stride; kp.dq_head_stride = p->dq_head_stride;
  kp.dk_batch_stride = p->dk_batch_stride; kp.dk_row_stride = p->dk_row_stride; kp.dk_head_stride = p->dk_head_stride;
  kp.dv_batch_stride = p->dv_batch_stride; kp.dv_row_stride = p->dv_row_stride; kp.dv_head_stride = p->dv_head_stride;
  kp.delta = delta;
  kp.lse2 = lse2;
  kp.sq_pad = sq_pad;
  kp.seqlen_q = p->seqlen_q; kp.seqlen_k = p->seqlen_k; kp.h = p->h; kp.h_k = p->h_k;
  kp.group = p->h / p->h_k;
  kp.scale = p->softmax_scale;
  kp.scale_log2 = p->softmax_scale * kLog2e;
  kp.is_causal = p->is_causal;
  kp.causal_shift = p->causal_shift;
  kp.cu_seqlens_q = p->cu_seqlens_q;
  kp.cu_seqlens_k = p->cu_seqlens_k;
  kp.status = device_status_ptr();
  kp.dq_acc = dq_acc;
  kp.dq_acc_rows = fused ? dq_acc_rows(p) : 0;
  kp.total_q = p->total_q;
  kp.sched = nullptr;  // set per launch of the dQ kernel
  kp.items_x = 0;
  kp.total_items = 0;
  kp.b = p->b;
  if (fused) {
    if (stage_mask & 2) {
      rc = launch_bwd_fused(kp, p, stream);
      if (rc != FA_OK) return rc;
    }
    if (stage_mask & 4) return launch_bwd_dq_finalize(kp, p, stream);
    return FA_OK;
  }
  if (p->d == 128) return launch_bwd<128>(kp, p, stage_mask, stream);
  return launch_bwd<64>(kp, p, stage_mask, stream);
}
