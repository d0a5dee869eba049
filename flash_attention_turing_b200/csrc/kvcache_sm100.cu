// KV-cache step for sm_100a: in-place append of the new tokens, split-KV attention of a few query
// rows against a contiguous or paged cache, and the log-sum-exp merge of the splits.
//
// The attend kernel is HBM-bound (every cached K and V byte is read exactly once per KV head; the
// query heads of a GQA group share the read), so it is built around the memory system:
//   * one CTA per (split, KV head, sequence), or for num_splits = 0, where that is faster, per even share of the batch
//     (decode_balanced_kernel, see uses_balanced_kernel()); a producer warp streams 64-token K and V tiles with
//     TMA (16-byte aligned bulk copies, 128-byte swizzle, no multicast) through a ring of
//     mbarrier-guarded stages, pages looked up in block_table per tile;
//   * four consumer warps each take 16 tokens of every tile: S = Q K^T and O += P V run on
//     mma.sync.m16n8k16 with ldmatrix from the swizzled tiles -- the up to 16 (query position, head
//     of the group) rows form the M dimension, so the tensor work is negligible and no CUDA-core
//     dot products or shuffle reductions sit on the critical path;
//   * online softmax in registers with a lazily updated reference maximum; the four warps merge
//     their (m, l, O) through shared memory at the end.
// Algorithmic bytes per (sequence, KV head): 2 * L * D * 2 (K and V rows) + q/out rows.
//
// Replaces paged_append_kernel, kvcache_decode_split_kernel, kvcache_split_kernel and
// kvcache_split_kernel_legacy of the reference (csrc/flash_attn/src/kvcache_native.cu:148-871),
// the contiguous append loop of mha_fwd_kvcache (csrc/flash_attn/flash_api.cpp:643-654) and the
// split heuristic choose_num_splits (kvcache_native.cu:913-952).  Query blocks with more than 16
// (position, head) rows per KV head go to the tiled tcgen05 forward kernel instead (the reference
// routes them to its tiled kernel too, flash_api.cpp:668-714).
#include <algorithm>
#include <mutex>

#include "combine.h"
#include "fwd.h"
#define FA_WAIT_INLINE  // two roles with a few waits each: code size is no concern here
#include "ptx.cuh"

namespace fa {
namespace {

constexpr int kTileTokens = 64;
constexpr int kConsumerWarps = 4;
constexpr int kDecodeThreads = (kConsumerWarps + 1) * 32;
constexpr int kMaxRows = 16;  // M of the mma: (query position, head in group) pairs
constexpr int kBalancedRows = 8;  // of them used by the balanced kernel at most, see uses_balanced_kernel()

struct DecodeParams {
  CUtensorMap tm_k;
  CUtensorMap tm_v;
  const __half* q;
  __half* o;        // final output (num_splits == 1)
  float* lse;       // final LSE (num_splits == 1)
  float* o_accum;   // (splits, rows_total, D) partials (num_splits > 1)
  float* lse_accum; // (splits, rows_total)
  int64_t q_batch_stride, q_row_stride, q_head_stride;
  int64_t o_batch_stride, o_row_stride, o_head_stride;
  int seqlen_q, seqlen_new, h, h_k, group;
  int64_t rows_total;  // b * h * seqlen_q
  float scale_log2;
  int is_causal;
  const int* cache_seqlens;
  const int* cache_batch_idx;
  const int* block_table;
  int64_t block_table_batch_stride;
  int page_size;     // tokens per page (paged) or capacity per cache row (contiguous)
  int capacity;      // tokens a sequence can hold: max_blocks_per_seq * page_size, or the cache row length
  int num_splits;    // grid.x
  int checked;       // the host refuses lengths beyond the capacity: neither read nor reported
  int chunk_tiles;   // split kernel: > 0: split s owns tiles [s*chunk, (s+1)*chunk); 0: proportional ranges
  int b;             // sequences
  int* arrivals;     // balanced kernel: a counter per CTA in scratch memory, zeroed by the kernel before
  int* status;
};

template <int D>
struct DCfg {
  static constexpr int kChunks = D / 64;
  static constexpr int kChunkBytes = kTileTokens * 128;     // 64 tokens x 128 B
  static constexpr int kTileBytes = kChunks * kChunkBytes;  // one K or V tile
  static constexpr int kStages = (D == 128) ? 3 : 6;
  static constexpr int kStageBytes = 2 * kTileBytes;
  static constexpr int kMergeBytes = kConsumerWarps * kMaxRows * (D + 2) * 4;
  static constexpr int kSmemBytes = kStages * kStageBytes + 2048 /*barriers, (m, l)*/ + 1024 /*align*/;
  static_assert(kMergeBytes <= kStages * kStageBytes, "merge buffer aliases the stage ring");
  static_assert(kConsumerWarps * 16 * D * 4 <= kStageBytes, "balanced kernel: the merge buffers are one stage");
};

struct DBarriers {
  uint64_t full[8];
  uint64_t empty[8];
  int abort_flag;
  int last;  // balanced kernel: this CTA merges the parts of the sequence
};
static_assert(sizeof(DBarriers) % 8 == 0 && sizeof(DBarriers) + 2 * kConsumerWarps * kBalancedRows * 8 <= 2048, "barrier block");

__device__ __forceinline__ int atomic_add_acq_rel_gpu(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                            uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1,
                                                  uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Byte offset of the 16-byte unit (token row r, 8-element column group c8) inside a swizzled tile.
template <int D>
__device__ __forceinline__ uint32_t tile_offset(int r, int c8) {
  return (c8 >> 3) * DCfg<D>::kChunkBytes + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
}

// What a consumer warp holds of its (up to 16) query rows: the Q fragments and the running (maximum, sum, O) over its tokens.
template <int D>
struct WarpRows {
  uint32_t qa[D / 16][4];
  int lim0, lim1;         // last visible key of fragment rows g and g + 8
  float oacc[D / 8][4];
  float m0, m1;           // reference maxima (raw score units)
  float l0, l1;           // per-thread partial row sums

  __device__ __forceinline__ void begin(const DecodeParams& p, int batch, int head_k, int len, int rows, int lane) {
    const int g = lane >> 2;   // fragment row (and row + 8)
    const int t4 = lane & 3;   // fragment column pair
    // Q fragments (A operand, 16 x D), straight from global memory; rows >= `rows` are zero.
    {
      auto q_ptr = [&](int r) -> const __half* {
        const int q_pos = r / p.group;
        const int head = head_k * p.group + (r - q_pos * p.group);
        return p.q + batch * p.q_batch_stride + q_pos * p.q_row_stride + head * p.q_head_stride;
      };
      const __half* r0p = g < rows ? q_ptr(g) : nullptr;
      const __half* r1p = (g + 8) < rows ? q_ptr(g + 8) : nullptr;
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const int c = k * 16 + t4 * 2;
        qa[k][0] = r0p ? *reinterpret_cast<const uint32_t*>(r0p + c) : 0u;
        qa[k][1] = r1p ? *reinterpret_cast<const uint32_t*>(r1p + c) : 0u;
        qa[k][2] = r0p ? *reinterpret_cast<const uint32_t*>(r0p + c + 8) : 0u;
        qa[k][3] = r1p ? *reinterpret_cast<const uint32_t*>(r1p + c + 8) : 0u;
      }
    }
    // causal limit per fragment row: key j visible iff j <= q_pos + len - seqlen_q
    lim0 = lim1 = len - 1;
    if (p.is_causal) {
      lim0 = min(lim0, g / p.group + len - p.seqlen_q);
      lim1 = min(lim1, (g + 8) / p.group + len - p.seqlen_q);
    }
#pragma unroll
    for (int n = 0; n < D / 8; ++n) oacc[n][0] = oacc[n][1] = oacc[n][2] = oacc[n][3] = 0.f;
    m0 = m1 = -INFINITY;
    l0 = l1 = 0.f;
  }

  // 16 tokens of a tile, the first of them token tok0 < len; sK, sV: the tiles, v_tile: the V tile's address, c: scale * log2(e)
  __device__ __forceinline__ void tokens(uint32_t sK, uint32_t sV, uint8_t* v_tile, int tok_in_tile, int tok0, int len, float c,
                                         int lane) {
    const int t4 = lane & 3;
    // ---- S = Q K^T for 16 tokens: two n8 tiles ----
    float sacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
      uint32_t b0, b1, b2, b3;
      const int mi = lane >> 3, rr = lane & 7;
      ldmatrix_x4(sK + tile_offset<D>(tok_in_tile + (mi >> 1) * 8 + rr, k * 2 + (mi & 1)), b0, b1,
                  b2, b3);
      mma_16816(sacc[0], qa[k], b0, b1);
      mma_16816(sacc[1], qa[k], b2, b3);
    }
    // ---- mask the tail / causal limit ----
    if (tok0 + 15 > min(lim0, lim1)) {
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int col = tok0 + n * 8 + t4 * 2;
        if (col > lim0) sacc[n][0] = -INFINITY;
        if (col + 1 > lim0) sacc[n][1] = -INFINITY;
        if (col > lim1) sacc[n][2] = -INFINITY;
        if (col + 1 > lim1) sacc[n][3] = -INFINITY;
      }
    }
    // Rows of V past the end of the sequence may hold anything (uninitialised cache memory):
    // zero them so that 0 * garbage cannot produce NaN.  Only this warp reads these rows.
    // (warp-uniform condition)
    if (tok0 + 15 >= len) {
      for (int idx = lane; idx < 16 * (D / 8); idx += 32) {
        const int r = idx / (D / 8), c8 = idx - r * (D / 8);
        if (tok0 + r >= len)
          *reinterpret_cast<uint4*>(v_tile +
                                    tile_offset<D>(tok_in_tile + r, c8)) = make_uint4(0, 0, 0, 0);
      }
      fence_proxy_async_smem();  // order these generic writes before the next TMA refill
      __syncwarp();
    }
    // ---- online softmax with a lazy reference maximum ----
    float mx0 = fmaxf(fmaxf(sacc[0][0], sacc[0][1]), fmaxf(sacc[1][0], sacc[1][1]));
    float mx1 = fmaxf(fmaxf(sacc[0][2], sacc[0][3]), fmaxf(sacc[1][2], sacc[1][3]));
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    float a0 = 1.f, a1 = 1.f;
    bool need = false;
    if (mx0 > m0) {
      if (m0 == -INFINITY) m0 = mx0;
      else if ((mx0 - m0) * c > 8.f) { a0 = ex2f((m0 - mx0) * c); m0 = mx0; need = true; }
    }
    if (mx1 > m1) {
      if (m1 == -INFINITY) m1 = mx1;
      else if ((mx1 - m1) * c > 8.f) { a1 = ex2f((m1 - mx1) * c); m1 = mx1; need = true; }
    }
    if (__any_sync(0xffffffffu, need)) {
      l0 *= a0;
      l1 *= a1;
#pragma unroll
      for (int n = 0; n < D / 8; ++n) {
        oacc[n][0] *= a0; oacc[n][1] *= a0;
        oacc[n][2] *= a1; oacc[n][3] *= a1;
      }
    }
    const float nm0 = (m0 == -INFINITY) ? 0.f : -m0 * c;
    const float nm1 = (m1 == -INFINITY) ? 0.f : -m1 * c;
    uint32_t pa[4];
    {
      const float p00 = ex2f(fmaf(sacc[0][0], c, nm0)), p01 = ex2f(fmaf(sacc[0][1], c, nm0));
      const float p02 = ex2f(fmaf(sacc[0][2], c, nm1)), p03 = ex2f(fmaf(sacc[0][3], c, nm1));
      const float p10 = ex2f(fmaf(sacc[1][0], c, nm0)), p11 = ex2f(fmaf(sacc[1][1], c, nm0));
      const float p12 = ex2f(fmaf(sacc[1][2], c, nm1)), p13 = ex2f(fmaf(sacc[1][3], c, nm1));
      l0 += (p00 + p01) + (p10 + p11);
      l1 += (p02 + p03) + (p12 + p13);
      pa[0] = pack_half2(p00, p01);
      pa[1] = pack_half2(p02, p03);
      pa[2] = pack_half2(p10, p11);
      pa[3] = pack_half2(p12, p13);
    }
    // ---- O += P V ----
#pragma unroll
    for (int n = 0; n < D / 16; ++n) {
      uint32_t b0, b1, b2, b3;
      const int mi = lane >> 3, rr = lane & 7;
      ldmatrix_x4_trans(sV + tile_offset<D>(tok_in_tile + (mi & 1) * 8 + rr, n * 2 + (mi >> 1)), b0,
                        b1, b2, b3);
      mma_16816(oacc[2 * n], pa, b0, b1);
      mma_16816(oacc[2 * n + 1], pa, b2, b3);
    }
  }
};

template <int D>
__global__ void __launch_bounds__(kDecodeThreads, (D == 128) ? 2 : 2)
decode_split_kernel(const __grid_constant__ DecodeParams p) {
  using C = DCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  const int split = blockIdx.x;
  const int head_k = blockIdx.y;
  const int batch = blockIdx.z;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rows = p.seqlen_q * p.group;  // valid rows of the 16-row M tile
  grid_launch_dependents();  // the merge waits for this grid by itself

  // ---- this CTA's token range ----
  // Lengths are clamped to the cache capacity on the device (the host does not have to read them back);
  // a clamp is reported through the status word.
  const CacheLength length = cache_length(p.cache_seqlens[batch], p.seqlen_new, p.capacity, p.checked);
  const int len = length.len;
  if (length.report && threadIdx.x == 0 && p.status) atomicOr(p.status, kStatusCapacityClamped);
  const int n_tiles = (len + kTileTokens - 1) / kTileTokens;
  int tile_begin, tile_end;
  if (p.chunk_tiles > 0) {
    tile_begin = min(n_tiles, split * p.chunk_tiles);
    tile_end = min(n_tiles, tile_begin + p.chunk_tiles);
  } else {
    tile_begin = static_cast<int>(static_cast<int64_t>(n_tiles) * split / p.num_splits);
    tile_end = static_cast<int>(static_cast<int64_t>(n_tiles) * (split + 1) / p.num_splits);
  }
  const int my_tiles = tile_end - tile_begin;

  // row r of the M tile -> (query position, head); output row index in (b, h, seqlen_q) order
  auto out_row_index = [&](int r) -> int64_t {
    const int q_pos = r / p.group;
    const int head = head_k * p.group + (r - q_pos * p.group);
    return (static_cast<int64_t>(batch) * p.h + head) * p.seqlen_q + q_pos;
  };

  const bool stop = cta_should_stop(p.status);  // CTA-uniform
  if (my_tiles <= 0 || stop) {
    if (threadIdx.x == 0) grid_dependency_wait();
    // empty split: neutral partial (or a zero row when there is nothing to attend to at all)
    for (int idx = threadIdx.x; idx < rows * (D / 2); idx += blockDim.x) {
      const int r = idx / (D / 2);
      const int c = (idx - r * (D / 2)) * 2;
      const int64_t orow = out_row_index(r);
      if (p.num_splits > 1) {
        float2* dst = reinterpret_cast<float2*>(p.o_accum + (split * p.rows_total + orow) * D + c);
        *dst = make_float2(0.f, 0.f);
      } else {
        const int q_pos = r / p.group;
        const int head = head_k * p.group + (r - q_pos * p.group);
        __half2* dst = reinterpret_cast<__half2*>(p.o + batch * p.o_batch_stride + q_pos * p.o_row_stride +
                                                  head * p.o_head_stride + c);
        *dst = __floats2half2_rn(0.f, 0.f);
      }
    }
    for (int r = threadIdx.x; r < rows; r += blockDim.x) {
      const int64_t orow = out_row_index(r);
      if (p.num_splits > 1) p.lse_accum[split * p.rows_total + orow] = -INFINITY;
      else p.lse[orow] = 0.f;
    }
    return;
  }

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  DBarriers* bars = reinterpret_cast<DBarriers*>(smem + C::kStages * C::kStageBytes);
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], kConsumerWarps);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
    grid_dependency_wait();  // the appended rows
  }
  __syncthreads();
  WaitCtx ctx{&bars->abort_flag, p.status};

  if (warp == kConsumerWarps) {
    // =========================== TMA producer ===========================
    if (lane == 0) {
      prefetch_tensormap(&p.tm_k);
      prefetch_tensormap(&p.tm_v);
      const int cache_row = p.cache_batch_idx ? p.cache_batch_idx[batch] : batch;
      for (int i = 0; i < my_tiles; ++i) {
        const int s = i % C::kStages;
        const uint32_t ph = (i / C::kStages) & 1;
        const int tok = (tile_begin + i) * kTileTokens;
        int row = tok, blk = cache_row;
        if (p.block_table) {
          blk = p.block_table[batch * p.block_table_batch_stride + tok / p.page_size];
          row = tok % p.page_size;
        }
        if (!mbar_wait(&bars->empty[s], ph ^ 1, ctx)) break;
        mbar_arrive_expect_tx(&bars->full[s], C::kStageBytes);
        uint8_t* dst = smem + s * C::kStageBytes;
#pragma unroll
        for (int c = 0; c < C::kChunks; ++c)
          tma_load_4d(dst + c * C::kChunkBytes, &p.tm_k, &bars->full[s], c * 64, head_k, row, blk);
#pragma unroll
        for (int c = 0; c < C::kChunks; ++c)
          tma_load_4d(dst + C::kTileBytes + c * C::kChunkBytes, &p.tm_v, &bars->full[s], c * 64,
                      head_k, row, blk);
      }
    }
  } else {
    // =========================== consumers ===========================
    const int g = lane >> 2;   // fragment row (and row + 8)
    const int t4 = lane & 3;   // fragment column pair
    WarpRows<D> w;
    w.begin(p, batch, head_k, len, rows, lane);
    const float c = p.scale_log2;
    const int tok_in_tile = warp * 16;     // this warp's 16 tokens of every tile
    bool ok = true;

    for (int i = 0; i < my_tiles; ++i) {
      const int s = i % C::kStages;
      const uint32_t ph = (i / C::kStages) & 1;
      ok = mbar_wait(&bars->full[s], ph, ctx);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const uint32_t sK = smem_u32(smem + s * C::kStageBytes);
      const int tok0 = (tile_begin + i) * kTileTokens + tok_in_tile;  // first token of this warp
      if (tok0 < len)
        w.tokens(sK, sK + C::kTileBytes, smem + s * C::kStageBytes + C::kTileBytes, tok_in_tile, tok0, len, c, lane);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->empty[s]);
    }

    // ---- merge the four warps: (m, l, O) through shared memory (aliases the stage ring) ----
    w.l0 += __shfl_xor_sync(0xffffffffu, w.l0, 1);
    w.l0 += __shfl_xor_sync(0xffffffffu, w.l0, 2);
    w.l1 += __shfl_xor_sync(0xffffffffu, w.l1, 1);
    w.l1 += __shfl_xor_sync(0xffffffffu, w.l1, 2);
    named_barrier_sync(1, kConsumerWarps * 32);  // every warp is done reading the ring
    float* mbuf = reinterpret_cast<float*>(smem);
    // layout: [warp][row][D + 2] with the last two floats = (m, l)
    {
      float* dst = mbuf + warp * kMaxRows * (D + 2);
#pragma unroll
      for (int n = 0; n < D / 8; ++n) {
        const int col = n * 8 + t4 * 2;
        *reinterpret_cast<float2*>(dst + g * (D + 2) + col) = make_float2(w.oacc[n][0], w.oacc[n][1]);
        *reinterpret_cast<float2*>(dst + (g + 8) * (D + 2) + col) = make_float2(w.oacc[n][2], w.oacc[n][3]);
      }
      if (t4 == 0) {
        dst[g * (D + 2) + D] = w.m0;
        dst[g * (D + 2) + D + 1] = w.l0;
        dst[(g + 8) * (D + 2) + D] = w.m1;
        dst[(g + 8) * (D + 2) + D + 1] = w.l1;
      }
    }
    named_barrier_sync(1, kConsumerWarps * 32);
    if (ok) {
      // 128 threads: thread -> (row, column slice)
      constexpr int kColsPerThread = D * kMaxRows / (kConsumerWarps * 32);  // 16 (D=128) or 8
      constexpr int kThreadsPerRow = D / kColsPerThread;                    // 8
      const int tid = threadIdx.x;
      const int r = tid / kThreadsPerRow;
      const int c0 = (tid - r * kThreadsPerRow) * kColsPerThread;
      if (r < rows) {
        float mw[kConsumerWarps], lw[kConsumerWarps];
        float mt = -INFINITY;
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) {
          mw[w] = mbuf[(w * kMaxRows + r) * (D + 2) + D];
          lw[w] = mbuf[(w * kMaxRows + r) * (D + 2) + D + 1];
          mt = fmaxf(mt, mw[w]);
        }
        float lt = 0.f, sc[kConsumerWarps];
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) {
          sc[w] = (mw[w] == -INFINITY) ? 0.f : ex2f((mw[w] - mt) * c);
          lt += lw[w] * sc[w];
        }
        const bool dead = (mt == -INFINITY) || (lt == 0.f);
        const float inv = dead ? 0.f : 1.f / lt;
        float acc[kColsPerThread];
#pragma unroll
        for (int j = 0; j < kColsPerThread; ++j) acc[j] = 0.f;
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) {
          const float* src = mbuf + (w * kMaxRows + r) * (D + 2) + c0;
#pragma unroll
          for (int j = 0; j < kColsPerThread; ++j) acc[j] = fmaf(src[j], sc[w], acc[j]);
        }
        const float lse_val = dead ? -INFINITY : (mt * c + __log2f(lt)) * kLn2;
        const int64_t orow = out_row_index(r);
        if (p.num_splits > 1) {
          float* dst = p.o_accum + (split * p.rows_total + orow) * D + c0;
#pragma unroll
          for (int j = 0; j < kColsPerThread; j += 4)
            *reinterpret_cast<float4*>(dst + j) =
                make_float4(acc[j] * inv, acc[j + 1] * inv, acc[j + 2] * inv, acc[j + 3] * inv);
          if (c0 == 0) p.lse_accum[split * p.rows_total + orow] = lse_val;
        } else {
          const int q_pos = r / p.group;
          const int head = head_k * p.group + (r - q_pos * p.group);
          __half* dst = p.o + batch * p.o_batch_stride + q_pos * p.o_row_stride + head * p.o_head_stride + c0;
#pragma unroll
          for (int j = 0; j < kColsPerThread; j += 8) {
            uint4 v;
            v.x = pack_half2(acc[j] * inv, acc[j + 1] * inv);
            v.y = pack_half2(acc[j + 2] * inv, acc[j + 3] * inv);
            v.z = pack_half2(acc[j + 4] * inv, acc[j + 5] * inv);
            v.w = pack_half2(acc[j + 6] * inv, acc[j + 7] * inv);
            *reinterpret_cast<uint4*>(dst + j) = v;
          }
          if (c0 == 0) p.lse[orow] = dead ? 0.f : lse_val;
        }
      }
    }
  }
  __syncthreads();
  if (bars->abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// num_splits == 0: the tiles of the whole batch shared out evenly
// ---------------------------------------------------------------------------------------------
// The host does not know the lengths.  Every CTA reads them, counts the 64-token tiles of the sequences, laid end to end, and takes
// its share of them for one KV head: an equal number of tiles whatever the spread of the lengths, one set-up per CTA, and the ring of
// stages runs on from one sequence into the next.  The CTAs of all heads go over the same tokens at the same time, whose rows lie
// next to each other in memory (a share of (sequence, head) pairs laid end to end, with heads far apart in time, read 3-10 % more slowly).
// A share holds the end of a sequence, whole ones and the beginning of another; the parts of a sequence that several CTAs
// share go to scratch memory (at most two per CTA), and the CTA that arrives last merges them, in the order of the tiles, so that the
// result does not depend on who that is.  Where a sequence is cut depends on the lengths of the others, and with it the last bits of its rows
// (P is rounded to fp16 against the maximum of a part).  Arrivals are counted in the call's own scratch memory, which calls that overlap do not share,
// and which the kernel before this one (append or prepare kernel) has zeroed.
// Bound by the K / V bytes for large batches, by a chain of latencies (lengths, Q and K / V tiles, merge) for small ones.  Append and
// attention, us, chunks of a fixed size per CTA and a merge kernel against this: 1 x 1500 tokens (Hq32 Hkv8 D128) 13.2 -> 10.4,
// 1 x 30000 42.1 -> 32.8, 16 x 1000-8000 56.3 -> 49.6 (6.0 TB/s), 64 x 1024-32768 620 -> 621 (6.9 TB/s), 128 x 20-64 (H32) 69.8 -> 43.1,
// 128 x 200-3000 (Hq8 Hkv2 D64) 34.4 -> 28.6.  Where the chunks are faster: see uses_balanced_kernel().
constexpr int kBalancedCtas = 2 * 148;  // two per SM are resident
constexpr int kMinShare = 2;            // tiles of a CTA at least
// A share of a sequence of n tiles is at least sqrt(kShareSlope * n * rows) of them (a warp merges a row): what a tile takes its CTA and
// what a part takes the CTA that merges the sequence are then about least together.  Half and twice the slope: 1.000 and 1.003 of the time over
// 400 shapes, 1.004 and 1.008 with one sequence, 1.004 and 1.005 with eight rows.  Sequences of up to kWholeTiles are not cut while there is a CTA for each, the merge takes as long: 60 x 50-250
// tokens (Hq8 Hkv2 D64) 12.4 -> 8.3.
constexpr float kShareSlope = 0.05f;
constexpr int kWholeTiles = 12;

__device__ __forceinline__ int kv_tiles(const DecodeParams& p, int batch, int& len) {
  len = cache_length(p.cache_seqlens[batch], p.seqlen_new, p.capacity, p.checked).len;
  return max(1, (len + kTileTokens - 1) / kTileTokens);  // an empty sequence has a share too: its rows are zero
}

// Tiles [begin, end) of CTA i of a head out of `ctas` that share `total`: the first `more` have one more than `each`.
struct Shares {
  int64_t total;
  int ctas, more;
  int64_t each;
  __device__ __forceinline__ Shares(int64_t total_, int ctas_) : total(total_), ctas(ctas_) {
    each = total / ctas;
    more = static_cast<int>(total - each * ctas);
  }
  __device__ __forceinline__ int64_t begin(int i) const { return i * each + min(i, more); }
  __device__ __forceinline__ int owner(int64_t tile) const {
    const int64_t first = more * (each + 1);
    return static_cast<int>(tile < first ? tile / (each + 1) : more + (tile - first) / each);
  }
};

// Walks a CTA's share sequence by sequence.
struct ShareWalk {
  int batch, tile, n_tiles, len;
  int64_t at, end;  // tiles counted over the batch, or over an uncut sequence

  // tiles [begin, end) of the batch, by a whole warp
  __device__ __forceinline__ void share_of_batch(const DecodeParams& p, int64_t begin, int64_t end_, int lane) {
    int64_t before = 0;  // tiles of the sequences before the current 32
    batch = 0, at = begin, end = end_;
    for (int b0 = 0; b0 < p.b; b0 += 32) {
      int unused, sum = b0 + lane < p.b ? kv_tiles(p, b0 + lane, unused) : 0;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, sum, off);
        if (lane >= off) sum += other;
      }
      const uint32_t past = __ballot_sync(0xffffffffu, before + sum > begin);
      if (past != 0) {
        const int first = __ffs(past) - 1;
        const int skipped = __shfl_sync(0xffffffffu, sum, max(first - 1, 0));
        batch = b0 + first;
        before += first > 0 ? skipped : 0;
        break;
      }
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    n_tiles = kv_tiles(p, batch, len);
    tile = static_cast<int>(begin - before);
  }
  __device__ __forceinline__ void whole_sequence(const DecodeParams& p, int cta) {
    batch = cta, tile = 0, at = 0;
    end = n_tiles = kv_tiles(p, batch, len);
  }
  __device__ __forceinline__ int count() const { return static_cast<int>(min(static_cast<int64_t>(n_tiles - tile), end - at)); }
  __device__ __forceinline__ void next(const DecodeParams& p) {
    at += count();
    tile = 0;
    if (at < end) n_tiles = kv_tiles(p, ++batch, len);
  }
};

// The tiles of the batch and of its longest sequence.
__device__ __forceinline__ int64_t all_tiles(const DecodeParams& p, int lane, int& longest) {
  int64_t sum = 0;
  longest = 0;
  for (int b0 = 0; b0 < p.b; b0 += 32) {
    int unused;
    const int n = b0 + lane < p.b ? kv_tiles(p, b0 + lane, unused) : 0;
    sum += __reduce_add_sync(0xffffffffu, n);
    longest = max(longest, __reduce_max_sync(0xffffffffu, n));
  }
  return sum;
}

// N (2 or 4) consecutive floats, aligned to their size
template <int N>
__device__ __forceinline__ void load_floats(const float* src, float (&x)[N]) {
  if constexpr (N == 4) {
    const float4 v = *reinterpret_cast<const float4*>(src);
    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
  } else {
    const float2 v = *reinterpret_cast<const float2*>(src);
    x[0] = v.x, x[1] = v.y;
  }
}
template <int N>
__device__ __forceinline__ void store_floats(float* dst, const float (&x)[N], float mul) {
  if constexpr (N == 4) {
    *reinterpret_cast<float4*>(dst) = make_float4(x[0] * mul, x[1] * mul, x[2] * mul, x[3] * mul);
  } else {
    *reinterpret_cast<float2*>(dst) = make_float2(x[0] * mul, x[1] * mul);
  }
}

// `bytes` (8 or 16) from global to shared memory, by each thread for itself
template <int kBytes>
__device__ __forceinline__ void async_copy(void* smem_dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(smem_dst)), "l"(src), "n"(kBytes) : "memory");
}
__device__ __forceinline__ void async_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One row of the merged parts of a sequence, by a warp: this lane's D / 32 columns, and the LSE.  first_slot: where the sequence begins;
// the later parts lie 2 * heads apart, from the slot before that on.  kPartsAtOnce rows are in flight at a time, through `buf` in shared
// memory (a lane reads what it copied itself): four at a time in registers, as many as they hold, took twice as long.
constexpr int kPartsAtOnce = 16;
template <int D>
__device__ __forceinline__ float merge_row(const float* o_accum, const float* lse_accum, int first_slot, int heads, int parts, int r,
                                           float* buf, int lane, float (&acc)[D / 32]) {
  constexpr int kPerLane = D / 32;
  auto slot_of = [&](int j) { return static_cast<int64_t>(first_slot + (j > 0 ? 2 * heads * j - 1 : 0)) * kBalancedRows + r; };
  auto lse_of = [&](int j) { return j < parts ? __ldcg(lse_accum + slot_of(j)) : -INFINITY; };
  float* mine = buf + lane * kPerLane;
  auto fetch = [&](int j0) {
#pragma unroll 4
    for (int u = 0; u < min(kPartsAtOnce, parts - j0); ++u)
      async_copy<kPerLane * 4>(mine + u * D, o_accum + slot_of(j0 + u) * D + lane * kPerLane);
  };
  fetch(0);
  const float first = lse_of(lane);
  float mx = first;
  for (int j = lane + 32; j < parts; j += 32) mx = fmaxf(mx, lse_of(j));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const bool dead = mx == -INFINITY;
  float sum = 0.f, weight = 0.f;
#pragma unroll
  for (int e = 0; e < kPerLane; ++e) acc[e] = 0.f;
  for (int j0 = 0; j0 < parts; j0 += kPartsAtOnce) {
    if (j0 > 0) fetch(j0);
    if (j0 % 32 == 0) {  // the weights of 32 parts sit in the lanes; 0 for a part without a visible key
      weight = dead ? 0.f : __expf((j0 == 0 ? first : lse_of(j0 + lane)) - mx);
      sum += weight;
    }
    async_copy_wait();
    for (int u = 0; u < min(kPartsAtOnce, parts - j0); ++u) {
      const float wu = __shfl_sync(0xffffffffu, weight, j0 % 32 + u);
      float x[kPerLane];
      load_floats(mine + u * D, x);
#pragma unroll
      for (int e = 0; e < kPerLane; ++e) acc[e] = fmaf(wu, x[e], acc[e]);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  const float inv = dead ? 0.f : 1.f / sum;
#pragma unroll
  for (int e = 0; e < kPerLane; ++e) acc[e] *= inv;
  return dead ? 0.f : mx + __logf(sum);
}

template <int D>
__global__ void __launch_bounds__(kDecodeThreads, 2)
decode_balanced_kernel(const __grid_constant__ DecodeParams p) {
  using C = DCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rows = p.seqlen_q * p.group;  // up to kBalancedRows: the upper half of the M tile is empty
  const int stop_probe = stop_probe_begin(p.status);
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  DBarriers* bars = reinterpret_cast<DBarriers*>(smem + C::kStages * C::kStageBytes);
  float2* ml_of_seqs = reinterpret_cast<float2*>(bars + 1);  // (m, l) of [sequence & 1][warp][row]: a warp may be a sequence ahead
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], kConsumerWarps);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  int longest;
  const int64_t total = all_tiles(p, lane, longest);
  const int least = max(kMinShare, static_cast<int>(sqrtf(kShareSlope * longest * max(rows, kConsumerWarps))));
  const bool uncut = longest <= kWholeTiles && p.b <= static_cast<int>(gridDim.y);
  const Shares shares(total, uncut ? p.b : static_cast<int>(min(static_cast<int64_t>(gridDim.y), (total + least - 1) / least)));
  const int cta = blockIdx.y, head_k = blockIdx.x;
  const bool stop = __syncthreads_or(stop_probe) != 0;
  if (cta >= shares.ctas) return;
  WaitCtx ctx{&bars->abort_flag, p.status};
  ShareWalk w;
  if (uncut) {
    w.whole_sequence(p, cta);
  } else {
    w.share_of_batch(p, shares.begin(cta), shares.begin(cta + 1), lane);
  }

  // row r of the M tile -> (query position, head)
  auto row_head = [&](int r, int& q_pos) {
    q_pos = r / p.group;
    return head_k * p.group + (r - q_pos * p.group);
  };

  if (stop) {  // sticky time-out bit: zeros, by the CTA where a sequence begins
    if (threadIdx.x == 0) grid_dependency_wait();
    for (; w.at < w.end; w.next(p)) {
      if (w.tile != 0) continue;
      for (int idx = threadIdx.x; idx < rows * (D / 8); idx += blockDim.x) {
        int q_pos;
        const int head = row_head(idx / (D / 8), q_pos);
        *reinterpret_cast<uint4*>(p.o + w.batch * p.o_batch_stride + q_pos * p.o_row_stride + head * p.o_head_stride +
                                  idx % (D / 8) * 8) = make_uint4(0, 0, 0, 0);
        if (idx % (D / 8) == 0) p.lse[(static_cast<int64_t>(w.batch) * p.h + head) * p.seqlen_q + q_pos] = 0.f;
      }
    }
    return;
  }

  if (warp == kConsumerWarps) {
    // =========================== TMA producer ===========================
    if (lane == 0) {
      prefetch_tensormap(&p.tm_k);
      prefetch_tensormap(&p.tm_v);
      grid_dependency_wait();  // the appended rows; nothing else here depends on the kernel before
      bool ok = true;
      int i = 0;  // ring position
      for (; ok && w.at < w.end; w.next(p)) {
        const int cache_row = p.cache_batch_idx ? p.cache_batch_idx[w.batch] : w.batch;
        const int n = w.len > 0 ? w.count() : 0;
        for (int t = 0; t < n; ++t, ++i) {
          const int s = i % C::kStages;
          const int tok = (w.tile + t) * kTileTokens;
          int row = tok, blk = cache_row;
          if (p.block_table) {
            blk = p.block_table[w.batch * p.block_table_batch_stride + tok / p.page_size];
            row = tok % p.page_size;
          }
          if (!(ok = mbar_wait(&bars->empty[s], ((i / C::kStages) & 1) ^ 1, ctx))) break;
          mbar_arrive_expect_tx(&bars->full[s], C::kStageBytes);
          uint8_t* dst = smem + s * C::kStageBytes;
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c)
            tma_load_4d(dst + c * C::kChunkBytes, &p.tm_k, &bars->full[s], c * 64, head_k, row, blk);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c)
            tma_load_4d(dst + C::kTileBytes + c * C::kChunkBytes, &p.tm_v, &bars->full[s], c * 64, head_k, row, blk);
        }
        // the stage behind the last tile of a sequence is where the consumers merge their rows
        if (ok && (ok = mbar_wait(&bars->empty[i % C::kStages], ((i / C::kStages) & 1) ^ 1, ctx))) {
          mbar_arrive(&bars->full[i % C::kStages]);
          ++i;
        }
      }
    }
  } else {
    // =========================== consumers ===========================
    const int g = lane >> 2;   // fragment row (and row + 8)
    const int t4 = lane & 3;   // fragment column pair
    const int tok_in_tile = warp * 16;  // this warp's 16 tokens of every tile
    const float c = p.scale_log2;
    constexpr int kPerLane = D / 32;    // columns of a lane when a warp merges a row
    auto wait_full = [&](int i) {
      const bool ok = mbar_wait(&bars->full[i % C::kStages], (i / C::kStages) & 1, ctx);
      return __all_sync(0xffffffffu, ok) != 0;
    };
    auto release = [&](int i) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->empty[i % C::kStages]);
    };
    int i = 0, n_seqs = 0;
    float2* ml = ml_of_seqs;
    bool ok = true;
    for (; ok && w.at < w.end; w.next(p)) {
      const int count = w.count(), n = w.len > 0 ? count : 0;
      const bool whole = count == w.n_tiles;
      if (w.tile == 0 && head_k == 0 && threadIdx.x == 0 && p.status &&
          cache_length(p.cache_seqlens[w.batch], p.seqlen_new, p.capacity, p.checked).report)
        atomicOr(p.status, kStatusCapacityClamped);
      WarpRows<D> mine;
      mine.begin(p, w.batch, head_k, w.len, rows, lane);
      for (int t = 0; t < n; ++t, ++i) {
        if (!(ok = wait_full(i))) break;
        uint8_t* stage = smem + (i % C::kStages) * C::kStageBytes;
        const uint32_t sK = smem_u32(stage);
        const int tok0 = (w.tile + t) * kTileTokens + tok_in_tile;
        if (tok0 < w.len) mine.tokens(sK, sK + C::kTileBytes, stage + C::kTileBytes, tok_in_tile, tok0, w.len, c, lane);
        release(i);
      }
      ok = ok && wait_full(i);

      // ---- merge the four warps through the stage that holds no tile: [warp][row][D], the columns of row r xor 8 * (r % 8) so
      // that the eight rows of a fragment column lie in different banks ----
      float* mbuf = reinterpret_cast<float*>(smem + (i % C::kStages) * C::kStageBytes);
      mine.l0 += __shfl_xor_sync(0xffffffffu, mine.l0, 1);
      mine.l0 += __shfl_xor_sync(0xffffffffu, mine.l0, 2);
      float* dst = mbuf + warp * kBalancedRows * D;
      ml = ml_of_seqs + (n_seqs++ & 1) * kConsumerWarps * kBalancedRows;
      if (ok) {
#pragma unroll
        for (int k = 0; k < D / 8; ++k) {
          const int col = ((k * 8) ^ (g * 8)) + t4 * 2;
          if (g < rows) *reinterpret_cast<float2*>(dst + g * D + col) = make_float2(mine.oacc[k][0], mine.oacc[k][1]);
        }
        if (t4 == 0) ml[warp * kBalancedRows + g] = make_float2(mine.m0, mine.l0);
      }
      // A warp may give up on a phase that the others see complete: all come here, and all leave or none (a warp that left by itself
      // would be at the end of the kernel while the others wait for it at this barrier, without a limit).
      if (!(ok = named_barrier_and(1, kConsumerWarps * 32, ok))) break;

      // a warp per row, a lane per kPerLane columns
      auto store = [&](int r, const float (&acc)[kPerLane], float mul, float lse) {
        int q_pos;
        const int head = row_head(r, q_pos);
        __half* out = p.o + w.batch * p.o_batch_stride + q_pos * p.o_row_stride + head * p.o_head_stride + lane * kPerLane;
        if constexpr (kPerLane == 4) {
          *reinterpret_cast<uint2*>(out) = make_uint2(pack_half2(acc[0] * mul, acc[1] * mul), pack_half2(acc[2] * mul, acc[3] * mul));
        } else {
          *reinterpret_cast<uint32_t*>(out) = pack_half2(acc[0] * mul, acc[1] * mul);
        }
        if (lane == 0) p.lse[(static_cast<int64_t>(w.batch) * p.h + head) * p.seqlen_q + q_pos] = lse;
      };
      // part of a sequence in scratch memory: slot 1 of the CTA where the sequence begins, slot 0 of the others
      auto part = [&](int owner, bool begins) { return 2 * (owner * static_cast<int>(gridDim.x) + head_k) + (begins ? 1 : 0); };
      for (int r = warp; r < rows; r += kConsumerWarps) {
        float2 of[kConsumerWarps];
        float mt = -INFINITY;
#pragma unroll
        for (int u = 0; u < kConsumerWarps; ++u) {
          of[u] = ml[u * kBalancedRows + r];
          mt = fmaxf(mt, of[u].x);
        }
        float lt = 0.f, acc[kPerLane];
#pragma unroll
        for (int e = 0; e < kPerLane; ++e) acc[e] = 0.f;
        const int col = (lane * kPerLane) ^ ((r & 7) * 8);
#pragma unroll
        for (int u = 0; u < kConsumerWarps; ++u) {
          const float scale = of[u].x == -INFINITY ? 0.f : ex2f((of[u].x - mt) * c);
          lt += of[u].y * scale;
          float x[kPerLane];
          load_floats(mbuf + (u * kBalancedRows + r) * D + col, x);
#pragma unroll
          for (int e = 0; e < kPerLane; ++e) acc[e] = fmaf(x[e], scale, acc[e]);
        }
        const bool dead = mt == -INFINITY || lt == 0.f;
        if (dead) {  // no visible key: 0 times a value that is hidden may be NaN
#pragma unroll
          for (int e = 0; e < kPerLane; ++e) acc[e] = 0.f;
        }
        const float inv = dead ? 0.f : 1.f / lt;
        const float lse = dead ? -INFINITY : (mt * c + __log2f(lt)) * kLn2;
        if (whole) {
          store(r, acc, inv, dead ? 0.f : lse);
        } else {
          const int slot = part(cta, w.tile == 0);
          store_floats(p.o_accum + (static_cast<int64_t>(slot) * kBalancedRows + r) * D + lane * kPerLane, acc, inv);
          if (lane == 0) p.lse_accum[slot * kBalancedRows + r] = lse;
        }
      }
      if (!whole) {
        // ---- the last of the CTAs that share the sequence merges its parts ----
        const int64_t first_tile = w.at - w.tile;
        const int c0 = shares.owner(first_tile), parts = shares.owner(first_tile + w.n_tiles - 1) - c0 + 1;
        named_barrier_sync(1, kConsumerWarps * 32);
        if (threadIdx.x == 0) {  // release: the barrier's other threads' writes too; acquire: those of the CTAs that came before
          grid_dependency_wait();  // the zeros; over long ago, the producer has waited for the same before the first tile
          bars->last = atomic_add_acq_rel_gpu(p.arrivals + c0 * gridDim.x + head_k, 1) == parts - 1;
        }
        named_barrier_sync(1, kConsumerWarps * 32);
        if (bars->last) {
          for (int r = warp; r < rows; r += kConsumerWarps) {
            float acc[kPerLane];
            const float lse = merge_row<D>(p.o_accum, p.lse_accum, part(c0, true), gridDim.x, parts, r, mbuf + warp * kPartsAtOnce * D, lane, acc);
            store(r, acc, 1.f, lse);
          }
        }
      }
      fence_proxy_async_smem();  // the merge buffer's writes, before TMA fills the stage again
      release(i);
      ++i;
    }
  }
  __syncthreads();
  if (bars->abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// append: k_new/v_new (b, s_new, h_k, d) -> cache rows / pages at cache_seqlens[b] + t
// ---------------------------------------------------------------------------------------------
struct AppendParams {
  __half* k_cache;
  __half* v_cache;
  const __half* k_new;
  const __half* v_new;
  int64_t kc_batch_stride, kc_row_stride, kc_head_stride;
  int64_t vc_batch_stride, vc_row_stride, vc_head_stride;
  int64_t kn_batch_stride, kn_row_stride, kn_head_stride;
  int64_t vn_batch_stride, vn_row_stride, vn_head_stride;
  int b, seqlen_new, h_k, d;
  int cache_batch, seqlen_cache;
  const int* cache_seqlens;
  const int* cache_batch_idx;
  const int* block_table;
  int64_t block_table_batch_stride;
  int max_blocks_per_seq;
  // fa_kvcache_checked(): nothing is written unless every length is at most max_length
  int* verdict;
  int token;
  int64_t max_length;
  // balanced kernel behind this one: its arrival counters, to be zeroed
  int* arrivals;
  int num_arrivals;
};

// By the threads of one block.
__device__ __forceinline__ void zero_arrivals(int* arrivals, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) arrivals[i] = 0;
}

// By all threads of a block.
__device__ __forceinline__ bool lengths_fit(const int* lengths, int b, int64_t max_length) {
  bool over = false;
  for (int i = threadIdx.x; i < b; i += blockDim.x) over |= lengths[i] > max_length;
  return !__syncthreads_or(over);
}
__device__ __forceinline__ void tell_host(int* verdict, int token, bool fits) {
  *reinterpret_cast<volatile int*>(verdict) = 2 * token + (fits ? 0 : 1);
  __threadfence_system();
}

// Calls without new tokens: what the append kernel does besides appending
__global__ void __launch_bounds__(256) prepare_kernel(const int* lengths, int b, int64_t max_length, int* verdict, int token, int* arrivals,
                                                      int num_arrivals) {
  grid_launch_dependents();
  zero_arrivals(arrivals, num_arrivals);
  if (verdict != nullptr) {
    const bool fits = lengths_fit(lengths, b, max_length);
    if (threadIdx.x == 0) tell_host(verdict, token, fits);
  }
}

// The 16-byte units of the first step are fetched before the lengths are looked at: two memory latencies in a row instead of four
// (lengths, the length again, the unit, the store), which is most of what a small append takes.
__global__ void __launch_bounds__(256) append_kernel(const __grid_constant__ AppendParams p) {
  grid_launch_dependents();
  const int unit_bits = p.d == 128 ? 4 : 3;  // d / 8 units of 16 bytes per (token, head)
  const int64_t total = (static_cast<int64_t>(p.b) * p.seqlen_new * p.h_k) << unit_bits;
  int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  int u, head, t, batch, cached;
  uint4 kv, vv;
  auto fetch = [&]() {
    u = static_cast<int>(idx) & ((1 << unit_bits) - 1);
    if (total <= 0x7fffffff) {  // divisions in 32 bits
      const int rest = static_cast<int>(idx) >> unit_bits, token = rest / p.h_k;
      head = rest - token * p.h_k, batch = token / p.seqlen_new, t = token - batch * p.seqlen_new;
    } else {
      const int64_t rest = idx >> unit_bits, token = rest / p.h_k;
      head = static_cast<int>(rest - token * p.h_k);
      batch = static_cast<int>(token / p.seqlen_new), t = static_cast<int>(token - static_cast<int64_t>(batch) * p.seqlen_new);
    }
    cached = p.cache_seqlens[batch];
    kv = *reinterpret_cast<const uint4*>(p.k_new + batch * p.kn_batch_stride + t * p.kn_row_stride + head * p.kn_head_stride + u * 8);
    vv = *reinterpret_cast<const uint4*>(p.v_new + batch * p.vn_batch_stride + t * p.vn_row_stride + head * p.vn_head_stride + u * 8);
  };
  if (idx < total) fetch();
  if (blockIdx.x == 0) zero_arrivals(p.arrivals, p.num_arrivals);
  if (p.verdict != nullptr) {  // every block looks at all lengths (b loads by its 256 threads, from L2 but for the first): no launch in between
    const bool fits = lengths_fit(p.cache_seqlens, p.b, p.max_length);
    if (blockIdx.x == 0 && threadIdx.x == 0) tell_host(p.verdict, p.token, fits);
    if (!fits) return;
  }
  while (idx < total) {
    const int pos = static_cast<int>(static_cast<uint32_t>(cached) + t);  // past 2^31: negative, not written
    int64_t blk = -1, row = pos;
    if (p.block_table) {
      const int slot = pos / p.seqlen_cache;
      if (pos >= 0 && slot < p.max_blocks_per_seq) {  // beyond capacity: never written
        blk = p.block_table[batch * p.block_table_batch_stride + slot];
        row = pos - slot * p.seqlen_cache;
      }
    } else if (pos >= 0 && pos < p.seqlen_cache) {
      blk = p.cache_batch_idx ? p.cache_batch_idx[batch] : batch;
    }
    if (blk >= 0 && blk < p.cache_batch) {
      *reinterpret_cast<uint4*>(p.k_cache + blk * p.kc_batch_stride + row * p.kc_row_stride + head * p.kc_head_stride + u * 8) = kv;
      *reinterpret_cast<uint4*>(p.v_cache + blk * p.vc_batch_stride + row * p.vc_row_stride + head * p.vc_head_stride + u * 8) = vv;
    }
    idx += static_cast<int64_t>(gridDim.x) * blockDim.x;
    if (idx < total) fetch();
  }
}

bool uses_decode_kernel(const FaKvcacheParams* p) {
  return static_cast<int64_t>(p->seqlen_q) * (p->h / p->h_k) <= kMaxRows;
}

int capacity_tokens(const FaKvcacheParams* p) {
  return p->block_table ? p->max_blocks_per_seq * p->seqlen_cache : p->seqlen_cache;
}

int64_t capacity_tiles(const FaKvcacheParams* p) {
  return std::max<int64_t>(1, (static_cast<int64_t>(capacity_tokens(p)) + p->seqlen_new + kTileTokens - 1) / kTileTokens);
}

// CTAs per KV head: as many as are resident together, and no more than can have a share
int balanced_shares(const FaKvcacheParams* p) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(kBalancedCtas / p->h_k, capacity_tiles(p) * p->b)));
}

// Chunk plan for num_splits == 0: the lengths are unknown on the host (no synchronisation), so work is cut into fixed chunks of tiles: every
// CTA gets at most `chunk` tiles and the grid covers the cache capacity; CTAs past a sequence's end return at once.  The chunk is chosen so
// that the sequences at full capacity would give about four CTAs per SM-slot (2 resident CTAs x 148 SMs), with a floor of 8 tiles (512
// tokens) so that the merge traffic stays small against the K/V bytes.
void plan_chunks(const FaKvcacheParams* p, int* num_splits, int* chunk_tiles) {
  const int64_t cap_tiles = capacity_tiles(p);
  const int64_t base_ctas = static_cast<int64_t>(p->b) * p->h_k;
  const int64_t target_ctas = 4 * 2 * 148;
  const int64_t want = std::min<int64_t>((target_ctas + base_ctas - 1) / base_ctas, 256);  // splits per (sequence, KV head)
  const int64_t chunk = std::max<int64_t>((cap_tiles + want - 1) / want, 8);
  *num_splits = static_cast<int>((cap_tiles + chunk - 1) / chunk);
  *chunk_tiles = *num_splits <= 1 ? 0 : static_cast<int>(chunk);
}

// Which kernel attends calls with num_splits == 0.  More than kBalancedRows rows per KV head: the chunks, because the balanced kernel's merge
// by a single CTA takes longer than it saves: 16 rows, 6 x 1000-5000 tokens (Hkv1 D128) 22.7 us against 15.5, 3 x 3000-12000 (Hkv4) 26.8 : 22.7.
// Else the balanced kernel, except where the chunks measured faster (append and attention, us, balanced : chunks; 4300 shapes of 1 to 4096
// sequences and 64 to 32768 tokens):
//  * Many sequences of one or two heads, since every CTA counts the tiles of all of them: 4096 x 10-100 (Hkv1) 95 : 77, 16384 x 1-60 374 : 199;
//    2048 x 10-60 (Hkv8) 0.70 of the chunks' time, 1024 x 200-1000 (Hkv4) 1.07.
//  * A head count that leaves resident CTAs over: 16 x 100-1500 (D64) Hkv149 1.49, Hkv99 1.19; Hkv120 and Hkv64 1.0 and 0.90.
//  * Chunks that need no merge, until they are several rounds of CTAs (33 x 105-285, Hkv12, 16.5 : 13.0; 128 x 20-64, Hkv32, 42 : 69), and with
//    more than four rows, two for a warp to merge, always.
//  * Large batches, bound by HBM whichever way, where the shares of sequences of equal lengths read more slowly: at least 700 (D64: 500) pairs of sequence
//    and head with 90000 tiles, and 1184 pairs whose chunks need no merge and are long: D64 97 x 3742 Hkv32 503 : 412, 137 x 8190 Hkv8 384 : 335,
//    D128 54 x 8200 Hkv16 442 : 425; 24 x 2000 and shorter 0.85-1.0, 64 x 1024-32768 Hkv8 (512 pairs) 645 : 657.
//  * A batch whose chunks all run at once, about one per SM: there is nothing to balance, and finer shares are more parts to merge.
//    75 to 148 chunks 1.02-1.09 (2 x 6000-9000 Hq8 Hkv2 D128 16.5 : 14.4), with more than four rows up to 148 chunks 1.1-1.3, up to 296 of shorter
//    sequences 1.05-1.13; beyond that 0.75-0.95 and 0.85-0.95.  One sequence alone gains from finer shares (0.85-0.95).
bool uses_balanced_kernel(const FaKvcacheParams* p, int splits) {  // splits: of the chunk plan
  const int64_t rows = static_cast<int64_t>(p->seqlen_q) * (p->h / p->h_k);
  if (rows > kBalancedRows) return false;
  const int64_t tiles = capacity_tiles(p), pairs = static_cast<int64_t>(p->b) * p->h_k;
  if (p->b > 256 && (p->h_k < 4 || (p->h_k < 8 && tiles > 8))) return false;
  const int used = kBalancedCtas / p->h_k * p->h_k;  // of the CTAs that are resident together
  if (p->b > 1 && 5 * used < (p->b > 4 ? 4 : 3) * kBalancedCtas) return false;
  const bool two_rows_a_warp = rows > kConsumerWarps;
  if (splits == 1) return !two_rows_a_warp && pairs > 1200 && tiles <= (p->d == 64 ? 28 : 12);
  if (pairs >= (p->d == 64 ? 500 : 700) && tiles * pairs >= 90000) return false;
  if (tiles <= kWholeTiles) return true;  // not cut, or rarely: 0.6-0.95
  const int64_t chunks = static_cast<int64_t>(splits) * pairs;
  if (two_rows_a_warp) return p->b == 1 ? tiles < 64 || chunks > 148 : chunks > (tiles < 192 ? 296 : 148);
  return p->b == 1 || tiles >= 300 || chunks > 148 || chunks <= (tiles < 128 ? 74 : 40);
}

// Whatever the lengths, no sequence is cut: each is in one CTA's share
bool never_cut(const FaKvcacheParams* p) {
  return balanced_shares(p) == 1 || (capacity_tiles(p) <= kWholeTiles && p->b <= balanced_shares(p));
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Scratch memory of the balanced kernel: the parts (two per CTA), their LSE, an arrival counter per CTA
struct BalancedScratch {
  size_t lse, arrivals, bytes;  // offsets of the second and third, and the size
  int num_arrivals;
  explicit BalancedScratch(const FaKvcacheParams* p) : num_arrivals(balanced_shares(p) * p->h_k) {
    const size_t rows = 2 * static_cast<size_t>(num_arrivals) * kBalancedRows;
    lse = align_up(rows * p->d * sizeof(float), 256);
    arrivals = lse + align_up(rows * sizeof(float), 256);
    bytes = arrivals + align_up(num_arrivals * sizeof(int), 256);
  }
};

// How a call is attended.  An explicit num_splits is honoured as given (proportional ranges per sequence).
struct Plan {
  bool balanced = false;  // the balanced kernel, else the split kernel (or the tiled forward: one split)
  bool may_lack = false;  // chunk plan of one split: without scratch memory that the balanced kernel would use, that is what runs
  int splits = 1;         // parts that the keys of a sequence are attended in (balanced kernel: at most)
  int chunk = 0;          // tiles of a split; 0: proportional ranges
  size_t lse = 0;         // scratch memory: offset of the LSE of the parts behind the parts, and the size
  size_t bytes = 0;
};
Plan plan_call(const FaKvcacheParams* p) {
  Plan plan;
  if (!uses_decode_kernel(p)) return plan;
  if (p->num_splits > 0) {
    plan.splits = std::min(p->num_splits, 256);
  } else {
    plan_chunks(p, &plan.splits, &plan.chunk);
    plan.may_lack = plan.splits == 1;
    plan.balanced = uses_balanced_kernel(p, plan.splits);
    if (plan.balanced) {
      plan.splits = never_cut(p) ? 1 : static_cast<int>(std::min<int64_t>(balanced_shares(p), capacity_tiles(p)));
      plan.chunk = 0;
    }
  }
  if (plan.splits > 1 && plan.balanced) {
    const BalancedScratch scratch(p);
    plan.lse = scratch.lse, plan.bytes = scratch.bytes;
  } else if (plan.splits > 1) {
    const size_t rows = static_cast<size_t>(plan.splits) * p->b * p->h * p->seqlen_q;
    plan.lse = align_up(rows * p->d * sizeof(float), 256);
    plan.bytes = plan.lse + align_up(rows * sizeof(float), 256);
  }
  return plan;
}

// kKernel: decode_split_kernel<D> or decode_balanced_kernel<D>
template <int D, auto kKernel>
int launch_decode(const DecodeParams& dp, dim3 grid, bool overlap, cudaStream_t stream) {
  using C = DCfg<D>;
  static bool configured[64] = {};
  int dev = 0;
  FA_CHECK_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    FA_CHECK_CUDA(cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
    configured[dev & 63] = true;
  }
  if (overlap) {
    FA_CHECK_CUDA(launch_overlapped(kKernel, grid, kDecodeThreads, C::kSmemBytes, stream, dp));
  } else {
    kKernel<<<grid, kDecodeThreads, C::kSmemBytes, stream>>>(dp);
    FA_CHECK_CUDA(cudaGetLastError());
  }
  return FA_OK;
}

int validate(const FaKvcacheParams* p, const char* who) {
  FA_CHECK_ARG(p != nullptr, std::string(who) + ": params is NULL");
  if (p->d != 64 && p->d != 128)
    return set_error(FA_ERR_UNSUPPORTED, std::string(who) + ": head_dim must be 64 or 128");
  FA_CHECK_ARG(p->b >= 1 && p->seqlen_q >= 1 && p->h >= 1 && p->h_k >= 1 && p->h % p->h_k == 0,
               std::string(who) + ": bad b / seqlen_q / h / h_k");
  FA_CHECK_ARG(p->seqlen_new >= 0 && p->num_splits >= 0, std::string(who) + ": negative seqlen_new or num_splits");
  FA_CHECK_ARG(p->cache_batch >= 1 && p->seqlen_cache >= 1, std::string(who) + ": empty cache");
  if (p->block_table) {
    FA_CHECK_ARG(p->seqlen_cache % kTileTokens == 0, std::string(who) + ": page size must be a multiple of 64");
    FA_CHECK_ARG(p->cache_batch_idx == nullptr, std::string(who) + ": block_table excludes cache_batch_idx");
    FA_CHECK_ARG(p->max_blocks_per_seq >= 1, std::string(who) + ": max_blocks_per_seq must be positive");
  }
  return FA_OK;
}

}  // namespace
}  // namespace fa

extern "C" int fa_kvcache_num_splits(const FaKvcacheParams* p) {
  using namespace fa;
  int rc = validate(p, "fa_kvcache_num_splits");
  if (rc != FA_OK) return rc;
  return plan_call(p).splits;
}

extern "C" size_t fa_kvcache_workspace_bytes(const FaKvcacheParams* p) {
  using namespace fa;
  if (validate(p, "fa_kvcache_workspace_bytes") != FA_OK) return 0;
  return plan_call(p).bytes;
}

namespace fa {
namespace {
// verdict: see fa_kvcache_checked(); NULL: lengths are clamped to the capacity
int run_kvcache(const FaKvcacheParams* p, int* verdict, int token, cudaStream_t stream) {
  int rc = validate(p, "fa_kvcache");
  if (rc != FA_OK) return rc;
  FA_CHECK_ARG(p->q && p->k_cache && p->v_cache && p->o && p->lse && p->cache_seqlens,
               "fa_kvcache: q, k_cache, v_cache, o, lse, cache_seqlens must be non-NULL");
  FA_CHECK_ARG((p->k_new == nullptr) == (p->v_new == nullptr), "fa_kvcache: k_new and v_new go together");
  FA_CHECK_ARG(p->k_new != nullptr || p->seqlen_new == 0, "fa_kvcache: seqlen_new > 0 without k_new");
  FA_CHECK_ARG(aligned16(p->q) && aligned16(p->o) && p->q_row_stride % 8 == 0 && p->q_head_stride % 8 == 0 &&
                   p->q_batch_stride % 8 == 0 && p->o_row_stride % 8 == 0 && p->o_head_stride % 8 == 0 &&
                   p->o_batch_stride % 8 == 0,
               "fa_kvcache: q and o must be 16-byte aligned with strides that are multiples of 8 elements");
  rc = check_device_sm100();
  if (rc != FA_OK) return rc;

  Plan plan = plan_call(p);
  uint8_t* scratch = nullptr;
  if (plan.bytes > 0) {
    const bool enough = p->workspace != nullptr && p->workspace_bytes >= plan.bytes;
    if (plan.may_lack && !(enough && aligned16(p->workspace))) {
      plan = Plan{};
    } else {
      if (!enough) return set_error(FA_ERR_WORKSPACE, "fa_kvcache: workspace smaller than fa_kvcache_workspace_bytes()");
      FA_CHECK_ARG(aligned16(p->workspace), "fa_kvcache: workspace must be 16-byte aligned");
      scratch = static_cast<uint8_t*>(p->workspace);
    }
  }
  int* arrivals = nullptr;
  int num_arrivals = 0;
  if (plan.balanced && scratch != nullptr) {
    const BalancedScratch layout(p);
    arrivals = reinterpret_cast<int*>(scratch + layout.arrivals), num_arrivals = layout.num_arrivals;
  }

  // The launches overlap (launch_overlapped): each kernel's set-up and launch run under its predecessor, and it waits inside for
  // what that writes.
  // ---- 1. append ----
  const bool appends = p->k_new && p->seqlen_new > 0;
  const int64_t max_length = (p->block_table ? static_cast<int64_t>(p->max_blocks_per_seq) : 1) * p->seqlen_cache - p->seqlen_new;
  if (!appends && (verdict != nullptr || num_arrivals > 0)) {
    prepare_kernel<<<1, 256, 0, stream>>>(p->cache_seqlens, p->b, max_length, verdict, token, arrivals, num_arrivals);
    FA_CHECK_CUDA(cudaGetLastError());
  }
  if (appends) {
    FA_CHECK_ARG(aligned16(p->k_new) && aligned16(p->v_new) && aligned16(p->k_cache) && aligned16(p->v_cache),
                 "fa_kvcache: k_new, v_new and the caches must be 16-byte aligned");
    const int64_t strides[] = {p->kc_batch_stride, p->kc_row_stride, p->kc_head_stride, p->vc_batch_stride,
                               p->vc_row_stride, p->vc_head_stride, p->kn_batch_stride, p->kn_row_stride,
                               p->kn_head_stride, p->vn_batch_stride, p->vn_row_stride, p->vn_head_stride};
    for (int64_t s : strides)
      FA_CHECK_ARG(s % 8 == 0, "fa_kvcache: cache and k_new/v_new strides must be multiples of 8 elements");
    AppendParams ap;
    ap.k_cache = static_cast<__half*>(p->k_cache);
    ap.v_cache = static_cast<__half*>(p->v_cache);
    ap.k_new = static_cast<const __half*>(p->k_new);
    ap.v_new = static_cast<const __half*>(p->v_new);
    ap.kc_batch_stride = p->kc_batch_stride; ap.kc_row_stride = p->kc_row_stride; ap.kc_head_stride = p->kc_head_stride;
    ap.vc_batch_stride = p->vc_batch_stride; ap.vc_row_stride = p->vc_row_stride; ap.vc_head_stride = p->vc_head_stride;
    ap.kn_batch_stride = p->kn_batch_stride; ap.kn_row_stride = p->kn_row_stride; ap.kn_head_stride = p->kn_head_stride;
    ap.vn_batch_stride = p->vn_batch_stride; ap.vn_row_stride = p->vn_row_stride; ap.vn_head_stride = p->vn_head_stride;
    ap.b = p->b; ap.seqlen_new = p->seqlen_new; ap.h_k = p->h_k; ap.d = p->d;
    ap.cache_batch = p->cache_batch; ap.seqlen_cache = p->seqlen_cache;
    ap.cache_seqlens = p->cache_seqlens; ap.cache_batch_idx = p->cache_batch_idx;
    ap.block_table = p->block_table; ap.block_table_batch_stride = p->block_table_batch_stride;
    ap.max_blocks_per_seq = p->max_blocks_per_seq;
    ap.verdict = verdict; ap.token = token; ap.max_length = max_length;
    ap.arrivals = arrivals; ap.num_arrivals = num_arrivals;
    const int64_t total = static_cast<int64_t>(p->b) * p->seqlen_new * p->h_k * (p->d / 8);
    const int blocks = static_cast<int>(std::min<int64_t>((total + 255) / 256, 148 * 8));
    append_kernel<<<blocks, 256, 0, stream>>>(ap);
    FA_CHECK_CUDA(cudaGetLastError());
  }

  // ---- 2. attend ----
  if (!uses_decode_kernel(p)) {
    // many query rows per KV head: tiled tcgen05 forward over the cache
    FaFwdParams f = {};
    f.q = p->q; f.k = p->k_cache; f.v = p->v_cache; f.o = p->o; f.lse = p->lse;
    f.q_batch_stride = p->q_batch_stride; f.q_row_stride = p->q_row_stride; f.q_head_stride = p->q_head_stride;
    f.k_batch_stride = p->kc_batch_stride; f.k_row_stride = p->kc_row_stride; f.k_head_stride = p->kc_head_stride;
    f.v_batch_stride = p->vc_batch_stride; f.v_row_stride = p->vc_row_stride; f.v_head_stride = p->vc_head_stride;
    f.o_batch_stride = p->o_batch_stride; f.o_row_stride = p->o_row_stride; f.o_head_stride = p->o_head_stride;
    f.lse_row_stride = p->seqlen_q;
    f.b = p->b; f.seqlen_q = p->seqlen_q; f.seqlen_k = p->seqlen_cache;
    f.h = p->h; f.h_k = p->h_k; f.d = p->d;
    f.k_batch = p->cache_batch;
    f.softmax_scale = p->softmax_scale; f.is_causal = p->is_causal;
    f.seqused_k = p->cache_seqlens;
    f.cache_batch_idx = p->cache_batch_idx;
    f.block_table = p->block_table;
    f.block_table_batch_stride = p->block_table_batch_stride;
    f.page_size = p->block_table ? p->seqlen_cache : 0;
    f.block_table_cols = p->block_table ? p->max_blocks_per_seq : 0;
    return run_fwd(&f, p->seqlen_new, stream, appends, verdict != nullptr);
  }

  const int64_t rows_total = static_cast<int64_t>(p->b) * p->h * p->seqlen_q;
  DecodeParams dp;
  rc = make_tensor_map_4d(&dp.tm_k, p->k_cache, p->d, p->h_k, p->seqlen_cache, p->cache_batch,
                          p->kc_head_stride, p->kc_row_stride, p->kc_batch_stride, kTileTokens,
                          "fa_kvcache: k_cache");
  if (rc != FA_OK) return rc;
  rc = make_tensor_map_4d(&dp.tm_v, p->v_cache, p->d, p->h_k, p->seqlen_cache, p->cache_batch,
                          p->vc_head_stride, p->vc_row_stride, p->vc_batch_stride, kTileTokens,
                          "fa_kvcache: v_cache");
  if (rc != FA_OK) return rc;
  dp.q = static_cast<const __half*>(p->q);
  dp.o = static_cast<__half*>(p->o);
  dp.lse = p->lse;
  dp.o_accum = reinterpret_cast<float*>(scratch);
  dp.lse_accum = scratch != nullptr ? reinterpret_cast<float*>(scratch + plan.lse) : nullptr;
  dp.q_batch_stride = p->q_batch_stride; dp.q_row_stride = p->q_row_stride; dp.q_head_stride = p->q_head_stride;
  dp.o_batch_stride = p->o_batch_stride; dp.o_row_stride = p->o_row_stride; dp.o_head_stride = p->o_head_stride;
  dp.seqlen_q = p->seqlen_q; dp.seqlen_new = p->seqlen_new; dp.h = p->h; dp.h_k = p->h_k;
  dp.group = p->h / p->h_k;
  dp.rows_total = rows_total;
  dp.scale_log2 = p->softmax_scale * kLog2e;
  dp.is_causal = p->is_causal;
  dp.cache_seqlens = p->cache_seqlens;
  dp.cache_batch_idx = p->cache_batch_idx;
  dp.block_table = p->block_table;
  dp.block_table_batch_stride = p->block_table_batch_stride;
  dp.page_size = p->seqlen_cache;
  dp.capacity = capacity_tokens(p);
  dp.num_splits = plan.splits;
  dp.chunk_tiles = plan.chunk;
  dp.b = p->b;
  dp.arrivals = arrivals;
  dp.checked = verdict != nullptr;
  dp.status = device_status_ptr();
  if (plan.balanced) {
    const dim3 grid(p->h_k, balanced_shares(p));
    const bool overlap = appends || num_arrivals > 0;
    return p->d == 128 ? launch_decode<128, decode_balanced_kernel<128>>(dp, grid, overlap, stream)
                       : launch_decode<64, decode_balanced_kernel<64>>(dp, grid, overlap, stream);
  }
  const dim3 grid(plan.splits, p->h_k, p->b);
  rc = p->d == 128 ? launch_decode<128, decode_split_kernel<128>>(dp, grid, appends, stream)
                   : launch_decode<64, decode_split_kernel<64>>(dp, grid, appends, stream);
  if (rc != FA_OK) return rc;

  // ---- 3. merge ----
  if (plan.splits > 1)
    return launch_combine(dp.o_accum, dp.lse_accum, p->o, p->lse, rows_total, plan.splits, p->h, p->seqlen_q, p->d,
                          p->o_batch_stride, p->o_row_stride, p->o_head_stride, stream, true);
  return FA_OK;
}
}  // namespace
}  // namespace fa

extern "C" int fa_kvcache(const FaKvcacheParams* p, fa_stream_t stream) {
  return fa::run_kvcache(p, nullptr, 0, static_cast<cudaStream_t>(stream));
}

extern "C" int fa_kvcache_checked(const FaKvcacheParams* p, int32_t* verdict, int32_t token, fa_stream_t stream) {
  using namespace fa;
  FA_CHECK_ARG(verdict != nullptr && token >= 0 && token < (1 << 30), "fa_kvcache_checked: verdict is NULL or token out of range");
  return run_kvcache(p, verdict, token, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------------
// fa_kvcache_noalloc: the same KV-cache step for hosts that cannot allocate device memory.
//
// Who needs it: a serving loop whose device memory pool is frozen after start-up, a plugin that runs
// inside another runtime's callback or graph node where cudaMalloc is not allowed, a language binding
// that can launch but not allocate.  The split partials (O fp32, LSE) then live in the array below,
// which is part of the library image: every GPU that loads the library holds these 32 MiB until exit.
//
// `g_noalloc_scratch` is a device symbol.  In host code its name is only a host-side stand-in for the
// device array, not a device address, so it must never be passed to a kernel as it is; the device
// address is looked up once per device with cudaGetSymbolAddress (with that device current) and that
// pointer is what the kernels receive.
// ---------------------------------------------------------------------------------------------
namespace fa {
namespace {

static __device__ __align__(256) unsigned char g_noalloc_scratch[FA_KVCACHE_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevicesNoAlloc = 64;
void* g_noalloc_ptr[kMaxDevicesNoAlloc] = {};
std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device (set-up on the first call per device).
int noalloc_scratch_ptr(void** out) {
  int dev = 0;
  FA_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevicesNoAlloc)
    return set_error(FA_ERR_UNSUPPORTED, "fa_kvcache_noalloc: device index out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    FA_CHECK_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    if (ptr == nullptr) return set_error(FA_ERR_CUDA, "fa_kvcache_noalloc: scratch symbol has no device address");
    g_noalloc_ptr[dev] = ptr;
  }
  *out = g_noalloc_ptr[dev];
  return FA_OK;
}

}  // namespace
}  // namespace fa

extern "C" int fa_kvcache_noalloc(const FaKvcacheParams* p, fa_stream_t stream) {
  using namespace fa;
  int rc = validate(p, "fa_kvcache_noalloc");
  if (rc != FA_OK) return rc;
  const size_t need = fa_kvcache_workspace_bytes(p);
  if (need > FA_KVCACHE_NOALLOC_SCRATCH_BYTES)
    return set_error(FA_ERR_WORKSPACE,
                     "fa_kvcache_noalloc: this call needs " + std::to_string(need) +
                         " bytes of split scratch, more than the built-in " +
                         std::to_string(static_cast<size_t>(FA_KVCACHE_NOALLOC_SCRATCH_BYTES)) +
                         " bytes; use fewer splits or fa_kvcache() with a caller-owned workspace");
  rc = check_device_sm100();
  if (rc != FA_OK) return rc;
  void* scratch = nullptr;
  rc = noalloc_scratch_ptr(&scratch);
  if (rc != FA_OK) return rc;
  FaKvcacheParams q = *p;
  q.workspace = scratch;
  q.workspace_bytes = FA_KVCACHE_NOALLOC_SCRATCH_BYTES;
  return fa_kvcache(&q, stream);
}
