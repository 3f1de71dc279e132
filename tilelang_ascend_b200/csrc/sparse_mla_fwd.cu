// Sparse MLA forward for sm_100a.
//
// For every query token the kernel gathers the latent KV rows its index list names, computes
// S = sm_scale * Q K^T over all D dims for all heads, an online softmax over the gathered keys, and
// O = P V over the first DV dims, and writes O (input dtype) and the natural-log LSE (fp32).
// Semantics follow ref_sparse_attention_fwd_interface
// (examples/sparse_flash_attention/example_sparse_flash_attn.py:255-292) and the -1 / length rules
// of the paged variant (example_sparse_flash_attn_mask_pa.py:221-238).
//
// Two kernels:
//  * sparse_mla_fwd_tc_kernel  -- D = 576 (or 512, rows without rope dims), DV = 512: tcgen05 MMAs with TMEM accumulators,
//    one 2-CTA cluster per (query, block of 128 heads); the two CTAs split the contraction dims of
//    Q K^T and the output columns of P V and exchange partial scores through distributed shared memory.
//  * sparse_mla_fwd_generic_kernel -- any D <= 640 / DV <= 512 (e.g. the GQA example with dim 128):
//    CUDA-core fp32, one warp per head.
#include <stdlib.h>
#include <type_traits>

#include "fwd_common.cuh"
#include "launch_util.h"
#include "params.h"
#include "ptx.cuh"

namespace dsa {

// -------------------------------------------------------------------------------------------------
// tcgen05 kernel: persistent 2-CTA clusters, one (query, block of 128 heads) item at a time
// -------------------------------------------------------------------------------------------------
// TMEM (512 columns x 128 lanes) cannot hold a 128 x 512 fp32 output tile plus a score tile, so the
// two CTAs of a cluster split the work of one query without duplicating any of it:
//   CTA r owns latent dims [256 r, 256 r + 256) and rope dims [512 + 32 r, 544 + 32 r):
//     * it gathers only those 576 bytes of every selected KV row,
//     * computes the PARTIAL scores S_r = Q[:, its dims] . K[:, its dims]^T (contraction split),
//     * sends S_r to its peer through distributed shared memory and adds the peer's S_(1-r),
//     * runs the (identical) online softmax, and
//     * accumulates O[:, 256 r : 256 r + 256] = P . V[:, its latent dims]   (output columns split).
// Per CTA: Q latent dims live in TMEM as the A operand, the Q rope dims in shared memory, KV tiles of 64
// keys in a 4-stage cp.async ring, two score buffers in TMEM that are released as soon as the softmax warps
// have read them, P (bf16) in two shared-memory buffers as the A operand of PV, one receive buffer for the
// peer's partial scores.  Warp roles: 8 softmax warps (32 rows x 32 score columns each), 4 warps that load Q
// and ship the partial scores to the peer CTA, 4 gather warps, one warp issuing the QK^T MMAs and one the PV
// MMAs.
//
// The grid is one cluster per SM pair; cluster c walks the items  n-1-c, n-1-c-C, ...  (late = long queries
// first).  Roles run ahead of each other across items: the gather warps build the next item's tile list and
// start its KV gathers while the current item is still being reduced, the exchange warps load the next Q as
// soon as the last QK^T of the current item is complete, and the first PV of an item only waits for the
// previous item's output tile to be drained.  Tiles are numbered cumulatively (g) over the items of a
// cluster; every ring buffer and barrier phase is a function of g.
namespace tc {
constexpr int kD = 576, kDV = 512;
constexpr int kM = 128;                               // heads per cluster = UMMA M
constexpr int kBK = 64;                               // keys per tile
constexpr int kStages = 4;
constexpr int kHalfDV = 256;                          // output columns (and latent dims) per CTA
constexpr int kMaxTiles = 128;                        // topk <= 8192
constexpr uint32_t kChunkBytes = kBK * 128;           // 8192: 64 keys x 64 dims, 128-byte swizzle
constexpr uint32_t kRopeOff = 4 * kChunkBytes;        // the CTA's 32 rope dims of the 64 keys: rows of 64 bytes, 64-byte swizzle
constexpr uint32_t kStageBytes = kRopeOff + kBK * 64; // 36864: 4 latent chunks + the rope chunk
constexpr uint32_t kQRopeBytes = kM * 64;             // Q rope dims, same 64-byte rows
constexpr uint32_t kXBytes = kM * kBK * 4;            // peer's partial scores [128 x 64] fp32
constexpr uint32_t kPBytes = kM * kBK * 2;            // P of one tile [128 x 64] bf16/fp16, 128-byte swizzle (A operand of PV)
constexpr uint32_t kOffQRope = kStages * kStageBytes;             // 147456
constexpr uint32_t kOffX = kOffQRope + kQRopeBytes;               // 155648
constexpr uint32_t kOffP = kOffX + kXBytes;                       // 188416: two P buffers
constexpr uint32_t kOffBar = kOffP + 2 * kPBytes;                 // 221184
constexpr uint32_t kOffHalfMax = kOffBar + 512;                   // [3][2][128] floats exchanged between the two column halves
constexpr uint32_t kOffMask = kOffHalfMax + 3 * 256 * 4;          // [2][kMaxTiles] 64-bit validity masks (per item parity)
constexpr uint32_t kOffList = kOffMask + 2 * kMaxTiles * 8;       // [2][kMaxTiles] 16-bit tile ids
constexpr uint32_t kOffInfo = kOffList + 2 * kMaxTiles * 2;       // [2] {tile count, run flag}
constexpr uint32_t kSmemBytes = kOffInfo + 64 + 1024;             // + slack to align the base to 1024 B
constexpr int kSoftmaxWarps = 8;                      // warp w: rows 32 (w & 3) .. +31, score columns 32 (w >> 2) .. +31
constexpr int kFirstExchangeWarp = 8;                 // warp w sends rows 32 (w & 3) .. +31 of the partial scores to the peer
constexpr int kFirstGatherWarp = 12;
constexpr int kMmaWarp = 16;                          // QK^T issuer
constexpr int kPvWarp = 17;                           // second MMA-issuing warp (PV), on another scheduler than the QK issuer
constexpr int kThreads = 576;                         // 8 softmax warps, 4 exchange warps, 4 gather warps, 2 MMA warps
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColO = 0, kColS = 256, kColQ = 384;  // O 256 | S0 64 | S1 64 | Q latent 128 (256 bf16 dims)
static_assert(kSmemBytes <= 232448, "shared memory per CTA");
constexpr float kRescaleThreshold = 8.0f;             // log2 units: P stays below 2^8
constexpr uint32_t kGatherBarrier = 5;                // named barrier of the 128 gather threads
}  // namespace tc

// kRope = false: rows of 512 dims without the 64 rope dims (D = DV = 512: the keys ARE the values, as in DeepSeek-V4's
// sparse_flash_mla); the rope buffers are zero-filled and the two rope MMA steps are left out, everything else is unchanged.
template <bool kBF16, bool kRope>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(tc::kThreads, 1) sparse_mla_fwd_tc_kernel(const FwdParams p) {
  using namespace tc;
  constexpr int kRowBytes = kRope ? kD * 2 : kDV * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sBase = smem_u32(smem);
  const uint32_t sQRope = sBase + kOffQRope, sX = sBase + kOffX;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffBar);
  uint64_t* kv_full = bars;         // [4] count 128: cp.async completion of the gather threads
  uint64_t* kv_empty = bars + 4;    // [4] count 1: commit after the PV MMAs of the stage
  uint64_t* s_full = bars + 8;      // [2] count 1: commit after the QK MMAs
  uint64_t* p_full = bars + 40;     // [2] count 8: softmax warps wrote P into this buffer (one barrier per buffer: the
                                    // softmax warps are not in step with each other, one may be a tile ahead of another)
  uint64_t* x_full = bars + 12;     // [4][2] count 1 + 4096 transaction bytes: 32 rows x 32 columns of the peer's partial scores landed here
  uint64_t* x_empty = bars + 20;    // [4][2] count 1: the peer's softmax warp of these rows and columns has read what this CTA sent
  uint64_t* info_full = bars + 28;  // [2] count 1: tile list of an item published by the gather warps
  uint64_t* info_empty = bars + 30; // [2] count 14: both MMA threads, softmax and exchange warps are done with the item's tile list
  uint64_t* q_ready = bars + 32;    // count 4: the exchange warps put the item's Q into TMEM / shared memory
  uint64_t* o_free = bars + 33;     // count 8: the softmax warps drained the previous item's output tile from TMEM
  uint64_t* s_free = bars + 34;     // [2] count 8: the softmax warps have read the scores of this buffer out of TMEM
  uint64_t* p_free = bars + 38;     // [2] count 1: commit after the PV MMAs that read this P buffer (= that tile's PV is complete)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 36);
  int* start_status = reinterpret_cast<int*>(bars + 37);
  float* halfmax = reinterpret_cast<float*>(smem + kOffHalfMax);
  unsigned long long* masks = reinterpret_cast<unsigned long long*>(smem + kOffMask);
  uint16_t* tile_list = reinterpret_cast<uint16_t*>(smem + kOffList);
  int* info = reinterpret_cast<int*>(smem + kOffInfo);  // [2][2]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();   // which half of the dims / output columns
  const uint32_t peer = rank ^ 1u;
  const int num_clusters = gridDim.x >> 1, cluster_id = blockIdx.x >> 1;
  const int head_blocks = (p.H + kM - 1) / kM;
  const int nsplit = p.nsplit > 1 ? p.nsplit : 1;
  const int num_items = p.B * p.S * head_blocks * nsplit;  // work units: (query, head block, share of the key tiles)
  const int ntiles = (p.topk + kBK - 1) / kBK;
  using T = typename std::conditional<kBF16, __nv_bfloat16, __half>::type;
  // k-th work unit of this cluster (late queries first), or -1; unit = (query, head block) * nsplit + share
  auto item_of = [&](int k) { const int it = num_items - 1 - cluster_id - k * num_clusters; return it; };

  // ---- setup ------------------------------------------------------------------------------------------
  if (tid == 0) {
    *start_status = *reinterpret_cast<volatile int*>(p.status);
    for (int i = 0; i < kStages; ++i) { mbar_init(&kv_full[i], 128); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&info_full[i], 1); mbar_init(&info_empty[i], 2 + kSoftmaxWarps + 4);
      mbar_init(&s_free[i], kSoftmaxWarps); mbar_init(&p_free[i], 1);
    }
    for (int i = 0; i < 8; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
    mbar_init(&p_full[0], kSoftmaxWarps); mbar_init(&p_full[1], kSoftmaxWarps);
    mbar_init(q_ready, 4);
    mbar_init(o_free, kSoftmaxWarps);
    for (int i = 0; i < 4; ++i) info[i] = 0;
    mbar_init_fence();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tO = tmem_base + kColO, tS = tmem_base + kColS, tQ = tmem_base + kColQ;
  // both CTAs must have their barriers initialised before any remote arrive; every thread takes part
  cluster_sync_all();
  const bool run_all = *start_status == kStatusOk;
  bool ok = true;

  if (warp >= kFirstExchangeWarp && warp < kFirstGatherWarp) {
    // ================================ Q loader + score exchange =====================================
    // Row r of the item's Q: the CTA's 256 latent dims go to TMEM (lane = row, column c = dims 2c, 2c+1), its 32
    // rope dims to shared memory.  Then, per tile, the CTA's partial scores of 32 rows x 64 keys go to the peer
    // as soon as the QK MMAs are done, in 16-byte units laid out [unit][row]; st.async signals the peer's barrier.
    const int q4 = warp & 3;
    const int r = q4 * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t peer_x = map_to_cta(sX, peer);
    const uint32_t peer_x_full = map_to_cta(smem_u32(x_full), peer);
    // pulls this thread's Q row of an item towards L2 (the CTA's 4 latent lines and its rope line)
    auto prefetch_q = [&](int it_unit) {
      if (it_unit < 0) return;
      const int it_item = it_unit / nsplit;
      const int nbt = it_item / head_blocks, nh = (it_item - nbt * head_blocks) * kM + r;
      if (nh >= p.H) return;
      const uint8_t* nq = reinterpret_cast<const uint8_t*>(p.q) + (static_cast<int64_t>(nbt) * p.H + nh) * kRowBytes;
#pragma unroll
      for (int j = 0; j < 4; ++j) prefetch_l2(nq + rank * 512 + j * 128);
      if (kRope) prefetch_l2(nq + 1024 + rank * 64);
    };
    if (run_all) prefetch_q(item_of(0));  // the first item's rows: behind the wait for its tile list
    int g = 0;
    for (int k = 0; run_all && ok; ++k) {
      const int unit = item_of(k);
      if (unit < 0) break;
      const int item = unit / nsplit;
      const int qp = k & 1;
      const int bt = item / head_blocks, h0 = (item - bt * head_blocks) * kM;
      if (!__all_sync(0xffffffffu, mbar_wait<true>(&info_full[qp], (k >> 1) & 1, p.status))) { ok = false; break; }
      const int nvt = info[qp * 2];
      if (nvt > 0) {
        // all QK MMAs of the previous item are complete (their last s_full was waited for below): Q can be replaced
        const bool row_ok = h0 + r < p.H;
        const uint8_t* qrow = reinterpret_cast<const uint8_t*>(p.q) + (static_cast<int64_t>(bt) * p.H + h0 + (row_ok ? r : 0)) * kRowBytes;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          cp_async16(sQRope + sw64_offset(r, u), kRope ? qrow + 1024 + (4 * rank + u) * 16 : qrow, (row_ok && kRope) ? 16u : 0u);
        cp_async_commit();
#pragma unroll 1
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t w[32];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row_ok) v = __ldg(reinterpret_cast<const uint4*>(qrow + rank * 512 + (cc * 8 + j) * 16));
            w[4 * j] = v.x; w[4 * j + 1] = v.y; w[4 * j + 2] = v.z; w[4 * j + 3] = v.w;
          }
          tmem_st32(tQ + lane_base + cc * 32, w);
        }
        cp_async_wait<0>();
        fence_proxy_async_smem();
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_ready);
      }
      prefetch_q(item_of(k + 1));  // the next item's rows, while this item is being worked on
      for (int it = 0; it < nvt; ++it, ++g) {
        const int sb = g & 1;
        uint32_t v[2][32];
        if (!__all_sync(0xffffffffu, mbar_wait<true>(&s_full[sb], (g >> 1) & 1, p.status))) { ok = false; break; }
        tc_fence_after();
        // both column halves of the rows are read at once; the sends below then only wait for their buffers
        tmem_ld32(tS + sb * kBK + lane_base, v[0]);
        tmem_ld32(tS + sb * kBK + 32 + lane_base, v[1]);
        tmem_wait_ld();
        // The receive buffer is handled in two column halves with their own barriers, so that the peer's first half
        // can be on its way while the second half of the previous tile is still being read there.
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int xb = q4 * 2 + hf;
          // the peer's softmax warp has read this half of tile g-1 out of its receive buffer
          if (g >= 1 && !__all_sync(0xffffffffu, mbar_wait<true>(&x_empty[xb], (g + 1) & 1, p.status))) { ok = false; break; }
          // this CTA's receive barrier is armed once per tile: its previous phase (tile g-1) must be complete first --
          // the peer's credit above says the peer read OUR data, not that ITS data has fully landed here
          if (g >= 1 && !__all_sync(0xffffffffu, mbar_wait<true>(&x_full[xb], (g + 1) & 1, p.status))) { ok = false; break; }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            st_async_v4(peer_x + (8 * hf + j) * (kM * 16) + r * 16, peer_x_full + xb * 8, __uint_as_float(v[hf][4 * j]),
                        __uint_as_float(v[hf][4 * j + 1]), __uint_as_float(v[hf][4 * j + 2]), __uint_as_float(v[hf][4 * j + 3]));
          // Arm this CTA's receive barrier for the same rows and columns only now: its completion then tells the softmax
          // warp of this block three things at once -- the peer's partial scores have landed, this CTA's own QK MMAs of
          // the tile are complete (s_full was waited for above), and this warp has read its copy of these scores out
          // of TMEM (the softmax warps report the score buffer free after their own read).
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_expect_tx(&x_full[xb], 32 * 128);
        }
        if (!ok) break;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&info_empty[qp]);
    }
  } else if (warp >= kFirstGatherWarp && warp < kMmaWarp) {
    // ================================ tile lists + gather producers =================================
    // These warps never leave their loops early: they meet at a named barrier twice per item.
    const int pw = warp - kFirstGatherWarp;  // keys [16 pw, 16 pw + 16) of every tile
    const uint8_t* kv_bytes = reinterpret_cast<const uint8_t*>(p.kv);
    int g = 0;
    for (int k = 0; run_all; ++k) {
      const int unit = item_of(k);
      if (unit < 0) break;
      const int item = unit / nsplit, share = unit - item * nsplit;
      const int qp = k & 1;
      const int bt = item / head_blocks;
      const RowCtx ctx = make_row_ctx(p, bt);
      if (k >= 2 && ok) ok = __all_sync(0xffffffffu, mbar_wait<true>(&info_empty[qp], ((k >> 1) + 1) & 1, p.status));
      // validity masks of all tiles of the item, then the list of tiles with at least one key taking part.  The indices
      // of eight tiles are loaded before the first of them is used, so that their latencies overlap (with a single
      // item per cluster -- decode -- this prologue is not hidden behind a previous item)
      for (int t0 = pw; t0 < ntiles; t0 += 32) {
        int i0[8], i1[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int tile = t0 + 4 * u;
          const int s0 = tile * kBK + lane, s1 = s0 + 32;
          i0[u] = (tile < ntiles && s0 < p.topk) ? __ldg(ctx.idx_row + s0) : -1;
          i1[u] = (tile < ntiles && s1 < p.topk) ? __ldg(ctx.idx_row + s1) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int tile = t0 + 4 * u;
          const uint32_t lo = __ballot_sync(0xffffffffu, ctx.active && index_valid(ctx, i0[u]));
          const uint32_t hi = __ballot_sync(0xffffffffu, ctx.active && index_valid(ctx, i1[u]));
          if (lane == 0 && tile < ntiles) masks[qp * kMaxTiles + tile] = (static_cast<unsigned long long>(hi) << 32) | lo;
        }
      }
      named_bar_sync(kGatherBarrier, 128);
      if (pw == 0) {
        int n = 0;
        for (int base = 0; base < ntiles; base += 32) {
          const int tile = base + lane;
          const bool nonempty = tile < ntiles && masks[qp * kMaxTiles + tile] != 0ull;
          const uint32_t bal = __ballot_sync(0xffffffffu, nonempty);
          if (nonempty) tile_list[qp * kMaxTiles + n + __popc(bal & ((1u << lane) - 1u))] = static_cast<uint16_t>(tile);
          n += __popc(bal);
        }
        if (nsplit > 1) {
          // this unit's share of the list: entries [lo, hi) move to the front (in chunks of 32, reading before writing)
          const int lo = static_cast<int>(static_cast<long long>(n) * share / nsplit);
          const int hi = static_cast<int>(static_cast<long long>(n) * (share + 1) / nsplit);
          __syncwarp();
          for (int base = 0; base < hi - lo; base += 32) {
            const int i = base + lane;
            const uint16_t v = i < hi - lo ? tile_list[qp * kMaxTiles + lo + i] : 0;
            __syncwarp();
            if (i < hi - lo) tile_list[qp * kMaxTiles + i] = v;
            __syncwarp();
          }
          n = hi - lo;
        }
        if (lane == 0) { info[qp * 2] = n; info[qp * 2 + 1] = ctx.active ? 1 : 0; }
        __syncwarp();
        if (lane == 0) mbar_arrive(&info_full[qp]);
      }
      named_bar_sync(kGatherBarrier, 128);
      const int nvt = info[qp * 2];
      for (int it = 0; it < nvt; ++it, ++g) {
        const int tile = tile_list[qp * kMaxTiles + it], s = g % kStages;
        // the row numbers are fetched before the wait for the stage, so their latency is hidden behind it
        const int slot = tile * kBK + pw * 16 + (lane & 15);
        const int my_idx = slot < p.topk ? __ldg(ctx.idx_row + slot) : -1;
        const bool my_valid = index_valid(ctx, my_idx);
        // row number inside kv (lanes 0..15 and 16..31 hold the same 16 keys), -1 for a key that does not take part: it is
        // fetched with a source size of zero, which fills the destination with zeros
        const int my_row = my_valid ? static_cast<int>(kv_row(p, ctx.b, my_idx)) : -1;
        int rows[16];
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) rows[kk] = __shfl_sync(0xffffffffu, my_row, kk);
        if (g >= kStages && ok) ok = mbar_wait<true>(&kv_empty[s], ((g / kStages) + 1) & 1, p.status);
        if (!ok) continue;
        const uint32_t stage = sBase + s * kStageBytes;
        const uint8_t* lat_src = kv_bytes + rank * 512 + lane * 16;
        const uint32_t lat_dst = stage + (lane >> 3) * kChunkBytes + pw * 2048;
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
          const uint32_t row = static_cast<uint32_t>(rows[kk] < 0 ? 0 : rows[kk]);
          cp_async16(lat_dst + sw128_offset(kk, lane & 7), lat_src + static_cast<size_t>(row) * kRowBytes, rows[kk] < 0 ? 0u : 16u);
        }
        // the 64 rope bytes of the 16 keys: 4 lanes per key, two instructions
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int kk = hh * 8 + (lane >> 2);
          const int row = __shfl_sync(0xffffffffu, my_row, kk);
          cp_async16(stage + kRopeOff + sw64_offset(pw * 16 + kk, lane & 3),
                     kv_bytes + static_cast<size_t>(row < 0 ? 0 : row) * kRowBytes + (kRope ? 1024 + (4 * rank + (lane & 3)) * 16 : 0),
                     (row < 0 || !kRope) ? 0u : 16u);
        }
        cp_async_arrive_noinc(&kv_full[s]);
      }
    }
    cp_async_wait<0>();
  } else if (warp == kMmaWarp) {
    // ================================ QK^T issuer ===================================================
    // S_r[128 x 64] = Q[:, dims of this CTA] . K^T : 16 steps with A in TMEM + 2 rope steps with A in smem.
    // Runs ahead of the PV issuer as far as the two score buffers allow.
    if (lane == 0) {
      constexpr uint32_t idesc_qk = make_idesc_f16(kBF16, kM, kBK, 0, 0);
      int g = 0, ne = 0;  // cumulative tile count, number of non-empty items so far
      for (int k = 0; run_all && ok; ++k) {
        const int item = item_of(k);
        if (item < 0) break;
        const int qp = k & 1;
        if (!mbar_wait(&info_full[qp], (k >> 1) & 1, p.status)) { ok = false; break; }
        const int nvt = info[qp * 2];
        if (nvt > 0) {  // items without a key neither load Q nor touch O: their barriers are skipped on both sides
          if (!mbar_wait(q_ready, ne & 1, p.status)) { ok = false; break; }
          ++ne;
        }
        for (int it = 0; ok && it < nvt; ++it, ++g) {
          const int s = g % kStages, sb = g & 1;
          const uint32_t stage = sBase + s * kStageBytes;
          if (!mbar_wait(&kv_full[s], (g / kStages) & 1, p.status)) { ok = false; break; }
          // the softmax warps must have read the scores of tile g-2 out of this buffer
          if (g >= 2 && !mbar_wait(&s_free[sb], ((g >> 1) + 1) & 1, p.status)) { ok = false; break; }
          fence_proxy_async_smem();  // the gathered rows were written by cp.async of other threads
          tc_fence_after();
          const uint64_t db0 = make_smem_desc(stage, 16, 1024, kSwizzle128B);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int kq = 0; kq < 4; ++kq)
              umma_ts(tS + sb * kBK, tQ + (c * 4 + kq) * 8, db0 + ((c * kChunkBytes + kq * 32) >> 4), idesc_qk, (c | kq) != 0);
          }
          const uint64_t da0 = make_smem_desc(sQRope, 16, 512, kSwizzle64B);
          const uint64_t dr0 = make_smem_desc(stage + kRopeOff, 16, 512, kSwizzle64B);
          if constexpr (kRope) {
#pragma unroll
            for (int kq = 0; kq < 2; ++kq) umma_ss(tS + sb * kBK, da0 + ((kq * 32) >> 4), dr0 + ((kq * 32) >> 4), idesc_qk, 1);
          }
          umma_commit(&s_full[sb]);
        }
        if (!ok) break;
        mbar_arrive(&info_empty[qp]);
      }
    }
  } else if (warp == kPvWarp) {
    // ================================ PV issuer =====================================================
    // O_r[128 x 256] += P[128 x 64] . V[64 x 256] : P K-major in shared memory (16 keys = 32 bytes per step), V MN-major.
    if (lane == 0) {
      constexpr uint32_t idesc_pv = make_idesc_f16(kBF16, kM, kHalfDV, 0, 1);
      int g = 0, ne = 0;
      for (int k = 0; run_all && ok; ++k) {
        const int item = item_of(k);
        if (item < 0) break;
        const int qp = k & 1;
        if (!mbar_wait(&info_full[qp], (k >> 1) & 1, p.status)) { ok = false; break; }
        const int nvt = info[qp * 2];
        for (int it = 0; ok && it < nvt; ++it, ++g) {
          if (!mbar_wait(&p_full[g & 1], (g >> 1) & 1, p.status)) { ok = false; break; }
          // the first PV of an item overwrites O: the previous non-empty item's output must have been read out
          if (it == 0 && ne > 0 && !mbar_wait(o_free, (ne - 1) & 1, p.status)) { ok = false; break; }
          fence_proxy_async_smem();
          tc_fence_after();
          const uint32_t stage = sBase + (g % kStages) * kStageBytes;
          const uint64_t db0 = make_smem_desc(stage, kChunkBytes, 1024, kSwizzle128B);
          const uint64_t dp0 = make_smem_desc(sBase + kOffP + (g & 1) * kPBytes, 16, 1024, kSwizzle128B);
#pragma unroll
          for (int ks = 0; ks < kBK / 16; ++ks)
            umma_ss(tO, dp0 + ((ks * 32) >> 4), db0 + ((ks * 2048) >> 4), idesc_pv, (it | ks) != 0);
          umma_commit(&kv_empty[g % kStages]);
          umma_commit(&p_free[g & 1]);
        }
        if (!ok) break;
        if (nvt > 0) ++ne;
        mbar_arrive(&info_empty[qp]);
      }
    }
  } else {
    // ================================ softmax + epilogue ============================================
    // thread = (row r, column half ch): r = TMEM lane, ch selects 32 of the tile's 64 score columns and 128 of the
    // CTA's 256 output columns.  The two warps of a row block combine their row maxima through shared memory and
    // a 64-thread named barrier once per tile; everything else is thread-local.  A failed wait clears `ok` but does
    // not leave the loops (the partner warp would wait at the named barrier): the remaining tiles are walked
    // without waiting.
    const int q4 = warp & 3, ch = warp >> 2;
    const int r = q4 * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t peer_x_empty = map_to_cta(smem_u32(x_empty), peer);
    int g = 0;
    for (int k = 0; run_all; ++k) {
      const int unit = item_of(k);
      if (unit < 0) break;
      const int item = unit / nsplit, share = unit - item * nsplit;
      const int qp = k & 1;
      const int bt = item / head_blocks, h0 = (item - bt * head_blocks) * kM;
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&info_full[qp], (k >> 1) & 1, p.status));
      const int nvt = info[qp * 2];  // read unconditionally: both warps of a row block must walk the same number of tiles
      float m_used = -INFINITY, l = 0.f;
      for (int it = 0; it < nvt; ++it, ++g) {
        const uint32_t mask = static_cast<uint32_t>(masks[qp * kMaxTiles + tile_list[qp * kMaxTiles + it]] >> (32 * ch));
        const int sb = g & 1;
        uint32_t sc[32];  // scores as raw bits (TMEM loads), used as floats below
        // one wait per tile: x_full completes after the peer's partial scores landed AND this CTA's exchange warp of the
        // same rows armed it, which it does after s_full and after its own read of the scores (see there)
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&x_full[q4 * 2 + ch], g & 1, p.status));
        // Pull the peer's partial scores (16-byte units, layout [unit][row]) into registers and return the credit before
        // anything else: the peer's next send into the single receive buffer waits for it.  The credit must not overtake
        // the loads.  A warp issues its instructions in order and a store cannot issue before its source register is
        // filled, so a (dummy) store of a word derived from all eight loads, placed before the arrive, holds the arrive
        // back until the values are in registers.  (Naming the value as an unused operand of the arrive would not: the
        // instruction would not read the register.)
        float4 xr[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) xr[j] = *reinterpret_cast<const float4*>(smem + kOffX + (8 * ch + j) * (kM * 16) + r * 16);
        {
          uint32_t dep = 0;
#pragma unroll
          for (int j = 0; j < 8; ++j) dep ^= __float_as_uint(xr[j].x);
          st_shared_u32_volatile(sBase + kOffInfo + 32 + warp * 4, dep);
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(peer_x_empty + (q4 * 2 + ch) * 8);
        }
        tc_fence_after();
        tmem_ld32(tS + sb * kBK + ch * 32 + lane_base, sc);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free[sb]);  // the QK^T of tile g+2 may overwrite the buffer
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 a = fadd2(make_float2(__uint_as_float(sc[4 * j]), __uint_as_float(sc[4 * j + 1])), make_float2(xr[j].x, xr[j].y));
          const float2 b = fadd2(make_float2(__uint_as_float(sc[4 * j + 2]), __uint_as_float(sc[4 * j + 3])), make_float2(xr[j].z, xr[j].w));
          sc[4 * j] = __float_as_uint(a.x); sc[4 * j + 1] = __float_as_uint(a.y);
          sc[4 * j + 2] = __float_as_uint(b.x); sc[4 * j + 3] = __float_as_uint(b.y);
        }
        const bool full = mask == 0xffffffffu;
        float mx;
        if (full) {
          float m4[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) m4[j] = fmaxf(__uint_as_float(sc[2 * j]), __uint_as_float(sc[2 * j + 1]));
#pragma unroll
          for (int j = 4; j < 16; ++j) m4[j & 3] = fmax3(m4[j & 3], __uint_as_float(sc[2 * j]), __uint_as_float(sc[2 * j + 1]));
          mx = fmaxf(fmax3(m4[0], m4[1], m4[2]), m4[3]);
        } else {
          mx = -INFINITY;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if ((mask >> j) & 1u) mx = fmaxf(mx, __uint_as_float(sc[j]));
        }
        // the other column half of this row lives in the warp with the same (w & 3): combine the maxima through shared
        // memory (double-buffered by tile parity)
        float* slot = halfmax + (g & 1) * 256;
        slot[ch * 128 + r] = mx;
        // exponentials relative to this half's own maximum, before the barrier: the MUFU work overlaps the wait for the
        // partner warp, and only one correction factor per thread is left for afterwards
        const float m_loc = mx * p.scale_log2;                      // -inf when no key of this half takes part
        const float neg_loc = (mx == -INFINITY) ? 0.f : -m_loc;
        float pe[32];
        float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), neg2 = make_float2(neg_loc, neg_loc);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 x = ffma2(make_float2(__uint_as_float(sc[2 * j]), __uint_as_float(sc[2 * j + 1])), scale2, neg2);
          float2 e = make_float2(exp2f(x.x), exp2f(x.y));
          if (!full) {
            e.x = ((mask >> (2 * j)) & 1u) ? e.x : 0.f;
            e.y = ((mask >> (2 * j + 1)) & 1u) ? e.y : 0.f;
          }
          pe[2 * j] = e.x; pe[2 * j + 1] = e.y;
          sum2[j & 1] = fadd2(sum2[j & 1], e);
        }
        named_bar_sync(1 + q4, 64);
        mx = fmaxf(slot[r], slot[128 + r]) * p.scale_log2;
        // ---- online softmax with a lazily updated reference maximum (identical in both warps of the row block) ----
        float factor = 1.f;
        if (mx > m_used + kRescaleThreshold || m_used == -INFINITY) {
          factor = (m_used == -INFINITY) ? 0.f : exp2f(m_used - mx);
          m_used = mx;
        }
        if (it > 0 && __any_sync(0xffffffffu, factor != 1.f)) {
          // O must be quiescent: the PV MMAs of the previous tile are done.  (Waited for on that tile's P buffer barrier:
          // its phase before -- tile g-3 -- was already waited for when P of tile g-1 was written, so the parity
          // test cannot be fooled by a barrier that is two phases behind.)
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&p_free[(g - 1) & 1], ((g - 1) >> 1) & 1, p.status));
          tc_fence_after();
          uint32_t o[32];
#pragma unroll 1
          for (int cc = 4 * ch; cc < 4 * ch + 4; ++cc) {  // this thread's half of the output columns
            tmem_ld32(tO + lane_base + cc * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * factor);
            tmem_st32(tO + lane_base + cc * 32, o);
          }
          tmem_wait_st();
          tc_fence_before();
        }
        const float corr = exp2f(m_loc - m_used);                  // <= 2^8; 0 for a half without keys
        l = l * factor + ((sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y)) * corr;
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 v = fmul2(make_float2(pe[2 * j], pe[2 * j + 1]), make_float2(corr, corr));
          pk[j] = pack2<kBF16>(v.x, v.y);
        }
        // P goes to shared memory as the K-major A operand of the PV MMAs: row r, keys 32 ch .. 32 ch + 31 = four 16-byte
        // units.  The buffer was last read by the PV MMAs of tile g-2.
        if (g >= 2 && ok) ok = __all_sync(0xffffffffu, mbar_wait(&p_free[sb], ((g >> 1) + 1) & 1, p.status));
        const uint32_t prow = sBase + kOffP + sb * kPBytes;
#pragma unroll
        for (int u = 0; u < 4; ++u) st_shared_v4(prow + sw128_offset(r, 4 * ch + u), pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
        fence_proxy_async_smem();  // read by the tensor core (async proxy)
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[sb]);
      }
      // ---- epilogue: each thread normalises and stores its 128 of the CTA's 256 output columns ----
      if (nvt > 0) {  // row sum = sum of the two column halves, exchanged like the maxima
        float* slot = halfmax + 2 * 256;
        slot[ch * 128 + r] = l;
        named_bar_sync(1 + q4, 64);
        l = slot[r] + slot[128 + r];  // (the slot is rewritten only after the next item's barriers)
      }
      const int h = h0 + r;
      T* orow = reinterpret_cast<T*>(p.out) + (static_cast<int64_t>(bt) * p.H + h) * kDV + rank * kHalfDV;
      // split-KV: this unit's normalised partial result and its log-sum-exp go to the workspace instead
      const int64_t prow_index = (static_cast<int64_t>(share) * p.B * p.S + bt) * p.H + h;
      float* part_row = nsplit > 1 ? p.part_out + prow_index * kDV + rank * kHalfDV : nullptr;
      if (nsplit > 1 && nvt == 0) {
        if (h < p.H) {  // nothing to add from this share (also for queries that do not exist: the combine step writes zeros)
          for (int j = 32 * ch; j < 32 * ch + 32; ++j) reinterpret_cast<float4*>(part_row)[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (rank == 0 && ch == 0) p.part_lse[prow_index] = -INFINITY;
        }
      } else if (nvt == 0) {  // no key takes part, or the query does not exist (beyond q_len_b): out = 0, lse = -inf
        if (h < p.H) {
          for (int j = 16 * ch; j < 16 * ch + 16; ++j) reinterpret_cast<uint4*>(orow)[j] = make_uint4(0, 0, 0, 0);
          if (rank == 0 && ch == 0 && p.lse) p.lse[static_cast<int64_t>(bt) * p.H + h] = -INFINITY;
        }
      } else if (nvt > 0) {
        // the last PV of the item is complete (same barrier and argument as for the rescale above)
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&p_free[(g - 1) & 1], ((g - 1) >> 1) & 1, p.status));
        tc_fence_after();
        const float inv_l = 1.f / l;
        uint32_t v[32];
#pragma unroll 1
        for (int cc = 4 * ch; cc < 4 * ch + 4; ++cc) {
          tmem_ld32(tO + lane_base + cc * 32, v);
          tmem_wait_ld();
          if (ok && h < p.H && nsplit > 1) {
#pragma unroll
            for (int gq = 0; gq < 8; ++gq)
              reinterpret_cast<float4*>(part_row + cc * 32)[gq] =
                  make_float4(__uint_as_float(v[4 * gq]) * inv_l, __uint_as_float(v[4 * gq + 1]) * inv_l, __uint_as_float(v[4 * gq + 2]) * inv_l,
                              __uint_as_float(v[4 * gq + 3]) * inv_l);
          } else if (ok && h < p.H) {
#pragma unroll
            for (int gq = 0; gq < 4; ++gq) {
              uint4 w;
              w.x = pack2<kBF16>(__uint_as_float(v[8 * gq + 0]) * inv_l, __uint_as_float(v[8 * gq + 1]) * inv_l);
              w.y = pack2<kBF16>(__uint_as_float(v[8 * gq + 2]) * inv_l, __uint_as_float(v[8 * gq + 3]) * inv_l);
              w.z = pack2<kBF16>(__uint_as_float(v[8 * gq + 4]) * inv_l, __uint_as_float(v[8 * gq + 5]) * inv_l);
              w.w = pack2<kBF16>(__uint_as_float(v[8 * gq + 6]) * inv_l, __uint_as_float(v[8 * gq + 7]) * inv_l);
              reinterpret_cast<uint4*>(orow + cc * 32)[gq] = w;
            }
          }
        }
        if (ok && rank == 0 && ch == 0 && h < p.H) {
          const float lse_v = m_used * 0.6931471805599453f + logf(l);
          if (nsplit > 1) p.part_lse[prow_index] = lse_v;
          else if (p.lse) p.lse[static_cast<int64_t>(bt) * p.H + h] = lse_v;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (nvt > 0) mbar_arrive(o_free);  // the output tile may be overwritten by the next item's first PV
        mbar_arrive(&info_empty[qp]);      // the item's tile list is no longer needed here
      }
    }
  }

  // ---- teardown: every thread of both CTAs comes here, also after a failed wait -----------------------
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
  cluster_sync_all();  // no CTA leaves while its peer may still write into its shared memory
}

// -------------------------------------------------------------------------------------------------
// generic CUDA-core kernel: one warp per head, fp32 arithmetic
// -------------------------------------------------------------------------------------------------
namespace gen {
constexpr int kBK = 32, kHeadsPerCta = 8, kMaxD = 640, kMaxDV = 512;
}

template <typename T>
__global__ void __launch_bounds__(256) sparse_mla_fwd_generic_kernel(const FwdParams p) {
  using namespace gen;
  extern __shared__ uint8_t smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // [kBK][D]
  __shared__ int s_idx[kBK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head_groups = (p.H + kHeadsPerCta - 1) / kHeadsPerCta;
  const int bt = blockIdx.x / head_groups;
  const int h = (blockIdx.x - bt * head_groups) * kHeadsPerCta + warp;
  const RowCtx ctx = make_row_ctx(p, bt);
  const int D = p.D, DV = p.DV;
  const bool head_ok = h < p.H;
  if (!ctx.active) {  // a query beyond q_len_b: out = 0, lse = -inf (uniform across the CTA)
    if (head_ok) {
      T* orow = reinterpret_cast<T*>(p.out) + (static_cast<int64_t>(bt) * p.H + h) * DV;
      for (int d = lane; d < DV; d += 32) orow[d] = static_cast<T>(0.f);
      if (lane == 0 && p.lse) p.lse[static_cast<int64_t>(bt) * p.H + h] = -INFINITY;
    }
    return;
  }

  float qreg[kMaxD / 32];
  float acc[kMaxDV / 32];
  const T* qrow = reinterpret_cast<const T*>(p.q) + (static_cast<int64_t>(bt) * p.H + (head_ok ? h : 0)) * D;
#pragma unroll
  for (int i = 0; i < kMaxD / 32; ++i) {
    const int d = lane + 32 * i;
    qreg[i] = (head_ok && d < D) ? static_cast<float>(qrow[d]) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kMaxDV / 32; ++i) acc[i] = 0.f;
  float m = -INFINITY, l = 0.f;

  const int ntiles = (p.topk + kBK - 1) / kBK;
  for (int tile_i = 0; tile_i < ntiles; ++tile_i) {
    __syncthreads();
    if (tid < kBK) {
      const int slot = tile_i * kBK + tid;
      const int idx = slot < p.topk ? ctx.idx_row[slot] : -1;
      s_idx[tid] = index_valid(ctx, idx) ? idx : -1;
    }
    __syncthreads();
    const int units = D / 8;  // 16-byte units per row (D % 8 == 0 is checked on the host)
    for (int u = tid; u < kBK * units; u += blockDim.x) {
      const int key = u / units, unit = u - key * units;
      const int idx = s_idx[key];
      uint4 val = make_uint4(0, 0, 0, 0);
      if (idx >= 0)
        val = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.kv) + kv_row(p, ctx.b, idx) * D + unit * 8);
      *reinterpret_cast<uint4*>(tile + key * D + unit * 8) = val;
    }
    __syncthreads();
    for (int j = 0; j < kBK; ++j) {
      if (s_idx[j] < 0) continue;  // uniform across the CTA
      const T* krow = tile + j * D;
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < kMaxD / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < D) dot += qreg[i] * static_cast<float>(krow[d]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      const float x = dot * p.scale_log2;
      const float m_new = fmaxf(m, x);
      const float f = (m == -INFINITY) ? 0.f : exp2f(m - m_new);
      const float pj = exp2f(x - m_new);
      l = l * f + pj;
      m = m_new;
#pragma unroll
      for (int i = 0; i < kMaxDV / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < DV) acc[i] = acc[i] * f + pj * static_cast<float>(krow[d]);
      }
    }
  }
  if (!head_ok) return;
  T* orow = reinterpret_cast<T*>(p.out) + (static_cast<int64_t>(bt) * p.H + h) * DV;
  const float inv_l = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int i = 0; i < kMaxDV / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < DV) orow[d] = static_cast<T>(acc[i] * inv_l);
  }
  if (lane == 0 && p.lse) p.lse[static_cast<int64_t>(bt) * p.H + h] = l > 0.f ? m * 0.6931471805599453f + logf(l) : -INFINITY;
}

// -------------------------------------------------------------------------------------------------
// split-KV combine: out = sum_s w_s part_out[s],  w_s = exp(lse_s - lse),  lse = log sum_s exp(lse_s)
// -------------------------------------------------------------------------------------------------
// (an attention sink of the row's head, sinks [H] or null, joins the denominator like a share without a value row)
template <typename T>
__global__ void __launch_bounds__(128) sparse_mla_fwd_combine_kernel(const float* __restrict__ part_out, const float* __restrict__ part_lse,
                                                                     T* __restrict__ out, float* __restrict__ lse, int64_t rows, int nsplit, int dv,
                                                                     const float* __restrict__ sinks, int H) {
  const int64_t row = blockIdx.x;
  const float sk = sinks ? sinks[row % H] : -INFINITY;
  float m = sk;
  for (int s = 0; s < nsplit; ++s) m = fmaxf(m, part_lse[s * rows + row]);
  float wsum = (m == -INFINITY) ? 0.f : expf(sk - m);
  for (int s = 0; s < nsplit; ++s) wsum += (m == -INFINITY) ? 0.f : expf(part_lse[s * rows + row] - m);
  for (int c = threadIdx.x * 4; c < dv; c += blockDim.x * 4) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < nsplit; ++s) {
      const float ls = part_lse[s * rows + row];
      if (ls == -INFINITY) continue;
      const float w = expf(ls - m) / wsum;
      const float4 v = *reinterpret_cast<const float4*>(part_out + (s * rows + row) * dv + c);
      acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
    }
    T* o = out + row * dv + c;
    o[0] = static_cast<T>(acc.x); o[1] = static_cast<T>(acc.y); o[2] = static_cast<T>(acc.z); o[3] = static_cast<T>(acc.w);
  }
  if (threadIdx.x == 0 && lse) lse[row] = (m == -INFINITY) ? -INFINITY : m + logf(wsum);
}

// -------------------------------------------------------------------------------------------------
// host launchers (return a cudaError_t as int; 0 = launched)
// -------------------------------------------------------------------------------------------------
bool sparse_mla_fwd_tc_supported(const FwdParams& p) {
  // (row numbers inside kv are kept in 32 bits by the gather warps)
  return (p.D == tc::kD || p.D == tc::kDV) && p.DV == tc::kDV && p.topk <= tc::kMaxTiles * tc::kBK && static_cast<long long>(p.B) * p.S_kv <= 0x7fffffffLL;
}

bool sparse_mla_fwd_pair_supported(const FwdParams& p);
int launch_sparse_mla_fwd_pair(const FwdParams& p, bool bf16, cudaStream_t stream);

static int launch_combine(const FwdParams& p, bool bf16, cudaStream_t stream) {
  // the rows that were split: all queries, or the first split_queries of them
  const int64_t all = static_cast<int64_t>(p.B) * p.S;
  const int64_t rows = ((p.split_queries > 0 && p.split_queries < all) ? p.split_queries : all) * p.H;
  if (bf16)
    sparse_mla_fwd_combine_kernel<__nv_bfloat16><<<static_cast<unsigned>(rows), 128, 0, stream>>>(p.part_out, p.part_lse, reinterpret_cast<__nv_bfloat16*>(p.out),
                                                                                                p.lse, rows, p.nsplit, p.DV, p.sinks, p.H);
  else
    sparse_mla_fwd_combine_kernel<__half><<<static_cast<unsigned>(rows), 128, 0, stream>>>(p.part_out, p.part_lse, reinterpret_cast<__half*>(p.out), p.lse,
                                                                                         rows, p.nsplit, p.DV, p.sinks, p.H);
  return static_cast<int>(cudaGetLastError());
}

// The SM-pair kernel followed, for a split call, by the combine kernel (for callers that need that kernel and no other).
int launch_sparse_mla_fwd_pair_combined(const FwdParams& p, bool bf16, cudaStream_t stream) {
  int rc = launch_sparse_mla_fwd_pair(p, bf16, stream);
  if (rc != 0 || p.nsplit <= 1) return rc;
  return launch_combine(p, bf16, stream);
}

int launch_sparse_mla_fwd_tc(const FwdParams& p, bool bf16, cudaStream_t stream) {
  // The kernel of sparse_mla_fwd_pair.cu (cta_group::2 MMAs) is the default; DSA_FWD_KERNEL=split in the environment selects
  // the kernel below (each CTA all 128 heads and half of the dims), which the tests use as a cross-check.
  const char* which = getenv("DSA_FWD_KERNEL");
  const bool tail_only = p.nsplit > 1 && p.split_queries > 0 && p.split_queries < static_cast<long long>(p.B) * p.S;  // pair kernel only
  if ((!(which && which[0] == 's') || tail_only) && sparse_mla_fwd_pair_supported(p)) {
    int rc = launch_sparse_mla_fwd_pair(p, bf16, stream);
    if (rc != 0 || p.nsplit <= 1) return rc;
    return launch_combine(p, bf16, stream);
  }
  const bool rope = p.D == tc::kD;
  auto kern = rope ? (bf16 ? sparse_mla_fwd_tc_kernel<true, true> : sparse_mla_fwd_tc_kernel<false, true>)
                   : (bf16 ? sparse_mla_fwd_tc_kernel<true, false> : sparse_mla_fwd_tc_kernel<false, false>);
  int dev = 0, sms = 0;
  cudaError_t e = current_device_sms(&dev, &sms);
  if (e != cudaSuccess) return static_cast<int>(e);
  if ((e = ensure_dynamic_smem(kern, dev, static_cast<int>(tc::kSmemBytes))) != cudaSuccess) return static_cast<int>(e);
  // persistent: one 2-CTA cluster per SM pair, each walking its share of the (query, head block) items
  const long long items = static_cast<long long>(p.B) * p.S * ((p.H + tc::kM - 1) / tc::kM);
  long long clusters = sms / 2 > 0 ? sms / 2 : 1;
  const long long units = items * (p.nsplit > 1 ? p.nsplit : 1);
  if (clusters > units) clusters = units;
  kern<<<dim3(static_cast<unsigned>(2 * clusters)), tc::kThreads, tc::kSmemBytes, stream>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess || p.nsplit <= 1) return static_cast<int>(e);
  const int64_t rows = static_cast<int64_t>(p.B) * p.S * p.H;
  if (bf16)
    sparse_mla_fwd_combine_kernel<__nv_bfloat16><<<static_cast<unsigned>(rows), 128, 0, stream>>>(p.part_out, p.part_lse, reinterpret_cast<__nv_bfloat16*>(p.out),
                                                                                                p.lse, rows, p.nsplit, p.DV, p.sinks, p.H);
  else
    sparse_mla_fwd_combine_kernel<__half><<<static_cast<unsigned>(rows), 128, 0, stream>>>(p.part_out, p.part_lse, reinterpret_cast<__half*>(p.out), p.lse,
                                                                                         rows, p.nsplit, p.DV, p.sinks, p.H);
  return static_cast<int>(cudaGetLastError());
}

// Number of shares that fills the GPU's cluster slots when there are fewer (query, head block) items than slots.
bool sparse_mla_fwd_narrow_shape(int H, int topk);

int sparse_mla_fwd_auto_nsplit(const FwdParams& p, int sms) {
  const long long items = static_cast<long long>(p.B) * p.S * ((p.H + tc::kM - 1) / tc::kM);
  const long long slots = sparse_mla_fwd_narrow_shape(p.H, p.topk) ? sms : sms / 2;   // a CTA or a pair of CTAs per item
  const long long clusters = slots > 0 ? slots : 1;
  const int ntiles = (p.topk + tc::kBK - 1) / tc::kBK;
  long long ns = clusters / (items > 0 ? items : 1);
  if (ns > 16) ns = 16;
  if (ns > ntiles / 2) ns = ntiles / 2;  // at least two tiles per share
  return ns < 2 ? 1 : static_cast<int>(ns);
}

int launch_sparse_mla_fwd_generic(const FwdParams& p, bool bf16, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(gen::kBK) * p.D * 2;
  // (query, group of 8 heads) on grid.x: B * S is not limited to 65535
  dim3 grid(static_cast<unsigned>(static_cast<long long>(p.B) * p.S * ((p.H + gen::kHeadsPerCta - 1) / gen::kHeadsPerCta)));
  if (bf16)
    sparse_mla_fwd_generic_kernel<__nv_bfloat16><<<grid, 256, smem, stream>>>(p);
  else
    sparse_mla_fwd_generic_kernel<__half><<<grid, 256, smem, stream>>>(p);
  return static_cast<int>(cudaGetLastError());
}


}  // namespace dsa
