// Sparse MLA forward for at most 64 heads (sm_100a): ONE CTA per query, D = 576 or 512, DV = 512.  Same semantics as the SM-pair
// kernel in sparse_mla_fwd_pair.cu, which takes 128 heads as the M dimension of every MMA and so spends half of it on rows that
// do not exist here (a tile of 64 keys takes a PAIR of SMs about 1.25 us whether the second CTA has heads or not).
//
//   * S = Q K^T: M = 64 heads, N = 32 keys of a tile, A = Q (dims 0..383 from tensor memory, the rest from shared memory), B = the
//     gathered rows.  M = 64 runs at half the tensor rate, but it puts a head's scores into one thread: the softmax needs no
//     exchange at all.
//   * O^T = V^T P^T: M = 128 of the 512 output dims (four MMAs), N = 64 heads: full rate.  A = V^T is the gathered tile itself
//     (MN-major), B = P as the softmax wrote it.  The accumulator has one output dim per lane and the heads in its columns, so
//     a rescale multiplies columns by factors that the softmax leaves in shared memory.
// What bounds it: ~1300 clocks per tile of 32 keys, the time from a stage's refill to its release (gather ~1000, Q K^T ~2000 with
// two in flight, softmax ~1100, P V ~600) over five (D = 512: six) stages, with 6.6 TB/s of rows coming out of L2.  Sending Q
// through the ring as the pair kernel does, instead of ~4000 clocks of loads at a unit's end, changed neither by more than
// the runs differ (310 -> 305, 976 -> 976 us).  Tiles of 32 keys rather than 64 are what gives the ring its stages.
// Measured (CUDA events, 8192 queries of 64 heads with 128 + 512 keys / 2 x 777 queries with 1024 keys): the pair kernel 1640 /
// 485 us; one Q K^T issuer, one softmax group 1230 / 457; two issuers 1058 / 334; two softmax groups, Q in tensor memory for one
// or two more stages, lists one unit ahead 990 / 321; Q in whole sectors, its second half requested before the rest 976 / 310.
//
// Persistent, one CTA per SM; work units as in the pair kernel (a query or one of the shares of its key tiles).
// Warp roles (19 warps): two groups of 4 softmax + epilogue, 4 gather, 4 Q loaders (+ tile lists), two Q K^T issuers (even and odd tiles: one
// issues while the other waits and fences, ~500 clocks), P V issuer.
#include "fwd_common.cuh"
#include "launch_util.h"
#include "params.h"
#include "ptx.cuh"

namespace dsa {

namespace nw {
constexpr int kD = 576, kDV = 512;
constexpr int kHeads = 64;
constexpr int kBK = 32;                                // keys per tile
// topk <= 2048.  Longer lists keep the pair kernel: not one has been timed here (masks and lists of 8192 keys would fit).
constexpr int kMaxTiles = 64;
constexpr int kQTmemChunks = 6;                        // Q dims 0..383 are a tensor-memory operand, the rest stays in shared memory
constexpr uint32_t kChunk = kBK * 128;                 // 4096: 32 keys x 64 dims, 128-byte swizzle
constexpr uint32_t kQChunk = kHeads * 128;             // 8192: 64 heads x 64 dims
constexpr uint32_t kPBytes = kHeads * 128;             // two tiles' P side by side: 64 heads x (32 + 32) keys
template <bool kRope>
struct Cfg {
  static constexpr int kChunks = kRope ? 9 : 8;
  static constexpr int kQSmemChunks = kChunks - kQTmemChunks;
  static constexpr int kStages = kRope ? 5 : 6;
  static constexpr uint32_t kStageBytes = kChunks * kChunk;
  static constexpr uint32_t kOffQ = kStages * kStageBytes;
  static constexpr uint32_t kOffP = kOffQ + kQSmemChunks * kQChunk;
  static constexpr uint32_t kOffMask = kOffP + kPBytes;              // [2][kMaxTiles] validity masks (per unit parity)
  static constexpr uint32_t kOffList = kOffMask + 2 * kMaxTiles * 4; // [2][kMaxTiles] tile numbers
  static constexpr uint32_t kOffFactor = kOffList + 2 * kMaxTiles;   // [4][64] rescale factors (tile number mod 4)
  static constexpr uint32_t kOffRef = kOffFactor + 4 * kHeads * 4;   // [2][64] reference maxima, [2][64] row sums (per softmax group)
  static constexpr uint32_t kOffInfo = kOffRef + 4 * kHeads * 4;  // [2] tile counts, start status, tensor-memory address
  static constexpr uint32_t kOffBar = kOffInfo + 16;
  static constexpr uint32_t kSmemBytes = kOffBar + 256;
  static_assert(kSmemBytes <= 232448, "shared memory per CTA");
};
constexpr int kGatherWarp = 8, kQWarp = 12, kQkWarp = 16, kQkWarpB = 17;   // Q K^T of the even / odd tiles; the P V issuer is warp 18
constexpr int kThreads = 608;
constexpr uint32_t kColO = 0, kColS = 256, kColQ = 320;  // O^T: four accumulators of 64 columns | S: two buffers of 32 | Q 192
constexpr int kSBufs = 2;
constexpr float kRescaleThreshold = 8.0f;              // log2 units: P stays below 2^8
// named barriers: the two softmax groups, the gather warps, hand-over of a row block's reference maximum (4 per direction), all softmax warps
constexpr uint32_t kGroupBarrier = 1, kGatherBarrier = 3, kHandBarrier = 4, kSoftmaxBarrier = 12;
constexpr int kMaxStages = 6;
constexpr int kBarKvFull = 0;                          // [6] count 128: cp.async completion of the gather threads
constexpr int kBarKvEmpty = kMaxStages;                // [6] count 1: commit after the P V MMAs of the stage
constexpr int kBarSFull = 2 * kMaxStages;              // [2] count 1: commit after the Q K^T MMAs
constexpr int kBarSFree = kBarSFull + 2;               // [2] count 4: the softmax warps have read the scores
constexpr int kBarPReady = kBarSFull + 4;              // [2] count 4: P is written and O rescaled
constexpr int kBarPFree = kBarSFull + 6;               // [2] count 1: commit after the P V MMAs of a tile
constexpr int kBarQTmem = kBarSFull + 8;               // count 4: the tensor-memory part of the unit's Q is there
constexpr int kBarQReady = kBarSFull + 9;              // count 128: cp.async completion of the rest
constexpr int kBarQFree = kBarSFull + 10;              // count 2: commits of both issuers after their last Q K^T of the unit
constexpr int kBarOFree = kBarSFull + 11;              // count 8: the softmax warps have read the unit's output
constexpr int kBarInfoFull = kBarSFull + 12;           // [2] count 1: a unit's tile list is published
constexpr int kBarInfoEmpty = kBarSFull + 14;          // [2] count 15: softmax 8, gather 4, issuers 3
constexpr int kBarCount = kBarSFull + 16;
static_assert(kBarCount * 8 <= 256, "barrier region");
}  // namespace nw

// Named barrier of `nthreads` threads that also tells every one of them whether any came with `pred` set.
__device__ __forceinline__ bool named_bar_any(uint32_t id, uint32_t nthreads, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(nthreads), "r"(static_cast<uint32_t>(pred))
      : "memory");
  return r != 0;
}

// 32-byte load (a whole sector); volatile: it stays in front of the wait that follows it.
__device__ __forceinline__ void ld_global_nc_32b(const uint8_t* src, uint32_t* v) {
  asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(src));
}

__device__ __forceinline__ void named_bar_arrive(uint32_t id, uint32_t nthreads) {
  asm volatile("barrier.cta.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

template <bool kBF16, bool kRope>
__global__ void __launch_bounds__(nw::kThreads, 1) sparse_mla_fwd_narrow_kernel(const FwdParams p) {
  using namespace nw;
  using C = Cfg<kRope>;
  constexpr int kChunks = C::kChunks, kStages = C::kStages;
  constexpr int kRowBytes = kRope ? kD * 2 : kDV * 2;
  using T = typename std::conditional<kBF16, __nv_bfloat16, __half>::type;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sBase = smem_u32(smem);
  if (sBase & 1023u) {  // the swizzled operand tiles need the alignment; same in every CTA of the launch
    if (threadIdx.x == 0) atomicCAS(p.status, kStatusOk, kStatusBadLayout);
    return;
  }
  const uint32_t sQ = sBase + C::kOffQ, sP = sBase + C::kOffP;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint32_t* masks = reinterpret_cast<uint32_t*>(smem + C::kOffMask);
  uint8_t* tile_list = smem + C::kOffList;
  float* factors = reinterpret_cast<float*>(smem + C::kOffFactor);
  float* refs = reinterpret_cast<float*>(smem + C::kOffRef);
  float* sums = refs + 2 * kHeads;                                  // (the first 64 become the final scales)
  int* info = reinterpret_cast<int*>(smem + C::kOffInfo);          // [0..1] tile counts, [2] start status, [3] tensor memory
  auto bar = [&](int slot) { return bars + slot; };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nsplit = p.nsplit > 1 ? p.nsplit : 1;
  const int queries = p.B * p.S;
  const int split_rows = nsplit > 1 ? ((p.split_queries > 0 && p.split_queries < queries) ? p.split_queries : queries) : 0;
  const int split_units = split_rows * nsplit;
  const int num_units = split_units + queries - split_rows;
  const int ntiles = (p.topk + kBK - 1) / kBK;
  auto unit_of = [&](int k) { return num_units - 1 - static_cast<int>(blockIdx.x) - k * static_cast<int>(gridDim.x); };
  auto query_and_share = [&](int u, int* share, int* shares) {
    if (u < split_units) {
      const int q = u / nsplit;
      *share = u - q * nsplit;
      *shares = nsplit;
      return q;
    }
    *share = 0;
    *shares = 1;
    return split_rows + (u - split_units);
  };

  // ---- setup ------------------------------------------------------------------------------------------
  if (tid == 0) {
    info[0] = info[1] = 0;
    info[2] = *reinterpret_cast<volatile int*>(p.status);
    for (int i = 0; i < kStages; ++i) { mbar_init(bar(kBarKvFull + i), 128); mbar_init(bar(kBarKvEmpty + i), 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(kBarSFull + i), 1); mbar_init(bar(kBarSFree + i), 4);
      mbar_init(bar(kBarPReady + i), 4); mbar_init(bar(kBarPFree + i), 1);
      mbar_init(bar(kBarInfoFull + i), 1); mbar_init(bar(kBarInfoEmpty + i), 15);
    }
    mbar_init(bar(kBarQTmem), 4); mbar_init(bar(kBarQReady), 128); mbar_init(bar(kBarQFree), 2); mbar_init(bar(kBarOFree), 8);
    mbar_init_fence();
  }
  if (warp == kQkWarp) {
    tmem_alloc(reinterpret_cast<uint32_t*>(info + 3), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = static_cast<uint32_t>(info[3]);
  const uint32_t tO = tmem_base + kColO, tS = tmem_base + kColS, tQ = tmem_base + kColQ;
  const bool run_all = info[2] == kStatusOk;
  bool ok = true;
  // Does index `idx` of a unit's list take part?  (Keys from two pools: inside its pool; see FwdParams::kv2.)
  auto takes_part = [&](const RowCtx& ctx, int idx) {
    if constexpr (!kRope) {
      if (p.kv2) return idx >= 0 && (idx & (kPool2Bit - 1)) < ((idx & kPool2Bit) ? p.kv2_rows : p.S_kv);
    }
    return index_valid(ctx, idx);
  };
  auto wait_all = [&](int slot, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar(slot), parity, p.status)); };
  auto wait_all_idle = [&](int slot, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait<true>(bar(slot), parity, p.status)); };

  if (warp < kGatherWarp) {
    // ================================ softmax + epilogue ============================================
    // Two groups of four warps take alternate tiles: a tile's softmax is a chain of ~1700 clocks from "scores there" to the next
    // tile's, longer than its MMAs.  What a tile needs from the one before is the reference maximum only, which the warps of
    // the same rows hand each other as soon as they have it; every group keeps the sum of its own tiles.
    // M = 64 accumulators occupy half of the lanes: lane l < 16 of warp w holds head 16 w + l (the others carry no data).  For
    // the output the thread is the lane of one of the four dims 128 a + 32 w + l.  A failed wait clears `ok` but does not
    // leave the loops (the partner warps would wait at the named barriers).
    const int w4 = warp & 3, grp = warp >> 2;
    const bool act = lane < 16;
    const int m = 16 * w4 + (lane & 15);
    const uint32_t lane_base = static_cast<uint32_t>(w4 * 32) << 16;
    int g0 = 0;
    for (int k = 0; run_all; ++k) {
      const int unit = unit_of(k);
      if (unit < 0) break;
      int share, shares;
      const int bt = query_and_share(unit, &share, &shares);
      const int qp = k & 1;
      if (ok) ok = wait_all(kBarInfoFull + qp, (k >> 1) & 1);
      const int nvt = info[qp];
      float m_own = -INFINITY, l = 0.f;   // reference of this group's last tile, sum of its tiles relative to it
      for (int it = (g0 ^ grp) & 1; it < nvt; it += 2) {
        const int g = g0 + it;
        const uint32_t mask = masks[qp * kMaxTiles + tile_list[qp * kMaxTiles + it]];
        const int sb = g & 1, pb = g & 1;
        uint32_t sc[32];
        if (ok) ok = wait_all(kBarSFull + sb, (g >> 1) & 1);
        tc_fence_after();
        tmem_ld32(tS + sb * kBK + lane_base, sc);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kBarSFree + sb));
        if (mask != 0xffffffffu) {  // scores of keys that do not take part count as -inf: their exponentials are exact zeros
#pragma unroll
          for (int j = 0; j < 32; ++j) sc[j] = ((mask >> j) & 1u) ? sc[j] : 0xff800000u;
        }
        float m4[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) m4[j] = fmaxf(__uint_as_float(sc[2 * j]), __uint_as_float(sc[2 * j + 1]));
#pragma unroll
        for (int j = 4; j < 16; ++j) m4[j & 3] = fmax3(m4[j & 3], __uint_as_float(sc[2 * j]), __uint_as_float(sc[2 * j + 1]));
        const float mx = fmaxf(fmax3(m4[0], m4[1], m4[2]), m4[3]) * p.scale_log2;
        // online softmax with a lazily updated reference maximum
        float m_prev = -INFINITY;
        if (it > 0) {
          named_bar_sync(kHandBarrier + (grp ^ 1) * 4 + w4, 64);
          m_prev = refs[(grp ^ 1) * kHeads + m];
        }
        float factor = 1.f, m_used = m_prev;
        if (mx > m_prev + kRescaleThreshold || m_prev == -INFINITY) {
          factor = (m_prev == -INFINITY) ? 0.f : exp2f(m_prev - mx);
          m_used = mx;
        }
        if (act) {
          refs[grp * kHeads + m] = m_used;
          factors[(g & 3) * kHeads + m] = factor;
        }
        if (it + 1 < nvt) named_bar_arrive(kHandBarrier + grp * 4 + w4, 64);
        const float neg = (m_used == -INFINITY) ? 0.f : -m_used;
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), neg2 = make_float2(neg, neg);
        float2 sum2 = make_float2(0.f, 0.f);
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 x = ffma2(make_float2(__uint_as_float(sc[2 * j]), __uint_as_float(sc[2 * j + 1])), scale2, neg2);
          const float2 e = make_float2(exp2f(x.x), exp2f(x.y));
          sum2 = fadd2(sum2, e);
          pk[j] = pack2<kBF16>(e.x, e.y);
        }
        l = l * ((m_own == -INFINITY) ? 0.f : exp2f(m_own - m_used)) + (sum2.x + sum2.y);
        m_own = m_used;
        const bool rescale = named_bar_any(kGroupBarrier + grp, 128, act && factor != 1.f);
        // P's buffer: its last reader were the P V MMAs of tile g - 2
        if (g >= 2 && ok) ok = wait_all(kBarPFree + pb, ((g >> 1) + 1) & 1);
        if (rescale && it > 0) {
          // O must be quiescent: the P V MMAs of the previous tile are done.  (Waited for on that tile's P barrier: its phase
          // before, tile g - 3, completed before that of tile g - 2, which has just been waited for.)
          if (ok) ok = wait_all(kBarPFree + ((g - 1) & 1), ((g - 1) >> 1) & 1);
          tc_fence_after();
#pragma unroll 1
          for (int cc = 0; cc < 8; ++cc) {  // 32 heads of one of the four accumulators
            uint32_t o[32];
            tmem_ld32(tO + lane_base + cc * 32, o);
            tmem_wait_ld();
            const float4* f4 = reinterpret_cast<const float4*>(factors + (g & 3) * kHeads + (cc & 1) * 32);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 f = f4[j];
              o[4 * j] = __float_as_uint(__uint_as_float(o[4 * j]) * f.x);
              o[4 * j + 1] = __float_as_uint(__uint_as_float(o[4 * j + 1]) * f.y);
              o[4 * j + 2] = __float_as_uint(__uint_as_float(o[4 * j + 2]) * f.z);
              o[4 * j + 3] = __float_as_uint(__uint_as_float(o[4 * j + 3]) * f.w);
            }
            tmem_st32(tO + lane_base + cc * 32, o);
          }
          tmem_wait_st();
          tc_fence_before();
        }
        // P: row m, keys 32 pb .. + 31 of the buffer (the issuer executes the proxy fence after it has seen the barrier)
        if (act) {
#pragma unroll
          for (int u = 0; u < 4; ++u) st_shared_v4(sP + sw128_offset(m, 4 * pb + u), pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kBarPReady + pb));
      }
      g0 += nvt;
      // ---- epilogue ----
      const int64_t prow0 = (static_cast<int64_t>(share) * split_rows + bt) * p.H;   // partial rows of a split unit
      const int64_t orow0 = static_cast<int64_t>(bt) * p.H;
      if (nvt == 0) {  // no key takes part (or the query does not exist): zeros, lse = the sink or -inf
        for (int64_t i = tid; i < static_cast<int64_t>(p.H) * kDV / 8; i += 256) {
          if (shares > 1) {
            reinterpret_cast<uint4*>(p.part_out + prow0 * kDV)[2 * i] = make_uint4(0, 0, 0, 0);
            reinterpret_cast<uint4*>(p.part_out + prow0 * kDV)[2 * i + 1] = make_uint4(0, 0, 0, 0);
          } else {
            reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + orow0 * kDV)[i] = make_uint4(0, 0, 0, 0);
          }
        }
        if (tid < p.H) {
          if (shares > 1) p.part_lse[prow0 + tid] = -INFINITY;
          else if (p.lse) p.lse[orow0 + tid] = p.sinks ? p.sinks[tid] : -INFINITY;
        }
      } else {
        // The unit's last two P V are complete, in this order (one of the two barriers is the other group's, whose phases this
        // group does not all wait for: the wait for tile n - 2 makes the parity of tile n - 1's unambiguous).  This also means
        // that every warp is done with the final scales of the unit before.
        if (nvt >= 2 && ok) ok = wait_all(kBarPFree + ((g0 - 2) & 1), ((g0 - 2) >> 1) & 1);
        if (ok) ok = wait_all(kBarPFree + ((g0 - 1) & 1), ((g0 - 1) >> 1) & 1);
        tc_fence_after();
        if (act) {
          refs[grp * kHeads + m] = m_own;
          sums[grp * kHeads + m] = l;
        }
        named_bar_sync(kSoftmaxBarrier, 256);
        if (act && grp == 0) {
          const float m_a = refs[m], m_b = refs[kHeads + m], m_used = fmaxf(m_a, m_b);
          l = (m_a == -INFINITY ? 0.f : sums[m] * exp2f(m_a - m_used)) + (m_b == -INFINITY ? 0.f : sums[kHeads + m] * exp2f(m_b - m_used));
          float inv_l, lse_v;
          if (p.sinks && shares == 1) {  // the sink joins the denominator, relative to the larger of the two (see the pair kernel)
            const float sk = (m < p.H ? p.sinks[m] : -INFINITY) * 1.4426950408889634f;
            const float m_all = fmaxf(m_used, sk), f = exp2f(m_used - m_all);
            const float den = l * f + exp2f(sk - m_all);
            inv_l = f / den;
            lse_v = m_all * 0.6931471805599453f + logf(den);
          } else {
            inv_l = 1.f / l;
            lse_v = m_used * 0.6931471805599453f + logf(l);
          }
          sums[m] = inv_l;   // the final scale of the head
          if (ok && m < p.H) {
            if (shares > 1) p.part_lse[prow0 + m] = lse_v;
            else if (p.lse) p.lse[orow0 + m] = lse_v;
          }
        }
        named_bar_sync(kSoftmaxBarrier, 256);
#pragma unroll 1
        for (int cc = 4 * grp; cc < 4 * grp + 4; ++cc) {  // a group reads two of the four accumulators
          const int h0 = (cc & 1) * 32, dim = 128 * (cc >> 1) + 32 * w4 + lane;
          if (h0 >= p.H) continue;
          uint32_t o[32];
          tmem_ld32(tO + lane_base + cc * 32, o);
          tmem_wait_ld();
          const float4* f4 = reinterpret_cast<const float4*>(sums + h0);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 f = f4[j];
            o[4 * j] = __float_as_uint(__uint_as_float(o[4 * j]) * f.x);
            o[4 * j + 1] = __float_as_uint(__uint_as_float(o[4 * j + 1]) * f.y);
            o[4 * j + 2] = __float_as_uint(__uint_as_float(o[4 * j + 2]) * f.z);
            o[4 * j + 3] = __float_as_uint(__uint_as_float(o[4 * j + 3]) * f.w);
          }
          if (shares > 1) {
            float* dst = p.part_out + (prow0 + h0) * kDV + dim;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (ok && h0 + j < p.H) dst[static_cast<int64_t>(j) * kDV] = __uint_as_float(o[j]);
          } else {
            // Two lanes hold neighbouring dims of every head: they trade so that the even one stores both dims of head j and the
            // odd one both dims of head j + 1 (a store writes 64 contiguous bytes of each of two heads).
            T* dst = reinterpret_cast<T*>(p.out) + (orow0 + h0 + (lane & 1)) * kDV + (dim & ~1);
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const bool odd = lane & 1;
              const float give = __uint_as_float(odd ? o[j] : o[j + 1]), keep = __uint_as_float(odd ? o[j + 1] : o[j]);
              const float got = __shfl_xor_sync(0xffffffffu, give, 1);
              const uint32_t w = odd ? pack2<kBF16>(got, keep) : pack2<kBF16>(keep, got);
              if (ok && h0 + j + (lane & 1) < p.H) *reinterpret_cast<uint32_t*>(dst + static_cast<int64_t>(j) * kDV) = w;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (nvt > 0) mbar_arrive(bar(kBarOFree));
        mbar_arrive(bar(kBarInfoEmpty + qp));
      }
    }
  } else if (warp < kQWarp) {
    // ================================ gather producers ==============================================
    const int pw = warp - kGatherWarp;  // keys [8 pw, 8 pw + 8) of a tile
    const uint8_t* kv_bytes = reinterpret_cast<const uint8_t*>(p.kv);
    // key rows in one piece or in two parts, or from two pools (see FwdParams)
    const size_t row_stride = (kRope && p.kv_rope) ? static_cast<size_t>(kDV * 2) : static_cast<size_t>(kRowBytes);
    const uint8_t* last_base = (kRope && p.kv_rope) ? reinterpret_cast<const uint8_t*>(p.kv_rope) : kv_bytes + 8 * 128;
    const size_t last_stride = (kRope && p.kv_rope) ? static_cast<size_t>((kD - kDV) * 2) : static_cast<size_t>(kRowBytes);
    int g = 0;
    for (int k = 0; run_all; ++k) {
      const int unit = unit_of(k);
      if (unit < 0) break;
      int share, shares;
      const int bt = query_and_share(unit, &share, &shares);
      const int qp = k & 1;
      const RowCtx ctx = make_row_ctx(p, bt);
      if (ok) ok = wait_all_idle(kBarInfoFull + qp, (k >> 1) & 1);
      const int nvt = ok ? info[qp] : 0;
      // lane l looks up key 8 pw + (l & 7); index two tiles ahead, row number one tile ahead: neither load's latency is in the
      // warp's per-tile period
      auto load_idx = [&](int it) {
        const int slot = it < nvt ? tile_list[qp * kMaxTiles + it] * kBK + pw * 8 + (lane & 7) : p.topk;
        return slot < p.topk ? __ldg(ctx.idx_row + slot) : -1;
      };
      auto row_of = [&](int idx) {
        if (!takes_part(ctx, idx)) return -1;
        if constexpr (!kRope) {
          if (p.kv2) return idx;
        }
        return static_cast<int>(kv_row(p, ctx.b, idx));
      };
      int idx_next = load_idx(0);
      int row_next = row_of(idx_next);
      idx_next = load_idx(1);
      for (int it = 0; it < nvt; ++it, ++g) {
        const int s = g % kStages;
        const int my_row = row_next;
        row_next = row_of(idx_next);
        idx_next = load_idx(it + 2);
        if (g >= kStages && ok) ok = mbar_wait<true>(bar(kBarKvEmpty + s), ((g / kStages) + 1) & 1, p.status);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) continue;
        const uint32_t stage = sBase + s * C::kStageBytes;
#pragma unroll
        for (int gh = 0; gh < 2; ++gh) {  // one instruction copies one 64-dim chunk (128 bytes, 8 lanes) of four keys
          const int kl = 4 * gh + (lane >> 3);
          const int row = __shfl_sync(0xffffffffu, my_row, kl);
          const uint32_t dst = stage + sw128_offset(pw * 8 + kl, lane & 7);
          const uint32_t nbytes = row < 0 ? 0u : 16u;   // a key that does not take part: zeros
          size_t r0 = static_cast<size_t>(row < 0 ? 0 : row);
          const uint8_t* base = kv_bytes;
          if constexpr (!kRope) {
            if (p.kv2 && row >= kPool2Bit) {
              base = reinterpret_cast<const uint8_t*>(p.kv2);
              r0 -= kPool2Bit;
            }
          }
          const uint8_t* src = base + r0 * row_stride + (lane & 7) * 16;
#pragma unroll
          for (int c = 0; c < 8; ++c) cp_async16(dst + c * kChunk, src + c * 128, nbytes);
          if (kRope) cp_async16(dst + 8 * kChunk, last_base + r0 * last_stride + (lane & 7) * 16, nbytes);
        }
        cp_async_arrive_noinc(bar(kBarKvFull + s));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kBarInfoEmpty + qp));
    }
    cp_async_wait<0>();
  } else if (warp < kQkWarp) {
    // ================================ Q loaders =====================================================
    // Dims 0..383 become the tensor-memory A operand (48 KB of shared memory are free for another stage or two): lane l < 16 of warp w needs row 16 w + l.  It
    // holds dims 0..191 of it and lane l + 16 the other half, in registers, the first half of it requested before the previous
    // unit's last Q K^T is complete.  The rest follows by cp.async; the issuers start on the first part meanwhile.
    const int qt = tid - kQWarp * 32, xw = warp - kQWarp;
    const bool two = kRope && p.q_rope;
    const int q_stride = two ? kDV * 2 : kRowBytes, r_stride = two ? (kD - kDV) * 2 : kRowBytes;
    const uint8_t* q_bytes = reinterpret_cast<const uint8_t*>(p.q);
    const uint8_t* r_bytes = two ? reinterpret_cast<const uint8_t*>(p.q_rope) : q_bytes + kDV * 2;
    const uint32_t lane_base = static_cast<uint32_t>(xw * 32) << 16;
    const int trow = 16 * xw + (lane & 15);
    // Validity masks and tile list of unit number k, published for the other warps.  One unit ahead: the chain of loads (lengths,
    // indices) takes several thousand clocks, during which the ring would run dry at every unit's end.  Runs whole whatever
    // `ok` is (these warps meet at a named barrier in it).
    auto build_list = [&](int k) {
      const int unit = unit_of(k);
      if (unit < 0) return;
      int share, shares;
      const int bt = query_and_share(unit, &share, &shares);
      const int qp = k & 1;
      const RowCtx ctx = make_row_ctx(p, bt);
      if (k >= 2 && ok) ok = wait_all_idle(kBarInfoEmpty + qp, ((k >> 1) + 1) & 1);
      for (int t0 = xw; t0 < ntiles; t0 += 32) {  // indices of eight tiles are loaded before the first of them is used
        int idx[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int slot = (t0 + 4 * u) * kBK + lane;
          idx[u] = slot < p.topk ? __ldg(ctx.idx_row + slot) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint32_t bits = __ballot_sync(0xffffffffu, ctx.active && takes_part(ctx, idx[u]));
          if (lane == 0 && t0 + 4 * u < ntiles) masks[qp * kMaxTiles + t0 + 4 * u] = bits;
        }
      }
      named_bar_sync(kGatherBarrier, 128);
      if (xw == 0) {
        int n = 0;
        for (int base = 0; base < ntiles; base += 32) {
          const int tile = base + lane;
          const bool nonempty = tile < ntiles && masks[qp * kMaxTiles + tile] != 0u;
          const uint32_t bal = __ballot_sync(0xffffffffu, nonempty);
          if (nonempty) tile_list[qp * kMaxTiles + n + __popc(bal & ((1u << lane) - 1u))] = static_cast<uint8_t>(tile);
          n += __popc(bal);
        }
        if (shares > 1) {  // this unit's share of the list moves to the front (in chunks of 32, reading before writing)
          const int lo = static_cast<int>(static_cast<long long>(n) * share / shares);
          const int hi = static_cast<int>(static_cast<long long>(n) * (share + 1) / shares);
          __syncwarp();
          for (int base = 0; base < hi - lo; base += 32) {
            const int i = base + lane;
            const uint8_t v = i < hi - lo ? tile_list[qp * kMaxTiles + lo + i] : 0;
            __syncwarp();
            if (i < hi - lo) tile_list[qp * kMaxTiles + i] = v;
            __syncwarp();
          }
          n = hi - lo;
        }
        if (lane == 0) info[qp] = n;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kBarInfoFull + qp));
      }
      named_bar_sync(kGatherBarrier, 128);
    };
    if (run_all) build_list(0);
    int ne = 0;
    for (int k = 0; run_all; ++k) {
      const int unit = unit_of(k);
      if (unit < 0) break;
      int share, shares;
      const int64_t row0 = static_cast<int64_t>(query_and_share(unit, &share, &shares)) * p.H;
      const int qp = k & 1;
      const int nvt = info[qp];   // written by the first of these warps
      if (nvt > 0) {
        uint32_t w[48];
        // (a row without a head reads the last one's: its scores and output rows are never stored)
        const uint8_t* src = q_bytes + (row0 + (trow < p.H ? trow : p.H - 1)) * q_stride + (lane >> 4) * 384;
        auto load_half = [&](int half) {   // dims 96 half .. + 95 of this lane's 192
#pragma unroll
          for (int u = 0; u < 6; ++u) ld_global_nc_32b(src + half * 192 + u * 32, w + 8 * u);
        };
        auto store_half = [&](int half) {
          tmem_st32(tQ + lane_base + half * 48, w);
          tmem_st16(tQ + lane_base + half * 48 + 32, w + 32);
          uint32_t x[48];
#pragma unroll
          for (int j = 0; j < 48; ++j) x[j] = __shfl_down_sync(0xffffffffu, w[j], 16);
          tmem_st32(tQ + lane_base + 96 + half * 48, x);
          tmem_st16(tQ + lane_base + 96 + half * 48 + 32, x + 32);
        };
        load_half(0);
        if (ne > 0 && ok) ok = wait_all(kBarQFree, (ne - 1) & 1);
        ++ne;
        tc_fence_after();
        store_half(0);
        load_half(1);
#pragma unroll 3
        for (int i = qt; i < C::kQSmemChunks * 512; i += 128) {
          const int unit16 = i & 7, row = (i >> 3) & 63, c = kQTmemChunks + (i >> 9);
          const bool v = row < p.H;
          const uint8_t* from = c < 8 ? q_bytes + (row0 + row) * q_stride + c * 128 : r_bytes + (row0 + row) * r_stride;
          cp_async16(sQ + (i >> 9) * kQChunk + sw128_offset(row, unit16), v ? from + unit16 * 16 : q_bytes, v ? 16u : 0u);
        }
        cp_async_arrive_noinc(bar(kBarQReady));
        store_half(1);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kBarQTmem));
      }
      const int next = unit_of(k + 1);
      if (next >= 0) {
        const int64_t nrow0 = static_cast<int64_t>(query_and_share(next, &share, &shares)) * p.H;
        for (int off = qt * 128; off < p.H * q_stride; off += 128 * 128) prefetch_l2(q_bytes + nrow0 * q_stride + off);
        if (two)
          for (int off = qt * 128; off < p.H * r_stride; off += 128 * 128) prefetch_l2(r_bytes + nrow0 * r_stride + off);
      }
      build_list(k + 1);
    }
    cp_async_wait<0>();
  } else if (warp == kQkWarp || warp == kQkWarpB) {
    // ================================ Q K^T issuers =================================================
    // the whole warp walks the loops and waits, converged; one elected lane issues through predicated instructions
    const int par = warp == kQkWarp ? 0 : 1;
    constexpr uint32_t idesc = make_idesc_f16(kBF16, kHeads, kBK, 0, 0);
    const uint32_t go = elect_one_lane();
    const uint64_t da0 = make_smem_desc(sQ, 16, 1024, kSwizzle128B);
    int g = 0, ne = 0;
    for (int k = 0; run_all && ok; ++k) {
      if (unit_of(k) < 0) break;
      const int qp = k & 1;
      if (!wait_all(kBarInfoFull + qp, (k >> 1) & 1)) { ok = false; break; }
      const int nvt = info[qp];
      const int first = (g ^ par) & 1;                                    // this warp's first tile of the unit ...
      const int last = nvt - 1 - ((g + nvt - 1 - par) & 1);               // ... and its last one
      if (nvt > 0) {
        // (waited for also when no tile of the unit is mine: a skipped phase would satisfy the next parity test too early)
        if (!wait_all(kBarQTmem, ne & 1)) { ok = false; break; }
        if (first >= nvt && !wait_all(kBarQReady, ne & 1)) { ok = false; break; }
        ++ne;
        // No tile of this unit is mine: done with its Q at once.  A commit, not a plain arrive, which could overtake the commit
        // that ended this warp's previous unit.
        if (first >= nvt) umma_commit_if(go, bar(kBarQFree));
      }
      for (int it = first; it < nvt; it += 2) {
        const int gg = g + it, s = gg % kStages, sb = par;
        if (!wait_all(kBarKvFull + s, (gg / kStages) & 1)) { ok = false; break; }
        if (gg >= kSBufs && !wait_all(kBarSFree + sb, ((gg >> 1) + 1) & 1)) { ok = false; break; }
        fence_proxy_async_smem();  // Q and the gathered rows were written by cp.async of other threads
        tc_fence_after();
        const uint64_t db0 = make_smem_desc(sBase + s * C::kStageBytes, 16, 1024, kSwizzle128B);
#pragma unroll 1
        for (int c = 0; c < kQTmemChunks; ++c) {
#pragma unroll
          for (int kq = 0; kq < 4; ++kq)
            umma_ts_if(go, tS + sb * kBK, tQ + (c * 4 + kq) * 8, db0 + ((c * kChunk + kq * 32) >> 4), idesc, (c | kq) != 0);
        }
        if (it == first) {  // the rest of Q has landed
          if (!wait_all(kBarQReady, (ne - 1) & 1)) { ok = false; break; }
          fence_proxy_async_smem();
        }
#pragma unroll 1
        for (int c = 0; c < C::kQSmemChunks; ++c) {
#pragma unroll
          for (int kq = 0; kq < 4; ++kq)
            umma_ss_if(go, tS + sb * kBK, da0 + ((c * kQChunk + kq * 32) >> 4), db0 + (((kQTmemChunks + c) * kChunk + kq * 32) >> 4), idesc, 1);
        }
        umma_commit_if(go, bar(kBarSFull + sb));
        if (it == last) umma_commit_if(go, bar(kBarQFree));
      }
      if (!ok) break;
      g += nvt;
      __syncwarp();
      if (go) mbar_arrive(bar(kBarInfoEmpty + qp));
    }
  } else {
    // ================================ P V issuer ====================================================
    // O^T[128 dims x 64 heads] += V^T[128 x 32 keys] . P^T[32 x 64]: A MN-major (two 64-dim chunks of the stage, 16 keys = 2048
    // bytes per step), B = the P rows of 64 heads, K-major.
    constexpr uint32_t idesc = make_idesc_f16(kBF16, 128, kHeads, 1, 0);
    const uint32_t go = elect_one_lane();
    int g = 0, ne = 0;
    for (int k = 0; run_all && ok; ++k) {
      if (unit_of(k) < 0) break;
      const int qp = k & 1;
      if (!wait_all(kBarInfoFull + qp, (k >> 1) & 1)) { ok = false; break; }
      const int nvt = info[qp];
      for (int it = 0; it < nvt; ++it, ++g) {
        const int s = g % kStages, pb = g & 1;
        if (!wait_all(kBarKvFull + s, (g / kStages) & 1)) { ok = false; break; }
        if (!wait_all(kBarPReady + pb, (g >> 1) & 1)) { ok = false; break; }
        // the first P V of a unit overwrites O: the output of the unit before must have been read out
        if (it == 0 && ne > 0 && !wait_all(kBarOFree, (ne - 1) & 1)) { ok = false; break; }
        fence_proxy_async_smem();
        tc_fence_after();
        const uint32_t stage = sBase + s * C::kStageBytes;
        const uint64_t dp0 = make_smem_desc(sP, 16, 1024, kSwizzle128B) + ((pb * 64) >> 4);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint64_t dv0 = make_smem_desc(stage + 2 * a * kChunk, kChunk, 1024, kSwizzle128B);
#pragma unroll
          for (int ks = 0; ks < 2; ++ks)
            umma_ss_if(go, tO + a * kHeads, dv0 + ((ks * 2048) >> 4), dp0 + ((ks * 32) >> 4), idesc, (it | ks) != 0);
        }
        umma_commit_if(go, bar(kBarKvEmpty + s));
        umma_commit_if(go, bar(kBarPFree + pb));
      }
      if (!ok) break;
      if (nvt > 0) ++ne;
      __syncwarp();
      if (go) mbar_arrive(bar(kBarInfoEmpty + qp));
    }
  }

  // ---- teardown: every thread comes here, also after a failed wait ------------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == kQkWarp) tmem_dealloc(tmem_base, 512);
}

// -------------------------------------------------------------------------------------------------
// host side
// -------------------------------------------------------------------------------------------------
bool sparse_mla_fwd_narrow_shape(int H, int topk) { return H <= nw::kHeads && topk <= nw::kMaxTiles * nw::kBK; }
bool sparse_mla_fwd_narrow_supported(const FwdParams& p) {
  return sparse_mla_fwd_narrow_shape(p.H, p.topk) && (reinterpret_cast<uintptr_t>(p.q) & 31u) == 0;   // (Q is read in 32-byte pieces)
}

int launch_sparse_mla_fwd_narrow(const FwdParams& p, bool bf16, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t e = current_device_sms(&dev, &sms);
  if (e != cudaSuccess) return static_cast<int>(e);
  const bool rope = p.D == nw::kD;
  auto kern = rope ? (bf16 ? sparse_mla_fwd_narrow_kernel<true, true> : sparse_mla_fwd_narrow_kernel<false, true>)
                   : (bf16 ? sparse_mla_fwd_narrow_kernel<true, false> : sparse_mla_fwd_narrow_kernel<false, false>);
  const uint32_t smem = rope ? nw::Cfg<true>::kSmemBytes : nw::Cfg<false>::kSmemBytes;
  if ((e = ensure_dynamic_smem(kern, dev, static_cast<int>(smem))) != cudaSuccess) return static_cast<int>(e);
  const long long rows = static_cast<long long>(p.B) * p.S;
  const long long split_rows = p.nsplit > 1 ? ((p.split_queries > 0 && p.split_queries < rows) ? p.split_queries : rows) : 0;
  const long long units = split_rows * (p.nsplit > 1 ? p.nsplit : 1) + (rows - split_rows);
  const long long ctas = units < sms ? units : sms;
  kern<<<static_cast<unsigned>(ctas), nw::kThreads, smem, stream>>>(p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dsa
