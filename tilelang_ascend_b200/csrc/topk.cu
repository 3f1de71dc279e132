// Row-wise top-k selector: value buckets, or radix select + sort of the survivors.
//
// For each fp32 row the kernel emits the indices of the `top_k` largest candidates in descending
// score order, equal scores in ascending index order (the stable-sort rule of
// cpu_lightning_indexer, examples/deepseek_v4/lightning_indexer.py:316-325); candidates are the first
// `limit[row]` entries whose score is > -1e30; slots left over hold -1 (value -inf).  For rows of
// distinct values this is also torch.topk's answer (examples/topk_selector/example_topk_selector.py:57-58).
//
// One CTA per row.  The ordered form buckets the row's values (see topk_bucket_kernel).  A row whose values crowd into few
// buckets, and the unordered form, take the radix select: the row is converted to order-preserving 32-bit keys in shared
// memory, four 8-bit most-significant-digit-first histogram passes find the k-th largest key, an index-ordered
// compaction (per-warp counts, prefix over warps, ordered write) takes everything above it plus the
// lowest-index ties, and the <= k survivors are sorted by buckets (bucket_sort) or by a stable least-significant-digit radix
// sort: the compaction leaves equal keys in ascending index order and a stable sort keeps them so.  With ordered = 0 the
// sort is left out and the selected SET comes out in ascending index order (what the sparse attention after the indexer
// needs, and the order in which its row gather is most local).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "launch_util.h"
#include "ptx.cuh"

namespace dsa {

namespace topk {
constexpr int kSelectThreads = 512;               // 4 rows (CTAs) per SM hide each other's barrier phases
constexpr int kBuckets = 4096;
constexpr int kMaxPerBucket = 96;                 // fuller buckets: radix select instead (bucket_sort: a second level of buckets)
constexpr size_t kMaxSmemBytes = 220 * 1024;       // rows whose keys do not fit are streamed from global memory
// dynamic, of a CTA of a cluster, beside 8 KB static: two of them per SM (228 KB), or one that has the SM alone (227 KB)
constexpr size_t kMaxClusterSmemBytes = 105 * 1024, kMaxLoneClusterSmemBytes = 219 * 1024;
// candidates of a row of n that each of c CTAs takes at most: whole groups of four
__host__ __device__ constexpr int cluster_slice(int n, int c) { return ((n + 3) / 4 + c - 1) / c * 4; }
}  // namespace topk

__device__ __forceinline__ uint32_t float_to_key(float f) {
  uint32_t u = __float_as_uint(f);
  if (u == 0x80000000u) u = 0u;  // -0.0 ties with +0.0, as in a floating-point comparison
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

// Shared memory of the CTA that a mapped address names.
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void st_cluster_u64(uint32_t addr, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t atom_add_cluster_u32(uint32_t addr, uint32_t v) {
  uint32_t old;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
  return old;
}

// Orders cnt survivors of the radix select by key, descending, equal keys by ascending index.  src holds them in ascending index
// order and receives the result; dst [cnt] and work [2048] are scratch.  False: nothing done, src as it was.
// 1024 equal buckets over the survivors' key range; a bucket of more than kMaxPerBucket elements is cut again, over the range
// of its own keys -- or, when they are all equal, of the indices -- into a share of 1024 fine buckets.  An element's place is
// its bucket's start plus the number of elements of the same bucket in front of it.  4096 rows of 8192 -> 2048 with 30 % of the
// entries at -1e4, whole call: 402 us with the four passes of the radix sort below, 268 with this (211 without any sort).  The
// radix sort stays for rows that crowd inside one fine bucket (mostly equal values and a few others within 2^-10 of the key range;
// the limit on the comparisons is about where the two cost the same) and for keys with few digits:
// `varies` receives the bits in which the keys differ: few distinct values have few of them, and a radix sort that skips the other
// digits is then the faster one (at most two digits: 16-bit scores, small whole numbers; N(0, 1) rounded to quarters, same call: 346 us
// by buckets, 305 by two passes of the radix sort).
template <int kThreads>
__device__ __forceinline__ bool bucket_sort(unsigned long long* src, unsigned long long* dst, uint32_t* work, const int cnt, uint32_t* varies) {
  using namespace topk;
  constexpr int kWarps = kThreads / 32, kCoarse = 1024, kFine = 1024, kPer = kCoarse / kThreads;
  constexpr int kSlots = 8192 / (kMaxPerBucket + 1) + 1;   // buckets that can be that full
  constexpr uint32_t kSlotFlag = 0x80000000u;
  uint32_t *coarse_ct = work, *fine_ct = work + kCoarse;
  __shared__ uint32_t w_a[kWarps], w_b[kWarps], w_c[kWarps];
  __shared__ uint32_t slot_start[kSlots], slot_count[kSlots], slot_kmin[kSlots], slot_kmax[kSlots];
  // largest key (0: all keys equal) | first fine bucket, their number << 16 | fine buckets per unit, fp32 | from "crowded elements
  // before" to the place in the whole order
  __shared__ uint4 slot_fine[kSlots];
  __shared__ uint32_t s_slots, s_cost;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto key_of = [](unsigned long long e) { return static_cast<uint32_t>(e >> 32); };
  auto index_of = [](unsigned long long e) { return 0xffffffffu - static_cast<uint32_t>(e & 0xffffffffull); };
  // replaces the counts c[0..1023] by each(i, elements before i, count)
  auto scan = [&](uint32_t* c, auto&& each) {
    uint32_t v[kPer], mine = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) { v[j] = c[tid * kPer + j]; mine += v[j]; }
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) w_a[warp] = incl;
    __syncthreads();
    uint32_t start = incl - mine;
    for (int w = 0; w < warp; ++w) start += w_a[w];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      c[tid * kPer + j] = each(tid * kPer + j, start, v[j]);
      start += v[j];
    }
    __syncthreads();
  };

  // ---- key range, coarse histogram ----
  uint32_t lo = 0xffffffffu, hi = 0u, bits = 0u;
  const uint32_t key0 = key_of(src[0]);
  for (int i = tid; i < cnt; i += kThreads) {
    const uint32_t k = key_of(src[i]);
    bits |= k ^ key0;
    lo = min(lo, k);
    hi = max(hi, k);
  }
  for (int i = tid; i < kCoarse + kFine; i += kThreads) work[i] = 0;
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  bits = __reduce_or_sync(0xffffffffu, bits);
  if (lane == 0) { w_a[warp] = lo; w_b[warp] = hi; w_c[warp] = bits; }
  if (tid == 0) { s_slots = 0; s_cost = 0; }
  __syncthreads();
  lo = __reduce_min_sync(0xffffffffu, w_a[lane % kWarps]);
  hi = __reduce_max_sync(0xffffffffu, w_b[lane % kWarps]);
  bits = __reduce_or_sync(0xffffffffu, w_c[lane % kWarps]);
  *varies = bits;
  if (lo >= hi) return true;   // equal keys (or none): in order as they are
  if (((bits & 0xffu) != 0u) + ((bits & 0xff00u) != 0u) + ((bits & 0xff0000u) != 0u) + ((bits & 0xff000000u) != 0u) <= 2) {
    __syncthreads();   // (the radix sort writes where the loop above cleared)
    return false;
  }
  const uint32_t index0 = index_of(src[0]), index_span = index_of(src[cnt - 1]) - index0;
  const int shift = max(0, 22 - __clz(hi - lo));   // (hi - lo) >> shift < 1024
  auto coarse_of = [&](unsigned long long e) { return (hi - key_of(e)) >> shift; };
  for (int i = tid; i < cnt; i += kThreads) atomicAdd(&coarse_ct[coarse_of(src[i])], 1u);
  __syncthreads();
  scan(coarse_ct, [&](int, uint32_t start, uint32_t c) -> uint32_t {
    if (c <= static_cast<uint32_t>(kMaxPerBucket)) return start;
    const uint32_t j = atomicAdd(&s_slots, 1u);   // (their numbering does not matter)
    slot_start[j] = start; slot_count[j] = c;
    slot_kmin[j] = 0xffffffffu; slot_kmax[j] = 0u;
    return kSlotFlag | j;
  });

  // ---- crowded buckets: fine buckets over their own ranges ----
  const int slots = static_cast<int>(s_slots);
  auto fine_of = [&](unsigned long long e, const uint4& f) {
    const uint32_t d = f.x ? f.x - key_of(e) : index_of(e) - index0;
    return (f.y & 0xffffu) + min((f.y >> 16) - 1u, static_cast<uint32_t>(static_cast<float>(d) * __uint_as_float(f.z)));
  };
  if (slots > 0) {
    for (int i = tid; i < cnt; i += kThreads) {
      const uint32_t k = key_of(src[i]), v = coarse_ct[(hi - k) >> shift], j = v & ~kSlotFlag;
      // (the look before the atomic leaves few of them: a bucket of equal keys is updated once)
      if ((v & kSlotFlag) && k < *static_cast<volatile uint32_t*>(&slot_kmin[j])) atomicMin(&slot_kmin[j], k);
      if ((v & kSlotFlag) && k > *static_cast<volatile uint32_t*>(&slot_kmax[j])) atomicMax(&slot_kmax[j], k);
    }
    __syncthreads();
    if (tid < slots) {   // fine buckets in proportion to the elements, at least one: at most kFine in all
      uint32_t crowd = 0, before = 0, base = 0;
      for (int j = 0; j < slots; ++j) crowd += slot_count[j];
      auto share = [&](int j) { return 1u + static_cast<uint32_t>(kFine - kSlots) * slot_count[j] / crowd; };
      for (int j = 0; j < tid; ++j) { before += slot_count[j]; base += share(j); }
      const bool equal = slot_kmax[tid] == slot_kmin[tid];
      const float span = static_cast<float>(equal ? index_span : slot_kmax[tid] - slot_kmin[tid]) + 1.f;
      slot_fine[tid] = make_uint4(equal ? 0u : slot_kmax[tid], base | share(tid) << 16, __float_as_uint(static_cast<float>(share(tid)) / span),
                                  slot_start[tid] - before);
    }
    __syncthreads();
    for (int i = tid; i < cnt; i += kThreads) {
      const uint32_t v = coarse_ct[coarse_of(src[i])];
      if (v & kSlotFlag) atomicAdd(&fine_ct[fine_of(src[i], slot_fine[v & ~kSlotFlag])], 1u);
    }
    __syncthreads();
    uint32_t cost = 0;   // (sum of squares of at most 8192: below 2^27)
    scan(fine_ct, [&](int, uint32_t start, uint32_t c) -> uint32_t { cost += c * c; return start; });
    cost = __reduce_add_sync(0xffffffffu, cost);
    if (lane == 0 && cost) atomicAdd(&s_cost, cost);
    __syncthreads();
    if (s_cost > 128u * static_cast<uint32_t>(cnt)) return false;
  }

  // ---- elements to their buckets' places (a bucket's entry moves from its start to its end), place inside the bucket ----
  for (int i = tid; i < cnt; i += kThreads) {
    const unsigned long long e = src[i];
    const uint32_t b = coarse_of(e), v = coarse_ct[b];
    uint32_t place;
    if (v & kSlotFlag) {
      const uint4 f = slot_fine[v & ~kSlotFlag];
      place = atomicAdd(&fine_ct[fine_of(e, f)], 1u) + f.w;
    } else {
      place = atomicAdd(&coarse_ct[b], 1u);
    }
    dst[place] = e;
  }
  __syncthreads();
  for (int i = tid; i < cnt; i += kThreads) {
    const unsigned long long e = dst[i];
    const uint32_t b = coarse_of(e), v = coarse_ct[b];
    uint32_t beg = 0, end = v;
    if (v & kSlotFlag) {
      const uint4 f = slot_fine[v & ~kSlotFlag];
      const uint32_t i_fine = fine_of(e, f);
      beg = i_fine > (f.y & 0xffffu) ? fine_ct[i_fine - 1] + f.w : slot_start[v & ~kSlotFlag];
      end = fine_ct[i_fine] + f.w;
    } else if (b > 0) {
      const uint32_t before = coarse_ct[b - 1], j = before & ~kSlotFlag;
      beg = (before & kSlotFlag) ? slot_start[j] + slot_count[j] : before;
    }
    uint32_t place = beg;
    for (uint32_t q = beg; q < end; ++q) place += dst[q] > e ? 1u : 0u;
    src[place] = e;
  }
  __syncthreads();
  return true;
}

// scores [rows, row_stride]; limits [rows] or null; out_idx [rows, top_k]; out_val [rows, top_k] or null.
// Dynamic shared memory: max(kpow2 * 8 (sort buffer), kWarps * 256 * 4 (per-warp first-digit histograms, used before the
// sort buffer)) + max(n * 4 (keys), kpow2 * 8 + kWarps * 256 * 2 (second sort buffer + digit counters, used after the keys)).
// kMaxRounds: 32-element rounds per warp in the sort, top_k <= kWarps * 32 * kMaxRounds.
// kStream: rows too long for shared memory (more than about 52 k candidates).  The keys are not kept: every pass -- the
// first-digit histogram, the three further select passes, the two passes of the compaction -- converts the scores again
// from global memory (six reads of a row that stays in L2 instead of one); the shared memory then holds the sort buffers
// only.  Same results bit for bit.
// kC > 1: the CTAs of a cluster share the row, [first, last) being this one's slice: they sum their histograms, and the survivors go to
// the first CTA, which sorts (32 crowded rows of 49152: 172 us with the first CTA of each cluster alone, 42 with all eight).
// kOrdered: sorted by value (the way out of topk_bucket_kernel); otherwise in index order (the body of topk_select_kernel).
template <int kThreads, int kMaxRounds, bool kStream, bool kOrdered, int kC = 1>
__device__ __forceinline__ void radix_select_row(uint8_t* smem_raw, const int row, const float* __restrict__ scores, int64_t row_stride, int n,
                                                 const int32_t* __restrict__ limits, int top_k, int kpow2, int32_t* __restrict__ out_idx,
                                                 float* __restrict__ out_val, int first = 0, int last = 0x7fffffff) {
  static_assert(kC == 1 || (kStream && kOrdered), "the cluster form streams its slices and sorts");
  using namespace topk;
  constexpr int kWarps = kThreads / 32;
  const size_t front = max(static_cast<size_t>(kpow2) * 8, static_cast<size_t>(kWarps) * 256 * 4);
  unsigned long long* sortbuf = reinterpret_cast<unsigned long long*>(smem_raw);  // [kpow2]
  uint32_t* whist = reinterpret_cast<uint32_t*>(smem_raw);                         // [kWarps][256], dead before sortbuf is written
  uint32_t* keys = reinterpret_cast<uint32_t*>(smem_raw + front);                  // [n]
  __shared__ uint32_t hist[256], dbase[256];
  __shared__ uint32_t warp_sums[kWarps], warp_ties[kWarps];
  __shared__ uint32_t s_prefix, s_remaining, s_nvalid, s_gt, s_eq;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* x = scores + static_cast<int64_t>(row) * row_stride;
  const bool whole_groups = (n & 3) == 0;  // 16-byte groups never reach past the end of the row
  int lim = limits ? limits[row] : n;
  lim = lim < 0 ? 0 : (lim > n ? n : lim);
  n = min(lim, last);  // entries at or beyond the limit are not candidates: none of the passes below looks at them
  const uint32_t rank = kC > 1 ? cluster_ctarank() : 0u;
  // key of candidate i (0 = not a candidate), from shared memory or again from the scores
  auto key_at = [&](int i) -> uint32_t {
    if constexpr (kStream) {
      const float f = __ldg(x + i);
      return f > -1e30f ? float_to_key(f) : 0u;
    } else {
      return keys[i];
    }
  };

  // keys of candidates i .. i + 3 (i a multiple of four; 0 beyond the end)
  const bool vec = whole_groups && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  auto keys4 = [&](int i) -> uint4 {
    uint4 k = make_uint4(0u, 0u, 0u, 0u);
    if (i + 3 < n && (!kStream || vec)) {
      if constexpr (kStream) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(x + i));
        k = make_uint4(f.x > -1e30f ? float_to_key(f.x) : 0u, f.y > -1e30f ? float_to_key(f.y) : 0u, f.z > -1e30f ? float_to_key(f.z) : 0u,
                       f.w > -1e30f ? float_to_key(f.w) : 0u);
      } else {
        k = *reinterpret_cast<const uint4*>(keys + i);
      }
    } else {
      if (i < n) k.x = key_at(i);
      if (i + 1 < n) k.y = key_at(i + 1);
      if (i + 2 < n) k.z = key_at(i + 2);
      if (i + 3 < n) k.w = key_at(i + 3);
    }
    return k;
  };

  if (tid == 0) s_nvalid = 0;
  for (int i = tid; i < kWarps * 256; i += kThreads) whist[i] = 0;
  __syncthreads();

  // ---- load, convert, count candidates, first-digit histogram ---------------------------------------
  uint32_t my_valid = 0;
  auto take = [&](int i, float f) {
    uint32_t k = 0;
    if (i < n && f > -1e30f) { k = float_to_key(f); ++my_valid; }
    if (!kStream && i < n) keys[i] = k;  // 0 marks "not a candidate" (a real key is never 0 for a score > -1e30)
    // sign + exponent bits crowd into a few bins: a private histogram per warp keeps the atomics apart
    if (k) atomicAdd(&whist[warp * 256 + (k >> 24)], 1u);
  };
  if (vec) {
    // 16-byte loads, four of them in flight per thread before the first is used: a row of 8192 scores is two round
    // trips to memory instead of sixteen
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const int n4 = (n + 3) >> 2;
    for (int base = first >> 2; base < n4; base += 4 * kThreads) {   // (a slice starts at a multiple of four)
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i4 = base + u * kThreads + tid;
        v[u] = i4 < n4 ? __ldg(x4 + i4) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = (base + u * kThreads + tid) * 4;
        take(i, v[u].x); take(i + 1, v[u].y); take(i + 2, v[u].z); take(i + 3, v[u].w);
      }
    }
  } else {
    for (int base = first; base < n; base += kThreads) {
      const int i = base + tid;
      take(i, i < n ? x[i] : 0.f);
    }
  }
  for (int o = 16; o > 0; o >>= 1) my_valid += __shfl_xor_sync(0xffffffffu, my_valid, o);
  if (lane == 0 && my_valid) atomicAdd(&s_nvalid, my_valid);
  __syncthreads();
  if (tid < 256) {
    uint32_t t = 0;
#pragma unroll 8
    for (int w = 0; w < kWarps; ++w) t += whist[w * 256 + tid];
    hist[tid] = t;
  }
  __syncthreads();
  // the counts of all CTAs of a cluster, in `total` (this CTA's own stay in hist)
  uint32_t* total = hist;
  uint32_t nvalid = s_nvalid;
  auto sum_over_cluster = [&]() {
    if constexpr (kC > 1) {
      total = dbase;
      cluster_sync_all();
      if (tid < 256) {
        uint32_t t = 0;
#pragma unroll
        for (int r = 0; r < kC; ++r) t += ld_cluster_u32(map_to_cta(smem_u32(hist + tid), r));
        dbase[tid] = t;
      }
      cluster_sync_all();
    }
  };
  sum_over_cluster();
  if constexpr (kC > 1) {
    nvalid = 0;
#pragma unroll
    for (int r = 0; r < kC; ++r) nvalid += ld_cluster_u32(map_to_cta(smem_u32(&s_nvalid), r));
  }
  const uint32_t kk = nvalid < static_cast<uint32_t>(top_k) ? nvalid : static_cast<uint32_t>(top_k);

  // ---- radix select: threshold key T = kk-th largest candidate key -----------------------------------
  uint32_t thresh = 0;     // everything is taken when nvalid <= top_k
  uint32_t need_ties = 0;  // how many keys equal to T are taken (lowest indices first)
  if (nvalid > static_cast<uint32_t>(top_k)) {
    if (tid == 0) { s_prefix = 0; s_remaining = kk; }
    __syncthreads();
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      if (pass > 0) {
        if (tid < 256) hist[tid] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix;
        const uint32_t pmask = 0xffffffffu << (shift + 8);
        // (four keys per load, two loads in flight: one key at a time, these passes were half of the select's instructions)
#pragma unroll 2
        for (int i = first + 4 * tid; i < n; i += 4 * kThreads) {
          const uint4 k4 = keys4(i);
          const uint32_t k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (k[j] && (k[j] & pmask) == prefix) atomicAdd(&hist[(k[j] >> shift) & 0xffu], 1u);  // few survivors, spread digits
        }
        __syncthreads();
        sum_over_cluster();
      }
      // warp 0 walks the 256 bins from the top: find digit dsel with  sum(bins > dsel) < remaining <= sum(bins >= dsel)
      if (warp == 0) {
        const uint32_t remaining = s_remaining;
        uint32_t c[8], tot = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) { c[j] = total[255 - (lane * 8 + j)]; tot += c[j]; }  // lane 0 holds the top 8 bins
        uint32_t incl = tot;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        uint32_t above = incl - tot;  // candidates in bins above this lane's 8 bins
        const bool mine = above < remaining && remaining <= incl;
        if (mine) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (above < remaining && remaining <= above + c[j]) {
              s_prefix = s_prefix | ((255u - (lane * 8 + j)) << shift);
              s_remaining = remaining - above;
            }
            above += c[j];
          }
        }
      }
      __syncthreads();
    }
    thresh = s_prefix;
    need_ties = s_remaining;
  }

  // ---- compaction: keys > T and the first need_ties keys == T, in ascending index order -- kOrdered: the former first, the
  // latter, which are then in their final places, behind them ----
  const bool take_all = nvalid <= static_cast<uint32_t>(top_k);
  {
    // warp w owns the contiguous index range [w * per, w * per + per): count, prefix over warps, then write in order
    const int per = ((max(n - first, 0) + kWarps - 1) / kWarps + 31) & ~31;
    const int beg = first + warp * per, end = min(n, beg + per);
    uint32_t n_gt = 0, n_eq = 0;
#pragma unroll 2
    for (int i = beg + 4 * lane; i < end; i += 128) {   // (end is a multiple of four from beg, or n)
      const uint4 k4 = keys4(i);
      const uint32_t k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        n_gt += (k[j] != 0u && (take_all || k[j] > thresh)) ? 1u : 0u;
        n_eq += (!take_all && k[j] != 0u && k[j] == thresh) ? 1u : 0u;
      }
    }
    n_gt = __reduce_add_sync(0xffffffffu, n_gt);
    n_eq = __reduce_add_sync(0xffffffffu, n_eq);
    if (lane == 0) { warp_sums[warp] = n_gt; warp_ties[warp] = n_eq; }
    __syncthreads();
    uint32_t tie_rank = 0, above = 0;  // elements equal to / above T before this warp's range
    if constexpr (kC > 1) {
      if (tid == 0) {
        uint32_t g = 0, e = 0;
        for (int w = 0; w < kWarps; ++w) { g += warp_sums[w]; e += warp_ties[w]; }
        s_gt = g;
        s_eq = e;
      }
      cluster_sync_all();   // (every CTA is also done with its histograms, where the first one's list begins)
      for (uint32_t r = 0; r < rank; ++r) {
        above += ld_cluster_u32(map_to_cta(smem_u32(&s_gt), r));
        tie_rank += ld_cluster_u32(map_to_cta(smem_u32(&s_eq), r));
      }
    }
    for (int w = 0; w < warp; ++w) { above += warp_sums[w]; tie_rank += warp_ties[w]; }
    const uint32_t lead_sort = kC > 1 ? map_to_cta(smem_u32(sortbuf), 0) : 0u;
    for (int base = beg; base < end; base += 128) {
      uint32_t k4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) k4[j] = base + 32 * j + lane < end ? key_at(base + 32 * j + lane) : 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t k = k4[j];
        const bool gt = k != 0 && (take_all || k > thresh);
        const bool eq = !take_all && k != 0 && k == thresh;
        const uint32_t bal_gt = __ballot_sync(0xffffffffu, gt), bal_eq = __ballot_sync(0xffffffffu, eq);
        const uint32_t my_above = above + __popc(bal_gt & ((1u << lane) - 1u)), my_rank = tie_rank + __popc(bal_eq & ((1u << lane) - 1u));
        if (gt || (eq && my_rank < need_ties)) {
          const uint32_t pos = !kOrdered ? my_above + min(my_rank, need_ties) : gt ? my_above : kk - need_ties + my_rank;
          const unsigned long long e =
              (static_cast<unsigned long long>(k) << 32) | static_cast<unsigned long long>(0xffffffffu - static_cast<uint32_t>(base + 32 * j + lane));
          if constexpr (kC > 1) st_cluster_u64(lead_sort + pos * 8, e);
          else sortbuf[pos] = e;
        }
        above += __popc(bal_gt);
        tie_rank += __popc(bal_eq);
      }
    }
  }
  if constexpr (kC > 1) {
    cluster_sync_all();
    if (rank != 0) return;
  }
  __syncthreads();

  // ---- sort of the survivors above the threshold, descending by key: by buckets, or a stable radix sort -------------
  // Radix sort: four passes over 8-bit digits, least significant first, ping-pong between the sort buffer and the (now free) key
  // array.  Warp w owns the contiguous slice [w * per, w * per + per) of the current order.  Rank of an element inside
  // its digit = (elements of that digit in earlier warps) + (in earlier 32-element rounds of this warp) + (in lower
  // lanes of this round, from match_any).  Per-warp digit counters are 16-bit and only ever touched by their own warp.
  unsigned long long* src = sortbuf;
  if constexpr (kOrdered) {
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(keys);
    uint16_t* wcnt = reinterpret_cast<uint16_t*>(keys) + static_cast<size_t>(kpow2) * 4;  // [kWarps][256], behind the second buffer
    if (kk <= 64u) {
      // up to 64 survivors: one warp sorts them in registers (two per lane, bitonic network, descending on the whole
      // 64-bit element = key, then lower index), no block barriers
      if (warp == 0) {
        const int i0 = lane, i1 = lane + 32;
        unsigned long long a = i0 < static_cast<int>(kk) ? sortbuf[i0] : 0ull, b = i1 < static_cast<int>(kk) ? sortbuf[i1] : 0ull;
        for (int size = 2; size <= 64; size <<= 1) {
          const bool d0 = (i0 & size) == 0, d1 = (i1 & size) == 0;
          int stride = min(size >> 1, 32);
          if (stride == 32) {
            if ((a < b) == d0) { const unsigned long long t = a; a = b; b = t; }
            stride = 16;
          }
          for (; stride > 0; stride >>= 1) {
            const bool lower = (lane & stride) == 0;
            const unsigned long long oa = __shfl_xor_sync(0xffffffffu, a, stride), ob = __shfl_xor_sync(0xffffffffu, b, stride);
            a = (lower == d0) ? (a > oa ? a : oa) : (a < oa ? a : oa);
            b = (lower == d1) ? (b > ob ? b : ob) : (b < ob ? b : ob);
          }
        }
        sortbuf[i0] = a;
        sortbuf[i1] = b;
      }
      __syncthreads();
    } else if (uint32_t varies = 0; !bucket_sort<kThreads>(sortbuf, dst, reinterpret_cast<uint32_t*>(wcnt), static_cast<int>(kk - need_ties), &varies)) {
      const int cnt = static_cast<int>(kk - need_ties);
      const int per = ((cnt + kWarps - 1) / kWarps + 31) & ~31;
      const int rounds = per >> 5;  // <= kMaxRounds (checked by the launcher)
      const int beg = warp * per;
      const int nw = (cnt + per - 1) / per;  // warps that own elements: the counters of the others are never looked at
      for (int pass = 0; pass < 4; ++pass) {
        const int shift = 32 + 8 * pass;  // the key is the upper word of the element
        if (((varies >> (8 * pass)) & 0xffu) == 0u) continue;   // all keys have the same digit
        for (int i = tid; i < nw * 256; i += kThreads) wcnt[i] = 0;
        __syncthreads();
        unsigned long long e[kMaxRounds];
        uint32_t dig[kMaxRounds], rk[kMaxRounds];
#pragma unroll
        for (int j = 0; j < kMaxRounds; ++j) {
          if (j < rounds) {
            const int i = beg + j * 32 + lane;
            const bool live = i < cnt;
            e[j] = live ? src[i] : 0ull;
            dig[j] = live ? static_cast<uint32_t>(e[j] >> shift) & 0xffu : 0x100u + lane;  // dead lanes match nobody
            const uint32_t peers = __match_any_sync(0xffffffffu, dig[j]);
            uint32_t old = 0;
            if (live) old = wcnt[warp * 256 + dig[j]];
            __syncwarp();
            if (live && (__ffs(peers) - 1) == lane) wcnt[warp * 256 + dig[j]] = static_cast<uint16_t>(old + __popc(peers));
            __syncwarp();
            rk[j] = old + __popc(peers & ((1u << lane) - 1u));
          }
        }
        __syncthreads();
        // per digit: exclusive prefix over the warps, total
        if (tid < 256) {
          uint32_t run = 0;
#pragma unroll 4
          for (int w = 0; w < nw; ++w) {
            const uint32_t c = wcnt[w * 256 + tid];
            wcnt[w * 256 + tid] = static_cast<uint16_t>(run);
            run += c;
          }
          hist[tid] = run;
        }
        __syncthreads();
        // descending order: digit d starts after all larger digits (warp 0, lane l holds digits 255 - 8l .. 248 - 8l)
        if (warp == 0) {
          uint32_t c[8], tot = 0;
#pragma unroll
          for (int j = 0; j < 8; ++j) { c[j] = hist[255 - (lane * 8 + j)]; tot += c[j]; }
          uint32_t incl = tot;
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          uint32_t above = incl - tot;
#pragma unroll
          for (int j = 0; j < 8; ++j) { dbase[255 - (lane * 8 + j)] = above; above += c[j]; }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kMaxRounds; ++j) {
          if (j < rounds) {
            const int i = beg + j * 32 + lane;
            if (i < cnt) dst[dbase[dig[j]] + wcnt[warp * 256 + dig[j]] + rk[j]] = e[j];
          }
        }
        __syncthreads();
        unsigned long long* t = src; src = dst; dst = t;
      }
      if (src != sortbuf) {   // an odd number of passes; the elements equal to T wait in the sort buffer
        for (int i = tid; i < cnt; i += kThreads) sortbuf[i] = src[i];
        src = sortbuf;
        __syncthreads();
      }
    }
  }
  const unsigned long long* sorted = src;

  // ---- output ---------------------------------------------------------------------------------------------
  int32_t* oi = out_idx + static_cast<int64_t>(row) * top_k;
  float* ov = out_val ? out_val + static_cast<int64_t>(row) * top_k : nullptr;
  for (int i = tid; i < top_k; i += kThreads) {
    if (static_cast<uint32_t>(i) < kk) {
      const unsigned long long e = sorted[i];
      oi[i] = static_cast<int32_t>(0xffffffffu - static_cast<uint32_t>(e & 0xffffffffull));
      if (ov) ov[i] = key_to_float(static_cast<uint32_t>(e >> 32));
    } else {
      oi[i] = -1;
      if (ov) ov[i] = -INFINITY;
    }
  }
}

template <bool kStream>
__global__ void __launch_bounds__(topk::kSelectThreads, 4)
    topk_select_kernel(const float* __restrict__ scores, int64_t row_stride, int n, const int32_t* __restrict__ limits, int top_k, int kpow2,
                       int32_t* __restrict__ out_idx, float* __restrict__ out_val) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  radix_select_row<topk::kSelectThreads, 1, kStream, false>(smem_raw, blockIdx.x, scores, row_stride, n, limits, top_k, kpow2, out_idx, out_val);
}

// Ordered top-k of one row per CTA by value buckets.  The radix select above is bound by its instructions (67 k warp
// instructions per row of 8192 -> 2048, two thirds of them in the four passes of the sort).  Here the row's range
// [min, max] is cut into 4096 equal buckets, largest values first -- (max - x) * scale is monotone in x, so buckets never
// disagree with the order of the values -- and one histogram gives both the bucket that holds the k-th value and every
// bucket's place in the output.  The elements of the buckets up to that one (k plus a few) are put into their bucket's
// places, and an element's final place is its bucket's start plus the number of elements of the same bucket in front of it
// (larger key, or equal key and lower index): a handful of comparisons, no sort, no search inside the threshold's bucket.
// Rows whose values crowd (more than kMaxPerBucket in a bucket that is needed, a range that is zero or not finite) take the
// radix select; by then they have cost a range pass and a histogram, which its sort by buckets has to win back against the
// radix select with a four-pass sort alone.  Whole calls, us, that one -> here: 4096 rows of 8192 -> 2048 with a finite mask 375 -> 268, with an
// outlier 375 -> 289, exp(3 x) 377 -> 274, rounded to quarters 301 -> 308 (the worst kind: few distinct values; 1024 rows of
// 16384 -> 512: 121 -> 131.  A sample of the row for equal values, looked at before the histogram, makes these two 273 and 110 but
// rows of distinct values 3 to 7 % slower); 32 rows of 49152 with a finite mask 63 -> 42, 300 rows 190 -> 174.  Rows that do not crowd: 4096
// rows of up to 8192 -> 2048: 380 -> 112 us; 64 rows of 4096 -> 2048, whole call: 22.5 -> 15.0 us.
// kC > 1: a cluster of kC CTAs per row, each with a contiguous slice of it (few long rows: one CTA per row leaves most SMs idle
// and is bound by its own shared-memory atomics).  The CTAs exchange their ranges, sum the histograms bucket range by bucket
// range into the first CTA's, and put the elements into its list; the rest is the first CTA's work.
// kCache: the row (slice) stays in shared memory after the first pass; longer rows are read three times (from L2).
template <int kThreads, bool kCache, int kMaxRounds, int kC>
__device__ __forceinline__ void bucket_select_row(uint8_t* smem_raw, const int row, const float* __restrict__ scores, int64_t row_stride, int n_all,
                                                  const int32_t* __restrict__ limits, int top_k, int kp, int32_t* __restrict__ out_idx,
                                                  float* __restrict__ out_val) {
  using namespace topk;
  constexpr int kWarps = kThreads / 32, kPer = kBuckets / kThreads;
  uint32_t* bucket = reinterpret_cast<uint32_t*>(smem_raw);                                    // [kBuckets] counts, then ends
  unsigned long long* list = reinterpret_cast<unsigned long long*>(smem_raw + kBuckets * 4);   // [kp + kMaxPerBucket]
  float* cache = reinterpret_cast<float*>(list + kp + kMaxPerBucket);                          // [n rounded up to 4]
  __shared__ float w_min[kWarps], w_max[kWarps];
  __shared__ uint32_t w_sum[kWarps], w_fullest[kWarps], w_total[kWarps];
  __shared__ int s_last;
  __shared__ uint32_t s_fullest;
  __shared__ float s_range[2];   // this CTA's minimum and maximum (kC > 1)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = kC > 1 ? cluster_ctarank() : 0u;
  const float* x = scores + static_cast<int64_t>(row) * row_stride;
  int n = limits ? limits[row] : n_all;
  n = n < 0 ? 0 : (n > n_all ? n_all : n);
  const int n4 = (n + 3) >> 2, per4 = (n4 + kC - 1) / kC;
  const int beg4 = static_cast<int>(rank) * per4, end4 = min(n4, beg4 + per4);   // this CTA's groups of four
  // (16-byte groups of the row: never past its end when its length is a multiple of four)
  const bool vec = (n_all & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  // candidates 4 i4 .. + 3; what is not a candidate reads as -inf
  auto load4 = [&](int i4) -> float4 {
    float4 v;
    if (vec) {
      v = __ldg(reinterpret_cast<const float4*>(x) + i4);
    } else {
      const int i = 4 * i4;
      v.x = __ldg(x + i);
      v.y = i + 1 < n ? __ldg(x + i + 1) : -INFINITY;
      v.z = i + 2 < n ? __ldg(x + i + 2) : -INFINITY;
      v.w = i + 3 < n ? __ldg(x + i + 3) : -INFINITY;
    }
    const int left = n - 4 * i4;
    v.x = v.x > -1e30f ? v.x : -INFINITY;
    v.y = (v.y > -1e30f && left > 1) ? v.y : -INFINITY;
    v.z = (v.z > -1e30f && left > 2) ? v.z : -INFINITY;
    v.w = (v.w > -1e30f && left > 3) ? v.w : -INFINITY;
    return v;
  };
  auto get4 = [&](int i4) -> float4 {
    if constexpr (kCache) return reinterpret_cast<const float4*>(cache)[i4 - beg4];
    else return load4(i4);
  };

  // ---- range of the candidates ----
  for (int i = tid; i < kBuckets; i += kThreads) bucket[i] = 0;
  float mn = INFINITY, mx = -INFINITY;
  for (int base = beg4 + tid; base < end4; base += 4 * kThreads) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i4 = base + u * kThreads;
      v[u] = i4 < end4 ? load4(i4) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i4 = base + u * kThreads;
      if (kCache && i4 < end4) reinterpret_cast<float4*>(cache)[i4 - beg4] = v[u];
      mx = fmaxf(fmaxf(fmaxf(mx, v[u].x), fmaxf(v[u].y, v[u].z)), v[u].w);
      const float f[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) mn = fminf(mn, f[j] == -INFINITY ? INFINITY : f[j]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) { w_min[warp] = mn; w_max[warp] = mx; }
  if (tid == 0) s_last = kBuckets - 1;
  __syncthreads();
  mn = w_min[lane % kWarps];
  mx = w_max[lane % kWarps];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if constexpr (kC > 1) {
    if (tid == 0) { s_range[0] = mn; s_range[1] = mx; }
    cluster_sync_all();
#pragma unroll
    for (int r = 0; r < kC; ++r) {
      const uint32_t a = map_to_cta(smem_u32(s_range), r);
      mn = fminf(mn, __uint_as_float(ld_cluster_u32(a)));
      mx = fmaxf(mx, __uint_as_float(ld_cluster_u32(a + 4)));
    }
  }
  // the way out of a row that the buckets do not suit, taken by every CTA of a cluster
  auto radix = [&]() {
    __syncthreads();
    radix_select_row<kThreads, kMaxRounds, (!kCache || kC > 1), true, kC>(smem_raw, row, scores, row_stride, n_all, limits, top_k, kp, out_idx, out_val,
                                                                           4 * beg4, 4 * end4);
  };
  const float scale = static_cast<float>(kBuckets) / (mx - mn);
  if (!(scale > 0.f && scale < 3e38f && mx - mn < 3e38f)) {  // no candidates, equal values, a range that is not finite
    radix();
    return;
  }
  auto bucket_of = [&](float f) { return min(static_cast<int>((mx - f) * scale), kBuckets - 1); };

  // ---- histogram ----
#pragma unroll 2
  for (int i4 = beg4 + tid; i4 < end4; i4 += kThreads) {
    const float4 v = get4(i4);
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (f[j] != -INFINITY) atomicAdd(&bucket[bucket_of(f[j])], 1u);
  }
  __syncthreads();

  const uint32_t lead_bucket = kC > 1 ? map_to_cta(smem_u32(bucket), 0) : 0u, lead_list = kC > 1 ? map_to_cta(smem_u32(list), 0) : 0u;
  if constexpr (kC > 1) {  // every CTA sums one range of the buckets over all of them, in the first one's histogram
    cluster_sync_all();
    for (int b = static_cast<int>(rank) * (kBuckets / kC) + tid; b < static_cast<int>(rank + 1) * (kBuckets / kC); b += kThreads) {
      uint32_t sum = 0;
#pragma unroll
      for (int r = 0; r < kC; ++r) sum += ld_cluster_u32(map_to_cta(smem_u32(bucket + b), r));
      st_cluster_u32(lead_bucket + b * 4, sum);
    }
    cluster_sync_all();
  }

  // ---- starts of the buckets, the last one that is needed, the fullest one of those ----
  const uint32_t want = static_cast<uint32_t>(top_k);
  uint32_t fullest = 0, total = 0;   // total: elements in the buckets up to the last one, fewer than top_k + kMaxPerBucket
  if (rank == 0) {
    uint32_t c[kPer], mine = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) { c[j] = bucket[tid * kPer + j]; mine += c[j]; }
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) w_sum[warp] = incl;
    __syncthreads();
    uint32_t start = incl - mine;
    for (int w = 0; w < warp; ++w) start += w_sum[w];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      bucket[tid * kPer + j] = start;
      if (start < want) {   // a bucket with places among the first top_k
        fullest = max(fullest, c[j]);
        total = start + c[j];
        if (start + c[j] >= want) s_last = tid * kPer + j;   // (one thread, one bucket: where the count passes top_k)
      }
      start += c[j];
    }
    fullest = __reduce_max_sync(0xffffffffu, fullest);
    total = __reduce_max_sync(0xffffffffu, total);
    if (lane == 0) { w_fullest[warp] = fullest; w_total[warp] = total; }
    __syncthreads();
    fullest = __reduce_max_sync(0xffffffffu, w_fullest[lane % kWarps]);
    total = __reduce_max_sync(0xffffffffu, w_total[lane % kWarps]);
    if (kC > 1 && tid == 0) s_fullest = fullest;
  }
  int last = 0;
  if constexpr (kC > 1) {
    cluster_sync_all();
    last = static_cast<int>(ld_cluster_u32(map_to_cta(smem_u32(&s_last), 0)));
    fullest = ld_cluster_u32(map_to_cta(smem_u32(&s_fullest), 0));
  } else {
    last = s_last;
  }
  if (fullest > static_cast<uint32_t>(kMaxPerBucket)) {
    radix();
    return;
  }

  // ---- elements of those buckets to their bucket's places (bucket[b] moves from its start to its end) ----
#pragma unroll 2
  for (int i4 = beg4 + tid; i4 < end4; i4 += kThreads) {
    const float4 v = get4(i4);
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (f[j] == -INFINITY) continue;
      const int b = bucket_of(f[j]);
      if (b <= last)
      {
        const unsigned long long e = (static_cast<unsigned long long>(float_to_key(f[j])) << 32) |
                                     static_cast<unsigned long long>(0xffffffffu - static_cast<uint32_t>(4 * i4 + j));
        if constexpr (kC > 1) st_cluster_u64(lead_list + atom_add_cluster_u32(lead_bucket + b * 4, 1u) * 8, e);
        else list[atomicAdd(&bucket[b], 1u)] = e;
      }
    }
  }
  if constexpr (kC > 1) {
    cluster_sync_all();
    if (rank != 0) return;
  } else {
    __syncthreads();
  }

  // ---- place inside the bucket, output ----
  int32_t* oi = out_idx + static_cast<int64_t>(row) * top_k;
  float* ov = out_val ? out_val + static_cast<int64_t>(row) * top_k : nullptr;
  for (uint32_t i = tid; i < total; i += kThreads) {
    const unsigned long long e = list[i];
    const float f = key_to_float(static_cast<uint32_t>(e >> 32));
    const int b = bucket_of(f);
    const uint32_t beg = b > 0 ? bucket[b - 1] : 0u, end = bucket[b];
    uint32_t place = beg;
    for (uint32_t j = beg; j < end; ++j) place += list[j] > e ? 1u : 0u;
    if (place < want) {
      oi[place] = static_cast<int32_t>(0xffffffffu - static_cast<uint32_t>(e & 0xffffffffull));
      if (ov) ov[place] = f;
    }
  }
  for (uint32_t i = total + tid; i < want; i += kThreads) {
    oi[i] = -1;
    if (ov) ov[i] = -INFINITY;
  }
}

// A cluster's row whose candidates fit the first CTA's slice is that CTA's alone, the others leave: score rows are as wide as the
// caller's block table, the sequence may be short (64 sequences of up to 3000 keys in a table for 131072, scores + selector:
// 36 -> 29 us; 26 under a table for 3000).
template <int kThreads, bool kCache, int kMaxRounds, int kC>
__global__ void __launch_bounds__(kThreads, (kThreads == 512 && kMaxRounds <= 4) ? 3 : 1)
    topk_bucket_kernel(const float* __restrict__ scores, int64_t row_stride, int n, const int32_t* __restrict__ limits, int top_k, int kp,
                       int32_t* __restrict__ out_idx, float* __restrict__ out_val) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int row = blockIdx.x / kC;
  if constexpr (kC > 1) {
    if (limits && limits[row] <= topk::cluster_slice(n, kC)) {
      if (cluster_ctarank() == 0)
        bucket_select_row<kThreads, kCache, kMaxRounds, 1>(smem_raw, row, scores, row_stride, n, limits, top_k, kp, out_idx, out_val);
      return;
    }
  }
  bucket_select_row<kThreads, kCache, kMaxRounds, kC>(smem_raw, row, scores, row_stride, n, limits, top_k, kp, out_idx, out_val);
}

// Shared memory of the kernel that keeps a row's keys (n > 0) or of the streaming kernel (n = 0).
template <int kThreads>
static size_t radix_smem_bytes(int n, int kp) {
  constexpr size_t kWarps = kThreads / 32;
  const size_t sort = static_cast<size_t>(kp) * 8, whist = kWarps * 256 * 4;
  const size_t back_sort = sort + kWarps * 256 * 2;
  return (sort > whist ? sort : whist) + (static_cast<size_t>(n) * 4 > back_sort ? static_cast<size_t>(n) * 4 : back_sort);
}

size_t topk_smem_bytes(int n, int top_k, int* kpow2_out) {
  int kp = 32;  // buffer length: top_k rounded up to a multiple of 32 (name kept from the power-of-two days of a bitonic sort)
  while (kp < top_k) kp += 32;
  if (kpow2_out) *kpow2_out = kp;
  return radix_smem_bytes<topk::kSelectThreads>(n, kp);
}

// Shared memory of topk_bucket_kernel (n = 0: the row is not kept), including what its way out needs.
template <int kThreads>
static size_t bucket_smem_bytes(int n, int kp) {
  const size_t own = topk::kBuckets * 4 + static_cast<size_t>(kp + topk::kMaxPerBucket) * 8 + ((static_cast<size_t>(n) + 3) & ~static_cast<size_t>(3)) * 4;
  const size_t radix = radix_smem_bytes<kThreads>(n, kp);
  return own > radix ? own : radix;
}

template <int kThreads>
static int launch_bucket(const float* scores, int64_t rows, int n, int64_t row_stride, const int32_t* limits, int top_k, int kp, int32_t* out_idx,
                         float* out_val, int dev, cudaStream_t stream) {
  const bool cache = bucket_smem_bytes<kThreads>(n, kp) <= topk::kMaxSmemBytes;
  const size_t smem = bucket_smem_bytes<kThreads>(cache ? n : 0, kp);
  constexpr int kFew = kThreads == 512 ? 4 : 2, kMany = kThreads == 512 ? 16 : 8;   // rounds of the way out's sort: 2048, 8192 survivors
  const bool small = top_k <= kThreads * kFew;
  auto kern = cache ? (small ? topk_bucket_kernel<kThreads, true, kFew, 1> : topk_bucket_kernel<kThreads, true, kMany, 1>)
                    : (small ? topk_bucket_kernel<kThreads, false, kFew, 1> : topk_bucket_kernel<kThreads, false, kMany, 1>);
  cudaError_t e = ensure_dynamic_smem(kern, dev, static_cast<int>(smem));
  if (e != cudaSuccess) return static_cast<int>(e);
  kern<<<static_cast<unsigned>(rows), kThreads, smem, stream>>>(scores, row_stride, n, limits, top_k, kp, out_idx, out_val);
  return static_cast<int>(cudaGetLastError());
}

// A cluster of kC CTAs of 512 threads per row.
template <int kC>
static int launch_bucket_cluster(const float* scores, int64_t rows, int n, int64_t row_stride, const int32_t* limits, int top_k, int kp,
                                 int32_t* out_idx, float* out_val, int dev, int sms, cudaStream_t stream) {
  const int slice = topk::cluster_slice(n, kC);
  const size_t most = rows * kC <= sms ? topk::kMaxLoneClusterSmemBytes : topk::kMaxClusterSmemBytes;
  const bool cache = bucket_smem_bytes<512>(slice, kp) <= most;
  const size_t smem = bucket_smem_bytes<512>(cache ? slice : 0, kp);   // (a row that one CTA takes alone fits a slice)
  auto kern = top_k <= 2048 ? (cache ? topk_bucket_kernel<512, true, 4, kC> : topk_bucket_kernel<512, false, 4, kC>)
                            : (cache ? topk_bucket_kernel<512, true, 16, kC> : topk_bucket_kernel<512, false, 16, kC>);
  cudaError_t e = ensure_dynamic_smem(kern, dev, static_cast<int>(smem));
  if (e != cudaSuccess) return static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows * kC));
  cfg.blockDim = dim3(512);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kC; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, scores, row_stride, n, limits, top_k, kp, out_idx, out_val));
}

int launch_topk_select(const float* scores, int64_t rows, int n, int64_t row_stride, const int32_t* limits, int top_k,
                       int32_t* out_idx, float* out_val, cudaStream_t stream, int ordered) {
  if (top_k > topk::kSelectThreads * 16) return static_cast<int>(cudaErrorInvalidValue);
  int kp = 0;
  const bool stream_rows = topk_smem_bytes(n, top_k, &kp) > topk::kMaxSmemBytes;
  int dev = 0, sms = 0;
  cudaError_t e = current_device_sms(&dev, &sms);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (ordered) {
    // Few rows that one CTA cannot keep in shared memory (more than about 47 k): a cluster per row, as long as the clusters are
    // resident at once.  49152 -> 2048: 1 row 20.8 -> 12.3 us, 32 rows 21.5 -> 16.3, 60 rows 21.6 -> 18.4; 4 rows of 131072 45.4 ->
    // 16.5.  Shorter rows do not repay the cluster's barriers and remote atomics (32 rows of 16384: 9.4 -> 17.2).
    const bool kept = bucket_smem_bytes<1024>(n, kp) <= topk::kMaxSmemBytes;
    if (!kept && rows * 8 <= 2 * sms)
      return launch_bucket_cluster<8>(scores, rows, n, row_stride, limits, top_k, kp, out_idx, out_val, dev, sms, stream);
    if (!kept && rows * 4 <= 2 * sms)
      return launch_bucket_cluster<4>(scores, rows, n, row_stride, limits, top_k, kp, out_idx, out_val, dev, sms, stream);
    // other rows that leave SMs idle get twice the threads
    return rows <= sms ? launch_bucket<1024>(scores, rows, n, row_stride, limits, top_k, kp, out_idx, out_val, dev, stream)
                       : launch_bucket<512>(scores, rows, n, row_stride, limits, top_k, kp, out_idx, out_val, dev, stream);
  }
  const size_t smem = topk_smem_bytes(stream_rows ? 0 : n, top_k, nullptr);
  auto kern = stream_rows ? topk_select_kernel<true> : topk_select_kernel<false>;
  if ((e = ensure_dynamic_smem(kern, dev, static_cast<int>(smem))) != cudaSuccess) return static_cast<int>(e);
  kern<<<static_cast<unsigned>(rows), topk::kSelectThreads, smem, stream>>>(scores, row_stride, n, limits, top_k, kp, out_idx, out_val);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dsa
