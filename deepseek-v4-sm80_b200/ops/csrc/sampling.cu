// Temperature / top-k / top-p sampling, one CTA per request row, replacing the reference's flashinfer calls
// (python/minisgl/engine/sample.py:69-90).
//
// Definition (the PyTorch oracle implements the same one): p = softmax(logits / T).  Order the vocabulary by
// (p descending, id ascending); entry of rank r is kept iff (top_k <= 0 or r < top_k) and the probability mass
// before it is < top_p.  The sample is the first kept id, in id order, whose running kept mass reaches
// u * kept_mass.  Rows with T <= 0 or top_k == 1 are greedy (lowest id among the maxima).
// Masses are accumulated as 2^-40 fixed point so that every reduction is order independent: the same logits
// and u always give the same token.  An optional mask adds -inf to given ids first (reasoning sampler).
#include "common.cuh"

namespace {

__device__ __forceinline__ uint32_t okey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// p * 2^40 truncated.  Multiplying a float by a power of two is exact, so the single-precision product equals the
// double-precision one the oracle computes; the FP64 pipe (slow on this part) stays out of the per-element path.
__device__ __forceinline__ unsigned long long fx(float p) { return __float2ull_rz(p * 1099511627776.0f); }

__device__ __forceinline__ unsigned long long block_scan_u64(unsigned long long v, unsigned long long* wt,
                                                             unsigned long long& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) wt[w] = x;
  __syncthreads();
  if (w == 0) {
    unsigned long long s = wt[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    wt[lane] = s;
  }
  __syncthreads();
  total = wt[31];
  return x - v + (w ? wt[w - 1] : 0ull);
}

// Any row: the key of the last kept rank byte by byte, each byte a pass over the whole row.  Rows that the kernel below cannot order come
// here: a maximum or a temperature that is not finite, values that are not numbers, more entries around the end of the kept set than its
// list holds (equal logits above all).  What is known by then is given: ztot, and that the last kept key is one of [kmin, kmax], which
// cnt_above entries of mass mass_above come before.  Bytes that kmin and kmax share need no pass, so equal logits need none.
template <class V>
__device__ __noinline__ int sample_exhaustive(V val, int v, float mx, int amax, float temp, int tk, float tp, float u,
                                              unsigned long long ztot, int cnt_above, unsigned long long mass_above, uint32_t kmin,
                                              uint32_t kmax) {
  __shared__ int si[32];
  __shared__ unsigned long long wt[32];
  __shared__ unsigned long long hmass[256];
  __shared__ int hcnt[256];
  __shared__ int sh_bin, sh_cnt_above;
  __shared__ unsigned long long sh_mass_above;
  const int tid = threadIdx.x, lane = tid & 31;
  const float inv_t = 1.f / temp;
  const unsigned long long p_limit = tp >= 1.f ? ~0ull : (unsigned long long)((double)ztot * (double)tp);
  const int k_limit = tk > 0 ? tk : 0x7fffffff;
  // radix descent: find the key of the last kept rank
  uint32_t prefix = 0, mask = 0;
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (((kmin ^ kmax) >> shift) == 0) {
      prefix = kmin & (~0u << shift), mask = ~0u << shift;
      continue;
    }
    for (int i = tid; i < 256; i += 1024) hcnt[i] = 0, hmass[i] = 0ull;
    __syncthreads();
    // Histogram of the candidates' next key byte.  The top bytes of nearly all logits agree, so per-element atomics
    // would serialise on a handful of addresses: a warp whose active lanes all hit one bin adds once (the masses are
    // fixed point, so any order gives the same sums).
    for (int i0 = 0; i0 < v; i0 += 1024) {
      const int i = i0 + tid;
      bool act = false;
      uint32_t bin = 0;
      unsigned long long m = 0;
      if (i < v) {
        const float x = val(i);
        const uint32_t key = okey(x);
        if ((key & mask) == prefix && key >= kmin && key <= kmax) {
          act = true;
          bin = (key >> shift) & 0xff;
          m = fx(expf((x - mx) * inv_t));
        }
      }
      // one pair of atomics per distinct bin of the warp: 64-bit shared atomics under same-address contention are
      // what made the first version of this loop take milliseconds
      unsigned todo = __ballot_sync(0xffffffffu, act);
      while (todo) {  // `todo` is warp-uniform
        const int leader = __ffs(todo) - 1;
        const uint32_t bin0 = __shfl_sync(0xffffffffu, bin, leader);
        const bool mine = act && bin == bin0;
        const unsigned grp = __ballot_sync(0xffffffffu, mine);
        unsigned long long sm = mine ? m : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, o);
        if (lane == leader) {
          atomicAdd(&hcnt[bin0], __popc(grp));
          atomicAdd(&hmass[bin0], sm);
        }
        todo &= ~grp;
      }
    }
    __syncthreads();
    if (tid == 0) {
      int c = cnt_above, bsel = 0;
      unsigned long long m = mass_above;
      for (int bb = 255; bb >= 0; --bb) {
        // does the kept set end inside this bin?  (it ends where count reaches k or mass reaches p)
        if (hcnt[bb] > 0 && (c + hcnt[bb] >= k_limit || m + hmass[bb] >= p_limit || bb == 0)) {
          bsel = bb;
          break;
        }
        c += hcnt[bb];
        m += hmass[bb];
        bsel = bb;
      }
      sh_bin = bsel;
      sh_cnt_above = c;
      sh_mass_above = m;
    }
    __syncthreads();
    prefix |= (uint32_t)sh_bin << shift;
    mask |= 0xffu << shift;
    kmin = max(kmin, prefix), kmax = min(kmax, prefix | ~mask);
    cnt_above = sh_cnt_above;
    mass_above = sh_mass_above;
    __syncthreads();
  }
  // kept: key > prefix, plus threshold ties in id order while count < k and mass before < p.
  // Every thread owns a contiguous range of ids, so "in id order" needs three block scans in total (ties before the
  // thread, tie mass before it, kept mass before it) and sequential walks inside the thread's own range.
  const int per = (v + 1023) / 1024;
  const int i_lo = min(tid * per, v), i_hi = min(i_lo + per, v);
  unsigned long long my_eq_mass = 0;
  int my_eq_cnt = 0;
  for (int i = i_lo; i < i_hi; ++i) {
    const float x = val(i);
    if (okey(x) == prefix) ++my_eq_cnt, my_eq_mass += fx(expf((x - mx) * inv_t));
  }
  unsigned long long tot;
  const int eqc_before = (int)block_scan_u64((unsigned long long)my_eq_cnt, wt, tot);
  const unsigned long long eqm_before = block_scan_u64(my_eq_mass, wt, tot);
  auto walk = [&](unsigned long long start, unsigned long long target, bool find) -> unsigned long long {
    // returns the kept mass of this thread's range, or (find) the id at which the running kept mass passes target
    unsigned long long run = start, em = eqm_before;
    int ec = eqc_before;
    for (int i = i_lo; i < i_hi; ++i) {
      const float x = val(i);
      const uint32_t key = okey(x);
      const unsigned long long pm = fx(expf((x - mx) * inv_t));
      const bool eq = key == prefix;
      const bool keep = key > prefix || (eq && cnt_above + ec < k_limit && mass_above + em < p_limit);
      if (eq) ++ec, em += pm;
      if (keep) {
        if (find && run + pm > target && run <= target) return (unsigned long long)i;
        run += pm;
      }
    }
    return find ? ~0ull : run - start;
  };
  const unsigned long long my_kept = walk(0ull, 0ull, false);
  unsigned long long kept_total;
  const unsigned long long kept_before = block_scan_u64(my_kept, wt, kept_total);
  unsigned long long target = (unsigned long long)((double)u * (double)kept_total);
  if (target >= kept_total && kept_total > 0) target = kept_total - 1;
  if (tid == 0) si[1] = amax;  // fallback (empty kept set cannot happen: the maximum is always kept)
  __syncthreads();
  if (my_kept > 0 && target >= kept_before && target < kept_before + my_kept) {
    const unsigned long long id = walk(kept_before, target, true);
    if (id != ~0ull) si[1] = (int)id;
  }
  __syncthreads();
  return si[1];
}

// Sums and a list per row of the route below.
constexpr int kBins = 2048;      // of (mx - x) / T, 1/64 wide: from 28 on (the last 256 bins) a mass is 0 in 2^-40
constexpr int kList = 4096;      // entries of the last kept bin that can be put in order
constexpr int kTopList = 256;    // top_k up to which the threads' maxima bound the kept set

struct SampleSmem {
  union {
    struct {
      uint32_t lo[kBins], hi[kBins];   // mass of a bin
      int cnt[kBins];
    } h;
    unsigned long long list[kList];
  };
  unsigned long long wt[32], seg[32];
  unsigned long long mass_above, last;
  int n, bin, cnt_above, found;
  uint32_t kmin, kmax;           // of the listed entries
};

// list[0..n) in descending order, n <= kList; all 1024 threads.
__device__ __forceinline__ void sort_list(unsigned long long* list, int n) {
  int p = 32;
  while (p < n) p <<= 1;
  __syncthreads();
  for (int i = n + threadIdx.x; i < p; i += 1024) list[i] = 0ull;
  __syncthreads();
  for (int size = 2; size <= p; size <<= 1)
    for (int step = size >> 1; step > 0; step >>= 1) {
      for (int i = threadIdx.x; i < (p >> 1); i += 1024) {
        const int a = 2 * i - (i & (step - 1)), b = a + step;
        const unsigned long long x = list[a], y = list[b];
        if ((x < y) == ((a & size) == 0)) list[a] = y, list[b] = x;
      }
      __syncthreads();
    }
}

__device__ __forceinline__ float key_value(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// What bounds it: passes over the row, which the L2 holds after the first (128 rows of 129 280 floats: 66 MB).  A warp reads one
// 32nd of the row, 16 bytes a lane and four loads in flight.  Two to three passes do: the maximum; the sum of the masses together
// with a histogram of (mx - x) / T, or, for a top_k of at most 256, with the list of what reaches the k-th largest of the threads'
// own maxima (at least k entries do); then, behind a histogram, the masses that the last kept bin's order decides.  Entries without a
// mass (-inf: a grammar's mask) are never drawn and never listed, so they do not fill the list.
// Only that bin's entries, about 200 of them for logits of a spread of 2.5, or that list are put in order.  The pass that finds the
// sample reads the one 32nd that it falls into.  128 rows of 129 280 at top_k 50 and top_p 0.95 take 55 us; the four passes of the
// descent, three walks over 126 consecutive ids a thread and the passes before them took 620 us.
__global__ void __launch_bounds__(1024) sample_kernel(const float* __restrict__ logits, int v,
                                                      const float* __restrict__ temperature,
                                                      const int* __restrict__ top_k, const float* __restrict__ top_p,
                                                      const float* __restrict__ uniform,
                                                      const int* __restrict__ mask_ids, int n_mask,
                                                      long long* __restrict__ out) {
  pdl_entry();
  using u64 = unsigned long long;
  __shared__ float sf[32];
  __shared__ int si[32], sbad;
  __shared__ SampleSmem sm;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const float* row = logits + (size_t)b * v;
  const int* mrow = mask_ids ? mask_ids + (size_t)b * n_mask : nullptr;
  auto masked = [mrow, n_mask](float x, int i) -> float {
    for (int m = 0; m < n_mask; ++m)
      if (mrow[m] == i) x = -INFINITY;
    return x;
  };
  // f(x, id) over this warp's ids [lo, hi); whole groups of four that start on 16 bytes are one load
  const int per_warp = ((v + 127) / 128) * 4;
  const int lo = min(w * per_warp, v), hi = min(lo + per_warp, v);
  auto each = [&](auto f) {
    const int head = min(hi, lo + (int)((4 - (((uintptr_t)(row + lo) >> 2) & 3)) & 3));
    if (lo + lane < head) f(masked(row[lo + lane], lo + lane), lo + lane);
    const float4* r4 = reinterpret_cast<const float4*>(row + head);
    const int n4 = (hi - head) >> 2;
    int i = lane;
    for (; i + 96 < n4; i += 128) {
      float4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = r4[i + 32 * u];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int id = head + 4 * (i + 32 * u);
        f(masked(x[u].x, id), id), f(masked(x[u].y, id + 1), id + 1);
        f(masked(x[u].z, id + 2), id + 2), f(masked(x[u].w, id + 3), id + 3);
      }
    }
    for (; i < n4; i += 32) {
      const float4 x = r4[i];
      const int id = head + 4 * i;
      f(masked(x.x, id), id), f(masked(x.y, id + 1), id + 1), f(masked(x.z, id + 2), id + 2), f(masked(x.w, id + 3), id + 3);
    }
    const int tail = head + 4 * n4 + lane;
    if (tail < hi) f(masked(row[tail], tail), tail);
  };
  // argmax (lowest id wins ties) -- also the softmax max
  if (tid == 0) sbad = 0, sm.n = 0, sm.kmin = ~0u, sm.kmax = 0;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  bool nan = false;
  each([&](float x, int i) {
    nan |= x != x;
    if (x > best || (x == best && i < bi)) best = x, bi = i;
  });
  const float own = best;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ob > best || (ob == best && oi < bi)) best = ob, bi = oi;
  }
  if (lane == 0) sf[w] = best, si[w] = bi;
  __syncthreads();
  if (nan) sbad = 1;
  if (w == 0) {
    best = sf[lane], bi = si[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) best = ob, bi = oi;
    }
    if (lane == 0) sf[0] = best, si[0] = bi;
  }
  __syncthreads();
  const float mx = sf[0];
  const int amax = si[0];
  const float temp = temperature ? temperature[b] : 0.f;
  const int tk = top_k ? top_k[b] : -1;
  const float tp = top_p ? top_p[b] : 1.f;
  if (temp <= 0.f || tk == 1) {
    if (tid == 0) out[b] = amax;
    return;
  }
  const float u = uniform ? uniform[b] : 0.5f;
  const float inv_t = 1.f / temp;
  auto mass = [&](float x) { return fx(expf((x - mx) * inv_t)); };
  auto exhaustive = [&](u64 ztot, int cnt_above, u64 mass_above, uint32_t kmin, uint32_t kmax) {
    const int id = sample_exhaustive([row, masked](int i) { return masked(row[i], i); }, v, mx, amax, temp, tk, tp, u, ztot, cnt_above, mass_above,
                                     kmin, kmax);
    if (tid == 0) out[b] = id;
  };
  u64 zl = 0, ztot;
  if (sbad || !isfinite(mx) || !isfinite(inv_t)) {
    each([&](float x, int) { zl += mass(x); });
    block_scan_u64(zl, sm.wt, ztot);
    exhaustive(ztot, 0, 0ull, 0u, ~0u);
    return;
  }
  auto entry = [](uint32_t key, int id) { return (u64)key << 32 | (0xffffffffu - (uint32_t)id); };   // larger: earlier in the order
  const int k_limit = tk > 0 ? tk : 0x7fffffff;
  const bool keep_all = tk <= 0 && tp >= 1.f, few = tk > 0 && tk <= kTopList;
  u64 last = 0;              // the last kept entry with a mass: kept are those not below it, and some without a mass
  bool none = false;         // top_p leaves nothing
  auto listed = [&](uint32_t key, int i) {
    const int at = atomicAdd(&sm.n, 1);
    if (at < kList) sm.list[at] = entry(key, i);
  };
  uint32_t bound = 0;
  if (few) {
    // at least k of the threads' maxima, so at least k values, are not below their k-th
    sm.list[tid] = (u64)okey(own) << 32 | (uint32_t)tid;
    sort_list(sm.list, 1024);
    bound = (uint32_t)(sm.list[tk - 1] >> 32);
    __syncthreads();
    each([&](float x, int i) {
      const u64 m = mass(x);
      zl += m;
      const uint32_t key = okey(x);
      if (key >= bound && m > 0) listed(key, i);
    });
  } else if (keep_all) {
    each([&](float x, int) { zl += mass(x); });
  } else {
    for (int i = tid; i < kBins; i += 1024) sm.h.lo[i] = sm.h.hi[i] = 0, sm.h.cnt[i] = 0;
    __syncthreads();
    const bool counted = tk > 0;
    each([&](float x, int) {
      const u64 m = mass(x);
      zl += m;
      const int bin = min(__float2int_rz(fminf((mx - x) * inv_t, 1e6f) * 64.f), kBins - 1);
      const uint32_t m_lo = (uint32_t)m;
      uint32_t m_hi = (uint32_t)(m >> 32);
      if (m_lo && atomicAdd(&sm.h.lo[bin], m_lo) + m_lo < m_lo) ++m_hi;    // a carry
      if (m_hi) atomicAdd(&sm.h.hi[bin], m_hi);
      if (counted) atomicAdd(&sm.h.cnt[bin], 1);
    });
  }
  block_scan_u64(zl, sm.wt, ztot);
  const u64 p_limit = tp >= 1.f ? ~0ull : (u64)((double)ztot * (double)tp);
  u64 mass_above = 0;
  int cnt_above = 0, bin_last = -1;
  if (!few && !keep_all) {
    // the first bin, from the largest values on, with which the count reaches k or the mass p
    const int b0 = 2 * tid;
    const u64 m0 = (u64)sm.h.hi[b0] << 32 | sm.h.lo[b0], m1 = (u64)sm.h.hi[b0 + 1] << 32 | sm.h.lo[b0 + 1];
    const int c0 = sm.h.cnt[b0], c1 = sm.h.cnt[b0 + 1];
    if (tid == 0) sm.bin = -1;
    u64 tot;
    const u64 m_before = block_scan_u64(m0 + m1, sm.wt, tot);
    const int c_before = (int)block_scan_u64((u64)(c0 + c1), sm.wt, tot);
    auto ends = [&](int c, u64 m) { return c >= k_limit || m >= p_limit; };
    const bool before = tid > 0 && ends(c_before, m_before);
    if (!before && ends(c_before + c0, m_before + m0))
      sm.bin = b0, sm.mass_above = m_before, sm.cnt_above = c_before;
    else if (!before && ends(c_before + c0 + c1, m_before + m0 + m1))
      sm.bin = b0 + 1, sm.mass_above = m_before + m0, sm.cnt_above = c_before + c0;
    __syncthreads();
    bin_last = sm.bin;
    if (bin_last >= 0) mass_above = sm.mass_above, cnt_above = sm.cnt_above;
    __syncthreads();
  }
  // the kept mass of each warp's ids; entries of the last bin are listed and counted once their order is known
  u64 own_mass = 0;
  if (keep_all || (!few && bin_last < 0)) {
    own_mass = zl;
  } else if (!few) {
    each([&](float x, int i) {
      const int bin = min(__float2int_rz(fminf((mx - x) * inv_t, 1e6f) * 64.f), kBins - 1);
      if (bin > bin_last) return;
      const u64 m = mass(x);
      if (bin < bin_last) own_mass += m;
      else if (m > 0) listed(okey(x), i);
    });
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) own_mass += __shfl_xor_sync(0xffffffffu, own_mass, o);
  if (lane == 0) sm.seg[w] = own_mass;
  __syncthreads();
  const int n = sm.n;
  if (n > kList) {
    uint32_t kmin = ~0u, kmax = 0;
    each([&](float x, int) {
      const uint32_t key = okey(x);
      const int bin = min(__float2int_rz(fminf((mx - x) * inv_t, 1e6f) * 64.f), kBins - 1);
      if ((few ? key >= bound : bin == bin_last) && mass(x) > 0) kmin = min(kmin, key), kmax = max(kmax, key);
    });
    kmin = __reduce_min_sync(0xffffffffu, kmin), kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) atomicMin(&sm.kmin, kmin), atomicMax(&sm.kmax, kmax);
    __syncthreads();
    exhaustive(ztot, cnt_above, mass_above, sm.kmin, sm.kmax);
    return;
  }
  if (n > 0) {
    sort_list(sm.list, n);
    u64 e[4], m[4], before, tot;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = 4 * tid + j < n ? sm.list[4 * tid + j] : 0ull;
      m[j] = 4 * tid + j < n ? mass(key_value((uint32_t)(e[j] >> 32))) : 0ull;
    }
    if (tid == 0) sm.last = 0ull;
    before = mass_above + block_scan_u64(m[0] + m[1] + m[2] + m[3], sm.wt, tot);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = 4 * tid + j;
      auto kept = [&](int rank, u64 mass_before) { return rank < n && cnt_above + rank < k_limit && mass_before < p_limit; };
      if (kept(r, before)) {
        atomicAdd(&sm.seg[(0xffffffffu - (uint32_t)e[j]) / per_warp], m[j]);
        if (!kept(r + 1, before + m[j])) sm.last = e[j];
      }
      before += m[j];
    }
    __syncthreads();
    last = sm.last;
    none = last == 0ull;
  }
  // the warp's ids that the running kept mass passes the target in, and then the id
  u64 kept_total;
  const u64 kept_before = block_scan_u64(lane == 0 ? sm.seg[w] : 0ull, sm.wt, kept_total);
  u64 target = (u64)((double)u * (double)kept_total);
  if (target >= kept_total && kept_total > 0) target = kept_total - 1;
  if (tid == 0) sm.found = amax, sm.bin = -1;
  __syncthreads();
  if (lane == 0 && !none && target >= kept_before && target < kept_before + sm.seg[w]) sm.bin = w, sm.mass_above = kept_before;
  __syncthreads();
  if (sm.bin >= 0) {
    const int first = sm.bin * per_warp, end = min(first + per_warp, v), per = (per_warp + 1023) / 1024;
    const int a = min(first + tid * per, end), z = min(a + per, end);
    auto kept_mass = [&](int i) -> u64 {
      const float x = masked(row[i], i);
      return entry(okey(x), i) >= last ? mass(x) : 0ull;
    };
    u64 mine = 0, tot;
    for (int i = a; i < z; ++i) mine += kept_mass(i);
    u64 run = sm.mass_above + block_scan_u64(mine, sm.wt, tot);
    if (target >= run && target < run + mine)
      for (int i = a; i < z; ++i) {
        const u64 pm = kept_mass(i);
        if (run <= target && run + pm > target) {
          sm.found = i;
          break;
        }
        run += pm;
      }
    __syncthreads();
  }
  if (tid == 0) out[b] = sm.found;
}

}  // namespace

DSV4_API int dsv4_sample(const float* logits, int rows, int v, const float* temperature, const int* top_k,
                         const float* top_p, const float* uniform, const int* mask_ids, int n_mask, long long* out,
                         cudaStream_t st) {
  if (rows <= 0) return 0;
  dsv4_launch(sample_kernel, rows, 1024, 0, st, logits, v, temperature, top_k, top_p, uniform, mask_ids, n_mask, out);
  return (int)cudaGetLastError();
}
