// Sparse-attention indexer: FP8 logits over a request's compressed (ratio 4) history and the deterministic top-k.
//
// logits[t, j] = k_scale[row_j] * sum_h relu(q[t,h,:] . k[row_j,:]) * w[t,h]   for j < (pos+1)/4, else -inf
// (python/minisgl/kernel/triton/deepseek_v4.py:1296-1384).  q and k are e4m3 codes; every product is exact in fp32.
// Each CTA owns one token and a 64-row slice of its history; a lane owns two heads, the key row is broadcast from
// shared memory, so there is one warp reduction per (token, row).
//
// top-k keeps the reference's contract (csrc/jit/dsv4_topk_v1.cu:275-479): rows shorter than k keep every entry,
// a non-finite score invalidates the row (len = -1), ties at the threshold are resolved towards the lower index.
// The selection finds the last selected entry in the order (score descending, index ascending) and writes what is not below it,
// so the result is deterministic and comes out sorted by index (attention does not depend on the order).
#include "common.cuh"

namespace {

constexpr int DI = 128;
constexpr int QLD = DI + 4;  // padded fp32 row stride: conflict-free 16-byte reads with lane = head

__device__ __forceinline__ float e4m3_to_float(uint8_t v) {
  return __half2float(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)v, __NV_E4M3)));
}

__global__ void __launch_bounds__(256) indexer_logits_kernel(const uint8_t* __restrict__ qc, const float* __restrict__ wf,
                                                             const uint8_t* __restrict__ kvals,
                                                             const float* __restrict__ kscale,
                                                             const int* __restrict__ slots, const int* __restrict__ pos,
                                                             const int* __restrict__ page_table, int ld_pt, int ps,
                                                             float* __restrict__ logits, int width, int heads) {
  pdl_entry();
  extern __shared__ __align__(16) float ix_smem[];
  float* qs = ix_smem;                  // [heads][QLD]
  float* ks = qs + heads * QLD;         // [8 warps][DI]
  const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j0 = blockIdx.y * 64;
  const int n = (pos[t] + 1) >> 2;
  if (j0 >= width) return;
  if (j0 >= n) {
    for (int j = j0 + tid; j < min(j0 + 64, width); j += 256) logits[(size_t)t * width + j] = -INFINITY;
    return;
  }
  for (int i = tid; i < heads * DI; i += 256) qs[(i / DI) * QLD + (i % DI)] = e4m3_to_float(qc[(size_t)t * heads * DI + i]);
  __syncthreads();
  const int* pt = page_table + (size_t)slots[t] * ld_pt;
  const int hpl = heads / 32;  // heads per lane (1 or 2)
  float w0 = wf[(size_t)t * heads + lane], w1 = hpl > 1 ? wf[(size_t)t * heads + lane + 32] : 0.f;
  float* kw = ks + warp * DI;
  for (int j = j0 + warp; j < min(j0 + 64, width); j += 8) {
    float out = -INFINITY;
    if (j < n) {
      const int loc = pt[4 * j + 3];
      const size_t row = (size_t)(loc / ps) * (ps / 4) + (loc % ps) / 4;
      const uint32_t kk = *reinterpret_cast<const uint32_t*>(kvals + row * DI + lane * 4);
      __syncwarp();
      kw[lane * 4 + 0] = e4m3_to_float(kk & 0xff);
      kw[lane * 4 + 1] = e4m3_to_float((kk >> 8) & 0xff);
      kw[lane * 4 + 2] = e4m3_to_float((kk >> 16) & 0xff);
      kw[lane * 4 + 3] = e4m3_to_float((kk >> 24) & 0xff);
      __syncwarp();
      float d0 = 0.f, d1 = 0.f;
      const float* q0 = qs + lane * QLD;
      const float* q1 = qs + (lane + 32) * QLD;
#pragma unroll 8
      for (int d = 0; d < DI; d += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(kw + d);
        const float4 a = *reinterpret_cast<const float4*>(q0 + d);
        d0 = fmaf(a.x, kv.x, d0), d0 = fmaf(a.y, kv.y, d0), d0 = fmaf(a.z, kv.z, d0), d0 = fmaf(a.w, kv.w, d0);
        if (hpl > 1) {
          const float4 b = *reinterpret_cast<const float4*>(q1 + d);
          d1 = fmaf(b.x, kv.x, d1), d1 = fmaf(b.y, kv.y, d1), d1 = fmaf(b.z, kv.z, d1), d1 = fmaf(b.w, kv.w, d1);
        }
      }
      float s = fmaxf(d0, 0.f) * w0 + fmaxf(d1, 0.f) * w1;
      s = warp_sum(s);
      out = s * kscale[row];
    }
    if (lane == 0) logits[(size_t)t * width + j] = out;
  }
}

// ------------------------------------------------------------------ top-k
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Exclusive prefix of v over the NT threads of the CTA, total = their sum.
template <int NT>
__device__ __forceinline__ int block_excl_scan(int v, int* warp_tot, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) warp_tot[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = lane < NT / 32 ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < NT / 32) warp_tot[lane] = s;
  }
  __syncthreads();
  total = warp_tot[NT / 32 - 1];
  return x - v + (w ? warp_tot[w - 1] : 0);
}

constexpr int kTopBins = 2048;   // equal parts of the row's range of values
constexpr int kTopList = 512;    // entries of the k-th one's part that are put in order

// One CTA per row.  The k-th largest value lies in one of 2 048 equal parts of the row's range of values, found by counting; the few
// entries of that part (about ten of 8 000 normal scores) are ranked against each other, which gives the last selected entry, and
// one ordered pass writes what is not below it.  A row whose part holds more than kTopList entries (equal scores, one far outlier)
// finds the k-th key byte by byte instead.  The four passes read registers: V float4 a thread hold the row of up to NT * 4 * V
// entries, a warp consecutive ones (V = 0: longer rows, read again by each pass).
// Bound by the steps of one row, not by its bytes: rows in flight hide them (512 threads for the rows of prompts: three CTAs an SM).
// In us, against four passes over key bytes whose 256 counts one thread walked: 4 096 rows of 8 192 normal scores 127 / 651, of equal ones
// 253 / 877, with one far outlier 258 / 650; 2 048 rows of 32 768: 255 / 823, equal 573 / 897; 512 rows of 65 536: 153 / 419, equal
// 298 / 452.  Rows with a score that is not finite, which end after the first pass, are the slower ones beyond 8 192 entries: 2 048 rows of
// 32 768 73 / 53, 512 of 65 536 37 / 28.
template <int NT, int V>
__global__ void __launch_bounds__(NT, NT == 512 ? 3 : 1) topk_kernel(const float* __restrict__ logits, int width,
                                                  const int* __restrict__ pos, int* __restrict__ idx,
                                                  int* __restrict__ out_len, int k) {
  pdl_entry();
  __shared__ int hist[kTopBins];
  __shared__ unsigned long long list[kTopList];
  __shared__ int wt[32];
  __shared__ float smin[32], smax[32];
  __shared__ int sh_bad, sh_bin, sh_above, sh_n;
  __shared__ unsigned long long sh_last;
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int n = min((pos[t] + 1) >> 2, width);
  int* oi = idx + (size_t)t * k;
  if (n <= k) {
    for (int i = tid; i < k; i += NT) oi[i] = i < n ? i : -1;
    if (tid == 0) out_len[t] = n;
    return;
  }
  const float* row = logits + (size_t)t * width;
  const bool vec = ((reinterpret_cast<uintptr_t>(logits) & 15) | (width & 3)) == 0;
  auto load = [&](int i) -> float4 {   // entries i .. i + 3 (i a multiple of four); those from n on are not looked at
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
      if (i < n) x = *reinterpret_cast<const float4*>(row + i);
    } else {
      if (i < n) x.x = row[i];
      if (i + 1 < n) x.y = row[i + 1];
      if (i + 2 < n) x.z = row[i + 2];
      if (i + 3 < n) x.w = row[i + 3];
    }
    return x;
  };
  // a warp's entries: `per` consecutive ones, 128 at a time
  const int per = V ? 128 * V : (((n + NT / 32 - 1) / (NT / 32) + 127) & ~127);
  const int first = w * per + 4 * lane;
  float4 held[V ? V : 1];
  if (V) {
#pragma unroll
    for (int u = 0; u < V; ++u) held[u] = load(first + 128 * u);
  }
  auto each4 = [&](auto f) {           // f(four values, id of the first); a warp's lanes stay together
    if (V) {
#pragma unroll
      for (int u = 0; u < V; ++u) f(held[u], first + 128 * u);
    } else {
      for (int i = 0; i < per && w * per + i < n; i += 512) {      // four loads in flight
        float4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = i + 128 * u < per ? load(first + i + 128 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + 128 * u < per && w * per + i + 128 * u < n) f(x[u], first + i + 128 * u);
      }
    }
  };
  auto each = [&](auto f) {
    each4([&](const float4& x, int i) {
      if (i < n) f(x.x, i);
      if (i + 1 < n) f(x.y, i + 1);
      if (i + 2 < n) f(x.z, i + 2);
      if (i + 3 < n) f(x.w, i + 3);
    });
  };
  for (int i = tid; i < kTopBins; i += NT) hist[i] = 0;
  if (tid == 0) sh_bad = 0, sh_n = 0;
  float mn = INFINITY, mx = -INFINITY;
  bool bad = false;
  each([&](float x, int) { bad |= !isfinite(x), mn = fminf(mn, x), mx = fmaxf(mx, x); });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o)), mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) smin[w] = mn, smax[w] = mx;
  __syncthreads();
  if (bad) sh_bad = 1;
  for (int i = 0; i < NT / 32; ++i) mn = fminf(mn, smin[i]), mx = fmaxf(mx, smax[i]);
  __syncthreads();
  if (sh_bad) {
    for (int i = tid; i < k; i += NT) oi[i] = -1;
    if (tid == 0) out_len[t] = -1;
    return;
  }
  // part 0 holds the largest values; a range that overflows or has no width puts all into one part, which the list then refuses
  const float scale = (float)kTopBins / (mx - mn);
  auto part = [&](float x) { return min(max(__float2int_rz((mx - x) * scale), 0), kTopBins - 1); };
  auto entry = [](uint32_t key, int id) { return (unsigned long long)key << 32 | (0xffffffffu - (uint32_t)id); };
  each([&](float x, int) { atomicAdd(&hist[part(x)], 1); });
  __syncthreads();
  {
    constexpr int B = kTopBins / NT;
    int c[B], sum = 0, tot;
#pragma unroll
    for (int j = 0; j < B; ++j) sum += c[j] = hist[B * tid + j];
    int above = block_excl_scan<NT>(sum, wt, tot);
#pragma unroll
    for (int j = 0; j < B; ++j) {
      if (above < k && above + c[j] >= k) sh_bin = B * tid + j, sh_above = above;
      above += c[j];
    }
  }
  __syncthreads();
  const int bin = sh_bin;
  each([&](float x, int i) {
    if (part(x) == bin) {
      const int at = atomicAdd(&sh_n, 1);
      if (at < kTopList) list[at] = entry(order_key(x), i);
    }
  });
  __syncthreads();
  const int m = sh_n, rem = k - sh_above;     // the rem-th largest of the list is the last selected
  if (m <= kTopList) {
    for (int i = tid; i < m; i += NT) {
      const unsigned long long e = list[i];
      int larger = 0;
      for (int j = 0; j < m; ++j) larger += list[j] > e;
      if (larger == rem - 1) sh_last = e;
    }
  } else {
    uint32_t prefix = 0, mask = 0;
    int left = k;  // how many still to take among entries matching the prefix
    for (int shift = 24; shift >= 0; shift -= 8) {
      __syncthreads();
      for (int i = tid; i < 256; i += NT) hist[i] = 0;
      __syncthreads();
      each([&](float x, int) {
        const uint32_t key = order_key(x);
        if ((key & mask) == prefix) atomicAdd(&hist[255 - ((key >> shift) & 0xff)], 1);
      });
      __syncthreads();
      int tot;
      const int c = tid < 256 ? hist[tid] : 0, above = block_excl_scan<NT>(c, wt, tot);
      if (above < left && above + c >= left) sh_bin = 255 - tid, sh_above = above;
      __syncthreads();
      prefix |= (uint32_t)sh_bin << shift;
      mask |= 0xffu << shift;
      left -= sh_above;
    }
    // of the entries equal to the k-th key the first `left` by index: the warp that holds the last of them names it
    int eq = 0, tot;
    each([&](float x, int) { eq += order_key(x) == prefix; });
    eq = __reduce_add_sync(0xffffffffu, eq);
    int before = block_excl_scan<NT>(lane == 0 ? eq : 0, wt, tot);
    before = __shfl_sync(0xffffffffu, before, 0);
    if (before < left && before + eq >= left) {
      each4([&](const float4& x, int i) {
        const float v[4] = {x.x, x.y, x.z, x.w};
        unsigned bits = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) bits |= (unsigned)(i + c < n && order_key(v[c]) == prefix) << c;
        int rank = before, here = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const unsigned all = __ballot_sync(0xffffffffu, bits >> c & 1);
          rank += __popc(all & ((1u << lane) - 1)), here += __popc(all);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (bits >> c & 1) {
            if (++rank == left) sh_last = entry(prefix, i + c);
          }
        before += here;
      });
    }
  }
  __syncthreads();
  const unsigned long long last = sh_last;
  int mine = 0, tot;
  each([&](float x, int i) { mine += entry(order_key(x), i) >= last; });
  mine = __reduce_add_sync(0xffffffffu, mine);
  int p = block_excl_scan<NT>(lane == 0 ? mine : 0, wt, tot);
  p = __shfl_sync(0xffffffffu, p, 0);
  if (mine > 0) {
    each4([&](const float4& x, int i) {
      const float v[4] = {x.x, x.y, x.z, x.w};
      unsigned bits = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) bits |= (unsigned)(i + c < n && entry(order_key(v[c]), i + c) >= last) << c;
      int at = p;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const unsigned all = __ballot_sync(0xffffffffu, bits >> c & 1);
        at += __popc(all & ((1u << lane) - 1)), p += __popc(all);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (bits >> c & 1) {
          if (at < k) oi[at] = i + c;
          ++at;
        }
    });
  }
  if (tid == 0) out_len[t] = k;
}

}  // namespace

DSV4_API int dsv4_indexer_logits(const void* qc, const float* wf, const void* kvals, const float* kscale,
                                 const int* slots, const int* pos, const int* page_table, int ld_pt, int ps,
                                 float* logits, int width, int t, int heads, int d, cudaStream_t st) {
  if (t <= 0 || width <= 0) return 0;
  if (d != DI || (heads != 32 && heads != 64)) return 400;
  const int smem = (heads * QLD + 8 * DI) * 4;
  dim3 grid(t, (width + 63) / 64);
  dsv4_launch(indexer_logits_kernel, grid, 256, smem, st, (const uint8_t*)qc, wf, (const uint8_t*)kvals, kscale, slots, pos,
                                                 page_table, ld_pt, ps, logits, width, heads);
  return (int)cudaGetLastError();
}

DSV4_API int dsv4_topk(const float* logits, int width, const int* pos, int* idx, int* out_len, int t, int k,
                       cudaStream_t st) {
  if (t <= 0) return 0;
  // 16 or 32 entries a thread in registers
  if (width <= 512 * 16)
    dsv4_launch(topk_kernel<512, 4>, t, 512, 0, st, logits, width, pos, idx, out_len, k);
  else if (width <= 1024 * 32)
    dsv4_launch(topk_kernel<1024, 8>, t, 1024, 0, st, logits, width, pos, idx, out_len, k);
  else
    dsv4_launch(topk_kernel<1024, 0>, t, 1024, 0, st, logits, width, pos, idx, out_len, k);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------ allocation-free entry point (see noalloc.h)
#include "noalloc.h"

#include <stdio.h>

namespace {
// The logits workspace of the allocation-free entry point.  In host code this name is only a handle for the runtime
// (taking its address on the host does NOT give a device pointer); kernels get the address from cudaGetSymbolAddress.
static __device__ __align__(256) float g_noalloc_logits[DSV4_NOALLOC_MAX_ELEMS];
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {};
thread_local char g_noalloc_err[256] = "";
}  // namespace

DSV4_API const char* dsv4_noalloc_last_error(void) { return g_noalloc_err; }

DSV4_API int dsv4_indexer_select_noalloc(const void* qc, const float* wf, const void* kvals, const float* kscale,
                                         const int* slots, const int* pos, const int* page_table, int ld_pt, int ps,
                                         int width, int t, int heads, int d, int* idx, int* out_len, int k,
                                         cudaStream_t stream) {
  g_noalloc_err[0] = 0;
  if (t <= 0) return 0;
  if (width <= 0 || (unsigned long long)t * (unsigned long long)width > DSV4_NOALLOC_MAX_ELEMS) {
    snprintf(g_noalloc_err, sizeof g_noalloc_err,
             "dsv4_indexer_select_noalloc: t * width = %d * %d exceeds the built-in workspace of %u floats; "
             "split the batch or use dsv4_indexer_logits + dsv4_topk with your own buffer",
             t, width, DSV4_NOALLOC_MAX_ELEMS);
    return 460;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    snprintf(g_noalloc_err, sizeof g_noalloc_err, "dsv4_indexer_select_noalloc: cannot identify the current device");
    return 461;
  }
  if (!g_noalloc_ptr[dev]) {  // once per device, with that device current
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_noalloc_logits);
    if (e != cudaSuccess || !p) {
      snprintf(g_noalloc_err, sizeof g_noalloc_err, "dsv4_indexer_select_noalloc: cudaGetSymbolAddress failed: %s",
               cudaGetErrorString(e));
      return 461;
    }
    g_noalloc_ptr[dev] = p;
  }
  float* logits = g_noalloc_ptr[dev];
  int rc = dsv4_indexer_logits(qc, wf, kvals, kscale, slots, pos, page_table, ld_pt, ps, logits, width, t, heads, d,
                               stream);
  if (rc == 0) rc = dsv4_topk(logits, width, pos, idx, out_len, t, k, stream);
  if (rc != 0) snprintf(g_noalloc_err, sizeof g_noalloc_err, "dsv4_indexer_select_noalloc: launch failed with code %d", rc);
  return rc;
}
