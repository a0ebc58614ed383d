// Projections of a few rows (decode of a few requests):  out[M,N] = X[M,K] W[N,K]^T  for M <= 24 in bf16 or M <= 16 in e4m3 with
// power-of-two block scales (as in gemm_tcgen05.cu); ops/gemm.py (few_rows) says which sizes come here.  Weights are read once and that
// is the time: 33.5 MB take 5.2 us at the HBM rate.
//
// One CTA per output tile with tensor memory, a TMA ring and a cluster reduction (gemm_tcgen05.cu) spends most of its life starting and
// ending at this size.  Here a warp loads 16 weight rows straight into registers, 16 bytes a lane, as the A operand of
// mma.sync m16n8k16 (rows of X are the 8 columns), one batch of loads ahead of the products; the 8 warps of a CTA share K between
// them as far as the output leaves SMs idle, and add their sums in order in shared memory.  Nothing waits on anything else before that.
// The first 8 columns are nearly free (4 096 x 4 096 in bf16: 8.1 us for one row, 8.7 for eight, 10.8 for 24; 28 to 19 in tiles).
// e4m3 has conversions in front of each product, which with 16 rows outweigh what tiles cost from about 8 192 weight rows on
// (32 768 x 1 024: 12.7 us for one row, 18.2 for 16; 15 in tiles).
//
// A lane's 16 bytes are consecutive places of K of one weight row, and the same places of one row of X: the order of the contraction
// is free as long as both operands agree.  e4m3 becomes f16 exactly, a product of two fits fp32, and every 128 places the fp32 sum is
// scaled by its exact power of two and added to the total.
//
// Weights do not depend on the kernel before: the first batch is asked for ahead of the dependent-launch wait.
#include "vec.cuh"

int dsv4_weight_prefetch();      // gemm_tcgen05.cu

namespace {

constexpr int kWarps = 8, kU = 4;          // segments (64 bytes of K) per batch

struct RowsArgs {
  const uint8_t *x, *w;
  void* out;
  const float *sa, *sb;
  int M, N, K;
  long long ldx, ldw, ldo;      // bytes, bytes, elements
  int kw;                       // warps that share K
  int accumulate, prefetch;
};

__device__ __forceinline__ uint4 ld_stream(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t f16_of(uint32_t two) {      // two e4m3 in the low half -> two f16
  const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)two, __NV_E4M3);
  return (uint32_t)h.x | (uint32_t)h.y << 16;
}
template <bool FP8>
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (FP8)
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int NTL, bool FP8, typename OutT>
__global__ void __launch_bounds__(kWarps * 32, 2) gemm_rows_kernel(const RowsArgs a) {
  __shared__ float part[kWarps][8 * NTL][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tiles = kWarps / a.kw, tile = warp / a.kw, kp = warp % a.kw;      // row tiles of the CTA, this warp's, its share of K
  const int batch = blockIdx.y, n0 = (blockIdx.x * tiles + tile) * 16;
  const int kbytes = a.K * (FP8 ? 1 : 2), nseg = kbytes / 64;
  const int per = ((nseg + a.kw - 1) / a.kw + 1) & ~1;
  const int lo = min(kp * per, nseg), hi = min(lo + per, nseg);
  const size_t wrow = (size_t)batch * a.N;
  const uint8_t* w0 = a.w + (wrow + min(n0 + g, a.N - 1)) * a.ldw + t * 16;
  const uint8_t* w1 = a.w + (wrow + min(n0 + g + 8, a.N - 1)) * a.ldw + t * 16;
  uint4 wv[kU][2];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (s0 + u < hi) wv[u][0] = ld_stream(w0 + (size_t)(s0 + u) * 64), wv[u][1] = ld_stream(w1 + (size_t)(s0 + u) * 64);
  };
  if (a.prefetch) fetch(lo);
  pdl_wait();
  pdl_launch_dependents();
  if (!a.prefetch) fetch(lo);
  const uint8_t* x[NTL];
#pragma unroll
  for (int j = 0; j < NTL; ++j) x[j] = a.x + min(8 * j + g, a.M - 1) * a.ldx + (size_t)batch * kbytes + t * 16;
  const int nkb = a.K / 128;
  const float* sb = FP8 ? a.sb + (size_t)(min(n0, a.N - 1) >> 7) * nkb : nullptr;
  float acc[NTL][4] = {}, sum[NTL][4] = {};
  uint32_t bits = 0;            // of all block scales read: no sign and no mantissa if each is a power of two
  for (int s0 = lo; s0 < hi; s0 += kU) {
    uint4 wc[kU][2], xv[kU][NTL];
    float f0[kU / 2][NTL], f1[kU / 2][NTL];      // scales of a block of 128 places and this lane's two rows of X
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      wc[u][0] = wv[u][0], wc[u][1] = wv[u][1];
      const int s = min(s0 + u, hi - 1);
#pragma unroll
      for (int j = 0; j < NTL; ++j) xv[u][j] = *reinterpret_cast<const uint4*>(x[j] + (size_t)s * 64);
      if (FP8 && (u & 1)) {
        const float sw = sb[s >> 1];
        bits |= __float_as_uint(sw);
#pragma unroll
        for (int j = 0; j < NTL; ++j) {
          const float r0 = a.sa[(size_t)min(8 * j + 2 * t, a.M - 1) * nkb + (s >> 1)];
          const float r1 = a.sa[(size_t)min(8 * j + 2 * t + 1, a.M - 1) * nkb + (s >> 1)];
          bits |= __float_as_uint(r0) | __float_as_uint(r1);
          f0[u >> 1][j] = r0 * sw, f1[u >> 1][j] = r1 * sw;
        }
      }
    }
    fetch(s0 + kU);
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (s0 + u >= hi) break;
      const uint32_t* p0 = reinterpret_cast<const uint32_t*>(&wc[u][0]);
      const uint32_t* p1 = reinterpret_cast<const uint32_t*>(&wc[u][1]);
      if constexpr (FP8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {      // four places of K per word: 2t, 2t + 1 and 2t + 8, 2t + 9 of a product
          const uint32_t a0 = f16_of(p0[i] & 0xffff), a2 = f16_of(p0[i] >> 16), a1 = f16_of(p1[i] & 0xffff), a3 = f16_of(p1[i] >> 16);
#pragma unroll
          for (int j = 0; j < NTL; ++j) {
            const uint32_t b = reinterpret_cast<const uint32_t*>(&xv[u][j])[i];
            mma<true>(sum[j], a0, a1, a2, a3, f16_of(b & 0xffff), f16_of(b >> 16));
          }
        }
        if (u & 1) {                       // the end of 128 places (a warp's share is whole blocks)
#pragma unroll
          for (int j = 0; j < NTL; ++j) {
            acc[j][0] = fmaf(sum[j][0], f0[u >> 1][j], acc[j][0]), acc[j][1] = fmaf(sum[j][1], f1[u >> 1][j], acc[j][1]);
            acc[j][2] = fmaf(sum[j][2], f0[u >> 1][j], acc[j][2]), acc[j][3] = fmaf(sum[j][3], f1[u >> 1][j], acc[j][3]);
            sum[j][0] = sum[j][1] = sum[j][2] = sum[j][3] = 0.f;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; i += 2)
#pragma unroll
          for (int j = 0; j < NTL; ++j) {
            const uint32_t* b = reinterpret_cast<const uint32_t*>(&xv[u][j]);
            mma<false>(acc[j], p0[i], p1[i], p0[i + 1], p1[i + 1], b[i], b[i + 1]);
          }
      }
    }
  }
  if (FP8 && (bits & 0x807fffffu)) dsv4_set_error(DSV4_ERR_BAD_INDEX, 41, (int)blockIdx.x);      // a scale that is not a power of two
#pragma unroll
  for (int j = 0; j < NTL; ++j) {
    part[warp][8 * j + 2 * t][g] = acc[j][0], part[warp][8 * j + 2 * t + 1][g] = acc[j][1];
    part[warp][8 * j + 2 * t][g + 8] = acc[j][2], part[warp][8 * j + 2 * t + 1][g + 8] = acc[j][3];
  }
  __syncthreads();
  const int cols = 16 * tiles;
  for (int i = threadIdx.x; i < a.M * cols; i += kWarps * 32) {
    const int m = i / cols, c = i % cols, n = blockIdx.x * cols + c;
    if (n >= a.N) continue;
    float v = 0.f;
    for (int k = 0; k < a.kw; ++k) v += part[(c >> 4) * a.kw + k][m][c & 15];
    OutT* dst = reinterpret_cast<OutT*>(a.out) + (size_t)m * a.ldo + wrow + n;
    if (a.accumulate) v += ld_f(dst);
    st_f(dst, v);
  }
}

template <bool FP8, typename OutT>
int launch(const RowsArgs& a, int batches, cudaStream_t st) {
  const int per_cta = 16 * (kWarps / a.kw);
  const dim3 grid((a.N + per_cta - 1) / per_cta, batches);
  if (a.M <= 8)
    dsv4_launch(gemm_rows_kernel<1, FP8, OutT>, grid, kWarps * 32, 0, st, a);
  else if (FP8 || a.M <= 16)
    dsv4_launch(gemm_rows_kernel<2, FP8, OutT>, grid, kWarps * 32, 0, st, a);
  else if constexpr (!FP8)
    dsv4_launch(gemm_rows_kernel<3, FP8, OutT>, grid, kWarps * 32, 0, st, a);
  return (int)cudaGetLastError();
}

// Warps that share K: as few as give two CTAs (16 warps, 64 KiB of weights in flight) to each SM.
int share_k(int N, int batches, int nseg) {
  int kw = 1;
  while (kw < kWarps && (long long)(N + 15) / 16 * batches * kw < 148 * 16 && nseg / (2 * kw) >= 4) kw *= 2;
  return kw;
}

}  // namespace

// bf16: batches as in dsv4_gemm_bf16 (batch b reads columns b K .. of x and rows b N .. of w, and writes columns b N ..).
// x, w and their rows start on 16 bytes; K a multiple of 32.
DSV4_API int dsv4_gemm_rows_bf16(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldo, int out_fp32,
                                 int accumulate, int batches, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 24 || K <= 0 || K % 32 || ldx % 8 || ldw % 8 || batches < 1 || batches > 65535 || (((uintptr_t)x | (uintptr_t)w) & 15)) return 680;
  const RowsArgs a{(const uint8_t*)x, (const uint8_t*)w, out, nullptr, nullptr, M, N, K, 2ll * ldx, 2ll * ldw, ldo,
                   share_k(N, batches, K / 32), accumulate, dsv4_weight_prefetch()};
  return out_fp32 ? launch<false, float>(a, batches, st) : launch<false, __nv_bfloat16>(a, batches, st);
}
// x: e4m3 [M,K] with sa fp32 [M, K/128];  w: e4m3 [N,K] with sb fp32 [ceil(N/128), K/128].
DSV4_API int dsv4_gemm_rows_fp8(const void* x, const void* w, void* out, const float* sa, const float* sb, int M, int N, int K, int ldx,
                                int ldw, int ldo, int out_fp32, int accumulate, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 16 || K <= 0 || K % 128 || ldx % 16 || ldw % 16 || (((uintptr_t)x | (uintptr_t)w) & 15)) return 681;
  const RowsArgs a{(const uint8_t*)x, (const uint8_t*)w, out, sa, sb, M, N, K, ldx, ldw, ldo, share_k(N, 1, K / 64), accumulate,
                   dsv4_weight_prefetch()};
  return out_fp32 ? launch<true, float>(a, 1, st) : launch<true, __nv_bfloat16>(a, 1, st);
}
