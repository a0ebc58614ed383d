// e4m3 projections of many rows with power-of-two block scales: the persistent counterpart of gemm_tcgen05.cu's FP8 path, as
// gemm_prefill.cu is for bf16.  out[M,N] = sum over 128-wide K blocks of  sa[row,kb] sw[n / 128,kb] (X W^T)_kb,  the scales applied by
// the block-scaled MMA, one fp32 accumulator over the whole K range.
//
// One CTA per SM walks 128 x 192 output tiles, with the accumulator in tensor memory twice, so that a tile's epilogue runs under the next
// tile's MMAs.  192 columns are the widest multiple of the 32 that the epilogue loads at once with which five stages fit shared memory
// (42 KiB each; 224 columns leave room for four).  Wider tiles ask less of shared memory: per MMA it reads 128 + 192 rows for 128 x 192
// results, a square tile of 128 a fifth more for each.
//   warp 0 TMA producer (5 stages of 128 K elements), warp 1 MMA issuer, warps 2-5 epilogue
//   warps 6-9 scales: each stage carries a 512-byte block of row scales and two of column scales (a tile's columns lie in two
//   128-row blocks of the weight), written next to the operands eight K blocks ahead of the loads' latency
#include "vec.cuh"

namespace {

constexpr int kM = 128, kN = 192, kStages = 5;
constexpr int kA = kM * 128, kB = kN * 128, kSf = 3 * 512, kStage = kA + kB + kSf;
constexpr int kOperands = kA + kB;
constexpr int kPad = (kStage + 1023) & ~1023;              // stages start on whole swizzle atoms
constexpr int kSmem = kStages * kPad + 1024 + 256;
constexpr int kGroupRows = 16;                             // row tiles that share a column of weight tiles before the next column
constexpr int kThreads = 320;

struct Args {
  int M, N, K, ldo, accumulate, mt, nt, w_blocks;
  const float *sa, *sb;      // [M, K / 128], [w_blocks, K / 128]
};

__device__ __forceinline__ void tile_of(const Args& g, int id, int& m, int& n) {
  const int gid = id / (kGroupRows * g.nt), m_first = gid * kGroupRows;
  const int rows = min(kGroupRows, g.mt - m_first), in = id - gid * kGroupRows * g.nt;
  m = m_first + in % rows;
  n = in / rows;
}

template <typename OutT>
__global__ void __launch_bounds__(kThreads, 1) gemm_prefill_fp8_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                       const __grid_constant__ CUtensorMap tmB,
                                                                       OutT* __restrict__ out, const Args g) {
  extern __shared__ uint8_t fsm_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fsm_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kPad);
  uint64_t *empty = full + kStages, *tfull = empty + kStages, *tempty = tfull + 2, *drain = tempty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) mbar_init(&full[i], 5), mbar_init(&empty[i], 1);    // the copies and four warps of scales
    for (int i = 0; i < 2; ++i) mbar_init(&tfull[i], 1), mbar_init(&tempty[i], 4);
    mbar_init(drain, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  pdl_wait();
  pdl_launch_dependents();
  const int total = g.mt * g.nt, nkt = g.K / 128;

  if (warp == 0) {
    if (lane == 0) {
      int i = 0;
      bool ok = true;
      for (int id = blockIdx.x; id < total && ok; id += gridDim.x) {
        int m, n;
        tile_of(g, id, m, n);
        for (int k = 0; k < nkt; ++k, ++i) {
          const int s = i % kStages;
          if (i >= kStages && !mbar_wait<20>(&empty[s], ((i / kStages) & 1) ^ 1, abort_flag, 61)) { ok = false; break; }
          uint8_t* st = smem + s * kPad;
          mbar_expect_tx(&full[s], kOperands);
          tma_load_2d(st, &tmA, &full[s], k * 128, m * kM);
          tma_load_2d(st + kA, &tmB, &full[s], k * 128, n * kN);
        }
      }
    }
  } else if (warp == 1) {
    // all lanes walk these loops: three copies of scales and four MMAs per stage, issued by a branch of one lane, took 815 us in the four
    // projections of an attention block, 730 us so
    const bool lead = elect_one();
    constexpr uint32_t kIdesc = umma_idesc_mx(kM, kN, 0, 0);
    int i = 0, it = 0;
    bool ok = true;
    for (int id = blockIdx.x; id < total && ok; id += gridDim.x, ++it) {
      const int acc = it & 1;
      if (it >= 2 && !mbar_wait(&tempty[acc], ((it >> 1) & 1) ^ 1, abort_flag, 62)) break;
      tc_fence_after();
      for (int k = 0; k < nkt; ++k, ++i) {
        const int s = i % kStages;
        if (!mbar_wait(&full[s], (i / kStages) & 1, abort_flag, 63)) { ok = false; break; }
        tc_fence_after();
        const uint8_t* st = smem + s * kPad;
        const uint32_t sft = tmem + 2 * kN + (i & 1) * 12;
        const uint64_t da = umma_desc_k128(st, 0), db = umma_desc_k128(st + kA, 0);
        if (lead) {
#pragma unroll
          for (int c = 0; c < 3; ++c) tmem_cp_sf(sft + 4 * c, st + kOperands + c * 512);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_mx(tmem + acc * kN, da + 2 * j, db + 2 * j, kIdesc, j, sft, sft + 4, k > 0 || j > 0);
          umma_commit(&empty[s]);
        }
      }
      if (ok && lead) umma_commit(&tfull[acc]);
    }
  } else if (warp >= 6) {
    // thread r: row r of the tile, columns r and 128 + r
    const int r = threadIdx.x - 192, word = (r & 31) * 4 + (r >> 5);
    int i = 0;
    bool ok = true, pow2 = true;
    for (int id = blockIdx.x; id < total && ok; id += gridDim.x) {
      int m, n;
      tile_of(g, id, m, n);
      const int row = m * kM + r;
      const float* sa = g.sa + (size_t)min(row, g.M - 1) * nkt;
      const float* sb0 = g.sb + (size_t)min((n * kN + r) >> 7, g.w_blocks - 1) * nkt;
      const float* sb1 = g.sb + (size_t)min((n * kN + 128 + r) >> 7, g.w_blocks - 1) * nkt;
      for (int k0 = 0; k0 < nkt && ok; k0 += 8) {
        uint32_t a[8], b0[8], b1[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int k = min(k0 + j, nkt - 1);
          a[j] = __float_as_uint(sa[k]), b0[j] = __float_as_uint(sb0[k]), b1[j] = __float_as_uint(sb1[k]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (k0 + j >= nkt || !ok) continue;
          const int s = i % kStages;
          if (i >= kStages) ok = mbar_wait<20>(&empty[s], ((i / kStages) & 1) ^ 1, abort_flag, 64);
          pow2 = pow2 && !((a[j] | b0[j] | b1[j]) & 0x807fffffu);
          uint32_t* blk = reinterpret_cast<uint32_t*>(smem + s * kPad + kOperands) + word;
          blk[0] = (a[j] >> 23) * 0x01010101u;
          blk[128] = (b0[j] >> 23) * 0x01010101u;
          blk[256] = (b1[j] >> 23) * 0x01010101u;
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[s]);
          ++i;
        }
      }
    }
    if (!pow2) dsv4_set_error(DSV4_ERR_BAD_INDEX, 41, (int)blockIdx.x);      // a scale that is not a power of two
  } else {
    const int q = warp & 3;
    int it = 0;
    for (int id = blockIdx.x; id < total; id += gridDim.x, ++it) {
      const int acc = it & 1;
      int m, n;
      tile_of(g, id, m, n);
      if (!mbar_wait<40>(&tfull[acc], (it >> 1) & 1, abort_flag, 65)) break;
      tc_fence_after();
      const int row = m * kM + q * 32 + lane;
      const uint32_t d0 = tmem + acc * kN + ((uint32_t)(q * 32) << 16);
      OutT* dst = out + (size_t)row * g.ldo + n * kN;
      const int cols = min(kN, g.N - n * kN);
      const bool vec = ((uintptr_t)dst & 15) == 0;
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(d0 + c, r);
        tmem_ld_wait();
        if (row < g.M) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          st_row32(dst + c, v, cols - c, vec, g.accumulate);
        }
        __syncwarp();      // the next columns are loaded by the warp as a whole
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) drain_after_abort(drain, elect_one());
    tmem_dealloc(tmem, 512);
  }
}

template <typename OutT>
int launch(const CUtensorMap& a, const CUtensorMap& b, void* out, const Args& g, int sms, cudaStream_t st) {
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(gemm_prefill_fp8_kernel<OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess)
      return 673;
    set = true;
  }
  const int total = g.mt * g.nt;
  dsv4_launch(gemm_prefill_fp8_kernel<OutT>, total < sms ? total : sms, kThreads, kSmem, st, a, b, (OutT*)out, g);
  return (int)cudaGetLastError();
}

}  // namespace

// x: e4m3 [M,K] with sa fp32 [M, K/128];  w: e4m3 [N,K] with sb fp32 [ceil(N/128), K/128].
DSV4_API int dsv4_gemm_prefill_fp8(const void* x, const void* w, void* out, const float* sa, const float* sb, int M, int N, int K,
                                   int ldx, int ldw, int ldo, int out_fp32, int accumulate, int sms, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 128 || K <= 0 || ldx % 16 || ldw % 16 || sms < 1) return 670;
  CUtensorMap ta, tb;
  if (dsv4_make_tmap_2d(&ta, x, 0, K, M, (uint64_t)ldx, 128, kM, 3)) return 671;
  if (dsv4_make_tmap_2d(&tb, w, 0, K, N, (uint64_t)ldw, 128, kN, 3)) return 672;
  const Args g{M, N, K, ldo, accumulate, (M + kM - 1) / kM, (N + kN - 1) / kN, (N + 127) / 128, sa, sb};
  return out_fp32 ? launch<float>(ta, tb, out, g, sms, st) : launch<__nv_bfloat16>(ta, tb, out, g, sms, st);
}
