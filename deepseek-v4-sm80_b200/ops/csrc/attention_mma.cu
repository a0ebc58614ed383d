// The sparse latent attention of attention.cu for 64 heads, on tcgen05.  Same entry point, same keys, same result up to the order
// of the sums.
//
// Both products are transposed, so that one token is enough for whole 128-row instructions: keys, then output dimensions lie along the
// 128 lanes, the token's 64 heads along the columns.
//   S^T [128 keys x 64]   =  K [128 x 512] Q^T              32 instructions 128 x 64 x 16
//   O^T [512 dims x 64]  +=  V^T [512 x 128] P^T            4 blocks of 128 dims, 8 instructions each
//   l   [64]             +=  1 [128 x 128] P^T              the rows' sums, from the same rounded weights as the product
// K = V: the gathered rows are stored once, as eight [128 keys][64 dims] blocks of 128-byte rows.  Read with the dims contiguous
// they are the K-major operand of S^T, with the keys running over rows the M-major operand of O^T.
//
//   warps 0-7    softmax: a thread holds one key (of its quarter) and 32 heads; a head's maximum is one warp reduction and four
//                values in shared memory.  A head's reference only moves when its maximum has grown by more than 2^8 since.
//   warp 8       tcgen05.mma issuer
//   warps 9-12   gather: a warp per 128-dim block of the key tile (and of Q), cp.async into 128-byte swizzled rows
// A key tile is 128 KiB, so one is resident: its blocks are refilled one after the other as the product with P frees them, under the
// rest of that product, and the next token's first tile loads under this one's epilogue.  CTAs stay and walk (token, split) items.
//
// What bounds it: the chain gather -> S -> softmax -> PV of a tile, and a token's epilogue, whose stores share the load/store path with
// the next gather; shared memory feeds an instruction of 64 columns at two thirds of the tensor core's rate.  8 prompts of 1 024
// tokens (4:1 entries): 840 us, against 2 340 us on the warp-level kernel (attention.cu), which spends four barriers on every 32 keys;
// 128 decoded tokens at 2 000: 43 and 87 us; one token: 16 and 51 us.
// The warp-level kernel stays for 8 to 32 heads, where columns would be padding.
//
// Splits leave unnormalised sums (fp32) with (reference, sum) per head; a second kernel merges them, four heads to a CTA.
#include "common.cuh"
#include "attention.cuh"
#include "mma16.cuh"
#include "rope.cuh"

namespace {

constexpr int D = 512, HL = 64, KT = 128;
constexpr int kSub = KT * 128;                  // bytes of a [128 keys][64 dims] block
constexpr int kQSub = HL * 128;                 // of a [64 heads][64 dims] block
constexpr int kThreads = 13 * 32;
constexpr int kColO = 0, kColS = 256, kColL = 320;

struct TcSmem {
  uint8_t k[8 * kSub];
  uint8_t q[8 * kQSub];
  uint8_t p[KT * 128];          // [key][64 heads] weights
  uint8_t ones[1024];           // an 8-row group of ones; every group of the operand is this one
  float wmax[8][32], ref[8][32], mul[8][32];
  const __nv_bfloat16* rows[2][KT];     // cache rows of a tile's keys, null if masked
  uint64_t full[4], empty[4], s_full, p_full, o_full, drain;
  uint32_t tmem;
  int abort_flag;
};
constexpr int kSmemBytes = (int)sizeof(TcSmem) + 1024;

__device__ __forceinline__ void cp16(uint32_t smem, const void* g, bool valid) {
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(g), "r"(sz) : "memory");
}
__device__ __forceinline__ float redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
// M- or N-major operand whose rows (of the K direction) hold 64 16-bit elements in 128 swizzled bytes: 8-row groups 1 024 bytes
// apart, further 64 elements of M or N kSub bytes apart.
__device__ __forceinline__ uint64_t desc_mn(const void* p) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(p) & 0x3FFFF) >> 4);
  d |= (uint64_t)(kSub >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ uint64_t desc_ones(const void* p) {
  uint64_t d = umma_desc_k128(p, 0);
  return d & ~((uint64_t)0x3FFF << 32);         // groups 0 bytes apart
}

struct Item {
  int t, split, pos, slot, nc, ns, lo, hi;      // keys [lo, hi) of nc + ns
};
__device__ __forceinline__ Item item_of(const AttnArgs& a, int id) {
  Item x;
  x.t = id / a.nsplit, x.split = id % a.nsplit;
  x.pos = a.pos[x.t], x.slot = a.slots[x.t];
  x.nc = 0;
  if (a.mode == 1) x.nc = max(a.topk_len[x.t], 0);
  if (a.mode == 2) x.nc = (x.pos + 1) / a.ratio;
  x.ns = min(x.pos + 1, a.window);
  const int ntot = a.num_valid && x.t >= *a.num_valid ? 0 : max(x.nc + x.ns, 0);
  const int per = ((ntot + KT - 1) / KT + a.nsplit - 1) / a.nsplit * KT;
  x.lo = min(x.split * per, ntot), x.hi = min(x.lo + per, ntot);
  return x;
}

__global__ void __launch_bounds__(kThreads, 1) sparse_attn_mma_kernel(const AttnArgs a, const int items) {
  extern __shared__ uint8_t tsm_raw[];
  TcSmem& sm = *reinterpret_cast<TcSmem*>((reinterpret_cast<uintptr_t>(tsm_raw) + 1023) & ~uintptr_t(1023));
  volatile int* abort_flag = &sm.abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(&sm.full[i], 1), mbar_init(&sm.empty[i], 1);
    mbar_init(&sm.s_full, 1), mbar_init(&sm.p_full, 8), mbar_init(&sm.o_full, 1), mbar_init(&sm.drain, 1);
    sm.abort_flag = 0;
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < 512; i += kThreads) reinterpret_cast<__nv_bfloat16*>(sm.ones)[i] = __float2bfloat16_rn(1.f);
  fence_proxy_async_smem();
  if (warp == 8) {
    tmem_alloc(&sm.tmem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem;
  pdl_wait();
  pdl_launch_dependents();

  if (warp >= 9) {
    const int db = warp - 9, mine = threadIdx.x - 9 * 32;      // dims [128 db, +128); the key of a tile that this thread looks up
    const int rpp = a.ratio > 0 ? max(a.ps / a.ratio, 1) : 1;
    const int side = lane >> 4, ch = lane & 15;                // two rows of 16 pieces at a time
    const uint32_t kb = smem_u32(sm.k + (2 * db + (ch >> 3)) * kSub) + side * 128;
    const uint32_t qb = smem_u32(sm.q + (2 * db + (ch >> 3)) * kQSub) + side * 128;
    uint32_t turn[4];                                          // place of the piece in rows 2 i + side, i % 4
#pragma unroll
    for (int i = 0; i < 4; ++i) turn[i] = ((ch ^ (2 * i + side)) & 7) << 4;
    // Cache row of key base + mine of an item, null if it is masked.  The chain of two or three dependent loads (behind an item's own)
    // runs one tile ahead.
    auto look_up = [&](const Item& x, int base) -> const __nv_bfloat16* {
      const int key = base + mine;
      if (key >= x.hi) return nullptr;
      const int* pt = a.page_table + (size_t)x.slot * a.ld_pt;
      if (key >= x.nc) {
        const int loc = pt[x.pos - x.ns + 1 + (key - x.nc)];
        const int sl = loc >= 0 ? a.swa_map[loc / a.ps] : -1;
        return sl >= 0 ? a.swa + ((size_t)sl * a.ps + loc % a.ps) * D : nullptr;
      }
      const int j = a.mode == 1 ? a.topk_idx[(size_t)x.t * a.topk_width + key] : key;
      const int loc = j >= 0 ? pt[j * a.ratio + a.ratio - 1] : -1;
      return loc >= 0 ? a.comp + ((size_t)(loc / a.ps) * rpp + (loc % a.ps) / a.ratio) * D : nullptr;
    };
    int fill = 0, id = blockIdx.x;
    Item x;
    auto next_item = [&]() {                                   // the first one with keys from id on
      for (; id < items; id += gridDim.x) {
        x = item_of(a, id);
        if (x.lo < x.hi) return;
      }
    };
    next_item();
    int base = id < items ? x.lo : 0;
    const __nv_bfloat16* row = id < items ? look_up(x, base) : nullptr;
    while (id < items) {
      // after a wait that ran out the warps still meet here, and copy nothing
      const __nv_bfloat16** rows = sm.rows[fill & 1];
      rows[mine] = row;
      asm volatile("bar.sync 3, 128;" ::: "memory");
      if (mbar_wait<20>(&sm.empty[db], (fill & 1) ^ 1, abort_flag, 51)) {
        if (base == x.lo) {
          const __nv_bfloat16* q = a.q + ((size_t)x.t * HL + side) * D + db * 128 + ch * 8;
#pragma unroll 1
          for (int i0 = 0; i0 < 32; i0 += 4)
#pragma unroll
            for (int i = 0; i < 4; ++i) cp16(qb + (i0 + i) * 256 + turn[i], q + (size_t)(i0 + i) * (2 * D), true);
        }
#pragma unroll 1
        for (int i0 = 0; i0 < 64; i0 += 8) {
          const __nv_bfloat16* r[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) r[i] = rows[2 * (i0 + i) + side];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            cp16(kb + (i0 + i) * 256 + turn[i & 3], (r[i] ? r[i] : a.swa) + db * 128 + ch * 8, r[i] != nullptr);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      base += KT;
      if (base >= x.hi) {
        id += gridDim.x;
        next_item();
        base = x.lo;
      }
      if (id < items) row = look_up(x, base);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.full[db]);
      ++fill;
    }
  } else if (warp == 8) {
    // all lanes walk these loops (elect_one)
    constexpr uint32_t kIdS = umma_idesc(128, HL, 1, 1);
    constexpr uint32_t kIdO = kIdS | (1u << 15) | (1u << 16);       // both operands M- / N-major
    constexpr uint32_t kIdL = kIdS | (1u << 16);
    const uint64_t ones = desc_ones(sm.ones), k_rows = umma_desc_k128(sm.k, 0), q_rows = umma_desc_k128(sm.q, 0);
    const uint64_t k_cols = desc_mn(sm.k), p_cols = desc_mn(sm.p);
    const bool lead = elect_one();
    int n = 0;
    bool ok = true;
    for (int id = blockIdx.x; id < items && ok; id += gridDim.x) {
      const Item x = item_of(a, id);
      for (int base = x.lo; base < x.hi && ok; base += KT, ++n) {
#pragma unroll 1
        for (int db = 0; db < 4 && ok; ++db) {
          ok = mbar_wait(&sm.full[db], n & 1, abort_flag, 52);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ka = k_rows + (uint64_t)(db * (2 * kSub / 16)), qa = q_rows + (uint64_t)(db * (2 * kQSub / 16));
          if (lead) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              umma_f16(tmem + kColS, ka + (k >> 2) * (kSub / 16) + (k & 3) * 2, qa + (k >> 2) * (kQSub / 16) + (k & 3) * 2, kIdS,
                       db > 0 || k > 0);
          }
        }
        if (!ok) break;
        if (lead) umma_commit(&sm.s_full);
        ok = mbar_wait(&sm.p_full, n & 1, abort_flag, 53);
        if (!ok) break;
        tc_fence_after();
        const uint32_t more = base > x.lo;
#pragma unroll 1
        for (int mb = 0; mb < 4; ++mb) {
          const uint64_t va = k_cols + (uint64_t)(mb * (2 * kSub / 16));
          if (lead) {
#pragma unroll
            for (int k = 0; k < 8; ++k) umma_f16(tmem + kColO + mb * HL, va + k * 128, p_cols + k * 128, kIdO, more || k > 0);
            umma_commit(&sm.empty[mb]);
          }
        }
        if (lead) {
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16(tmem + kColL, ones, p_cols + k * 128, kIdL, more || k > 0);
        }
      }
      if (lead && ok && x.lo < x.hi) umma_commit(&sm.o_full);
    }
  } else {
    const int hf = warp >> 2, q = warp & 3, key = q * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16) + hf * 32;
    const float scale2 = a.scale * kLog2e;
    const int head = hf * 32 + lane;                 // of the reference that this lane keeps
    const float sink2 = a.sink[head] * kLog2e;
    const int d0 = q * 32 + (lane & ~1);             // first of the pair of dims (within a block of 128) that this lane stores
    int n = 0, done = 0;
    // False after a wait that ran out.  The warps of a half still meet at every tile's barrier, which a warp that left would keep the
    // others at for good; they wait for nothing more and store nothing.
    bool ok = true;
    for (int id = blockIdx.x; id < items; id += gridDim.x) {
      const Item x = item_of(a, id);
      const size_t part = (size_t)id * HL;           // [t][split][head]
      if (x.lo >= x.hi) {
        if (a.nsplit > 1) {
          if (q == 0) reinterpret_cast<float2*>(a.part_ml)[part + head] = make_float2(-1e30f, 0.f);
        } else {
          for (int i = threadIdx.x; i < HL * D / 8; i += 256)
            reinterpret_cast<uint4*>(a.o + (size_t)x.t * HL * D)[i] = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
      float ref = x.split == 0 ? sink2 : -1e30f;
      for (int base = x.lo; base < x.hi; base += KT, ++n) {
        ok = ok && mbar_wait<16>(&sm.s_full, n & 1, abort_flag, 54) && mbar_wait(&sm.full[0], n & 1, abort_flag, 55);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        uint32_t r[32];
        float s[32];
        tmem_ld_32x32(lanes + kColS, r);
        tmem_ld_wait();
        const bool valid = sm.rows[n & 1][key] != nullptr;
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = valid ? __uint_as_float(r[j]) * scale2 : -INFINITY;
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float w = redux_max(s[j]);
          if (lane == j) mx = w;
        }
        sm.wmax[warp][lane] = mx;
        if (hf)
          asm volatile("bar.sync 2, 128;" ::: "memory");
        else
          asm volatile("bar.sync 1, 128;" ::: "memory");
        if (!ok) continue;
        mx = fmaxf(fmaxf(sm.wmax[hf * 4][lane], sm.wmax[hf * 4 + 1][lane]), fmaxf(sm.wmax[hf * 4 + 2][lane], sm.wmax[hf * 4 + 3][lane]));
        const bool first = base == x.lo, grow = first ? mx > ref : mx > ref + 8.f;
        const float now = grow ? mx : ref;
        sm.ref[warp][lane] = now;
        sm.mul[warp][lane] = ex2(ref - now);
        ref = now;
        __syncwarp();
        if (!first && __any_sync(0xffffffffu, grow)) {
          // columns of O and l to the new references
#pragma unroll 1
          for (int b = 0; b < 5; ++b) {
            const uint32_t col = lanes + (b < 4 ? kColO + b * HL : kColL);
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
              uint32_t v[16];
              tmem_ld_32x16(col + c, v);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * sm.mul[warp][c + j]);
              tmem_st_32x16(col + c, v);
            }
          }
          tmem_st_wait();
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 m = *reinterpret_cast<const float2*>(&sm.ref[warp][8 * c + 2 * j]);
            const __nv_bfloat162 p = __floats2bfloat162_rn(ex2(s[8 * c + 2 * j] - m.x), ex2(s[8 * c + 2 * j + 1] - m.y));
            w[j] = *reinterpret_cast<const uint32_t*>(&p);
          }
          *reinterpret_cast<uint4*>(sm.p + key * 128 + (((hf * 4 + c) ^ (key & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.p_full);
      }
      ok = __all_sync(0xffffffffu, ok && mbar_wait<16>(&sm.o_full, done & 1, abort_flag, 56));
      ++done;
      if (!ok) continue;
      tc_fence_after();
      float l[32];
      {
        uint32_t r[32];
        tmem_ld_32x32(lanes + kColL, r);
        tmem_ld_wait();
        __syncwarp();
        sm.mul[warp][lane] = x.split == 0 ? ex2(sink2 - ref) : 0.f;      // the sink adds to the sum only
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = __uint_as_float(r[j]) + sm.mul[warp][j];
      }
      if (a.nsplit > 1) {
        float mine = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (lane == j) mine = l[j];
        if (q == 0) reinterpret_cast<float2*>(a.part_ml)[part + head] = make_float2(ref, mine);
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
          uint32_t r[32];
          tmem_ld_32x32(lanes + kColO + b * HL, r);
          tmem_ld_wait();
          float* dst = a.part_acc + (part + hf * 32) * D + b * 128 + key;
#pragma unroll
          for (int j = 0; j < 32; ++j) dst[(size_t)j * D] = __uint_as_float(r[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = 1.f / l[j];
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
          uint32_t r[32];
          tmem_ld_32x32(lanes + kColO + b * HL, r);
          tmem_ld_wait();
          const int d = b * 128 + d0;
          const bool turn = a.out_rope && d >= D - a.rp.rotary_dim;
          float cs = 1.f, sn = 0.f;
          if (turn) rope_cos_sin(a.rp, (float)x.pos, (d - (D - a.rp.rotary_dim)) >> 1, 1, cs, sn);
          // neighbouring lanes trade dims for heads: even lanes store the pair of head j, odd ones that of head j + 1
          __nv_bfloat16* dst = a.o + ((size_t)x.t * HL + hf * 32 + (lane & 1)) * D + d;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float v0 = __uint_as_float(r[j]) * l[j], v1 = __uint_as_float(r[j + 1]) * l[j + 1];
            const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? v0 : v1, 1);
            __nv_bfloat162 v = lane & 1 ? __floats2bfloat162_rn(got, v1) : __floats2bfloat162_rn(v0, got);
            if (turn) {
              const float2 f = __bfloat1622float2(v);
              v = __floats2bfloat162_rn(f.x * cs - f.y * sn, f.x * sn + f.y * cs);
            }
            *reinterpret_cast<__nv_bfloat162*>(dst + (size_t)j * D) = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    if (*abort_flag) drain_after_abort(&sm.drain, elect_one());
    tmem_dealloc(tmem, 512);
  }
}

// out[t][head] = sum_s acc_s 2^(ref_s - M) / sum_s l_s 2^(ref_s - M); one warp per head, 16 dims a lane.
__global__ void __launch_bounds__(128) sparse_attn_merge_kernel(const AttnArgs a) {
  pdl_entry();
  const int t = blockIdx.x, head = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const float2* ml = reinterpret_cast<const float2*>(a.part_ml) + (size_t)t * a.nsplit * HL + head;
  float top = -1e30f, sum = 0.f;
  const float2 mine = lane < a.nsplit ? ml[(size_t)lane * HL] : make_float2(-1e30f, 0.f);
  top = warp_max(mine.y > 0.f ? mine.x : -1e30f);
  const float f = mine.y > 0.f ? ex2(mine.x - top) : 0.f;
  sum = warp_sum(mine.y * f);
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  for (int s = 0; s < a.nsplit; ++s) {
    const float w = __shfl_sync(0xffffffffu, f, s);
    if (w == 0.f) continue;
    const float4* src = reinterpret_cast<const float4*>(a.part_acc + (((size_t)t * a.nsplit + s) * HL + head) * D) + lane;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 v = src[32 * c];
      acc[4 * c] = fmaf(v.x, w, acc[4 * c]), acc[4 * c + 1] = fmaf(v.y, w, acc[4 * c + 1]);
      acc[4 * c + 2] = fmaf(v.z, w, acc[4 * c + 2]), acc[4 * c + 3] = fmaf(v.w, w, acc[4 * c + 3]);
    }
  }
  const float inv = sum > 0.f ? 1.f / sum : 0.f;
  __nv_bfloat16* o = a.o + ((size_t)t * HL + head) * D;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int d = 128 * c + 4 * lane;
    __nv_bfloat162 v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      v[i] = __floats2bfloat162_rn(acc[4 * c + 2 * i] * inv, acc[4 * c + 2 * i + 1] * inv);
      const int dp = d + 2 * i;
      if (a.out_rope && dp >= D - a.rp.rotary_dim) {
        float cs, sn;
        rope_cos_sin(a.rp, (float)a.pos[t], (dp - (D - a.rp.rotary_dim)) >> 1, 1, cs, sn);
        const float2 x = __bfloat1622float2(v[i]);
        v[i] = __floats2bfloat162_rn(x.x * cs - x.y * sn, x.x * sn + x.y * cs);
      }
    }
    *reinterpret_cast<uint2*>(o + d) = make_uint2(*reinterpret_cast<uint32_t*>(&v[0]), *reinterpret_cast<uint32_t*>(&v[1]));
  }
}

}  // namespace

int launch_attn_mma(const AttnArgs& a, int t, cudaStream_t st) {
  if (a.nsplit > 32) return 304;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(sparse_attn_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess)
      return 306;
    set = true;
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 307;
  const int items = t * a.nsplit;
  dsv4_launch(sparse_attn_mma_kernel, items < sms ? items : sms, kThreads, kSmemBytes, st, a, items);
  if (a.nsplit > 1) dsv4_launch(sparse_attn_merge_kernel, dim3(t, HL / 4), 128, 0, st, a);
  return (int)cudaGetLastError();
}
