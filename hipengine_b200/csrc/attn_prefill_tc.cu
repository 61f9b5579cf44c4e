// Causal paged GQA prefill attention for heads of 256 columns on the 5th-generation tensor cores (the arguments and the
// fused sigmoid gate of attn_prefill.cu, without window, soft cap, sink and head gate).
//
//   warps 0-3 : softmax; a thread owns one of the tile's 128 query rows (= a TMEM lane)
//   warp 4, 5 : TMA producers of keys / values: a tile is 64 keys = 4 pages x 4 boxes of 16 keys x 64 columns, one box a lane
//   warp 6    : MMA issuer; owns the tensor memory
// Tensor memory: two score buffers of 64 columns and the 256-column accumulator; the weights overwrite the scores they came from
// and are the A operand of the value product.  Queries and keys are K-major operands as they lie in memory; values
// are too -- [key][column] rows are the MN-major form of the B operand, so the cache is read in place by both products.
// While the softmax of a tile runs, the scores of the next tile and the value product of the last one occupy the tensor
// cores.  The accumulator is rescaled only when a row's maximum has grown by more than 2^8: sums and weights use the same
// reference, but the largest weight is then not 1 and a bf16 weight would be off by its rounding, which it is not in the register
// form.  So a weight is two bf16 numbers, its upper 16 bits and the rest (64 columns of 64 keys: the buffer that the scores had), and
// the value product takes both.  Error against 64 bits at 600 rows after 2000, queries of twice unit size: 1.66e-3, the rounding of
// the output; 2.19e-3 with one number, 1.89e-3 in the register form.  It costs 14-24 % (4096 rows 406 -> 462 us, after 12288 tokens
// 1516 -> 1878 us); rescaling at every growth instead, with one number, 493 / 1924 us.
//
// What bounds it: a tile of 64 keys costs 1536 tensor-core cycles, about 1750 cycles of operand reads from shared memory by count
// (the 64 KB of queries are read again for every tile, 64-wide score products cannot do better) and 64 KB from L2; with one
// bf16 number a weight 1024 and 1500.  The register form (mma.sync, 64 query rows) is bound by the rate of mma.sync and re-reads keys
// and values twice as often: 24 heads on 4, 4096 rows 1159 us there, 462 us here (447 TFLOP/s); after 12288 tokens 6694 / 1878 us (769
// TFLOP/s); 777 rows 107 / 91 us; 16 heads on 2, 2048 rows 287 / 147 us.  Counters at 4096 rows after 4096 tokens: tensor pipe 62 %,
// L2 5.5 TB/s, issue 27 %, DRAM 2 %.
#include "common.cuh"
#include "sm100.cuh"
#include "tmap.cuh"

using namespace he;
using namespace sm100;

namespace {

constexpr int QM = 128, KN = 64, D = 256, PAGE_KEYS = 16, NGRP = D / 64, KS = 3, VS = 2, NTHR = 224;
constexpr int Q_SUB = QM * 128, KV_SUB = KN * 128, KV_STAGE = NGRP * KV_SUB;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LAZY = 8.f;                  // log2 growth of a maximum that is tolerated without rescaling

struct FlashTcArgs {
  const __nv_bfloat16* gate;   // [T][H][D] or null
  const int* block_table;      // row of the segment's slot
  __nv_bfloat16* out;          // [T][H * D]
  int* status;
  int T, H, Hkv, pos0;
  float scale_log2;
};

struct __align__(8) Bars {
  uint64_t q_full, k_full[KS], k_empty[KS], v_full[VS], v_empty[VS];
  uint64_t s_full[2], p_full[2];     // per buffer: a softmax may be one tile ahead of the issuer
  uint64_t o_done, drain;
  uint32_t tmem_base;
  int abort_flag;
};

constexpr size_t SMEM_TC = (size_t)NGRP * Q_SUB + (KS + VS) * (size_t)KV_STAGE + sizeof(Bars) + 1024;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// The upper half of a float: a bf16 number; what it leaves fits another one to 2^-9 of itself.
__device__ __forceinline__ float upper(float x) { return __uint_as_float(__float_as_uint(x) & 0xFFFF0000u); }
// Bounded wait that goes on after an abort.
__device__ __forceinline__ void drain_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return;
    if (i > 64) __nanosleep(32);
  }
}
// MN-major operand (rows of 64 columns = 128 bytes, 128-byte swizzle, 8-row groups 1 KB apart): the leading offset is the
// distance between groups of 64 columns, the stride offset the one between groups of 8 rows along K.
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(KV_SUB >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// grid (query tiles, H)
__global__ void __launch_bounds__(NTHR, 1)
flash_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                        const __grid_constant__ FlashTcArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                                   // [4 groups][128 rows][128 bytes]
  uint8_t* sK = sQ + NGRP * Q_SUB;                      // [KS][4 groups][64 keys][128 bytes]
  uint8_t* sV = sK + KS * KV_STAGE;                     // [VS][4 groups][64 keys][128 bytes]
  Bars* bar = reinterpret_cast<Bars*>(sV + VS * KV_STAGE);
  volatile int* abort_flag = &bar->abort_flag;

  const int tile = (int)gridDim.x - 1 - (int)blockIdx.x;          // heavy (late) tiles first
  const int h = blockIdx.y, hk = h / (a.H / a.Hkv);
  const int t0 = tile * QM, rows = min(QM, a.T - t0);
  const int kv_end = a.pos0 + t0 + rows, n_tiles = (kv_end + KN - 1) / KN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&bar->q_full, 1);
    for (int s = 0; s < KS; ++s) {
      mbar_init(&bar->k_full[s], 1);
      mbar_init(&bar->k_empty[s], 1);
    }
    for (int s = 0; s < VS; ++s) {
      mbar_init(&bar->v_full[s], 1);
      mbar_init(&bar->v_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bar->s_full[b], 1);
      mbar_init(&bar->p_full[b], 4);
    }
    mbar_init(&bar->o_done, 1);
    mbar_init(&bar->drain, 1);
    bar->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 6) {
    tmem_alloc(&bar->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = bar->tmem_base, o_col = tm + 256;
  const auto s_col = [&](int b) { return tm + (uint32_t)(b * KN); };

  if (warp == 4 || warp == 5) {
    const bool keys = warp == 4;
    const int depth = keys ? KS : VS;
    uint64_t *full = keys ? bar->k_full : bar->v_full, *empty = keys ? bar->k_empty : bar->v_empty;
    uint8_t* ring = keys ? sK : sV;
    if (keys && lane == 0) {
      mbar_expect_tx(&bar->q_full, NGRP * Q_SUB);
      for (int k = 0; k < NGRP; ++k) tma_load_2d(sQ + k * Q_SUB, &tmQ, &bar->q_full, h * D + k * 64, t0);
    }
    __syncwarp();
    // lane = (page of the tile, group of 64 columns); pages past the last visible one repeat it (masked, see below)
    const int pg = (lane >> 2) & 3, grp = lane & 3, last_page = (kv_end - 1) / PAGE_KEYS;
    int page = __ldg(a.block_table + min(pg, last_page));
    int s = 0, n = 0;
    uint32_t ph = 0;
    for (int j = 0; j < n_tiles; ++j) {
      const int next = __ldg(a.block_table + min((j + 1) * 4 + pg, last_page));
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], ph ^ 1, abort_flag, a.status, keys ? 701 : 702));
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(&full[s], KV_STAGE);
      __syncwarp();
      if (lane < 16)
        tma_load_2d(ring + s * KV_STAGE + grp * KV_SUB + pg * (PAGE_KEYS * 128), &tmKV, &full[s], grp * 64,
                    ((page * 2 + (keys ? 0 : 1)) * a.Hkv + hk) * PAGE_KEYS);
      page = next;
      ++n;
      if (++s == depth) { s = 0; ph ^= 1u; }
    }
    // no copy may still be in flight when the CTA leaves (matters only after an abort)
    if (lane == 0) {
      if (keys) drain_wait(&bar->q_full, 0);
      for (int i = 0; i < depth; ++i)
        if (i < n) drain_wait(&full[i], ((n - 1 - i) / depth) & 1);
    }
  } else if (warp == 6) {
    if (elect_one()) {
      constexpr uint32_t id_s = umma_idesc_bf16(QM, KN), id_o = umma_idesc_bf16(QM, D) | (1u << 16);   // B is MN-major
      bool ok = mbar_wait(&bar->q_full, 0, abort_flag, a.status, 703);
      const auto scores = [&](int j) {
        const int s = j % KS, b = j & 1;
        if (!mbar_wait(&bar->k_full[s], (j / KS) & 1, abort_flag, a.status, 704)) return false;
        // the buffer still holds the weights of two tiles ago until their value product is done
        if (j >= 2 && !mbar_wait(&bar->o_done, j & 1, abort_flag, a.status, 705)) return false;
        tc_fence_after();
        const uint32_t qa = smem_u32(sQ), ka = smem_u32(sK + s * KV_STAGE);
#pragma unroll
        for (int k = 0; k < NGRP; ++k)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            umma_f16(s_col(b), umma_desc_k_sw128(qa + k * Q_SUB + u * 32), umma_desc_k_sw128(ka + k * KV_SUB + u * 32), id_s,
                     (k > 0 || u > 0) ? 1u : 0u);
        umma_commit(&bar->s_full[b]);
        umma_commit(&bar->k_empty[s]);
        return true;
      };
      ok = ok && scores(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles && !scores(j + 1)) break;
        const int s = j % VS, b = j & 1;
        if (!mbar_wait(&bar->p_full[b], (j >> 1) & 1, abort_flag, a.status, 706)) break;
        if (!mbar_wait(&bar->v_full[s], (j / VS) & 1, abort_flag, a.status, 707)) break;
        tc_fence_after();
        const uint32_t va = smem_u32(sV + s * KV_STAGE);
#pragma unroll
        for (int u = 0; u < KN / 16; ++u) {
          const uint64_t vd = desc_mn_sw128(va + u * 2048);
          umma_f16_ts(o_col, s_col(b) + u * 8, vd, id_o, (j > 0 || u > 0) ? 1u : 0u);
          umma_f16_ts(o_col, s_col(b) + KN / 2 + u * 8, vd, id_o, 1u);        // the weights' low parts
        }
        umma_commit(&bar->o_done);
        umma_commit(&bar->v_empty[s]);
      }
      umma_commit(&bar->drain);
      drain_wait(&bar->drain, 0);
    }
  } else {
    // ------------------------------------------------------------ softmax, one row per thread
    const int row = warp * 32 + lane;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    const int q_first = a.pos0 + t0 + warp * 32, q_pos = q_first + lane;
    const float sc = a.scale_log2;
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    int j = 0;
    for (; j < n_tiles; ++j) {
      const int b = j & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->s_full[b], (j >> 1) & 1, abort_flag, a.status, 708));
      if (!ok) break;
      tc_fence_after();
      uint32_t r0[32], r1[32];
      tmem_ld_32x32(s_col(b) + lane_off, r0);
      tmem_ld_32x32(s_col(b) + lane_off + 32, r1);
      tmem_ld_wait();
      const int k0 = j * KN;
      if (k0 + KN - 1 > q_first) {
        const int hi = q_pos - k0;
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (c > hi) r0[c] = 0xff800000u;
          if (c + 32 > hi) r1[c] = 0xff800000u;
        }
      }
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 32; ++c) mx = fmaxf(mx, fmaxf(__uint_as_float(r0[c]), __uint_as_float(r1[c])));
      mx *= sc;                                        // the scale is positive (checked by the launcher)
      const bool grow = mx > m_ref + LAZY;
      if (__any_sync(0xffffffffu, grow)) {
        const float m_new = grow ? mx : m_ref, f = m_ref == -INFINITY ? 0.f : ex2(m_ref - m_new);
        m_ref = m_new;
        l *= f;
        if (j > 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(&bar->o_done, (j - 1) & 1, abort_flag, a.status, 709));
          if (!ok) break;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t o[32];
            tmem_ld_32x32(o_col + lane_off + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
            tmem_st_32x32(o_col + lane_off + c, o);
          }
        }
      }
      const float neg = m_ref == -INFINITY ? 0.f : -m_ref;     // nothing seen yet: every weight is 2^-inf = 0
      float s0 = 0.f, s1 = 0.f;
      uint32_t hi[32], lo[32];                                 // 32 columns each: weights of 64 keys, two to a column
#pragma unroll
      for (int c = 0; c < 32; c += 2) {
        const float p0 = ex2(fmaf(__uint_as_float(r0[c]), sc, neg)), p1 = ex2(fmaf(__uint_as_float(r0[c + 1]), sc, neg));
        const float p2 = ex2(fmaf(__uint_as_float(r1[c]), sc, neg)), p3 = ex2(fmaf(__uint_as_float(r1[c + 1]), sc, neg));
        s0 += p0 + p1;
        s1 += p2 + p3;
        hi[c >> 1] = __byte_perm(__float_as_uint(p0), __float_as_uint(p1), 0x7632);
        hi[16 + (c >> 1)] = __byte_perm(__float_as_uint(p2), __float_as_uint(p3), 0x7632);
        lo[c >> 1] = pack2(p0 - upper(p0), p1 - upper(p1));
        lo[16 + (c >> 1)] = pack2(p2 - upper(p2), p3 - upper(p3));
      }
      l += s0 + s1;
      tmem_st_32x32(s_col(b) + lane_off, hi);
      tmem_st_32x32(s_col(b) + lane_off + KN / 2, lo);
      tmem_st_wait();
      if (k0 + KN > kv_end) {
        // keys past the last visible one: their weights are zero, their values may be anything (also NaN): zero them
        const int s = j % VS, bad = k0 + KN - kv_end;
        ok = __all_sync(0xffffffffu, mbar_wait(&bar->v_full[s], (j / VS) & 1, abort_flag, a.status, 710));
        if (!ok) break;
        for (int i = threadIdx.x; i < bad * NGRP * 8; i += 128) {
          const int r = KN - bad + i / (NGRP * 8), c = i % (NGRP * 8);
          *reinterpret_cast<uint4*>(sV + s * KV_STAGE + (c >> 3) * KV_SUB + r * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async_smem();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->p_full[b]);
    }
    if (ok) {
      // the last two value products may both be outstanding: wait for them in turn, a parity tells only neighbours apart
      if (j > 1) ok = __all_sync(0xffffffffu, mbar_wait(&bar->o_done, j & 1, abort_flag, a.status, 711));
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&bar->o_done, (j - 1) & 1, abort_flag, a.status, 712));
      if (ok) {
        tc_fence_after();
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const bool live = row < rows;
        const size_t at = (size_t)(t0 + (live ? row : 0)) * a.H * D + (size_t)h * D;
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32(o_col + lane_off + c, o);
          tmem_ld_wait();
          if (live) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 pk, gt = make_uint4(0u, 0u, 0u, 0u);
              if (a.gate != nullptr) gt = __ldg(reinterpret_cast<const uint4*>(a.gate + at + c + v * 8));
              uint32_t *pw = reinterpret_cast<uint32_t*>(&pk), *gw = reinterpret_cast<uint32_t*>(&gt);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float x = __uint_as_float(o[v * 8 + 2 * e]) * inv, y = __uint_as_float(o[v * 8 + 2 * e + 1]) * inv;
                if (a.gate != nullptr) {     // the output is rounded to bf16 before the gate (cpu_reference/ops.py:2250)
                  const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[e]));
                  x = bf16_to_f32(f32_to_bf16(x)) * sigmoid_f(gf.x);
                  y = bf16_to_f32(f32_to_bf16(y)) * sigmoid_f(gf.y);
                }
                pw[e] = pack2(x, y);
              }
              *reinterpret_cast<uint4*>(a.out + at + c + v * 8) = pk;
            }
          }
        }
        tc_fence_before();
      }
    }
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 6) tmem_dealloc(tm, 512);
}

}  // namespace

// One segment, as he_flash_prefill, for D = 256, pages of 16 keys, no window.  `n_pages`: pages of the cache.
HE_API int he_flash_prefill_tc(const void* q, const void* gate, const void* kv_cache, long long n_pages,
                               const void* block_table_row, void* out, int T, int H, int Hkv, int pos0, float scale,
                               void* status, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (Hkv <= 0 || H % Hkv != 0 || n_pages <= 0 || pos0 < 0 || !(scale > 0.f) ||
      (reinterpret_cast<uintptr_t>(out) & 15) != 0 || (reinterpret_cast<uintptr_t>(gate) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  CUtensorMap mq, mkv;
  int rc = make_map(&mq, q, T, (long long)H * D, (long long)H * D, QM);
  if (rc == 0) rc = make_map(&mkv, kv_cache, n_pages * 2 * Hkv * PAGE_KEYS, D, D, PAGE_KEYS);
  if (rc != 0) return rc;
  FlashTcArgs a = {};
  a.gate = (const __nv_bfloat16*)gate;
  a.block_table = (const int*)block_table_row;
  a.out = (__nv_bfloat16*)out;
  a.status = (int*)status;
  a.T = T; a.H = H; a.Hkv = Hkv; a.pos0 = pos0;
  a.scale_log2 = scale * LOG2E;
  // set per call (cheap): the attribute belongs to the (function, device) pair, not to the process
  const cudaError_t e = cudaFuncSetAttribute(flash_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_TC);
  if (e != cudaSuccess) return (int)e;
  flash_prefill_tc_kernel<<<dim3((T + QM - 1) / QM, H), NTHR, SMEM_TC, stream>>>(mq, mkv, a);
  HE_LAUNCH_CHECK();
  return 0;
}
