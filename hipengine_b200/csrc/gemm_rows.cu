// Products of a few activation rows (1..64) with QUANTISED weights (Q4_K / Q6_K / Q8_0 in their device layouts):
// out[r][n] = sum_k x[r][k] W[n][k], the weights streamed once whatever the row count.  Decode steps, verify chains and
// short prompts are these products and little else.  This file: the rows' image for all of them, and the products of up to 24
// rows on mma.sync; more rows run on tcgen05 (gemm_rows_tc.cu; ops/rows.py has the line).
//
// What has to move is the weight stream (HBM).  What bounds it in fact (17408 x 5120 Q4_K, 4 / 16 rows: 18.4 / 22.2 us): ramp,
// image wait and the sum of shared tiles around a steady part that the expansion of blocks sets (DRAM 25 / 22 %, issue 44 / 43 %,
// tensor pipe 14 / 23 %).
//   operands : fp16 m16n8k16 MMAs with the WEIGHT as the A operand.  A k-quant weight is d * (sc * q) - dmin * m with
//              sc * q an integer below 2^10 and m one below 2^6: both are exact in fp16, so ONE packed fp16 FMA makes two
//              operands (1024 + q is the nibble under an exponent byte; (1024 + q) * sc - 1024 * sc), the 256-column block
//              accumulates in fp32, and d / dmin come in once per block.  The minima are one more MMA against the sums of
//              the activations per 32 columns (as an fp16 high and low part).  Q8_0, and Q6_K up to 8 rows: the integers
//              themselves are the operands, an MMA (two for Q8_0) covers one sub-block, and the sub-block's scale meets
//              its fp32 sums: exact as well, and for Q8_0 cheaper than a product per operand (17408 x 5120, 4 / 16 / 32 rows
//              24.7 / 29.2 / 48.1 -> 21.4 / 24.0 / 42.5 us).  Q6_K above 8 rows: sc * (q - 32), 13 bits, rounded to 11: the exact
//              form costs two packed FMAs per MMA (17408 x 5120, 16 rows 27.5 us against 25.0; at 8 rows 22.1 against 22.8).
//   activations: fp16 under a power of two per row and block of 256 columns, 11 bits each down to 2^-14 of the block's largest
//              value and 2^-25 of it below (bf16 values down to 2^-17 of it exactly), written once per launch by he_rows_image
//              in the order of the MMA's B fragments (one 16-byte load per lane feeds two MMAs), so no CTA repeats the
//              normalisation.
//   k order  : lane (g, t) of an MMA with scaled operands holds columns of ITS OWN sub-blocks -- t = (h, u) owns, in half h of
//              the block, the 16 positions of half u of each of the four 32-column groups -- because that is what a 16-byte load
//              of Q6_K low nibbles, high nibbles and Q4_K nibbles delivers; the scale is then a per-lane constant.
//   split    : the (tile of 128 weight rows) x (block) units of all segments are dealt out as one contiguous range
//              per SM (equal to one unit), so there is no last wave.  A tile that several CTAs share leaves fp32 partial
//              tiles in `ws`; whoever arrives last (a counter per tile, reset by it) adds them in CTA order:
//              bit-reproducible for a given number of rows.  (A row's last bits depend on that number: up to 16 rows sum a
//              block in two chains, more in one, on tcgen05 in the order of its sums.)  The host divides: with the CTAs' ranges
//              from eight 64-bit divisions a thread and old residual values loaded one by one 4 / 16 rows took 20.0 / 23.1 us.
//   roles    : one producer warp (TMA boxes of weight rows x 1 block, bulk copies of the image), one warp that signals shared
//              tiles, 16 MMA warps.  The ring holds ~200 KB: with programmatic dependent launch the
//              next product's weights arrive while the previous kernels drain.
//
// Counterparts in the reference: hipengine/kernels/hip_gfx1100/quant/gguf_q4_k_gemv.hip and the packed-row forms in
// quant/gguf_q4_k_prefill.hip.
#include "rows_mma.cuh"

using namespace he;
using namespace herows;

namespace {

struct RowsShared {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  int abort_flag;
  int last[2];                // was this CTA the last to arrive at its first / last shared tile
};

constexpr int TILE = 128, HALF = 64;                  // weight rows of a tile; of a TMA box, of each weight of a pair

// MMA warps: two groups of eight side by side, 16 weight rows each, that take every other block (their sums meet in shared memory
// at the end of a tile).
constexpr int MMA_WARPS = 16, THREADS = MMA_WARPS * 32 + 64;       // + producer warp + signal warp
template <int NT>
struct Shape {
  static constexpr int XBUF = TILE * 8 * NT * 4;                   // exchange of the second group's sums
};

template <int NT>
__global__ void __launch_bounds__(THREADS, 1)
rows_gemm_kernel(const __grid_constant__ RowsMaps maps, const __grid_constant__ HeRowsArgs a, const RowsPlan plan) {
  using S = Shape<NT>;
  constexpr int IMG = IMG_COL * 8 * NT, SLOT = TILE * 8 * NT;      // image bytes of a block, floats of a partial tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* xbuf = reinterpret_cast<float*>(smem + (size_t)a.stages * a.stage_bytes);
  RowsShared* sh = reinterpret_cast<RowsShared*>(smem + (size_t)a.stages * a.stage_bytes + S::XBUF);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = a.K >> 8, b = blockIdx.x, u0 = plan.begin(b), u1 = plan.begin(b + 1);
  // CTAs that share a tile: those that hold its first and last unit and all between
  const auto first_cta = [&](int tile) { return plan.cta_of(tile * nb); };
  const auto last_cta = [&](int tile) { return plan.cta_of((tile + 1) * nb - 1); };
  const int tile_a = u0 / nb, tile_z = (u1 - 1) / nb;           // only the first and the last tile can be shared
  const bool share_a = u0 > tile_a * nb || u1 < (tile_a + 1) * nb, share_z = tile_z != tile_a && u1 < (tile_z + 1) * nb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      sm100::mbar_init(&sh->full[s], 1);
      sm100::mbar_init(&sh->empty[s], 8);
    }
    sh->abort_flag = 0;
    sm100::mbar_fence_init();
  }
  __syncthreads();
  pdl_launch();
  volatile int* abort_flag = &sh->abort_flag;

  if (warp >= MMA_WARPS) {
    if (warp == MMA_WARPS) {
      // ------------------------------------------------------------ producer
      if (sm100::elect_one()) {
        const uint8_t* image = reinterpret_cast<const uint8_t*>(a.image);
        int si = 0, tile = u0 / nb, blk = u0 % nb;
        auto weights = [&](int s) {
          while (si + 1 < a.n_seg && tile >= a.seg[si + 1].tile0) ++si;
          const HeRowsSeg& sg = a.seg[si];
          uint8_t* dst = smem + (size_t)s * a.stage_bytes;
          const int bb = rows_block_bytes(sg.qtype);
          sm100::mbar_expect_tx(&sh->full[s], (uint32_t)(TILE * bb + IMG));
          const bool pair = sg.epi >= 3;
          const int n0 = (tile - sg.tile0) * (pair ? HALF : TILE);
#pragma unroll 1
          for (int r = 0; r < 2; ++r) {
            const CUtensorMap* m = &maps.m[si][pair && r ? 2 : 0];
            const int row = pair ? n0 : n0 + r * HALF;
            uint8_t* d = dst + r * HALF * bb;
            if (sg.qtype == HE_Q8_0) {
              sm100::tma_load_2d(d, m, &sh->full[s], blk * 256, row);
              sm100::tma_load_2d(d + HALF * 128, m, &sh->full[s], blk * 256 + 128, row);
              sm100::tma_load_2d(d + 2 * HALF * 128, m + 1, &sh->full[s], a.K + 16 * blk, row);
            } else {
              sm100::tma_load_2d(d, m, &sh->full[s], blk * bb, row);
            }
          }
          if (++blk == nb) { blk = 0; ++tile; }
        };
        const int n = u1 - u0, pre = min(n, a.stages);
        for (int i = 0; i < pre; ++i) weights(i);
        pdl_wait();                       // the rows (and so their image) come from the kernels before
        for (int i = 0; i < pre; ++i)
          bulk_load(sm100::smem_u32(smem + (size_t)i * a.stage_bytes + a.w_bytes), image + (size_t)((u0 + i) % nb) * IMG,
                    IMG, &sh->full[i]);
        int s = 0;
        uint32_t ph = 0;
        int issued = pre;
        for (int i = pre; i < n; ++i) {
          if (!wait_long(&sh->empty[s], ph, abort_flag, a.status, 401)) break;
          const int bi = blk;
          weights(s);
          bulk_load(sm100::smem_u32(smem + (size_t)s * a.stage_bytes + a.w_bytes), image + (size_t)bi * IMG, IMG,
                    &sh->full[s]);
          ++issued;
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
        if (issued < n) {                 // gave up: let the copies in flight land before the CTA leaves
          for (int i = max(0, issued - a.stages); i < issued; ++i)
            for (int p = 0; p < (1 << 16) && !sm100::mbar_test_wait(&sh->full[i % a.stages], (i / a.stages) & 1); ++p)
              __nanosleep(64);
        }
      }
    } else {
      // ------------------------------------------------------------ arrivals at shared tiles
      // A fence and an atomic take a round trip to L2 each; this warp makes it while the MMA warps go on.
      pdl_wait();
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        if (!(i == 0 ? share_a : share_z)) continue;
        const int tile = i == 0 ? tile_a : tile_z;
        // the partial tile is written (one barrier each: the MMA warps may be at the second before this warp is at the first)
        if (i == 0) named_sync(1, 256 + 32);
        else named_sync(2, 256 + 32);
        if (lane == 0) {
          __threadfence();
          const int n = last_cta(tile) - first_cta(tile);
          const bool last = atomicAdd(a.counters + tile, 1) == n;
          if (last) a.counters[tile] = 0;
          __threadfence();
          sh->last[i] = last;
        }
        __syncwarp();
      }
      if (share_a || share_z) named_arrive(3, 256 + 32);
    }
    return;
  }

  // -------------------------------------------------------------- MMA warps
  const uint32_t mg = opaque(MAGIC);
  const int grp = warp >> 3, w = warp & 7, g = lane >> 2, t = lane & 3;
  pdl_wait();
  // this group's stages: the slots of its parity
  const uint32_t ring = sm100::smem_u32(smem), step = (uint32_t)(2 * a.stage_bytes);
  const uint32_t first = ring + (uint32_t)(grp * a.stage_bytes), end = ring + (uint32_t)(a.stages * a.stage_bytes);
  const uint32_t w_bytes = (uint32_t)a.w_bytes;
  uint32_t st = first, ph = 0;
  uint64_t *full = sh->full + grp, *empty = sh->empty + grp;

  auto epilogue = [&](const HeRowsSeg& sg, int tile, const float (&acc)[NT][4]) {
    const int tl = tile - sg.tile0;
    if (sg.epi >= 3) {
      const int row = tl * HALF + 8 * w + g;
      if (row >= sg.n_rows) return;
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(sg.out) + row;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int r = 8 * n + 2 * t + j;
          const float ga = sg.epi == 3 ? silu_f(acc[n][j]) : gelu_tanh_f(acc[n][j]);
          if (r < a.R) o[(size_t)r * sg.out_stride] = f32_to_bf16(ga * acc[n][2 + j]);
        }
      return;
    }
    // a residual's old values first, all of them: they could lie where the stores go, for the compiler
    float old[NT][4];
    if (sg.epi == 2) {
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = tl * TILE + 16 * w + g + 8 * (i >> 1), r = 8 * n + 2 * t + (i & 1);
          old[n][i] = row < sg.n_rows && r < a.R ? reinterpret_cast<const float*>(sg.out)[(size_t)r * sg.out_stride + row] : 0.f;
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int row = tl * TILE + 16 * w + g + 8 * k;
      if (row >= sg.n_rows) continue;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int r = 8 * n + 2 * t + j;
          if (r >= a.R) continue;
          const size_t off = (size_t)r * sg.out_stride + row;
          const float v = acc[n][2 * k + j];
          if (sg.epi == 1) reinterpret_cast<__nv_bfloat16*>(sg.out)[off] = f32_to_bf16(v);
          else reinterpret_cast<float*>(sg.out)[off] = sg.epi == 2 ? old[n][2 * k + j] + v : v;
        }
    }
  };
  const auto segment = [&](int tile) {
    int si = 0;
    while (si + 1 < a.n_seg && tile >= a.seg[si + 1].tile0) ++si;
    return si;
  };

  int u = u0;
  bool wrote = false;
  while (u < u1) {
    const int tile = u / nb, blk0 = u - tile * nb, n_blk = min(nb - blk0, u1 - u);
    const HeRowsSeg& sg = a.seg[segment(tile)];
    const bool pair = sg.epi >= 3;
    const int qtype = sg.qtype, bb = rows_block_bytes(qtype);
    // rows g and g + 8 of this warp's MMA: (region, row in region); a tile of a pair holds HALF gate rows and HALF up rows,
    // row g is a gate row and row g + 8 its up row
    const int i0 = pair ? 8 * w + g : (w & 3) * 16 + g, i1 = pair ? i0 : i0 + 8;
    const uint32_t p0 = (pair ? 0 : w >> 2) * HALF * bb, p1 = (pair ? 1 : w >> 2) * HALF * bb;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    const int skip = (u - u0 + grp) & 1;    // the tile's first unit is the other group's
    auto blocks = [&](auto&& one) {
      for (int i = skip; i < n_blk; i += 2) {
        if (wait_long(full, ph, abort_flag, a.status, 402)) {
          one(st, st + w_bytes);
          __syncwarp();
          if (lane == 0) sm100::mbar_arrive(empty);
        }
        st += step;
        full += 2;
        empty += 2;
        if (st >= end) {
          st = first;
          full = sh->full + grp;
          empty = sh->empty + grp;
          ph ^= 1u;
        }
      }
    };
    if (qtype == HE_Q4_K) {
      const uint32_t o0 = p0 + i0 * 144, o1 = p1 + i1 * 144;
      blocks([&](uint32_t st0, uint32_t img) { block_q4k<NT, NT, NT <= 2>(st0 + o0, st0 + o1, img, lane, mg, acc); });
    } else if (qtype == HE_Q6_K) {
      const uint32_t o0 = p0 + i0 * 224, o1 = p1 + i1 * 224;
      blocks([&](uint32_t st0, uint32_t img) {
        if constexpr (NT == 1) block_q6k_exact<NT, NT>(st0 + o0, st0 + o1, img, lane, mg, acc);
        else block_q6k<NT, NT, NT <= 2>(st0 + o0, st0 + o1, img, lane, mg, acc);
      });
    } else {
      blocks([&](uint32_t st0, uint32_t img) { block_q80<NT, NT, HALF>(st0 + p0, i0, st0 + p1, i1, img, lane, mg, acc); });
    }
    u += n_blk;
    float4* xb = reinterpret_cast<float4*>(xbuf) + w * NT * 32 + lane;
    if (grp == 1) {
      if (wrote) named_sync(5, 512);          // group 0 has read the previous tile's sums
      wrote = true;
#pragma unroll
      for (int n = 0; n < NT; ++n) xb[n * 32] = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
      named_arrive(4, 512);
      continue;
    }
    named_sync(4, 512);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const float4 v = xb[n * 32];
      acc[n][0] += v.x; acc[n][1] += v.y; acc[n][2] += v.z; acc[n][3] += v.w;
    }
    named_arrive(5, 512);
    if ((tile == tile_a && share_a) || (tile == tile_z && share_z)) {
      // a partial tile: the CTA's own slot 1 if it holds the tile's first unit, else slot 0
      float* mine = a.ws + (size_t)(2 * b + (blk0 == 0 ? 1 : 0)) * SLOT + (w * NT * 32 + lane) * 4;
#pragma unroll
      for (int n = 0; n < NT; ++n)
        *reinterpret_cast<float4*>(mine + n * 128) = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
      if (tile == tile_a) named_arrive(1, 256 + 32);
      else named_arrive(2, 256 + 32);
      continue;
    }
    epilogue(sg, tile, acc);
  }
  if (grp == 1) {
    if (wrote) named_sync(5, 512);
    return;
  }
  if (!(share_a || share_z)) return;
  named_sync(3, 256 + 32);
#pragma unroll 1
  for (int i = 0; i < 2; ++i) {
    if (!(i == 0 ? share_a : share_z) || !sh->last[i]) continue;
    const int tile = i == 0 ? tile_a : tile_z, c0 = first_cta(tile), c1 = last_cta(tile);
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    constexpr int FLY = NT == 1 ? 8 : 4;         // partial tiles in flight (one after the other each took a trip to L2)
    for (int c = c0; c <= c1; c += FLY) {
      float4 v[FLY][NT];
#pragma unroll
      for (int e = 0; e < FLY; ++e) {
        // the first of them holds the tile's first unit (slot 1 of its CTA), the others' ranges start inside it (slot 0)
        const float* p = a.ws + (size_t)(2 * (c + e) + (c + e == c0 ? 1 : 0)) * SLOT + (w * NT * 32 + lane) * 4;
#pragma unroll
        for (int n = 0; n < NT; ++n) v[e][n] = c + e <= c1 ? ldcg4(p + n * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int e = 0; e < FLY; ++e)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          acc[n][0] += v[e][n].x; acc[n][1] += v[e][n].y; acc[n][2] += v[e][n].z; acc[n][3] += v[e][n].w;
        }
    }
    epilogue(a.seg[segment(tile)], tile, acc);
  }
}

// Two fp32 weight rows against all activation rows, in fp32 (the few projections that checkpoints keep as floats: expert
// routers, the gates of the delta rule).  They ride in the image's launch because they need the same rows at the same
// time and leave nearly all of the chip free.  The weight rows times the norm wait in shared memory; a warp takes a row,
// or with fewer rows than warps a slice of one; the row's sum of squares falls out of the same pass.  `steady`: all warps a slice of
// one row after the other, so that a row's sums do not depend on how many rows there are.
__device__ void side_rows(const float* w, int n, int n0, float* out, long long ld, const void* x, int x_dtype,
                          long long x_stride, const float* norm_w, float eps, int K, int R, bool steady, float* wsm) {
  __shared__ float part[16][3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool two = n0 + 1 < n;
  for (int i = threadIdx.x * 4; i < K; i += 2048) {
    const float4 m = norm_w != nullptr ? *reinterpret_cast<const float4*>(norm_w + i) : make_float4(1.f, 1.f, 1.f, 1.f);
    const float4 a = *reinterpret_cast<const float4*>(w + (size_t)n0 * K + i);
    const float4 b = *reinterpret_cast<const float4*>(w + (size_t)(n0 + (two ? 1 : 0)) * K + i);
    *reinterpret_cast<float4*>(wsm + i) = make_float4(a.x * m.x, a.y * m.y, a.z * m.z, a.w * m.w);
    *reinterpret_cast<float4*>(wsm + K + i) = make_float4(b.x * m.x, b.y * m.y, b.z * m.z, b.w * m.w);
  }
  pdl_wait();
  __syncthreads();
  int slices = 1;
  if (steady) slices = 16;
  else while (slices * R <= 8) slices <<= 1;                  // R * slices <= 16 warps
  const int sl = warp % slices, r_step = 16 / slices;
  for (int r0 = 0; r0 < R; r0 += r_step) {
    const int r = r0 + warp / slices;
    float ss = 0.f, da = 0.f, db = 0.f;
    if (r < R) {
#pragma unroll 4
      for (int i = (sl * 32 + lane) * 4; i < K; i += slices * 128) {
        float4 v;
        if (x_dtype == 0) {
          v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + (size_t)r * x_stride + i);
        } else {
          const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(x) + (size_t)r * x_stride + i);
          const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
          const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
          v = make_float4(f0.x, f0.y, f1.x, f1.y);
        }
        const float4 a = *reinterpret_cast<const float4*>(wsm + i), b = *reinterpret_cast<const float4*>(wsm + K + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        da += v.x * a.x + v.y * a.y + v.z * a.z + v.w * a.w;
        db += v.x * b.x + v.y * b.y + v.z * b.z + v.w * b.w;
      }
    }
    ss = warp_sum(ss);
    da = warp_sum(da);
    db = warp_sum(db);
    if (lane == 0) {
      part[warp][0] = ss;
      part[warp][1] = da;
      part[warp][2] = db;
    }
    __syncthreads();
    if (sl == 0 && lane == 0 && r < R) {
      ss = da = db = 0.f;
      for (int i = 0; i < slices; ++i) {
        ss += part[warp + i][0];
        da += part[warp + i][1];
        db += part[warp + i][2];
      }
      const float inv = norm_w != nullptr ? rsqrtf(ss / (float)K + eps) : 1.f;
      out[(size_t)r * ld + n0] = da * inv;
      if (two) out[(size_t)r * ld + n0 + 1] = db * inv;
    }
    __syncthreads();
  }
}

// With a norm: one CTA per row, the row kept in registers between the statistics and the fragments (up to 4 blocks a
// warp), a warp per block; CTAs from `R` on take two side rows each.  Without: the blocks of a row are spread over CTAs.
template <bool TC>                    // the image for tcgen05
__global__ void __launch_bounds__(512) rows_image_kernel(const void* __restrict__ x, int x_dtype, long long x_stride,
                                                         const float* __restrict__ norm_w, float eps, int K, int R,
                                                         int pad_rows, int parts, uint8_t* __restrict__ image,
                                                         uint8_t* __restrict__ by_row,
                                                         const float* __restrict__ side_w, int side_n,
                                                         float* __restrict__ side_out, long long side_ld, bool steady) {
  extern __shared__ __align__(16) float side_sm[];
  __shared__ float red[33];
  pdl_launch();
  if ((int)blockIdx.x >= R * parts) {
    side_rows(side_w, side_n, ((int)blockIdx.x - R * parts) * 2, side_out, side_ld, x, x_dtype, x_stride, norm_w, eps, K, R,
              steady, side_sm);
    return;
  }
  const int r = blockIdx.x / parts, nb = K >> 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = (int)(blockDim.x >> 5) * parts, w0 = (int)(blockIdx.x % parts) * (int)(blockDim.x >> 5) + warp;
  const auto store = [&](int blk, const float (&v)[8]) {
    uint8_t* row = by_row == nullptr ? nullptr : by_row + ((size_t)r * nb + blk) * IMG_COL;
    if (TC) image_store<true>(image + (size_t)blk * tc_image(pad_rows), row, pad_rows, r, lane, v);
    else if (image == nullptr) image_store<false>(row, nullptr, 0, 0, lane, v);
    else image_store<false>(image + ((size_t)blk * pad_rows + r) * IMG_COL, row, 0, 0, lane, v);
  };
  constexpr int KEEP = 4;
  float nwv[KEEP][8];
  if (norm_w != nullptr) {              // constants: ahead of the wait
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
      if (w0 + i * nw < nb) load_cols(norm_w, 0, (size_t)(w0 + i * nw) * 256 + lane * 8, nwv[i]);
  }
  pdl_wait();
  const size_t base = (size_t)r * x_stride + lane * 8;
  if (norm_w == nullptr) {
    for (int blk = w0; blk < nb; blk += nw) {
      float v[8];
      load_cols(x, x_dtype, base + (size_t)blk * 256, v);
      store(blk, v);
    }
    return;
  }
  float v[KEEP][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    if (w0 + i * nw >= nb) continue;
    load_cols(x, x_dtype, base + (size_t)(w0 + i * nw) * 256, v[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[i][j] * v[i][j];
  }
  for (int blk = w0 + KEEP * nw; blk < nb; blk += nw) {
    float y[8];
    load_cols(x, x_dtype, base + (size_t)blk * 256, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += y[j] * y[j];
  }
  ss = block_sum(ss, red);
  const float inv = rsqrtf(ss / (float)K + eps);
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    if (w0 + i * nw >= nb) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] *= inv * nwv[i][j];
    store(w0 + i * nw, v[i]);
  }
  for (int blk = w0 + KEEP * nw; blk < nb; blk += nw) {
    float y[8], m[8];
    load_cols(x, x_dtype, base + (size_t)blk * 256, y);
    load_cols(norm_w, 0, (size_t)blk * 256 + lane * 8, m);
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] *= inv * m[j];
    store(blk, y);
  }
}

template <int NT>
int launch_rows(HeRowsArgs a, int num_sms, cudaStream_t stream) {
  using S = Shape<NT>;
  constexpr int IMG = IMG_COL * 8 * NT;
  RowsMaps maps;
  a.tiles = 0;
  a.w_bytes = 0;
  for (int i = 0; i < a.n_seg; ++i) {
    HeRowsSeg& sg = a.seg[i];
    if (sg.n_rows < 1 || sg.out == nullptr || sg.epi < 0 || sg.epi > 4) return -HE_ERR_BAD_ARG;
    int rc = weight_maps(&maps.m[i][0], sg.w, sg.qtype, sg.n_rows, a.K, HALF);
    if (rc == 0 && sg.epi >= 3) rc = weight_maps(&maps.m[i][2], sg.w2, sg.qtype, sg.n_rows, a.K, HALF);
    if (rc != 0) return rc;
    sg.tile0 = a.tiles;
    const int per = sg.epi >= 3 ? HALF : TILE;
    a.tiles += (sg.n_rows + per - 1) / per;
    const int wb = TILE * rows_block_bytes(sg.qtype);
    if (wb > a.w_bytes) a.w_bytes = wb;
  }
  a.stage_bytes = (a.w_bytes + IMG + 1023) & ~1023;
  a.stages = (SMEM_TOTAL - S::XBUF - (int)sizeof(RowsShared) - 1024) / a.stage_bytes;
  if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
  // an even ring, so that a slot always belongs to one group.  A phase bit tells only neighbours apart: a
  // group that skipped the other group's use of a slot could take the phase before that use for its own
  a.stages &= ~1;
  if (a.stages < 2) return -HE_ERR_BAD_ARG;
  const size_t smem = (size_t)a.stages * a.stage_bytes + S::XBUF + sizeof(RowsShared) + 1024;
  static std::atomic<unsigned long long> allowed{0};
  const cudaError_t e = allow_smem(rows_gemm_kernel<NT>, SMEM_TOTAL, allowed);
  if (e != cudaSuccess) return (int)e;
  const long long units = (long long)a.tiles * (a.K >> 8);
  const int grid = (int)(units < num_sms ? units : num_sms);
  if (units > 0x7FFFFFFF || 2ll * grid * TILE * 8 * NT > a.ws_floats || a.tiles > a.n_counters) return -HE_ERR_BAD_ARG;
  return (int)launch_pdl(rows_gemm_kernel<NT>, dim3(grid), dim3(THREADS), smem, stream, maps, a,
                         RowsPlan{(int)(units / grid), (int)(units % grid)});
}

}  // namespace

// Bytes of the activation image of R rows of K columns.
HE_API long long he_rows_image_bytes(int R, int K, int tc) {
  return (long long)(K >> 8) * (tc ? tc_image(tc_rows(R)) : col_groups(R) * 8 * IMG_COL);
}
// Floats of the partial-tile workspace for R rows.
HE_API long long he_rows_ws_floats(int R, int num_sms, int tc) {
  return 2ll * num_sms * TILE * (tc ? tc_rows(R) : col_groups(R) * 8);
}

// Images of (RMSNorm with norm_w of) the R rows x[r][0..K), fp32 or bf16.  K % 256 == 0, 16-byte rows.  `image` (may be
// null): block by block, for a product of 1..64 rows; `by_row` (may be null): row by row, for he_rows_experts, any R; both null:
// the side rows alone.
// With `side_n` > 0 (at most 64 rows) also side_out[r][j] = (normalised row r) . side_w[j], j < side_n: fp32 weights
// [side_n][K], in fp32.  `side_steady`: a row's are the same bits beside any number of others.
HE_API int he_rows_image(const void* x, int x_dtype, long long x_stride, const float* norm_w, float eps, int K, int R,
                         void* image, int tc, void* by_row, const float* side_w, int side_n, float* side_out, long long side_ld,
                         int side_steady, cudaStream_t stream) {
  if (K <= 0 || K % 256 != 0 || R < 1 || ((image != nullptr || side_n > 0) && R > (image != nullptr && !tc ? MMA_MAX_ROWS : 64)) || x == nullptr ||
      (image == nullptr && by_row == nullptr && side_n <= 0) || (reinterpret_cast<uintptr_t>(by_row) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  const int es = x_dtype == 0 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0 || (x_stride * es) % 16 != 0 ||
      (reinterpret_cast<uintptr_t>(norm_w) & 15) != 0 || (reinterpret_cast<uintptr_t>(image) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  const int nb = K >> 8;
  if (image == nullptr) tc = 0;
  size_t smem = 0;
  if (side_n > 0) {
    if (norm_w == nullptr || side_w == nullptr || side_out == nullptr || (reinterpret_cast<uintptr_t>(side_w) & 15) != 0)
      return -HE_ERR_BAD_ARG;
    smem = (size_t)2 * K * sizeof(float);
    constexpr int most = 200 * 1024;
    if (smem > most) return -HE_ERR_BAD_ARG;
    static std::atomic<unsigned long long> allowed[2];
    const cudaError_t e = tc ? allow_smem(rows_image_kernel<true>, most, allowed[1]) : allow_smem(rows_image_kernel<false>, most, allowed[0]);
    if (e != cudaSuccess) return (int)e;
  }
  const int parts = image == nullptr && by_row == nullptr ? 0 : norm_w != nullptr ? 1 : (nb + 3) / 4;
  const unsigned grid = (unsigned)(R * parts + (side_n > 0 ? (side_n + 1) / 2 : 0));
  return (int)launch_pdl(tc ? rows_image_kernel<true> : rows_image_kernel<false>, dim3(grid), dim3(norm_w != nullptr ? 512 : 128), smem, stream, x, x_dtype,
                         x_stride, norm_w, eps, K, R, tc ? tc_rows(R) : col_groups(R) * 8, parts, (uint8_t*)image, (uint8_t*)by_row, side_w, side_n,
                         side_out, side_ld, side_steady != 0);
}

HE_API int he_rows_gemm(const HeRowsArgs* args, int num_sms, cudaStream_t stream) {
  HeRowsArgs a = *args;
  if (a.K <= 0 || a.K % 256 != 0 || a.R < 1 || a.R > 64 || a.n_seg < 1 || a.n_seg > ROWS_MAX_SEG || num_sms < 1 ||
      a.image == nullptr || a.ws == nullptr || a.counters == nullptr || (reinterpret_cast<uintptr_t>(a.image) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(a.ws) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  if (a.tc) return launch_rows_tc(a, num_sms, stream);
  switch (col_groups(a.R)) {
    case 1: return launch_rows<1>(a, num_sms, stream);
    case 2: return launch_rows<2>(a, num_sms, stream);
    case 3: return launch_rows<3>(a, num_sms, stream);
    default: return -HE_ERR_BAD_ARG;
  }
}
HE_API int he_rows_args_size() { return (int)sizeof(HeRowsArgs); }
