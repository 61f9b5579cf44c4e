// Products of 17..64 activation rows with QUANTISED weights on the 5th-generation tensor cores (gemm_rows.cu has the rows' image, the
// smaller batches and the arguments).  The weight is the MMA's A operand, 128 rows of it in tensor memory, the rows are its N.
//
//   operands : as in the mma.sync form: sc * q of a k-quant exactly in fp16 (one packed FMA makes two), fp32 sums of a 256-column
//              block, d / dmin / the rows' powers of two once per block, the minima as one more MMA (16 columns, from shared memory)
//              against the rows' sums.  Q8_0 (integer * fp16 scale: 19 bits) takes a second operand for what the first one's
//              rounding leaves, into the accumulator of the minima (64 columns of both in half a slot): exact down to 2^-22 of a
//              block's largest scale.  Q6_K: scale * (q - 32), 13 bits rounded to 11.
//   split    : (tile of 128 weight rows) x (block) units in one contiguous range per SM, shared tiles summed in CTA order by whoever
//              arrives last, as in gemm_rows.cu
//   roles    : eight unpacking warps in two groups, a slot of the tensor memory each: a thread expands a weight row (64 columns at a
//              time, two k-blocks to a barrier).  Two issuers, one for each slot.  Eight summing warps: accumulators -> registers,
//              scaled, over all blocks of the tile.  Producer and signal warp.
//
// What bounds it (counters in profiles/few_row_products_and_expert_jobs.md: issue slots 33 %, tensor pipe 10-16 %, DRAM 18-22 %): chains of instructions in the warps that expand (a block costs a warp 2500 cycles at 1.9 GHz, half of them waits that
// are over, branches and the hand-over; the two groups take turns), above 48 rows also the image, 35 KB from L2 for 18 KB of weights.
// Tried: 16 unpacking warps (22.9 / 25.3 / 27.8 us at 32 / 48 / 64 rows where eight took 21.3 / 22.9 / 26.3), one issuer (23.3 / 24.3 /
// 27.1), tiles of 256 rows that share an image (22.3 / 25.0 / 29.0: 19 % off a block, twice the partial tiles to sum).
// Against mma.sync, whose warps each read the whole image for 16 weight rows (17408 x 5120, 32 / 48 / 64 rows, us in a graph):
// Q4_K 30.7 / 37.9 / 46.8 -> 20.0 / 21.7 / 24.8, Q8_0 44.5 / 42.5 / 54.4 -> 34.3 / 36.5 / 39.2, Q6_K (5120 x 17408) 35.2 / 37.7 / 45.8
// -> 26.1 / 27.8 / 31.9; a step of 64 rows after 1000 tokens, 8 layers of the 27B, 3279 -> 2354 us.
// Experts of prompts: the same pipeline over (job of up to 64 rows of an expert, tile) items.  A job's rows are first gathered into an
// image of their own (43 us for 16384 rows of 2048 columns), which its tiles read from L2.  2048 rows, 256 experts, 8 used, hidden 2048,
// width 512 (Q4_K, Q6_K): gate/up 180-215 us and down 163 us a layer; the grouped GEMM took 130 + 124 + 52 (activation) and 190, with
// 128-row tiles half padding, and rounds its weights to bf16, which these do not.  With Q8_0 experts it is the faster one above 64 pairs an
// expert (models/moe.py).
#include "rows_tc.cuh"

using namespace he;
using namespace herows;

namespace {

struct TcExperts {
  const int4* jobs;        // (expert, first entry, entries, 0)
  const int* entries;      // pairs
  const int* meta;         // [0]: number of jobs
  int expert_rows;
};

constexpr int TILE = 128, HALF = TC_HALF;              // weight rows of a tile, of each weight of a pair
constexpr int TC_JOB_ROWS = 64;                        // rows of an expert job

// N: activation rows, padded to the next multiple of 16; TYPE: block type of all segments, or 0 where they differ.
// EXPERTS: instead of units dealt out, whole (job, tile) items in turn; segment 0 describes an expert's weights, a job's rows have an
// image of their own (he_tc_gather) and results go to the rows of their pairs.
template <int N, int TYPE, bool EXPERTS>
__global__ void __launch_bounds__(TC_THREADS, 1)
rows_gemm_kernel(const __grid_constant__ RowsMaps maps, const __grid_constant__ HeRowsArgs a, const RowsPlan plan,
                 const TcExperts x) {
  constexpr int SUMS = TC_SUM_WARPS, NC = 4 * N / SUMS, SLOT = TILE * N;   // columns of a summing thread, floats of a partial tile
  constexpr int IMG = tc_image(N), IMG_PAD = tc_image_pad(N);
  constexpr int PRODUCER = TC_UNPACK_WARPS + SUMS, SIGNAL = PRODUCER + 1, ISSUER = PRODUCER + 2;     // two issuers
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  // what the loops use is kept in registers: a kernel with 2 KB of maps in its parameters finds others pushed out of the cache
  const int stages = (int)opaque((uint32_t)a.stages);
  const uint32_t stage_bytes = opaque((uint32_t)a.stage_bytes);
  const uint32_t ring = sm100::smem_u32(smem), minima = ring + (uint32_t)stages * stage_bytes;
  TcBars* bar = reinterpret_cast<TcBars*>(smem + (size_t)stages * stage_bytes + 2 * TC_MIN_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (EXPERTS) pdl_wait();               // the jobs come from the kernels before
  const int nb = a.K >> 8, b = blockIdx.x, u0 = EXPERTS ? b : plan.begin(b);
  const int u1 = EXPERTS ? *reinterpret_cast<const volatile int*>(x.meta) * a.tiles : plan.begin(b + 1);
  const int step = EXPERTS ? (int)gridDim.x : 0;        // to a CTA's next item
  // CTAs that share a tile: those that hold its first and last unit and all between
  const auto first_cta = [&](int tile) { return plan.cta_of(tile * nb); };
  const auto last_cta = [&](int tile) { return plan.cta_of((tile + 1) * nb - 1); };
  const int tile_a = u0 / nb, tile_z = (u1 - 1) / nb;           // only the first and the last tile can be shared
  const bool share_a = !EXPERTS && (u0 > tile_a * nb || u1 < (tile_a + 1) * nb);
  const bool share_z = !EXPERTS && tile_z != tile_a && u1 < (tile_z + 1) * nb;
  const auto segment = [&](int tile) {
    if (EXPERTS) return 0;
    int si = 0;
    while (si + 1 < a.n_seg && tile >= a.seg[si + 1].tile0) ++si;
    return si;
  };
  const auto type_of = [&](const HeRowsSeg& sg) { return TYPE ? TYPE : sg.qtype; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      sm100::mbar_init(&bar->full[0][s], 1);
      sm100::mbar_init(&bar->full[1][s], 1);
      sm100::mbar_init(&bar->empty[s], SUMS);
    }
    for (int s = 0; s < 4; ++s) {
      sm100::mbar_init(&bar->ready[s], TC_UNPACK_WARPS / 2);
      sm100::mbar_init(&bar->done[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      sm100::mbar_init(&bar->filled[s], 1);
      sm100::mbar_init(&bar->drained[s], SUMS);
      sm100::mbar_init(&bar->fin[s], 1);
    }
    bar->abort_flag = 0;
    sm100::mbar_fence_init();
  }
  if (warp == ISSUER) {
    sm100::tmem_alloc(&bar->tmem_base, 512);
    sm100::tmem_relinquish();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  pdl_launch();
  const uint32_t tmem = bar->tmem_base;
  volatile int* abort_flag = &bar->abort_flag;
  // (the first poll stands alone: of a barrier that is ready it costs 60 cycles, through the loop 140)
  const auto wait = [&](uint64_t* m, uint32_t parity, int code) {
    return sm100::mbar_test_wait(m, parity) || wait_long(m, parity, abort_flag, a.status, code);
  };

  // The results of weight row 32 q + lane of a tile for columns col .. col + C (C even)
  const auto epilogue = [&](const HeRowsSeg& sg, int tile, int q, int col, const auto& acc) {
    constexpr int C = sizeof(acc) / sizeof(float);
    const int tl = EXPERTS ? tile % a.tiles : tile - sg.tile0;
    int4 job = make_int4(0, 0, a.R, 0);
    if (EXPERTS) job = x.jobs[tile / a.tiles];
    const auto to = [&](int r) { return (size_t)(EXPERTS ? x.entries[job.y + r] : r) * sg.out_stride; };
    if (sg.epi >= 3) {
      // lanes l and l + 16 hold the gate row and its up row: the lower one finishes the first half of the columns
      const bool up = lane >= 16;
      const int row = tl * HALF + 16 * q + (lane & 15);
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(sg.out) + row;
#pragma unroll
      for (int j = 0; j < C / 2; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, up ? acc[j] : acc[j + C / 2], 16);
        const float gv = up ? other : acc[j], uv = up ? acc[j + C / 2] : other;
        const int r = col + j + (up ? C / 2 : 0);
        const float ga = sg.epi == 3 ? silu_f(gv) : gelu_tanh_f(gv);
        if (r < job.z && row < sg.n_rows) o[to(r)] = f32_to_bf16(ga * uv);
      }
      return;
    }
    const int row = tl * TILE + 32 * q + lane;
    if (row >= sg.n_rows) return;
    const int n = min(C, job.z - col);
    if (sg.epi == 1) {
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(sg.out) + row;
#pragma unroll
      for (int j = 0; j < C; ++j)
        if (j < n) o[to(col + j)] = f32_to_bf16(acc[j]);
      return;
    }
    float* o = reinterpret_cast<float*>(sg.out) + row;
    float old[C];                       // all loads before the first store: they could be of the same address, for the compiler
#pragma unroll
    for (int j = 0; j < C; ++j) old[j] = sg.epi == 2 && j < n ? o[to(col + j)] : 0.f;
#pragma unroll
    for (int j = 0; j < C; ++j)
      if (j < n) o[to(col + j)] = sg.epi == 2 ? old[j] + acc[j] : acc[j];
  };
  // Shared tiles that this CTA was the last to arrive at: sums of the partial tiles in CTA order, by all unpacking and summing
  // warps with four partial tiles in flight (by the summing warps alone, one after the other: 4 us of a launch)
  const auto finish = [&](int w) {
    if (!(share_a || share_z)) return;
    named_sync(3, 32 * (TC_UNPACK_WARPS + SUMS) + 32);
    constexpr int V = N / 16;           // float4 of a thread: a quarter of the columns
    const int q = w & 3, g = w >> 2;
    const uint32_t from = (uint32_t)((((g >> 1) * 4 + q) * (NC / 4) + (g & 1) * V) * 32 + lane) * 4;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      if (!(i == 0 ? share_a : share_z) || !bar->last[i]) continue;
      const int tile = i == 0 ? tile_a : tile_z, c0 = first_cta(tile), c1 = last_cta(tile);
      float acc[4 * V];
#pragma unroll
      for (int k = 0; k < 4 * V; ++k) acc[k] = 0.f;
      for (int c = c0; c <= c1; c += 4) {
        float4 v[4][V];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // the first of them holds the tile's first unit (slot 1 of its CTA), the others' ranges start inside it (slot 0)
          const float* p = a.ws + (size_t)(2 * (c + e) + (c + e == c0 ? 1 : 0)) * SLOT + from;
#pragma unroll
          for (int k = 0; k < V; ++k) v[e][k] = c + e <= c1 ? ldcg4(p + k * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int k = 0; k < V; ++k) {
            acc[4 * k] += v[e][k].x; acc[4 * k + 1] += v[e][k].y; acc[4 * k + 2] += v[e][k].z; acc[4 * k + 3] += v[e][k].w;
          }
      }
      epilogue(a.seg[segment(tile)], tile, q, (g >> 1) * NC + (g & 1) * (4 * V), acc);
    }
  };

  if (warp < TC_UNPACK_WARPS) {
    // -------------------------------------------------------------- unpack: two groups of four warps, one for each operand slot; a
    // thread takes a weight row.  (Reads nothing that the kernels before wrote.)
    const uint32_t mg = opaque(MAGIC), grp = (uint32_t)warp >> 2;
    const int q = warp & 3;
    const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + TC_A_COL + grp * TC_A_SLOT;
    const uint32_t mins = minima + grp * TC_MIN_BYTES + (uint32_t)((4 * q + (lane >> 3)) * 256 + (lane & 7) * 16);
    uint64_t* full = bar->full[grp];
    uint32_t j = 0, done_ph = 1;
    TcWalk at_stage;
    bool ok = true;
    const auto slot_free = [&](int half) {
      ok = ok && wait(&bar->done[2 * grp + half], done_ph, 403);
      sm100::tc_fence_after();
    };
    const auto stored = [&]() {
      sm100::tmem_st_wait();
      sm100::tc_fence_before();
      __syncwarp();
    };
    for (int u = u0; u < u1 && ok;) {
      const int tile = EXPERTS ? u : u / nb, n_blk = EXPERTS ? nb : min(nb - (u - tile * nb), u1 - u);
      const HeRowsSeg& sg = a.seg[segment(tile)];
      const bool pair = sg.epi >= 3;
      const int qtype = type_of(sg), bb = rows_block_bytes(qtype);
      const TcRow at_row(pair, q, lane, bb, qtype);
      u += EXPERTS ? step : n_blk;
      for (int k = 0; k < n_blk; ++k, ++j) {
        const bool mine = (j & 1) == grp;
        if (mine) {
          ok = wait(&full[at_stage.s], at_stage.ph, 402);
          if (!ok) break;
        }
        const uint32_t row = ring + (uint32_t)at_stage.s * stage_bytes + IMG_PAD + at_row.off;
        if (mine && qtype == HE_Q8_0) {
          // 64 columns at a time: first and second operands in a half of the slot
          const float inv = tc_q80_inv(tc_q80_pow(row, at_row));
#pragma unroll 2
          for (int c = 0; c < 4; ++c) {
            uint32_t x[32], f[2], r[32];
            tc_q80(row, at_row, c, inv, mg, x, f);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = h2_mul(x[i], f[i >> 4]);
            slot_free(c & 1);
            sm100::tmem_st_32x32(at + 64 * (c & 1), r);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = h2_rest(x[i], f[i >> 4], r[i]);
            sm100::tmem_st_32x32(at + 64 * (c & 1) + 32, r);
            stored();
            if (lane == 0) sm100::mbar_arrive(&bar->ready[2 * grp + (c & 1)]);
            if (c & 1) done_ph ^= 1u;
          }
        } else if (mine) {
          uint4 meta;
          if (qtype == HE_Q4_K) meta = lds128(row);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            if (qtype == HE_Q4_K) tc_q4k(row, c, meta, mg, r);
            else tc_q6k(row, c, mg, r);
            if ((c & 1) == 0) slot_free(c >> 1);               // a half of the block has half the slot and barriers of its own
            sm100::tmem_st_32x32(at + 32 * c, r);
            if (c & 1) {
              if (qtype == HE_Q4_K && c == 3) {
                const uint4 mn = tc_q4k_minima(meta);
                sts128(mins, mn);
                sts128(mins + 128, mn);
                sm100::fence_proxy_async_smem();
              }
              stored();
              if (lane == 0) sm100::mbar_arrive(&bar->ready[2 * grp + (c >> 1)]);
            }
          }
          done_ph ^= 1u;
        }
        if (!ok) break;
        at_stage.next(stages);
      }
    }
    pdl_wait();
    finish(warp);
  } else if (warp < PRODUCER) {
    // -------------------------------------------------------------- sums over the blocks: a thread has NC columns of a weight row
    const int w = warp - TC_UNPACK_WARPS, q = w & 3, h = w >> 2;
    const uint32_t dt = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * NC);
    pdl_wait();
    const uint32_t part = (uint32_t)((w * (NC / 4) * 32 + lane) * 4);
    uint32_t j = 0;
    int s = 0;
    for (int u = u0; u < u1;) {
      const int tile = EXPERTS ? u : u / nb, blk0 = EXPERTS ? 0 : u - tile * nb, n_blk = min(nb - blk0, EXPERTS ? nb : u1 - u);
      const HeRowsSeg& sg = a.seg[segment(tile)];
      const bool pair = sg.epi >= 3;
      const int qtype = type_of(sg), bb = rows_block_bytes(qtype);
      const TcRow at_row(pair, q, lane, bb, qtype);
      uint64_t sum[NC / 2];
#pragma unroll
      for (int k = 0; k < NC / 2; ++k) sum[k] = 0;
      u += EXPERTS ? step : n_blk;
      for (int k = 0; k < n_blk; ++k, ++j) {
        const uint32_t slot = j & 1;
        const uint32_t st = ring + (uint32_t)s * stage_bytes, t = dt + slot * (2 * N);
        // (the products of a block follow its arrival: what the unpacking warps saw, whoever sees their products sees)
        const bool ok = wait(&bar->filled[slot], (j >> 1) & 1, 407);
        if (ok) {
          const uint32_t row = st + IMG_PAD + at_row.off;
          const uint32_t xs = st + tc_scales(N) + (uint32_t)(h * NC * 4);
          sm100::tc_fence_after();
          if (qtype == HE_Q4_K) {
            const uint32_t dm = lds32(row);
            const float2 dv = __half22float2(*reinterpret_cast<const __half2*>(&dm));
            tc_add<NC, true>(t, N, xs, dv.x, -dv.y, sum);
          } else {
            const float d = qtype == HE_Q6_K ? half_bits_to_f32((uint16_t)lds32(row + 208)) : tc_q80_pow(row, at_row) * TC_Q80_SCALE;
            if (tc_two(qtype)) tc_add<NC, true>(t, N, xs, d, d, sum);
            else tc_add<NC, false>(t, N, xs, d, 0.f, sum);
          }
          sm100::tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            sm100::mbar_arrive(&bar->drained[slot]);
            sm100::mbar_arrive(&bar->empty[s]);
          }
        }
        if (++s == stages) s = 0;
      }
      float acc[NC];
#pragma unroll
      for (int k = 0; k < NC / 2; ++k) f2_get(sum[k], acc[2 * k], acc[2 * k + 1]);
      if ((tile == tile_a && share_a) || (tile == tile_z && share_z)) {
        // a partial tile: the CTA's own slot 1 if it holds the tile's first unit, else slot 0
        float* mine = a.ws + (size_t)(2 * b + (blk0 == 0 ? 1 : 0)) * SLOT + part;
#pragma unroll
        for (int k = 0; k < NC / 4; ++k)
          *reinterpret_cast<float4*>(mine + k * 128) = make_float4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
        if (tile == tile_a) named_arrive(1, 32 * SUMS + 32);
        else named_arrive(2, 32 * SUMS + 32);
        continue;
      }
      epilogue(sg, tile, q, h * NC, acc);
    }
    finish(TC_UNPACK_WARPS + w);
  } else if (warp == PRODUCER) {
    // -------------------------------------------------------------- producer
    const uint8_t* image = reinterpret_cast<const uint8_t*>(a.image);
    const bool leader = sm100::elect_one();
    int si = EXPERTS ? 0 : segment(u0 / nb), tile = EXPERTS ? u0 : u0 / nb, blk = EXPERTS ? 0 : u0 % nb;
    const auto weights = [&](int i, int s) {
      while (!EXPERTS && si + 1 < a.n_seg && tile >= a.seg[si + 1].tile0) ++si;
      const HeRowsSeg& sg = a.seg[si];
      const int qtype = type_of(sg), bb = rows_block_bytes(qtype);
      const bool pair = sg.epi >= 3;
      if (leader) {
        uint8_t* dst = smem + (size_t)s * stage_bytes + IMG_PAD;
        uint64_t* full = &bar->full[i & 1][s];
        sm100::mbar_expect_tx(full, (uint32_t)(TILE * bb + IMG));
        const int n0 = EXPERTS ? x.jobs[tile / a.tiles].x * x.expert_rows + tile % a.tiles * (pair ? HALF : TILE)
                               : (tile - sg.tile0) * (pair ? HALF : TILE);
        if (qtype == HE_Q8_0) {
          const int h = pair ? HALF : TILE;
#pragma unroll 1
          for (int r = 0; r < (pair ? 2 : 1); ++r) {
            uint8_t* d = dst + r * HALF * 272;
            sm100::tma_load_2d(d, &maps.m[si][2 * r], full, blk * 256, n0);
            sm100::tma_load_2d(d + h * 128, &maps.m[si][2 * r], full, blk * 256 + 128, n0);
            sm100::tma_load_2d(d + 2 * h * 128, &maps.m[si][2 * r + 1], full, a.K + 16 * blk, n0);
          }
        } else {
          sm100::tma_load_2d(dst, &maps.m[si][0], full, blk * bb, n0);
          if (pair) sm100::tma_load_2d(dst + HALF * bb, &maps.m[si][2], full, blk * bb, n0);
        }
      }
      __syncwarp();
      if (++blk == nb) { blk = 0; tile += EXPERTS ? step : 1; }
    };
    const auto rows = [&](int i, int s, int blk) {
      if (leader) bulk_load(ring + (uint32_t)s * stage_bytes, image + (size_t)blk * IMG, IMG, &bar->full[i & 1][s]);
      __syncwarp();
    };
    const int n = EXPERTS ? (u1 > u0 ? (u1 - u0 + step - 1) / step * nb : 0) : u1 - u0, pre = EXPERTS ? 0 : min(n, stages);
    for (int i = 0; i < pre; ++i) weights(i, i);
    pdl_wait();                         // the rows (and so their image) come from the kernels before
    for (int i = 0; i < pre; ++i) rows(i, i, (u0 + i) % nb);
    int s = 0;
    uint32_t ph = 0;
    int issued = pre;
    for (int i = pre; i < n; ++i) {
      if (EXPERTS ? i >= stages && !wait(&bar->empty[s], ph ^ 1u, 401) : !wait(&bar->empty[s], ph, 401)) break;
      const int bi = EXPERTS ? tile / a.tiles * nb + blk : blk;
      weights(i, s);
      rows(i, s, bi);
      ++issued;
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
    if (issued < n) {                   // gave up: let the copies in flight land before the CTA leaves
      TcWalk at_stage;
      for (int i = 0; i < issued; ++i, at_stage.next(stages))
        for (int p = 0; i >= issued - stages && p < (1 << 16) && !sm100::mbar_test_wait(&bar->full[i & 1][at_stage.s], at_stage.ph); ++p)
          __nanosleep(64);
    }
  } else if (warp >= ISSUER) {
    // -------------------------------------------------------------- issuers of the products, one for each slot (and its accumulators).
    // The whole warp walks (addresses stay in uniform registers), one lane issues
    constexpr uint32_t IDESC = idesc_f16(N);
    const bool leader = sm100::elect_one();
    const uint32_t me = (uint32_t)(warp - ISSUER), t = __shfl_sync(0xffffffffu, tmem, 0) + TC_A_COL + me * TC_A_SLOT;
    const uint32_t d = t - TC_A_COL - me * TC_A_SLOT + me * (2 * N);
    const uint64_t mins = desc_k16(minima + me * TC_MIN_BYTES);
    uint64_t *ready = bar->ready + 2 * me, *done = bar->done + 2 * me;
    uint32_t j = 0, ph = 0, free_ph = 1;
    int s = 0;
    bool ok = true;
    for (int u = u0; u < u1 && ok;) {
      const int tile = EXPERTS ? u : u / nb, n_blk = EXPERTS ? nb : min(nb - (u - tile * nb), u1 - u);
      const int qtype = type_of(a.seg[segment(tile)]);
      u += EXPERTS ? step : n_blk;
      for (int k = 0; k < n_blk && ok; ++k, ++j) {
        if ((j & 1) == me) {
          const uint32_t img = ring + (uint32_t)s * stage_bytes;
          const uint64_t x = sm100::umma_desc_k_sw128(img);
          ok = wait(&bar->drained[me], free_ph, 409);
          free_ph ^= 1u;
          if (tc_two(qtype)) {
            // second operands have the accumulator of the minima, which their types do without
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              ok = ok && wait(ready + (c & 1), ph, 405);
              sm100::tc_fence_after();
              if (leader && ok) {
                const uint32_t o = t + 64 * (c & 1);
                const uint64_t xc = x + (uint64_t)(c * N * 8);
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  sm100::umma_f16_ts(e < 4 ? d : d + N, o + e * 8, xc + (uint64_t)((e & 3) * 2), IDESC, c > 0 || (e & 3) > 0);
                sm100::umma_commit(done + (c & 1));
              }
              __syncwarp();
              if (c & 1) ph ^= 1u;
            }
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              ok = ok && wait(ready + h, ph, 405);
              sm100::tc_fence_after();
              if (leader && ok) {
#pragma unroll
                for (int e = 8 * h; e < 8 * h + 8; ++e)
                  sm100::umma_f16_ts(d, t + e * 8, x + (uint64_t)((e >> 2) * (N * 8) + (e & 3) * 2), IDESC, e > 0);
                if (qtype == HE_Q4_K && h == 1) sm100::umma_f16(d + N, mins, desc_k16(img + tc_sums(N)), IDESC, 0);
                sm100::umma_commit(done + h);
              }
              __syncwarp();
            }
            ph ^= 1u;
          }
          if (leader && ok) sm100::umma_commit(&bar->filled[me]);
          __syncwarp();
        }
        if (++s == stages) s = 0;
      }
    }
    if (!ok && leader) {                // gave up: let the products in flight end before the tensor memory goes
      sm100::umma_commit(&bar->fin[me]);
      for (int p = 0; p < (1 << 16) && !sm100::mbar_test_wait(&bar->fin[me], 0); ++p) __nanosleep(64);
    }
    __syncwarp();
  } else if (warp == SIGNAL) {
    // -------------------------------------------------------------- arrivals at shared tiles
    // A fence and an atomic take a round trip to L2 each; this warp makes it while the summing warps go on.
    pdl_wait();
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      if (!(i == 0 ? share_a : share_z)) continue;
      const int tile = i == 0 ? tile_a : tile_z;
      // the partial tile is written (one barrier each: the summing warps may be at the second before this warp is at the first)
      if (i == 0) named_sync(1, 32 * SUMS + 32);
      else named_sync(2, 32 * SUMS + 32);
      if (lane == 0) {
        __threadfence();
        const int n = last_cta(tile) - first_cta(tile);
        const bool last = atomicAdd(a.counters + tile, 1) == n;
        if (last) a.counters[tile] = 0;
        __threadfence();
        bar->last[i] = last;
      }
      __syncwarp();
    }
    if (share_a || share_z) named_arrive(3, 32 * (TC_UNPACK_WARPS + SUMS) + 32);
  }

  sm100::tc_fence_before();
  __syncthreads();
  if (warp == ISSUER) {
    sm100::tc_fence_after();
    sm100::tmem_dealloc(tmem, 512);
  }
}

template <int N, int TYPE, bool EXPERTS>
int launch_typed(const RowsMaps& maps, const HeRowsArgs& a, size_t smem, int grid, const RowsPlan& plan, const TcExperts& x,
                 cudaStream_t stream) {
  static std::atomic<unsigned long long> allowed{0};
  const cudaError_t e = allow_smem(rows_gemm_kernel<N, TYPE, EXPERTS>, TC_SMEM, allowed);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_pdl(rows_gemm_kernel<N, TYPE, EXPERTS>, dim3(grid), dim3(TC_THREADS), smem, stream, maps, a, plan, x);
}

constexpr int TC_FIXED = 1024 + 2 * TC_MIN_BYTES + (int)sizeof(TcBars);

// Stages of a ring for n activation rows and a block of `w_bytes` of weights
int ring_stages(int n, int w_bytes) {
  int s = (TC_SMEM - TC_FIXED) / (tc_image_pad(n) + ((w_bytes + 1023) & ~1023));
  if (s > TC_MAX_STAGES) s = TC_MAX_STAGES;
  return s > 4 ? s & ~1 : s;
}

// Stages of the ring, set in `a`; dynamic shared memory of a block, or 0 where it does not hold two stages
template <int N>
size_t ring(HeRowsArgs& a) {
  a.stage_bytes = tc_image_pad(N) + ((a.w_bytes + 1023) & ~1023);
  a.stages = ring_stages(N, a.w_bytes);
  return a.stages < 2 ? 0 : (size_t)a.stages * a.stage_bytes + TC_FIXED;
}

template <int N>
int launch_rows(HeRowsArgs a, int num_sms, cudaStream_t stream) {
  RowsMaps maps;
  a.tiles = 0;
  a.w_bytes = 0;
  int type = a.seg[0].qtype;
  for (int i = 0; i < a.n_seg; ++i) {
    HeRowsSeg& sg = a.seg[i];
    if (sg.n_rows < 1 || sg.out == nullptr || sg.epi < 0 || sg.epi > 4) return -HE_ERR_BAD_ARG;
    const int per = sg.epi >= 3 ? HALF : TILE;
    int rc = weight_maps(&maps.m[i][0], sg.w, sg.qtype, sg.n_rows, a.K, per);
    if (rc == 0 && sg.epi >= 3) rc = weight_maps(&maps.m[i][2], sg.w2, sg.qtype, sg.n_rows, a.K, per);
    if (rc != 0) return rc;
    sg.tile0 = a.tiles;
    a.tiles += (sg.n_rows + per - 1) / per;
    const int wb = TILE * rows_block_bytes(sg.qtype);
    if (wb > a.w_bytes) a.w_bytes = wb;
    if (sg.qtype != type) type = 0;
  }
  const size_t smem = ring<N>(a);
  if (smem == 0) return -HE_ERR_BAD_ARG;
  const long long units = (long long)a.tiles * (a.K >> 8);
  const int grid = (int)(units < num_sms ? units : num_sms);
  if (units > 0x7FFFFFFF || 2ll * grid * TILE * N > a.ws_floats || a.tiles > a.n_counters) return -HE_ERR_BAD_ARG;
  const RowsPlan plan{(int)(units / grid), (int)(units % grid)};
  switch (type) {
    case HE_Q4_K: return launch_typed<N, HE_Q4_K, false>(maps, a, smem, grid, plan, TcExperts{}, stream);
    case HE_Q6_K: return launch_typed<N, HE_Q6_K, false>(maps, a, smem, grid, plan, TcExperts{}, stream);
    case HE_Q8_0: return launch_typed<N, HE_Q8_0, false>(maps, a, smem, grid, plan, TcExperts{}, stream);
    default: return launch_typed<N, 0, false>(maps, a, smem, grid, plan, TcExperts{}, stream);
  }
}

int launch_experts(HeRowsArgs a, const TcExperts& x, long long rows, int num_sms, cudaStream_t stream) {
  constexpr int N = TC_JOB_ROWS;
  const HeRowsSeg& sg = a.seg[0];
  const int per = sg.epi >= 3 ? HALF : TILE;
  RowsMaps maps;
  int rc = weight_maps(&maps.m[0][0], sg.w, sg.qtype, rows, a.K, per);
  if (rc == 0 && sg.epi >= 3) rc = weight_maps(&maps.m[0][2], sg.w2, sg.qtype, rows, a.K, per);
  if (rc != 0) return rc;
  a.n_seg = 1;
  a.tiles = (sg.n_rows + per - 1) / per;
  a.w_bytes = TILE * rows_block_bytes(sg.qtype);
  const size_t smem = ring<N>(a);
  if (smem == 0) return -HE_ERR_BAD_ARG;
  const RowsPlan plan{1, 0};
  switch (sg.qtype) {
    case HE_Q4_K: return launch_typed<N, HE_Q4_K, true>(maps, a, smem, num_sms, plan, x, stream);
    case HE_Q6_K: return launch_typed<N, HE_Q6_K, true>(maps, a, smem, num_sms, plan, x, stream);
    case HE_Q8_0: return launch_typed<N, HE_Q8_0, true>(maps, a, smem, num_sms, plan, x, stream);
    default: return -HE_ERR_BAD_ARG;
  }
}

// Images of the jobs' rows: row entries[first + c] / per_row of x becomes row c of its job's image.  A CTA a (job, block), a warp a row,
// four rows of a warp in flight.  (A CTA a job: 52 us for 16384 rows of 2048 columns, a chain of loads a warp.)
__global__ void __launch_bounds__(512) gather_kernel(const void* __restrict__ rows, int dtype, long long stride, int K,
                                                     const int4* __restrict__ jobs, const int* __restrict__ entries,
                                                     const int* __restrict__ meta, int per_row, uint8_t* __restrict__ image) {
  constexpr int n = TC_JOB_ROWS;
  pdl_wait();
  pdl_launch();
  if ((int)blockIdx.x >= *meta) return;
  const int4 job = jobs[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, blk = blockIdx.y;
  uint8_t* img = image + ((size_t)blockIdx.x * (K >> 8) + blk) * tc_image(n);
  float v[4][8];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int c = warp + 16 * e;
    if (c < job.z)
      load_cols(rows, dtype, (size_t)(entries[job.y + c] / per_row) * stride + blk * 256 + lane * 8, v[e]);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int c = warp + 16 * e;
    if (c < job.z) image_store<true>(img, nullptr, n, c, lane, v[e]);
  }
}

}  // namespace

int herows::launch_rows_tc(const HeRowsArgs& a, int num_sms, cudaStream_t stream) {
  switch (tc_rows(a.R)) {
    case 32: return launch_rows<32>(a, num_sms, stream);
    case 48: return launch_rows<48>(a, num_sms, stream);
    default: return launch_rows<64>(a, num_sms, stream);
  }
}

// The way of blocks 0 .. n through the ring of a product of R rows (blocks of the largest type `qtype`): stage and parity of the
// arrival of each.  Returns the stages.
HE_API int he_rows_tc_walk(int R, int qtype, int n, int* stage, int* parity) {
  const int stages = ring_stages(tc_rows(R), TILE * rows_block_bytes(qtype));
  TcWalk w;
  for (int j = 0; j < n; ++j, w.next(stages)) {
    stage[j] = w.s;
    parity[j] = (int)w.ph;
  }
  return stages;
}

// Bytes of the images of `jobs` jobs of up to 64 rows of K columns.
HE_API long long he_tc_gather_bytes(long long jobs, int K) { return jobs * (K >> 8) * (long long)tc_image(TC_JOB_ROWS); }

// Images of the rows of `max_jobs` jobs at most (he_moe_jobs with 64 columns): fp32 or bf16 rows, 16-byte aligned.
HE_API int he_tc_gather(const void* rows, int dtype, long long stride, int K, const void* jobs, const int* entries, const int* meta,
                        int per_row, int max_jobs, void* image, cudaStream_t stream) {
  if (K <= 0 || K % 256 != 0 || per_row < 1 || max_jobs < 1 || rows == nullptr || image == nullptr ||
      (reinterpret_cast<uintptr_t>(rows) & 15) != 0 || (stride * (dtype == 0 ? 4 : 2)) % 16 != 0 ||
      (reinterpret_cast<uintptr_t>(image) & 15) != 0 || (reinterpret_cast<uintptr_t>(jobs) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  return (int)launch_pdl(gather_kernel, dim3(max_jobs, K >> 8), dim3(512), 0, stream, rows, dtype, stride, K, (const int4*)jobs, entries,
                         meta, per_row, (uint8_t*)image);
}

// Products of the jobs' rows with their experts' weights, from the images of he_tc_gather; see he_rows_experts.  `a`: segment 0 (n_rows
// of an expert, out by pair), K, image, status.
HE_API int he_tc_experts(const HeRowsArgs* args, int experts, const void* jobs, const int* entries, const int* meta,
                         int num_sms, cudaStream_t stream) {
  HeRowsArgs a = *args;
  const HeRowsSeg& sg = a.seg[0];
  if (a.K <= 0 || a.K % 256 != 0 || sg.n_rows < 1 || experts < 1 || num_sms < 1 || a.image == nullptr || sg.out == nullptr ||
      (reinterpret_cast<uintptr_t>(a.image) & 15) != 0 || jobs == nullptr || entries == nullptr || meta == nullptr ||
      !(sg.epi == 0 || sg.epi == 1 || sg.epi == 3 || sg.epi == 4))
    return -HE_ERR_BAD_ARG;
  const TcExperts x{(const int4*)jobs, entries, meta, sg.n_rows};
  return launch_experts(a, x, (long long)experts * sg.n_rows, num_sms, stream);
}
