// Routed experts over the rows that chose them: every expert's quantised weights are streamed once per 8, 16 or 32 of its rows,
// with the operands of the few-row products (rows_mma.cuh).
//
//   he_moe_jobs      : the (row, expert) pairs sorted by expert, ascending within one, and cut into jobs of at most `cols` rows
//   he_rows_experts  : a CTA takes (job, tile of 256 weight rows) items; the activation image is gathered row by row with
//                      bulk copies while the tile's blocks arrive by TMA.  Gate/up: act(g) * u per pair as bf16; down: one
//                      row per pair
//   he_moe_sum_pairs : residual += sum over a token's k pairs of weight * row, in order
// Expert ids never leave the device.
//
// Why: a decode batch (256 pairs over ~160 of 256 experts at 32 rows, top 8) had one CTA group per PAIR that normalised and
// quantised its row again and read the expert's blocks with 16-byte loads; a prompt (64 rows per expert at 2048) had its
// rows padded to 128 for a tile of the tcgen05 GEMM, whose expansion of 128 x 256 weights costs the same whatever the rows.
// At 32 rows DRAM is at 43-47 % and the issue slots at 60 % (expansion of the blocks); with more rows per expert mma.sync and the
// image reads grow.  A layer's experts (256, 8 used, hidden 2048,
// width 512): 32 rows 100 us for both products (172 us before), a step of 8 layers 2471 -> 1893 us; prompts of 72 / 256 / 1024
// rows 6.1 / 7.3 / 8.6 ms -> 3.9 / 4.4 / 7.1 ms, of 2048 rows 10.6 -> 12.4 ms (those take the jobs of gemm_rows_tc.cu).
// Reference: hipengine/kernels/hip_gfx1100/quant/gguf_q4_k_selected_prefill.hip, moe/group_scatter.hip.
#include "rows_mma.cuh"

using namespace he;
using namespace herows;

namespace {

struct MoeJob {
  int expert, first, count, pad;      // rows entries[first .. first + count)
};

constexpr int JOB_WARPS = 16, MAX_EXPERTS = JOB_WARPS * 32;

// One CTA, a contiguous part of the pairs per warp.  entries: pair ids sorted by expert, in ascending order within one, so that
// the jobs (and the sums of their rows) are the same in every run; meta[0] = number of jobs.
__global__ void __launch_bounds__(MAX_EXPERTS) moe_jobs_kernel(const int* __restrict__ ids, int P, int E, int cols,
                                                               int* __restrict__ entries, MoeJob* __restrict__ jobs,
                                                               int max_jobs, int* __restrict__ meta) {
  __shared__ int at[JOB_WARPS][MAX_EXPERTS];      // pairs of a warp's part per expert, then where its next one goes
  __shared__ int wsum[2][JOB_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = (P + MAX_EXPERTS - 1) / MAX_EXPERTS * 32, p0 = warp * part, p1 = min(P, p0 + part);
  pdl_wait();
  pdl_launch();
  for (int w = 0; w < JOB_WARPS; ++w) at[w][tid] = 0;
  __syncthreads();
  for (int p = p0 + lane; p < p1; p += 32) {
    const int e = ids[p];
    if (HE_INDEX_OK(e, E, HE_SITE_MOE_EXPERT_ID) && e >= 0 && e < E) atomicAdd(&at[warp][e], 1);
  }
  __syncthreads();
  // exclusive sums: of an expert's pairs over the parts before, of the pairs and the jobs of the experts before
  int n = 0;
  for (int w = 0; w < JOB_WARPS; ++w) {
    const int c = at[w][tid];
    at[w][tid] = n;
    n += c;
  }
  const int nj = (n + cols - 1) / cols;
  int a = n, b = nj;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int va = __shfl_up_sync(0xffffffffu, a, o), vb = __shfl_up_sync(0xffffffffu, b, o);
    if (lane >= o) { a += va; b += vb; }
  }
  if (lane == 31) { wsum[0][warp] = a; wsum[1][warp] = b; }
  __syncthreads();
  for (int w = 0; w < warp; ++w) { a += wsum[0][w]; b += wsum[1][w]; }
  for (int w = 0; w < JOB_WARPS; ++w) at[w][tid] += a - n;
  for (int i = 0; i < nj; ++i)
    if (b - nj + i < max_jobs) jobs[b - nj + i] = MoeJob{tid, a - n + i * cols, min(cols, n - i * cols), 0};
  if (tid == MAX_EXPERTS - 1) meta[0] = min(b, max_jobs);
  __syncthreads();
  for (int q = p0; q < p1; q += 32) {
    const int p = q + lane, e = p < p1 ? ids[p] : -1;
    const bool ok = e >= 0 && e < E;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int rank = __popc(same & ((1u << lane) - 1u)), first = ok ? at[warp][e] : 0;
    if (ok) entries[first + rank] = p;
    __syncwarp();
    if (ok && rank == 0) at[warp][e] = first + __popc(same);
    __syncwarp();
  }
}

struct RowsExpertsArgs {
  const void* image;        // row-by-row image of the activation rows
  const MoeJob* jobs;
  const int* entries;
  const int* meta;          // [0]: number of jobs
  void* out;                // [pairs][out_stride]
  long long out_stride;
  int* status;
  int rows_per_image_row;   // pairs that share an image row (k: rows are tokens; 1: rows are pairs)
  int N, K, E;              // weight rows per expert, columns, experts
  int expert_rows;          // rows between consecutive experts in the stacked weights
  int qtype;
  int epi;                  // 0: f32 store, 1: bf16 store, 3: silu(g) * u -> bf16, 4: gelu_tanh(g) * u -> bf16
  int stages, stage_bytes, w_bytes;      // set by the launcher
};

struct ExpertMaps {
  CUtensorMap m[4];         // [2 * (up weight) + (scale plane of Q8_0)]
};

template <int V>
struct Count {
  static constexpr int value = V;
};

constexpr int XT = 256, XH = 128, XTHREADS = 640;     // tile rows, rows of a TMA box, threads (16 MMA warps + helpers)

struct ExpertShared {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  int abort_flag;
};

template <int NT>
__global__ void __launch_bounds__(XTHREADS, 1)
rows_experts_kernel(const __grid_constant__ ExpertMaps maps, const __grid_constant__ RowsExpertsArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  ExpertShared* sh = reinterpret_cast<ExpertShared*>(smem + (size_t)a.stages * a.stage_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = a.K >> 8, bb = rows_block_bytes(a.qtype);
  const bool pair = a.epi >= 3;
  const int per = pair ? XH : XT, tiles = (a.N + per - 1) / per;
  volatile int* abort_flag = &sh->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      sm100::mbar_init(&sh->full[s], 1);
      sm100::mbar_init(&sh->empty[s], 16);
    }
    sh->abort_flag = 0;
    sm100::mbar_fence_init();
  }
  __syncthreads();
  pdl_launch();
  pdl_wait();                      // the jobs and the image come from the kernels before
  const int items = *reinterpret_cast<const volatile int*>(a.meta) * tiles;

  if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == 16) {
      // ------------------------------------------------------------ producer: lane 0 the weights, every lane image rows
      const uint8_t* image = reinterpret_cast<const uint8_t*>(a.image);
      int s = 0, n = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        const MoeJob job = a.jobs[it / tiles];
        const int n0 = (it % tiles) * per;
        const uint8_t* src = image;                  // a job has at most 32 rows: one a lane
        if (lane < job.count) src += (size_t)(a.entries[job.first + lane] / a.rows_per_image_row) * nb * IMG_COL;
        for (int blk = 0; blk < nb; ++blk, ++n) {
          ok = __all_sync(0xffffffffu, wait_long(&sh->empty[s], ph ^ 1u, abort_flag, a.status, 411));
          if (!ok) break;
          uint8_t* dst = smem + (size_t)s * a.stage_bytes;
          if (lane == 0) {
            sm100::mbar_expect_tx(&sh->full[s], (uint32_t)(XT * bb + job.count * IMG_COL));
#pragma unroll 1
            for (int r = 0; r < 2; ++r) {
              const CUtensorMap* m = &maps.m[pair && r ? 2 : 0];
              const int row = job.expert * a.expert_rows + (pair ? n0 : n0 + r * XH);
              uint8_t* d = dst + r * XH * bb;
              if (a.qtype == HE_Q8_0) {
                sm100::tma_load_2d(d, m, &sh->full[s], blk * 256, row);
                sm100::tma_load_2d(d + XH * 128, m, &sh->full[s], blk * 256 + 128, row);
                sm100::tma_load_2d(d + 2 * XH * 128, m + 1, &sh->full[s], a.K + 16 * blk, row);
              } else {
                sm100::tma_load_2d(d, m, &sh->full[s], blk * bb, row);
              }
            }
          }
          __syncwarp();
          if (lane < job.count)
            bulk_load(sm100::smem_u32(dst + a.w_bytes + lane * IMG_COL), src + (size_t)blk * IMG_COL, IMG_COL, &sh->full[s]);
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok && lane == 0) {      // gave up: let the copies in flight land before the CTA leaves
        for (int i = max(0, n - a.stages); i < n; ++i)
          for (int p = 0; p < (1 << 16) && !sm100::mbar_test_wait(&sh->full[i % a.stages], (i / a.stages) & 1); ++p)
            __nanosleep(64);
      }
    }
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");

  // -------------------------------------------------------------- MMA warps: 16 weight rows each
  const uint32_t mg = opaque(MAGIC);
  const int w = warp, g = lane >> 2, t = lane & 3;
  const uint32_t ring = sm100::smem_u32(smem), w_bytes = (uint32_t)a.w_bytes;
  const int i0 = pair ? 8 * w + g : (w & 7) * 16 + g, i1 = pair ? i0 : i0 + 8;
  const uint32_t p0 = (pair ? 0 : w >> 3) * XH * bb, p1 = (pair ? 1 : w >> 3) * XH * bb;
  int s = 0;
  uint32_t ph = 0;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const MoeJob job = a.jobs[it / tiles];
    const int tl = it % tiles, live = (job.count + 7) >> 3;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    auto blocks = [&](auto groups) {       // of eight rows
      constexpr int L = decltype(groups)::value;
      for (int blk = 0; blk < nb; ++blk) {
        if (wait_long(&sh->full[s], ph, abort_flag, a.status, 412)) {
          const uint32_t st = ring + (uint32_t)s * a.stage_bytes, img = st + w_bytes;
          if (a.qtype == HE_Q4_K) block_q4k<NT, L, L <= 2>(st + p0 + i0 * 144, st + p1 + i1 * 144, img, lane, mg, acc);
          else if (a.qtype == HE_Q6_K) {      // prompts: 11 bits; the exact form takes 15-20 % longer at 32 rows a job
            if constexpr (NT <= 2) block_q6k_exact<NT, L>(st + p0 + i0 * 224, st + p1 + i1 * 224, img, lane, mg, acc);
            else block_q6k<NT, L, L <= 2>(st + p0 + i0 * 224, st + p1 + i1 * 224, img, lane, mg, acc);
          }
          else block_q80<NT, L, XH>(st + p0, i0, st + p1, i1, img, lane, mg, acc);
          __syncwarp();
          if (lane == 0) sm100::mbar_arrive(&sh->empty[s]);
        }
        if (++s == a.stages) { s = 0; ph ^= 1u; }
      }
    };
    if (NT == 1 || live * 2 > NT) blocks(Count<NT>{});
    else blocks(Count<(NT + 1) / 2>{});
    if (*abort_flag) break;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      if (n >= live) break;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = 8 * n + 2 * t + j;
        if (c >= job.count) continue;
        const size_t at = (size_t)a.entries[job.first + c] * a.out_stride;
        if (pair) {
          const int row = tl * XH + 8 * w + g;
          const float ga = a.epi == 3 ? silu_f(acc[n][j]) : gelu_tanh_f(acc[n][j]);
          if (row < a.N) reinterpret_cast<__nv_bfloat16*>(a.out)[at + row] = f32_to_bf16(ga * acc[n][2 + j]);
        } else {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int row = tl * XT + 16 * w + g + 8 * k;
            const float v = acc[n][2 * k + j];
            if (row >= a.N) continue;
            if (a.epi == 0) reinterpret_cast<float*>(a.out)[at + row] = v;
            else reinterpret_cast<__nv_bfloat16*>(a.out)[at + row] = f32_to_bf16(v);
          }
        }
      }
    }
  }
}

// h[t][:] += sum_j wts[t][j] * y[t * k + j][:]  (+ sigmoid(sg[t]) * ysh[t][:]); y fp32 or bf16, four columns a thread
template <typename Y>
__global__ void __launch_bounds__(256) moe_sum_pairs_kernel(float* __restrict__ h, long long ldh, const Y* __restrict__ y,
                                                            long long ldy, const float* __restrict__ wts, int k,
                                                            const __nv_bfloat16* __restrict__ ysh, long long ldsh,
                                                            const float* __restrict__ sg, long long ldsg, int N) {
  pdl_wait();
  pdl_launch();
  const int t = blockIdx.y, n = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (n >= N) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = 0; j < k; ++j) {
    const float w = wts[(size_t)t * k + j];
    float4 v;
    if constexpr (sizeof(Y) == 4) {
      v = *reinterpret_cast<const float4*>(y + (size_t)(t * k + j) * ldy + n);
    } else {
      const uint2 u = *reinterpret_cast<const uint2*>(y + (size_t)(t * k + j) * ldy + n);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
      v = make_float4(a.x, a.y, b.x, b.y);
    }
    s.x += w * v.x; s.y += w * v.y; s.z += w * v.z; s.w += w * v.w;
  }
  if (ysh != nullptr) {
    const float gt = sg != nullptr ? sigmoid_f(sg[(size_t)t * ldsg]) : 1.f;
    const uint2 u = *reinterpret_cast<const uint2*>(ysh + (size_t)t * ldsh + n);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    s.x += gt * a.x; s.y += gt * a.y; s.z += gt * b.x; s.w += gt * b.y;
  }
  float4* hp = reinterpret_cast<float4*>(h + (size_t)t * ldh + n);
  float4 v = *hp;
  v.x += s.x; v.y += s.y; v.z += s.z; v.w += s.w;
  *hp = v;
}

// The kernel moves registers from its helper warps to the MMA warps (setmaxnreg: 128 x 32 + 512 x 112 of a block's
// 640 x 96).  A build that gave them fewer registers at launch would wait for the difference for good: refuse it.
template <typename F>
inline bool registers_ok(F kernel) {
  cudaFuncAttributes fa;
  return cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs * 640 >= 128 * 32 + 512 * 112;
}

template <int NT>
int launch_experts(const ExpertMaps& maps, RowsExpertsArgs a, int num_sms, cudaStream_t stream) {
  a.w_bytes = XT * rows_block_bytes(a.qtype);
  a.stage_bytes = (a.w_bytes + IMG_COL * 8 * NT + 1023) & ~1023;
  a.stages = (SMEM_TOTAL - (int)sizeof(ExpertShared) - 1024) / a.stage_bytes;
  if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
  if (a.stages < 2) return -HE_ERR_BAD_ARG;
  const size_t smem = (size_t)a.stages * a.stage_bytes + sizeof(ExpertShared) + 1024;
  static const bool ok = registers_ok(rows_experts_kernel<NT>);
  if (!ok) return -HE_ERR_BAD_ARG;
  static std::atomic<unsigned long long> allowed{0};
  const cudaError_t e = allow_smem(rows_experts_kernel<NT>, SMEM_TOTAL, allowed);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_pdl(rows_experts_kernel<NT>, dim3(num_sms), dim3(XTHREADS), smem, stream, maps, a);
}

}  // namespace

// Jobs that P pairs over E experts can make at most, with up to `cols` rows each.
HE_API long long he_moe_jobs_bound(long long P, int E, int cols) {
  const long long full = P / cols + E;
  return full < P ? full : P;
}

// ids[P] (0 <= id < E <= 512; pairs with others are in no job) -> entries[P], jobs (4 ints each), meta[0].  cols: 8, 16 or 32 for
// he_rows_experts, 64 for he_tc_experts.
HE_API int he_moe_jobs(const int* ids, int P, int E, int cols, int* entries, void* jobs, int max_jobs, int* meta,
                       cudaStream_t stream) {
  if (P <= 0) return 0;
  if (E < 1 || E > MAX_EXPERTS || cols < 1 || max_jobs < he_moe_jobs_bound(P, E, cols)) return -HE_ERR_BAD_ARG;
  return (int)launch_pdl(moe_jobs_kernel, dim3(1), dim3(MAX_EXPERTS), 0, stream, ids, P, E, cols, entries, (MoeJob*)jobs, max_jobs,
                         meta);
}

// Products of the jobs' rows with their experts' weights `w` (and `w2`: the up weights of epi 3, 4), [E * expert_rows][K]
// blocks of one type.  `cols` as given to he_moe_jobs.
HE_API int he_rows_experts(const RowsExpertsArgs* args, const void* w, const void* w2, int cols, int num_sms,
                           cudaStream_t stream) {
  const RowsExpertsArgs& a = *args;
  if (a.K <= 0 || a.K % 256 != 0 || a.N < 1 || a.E < 1 || a.expert_rows < a.N || a.rows_per_image_row < 1 || num_sms < 1 ||
      a.image == nullptr || (reinterpret_cast<uintptr_t>(a.image) & 15) != 0 || a.out == nullptr || a.jobs == nullptr ||
      a.entries == nullptr || a.meta == nullptr || !(a.epi == 0 || a.epi == 1 || a.epi == 3 || a.epi == 4))
    return -HE_ERR_BAD_ARG;
  ExpertMaps maps;
  const long long rows = (long long)a.E * a.expert_rows;
  int rc = weight_maps(&maps.m[0], w, a.qtype, rows, a.K, XH);
  if (rc == 0 && a.epi >= 3) rc = weight_maps(&maps.m[2], w2, a.qtype, rows, a.K, XH);
  if (rc != 0) return rc;
  switch (cols) {
    case 8: return launch_experts<1>(maps, a, num_sms, stream);
    case 16: return launch_experts<2>(maps, a, num_sms, stream);
    case 32: return launch_experts<4>(maps, a, num_sms, stream);
    default: return -HE_ERR_BAD_ARG;
  }
}
HE_API int he_rows_experts_args_size() { return (int)sizeof(RowsExpertsArgs); }

HE_API int he_moe_sum_pairs(float* h, long long ldh, const void* y, int y_dtype, long long ldy, const float* wts, int T, int k,
                            const void* ysh, long long ldsh, const float* sg, long long ldsg, int N, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (N % 4 != 0 || ldh % 4 != 0 || ldy % 4 != 0 || ldsh % 4 != 0 || (reinterpret_cast<uintptr_t>(h) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(y) & (y_dtype == 0 ? 15 : 7)) != 0 || (reinterpret_cast<uintptr_t>(ysh) & 7) != 0)
    return -HE_ERR_BAD_ARG;
  const dim3 grid((N / 4 + 255) / 256, T);
  if (y_dtype == 0)
    return (int)launch_pdl(moe_sum_pairs_kernel<float>, grid, dim3(256), 0, stream, h, ldh, (const float*)y, ldy, wts, k,
                           (const __nv_bfloat16*)ysh, ldsh, sg, ldsg, N);
  return (int)launch_pdl(moe_sum_pairs_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, h, ldh, (const __nv_bfloat16*)y, ldy,
                         wts, k, (const __nv_bfloat16*)ysh, ldsh, sg, ldsg, N);
}
