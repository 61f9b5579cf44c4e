// Gated DeltaNet (linear attention): prepare (L2-norm q,k + gates), the recurrent scan over packed
// segments (decode rows, verify chains and prefill share one kernel), and the gated output RMSNorm.
//
// Per V head the state S is [Dk x Dv] fp32 and each step is
//     S <- decay*S ;  kv = k^T S ;  delta = beta*(v - kv) ;  S <- S + k (x) delta ;  o = q^T S
// (hipengine/kernels/hip_gfx1100/linear_attn/gdn.hip:126-330; oracle hipengine/kernels/cpu_reference/ops.py:1967-2012).
// Columns of S are independent, so a head is split into Dv/32 column slices, one CTA each: with 48 heads x 4
// slices a single request already fills the 148 SMs.  Inside a CTA a column is owned by 4 lanes of one warp
// (rows r = lane%4 + 4*i), so the two reductions per token are two xor-shuffles and no block barrier.
// GGUF head order: V head h reads K head h % num_k_heads (gdn.hip:106-118).
#include "common.cuh"

using namespace he;

namespace {

struct GdnPrepArgs {
  float* qkv;            // [T][C] conv output, q and k normalised in place
  const float* a;        // [T][a_stride]
  const float* b;        // [T][b_stride]
  long long a_stride, b_stride;
  const float* ssm_a;    // [Hv]  (negative coefficient)
  const float* dt_bias;  // [Hv]
  float* decay;          // [T][Hv]
  float* beta;           // [T][Hv]
  int C, G, Hv, S, T;
};

// grid T, block 256
__global__ void __launch_bounds__(256) gdn_prepare_kernel(const GdnPrepArgs p) {
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  float* row = p.qkv + (size_t)t * p.C;
  const float qscale = rsqrtf((float)p.S);
  for (int h = warp; h < 2 * p.G; h += nwarp) {
    float* v = row + (size_t)h * p.S;
    float ss = 0.f;
    for (int i = lane; i < p.S; i += 32) ss += v[i] * v[i];
    ss = warp_sum(ss);
    float inv = 1.f / fmaxf(sqrtf(ss), 1e-6f);
    if (h < p.G) inv *= qscale;
    for (int i = lane; i < p.S; i += 32) v[i] *= inv;
  }
  for (int h = threadIdx.x; h < p.Hv; h += blockDim.x) {
    const float av = p.a[(size_t)t * p.a_stride + h], bv = p.b[(size_t)t * p.b_stride + h];
    p.beta[(size_t)t * p.Hv + h] = sigmoid_f(bv);
    p.decay[(size_t)t * p.Hv + h] = __expf(p.ssm_a[h] * softplus20_f(av + p.dt_bias[h]));
  }
}

struct GdnScanArgs {
  const float* qkv;       // [T][C]  prepared conv output: q | k | v
  const float* decay;     // [T][Hv]
  const float* beta;      // [T][Hv]
  float* state;           // [n_slots][Hv][Dk][Dv]
  const int* seg_start;   // [n_seg+1]
  const int* seg_slot;    // [n_seg]
  float* out;             // [T][Hv][Dv]
  float* journal;         // optional [T][Hv][Dk][Dv] state after each token
  int C, G, Hv, T, n_seg;
  int write_state;        // 1: store the final state back to `state`
};

constexpr int DK = 128;       // state rows (key dim)
constexpr int DV = 128;       // state cols (value dim)
constexpr int SLICE = 32;     // columns per CTA
constexpr int TCH = 16;       // tokens staged per shared-memory chunk

constexpr int KPAD = DK + DK / 8;   // 4 pad floats per 32 so the 4 row groups of a column land in different banks

// grid (n_seg, Hv, DV/SLICE), block 32*LPC.  A column of S is owned by LPC lanes of one warp; lane ks owns rows
// ks*RPL .. ks*RPL+RPL-1 (RPL = 128/LPC).  LPC = 4 keeps more of the state per thread (fewer shuffles per token);
// LPC = 8 doubles the warps when only a few (segment, head) pairs exist, which is what hides the issue latency of
// this strictly sequential recurrence during a single-request prefill.
template <int LPC>
__global__ void __launch_bounds__(32 * LPC) gdn_scan_kernel(const GdnScanArgs p) {
  constexpr int RPL = DK / LPC;            // rows per lane: 32 or 16
  constexpr int NT = 32 * LPC;             // threads
  constexpr int CPW = 32 / LPC;            // columns per warp
  __shared__ __align__(16) float sq[TCH][KPAD];
  __shared__ __align__(16) float sk[TCH][KPAD];
  __shared__ float sv[TCH][SLICE];
  __shared__ float sdec[TCH], sbeta[TCH];
  const int sg = blockIdx.x, h = blockIdx.y, sl = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cw = warp * CPW + lane / LPC;               // column inside the slice
  const int col = sl * SLICE + cw;                      // column of S owned (with LPC-1 other lanes)
  const int ks = lane % LPC;
  const int kh = h % p.G;
  const int s0 = p.seg_start[sg], s1 = p.seg_start[sg + 1];
  float* Sg = p.state + (((size_t)p.seg_slot[sg] * p.Hv + h) * DK) * DV;
  float S[RPL];
#pragma unroll
  for (int i = 0; i < RPL; ++i) S[i] = Sg[(size_t)(ks * RPL + i) * DV + col];
  const int koff = ks * RPL + ((ks * RPL) >> 5) * 4;    // padded offset of this lane's rows in sq / sk

  const size_t q_off = (size_t)kh * DK, k_off = (size_t)p.G * DK + (size_t)kh * DK;
  const size_t v_off = (size_t)2 * p.G * DK + (size_t)h * DV + sl * SLICE;

  for (int c0 = s0; c0 < s1; c0 += TCH) {
    const int n = min(TCH, s1 - c0);
    __syncthreads();
    for (int i = tid; i < n * (DK / 4); i += NT) {
      const int tt = i / (DK / 4), d4 = (i % (DK / 4)) * 4;
      const float* row = p.qkv + (size_t)(c0 + tt) * p.C;
      const int dst = d4 + (d4 >> 5) * 4;
      *reinterpret_cast<float4*>(&sq[tt][dst]) = *reinterpret_cast<const float4*>(row + q_off + d4);
      *reinterpret_cast<float4*>(&sk[tt][dst]) = *reinterpret_cast<const float4*>(row + k_off + d4);
    }
    for (int i = tid; i < n * SLICE; i += NT) {
      const int tt = i / SLICE, d = i % SLICE;
      sv[tt][d] = p.qkv[(size_t)(c0 + tt) * p.C + v_off + d];
    }
    if (tid < n) {
      sdec[tid] = p.decay[(size_t)(c0 + tid) * p.Hv + h];
      sbeta[tid] = p.beta[(size_t)(c0 + tid) * p.Hv + h];
    }
    __syncthreads();
    for (int tt = 0; tt < n; ++tt) {
      const float dec = sdec[tt], bet = sbeta[tt];
      float kr[RPL];
#pragma unroll
      for (int i4 = 0; i4 < RPL / 4; ++i4) {
        const float4 kv4 = *reinterpret_cast<const float4*>(&sk[tt][koff + i4 * 4]);
        kr[i4 * 4] = kv4.x; kr[i4 * 4 + 1] = kv4.y; kr[i4 * 4 + 2] = kv4.z; kr[i4 * 4 + 3] = kv4.w;
      }
      // four independent partial sums per reduction keep the FMA pipe busy (the chains are otherwise serial)
      float kv4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        S[i] *= dec;
        kv4[i & 3] += kr[i] * S[i];
      }
      float kv = (kv4[0] + kv4[1]) + (kv4[2] + kv4[3]);
#pragma unroll
      for (int o = 1; o < LPC; o <<= 1) kv += __shfl_xor_sync(0xffffffffu, kv, o);
      const float delta = (sv[tt][cw] - kv) * bet;
      float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i4 = 0; i4 < RPL / 4; ++i4) {
        const float4 q4 = *reinterpret_cast<const float4*>(&sq[tt][koff + i4 * 4]);
        S[i4 * 4] += kr[i4 * 4] * delta;         o4[0] += q4.x * S[i4 * 4];
        S[i4 * 4 + 1] += kr[i4 * 4 + 1] * delta; o4[1] += q4.y * S[i4 * 4 + 1];
        S[i4 * 4 + 2] += kr[i4 * 4 + 2] * delta; o4[2] += q4.z * S[i4 * 4 + 2];
        S[i4 * 4 + 3] += kr[i4 * 4 + 3] * delta; o4[3] += q4.w * S[i4 * 4 + 3];
      }
      float o = (o4[0] + o4[1]) + (o4[2] + o4[3]);
#pragma unroll
      for (int of = 1; of < LPC; of <<= 1) o += __shfl_xor_sync(0xffffffffu, o, of);
      if (ks == 0) p.out[((size_t)(c0 + tt) * p.Hv + h) * DV + col] = o;
      if (p.journal != nullptr) {
        float* J = p.journal + (((size_t)(c0 + tt) * p.Hv + h) * DK) * DV;
#pragma unroll
        for (int i = 0; i < RPL; ++i) J[(size_t)(ks * RPL + i) * DV + col] = S[i];
      }
    }
  }
  if (p.write_state) {
#pragma unroll
    for (int i = 0; i < RPL; ++i) Sg[(size_t)(ks * RPL + i) * DV + col] = S[i];
  }
}

// out[t][h][:] = RMSNorm(o[t][h][:]) * w * SiLU(z[t][h][:])  -> bf16.  One warp per (t, h).
__global__ void gdn_gated_norm_kernel(const float* __restrict__ o, const void* __restrict__ z, int z_dtype,
                                      long long z_stride, const float* __restrict__ w,
                                      __nv_bfloat16* __restrict__ out, long long out_stride, int T, int Hv, int Dv,
                                      float eps) {
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= (long long)T * Hv) return;
  const int t = (int)(gw / Hv), h = (int)(gw % Hv);
  const float* orow = o + ((size_t)t * Hv + h) * Dv;
  float ss = 0.f;
  for (int i = lane; i < Dv; i += 32) ss += orow[i] * orow[i];
  ss = warp_sum(ss);
  const float inv = rsqrtf(ss / (float)Dv + eps);
  for (int i = lane; i < Dv; i += 32) {
    const size_t zi = (size_t)t * z_stride + (size_t)h * Dv + i;
    const float zv = z_dtype == 0 ? reinterpret_cast<const float*>(z)[zi]
                                  : bf16_to_f32(reinterpret_cast<const __nv_bfloat16*>(z)[zi]);
    out[(size_t)t * out_stride + (size_t)h * Dv + i] = f32_to_bf16(orow[i] * inv * w[i] * silu_f(zv));
  }
}

// The same for heads of 128 columns, 16-byte aligned: four columns a lane, one load each of the output and the gate
// (128 bytes apart per lane and four passes before: 94 us at 4096 x 48 heads, 47 us now; 200 MB).
__global__ void __launch_bounds__(256) gdn_gated_norm128_kernel(const float* __restrict__ o, const void* __restrict__ z,
                                                                int z_dtype, long long z_stride,
                                                                const float* __restrict__ w,
                                                                __nv_bfloat16* __restrict__ out, long long out_stride,
                                                                int T, int Hv, float eps) {
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= (long long)T * Hv) return;
  const int t = (int)(gw / Hv), h = (int)(gw % Hv);
  const float4 v = *reinterpret_cast<const float4*>(o + (size_t)gw * 128 + lane * 4);
  const size_t zi = (size_t)t * z_stride + (size_t)h * 128 + lane * 4;
  float4 g;
  if (z_dtype == 0) {
    g = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(z) + zi);
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(z) + zi);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    g = make_float4(a.x, a.y, b.x, b.y);
  }
  const float4 wv = *reinterpret_cast<const float4*>(w + lane * 4);
  const float ss = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
  const float inv = rsqrtf(ss / 128.f + eps);
  __nv_bfloat162 r[2] = {__floats2bfloat162_rn(v.x * inv * wv.x * silu_f(g.x), v.y * inv * wv.y * silu_f(g.y)),
                         __floats2bfloat162_rn(v.z * inv * wv.z * silu_f(g.z), v.w * inv * wv.w * silu_f(g.w))};
  *reinterpret_cast<uint2*>(out + (size_t)t * out_stride + (size_t)h * 128 + lane * 4) = *reinterpret_cast<const uint2*>(r);
}

// ---------------------------------------------------------------------------------------------- prompt front end
// Everything between the projections and the scan of a prompt portion in one pass: convolution of four taps + SiLU with
// the rolling window in registers (a row is read once, not four times), L2 norm of the q / k heads, the new window, and the
// gates.  A warp owns the 128 channels of one head for FRONT_TOK tokens of one segment, four channels a lane.  Three
// kernels before (convolution 137 us, window 18 us, norm and gates 30 us at 4096 x 10240), 82 us now; 252 MB.
// The warp of a segment's first tokens is the only reader of the old window and therefore the writer of the new one.
struct GdnFrontArgs {
  const void* x;          // [T][x_stride] projections q | k | v, fp32 or bf16
  int in_dtype;
  long long x_stride;
  const float* w;         // [C][4]
  float* conv_state;      // [n_slots][C][3], oldest first
  const int* seg_start;   // [n_seg + 1]
  const int* seg_slot;    // [n_seg]
  float* out;             // [T][C]
  const float* a;
  const float* b;
  long long a_stride, b_stride;
  const float* ssm_a;
  const float* dt_bias;
  float* decay;           // [T][Hv]
  float* beta;            // [T][Hv]
  int C, G, Hv, T, n_seg;
};

constexpr int FRONT_TOK = 16;

__device__ __forceinline__ float4 front_load(const GdnFrontArgs& p, int t, int c) {
  const size_t i = (size_t)t * p.x_stride + c;
  if (p.in_dtype == 0) return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.x) + i);
  const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.x) + i);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// grid (token groups of all segments, ceil(heads / 8)), block 256
__global__ void __launch_bounds__(256) gdn_front_kernel(const GdnFrontArgs p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int sg = 0, grp = blockIdx.x;
  for (; sg < p.n_seg; ++sg) {
    const int n = (p.seg_start[sg + 1] - p.seg_start[sg] + FRONT_TOK - 1) / FRONT_TOK;
    if (grp < n) break;
    grp -= n;
  }
  if (sg == p.n_seg) return;
  const int s0 = p.seg_start[sg], s1 = p.seg_start[sg + 1], t0 = s0 + grp * FRONT_TOK, t1 = min(s1, t0 + FRONT_TOK);
  if (blockIdx.y == 0) {
    for (int i = threadIdx.x; i < (t1 - t0) * p.Hv; i += 256) {
      const int t = t0 + i / p.Hv, h = i % p.Hv;
      const float av = p.a[(size_t)t * p.a_stride + h], bv = p.b[(size_t)t * p.b_stride + h];
      p.beta[(size_t)t * p.Hv + h] = sigmoid_f(bv);
      p.decay[(size_t)t * p.Hv + h] = __expf(p.ssm_a[h] * softplus20_f(av + p.dt_bias[h]));
    }
  }
  const int head = blockIdx.y * 8 + warp, c = head * 128 + lane * 4;
  if (c >= p.C) return;
  float4 w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) w[e] = __ldg(reinterpret_cast<const float4*>(p.w + (size_t)(c + e) * 4));
  float4 x0, x1, x2;                                     // the three inputs before token t, oldest first
  if (grp == 0) {
    float* st = p.conv_state + ((size_t)p.seg_slot[sg] * p.C + c) * 3;
    float4 q[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) q[i] = reinterpret_cast<const float4*>(st)[i];
    x0 = make_float4(q[0].x, q[0].w, q[1].z, q[2].y);
    x1 = make_float4(q[0].y, q[1].x, q[1].w, q[2].z);
    x2 = make_float4(q[0].z, q[1].y, q[2].x, q[2].w);
    const int n = s1 - s0;
    const float4 n0 = n >= 3 ? front_load(p, s1 - 3, c) : (n == 2 ? x2 : x1);
    const float4 n1 = n >= 2 ? front_load(p, s1 - 2, c) : x2;
    const float4 n2 = front_load(p, s1 - 1, c);
    reinterpret_cast<float4*>(st)[0] = make_float4(n0.x, n1.x, n2.x, n0.y);
    reinterpret_cast<float4*>(st)[1] = make_float4(n1.y, n2.y, n0.z, n1.z);
    reinterpret_cast<float4*>(st)[2] = make_float4(n2.z, n0.w, n1.w, n2.w);
  } else {
    x0 = front_load(p, t0 - 3, c);
    x1 = front_load(p, t0 - 2, c);
    x2 = front_load(p, t0 - 1, c);
  }
  const bool unit = head < 2 * p.G;
  const float qscale = head < p.G ? rsqrtf(128.f) : 1.f;
  for (int t = t0; t < t1; t += 4) {
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = t + i < t1 ? front_load(p, t + i, c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 x3 = v[i];
      float4 y;
      y.x = silu_f(x0.x * w[0].x + x1.x * w[0].y + x2.x * w[0].z + x3.x * w[0].w);
      y.y = silu_f(x0.y * w[1].x + x1.y * w[1].y + x2.y * w[1].z + x3.y * w[1].w);
      y.z = silu_f(x0.z * w[2].x + x1.z * w[2].y + x2.z * w[2].z + x3.z * w[2].w);
      y.w = silu_f(x0.w * w[3].x + x1.w * w[3].y + x2.w * w[3].z + x3.w * w[3].w);
      if (unit) {
        const float ss = warp_sum(y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w);
        const float inv = qscale / fmaxf(sqrtf(ss), 1e-6f);
        y.x *= inv; y.y *= inv; y.z *= inv; y.w *= inv;
      }
      if (t + i < t1) *reinterpret_cast<float4*>(p.out + (size_t)(t + i) * p.C + c) = y;
      x0 = x1;
      x1 = x2;
      x2 = x3;
    }
  }
}

// Copy one journalled state row into the canonical slot (speculative commit): dst[slot] = journal[row].
__global__ void gdn_commit_kernel(float* __restrict__ state, const float* __restrict__ journal,
                                  const int* __restrict__ seg_slot, const int* __restrict__ commit_row,
                                  long long per_slot) {
  const int sg = blockIdx.y;
  const int row = commit_row[sg];
  if (row < 0) return;
  const float4* src = reinterpret_cast<const float4*>(journal + (size_t)row * per_slot);
  float4* dst = reinterpret_cast<float4*>(state + (size_t)seg_slot[sg] * per_slot);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < per_slot / 4;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// ---------------------------------------------------------------------------------------------- decode fast path
// For single-token segments (plain decode) the five kernels conv -> conv state -> prepare -> scan -> gated norm
// collapse into two launches; a decode step is bound by launch latency, not by this arithmetic.
struct GdnDecodeArgs {
  const float* x;         // [R][x_stride] pre-conv projections q | k | v (fp32)
  long long x_stride;
  const float* conv_w;    // [C][4]
  float* conv_state;      // [n_slots][C][3]
  const float* a;         // [R][a_stride]
  const float* b;         // [R][b_stride]
  long long a_stride, b_stride;
  const float* ssm_a;     // [Hv]
  const float* dt_bias;   // [Hv]
  const int* slot;        // [R]
  float* qkv;             // [R][C] conv output (q, k normalised)
  float* decay;           // [R][Hv]
  float* beta;            // [R][Hv]
  float* state;           // [n_slots][Hv][128][128]
  const void* z;          // [R][z_stride] gate input
  int z_dtype;
  long long z_stride;
  const float* norm_w;    // [128]
  __nv_bfloat16* out;     // [R][out_stride]
  long long out_stride;
  float eps;
  int C, G, Hv, R;
  // one row, gates from the residual (gate_w non-null; then a and b are not read): alpha and beta rows of all heads
  // [2 Hv][K] fp32, the residual row [K] fp32 and the norm in front of them
  const float* gate_w;
  const float* gate_x;
  const float* gate_norm;
  float gate_eps;
  int K;
};

// Alpha and beta of one head and their gates, in fp32, by a block of 128 threads: the two weight rows are requested ahead
// of the predecessor's end.  As a product of their own (two 48-row weights, 8-bit) they cost a launch of ~5 us per layer.
__device__ __forceinline__ void gate_block(const GdnDecodeArgs& p, int h, float* red) {
  constexpr int KEEP = 12;                     // float4 per thread and row: 6144 columns; the rest is loaded in place
  const int n4 = p.K >> 2, tid = threadIdx.x;
  const float4* wa = reinterpret_cast<const float4*>(p.gate_w + (size_t)h * p.K);
  const float4* wb = reinterpret_cast<const float4*>(p.gate_w + (size_t)(p.Hv + h) * p.K);
  const float4* nw = reinterpret_cast<const float4*>(p.gate_norm);
  float4 a[KEEP], b[KEEP];
#pragma unroll
  for (int i = 0; i < KEEP; ++i)
    if (i * 128 + tid < n4) {
      const float4 m = __ldg(nw + i * 128 + tid);
      a[i] = __ldg(wa + i * 128 + tid);
      b[i] = __ldg(wb + i * 128 + tid);
      a[i] = make_float4(a[i].x * m.x, a[i].y * m.y, a[i].z * m.z, a[i].w * m.w);
      b[i] = make_float4(b[i].x * m.x, b[i].y * m.y, b[i].z * m.z, b[i].w * m.w);
    }
  pdl_wait();
  pdl_launch();
  const float4* x = reinterpret_cast<const float4*>(p.gate_x);
  float ss = 0.f, da = 0.f, db = 0.f;
  const auto add = [&](const float4& v, const float4& fa, const float4& fb) {
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    da += v.x * fa.x + v.y * fa.y + v.z * fa.z + v.w * fa.w;
    db += v.x * fb.x + v.y * fb.y + v.z * fb.z + v.w * fb.w;
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i)
    if (i * 128 + tid < n4) add(x[i * 128 + tid], a[i], b[i]);
  for (int i = KEEP * 128 + tid; i < n4; i += 128) {
    const float4 m = __ldg(nw + i), fa = __ldg(wa + i), fb = __ldg(wb + i);
    add(x[i], make_float4(fa.x * m.x, fa.y * m.y, fa.z * m.z, fa.w * m.w),
        make_float4(fb.x * m.x, fb.y * m.y, fb.z * m.z, fb.w * m.w));
  }
  ss = warp_sum(ss);
  da = warp_sum(da);
  db = warp_sum(db);
  if ((tid & 31) == 0) {
    red[tid >> 5] = ss;
    red[4 + (tid >> 5)] = da;
    red[8 + (tid >> 5)] = db;
  }
  __syncthreads();
  if (tid == 0) {
    const float inv = rsqrtf(((red[0] + red[1]) + (red[2] + red[3])) / (float)p.K + p.gate_eps);
    const float av = ((red[4] + red[5]) + (red[6] + red[7])) * inv, bv = ((red[8] + red[9]) + (red[10] + red[11])) * inv;
    p.beta[h] = sigmoid_f(bv);
    p.decay[h] = __expf(p.ssm_a[h] * softplus20_f(av + p.dt_bias[h]));
  }
}

// grid (C/128 [+ Hv], R), block 128: one channel per thread.  conv(k=4)+SiLU, rolling state shift, L2 norm of q/k heads,
// and (block 0, or Hv blocks of their own) the decay / beta gates of the row.
__global__ void __launch_bounds__(128) gdn_decode_pre_kernel(const GdnDecodeArgs p) {
  __shared__ float red[32];
  if ((int)blockIdx.x >= p.C / 128) {
    gate_block(p, (int)blockIdx.x - p.C / 128, red);
    return;
  }
  pdl_wait();
  pdl_launch();
  const int r = blockIdx.y, blk = blockIdx.x, c = blk * 128 + threadIdx.x;
  float* st = p.conv_state + ((size_t)p.slot[r] * p.C + c) * 3;
  const float4 w = __ldg(reinterpret_cast<const float4*>(p.conv_w + (size_t)c * 4));
  const float xv = p.x[(size_t)r * p.x_stride + c];
  const float s0 = st[0], s1 = st[1], s2 = st[2];
  float y = silu_f(w.x * s0 + w.y * s1 + w.z * s2 + w.w * xv);
  st[0] = s1; st[1] = s2; st[2] = xv;
  if (blk < 2 * p.G) {
    const float ss = block_sum(y * y, red);
    float inv = 1.f / fmaxf(sqrtf(ss), 1e-6f);
    if (blk < p.G) inv *= rsqrtf(128.f);
    y *= inv;
  }
  p.qkv[(size_t)r * p.C + c] = y;
  if (blk == 0 && p.gate_w == nullptr) {
    for (int h = threadIdx.x; h < p.Hv; h += 128) {
      const float av = p.a[(size_t)r * p.a_stride + h], bv = p.b[(size_t)r * p.b_stride + h];
      p.beta[(size_t)r * p.Hv + h] = sigmoid_f(bv);
      p.decay[(size_t)r * p.Hv + h] = __expf(p.ssm_a[h] * softplus20_f(av + p.dt_bias[h]));
    }
  }
}

// grid (Hv, R), block 512: thread (ks = tid / 128, col = tid % 128) owns rows ks*32..+31 of one column of S, so that a
// warp's access covers whole 128-byte lines of the state; the four partial sums of a column meet in shared memory.
// One recurrent step, then RMSNorm over the head's 128 outputs * w * SiLU(z) -> bf16.
// Bound by the state (read and written once, 128 KB per head and row).
__global__ void __launch_bounds__(512, 2) gdn_decode_step_kernel(const GdnDecodeArgs p) {
  __shared__ __align__(16) float sq[DK];
  __shared__ __align__(16) float sk[DK];
  __shared__ float part[2][4][DV];
  __shared__ float red[4];
  const int h = blockIdx.x, r = blockIdx.y, tid = threadIdx.x;
  const int col = tid & 127, ks = tid >> 7;
  const int kh = h % p.G;
  const float* row = p.qkv + (size_t)r * p.C;
  pdl_wait();
  pdl_launch();
  float* Sg = p.state + (((size_t)p.slot[r] * p.Hv + h) * DK + ks * 32) * DV + col;
  float S[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) S[i] = Sg[(size_t)i * DV];
  if (ks == 0) sq[col] = row[(size_t)kh * DK + col];
  if (ks == 1) sk[col] = row[(size_t)p.G * DK + (size_t)kh * DK + col];
  const float v = row[(size_t)2 * p.G * DK + (size_t)h * DV + col];
  const float dec = p.decay[(size_t)r * p.Hv + h], bet = p.beta[(size_t)r * p.Hv + h];
  __syncthreads();
  float kv4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i4 = 0; i4 < 8; ++i4) {
    const float4 k4 = *reinterpret_cast<const float4*>(&sk[ks * 32 + i4 * 4]);
    S[i4 * 4] *= dec;     kv4[0] += k4.x * S[i4 * 4];
    S[i4 * 4 + 1] *= dec; kv4[1] += k4.y * S[i4 * 4 + 1];
    S[i4 * 4 + 2] *= dec; kv4[2] += k4.z * S[i4 * 4 + 2];
    S[i4 * 4 + 3] *= dec; kv4[3] += k4.w * S[i4 * 4 + 3];
  }
  part[0][ks][col] = (kv4[0] + kv4[1]) + (kv4[2] + kv4[3]);
  __syncthreads();
  const float kv = (part[0][0][col] + part[0][1][col]) + (part[0][2][col] + part[0][3][col]);
  const float delta = (v - kv) * bet;
  float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i4 = 0; i4 < 8; ++i4) {
    const float4 k4 = *reinterpret_cast<const float4*>(&sk[ks * 32 + i4 * 4]);
    const float4 q4 = *reinterpret_cast<const float4*>(&sq[ks * 32 + i4 * 4]);
    S[i4 * 4] += k4.x * delta;     o4[0] += q4.x * S[i4 * 4];
    S[i4 * 4 + 1] += k4.y * delta; o4[1] += q4.y * S[i4 * 4 + 1];
    S[i4 * 4 + 2] += k4.z * delta; o4[2] += q4.z * S[i4 * 4 + 2];
    S[i4 * 4 + 3] += k4.w * delta; o4[3] += q4.w * S[i4 * 4 + 3];
  }
  part[1][ks][col] = (o4[0] + o4[1]) + (o4[2] + o4[3]);
#pragma unroll
  for (int i = 0; i < 32; ++i) Sg[(size_t)i * DV] = S[i];
  __syncthreads();
  if (ks != 0) return;
  const float o = (part[1][0][col] + part[1][1][col]) + (part[1][2][col] + part[1][3][col]);
  const float sw = warp_sum(o * o);
  if ((tid & 31) == 0) red[tid >> 5] = sw;
  asm volatile("bar.sync 1, 128;" ::: "memory");
  const float inv = rsqrtf(((red[0] + red[1]) + (red[2] + red[3])) / (float)DV + p.eps);
  const size_t zi = (size_t)r * p.z_stride + (size_t)h * DV + col;
  const float zv = p.z_dtype == 0 ? reinterpret_cast<const float*>(p.z)[zi]
                                  : bf16_to_f32(reinterpret_cast<const __nv_bfloat16*>(p.z)[zi]);
  p.out[(size_t)r * p.out_stride + (size_t)h * DV + col] = f32_to_bf16(o * inv * p.norm_w[col] * silu_f(zv));
}

}  // namespace

HE_API int he_gdn_prepare(const GdnPrepArgs* args, cudaStream_t stream) {
  if (args->T <= 0) return 0;
  gdn_prepare_kernel<<<args->T, 256, 0, stream>>>(*args);
  HE_LAUNCH_CHECK();
  return 0;
}
HE_API int he_gdn_prep_args_size() { return (int)sizeof(GdnPrepArgs); }

// Prompt front end (state size 128, four taps, no journal): see GdnFrontArgs.
HE_API int he_gdn_front(const GdnFrontArgs* args, cudaStream_t stream) {
  const GdnFrontArgs& a = *args;
  if (a.T <= 0 || a.n_seg <= 0) return 0;
  const int es = a.in_dtype == 0 ? 4 : 2;
  if (a.C != 2 * a.G * 128 + a.Hv * 128 || (reinterpret_cast<uintptr_t>(a.x) & 15) != 0 || (a.x_stride * es) % 8 != 0 ||
      (a.in_dtype == 0 && a.x_stride % 4 != 0) ||
      ((reinterpret_cast<uintptr_t>(a.conv_state) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.out)) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  gdn_front_kernel<<<dim3(a.T / FRONT_TOK + a.n_seg, (a.C / 128 + 7) / 8), 256, 0, stream>>>(a);
  HE_LAUNCH_CHECK();
  return 0;
}
HE_API int he_gdn_front_args_size() { return (int)sizeof(GdnFrontArgs); }

HE_API int he_gdn_scan(const GdnScanArgs* args, cudaStream_t stream) {
  if (args->T <= 0 || args->n_seg <= 0) return 0;
  dim3 grid(args->n_seg, args->Hv, DV / SLICE);
  // few (segment, head) pairs and long segments: spread every column over 8 lanes to double the resident warps
  const bool wide = (long long)args->n_seg * args->Hv * (DV / SLICE) <= 1024 && args->T >= 64 * args->n_seg;
  if (wide) gdn_scan_kernel<8><<<grid, 256, 0, stream>>>(*args);
  else gdn_scan_kernel<4><<<grid, 128, 0, stream>>>(*args);
  HE_LAUNCH_CHECK();
  return 0;
}
HE_API int he_gdn_scan_args_size() { return (int)sizeof(GdnScanArgs); }

HE_API int he_gdn_gated_norm(const void* o, const void* z, int z_dtype, long long z_stride, const void* w, void* out,
                             long long out_stride, int T, int Hv, int Dv, float eps, cudaStream_t stream) {
  if (T <= 0) return 0;
  const long long warps = (long long)T * Hv;
  const int zs = z_dtype == 0 ? 4 : 2;
  if (Dv == 128 && (reinterpret_cast<uintptr_t>(o) & 15) == 0 && (reinterpret_cast<uintptr_t>(z) & 15) == 0 &&
      (z_stride * zs) % 16 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0 && out_stride % 4 == 0 &&
      (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
    gdn_gated_norm128_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, stream>>>(
        (const float*)o, z, z_dtype, z_stride, (const float*)w, (__nv_bfloat16*)out, out_stride, T, Hv, eps);
    HE_LAUNCH_CHECK();
    return 0;
  }
  gdn_gated_norm_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, stream>>>(
      (const float*)o, z, z_dtype, z_stride, (const float*)w, (__nv_bfloat16*)out, out_stride, T, Hv, Dv, eps);
  HE_LAUNCH_CHECK();
  return 0;
}

// state[seg_slot[s]] = journal[commit_row[s]] for each segment s with commit_row[s] >= 0.
// per_slot = floats per slot (Hv*Dk*Dv for GDN state, C*(KW-1) for conv state); must be a multiple of 4.
HE_API int he_state_commit(void* state, const void* journal, const void* seg_slot, const void* commit_row, int n_seg,
                           long long per_slot, cudaStream_t stream) {
  if (n_seg <= 0) return 0;
  if (per_slot % 4 != 0) return -HE_ERR_BAD_ARG;
  dim3 grid(64, n_seg);
  gdn_commit_kernel<<<grid, 256, 0, stream>>>((float*)state, (const float*)journal, (const int*)seg_slot,
                                              (const int*)commit_row, per_slot);
  HE_LAUNCH_CHECK();
  return 0;
}

// Decode fast path (every row is a single-token segment, no journal): conv + gates + one scan step + gated norm
// in two launches.  Requires state size 128, conv kernel 4, C % 128 == 0.
HE_API int he_gdn_decode(const GdnDecodeArgs* args, cudaStream_t stream) {
  const GdnDecodeArgs& a = *args;
  if (a.R <= 0) return 0;
  if (a.C % 128 != 0 || a.C != 2 * a.G * 128 + a.Hv * 128 || a.Hv % a.G != 0) return -HE_ERR_BAD_ARG;
  if (a.gate_w != nullptr && (a.R != 1 || a.K <= 0 || a.K % 4 != 0 || a.gate_x == nullptr || a.gate_norm == nullptr ||
                              ((reinterpret_cast<uintptr_t>(a.gate_w) | reinterpret_cast<uintptr_t>(a.gate_x) |
                                reinterpret_cast<uintptr_t>(a.gate_norm)) & 15) != 0))
    return -HE_ERR_BAD_ARG;
  const int gates = a.gate_w != nullptr ? a.Hv : 0;
  cudaError_t e = launch_pdl(gdn_decode_pre_kernel, dim3(a.C / 128 + gates, a.R), dim3(128), 0, stream, a);
  if (e != cudaSuccess) return (int)e;
  e = launch_pdl(gdn_decode_step_kernel, dim3(a.Hv, a.R), dim3(512), 0, stream, a);
  if (e != cudaSuccess) return (int)e;
  return 0;
}
HE_API int he_gdn_decode_args_size() { return (int)sizeof(GdnDecodeArgs); }
