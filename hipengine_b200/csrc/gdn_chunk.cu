// Gated DeltaNet prefill scan in chunked (WY) form on the tensor cores, split into a parallel and a serial kernel.
//
// The recurrence  S_t = g_t S_{t-1} + k_t d_t^T,  d_t = beta_t (v_t - (g_t S_{t-1})^T k_t),  o_t = S_t^T q_t
// (hipengine/kernels/cpu_reference/ops.py:1967-2012; chunked algebra oracle :2015-2141) is evaluated 32 tokens at
// a time.  With G_t = prod_{s<=t} g_s inside the chunk (kept as log-sums, ratios G_t/G_j <= 1 for j <= t):
//     A_tj = beta_t (G_t/G_j)(k_t.k_j), j < t          (strictly lower 32x32)
//     [U | W] = (I + A)^-1 [beta*V | beta*G*K]
//     D = U - W S_0                                     (the 32 delta rows)
//     O = G*(Q S_0) + P D,  P_tj = (G_t/G_j)(q_t.k_j), j <= t
//     S_32 = G_32 S_0 + Kt^T D,  Kt_j = (G_32/G_j) k_j
// Everything but the last three lines does not depend on the state.  One kernel with all of it in the loop over the
// chunks (16 tokens each) was a chain of 256 steps of 3.7 us for 4096 tokens -- products too small to fill anything,
// and an inverse, between barriers.  So:
//   gdn_prepare_chunks : one CTA per (chunk, V head), all chunks at once: W, U, P and the log-sums to a workspace
//   gdn_chain          : one CTA per (segment, V head, 32 or 64 columns of the state), the chunks in order: three products per
//                        step, the state in registers, the next chunk's operands in flight (cp.async)
// The chain is bound by latency: dependent products and conversions, operands from shared memory, two barriers per step, on the
// 96 SMs that 48 heads fill (issue 42 %, shared memory 41 %, tensor pipe 26 %, L2 2.8 TB/s); a step needs 56 KB from L2 per CTA of
// 32 columns, 60 KB of 64.  32 tokens per chunk halve the steps of 16 and keep the inverse cheap.  (64 were not built: the same
// bytes per token and an inverse of eight times the work.)  Measured on B200, 4096 tokens: 48 heads 585 us (147 + 438) against
// 938 us, 2048 tokens x 32 heads 207 us (54 + 153) against 395 us.
// All products run as mma.sync m16n8k8 TF32 with rounded operands (fp32 accumulate).  Used for prefill segments without a
// state journal; decode rows, verify chains and short segments keep the serial kernel in gdn.cu.  V head h reads K head
// h % G (GGUF order).
#include "common.cuh"

using namespace he;

namespace {

constexpr int CK = 32;          // tokens per chunk
constexpr int DK = 128;         // state rows (key dim) and columns
constexpr int LDK = DK + 16;    // row stride (floats) of K / Q / W / transposed S: conflict-free 128-bit fragment reads
constexpr int LDV = DK + 8;     // row stride of V
constexpr int LDA = CK + 4;     // row stride of the 32 x 32 matrices

// workspace of one (chunk, head), in floats
constexpr int WS_W = 0, WS_U = WS_W + CK * DK, WS_P = WS_U + CK * DK, WS_B = WS_P + CK * CK, WS_UNIT = WS_B + CK;

// Fragment convention for the 128-deep products: the k index is relabelled so that the four k values a lane feeds into
// two consecutive m16n8k8 steps are contiguous in memory (one 128-bit load); A and B use the same relabelling.
struct GdnChunkArgs {
  const float* qkv;       // [T][C] prepared conv output: q | k | v (q, k normalised)
  const float* decay;     // [T][Hv]
  const float* beta;      // [T][Hv]
  float* state;           // [n_slots][Hv][128][128]
  const int* seg_start;   // [n_seg+1]
  const int* seg_slot;    // [n_seg]
  float* out;             // [T][Hv][128]
  int C, G, Hv, T, n_seg;
  int write_state;
  float* ws;              // he_gdn_chunk_ws_floats
  long long ws_floats;
  int longest;            // tokens of the longest segment, or 0 where the caller does not know it
  int c_lo, c_hi;         // chunks [c_lo, c_hi) of every segment (set by the launcher)
};

__device__ __forceinline__ float rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
__device__ __forceinline__ uint32_t tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ float4 ld4f(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ uint4 ld4r(const float* p) {      // rounded operands
  const float4 v = ld4f(p);
  return make_uint4(tf32(v.x), tf32(v.y), tf32(v.z), tf32(v.w));
}
__device__ __forceinline__ uint4 ld4u(const float* p) { return *reinterpret_cast<const uint4*>(p); }   // stored rounded

// First workspace unit of a segment's window: the windows of the segments before it come first.
__device__ __forceinline__ int window(const GdnChunkArgs& p, int s) {
  const int n = (p.seg_start[s + 1] - p.seg_start[s] + CK - 1) / CK;
  return max(0, min(n, p.c_hi) - p.c_lo);
}

struct PrepSmem {
  float K[CK][LDK];
  float Q[CK][LDK];
  float V[CK][LDV];
  float A[CK][LDA];        // strictly lower
  float T[CK][LDA];        // (I + A)^-1
  float L[16][20];         // L21 T11
  float b[CK], bt[CK];
};

// grid (chunks of all windows, Hv), block 128
__global__ void __launch_bounds__(128) gdn_prepare_chunks_kernel(const GdnChunkArgs p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  PrepSmem& sm = *reinterpret_cast<PrepSmem*>(smem_raw);
  const int h = blockIdx.y, kh = h % p.G, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  int sg = 0, c = blockIdx.x;
  for (; sg < p.n_seg; ++sg) {
    const int n = window(p, sg);
    if (c < n) break;
    c -= n;
  }
  if (sg == p.n_seg) return;
  const int s1 = p.seg_start[sg + 1], t0 = p.seg_start[sg] + (p.c_lo + c) * CK;
  float* ws = p.ws + ((size_t)blockIdx.x * p.Hv + h) * WS_UNIT;

  for (int i = tid; i < CK * (DK / 4); i += 128) {
    const int tt = i / (DK / 4), d4 = (i % (DK / 4)) * 4;
    const bool ok = t0 + tt < s1;
    const float* row = p.qkv + (size_t)(ok ? t0 + tt : t0) * p.C;
    cp_async16(&sm.K[tt][d4], row + (size_t)p.G * DK + (size_t)kh * DK + d4, ok ? 16 : 0);
    cp_async16(&sm.Q[tt][d4], row + (size_t)kh * DK + d4, ok ? 16 : 0);
    cp_async16(&sm.V[tt][d4], row + (size_t)2 * p.G * DK + (size_t)h * DK + d4, ok ? 16 : 0);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (warp == 0) {         // tokens past the segment's end are identity steps (decay 1, beta 0)
    const bool ok = t0 + lane < s1;
    float lg = ok ? __logf(fmaxf(p.decay[(size_t)(t0 + lane) * p.Hv + h], 1e-37f)) : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, lg, o);
      if (lane >= o) lg += v;
    }
    sm.b[lane] = lg;
    sm.bt[lane] = ok ? p.beta[(size_t)(t0 + lane) * p.Hv + h] : 0.f;
    ws[WS_B + lane] = lg;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // warps 0, 1: K K^T (rows 16w .. +15), warps 2, 3: Q K^T; tiles above the diagonal are zero
  {
    const int m0 = (warp & 1) * 16;
    const float (*X)[LDK] = warp < 2 ? sm.K : sm.Q;
    float c4[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) c4[n][0] = c4[n][1] = c4[n][2] = c4[n][3] = 0.f;
    const int nt = m0 == 0 ? 2 : 4;
#pragma unroll 4
    for (int kk = 0; kk < DK; kk += 16) {
      const uint4 lo = ld4r(&X[m0 + g][kk + 4 * t]), hi = ld4r(&X[m0 + g + 8][kk + 4 * t]);
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (n < nt) {
          const uint4 bb = ld4r(&sm.K[n * 8 + g][kk + 4 * t]);
          mma_tf32(c4[n], lo.x, hi.x, lo.y, hi.y, bb.x, bb.y);
          mma_tf32(c4[n], lo.z, hi.z, lo.w, hi.w, bb.z, bb.w);
        }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = m0 + g + (e >> 1) * 8, j = n * 8 + 2 * t + (e & 1);
        const float r = j <= i ? __expf(sm.b[i] - sm.b[j]) * c4[n][e] : 0.f;
        if (warp < 2) sm.A[i][j] = j < i ? sm.bt[i] * r : 0.f;
        else ws[WS_P + i * CK + j] = rna(r);
      }
  }
  __syncthreads();
  // (I + A)^-1 by halves: both 16 x 16 diagonal blocks by forward substitution (lane = column; lanes 16.. the second)
  if (warp == 0) {
    const int o = lane & 16, cl = lane & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float r = i == cl ? 1.f : 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) r -= sm.A[o + i][o + m] * x[m];
      x[i] = r;
      sm.T[o + i][o + cl] = r;
      sm.T[i][16 + cl] = 0.f;
    }
  }
  __syncthreads();
  // ... and T21 = -T22 (A21 T11)
  for (int e = tid; e < 256; e += 128) {
    const int i = e >> 4, j = e & 15;
    float r = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) r += sm.A[16 + i][m] * sm.T[m][j];
    sm.L[i][j] = r;
  }
  __syncthreads();
  for (int e = tid; e < 256; e += 128) {
    const int i = e >> 4, j = e & 15;
    float r = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) r += sm.T[16 + i][16 + m] * sm.L[m][j];
    sm.T[16 + i][j] = -r;
  }
  __syncthreads();
  // [W | U] = T [beta G K | beta V]: warps 0, 1 -> W, 2, 3 -> U, 64 columns each
  {
    const bool is_w = warp < 2;
    const int c0 = (warp & 1) * 64;
    uint32_t ta[2][4][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        ta[m][ks][0] = tf32(sm.T[m * 16 + g][ks * 8 + t]);
        ta[m][ks][1] = tf32(sm.T[m * 16 + g + 8][ks * 8 + t]);
        ta[m][ks][2] = tf32(sm.T[m * 16 + g][ks * 8 + t + 4]);
        ta[m][ks][3] = tf32(sm.T[m * 16 + g + 8][ks * 8 + t + 4]);
      }
    float sc[4][2];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j = ks * 8 + t + 4 * u;
        sc[ks][u] = sm.bt[j] * (is_w ? __expf(sm.b[j]) : 1.f);
      }
    const float* X = is_w ? &sm.K[0][0] : &sm.V[0][0];
    const int ld = is_w ? LDK : LDV;
    float* dst = ws + (is_w ? WS_W : WS_U);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int n0 = c0 + n * 8;
      float c4[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m) c4[m][0] = c4[m][1] = c4[m][2] = c4[m][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint32_t b0 = tf32(X[(ks * 8 + t) * ld + n0 + g] * sc[ks][0]);
        const uint32_t b1 = tf32(X[(ks * 8 + t + 4) * ld + n0 + g] * sc[ks][1]);
#pragma unroll
        for (int m = 0; m < 2; ++m)
          if (m == 1 || ks < 2) mma_tf32(c4[m], ta[m][ks][0], ta[m][ks][1], ta[m][ks][2], ta[m][ks][3], b0, b1);
      }
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float2 v = make_float2(c4[m][2 * e], c4[m][2 * e + 1]);
          if (is_w) v = make_float2(rna(v.x), rna(v.y));
          *reinterpret_cast<float2*>(dst + (size_t)(m * 16 + g + 8 * e) * DK + n0 + 2 * t) = v;
        }
    }
  }
}

template <int NV>
struct ChainStage {
  float K[CK][LDK];
  float Q[CK][LDK];
  float W[CK][LDK];
  float P[CK][LDA];
  float U[CK][NV + 8];
  float b[CK];
};
template <int NV>
struct ChainSmem {
  ChainStage<NV> st[2];
  float S[NV][LDK];        // rounded state slice, transposed: S[n][k]
  float D[CK][NV + 8];     // rounded delta rows
};

// grid (n_seg, Hv, 128 / NV), block 256
template <int NV>
__global__ void __launch_bounds__(256) gdn_chain_kernel(const GdnChunkArgs p) {
  constexpr int NT = NV / 8, HT = NT / 2;     // column tiles of the slice, and of one warp of the 32-row products
  extern __shared__ __align__(16) uint8_t smem_raw[];
  ChainSmem<NV>& sm = *reinterpret_cast<ChainSmem<NV>*>(smem_raw);
  const int sg = blockIdx.x, h = blockIdx.y, sl = blockIdx.z, kh = h % p.G;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  int base = 0;
  for (int s = 0; s < sg; ++s) base += window(p, s);
  const int n_chunks = window(p, sg);
  if (n_chunks == 0) return;
  const int s1 = p.seg_start[sg + 1], first = p.seg_start[sg] + p.c_lo * CK;
  float* Sg = p.state + (((size_t)p.seg_slot[sg] * p.Hv + h) * DK) * DK + sl * NV;

  auto fetch = [&](int c) {
    ChainStage<NV>& st = sm.st[c & 1];
    const float* ws = p.ws + ((size_t)(base + c) * p.Hv + h) * WS_UNIT;
    for (int i = tid; i < CK * (DK / 4); i += 256) {
      const int tt = i / (DK / 4), d4 = (i % (DK / 4)) * 4, tok = first + c * CK + tt;
      const bool ok = tok < s1;
      const float* row = p.qkv + (size_t)(ok ? tok : first) * p.C + (size_t)kh * DK + d4;
      cp_async16(&st.Q[tt][d4], row, ok ? 16 : 0);
      cp_async16(&st.K[tt][d4], row + (size_t)p.G * DK, ok ? 16 : 0);
      cp_async16(&st.W[tt][d4], ws + WS_W + tt * DK + d4, 16);
    }
    cp_async16(&st.P[tid >> 3][(tid & 7) * 4], ws + WS_P + tid * 4, 16);
    for (int i = tid; i < CK * (NV / 4); i += 256) {
      const int tt = i / (NV / 4), d4 = (i % (NV / 4)) * 4;
      cp_async16(&st.U[tt][d4], ws + WS_U + tt * DK + sl * NV + d4, 16);
    }
    if (tid < CK / 4) cp_async16(&st.b[tid * 4], ws + WS_B + tid * 4, 16);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // warp w keeps state rows [16 w, +16) of the slice in registers, in accumulator layout; shared memory holds the rounded
  // copy that all warps read as a B operand
  float s[NT][4];
  const int m0 = warp * 16;
  auto publish = [&]() {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      sm.S[n * 8 + 2 * t][m0 + g] = rna(s[n][0]);
      sm.S[n * 8 + 2 * t + 1][m0 + g] = rna(s[n][1]);
      sm.S[n * 8 + 2 * t][m0 + g + 8] = rna(s[n][2]);
      sm.S[n * 8 + 2 * t + 1][m0 + g + 8] = rna(s[n][3]);
    }
  };
  fetch(0);
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 v = *reinterpret_cast<const float2*>(Sg + (size_t)(m0 + g + 8 * e) * DK + n * 8 + 2 * t);
      s[n][2 * e] = v.x;
      s[n][2 * e + 1] = v.y;
    }
  publish();
  const int mt = (warp & 1) * 16, nt = ((warp >> 1) & 1) * HT;     // this warp's tile row and first tile column
  for (int c = 0; c < n_chunks; ++c) {
    ChainStage<NV>& st = sm.st[c & 1];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                   // operands and the previous state are visible, D is free
    if (c + 1 < n_chunks) fetch(c + 1);
    // warps 0..3: D = U - W S;  warps 4..7: Q S (kept in registers).  Two independent chains per tile.
    float c0[HT][4], c1[HT][4];
#pragma unroll
    for (int n = 0; n < HT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) c0[n][e] = c1[n][e] = 0.f;
    const float (*X)[LDK] = warp < 4 ? st.W : st.Q;
#pragma unroll
    for (int kk = 0; kk < DK; kk += 16) {
      const uint4 lo = warp < 4 ? ld4u(&X[mt + g][kk + 4 * t]) : ld4r(&X[mt + g][kk + 4 * t]);
      const uint4 hi = warp < 4 ? ld4u(&X[mt + g + 8][kk + 4 * t]) : ld4r(&X[mt + g + 8][kk + 4 * t]);
#pragma unroll
      for (int n = 0; n < HT; ++n) {
        const uint4 bb = ld4u(&sm.S[(nt + n) * 8 + g][kk + 4 * t]);
        mma_tf32(c0[n], lo.x, hi.x, lo.y, hi.y, bb.x, bb.y);
        mma_tf32(c1[n], lo.z, hi.z, lo.w, hi.w, bb.z, bb.w);
      }
    }
    if (warp < 4) {
#pragma unroll
      for (int n = 0; n < HT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = mt + g + 8 * e, j = (nt + n) * 8 + 2 * t;
          const float2 u = *reinterpret_cast<const float2*>(&st.U[i][j]);
          *reinterpret_cast<float2*>(&sm.D[i][j]) =
              make_float2(rna(u.x - (c0[n][2 * e] + c1[n][2 * e])), rna(u.y - (c0[n][2 * e + 1] + c1[n][2 * e + 1])));
        }
    }
    __syncthreads();                                   // D complete; every read of S is done
    if (warp >= 4) {                                   // O = G (Q S) + P D
      const float ga = __expf(st.b[mt + g]), gb = __expf(st.b[mt + g + 8]);
      float o[HT][4];
#pragma unroll
      for (int n = 0; n < HT; ++n) {
        o[n][0] = ga * (c0[n][0] + c1[n][0]);
        o[n][1] = ga * (c0[n][1] + c1[n][1]);
        o[n][2] = gb * (c0[n][2] + c1[n][2]);
        o[n][3] = gb * (c0[n][3] + c1[n][3]);
      }
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (mt == 0 && ks >= 2) break;                 // P is lower triangular
        const uint32_t a0 = __float_as_uint(st.P[mt + g][ks * 8 + t]), a1 = __float_as_uint(st.P[mt + g + 8][ks * 8 + t]);
        const uint32_t a2 = __float_as_uint(st.P[mt + g][ks * 8 + t + 4]);
        const uint32_t a3 = __float_as_uint(st.P[mt + g + 8][ks * 8 + t + 4]);
#pragma unroll
        for (int n = 0; n < HT; ++n)
          mma_tf32(o[n], a0, a1, a2, a3, __float_as_uint(sm.D[ks * 8 + t][(nt + n) * 8 + g]),
                   __float_as_uint(sm.D[ks * 8 + t + 4][(nt + n) * 8 + g]));
      }
#pragma unroll
      for (int n = 0; n < HT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int tok = first + c * CK + mt + g + 8 * e;
          if (tok < s1)
            *reinterpret_cast<float2*>(p.out + ((size_t)tok * p.Hv + h) * DK + sl * NV + (nt + n) * 8 + 2 * t) =
                make_float2(o[n][2 * e], o[n][2 * e + 1]);
        }
    }
    // S <- G_32 S + Kt^T D
    const float bl = st.b[CK - 1], gall = __expf(bl);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] *= gall;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const float ea = __expf(bl - st.b[ks * 8 + t]), eb = __expf(bl - st.b[ks * 8 + t + 4]);
      const uint32_t a0 = tf32(st.K[ks * 8 + t][m0 + g] * ea), a1 = tf32(st.K[ks * 8 + t][m0 + g + 8] * ea);
      const uint32_t a2 = tf32(st.K[ks * 8 + t + 4][m0 + g] * eb), a3 = tf32(st.K[ks * 8 + t + 4][m0 + g + 8] * eb);
#pragma unroll
      for (int n = 0; n < NT; ++n)
        mma_tf32(s[n], a0, a1, a2, a3, __float_as_uint(sm.D[ks * 8 + t][n * 8 + g]),
                 __float_as_uint(sm.D[ks * 8 + t + 4][n * 8 + g]));
    }
    publish();
  }
  if (p.write_state) {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<float2*>(Sg + (size_t)(m0 + g + 8 * e) * DK + n * 8 + 2 * t) =
            make_float2(s[n][2 * e], s[n][2 * e + 1]);
  }
}

// Chunks that one pass of both kernels covers, over all segments: 160 of them bound the workspace (37 KB per chunk and head)
// whatever the number of tokens.  What fits is one pass, a longer scan goes in windows of as many chunks of every segment.
constexpr int WINDOW_CHUNKS = 160;

struct Windows {
  long long units;        // workspace units of one pass
  int per, count;         // chunks of a segment in one pass; passes
};
// (A scan that leaves the state alone has no place to carry it between windows: one window.)
inline Windows windows(int T, int n_seg, int write_state, int longest) {
  const long long all = T / CK + n_seg;                                // at least the sum of the rounded-up counts
  const int chunks = ((longest > 0 && longest < T ? longest : T) + CK - 1) / CK;
  if (!write_state || all <= WINDOW_CHUNKS) return {all, chunks, 1};
  const int per = n_seg >= WINDOW_CHUNKS ? 1 : WINDOW_CHUNKS / n_seg;
  const long long most = (long long)n_seg * per;
  return {all < most ? all : most, per, (chunks + per - 1) / per};
}

}  // namespace

// Floats of workspace that a scan of T tokens in n_seg segments needs.
HE_API long long he_gdn_chunk_ws_floats(int T, int n_seg, int Hv, int write_state) {
  if (T <= 0 || n_seg <= 0) return 0;
  return windows(T, n_seg, write_state, 0).units * Hv * WS_UNIT;
}
// Passes (of two launches each) that it makes; `longest` as in GdnChunkArgs.
HE_API int he_gdn_chunk_windows(int T, int n_seg, int write_state, int longest) {
  return T <= 0 || n_seg <= 0 ? 0 : windows(T, n_seg, write_state, longest).count;
}

// Chunked tensor-core scan.  Same arguments as he_gdn_scan minus the journal, plus the workspace; state size must be 128.
HE_API int he_gdn_scan_chunked(const GdnChunkArgs* args, cudaStream_t stream) {
  GdnChunkArgs a = *args;
  if (a.T <= 0 || a.n_seg <= 0) return 0;
  const Windows w = windows(a.T, a.n_seg, a.write_state, a.longest);
  if (a.C != 2 * a.G * DK + a.Hv * DK || a.ws == nullptr || a.longest < 0 || a.ws_floats < w.units * a.Hv * WS_UNIT ||
      ((reinterpret_cast<uintptr_t>(a.ws) | reinterpret_cast<uintptr_t>(a.qkv)) & 15) != 0)
    return -HE_ERR_BAD_ARG;
  // set per call (cheap): the attribute belongs to the (function, device) pair, not to the process
  cudaError_t e = cudaFuncSetAttribute(gdn_prepare_chunks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(PrepSmem));
  // one CTA per SM (its two stages fill shared memory): 32 state columns each while those CTAs fit the chip at once, else 64
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool narrow = (long long)a.n_seg * a.Hv * 4 <= sms;
  const size_t chain_smem = narrow ? sizeof(ChainSmem<32>) : sizeof(ChainSmem<64>);
  if (e == cudaSuccess)
    e = narrow ? cudaFuncSetAttribute(gdn_chain_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chain_smem)
               : cudaFuncSetAttribute(gdn_chain_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chain_smem);
  if (e != cudaSuccess) return (int)e;
  for (int i = 0; i < w.count; ++i) {
    a.c_lo = i * w.per;
    a.c_hi = a.c_lo + w.per;
    gdn_prepare_chunks_kernel<<<dim3((unsigned)w.units, a.Hv), 128, sizeof(PrepSmem), stream>>>(a);
    HE_LAUNCH_CHECK();
    if (narrow) gdn_chain_kernel<32><<<dim3(a.n_seg, a.Hv, 4), 256, chain_smem, stream>>>(a);
    else gdn_chain_kernel<64><<<dim3(a.n_seg, a.Hv, 2), 256, chain_smem, stream>>>(a);
    HE_LAUNCH_CHECK();
  }
  return 0;
}
HE_API int he_gdn_chunk_args_size() { return (int)sizeof(GdnChunkArgs); }
