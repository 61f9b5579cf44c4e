// Parts of the few-row products on the 5th-generation tensor cores: quantised weight blocks as fp16 operands in tensor memory, the
// sum over blocks.  See gemm_rows_tc.cu for the method.
#pragma once
#include "rows_mma.cuh"

namespace herows {

constexpr int TC_UNPACK_WARPS = 8, TC_SUM_WARPS = 8, TC_THREADS = 32 * (TC_UNPACK_WARPS + TC_SUM_WARPS + 4);
// Tensor memory: [2 slots][sums, sums of the minima][n columns], then two operands of 256 fp16 columns
constexpr uint32_t TC_A_COL = 256, TC_A_SLOT = 128;
constexpr int TC_MAX_STAGES = 8;
constexpr int TC_SMEM = 227 * 1024;                 // dynamic shared memory of a block
constexpr int TC_HALF = 64;                         // rows of each weight of a gate/up pair in a tile
constexpr int TC_MIN_BYTES = 128 * 32;              // operand of the minima: 128 rows x 16 fp16
// The way of a group of unpacking warps through the ring: a block's stage and the parity of its arrival.  Blocks go to the two groups in
// turn, and an arrival is signalled to the group that takes the block alone: a phase bit tells only neighbours apart, and in an odd ring
// a stage holds a block of each group in turn.  A group comes by all its barriers in one lap of an even ring, in two of an odd one.
struct TcWalk {
  int s = 0;
  uint32_t ph = 0, lap = 0;
  __host__ __device__ __forceinline__ void next(int stages) {
    if (++s == stages) {
      s = 0;
      lap ^= 1u;
      ph ^= (stages & 1) != 0 ? lap ^ 1u : 1u;
    }
  }
};

// Does a block of this type take a second operand for what the first one's rounding to 11 bits leaves?
__host__ __device__ constexpr bool tc_two(int qtype) { return qtype == HE_Q8_0; }

struct TcBars {
  uint64_t full[2][TC_MAX_STAGES];  // blocks and image have landed, for the group of unpacking warps that takes them
  uint64_t empty[TC_MAX_STAGES];    // ... and are read (by the summing warps, the last to do so)
  uint64_t ready[4];                // [2 slot + half]: the operand is stored
  uint64_t done[4];                 // the products of this half are complete
  uint64_t filled[2];               // the products of the block in this slot are complete
  uint64_t drained[2];              // the slot's accumulators are read
  uint64_t fin[2];
  uint32_t tmem_base;
  int abort_flag;
  int last[2];                      // was this CTA the last to arrive at its first / last shared tile
};

__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void tmem_ld_8(uint32_t a, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(a) : "memory");
}
// K-major operand of 16 columns without swizzle: matrices of 8 rows x 16 bytes, the two of a row group 128 bytes apart, row groups 256.
__device__ __forceinline__ uint64_t desc_k16(uint32_t a) {
  return (uint64_t)((a & 0x3FFFFu) >> 4) | (uint64_t)(128 >> 4) << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46;
}
// kind::f16 with fp16 operands, K-major both, fp32 sums, 128 x n
__host__ __device__ constexpr uint32_t idesc_f16(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (128u >> 4 << 24); }

// Where a thread's weight row lies in a stage: TMEM lane 32 q + lane.  Of a pair, whose two weights are staged one behind the other,
// lanes l and l + 16 hold a gate row and its up row.
struct TcRow {
  uint32_t off;             // from the stage's weights: of the row, or (Q8_0) of its weight's planes
  int i, rows;              // Q8_0: row in the planes, rows of them
  __device__ __forceinline__ TcRow(bool pair, int q, int lane, int bb, int qtype) {
    i = pair ? 16 * q + (lane & 15) : 32 * q + lane;
    rows = pair ? TC_HALF : 2 * TC_HALF;
    off = (uint32_t)((pair ? (lane >> 4) * TC_HALF * bb : 0) + (qtype == HE_Q8_0 ? 0 : i * bb));
  }
};

// ---------------------------------------------------------------- operands: 64 columns (k-block c) of a weight row
// Q4_K: sc * q, exact (see gemm_rows.cu).
__device__ __forceinline__ void tc_q4k(uint32_t row, int c, const uint4& meta, uint32_t mg, uint32_t (&r)[32]) {
  const uint4 qa = lds128(row + 16 + 32 * c), qb = lds128(row + 32 + 32 * c);
  const uint32_t sc = c < 2 ? meta.y : ((meta.w & 0x0F0F0F0Fu) | ((meta.y >> 2) & 0x30303030u));
  const uint32_t s6 = (sc & 0x3F3F3F3Fu) >> (16 * (c & 1));
  const uint32_t sl = h2_add(dup_byte(s6, 0), M1024), s2 = h2_add(dup_byte(s6, 1), M1024);
  const uint32_t cl = h2_mul(sl, M1024), ch = h2_mul(s2, M64), sh = h2_mul(s2, P1_16);     // high nibbles stay in place: 16 q
  const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t a = w[i], a8 = a >> 8;
    r[2 * i] = h2_fma(and_or<0x000F000Fu>(a, mg), sl, cl);
    r[2 * i + 1] = h2_fma(and_or<0x000F000Fu>(a8, mg), sl, cl);
    r[16 + 2 * i] = h2_fma(and_or<0x00F000F0u>(a, mg), sh, ch);
    r[16 + 2 * i + 1] = h2_fma(and_or<0x00F000F0u>(a8, mg), sh, ch);
  }
}
// The row's eight 6-bit minima as fp16
__device__ __forceinline__ uint4 tc_q4k_minima(const uint4& meta) {
  const uint32_t a = meta.z & 0x3F3F3F3Fu, b = ((meta.w >> 4) & 0x0F0F0F0Fu) | ((meta.z >> 2) & 0x30303030u);
  return make_uint4(h2_add(prmt(a, 0x64646464u, 0x4140u), M1024), h2_add(prmt(a, 0x64646464u, 0x4342u), M1024),
                    h2_add(prmt(b, 0x64646464u, 0x4140u), M1024), h2_add(prmt(b, 0x64646464u, 0x4342u), M1024));
}
// Q6_K: scale * (q - 32), 13 bits rounded to 11
__device__ __forceinline__ void tc_q6k(uint32_t row, int c, uint32_t mg, uint32_t (&r)[32]) {
  const int half = c >> 1, cb = c & 1;
  const uint32_t scw = lds32(row + 192 + 8 * half + 4 * cb) ^ 0x80808080u;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint4 hv = lds128(row + 128 + 32 * half + 16 * u);
    const uint32_t h[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const uint4 lv = lds128(row + 64 * half + 32 * t + 16 * u);
      const uint32_t l[4] = {lv.x, lv.y, lv.z, lv.w};
      uint32_t f = h2_add(dup_byte(scw, 2 * t + u), M1152);
      if (cb) f = h2_mul(f, P1_16);                 // high nibbles stay in place: 16 (q - 32)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t x = t ? h[i] << 2 : h[i] << 4, y = t ? h[i] >> 6 : h[i] >> 4;
        uint32_t a0, a1;
        if (cb == 0) {
          a0 = h2_add(and_or<0x00300030u>(x, and_or<0x000F000Fu>(l[i], mg)), M1056);
          a1 = h2_add(and_or<0x00300030u>(y, and_or<0x000F000Fu>(l[i] >> 8, mg)), M1056);
        } else {
          a0 = h2_add(and_or<0x03000300u>(x, and_or<0x00F000F0u>(l[i], mg)), M1536);
          a1 = h2_add(and_or<0x03000300u>(y, and_or<0x00F000F0u>(l[i] >> 8, mg)), M1536);
        }
        r[16 * t + 8 * u + 2 * i] = h2_mul(a0, f);
        r[16 * t + 8 * u + 2 * i + 1] = h2_mul(a1, f);
      }
    }
  }
}
// Q8_0: the power of two of the largest scale of a row's block; integers, and the scales under 2^-8 of it (`inv`: 511.75, the largest then,
// times -128 is fp16's largest number) of 32 columns each.  x * f rounds to 11 bits; what that leaves of the
// 19, fma(x, f, -that), is exact down to 2^-24.  So scales down to 2^-22 of the block's largest are exact; smaller ones become multiples
// of 2^-32 of its power of two.
__device__ __forceinline__ float tc_q80_pow(uint32_t plane, const TcRow& at) {
  const uint4 s = lds128(plane + at.rows * 256 + at.i * 16);
  const uint32_t m = 0x7FFF7FFFu;
  const uint32_t v = __vmaxu2(__vmaxu2(s.x & m, s.y & m), __vmaxu2(s.z & m, s.w & m));
  const uint16_t top = (uint16_t)max(v & 0xFFFFu, v >> 16);
  const uint32_t e = __float_as_uint(half_bits_to_f32(top)) & 0x7F800000u;
  return e == 0 ? 1.f : __uint_as_float(min(e, 143u << 23));        // (a scale that is not finite stays so)
}
constexpr float TC_Q80_SCALE = 1.f / 256.f;
__device__ __forceinline__ float tc_q80_inv(float pow) { return __uint_as_float(0x7F000000u + (8u << 23) - __float_as_uint(pow)); }
__device__ __forceinline__ void tc_q80(uint32_t plane, const TcRow& at, int c, float inv, uint32_t mg, uint32_t (&x)[32],
                                       uint32_t (&f)[2]) {
  const uint32_t scw = lds32(plane + at.rows * 256 + at.i * 16 + 4 * c);
  const uint32_t base = plane + (c >> 1) * at.rows * 128 + at.i * 128;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const __half2 d2 = __half2half2(__float2half_rn(half_bits_to_f32((uint16_t)(k ? scw >> 16 : scw)) * inv));
    f[k] = *reinterpret_cast<const uint32_t*>(&d2);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint4 q = lds128(base + (((4 * (c & 1) + k) ^ (at.i & 7)) << 4));
    const uint32_t w[4] = {q.x ^ 0x80808080u, q.y ^ 0x80808080u, q.z ^ 0x80808080u, q.w ^ 0x80808080u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[8 * k + 2 * j] = h2_add(and_or<0x00FF00FFu>(w[j], mg), M1152);
      x[8 * k + 2 * j + 1] = h2_add(and_or<0x00FF00FFu>(w[j] >> 8, mg), M1152);
    }
  }
}

// What p = x * f left of the product
__device__ __forceinline__ uint32_t h2_rest(uint32_t x, uint32_t f, uint32_t p) {
  uint32_t d;
  asm("{\n\t.reg .b32 t;\n\tneg.f16x2 t, %3;\n\tfma.rn.f16x2 %0, %1, %2, t;\n\t}" : "=r"(d) : "r"(x), "r"(f), "r"(p));
  return d;
}

// ---------------------------------------------------------------- sum over blocks
__device__ __forceinline__ uint64_t f2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void f2_get(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// acc[j] += scale[j] * (d * D[j] + m * M[j]) over NC columns (pairs of them); `t`: D, and with MIN M n columns on; `xs`: scales
template <int NC, bool MIN>
__device__ __forceinline__ void tc_add(uint32_t t, int n, uint32_t xs, float d, float m, uint64_t (&acc)[NC / 2]) {
  const uint64_t dd = f2(d, d), mm = f2(m, m);
#pragma unroll
  for (int c = 0; c < NC; c += 8) {
    uint32_t D[8], M[8];
    tmem_ld_8(t + c, D);
    if (MIN) tmem_ld_8(t + n + c, M);
    const uint4 p0 = lds128(xs + 4 * c), p1 = lds128(xs + 4 * c + 16);
    sm100::tmem_ld_wait();
    const uint64_t p[4] = {f2(p0.x, p0.y), f2(p0.z, p0.w), f2(p1.x, p1.y), f2(p1.z, p1.w)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint64_t v = f2_mul(dd, f2(D[2 * j], D[2 * j + 1]));
      if (MIN) v = f2_fma(mm, f2(M[2 * j], M[2 * j + 1]), v);
      acc[c / 2 + j] = f2_fma(p[j], v, acc[c / 2 + j]);
    }
  }
}

}  // namespace herows
