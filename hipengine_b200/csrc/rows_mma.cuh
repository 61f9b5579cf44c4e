// Operands and host helpers of the few-row products (gemm_rows.cu, moe_rows.cu): quantised weight blocks as fp16 MMA
// operands, the activation image, waits, tensor maps of weight rows.  See gemm_rows.cu for the method.
#pragma once
#include <atomic>
#include <cfloat>

#include "common.cuh"
#include "sm100.cuh"
#include "tmap.cuh"

constexpr int ROWS_MAX_SEG = 4;

struct HeRowsSeg {
  const void* w;
  const void* w2;          // second weight of a gate/up pair (epi 3, 4), same block type
  void* out;
  long long out_stride;    // elements between the outputs of two activation rows
  int n_rows;
  int qtype;
  int epi;                 // 0: f32 store, 1: bf16 store, 2: f32 +=, 3: silu(g) * u -> bf16, 4: gelu_tanh(g) * u -> bf16
  int tile0;               // first tile of the segment (set by the launcher)
};

struct HeRowsArgs {
  HeRowsSeg seg[ROWS_MAX_SEG];
  int n_seg;
  int K, R;
  int tc;                  // products and image on tcgen05 (up to 64 rows), else on mma.sync (up to MMA_MAX_ROWS)
  const void* image;       // he_rows_image of the R rows, with the same `tc`
  float* ws;               // partial tiles (he_rows_ws_floats)
  long long ws_floats;
  int* counters;           // zero before the first launch; every launch leaves them zero
  int n_counters;
  int* status;
  int stages, stage_bytes, w_bytes, tiles;   // set by the launcher
};

namespace herows {

using namespace he;

// Image of one block of one activation row: four parts v of 144 bytes.  Part v holds the quads v (columns 4 v .. + 3) of all
// 16-column groups (h, qt, u): unit c = qt / 2 of 64 bytes, in it 16 bytes per (h, u), quads of qt = 2 c and 2 c + 1.  The last 16
// bytes of parts 0 and 1 hold the eight sums per 32 columns in two parts, those of part 2 the scale.  With them lanes that read one
// part and lanes that read one place of four parts both meet no bank twice; 576 bytes put neighbouring rows half a bank cycle apart.
constexpr int IMG_COL = 576, PART = 144, SX_OFF = 128, XS_OFF = 2 * PART + 128;
// Products of more rows than a few run on tcgen05 (gemm_rows_tc.cu), from an image of their own: of one block of n rows (32, 48 or 64)
//   [4 groups of 64 columns][n rows][128 bytes], 128-byte swizzle : the B operand, columns of a quad in the order 0 2 1 3
//   [n / 8][2: high, low parts][8 rows][8 sums per 32 columns], fp16: the B operand of the minima (no swizzle)
//   [n] fp32                                                      : the rows' powers of two
constexpr int MMA_MAX_ROWS = 24;
__host__ __device__ constexpr int tc_rows(int R) { return R <= 32 ? 32 : (R + 15) & ~15; }
__host__ __device__ constexpr int tc_sums(int n) { return n * 512; }
__host__ __device__ constexpr int tc_scales(int n) { return n * 544; }
__host__ __device__ constexpr int tc_image(int n) { return n * 548; }
__host__ __device__ constexpr int tc_image_pad(int n) { return (tc_image(n) + 1023) & ~1023; }

constexpr int MAX_STAGES = 8;
constexpr int SMEM_TOTAL = 220 * 1024;

__host__ __device__ inline int rows_block_bytes(int qt) { return qt == HE_Q4_K ? 144 : qt == HE_Q6_K ? 224 : 272; }
__host__ __device__ inline int col_groups(int R) { return (R + 7) / 8; }       // n8 tiles of R rows

__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ... and one that starts a sum (`first`) instead of adding to it
__device__ __forceinline__ void mma_from(bool first, float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  if (!first) {
    mma(d, a0, a1, a2, a3, b0, b1);
    return;
  }
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// fp16 pairs (bit patterns)
constexpr uint32_t MAGIC = 0x64006400u;       //  1024
constexpr uint32_t M1024 = 0xE400E400u;       // -1024
constexpr uint32_t M1056 = 0xE420E420u;       // -1056 = -(1024 + 32)
constexpr uint32_t M1536 = 0xE600E600u;       // -1536 = -(1024 + 16 * 32)
constexpr uint32_t M1152 = 0xE480E480u;       // -1152 = -(1024 + 128)
constexpr uint32_t M64 = 0xD400D400u;         //   -64
constexpr uint32_t P1_16 = 0x2C002C00u;       //  1/16

// (x & mask) | c as ONE instruction: LOP3 takes a single immediate, so `c` has to be a register the compiler cannot see
// through (with both constants visible it emits two; the integer pipe is the busiest one here)
template <uint32_t MASK>
__device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(x), "n"(MASK), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t opaque(uint32_t c) {
  uint32_t r;
  asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(c));
  return r;
}

// byte i of w as the fp16 pair (1024 + byte, 1024 + byte)
__device__ __forceinline__ uint32_t dup_byte(uint32_t w, uint32_t i) { return prmt(w, 0x64646464u, 0x4040u | i | (i << 8)); }

// One block (256 columns) of the 16 weight rows of a warp: `r0`, `r1` are the shared addresses of rows g and g + 8 in
// the stage, `img` that of the block's image.  acc[nt] += the block's product in the MMA's C layout (rows g / g + 8,
// activation rows 8 nt + 2t, + 1); only the first L groups of eight rows are computed.  SPLIT: two accumulators of a block, half
// the dependent MMAs in a row.  A row's sum is the same for every L of one SPLIT.
template <int NT, int L, bool SPLIT>
__device__ __forceinline__ void block_q4k(uint32_t r0, uint32_t r1, uint32_t img, int lane, uint32_t mg,
                                          float (&acc)[NT][4]) {
  const int g = lane >> 2, t = lane & 3, h = t >> 1, u = t & 1;
  const uint4 ma = lds128(r0), mb = lds128(r1);
  const uint32_t qo = 16 + 64 * h + 16 * u;
  const uint4 qa[2] = {lds128(r0 + qo), lds128(r0 + qo + 32)}, qb[2] = {lds128(r1 + qo), lds128(r1 + qo + 32)};
  // 6-bit scales and minima of sub-blocks 4h .. 4h + 3, one per byte: the upper half's are split into four and two bits
  const uint32_t low_bits = h ? 0x0F0F0F0Fu : 0x3F3F3F3Fu, high_bits = h ? 0x30303030u : 0u;
  const uint32_t sca = ((h ? ma.w : ma.y) & low_bits) | ((ma.y >> 2) & high_bits);
  const uint32_t scb = ((h ? mb.w : mb.y) & low_bits) | ((mb.y >> 2) & high_bits);
  const uint32_t mna = ((h ? ma.w >> 4 : ma.z) & low_bits) | ((ma.z >> 2) & high_bits);
  const uint32_t mnb = ((h ? mb.w >> 4 : mb.z) & low_bits) | ((mb.z >> 2) & high_bits);
  float D[L][4], E[SPLIT ? L : 1][4];
  const uint32_t xb = img + g * IMG_COL + t * 16;
#pragma unroll
  for (int c = 0; c < 2; ++c) {      // chunk 2h + c: low nibbles are group 2c of the half, high nibbles group 2c + 1
    const uint32_t sla = h2_add(dup_byte(sca, 2 * c), M1024), slb = h2_add(dup_byte(scb, 2 * c), M1024);
    const uint32_t sha_ = h2_add(dup_byte(sca, 2 * c + 1), M1024), shb_ = h2_add(dup_byte(scb, 2 * c + 1), M1024);
    const uint32_t cla = h2_mul(sla, M1024), clb = h2_mul(slb, M1024);
    const uint32_t cha = h2_mul(sha_, M64), chb = h2_mul(shb_, M64);         // high nibbles stay in place: 16 q
    const uint32_t sha = h2_mul(sha_, P1_16), shb = h2_mul(shb_, P1_16);
    const uint32_t wa[4] = {qa[c].x, qa[c].y, qa[c].z, qa[c].w}, wb[4] = {qb[c].x, qb[c].y, qb[c].z, qb[c].w};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint32_t a = wa[v], b = wb[v], a8 = a >> 8, b8 = b >> 8;
      const uint32_t l0 = h2_fma(and_or<0x000F000Fu>(a, mg), sla, cla), l1 = h2_fma(and_or<0x000F000Fu>(b, mg), slb, clb);
      const uint32_t l2 = h2_fma(and_or<0x000F000Fu>(a8, mg), sla, cla), l3 = h2_fma(and_or<0x000F000Fu>(b8, mg), slb, clb);
      const uint32_t u0 = h2_fma(and_or<0x00F000F0u>(a, mg), sha, cha), u1 = h2_fma(and_or<0x00F000F0u>(b, mg), shb, chb);
      const uint32_t u2 = h2_fma(and_or<0x00F000F0u>(a8, mg), sha, cha), u3 = h2_fma(and_or<0x00F000F0u>(b8, mg), shb, chb);
#pragma unroll
      for (int n = 0; n < L; ++n) {
        const uint4 x = lds128(xb + n * 8 * IMG_COL + v * PART + c * 64);
        mma_from(v + c == 0, D[n], l0, l1, l2, l3, x.x, x.y);
        mma_from(SPLIT && v + c == 0, SPLIT ? E[SPLIT ? n : 0] : D[n], u0, u1, u2, u3, x.z, x.w);
      }
    }
  }
  if (SPLIT) {
#pragma unroll
    for (int n = 0; n < L; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) D[n][i] += E[SPLIT ? n : 0][i];
  }
  // minima: slots (2t, 2t + 1) meet the high parts of the sums of sub-blocks 2t, 2t + 1, slots + 8 the low parts
  const uint32_t msel = 0x4040u | (2 * u) | ((2 * u + 1) << 8);
  const uint32_t na = h2_add(prmt(mna, 0x64646464u, msel), M1024), nb = h2_add(prmt(mnb, 0x64646464u, msel), M1024);
  const float2 da = __half22float2(*reinterpret_cast<const __half2*>(&ma.x));
  const float2 db = __half22float2(*reinterpret_cast<const __half2*>(&mb.x));
  const uint32_t sx = img + g * IMG_COL + SX_OFF + (t >> 1) * PART + (t & 1) * 8, xs = img + 2 * t * IMG_COL + XS_OFF;
#pragma unroll
  for (int n = 0; n < L; ++n) {
    float M[4];
    const uint2 s = lds64(sx + n * 8 * IMG_COL);
    mma_from(true, M, na, nb, na, nb, s.x, s.y);
    const float p0 = __uint_as_float(lds32(xs + n * 8 * IMG_COL)), p1 = __uint_as_float(lds32(xs + (n * 8 + 1) * IMG_COL));
    acc[n][0] += p0 * (da.x * D[n][0] - da.y * M[0]);
    acc[n][1] += p1 * (da.x * D[n][1] - da.y * M[1]);
    acc[n][2] += p0 * (db.x * D[n][2] - db.y * M[2]);
    acc[n][3] += p1 * (db.x * D[n][3] - db.y * M[3]);
  }
}

template <int NT, int L>
__device__ __forceinline__ void block_scale(uint32_t img, int t, float da, float db, const float (&D)[L][4],
                                            float (&acc)[NT][4]) {
  const uint32_t xs = img + 2 * t * IMG_COL + XS_OFF;
#pragma unroll
  for (int n = 0; n < L; ++n) {
    const float p0 = __uint_as_float(lds32(xs + n * 8 * IMG_COL)), p1 = __uint_as_float(lds32(xs + (n * 8 + 1) * IMG_COL));
    acc[n][0] += p0 * da * D[n][0];
    acc[n][1] += p1 * da * D[n][1];
    acc[n][2] += p0 * db * D[n][2];
    acc[n][3] += p1 * db * D[n][3];
  }
}

template <int NT, int L, bool SPLIT>
__device__ __forceinline__ void block_q6k(uint32_t r0, uint32_t r1, uint32_t img, int lane, uint32_t mg,
                                          float (&acc)[NT][4]) {
  const int g = lane >> 2, t = lane & 3, h = t >> 1, u = t & 1;
  const uint32_t lo = 64 * h + 16 * u, ho = 128 + 32 * h + 16 * u;
  const uint4 la = lds128(r0 + lo), lb = lds128(r0 + lo + 32), lh = lds128(r0 + ho);
  const uint4 ka = lds128(r1 + lo), kb = lds128(r1 + lo + 32), kh = lds128(r1 + ho);
  const uint2 sa = lds64(r0 + 192 + 8 * h), sb = lds64(r1 + 192 + 8 * h);
  // signed scales of the four groups (byte 2 qt + u), one per byte, as byte + 128
  const uint32_t ssel = u ? 0x7531u : 0x6420u;
  const uint32_t sca = prmt(sa.x, sa.y, ssel) ^ 0x80808080u, scb = prmt(sb.x, sb.y, ssel) ^ 0x80808080u;
  float D[L][4], E[SPLIT ? L : 1][4];
  const uint32_t xb = img + g * IMG_COL + t * 16;
  uint32_t fa[4], fb[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    fa[q] = h2_add(dup_byte(sca, q), M1152);
    fb[q] = h2_add(dup_byte(scb, q), M1152);
    if (q >= 2) {                     // groups 2, 3 come from high nibbles left in place: 16 (q - 32)
      fa[q] = h2_mul(fa[q], P1_16);
      fb[q] = h2_mul(fb[q], P1_16);
    }
  }
  const uint32_t lav[4] = {la.x, la.y, la.z, la.w}, lbv[4] = {lb.x, lb.y, lb.z, lb.w}, lhv[4] = {lh.x, lh.y, lh.z, lh.w};
  const uint32_t kav[4] = {ka.x, ka.y, ka.z, ka.w}, kbv[4] = {kb.x, kb.y, kb.z, kb.w}, khv[4] = {kh.x, kh.y, kh.z, kh.w};
  auto low = [mg](uint32_t l, uint32_t hs, uint32_t f) {
    return h2_mul(h2_add(and_or<0x00300030u>(hs, and_or<0x000F000Fu>(l, mg)), M1056), f);
  };
  auto high = [mg](uint32_t l, uint32_t hs, uint32_t f) {
    return h2_mul(h2_add(and_or<0x03000300u>(hs, and_or<0x00F000F0u>(l, mg)), M1536), f);
  };
#pragma unroll
  for (int v = 0; v < 4; ++v) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t e[4], o[4];            // the MMA's a0..a3 of groups 2c and 2c + 1
      const uint32_t hA = lhv[v], hB = khv[v], hA8 = hA >> 8, hB8 = hB >> 8;
      if (c == 0) {
        e[0] = low(lav[v], hA << 4, fa[0]);
        e[1] = low(kav[v], hB << 4, fb[0]);
        e[2] = low(lav[v] >> 8, hA8 << 4, fa[0]);
        e[3] = low(kav[v] >> 8, hB8 << 4, fb[0]);
        o[0] = low(lbv[v], hA << 2, fa[1]);
        o[1] = low(kbv[v], hB << 2, fb[1]);
        o[2] = low(lbv[v] >> 8, hA8 << 2, fa[1]);
        o[3] = low(kbv[v] >> 8, hB8 << 2, fb[1]);
      } else {
        e[0] = high(lav[v], hA << 4, fa[2]);
        e[1] = high(kav[v], hB << 4, fb[2]);
        e[2] = high(lav[v] >> 8, hA8 << 4, fa[2]);
        e[3] = high(kav[v] >> 8, hB8 << 4, fb[2]);
        o[0] = high(lbv[v], hA << 2, fa[3]);
        o[1] = high(kbv[v], hB << 2, fb[3]);
        o[2] = high(lbv[v] >> 8, hA8 << 2, fa[3]);
        o[3] = high(kbv[v] >> 8, hB8 << 2, fb[3]);
      }
#pragma unroll
      for (int n = 0; n < L; ++n) {
        const uint4 x = lds128(xb + n * 8 * IMG_COL + v * PART + c * 64);
        mma_from(v + c == 0, D[n], e[0], e[1], e[2], e[3], x.x, x.y);
        mma_from(SPLIT && v + c == 0, SPLIT ? E[SPLIT ? n : 0] : D[n], o[0], o[1], o[2], o[3], x.z, x.w);
      }
    }
  }
  if (SPLIT) {
#pragma unroll
    for (int n = 0; n < L; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) D[n][i] += E[SPLIT ? n : 0][i];
  }
  const uint32_t dwa = lds32(r0 + 208), dwb = lds32(r1 + 208);
  block_scale<NT, L>(img, t, __low2float(*reinterpret_cast<const __half2*>(&dwa)),
                  __low2float(*reinterpret_cast<const __half2*>(&dwb)), D, acc);
}

// Byte i of w, an integer - 128 with its sign bit flipped, as a float times 1 / div (exact: 2^23 + byte).
template <int DIV>
__device__ __forceinline__ float byte_scale(uint32_t w, uint32_t i) {
  const float f = __uint_as_float(prmt(w, 0x4B000000u, 0x7440u | i));
  return DIV == 1 ? f - 8388736.f : fmaf(f, 1.f / DIV, -8388736.f / DIV);
}
// acc += (row g's scale, row g + 8's scale) * D, two sums an instruction
__device__ __forceinline__ void add_scaled(float (&acc)[4], float sa, float sb, const float (&D)[4]) {
  asm("{\n\t.reg .b64 x, y, s;\n\t"
      "mov.b64 s, {%4, %4};\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%6, %7};\n\t"
      "fma.rn.f32x2 x, s, y, x;\n\tmov.b64 {%0, %1}, x;\n\t"
      "mov.b64 s, {%5, %5};\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%8, %9};\n\t"
      "fma.rn.f32x2 x, s, y, x;\n\tmov.b64 {%2, %3}, x;\n\t}"
      : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
      : "f"(sa), "f"(sb), "f"(D[0]), "f"(D[1]), "f"(D[2]), "f"(D[3]));
}

// The same with exact weights: an MMA takes the 16 columns of one sub-block (lane t its quad t), its integers q - 32 as they are,
// and the sub-block's scale meets the fp32 sums.
template <int NT, int L>
__device__ __forceinline__ void block_q6k_exact(uint32_t r0, uint32_t r1, uint32_t img, int lane, uint32_t mg,
                                                float (&acc)[NT][4]) {
  const int g = lane >> 2, t = lane & 3;
  const uint4 sa = lds128(r0 + 192), sb = lds128(r1 + 192);
  const uint32_t wa[4] = {sa.x ^ 0x80808080u, sa.y ^ 0x80808080u, sa.z ^ 0x80808080u, sa.w ^ 0x80808080u};
  const uint32_t wb[4] = {sb.x ^ 0x80808080u, sb.y ^ 0x80808080u, sb.z ^ 0x80808080u, sb.w ^ 0x80808080u};
  const uint32_t xb = img + g * IMG_COL + t * PART, q0 = r0 + 4 * t, q1 = r1 + 4 * t;
  auto low = [mg](uint32_t l, uint32_t hs) { return h2_add(and_or<0x00300030u>(hs, and_or<0x000F000Fu>(l, mg)), M1056); };
  auto high = [mg](uint32_t l, uint32_t hs) {       // 16 (q - 32)
    return h2_add(and_or<0x03000300u>(hs, and_or<0x00F000F0u>(l, mg)), M1536);
  };
  float D[L][4];
#pragma unroll
  for (int n = 0; n < L; ++n) D[n][0] = D[n][1] = D[n][2] = D[n][3] = 0.f;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int h = s >> 1, u = s & 1, lo = 64 * h + 16 * u, ho = 128 + 32 * h + 16 * u;
    const uint32_t la = lds32(q0 + lo), lb = lds32(q0 + lo + 32), lh = lds32(q0 + ho);
    const uint32_t ka = lds32(q1 + lo), kb = lds32(q1 + lo + 32), kh = lds32(q1 + ho);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t e[4], o[4];            // groups 2c and 2c + 1
      if (c == 0) {
        e[0] = low(la, lh << 4);
        e[1] = low(ka, kh << 4);
        e[2] = low(la >> 8, lh >> 4);
        e[3] = low(ka >> 8, kh >> 4);
        o[0] = low(lb, lh << 2);
        o[1] = low(kb, kh << 2);
        o[2] = low(lb >> 8, lh >> 6);
        o[3] = low(kb >> 8, kh >> 6);
      } else {
        e[0] = high(la, lh << 4);
        e[1] = high(ka, kh << 4);
        e[2] = high(la >> 8, lh >> 4);
        e[3] = high(ka >> 8, kh >> 4);
        o[0] = high(lb, lh << 2);
        o[1] = high(kb, kh << 2);
        o[2] = high(lb >> 8, lh >> 6);
        o[3] = high(kb >> 8, kh >> 6);
      }
      constexpr int W = 16;
      const float ea = c == 0 ? byte_scale<1>(wa[2 * h], u) : byte_scale<W>(wa[2 * h + 1], u);
      const float eb = c == 0 ? byte_scale<1>(wb[2 * h], u) : byte_scale<W>(wb[2 * h + 1], u);
      const float oa = c == 0 ? byte_scale<1>(wa[2 * h], 2 + u) : byte_scale<W>(wa[2 * h + 1], 2 + u);
      const float ob = c == 0 ? byte_scale<1>(wb[2 * h], 2 + u) : byte_scale<W>(wb[2 * h + 1], 2 + u);
#pragma unroll
      for (int n = 0; n < L; ++n) {
        const uint4 x = lds128(xb + n * 8 * IMG_COL + s * 16 + c * 64);
        float P[4], R[4];
        mma_from(true, P, e[0], e[1], e[2], e[3], x.x, x.y);
        mma_from(true, R, o[0], o[1], o[2], o[3], x.z, x.w);
        add_scaled(D[n], ea, eb, P);
        add_scaled(D[n], oa, ob, R);
      }
    }
  }
  const uint32_t dwa = lds32(r0 + 208), dwb = lds32(r1 + 208);
  block_scale<NT, L>(img, t, __low2float(*reinterpret_cast<const __half2*>(&dwa)),
                  __low2float(*reinterpret_cast<const __half2*>(&dwb)), D, acc);
}

// Q8_0: `p0` / `p1` are the region's planes [2][HT rows][128 bytes] (128-byte swizzle) and [HT rows][8 scales]; rows i0, i1.
// Two MMAs take the 32 columns of one sub-block, its bytes as they are (lane t the quads 2 (t / 2), + 1 of the 16 columns
// t % 2), and the sub-block's scale meets the fp32 sums: exact weights.
template <int NT, int L, int HT>
__device__ __forceinline__ void block_q80(uint32_t p0, int i0, uint32_t p1, int i1, uint32_t img, int lane,
                                          uint32_t mg, float (&acc)[NT][4]) {
  const int g = lane >> 2, t = lane & 3, u = t & 1;
  const uint4 sa = lds128(p0 + 2 * HT * 128 + i0 * 16), sb = lds128(p1 + 2 * HT * 128 + i1 * 16);
  const uint32_t wa[4] = {sa.x, sa.y, sa.z, sa.w}, wb[4] = {sb.x, sb.y, sb.z, sb.w};
  const uint32_t ra = p0 + i0 * 128 + (t >> 1) * 8, rb = p1 + i1 * 128 + (t >> 1) * 8;
  const uint32_t xb = img + g * IMG_COL + (t >> 1) * 2 * PART + u * 16;
  auto up = [mg](uint32_t w) { return h2_add(and_or<0x00FF00FFu>(w, mg), M1152); };
  float D[L][4];
#pragma unroll
  for (int n = 0; n < L; ++n) D[n][0] = D[n][1] = D[n][2] = D[n][3] = 0.f;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint2 va[2], vb[2];             // sub-blocks 2c, 2c + 1 of the half
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int chunk = 2 * (2 * c + q) + u;
        va[q] = lds64(ra + h * HT * 128 + ((chunk ^ (i0 & 7)) << 4));
        vb[q] = lds64(rb + h * HT * 128 + ((chunk ^ (i1 & 7)) << 4));
      }
      const float2 da = __half22float2(*reinterpret_cast<const __half2*>(&wa[2 * h + c]));
      const float2 db = __half22float2(*reinterpret_cast<const __half2*>(&wb[2 * h + c]));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t a[2][4];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t ka = (i ? va[q].y : va[q].x) ^ 0x80808080u, kb = (i ? vb[q].y : vb[q].x) ^ 0x80808080u;
          a[q][0] = up(ka);
          a[q][1] = up(kb);
          a[q][2] = up(ka >> 8);
          a[q][3] = up(kb >> 8);
        }
#pragma unroll
        for (int n = 0; n < L; ++n) {
          const uint4 x = lds128(xb + n * 8 * IMG_COL + i * PART + c * 64 + h * 32);
          float P[4], R[4];
          mma_from(true, P, a[0][0], a[0][1], a[0][2], a[0][3], x.x, x.y);
          mma_from(true, R, a[1][0], a[1][1], a[1][2], a[1][3], x.z, x.w);
          add_scaled(D[n], da.x, db.x, P);
          add_scaled(D[n], da.y, db.y, R);
        }
      }
    }
  block_scale<NT, L>(img, t, 1.f, 1.f, D, acc);
}

// Bounded wait whose polls the hardware suspends for up to ~10 us each: the polling loop of a waiting warp would take
// issue slots from the warps that compute.
__device__ __forceinline__ bool wait_long(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  for (uint32_t i = 0; i < (1u << 20); ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(sm100::smem_u32(bar)), "r"(parity), "r"(10000u)
        : "memory");
    if (ok) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  if (status != nullptr) atomicCAS(status, 0, code);
  return false;
}

__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(sm100::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ float4 ldcg4(const float* p) {
  float4 v;
  asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Eight consecutive columns (8 * lane) of a block of an activation row, as the fp16 fragments that the products load: x over the
// power of two of the block's largest value (at most 2^126, whose reciprocal is the smallest normal number: up to 4 then); the
// sums of the rounded values per 32 columns in two parts.  Into the row's unit `unit` or, TC, as row r of the block's image `unit` of n
// rows; and into the row's unit `also` (or null).
template <bool TC>
__device__ __forceinline__ void image_store(uint8_t* unit, uint8_t* also, int n, int r, int lane, const float (&v)[8]) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
  bool odd = false;                     // a NaN or an infinity stays one, under scale 1
#pragma unroll
  for (int i = 0; i < 8; ++i) odd |= !(fabsf(v[i]) <= FLT_MAX);
  amax = warp_max(amax);
  uint32_t e = min(__float_as_uint(amax) & 0x7F800000u, 0x7E800000u);
  if (__any_sync(0xffffffffu, odd)) e = 0x3F800000u;
  const float inv = __uint_as_float(0x7F000000u - e);
  __half hv[8];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    hv[i] = __float2half_rn(v[i] * inv);
    s += __half2float(hv[i]);
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  const int sub = lane >> 2;
  if (TC) {
    const __half2 p[4] = {__halves2half2(hv[0], hv[2]), __halves2half2(hv[1], hv[3]), __halves2half2(hv[4], hv[6]),
                          __halves2half2(hv[5], hv[7])};
    *reinterpret_cast<uint4*>(unit + (lane >> 3) * n * 128 + r * 128 + (((lane & 7) ^ (r & 7)) << 4)) =
        *reinterpret_cast<const uint4*>(p);
    if ((lane & 3) == 0) {
      const __half hi = __float2half_rn(s), lo = __float2half_rn(s - __half2float(hi));
      uint8_t* at = unit + tc_sums(n) + (r >> 3) * 256 + (r & 7) * 16 + sub * 2;
      *reinterpret_cast<__half*>(at) = hi;
      *reinterpret_cast<__half*>(at + 128) = lo;
    }
    if (lane == 0) *reinterpret_cast<float*>(unit + tc_scales(n) + r * 4) = __uint_as_float(e);
    if (also == nullptr) return;
    unit = also;
  }
  const int h = lane >> 4, qt = (lane >> 2) & 3, u = (lane >> 1) & 1, v0 = (lane & 1) * 2, t = 2 * h + u;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    __half2 p[2] = {__halves2half2(hv[4 * q], hv[4 * q + 2]), __halves2half2(hv[4 * q + 1], hv[4 * q + 3])};
    const int at = (v0 + q) * PART + (qt >> 1) * 64 + t * 16 + (qt & 1) * 8;
    *reinterpret_cast<uint2*>(unit + at) = *reinterpret_cast<const uint2*>(p);
    if (!TC && also != nullptr) *reinterpret_cast<uint2*>(also + at) = *reinterpret_cast<const uint2*>(p);
  }
  if ((lane & 3) == 0) {
    const __half hi = __float2half_rn(s), lo = __float2half_rn(s - __half2float(hi));
    const int at = SX_OFF + (sub >> 2) * PART + ((sub >> 1) & 1) * 8 + (sub & 1) * 2;
    *reinterpret_cast<__half*>(unit + at) = hi;
    *reinterpret_cast<__half*>(unit + at + 4) = lo;
    if (!TC && also != nullptr) {
      *reinterpret_cast<__half*>(also + at) = hi;
      *reinterpret_cast<__half*>(also + at + 4) = lo;
    }
  }
  if (lane == 0) {
    *reinterpret_cast<float*>(unit + XS_OFF) = __uint_as_float(e);
    if (!TC && also != nullptr) *reinterpret_cast<float*>(also + XS_OFF) = __uint_as_float(e);
  }
}

__device__ __forceinline__ void load_cols(const void* x, int dtype, size_t off, float (&v)[8]) {
  if (dtype == 0) {
    const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + off);
    const float4 a = p[0], b = p[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(x) + off);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
  }
}

// Dynamic shared memory that a kernel may ask for, set once per device.  `bytes` is the kernel's largest need, the same in every
// call: threads that set it at the same time agree, and none takes back what another one's launch relies on.
template <typename F>
inline cudaError_t allow_smem(F kernel, int bytes, std::atomic<unsigned long long>& devices) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (e == cudaSuccess && (devices.load(std::memory_order_acquire) & bit) == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_release);
  }
  return e;
}

// Weight rows as bytes: [rows][row_bytes], box {box_bytes, box_rows}
inline int byte_map(CUtensorMap* m, const void* ptr, long long rows, long long row_bytes, int box_bytes, bool swizzle, int box_rows) {
  const EncodeTiledFn enc = get_encode();
  if (enc == nullptr || (reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || row_bytes % 16 != 0) return -HE_ERR_BAD_ARG;
  const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)box_bytes, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1000 + (int)r;
}

inline int weight_maps(CUtensorMap* m, const void* w, int qtype, long long rows, int K, int box) {
  if (w == nullptr) return -HE_ERR_BAD_ARG;
  if (qtype == HE_Q4_K) return byte_map(m, w, rows, (long long)(K >> 8) * 144, 144, false, box);
  if (qtype == HE_Q6_K) return byte_map(m, w, rows, (long long)(K >> 8) * 224, 224, false, box);
  if (qtype != HE_Q8_0) return -HE_ERR_BAD_ARG;
  const long long rb = (long long)K + (((K >> 4) + 15) / 16) * 16;
  const int rc = byte_map(m, w, rows, rb, 128, true, box);
  return rc != 0 ? rc : byte_map(m + 1, w, rows, rb, 16, false, box);
}

struct RowsMaps {
  CUtensorMap m[ROWS_MAX_SEG][4];   // [2 * (second weight of a pair) + (scale plane of Q8_0)]
};

// Units per CTA: the first `rem` take base + 1, the others base.  (Divided once, by the host: eight 64-bit divisions a thread were
// 3 us at the start of every launch.)
struct RowsPlan {
  int base, rem;
  __host__ __device__ int begin(int cta) const { return base * cta + (cta < rem ? cta : rem); }
  __host__ __device__ int cta_of(int unit) const {
    const unsigned big = (unsigned)rem * (unsigned)(base + 1), x = (unsigned)unit;
    return x < big ? (int)(x / (unsigned)(base + 1)) : rem + (int)((x - big) / (unsigned)base);
  }
};

// Products of up to 64 rows on tcgen05 (gemm_rows_tc.cu)
int launch_rows_tc(const HeRowsArgs& a, int num_sms, cudaStream_t stream);

}  // namespace herows
