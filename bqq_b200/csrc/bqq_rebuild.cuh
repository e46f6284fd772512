// One 32x32 block of the dense weight from its plane words, in registers:
//   W[p][q] = sum_b ( a_b sum_k Y_b[p][k] Z_b[k][q] + b_b sum_k Y_b[p][k] + c_b sum_k Z_b[k][q] ) + d
// by one warp.  Bound: issue and fixed-latency dependences at four warps per scheduler (registers), with the int8 tensor
// pipe (10 products m16n8k32 of 9 clocks per bit layer and 32 ranks) beside them; what is not a product is kept as short
// as possible.  Measured, 4096 x 14336 with 4 bit layers to bf16: 62.9 us with 14 products and scalar multiply-adds -> 55.3.
//  * A count leaves the tensor core as an integer n 2^s (s: the powers of two that the operand masks below leave in).
//    Its bit pattern, read as a float, IS the subnormal number n 2^(s-149), and a multiply-add takes subnormal inputs at
//    full rate: with coefficients scaled by 2^84 the sums are ordinary floats of full precision, and one multiply-add
//    per entry and bit layer is all there is - no conversion, no start value.  The powers of two are taken out once at
//    the end.  (Coefficients beyond 2^43 would overflow; products below 2^-87 would lose bits.)
//  * Y (A operand): a lane's plane word holds rows g + 8 rr and ranks 16 kh + 4 t + e at bit 8 e + 4 kh + rr, so
//    word & (0x01010101 << rr) is an operand register (bytes 0 or 2^rr).
//  * Z (B operand): the four ranks of one column are one nibble of a plane word.  byte * 0x08040201 repeats the byte
//    at a pitch of 9 bits, so bit 3 of byte s is bit 3 - s of the low nibble and bit 7 of byte s that of the high one:
//    one multiplication and two masks make the registers of two 8-column tiles (bytes 0 or 8 and 0 or 128).  The ranks
//    come out in reverse, so the bytes of the Y word are reversed too (any common order of the contraction serves).
//  * Row sums are products with an operand of ones.  Column sums as such products would be four of the fourteen products
//    of a bit layer; here every lane adds up the bytes of its own B registers (dp4a), and the four lanes of a column are
//    added once per block.
//  * Entries are accumulated two at a time (fma.rn.f32x2), which halves the issue slots of what is left.
// Column order: the tile nt = 2 qh + x holds, at column n, q = 16 qh + 4 (n >> 1) + 2 x + (n & 1); a lane thus owns
// q = 16 qh + 4 t + {0..3} of every row, in two pairs (x = 0, 1): 8- or 16-byte global stores that fill 32-byte sectors, or
// the registers of a 16x256b tensor-memory store.
#pragma once
#include "bqq_common.cuh"

namespace bqq {

__device__ __forceinline__ void mma_u8u8_zero(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_u8u8_add(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kCoefExp = 84;                         // coefficients come in multiplied by 2^84
constexpr float kCoefScale = 19342813113834066795298816.f;
// 2^(62 - e): takes the powers of two out of a sum (62 = 149 - 84 - 3)
template <int E>
__device__ __forceinline__ float rebuild_unscale() {
  static_assert(62 - E > -126 && 62 - E < 127, "");
  return __int_as_float((127 + 62 - E) << 23);
}

// Where a lane finds its Z bytes.
struct RebuildLane {
  uint32_t zsel[2];            // byte of tile x, zeros above it
  int zfrom;                   // plane lane of rank half 0 (rank half 1: + 16)
};
__device__ __forceinline__ RebuildLane rebuild_lane(int lane) {
  const int g = lane >> 2, t = lane & 3;
  const uint32_t e = g & 1;
  RebuildLane L;
  L.zsel[0] = 0x4440u | e;
  L.zsel[1] = 0x4440u | (e ^ 2u);
  L.zfrom = 4 * t + (g >> 1);
  return L;
}

// Sums of a block so far: acc[rr][nt] = rows g + 8 rr, columns 2 t and 2 t + 1; what depends on the row or on the column only is
// kept apart until the end: row[rr] whole, col[nt] for column g over this lane's ranks.
struct RebuildAcc {
  float2 acc[4][4];
  float row[4];
  float col[4];
  float2 colsum[4];                                  // columns 2 t, 2 t + 1, after rebuild_end
};
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
// Takes the powers of two out of the row and column terms (d joins the rows), adds up the column terms of the four lanes of
// a column (each keeps the tile nt = t) and hands every lane those of its columns ...
__device__ __forceinline__ void rebuild_end(RebuildAcc& r, float d, int lane) {
  r.row[0] = fmaf(r.row[0], rebuild_unscale<0>(), d);
  r.row[1] = fmaf(r.row[1], rebuild_unscale<1>(), d);
  r.row[2] = fmaf(r.row[2], rebuild_unscale<2>(), d);
  r.row[3] = fmaf(r.row[3], rebuild_unscale<3>(), d);
  const int t = lane & 3;
  const float c0 = r.col[0] * rebuild_unscale<0>(), c1 = r.col[1] * rebuild_unscale<0>();
  const float c2 = r.col[2] * rebuild_unscale<4>(), c3 = r.col[3] * rebuild_unscale<4>();
  const float k0 = (t & 1 ? c1 : c0) + __shfl_xor_sync(0xffffffffu, t & 1 ? c0 : c1, 1);
  const float k1 = (t & 1 ? c3 : c2) + __shfl_xor_sync(0xffffffffu, t & 1 ? c2 : c3, 1);
  const float full = (t & 2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, t & 2 ? k0 : k1, 2);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
    r.colsum[nt] = make_float2(__shfl_sync(0xffffffffu, full, 8 * t + nt), __shfl_sync(0xffffffffu, full, 8 * t + 4 + nt));
}
// ... and gives the entries of row g + 8 RR in tile NT: acc 2^(62-e) + (col + row), two at a time.
template <int RR, int NT>
__device__ __forceinline__ float2 rebuild_entry(const RebuildAcc& r) {
  constexpr int E = RR + (NT < 2 ? 0 : 4);
  unsigned long long v;
  float2 o;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(pack2(r.colsum[NT].x, r.colsum[NT].y)), "l"(pack2(r.row[RR], r.row[RR])));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(pack2(r.acc[RR][NT].x, r.acc[RR][NT].y)), "l"(pack2(rebuild_unscale<E>(), rebuild_unscale<E>())));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(v));
  return o;
}

// acc += (k, k) * (n0, n1), the integers' bit patterns taken as floats
template <bool FIRST>
__device__ __forceinline__ void fma_pair(float2& acc, float k, int n0, int n1) {
  const unsigned long long n = pack2(__int_as_float(n0), __int_as_float(n1)), kk = pack2(k, k);
  unsigned long long v;
  if (FIRST) {
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(n), "l"(kk));
  } else {
    v = pack2(acc.x, acc.y);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(n), "l"(kk));
  }
  asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.x), "=f"(acc.y) : "l"(v));
}

// Adds one bit layer (FIRST: starts the sums with it).  y, z: the words of this lane's col patch in RT blocks of 32 lanes x 4 col patches of Y and of Z
// (shared memory).
template <int RT, bool FIRST>
__device__ __forceinline__ void rebuild_bit(RebuildAcc& r, const RebuildLane& L, const uint32_t* y, const uint32_t* z,
                                            int lane, float a, float b, float c) {
  uint32_t A[RT][2][4], B[RT][4][2];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt) {
    const uint32_t w = __byte_perm(y[rt * 128 + lane * 4], 0u, 0x0123);
    const uint32_t w4 = w >> 4;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      A[rt][mt][0] = w & (0x01010101u << (2 * mt));
      A[rt][mt][1] = w & (0x02020202u << (2 * mt));
      A[rt][mt][2] = w4 & (0x01010101u << (2 * mt));
      A[rt][mt][3] = w4 & (0x02020202u << (2 * mt));
    }
#pragma unroll
    for (int kh = 0; kh < 2; ++kh) {
      const uint32_t v = z[rt * 128 + (L.zfrom + 16 * kh) * 4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const uint32_t m = __byte_perm(v, 0u, L.zsel[x]) * 0x08040201u;
        B[rt][x][kh] = m & 0x08080808u;
        B[rt][2 + x][kh] = m & 0x80808080u;
      }
    }
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {                   // row sums: B = 8 everywhere
    int d[4];
    mma_u8u8_zero(d, A[0][mt], 0x08080808u, 0x08080808u);
    if (RT == 2) mma_u8u8_add(d, A[RT - 1][mt], 0x08080808u, 0x08080808u);
    r.row[2 * mt] = FIRST ? b * __int_as_float(d[0]) : fmaf(b, __int_as_float(d[0]), r.row[2 * mt]);
    r.row[2 * mt + 1] = FIRST ? b * __int_as_float(d[2]) : fmaf(b, __int_as_float(d[2]), r.row[2 * mt + 1]);
  }
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    int d0[4], d1[4];
    mma_u8u8_zero(d0, A[0][0], B[0][nt][0], B[0][nt][1]);
    mma_u8u8_zero(d1, A[0][1], B[0][nt][0], B[0][nt][1]);
    uint32_t zs = __dp4a(B[0][nt][1], 0x01010101u, __dp4a(B[0][nt][0], 0x01010101u, 0u));
    if (RT == 2) {
      zs = __dp4a(B[RT - 1][nt][1], 0x01010101u, __dp4a(B[RT - 1][nt][0], 0x01010101u, zs));
      mma_u8u8_add(d0, A[RT - 1][0], B[RT - 1][nt][0], B[RT - 1][nt][1]);
      mma_u8u8_add(d1, A[RT - 1][1], B[RT - 1][nt][0], B[RT - 1][nt][1]);
    }
    r.col[nt] = FIRST ? c * __uint_as_float(zs) : fmaf(c, __uint_as_float(zs), r.col[nt]);
    fma_pair<FIRST>(r.acc[0][nt], a, d0[0], d0[1]);
    fma_pair<FIRST>(r.acc[1][nt], a, d0[2], d0[3]);
    fma_pair<FIRST>(r.acc[2][nt], a, d1[0], d1[1]);
    fma_pair<FIRST>(r.acc[3][nt], a, d1[2], d1[3]);
  }
}

// n bit layers in a row; words of bit layer b at y + b step and z + b step, its {a, b, c, .} at k[b kstep], to be multiplied
// by f.  FIRST: they start the sums.
template <int RT>
__device__ __forceinline__ void rebuild_bits(RebuildAcc& r, const RebuildLane& L, const uint32_t* y, const uint32_t* z, int step,
                                             const float4* k, int kstep, float f, int lane, int n, bool first) {
  if (first) {
    const float4 c = *k;
    rebuild_bit<RT, true>(r, L, y, z, lane, c.x * f, c.y * f, c.z * f);
    --n; y += step; z += step; k += kstep;
  }
#pragma unroll 1
  for (; n > 0; --n, y += step, z += step, k += kstep) {
    const float4 c = *k;
    rebuild_bit<RT, false>(r, L, y, z, lane, c.x * f, c.y * f, c.z * f);
  }
}

}  // namespace bqq
