// The state pass of the decode step on the tensor pipe (states scaled along k, head dim 128).
//
// The read-out vectors q and k are held as 30-bit fixed point with one power-of-two scale per vector and cut into four
// BALANCED byte digits (each in [-128, 127]: x = d3 2^24 + d2 2^16 + d1 2^8 + d0).  The eight digit vectors are the
// eight columns of the B operand of an integer tensor-core product
//     D[row][n] = sum_k code[row][k] * digit_n[k]          (mma.sync m16n8k32, int8 x int8 -> int32, exact)
// taken per 32-column unit; the units of one scale group accumulate in the same registers, the group's fp16 scale is
// applied to the exact integer sums, and the four digits of a vector are recombined with powers of two.  No code is
// ever converted to floating point.  A fixed-point element is exact when it lies within 2^-6 of the vector's largest
// one and is otherwise rounded to 2^-30 of it, so the pass is at least as accurate as an fp32 accumulation.
//
// Shared-memory layout of a stage's codes (128 state rows): the rows as they lie in the slot, the 16-byte chunks of a row
// permuted by the copy engine's swizzle (a tensor-map copy, one instruction a stage): 128-byte rows (8-bit codes) chunk ^= row
// mod 8, 64-byte rows (4-bit) chunk ^= row / 2 mod 4, so that the eight row addresses of an ldmatrix 8x8 tile fall on distinct
// banks.
// A warp takes rows 32 w .. 32 w + 31 (two blocks of 16) and ends up with one finished row per lane: lane (i = lane / 4, t = lane
// % 4) owns row 32 w + 8 t + i.
//
// Column n of B: vector n / 4 (0: q, 1: k), digit 3 - n % 4, so that a thread's two accumulator columns (2t, 2t + 1)
// are the upper digit pair (t even) or the lower digit pair (t odd) of one vector.
// Units: 8-bit codes: unit j = columns 32 j .. 32 j + 31, k index = column - 32 j.  4-bit codes: unit j = the same
// columns = 16 bytes; the low nibbles (even columns) are k 0..15, the high nibbles (odd columns) k 16..31; nibbles
// carry an offset of 8, which the start value of the accumulators takes off (8 * column sum of the digits, itself
// computed by a product with an all-ones A operand).
#pragma once
#include "common.cuh"

namespace sqb {

constexpr int MAGIC_I = 0x4B400000;      // bit pattern of 1.5 * 2^23: an int32 accumulator started here reads, as a
                                          // float, 1.5 * 2^23 + sum (exact while |sum| < 2^22)

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr));
}
// D += A B: A 16 x 32 bytes (unsigned if AU), B 32 x 8 signed bytes, int32 accumulators
template <bool AU>
__device__ __forceinline__ void mma_i8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  if constexpr (AU)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- fixed point ----------------------------------------------------------------------------------------------------
// Multipliers m1 m2 = 2^(TOP - e) (e: exponent of the vector's largest magnitude, which lands in [2^TOP, 2^(TOP + 1))) as two
// factors that are both normal floats over the whole float range, and their inverses.  A non-finite amax poisons the
// inverse (outputs become NaN).
struct FxScale { float m1, m2, i1, i2; };
template <int TOP>
__device__ __forceinline__ FxScale fx_scale(float amax) {
  int e = static_cast<int>((__float_as_uint(amax) >> 23) & 0xFFu) - 127;
  e = max(e, -126);
  const int sh = TOP - e;
  const int h2 = sh >> 1, h1 = sh - h2;
  FxScale s;
  s.m1 = __uint_as_float(static_cast<uint32_t>(127 + h1) << 23);
  s.m2 = __uint_as_float(static_cast<uint32_t>(127 + h2) << 23);
  s.i1 = __uint_as_float(static_cast<uint32_t>(127 - h1) << 23);
  s.i2 = __uint_as_float(static_cast<uint32_t>(127 - h2) << 23);
  if (!(amax <= 3.0e38f)) { s.m1 = 0.f; s.m2 = 0.f; s.i1 = __uint_as_float(0x7FC00000u); }
  return s;
}
__device__ __forceinline__ FxScale fx30_scale(float amax) { return fx_scale<29>(amax); }
// the four balanced digits of x (|x| <= 2^30, rounded to an integer) as the bytes of the result, lowest digit in byte 0
__device__ __forceinline__ uint32_t byte_digits(float x) {
  return (static_cast<uint32_t>(__float2int_rn(x)) + 0x80808080u) ^ 0x80808080u;
}
__device__ __forceinline__ uint32_t fx30_digits(float v, const FxScale& s) { return byte_digits((v * s.m1) * s.m2); }

// One lane's four consecutive columns (4 lane .. 4 lane + 3) of vector `vec` -> its words of the B fragments in
// shared memory, Bf[(unit * 2 + reg) * 32 + n * 4 + t].  All 32 lanes call this together.
template <int BITS>
__device__ __forceinline__ void put_b_words(uint32_t* Bf, int lane, int vec, uint32_t y0, uint32_t y1, uint32_t y2,
                                            uint32_t y3) {
  const uint32_t t0 = __byte_perm(y0, y1, 0x5140), t1 = __byte_perm(y2, y3, 0x5140);
  const uint32_t t2 = __byte_perm(y0, y1, 0x7362), t3 = __byte_perm(y2, y3, 0x7362);
  uint32_t W[4] = {__byte_perm(t0, t1, 0x5410), __byte_perm(t0, t1, 0x7632), __byte_perm(t2, t3, 0x5410),
                   __byte_perm(t2, t3, 0x7632)};                 // W[s]: digit s of the four columns
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int n = vec * 4 + (3 - s);
    if constexpr (BITS == 8) {
      Bf[(lane >> 2) * 32 + n * 4 + (lane & 3)] = W[s];           // unit lane / 8, reg (lane / 4) & 1, t lane % 4
    } else {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, W[s], 1);
      const uint32_t w = (lane & 1) ? __byte_perm(o, W[s], 0x7531) : __byte_perm(W[s], o, 0x6420);
      const int p = lane >> 1;                                   // span of 8 columns; unit p / 4, t p % 4
      Bf[((p >> 2) * 2 + (lane & 1)) * 32 + n * 4 + (p & 3)] = w;
    }
  }
}

// Start values of the accumulators of scale group g (two columns per thread): the magic integer, minus 8 * the column
// sums of the digits over the group's units for nibble codes.
template <int BITS, int UPG>
__device__ __forceinline__ void acc_start(const uint32_t (&bf)[8], int (&ci)[4 / UPG][2]) {
  constexpr int NG = 4 / UPG;
#pragma unroll
  for (int g = 0; g < NG; g++) {
    if constexpr (BITS == 4) {
      int d[4] = {0, 0, 0, 0};
#pragma unroll
      for (int u = 0; u < UPG; u++) {
        const int j = g * UPG + u;
        mma_i8<true>(d, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, bf[2 * j], bf[2 * j + 1]);
      }
      ci[g][0] = MAGIC_I - 8 * d[0];
      ci[g][1] = MAGIC_I - 8 * d[1];
    } else {
      ci[g][0] = MAGIC_I;
      ci[g][1] = MAGIC_I;
    }
  }
}

// Shared address of 16-byte chunk `chunk` of row `row` in a stage at `codes` (aligned to the swizzle's 1024 or 512 bytes).  The
// chunk's bits are XORed with the row's, so chunk c's address is chunk 0's ^ 16 c.
template <int BITS>
__device__ __forceinline__ uint32_t tile_addr(uint32_t codes, int row, int chunk) {
  constexpr int ROWB = 128 * BITS / 8;
  return codes + row * ROWB + ((chunk ^ (BITS == 8 ? row & 7 : (row >> 1) & 3)) << 4);
}
// the row address this lane supplies to an ldmatrix.x4 of block bb of warp w's rows: matrices (rows 0 .. 7, rows 8 .. 15) x (chunk 0,
// chunk 1)
template <int BITS>
__device__ __forceinline__ uint32_t tile_lrow(uint32_t codes, int w, int lane, int bb) {
  return tile_addr<BITS>(codes, 32 * w + 16 * bb + (lane & 15), lane >> 4);
}
__device__ __forceinline__ int tile_row(int w, int lane) { return 32 * w + 8 * (lane & 3) + (lane >> 2); }

// the NG fp16 scales of a row
template <int NG>
__device__ __forceinline__ void row_scales(const unsigned short* sc, float (&s)[NG]) {
  if constexpr (NG == 4) {
    const uint2 w = *reinterpret_cast<const uint2*>(sc);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
    s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
  } else if constexpr (NG == 2) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(sc));
    s[0] = a.x; s[1] = a.y;
  } else {
    s[0] = __half2float(__ushort_as_half(*sc));
  }
}

// One 16-row block against all units: p[0..3] += scale * sums for (row0, col 2t), (row0, col 2t + 1), (row1, ...).
// a_addr: this lane's ldmatrix row address for the block's first 32 bytes; sc0, sc1: the NG scales of the two rows (SCALED), or not
// looked at: the blocks of a state scaled along v carry no scale of their own.
template <int BITS, int UPG, bool SCALED = true>
__device__ __forceinline__ void block_pass(uint32_t a_addr, const unsigned short* sc0, const unsigned short* sc1, const uint32_t (&bf)[8],
                                           const int (&ci)[4 / UPG][2], float (&p)[4]) {
  constexpr int NG = 4 / UPG;
  float s0[NG], s1[NG];
  if constexpr (SCALED) { row_scales<NG>(sc0, s0); row_scales<NG>(sc1, s1); }
  int acc[NG][4];
#pragma unroll
  for (int g = 0; g < NG; g++) { acc[g][0] = ci[g][0]; acc[g][1] = ci[g][1]; acc[g][2] = ci[g][0]; acc[g][3] = ci[g][1]; }
  if constexpr (BITS == 8) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t m[4];
      ldsm_x4(m, a_addr ^ (32 * j));
      mma_i8<false>(acc[j / UPG], m[0], m[1], m[2], m[3], bf[2 * j], bf[2 * j + 1]);
    }
  } else {
#pragma unroll
    for (int J = 0; J < 2; J++) {
      uint32_t m[4];
      ldsm_x4(m, a_addr ^ (32 * J));
      const uint32_t l0 = m[0] & 0x0F0F0F0Fu, l1 = m[1] & 0x0F0F0F0Fu, l2 = m[2] & 0x0F0F0F0Fu, l3 = m[3] & 0x0F0F0F0Fu;
      const uint32_t h0 = (m[0] >> 4) & 0x0F0F0F0Fu, h1 = (m[1] >> 4) & 0x0F0F0F0Fu, h2 = (m[2] >> 4) & 0x0F0F0F0Fu,
                     h3 = (m[3] >> 4) & 0x0F0F0F0Fu;
      mma_i8<true>(acc[(2 * J) / UPG], l0, l1, h0, h1, bf[4 * J], bf[4 * J + 1]);
      mma_i8<true>(acc[(2 * J + 1) / UPG], l2, l3, h2, h3, bf[4 * J + 2], bf[4 * J + 3]);
    }
  }
  // (the accumulators of a row are a register pair: packed f32x2 arithmetic, same roundings)
  float2 p01 = make_float2(p[0], p[1]), p23 = make_float2(p[2], p[3]);
  const float2 nm = make_float2(-12582912.0f, -12582912.0f);
#pragma unroll
  for (int g = 0; g < NG; g++) {
    const float2 a01 = __fadd2_rn(make_float2(__int_as_float(acc[g][0]), __int_as_float(acc[g][1])), nm);
    const float2 a23 = __fadd2_rn(make_float2(__int_as_float(acc[g][2]), __int_as_float(acc[g][3])), nm);
    if constexpr (SCALED) {
      p01 = __ffma2_rn(a01, make_float2(s0[g], s0[g]), p01);
      p23 = __ffma2_rn(a23, make_float2(s1[g], s1[g]), p23);
    } else {
      p01 = a01;
      p23 = a23;
    }
  }
  p[0] = p01.x; p[1] = p01.y; p[2] = p23.x; p[3] = p23.y;
}

// Recombine the digit pair of a thread: after this, lane t = 0 holds vector 0 of row0, t = 1 vector 0 of row1,
// t = 2 vector 1 of row0, t = 3 vector 1 of row1 (still in fixed-point units).
__device__ __forceinline__ float join_digits(const float (&p)[4], int t) {
  const float wa = (t & 1) ? 256.0f : 16777216.0f, wb = (t & 1) ? 1.0f : 65536.0f;
  const float x0 = fmaf(p[0], wa, p[1] * wb), x1 = fmaf(p[2], wa, p[3] * wb);
  const float recv = __shfl_xor_sync(0xffffffffu, (t & 1) ? x0 : x1, 1);
  return ((t & 1) ? x1 : x0) + recv;
}

// The pass of one tile (32 rows of a stage): on return lane (i, t) holds the sums of stage row tile_row(w, lane) against vector 0
// (tq) and vector 1 (tk), in fixed-point units.  codes: shared address of the stage; scs: its scales [row][NG].
template <int BITS, int UPG>
__device__ __forceinline__ void tile_pass(uint32_t codes, const unsigned short* scs, const uint32_t (&bf)[8],
                                          const int (&ci)[4 / UPG][2], int w, int lane, float& tq, float& tk) {
  constexpr int NG = 4 / UPG;
  const int t = lane & 3;
  const uint32_t lrow = tile_lrow<BITS>(codes, w, lane, 0);
  const unsigned short* sr = scs + (32 * w + (lane >> 2)) * NG;
  float T[2];
#pragma unroll
  for (int bb = 0; bb < 2; bb++) {
    float p[4] = {0.f, 0.f, 0.f, 0.f};
    block_pass<BITS, UPG>(lrow + bb * 16 * (128 * BITS / 8), sr + bb * 16 * NG, sr + (bb * 16 + 8) * NG, bf, ci, p);
    T[bb] = join_digits(p, t);
  }
  const float recv = __shfl_xor_sync(0xffffffffu, t < 2 ? T[1] : T[0], 2);
  tq = t < 2 ? T[0] : recv;
  tk = t < 2 ? recv : T[1];
}

// ---- states scaled along v (one scale per column for every group of 32 rows) ------------------------------------------
// The scale varies along the contraction, so it goes into the read-out vectors: group G of a head is read against
// q * scale_G and k * scale_G, in fixed point as above, and the integer sums need no scale afterwards.  A warp's 32 rows are
// exactly one group, and it builds its own B fragments for it.

// The warp's B fragments for its group: sg = the group's 128 column scales (fp16), vq / vk = the read-out vectors
// (fp32, 128 each; vk unused if !TWO).  Bf: the warp's own 1 KB of shared memory.  Returns the fixed-point scales.
template <int BITS, bool TWO>
__device__ __forceinline__ void build_b_v(uint32_t* Bf, const unsigned short* sg, const float* vq, const float* vk, int lane,
                                          uint32_t (&bf)[8], FxScale& fq, FxScale& fk) {
  const uint2 sw = *reinterpret_cast<const uint2*>(sg + 4 * lane);
  const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sw.x)), s23 = __half22float2(*reinterpret_cast<const __half2*>(&sw.y));
  const float4 q4 = *reinterpret_cast<const float4*>(vq + 4 * lane);
  float eq[4] = {q4.x * s01.x, q4.y * s01.y, q4.z * s23.x, q4.w * s23.y};
  float ek[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (TWO) {
    const float4 k4 = *reinterpret_cast<const float4*>(vk + 4 * lane);
    ek[0] = k4.x * s01.x; ek[1] = k4.y * s01.y; ek[2] = k4.z * s23.x; ek[3] = k4.w * s23.y;
  }
  float mq = fmaxf(fmaxf(fabsf(eq[0]), fabsf(eq[1])), fmaxf(fabsf(eq[2]), fabsf(eq[3])));
  float mk = fmaxf(fmaxf(fabsf(ek[0]), fabsf(ek[1])), fmaxf(fabsf(ek[2]), fabsf(ek[3])));
  mq = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mq)));
  if constexpr (TWO) mk = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mk)));
  fq = fx30_scale(mq);
  fk = fx30_scale(mk);
  uint32_t yq[4], yk[4];
#pragma unroll
  for (int j = 0; j < 4; j++) { yq[j] = fx30_digits(eq[j], fq); yk[j] = TWO ? fx30_digits(ek[j], fk) : 0u; }
  __syncwarp();                                        // the fragments of the previous stage have been read
  put_b_words<BITS>(Bf, lane, 0, yq[0], yq[1], yq[2], yq[3]);
  put_b_words<BITS>(Bf, lane, 1, yk[0], yk[1], yk[2], yk[3]);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 8; r++) bf[r] = Bf[r * 32 + lane];
}

template <int BITS>
__device__ __forceinline__ void tile_pass_v(uint32_t codes, const uint32_t (&bf)[8], int w, int lane, float& tq, float& tk) {
  const int t = lane & 3;
  int ci[1][2];
  acc_start<BITS, 4>(bf, ci);
  const uint32_t lrow = tile_lrow<BITS>(codes, w, lane, 0);
  float T[2];
#pragma unroll
  for (int bb = 0; bb < 2; bb++) {
    float p[4] = {0.f, 0.f, 0.f, 0.f};
    block_pass<BITS, 4, false>(lrow + bb * 16 * (128 * BITS / 8), nullptr, nullptr, bf, ci, p);
    T[bb] = join_digits(p, t);
  }
  const float recv = __shfl_xor_sync(0xffffffffu, t < 2 ? T[1] : T[0], 2);
  tq = t < 2 ? T[0] : recv;
  tk = t < 2 ? recv : T[1];
}

}  // namespace sqb
