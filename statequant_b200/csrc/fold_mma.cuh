// The fold of a stage (128 state rows) on the tensor pipe, for the tensor-core decode kernel (step_mma.cuh), buffer
// length 8, decays per head (Gated DeltaNet, Mamba2):
//     S[v][k] = alpha (code[v][k] scale) + sum_i L_i[v] key_i[k],     L_i[v] = (dec_i u_i[v]) ks_i,  key_i = int8 codes
// The sum over the 8 buffer slots is a K = 8 contraction.  L is fp32: it is cut into three bf16 pieces (8 + 8 + 8
// mantissa bits: exact), the int8 key codes are exact in bf16, so every product of an mma.m16n8k16 (bf16 x bf16 -> fp32)
// is exact and only the accumulation (fp32, in the tensor core's order) rounds.  K index = piece * 8 + slot: an
// m16n8k16 takes pieces 0 and 1, an m16n8k8 piece 2.  The stored state enters as the start value of the
// accumulators, rounded twice as the reference does (code * scale, then * alpha).
//
// The codes never leave the ldmatrix fragment layout of the state pass (mma_pass.cuh): a span = 16 rows x 32 bytes is
// one ldmatrix.x4; its values are the C fragments of 4 (8-bit) or 8 (4-bit) N-blocks whose column order is chosen to
// match (a thread's bytes are its accumulator columns), re-rounded in registers and put back with stmatrix.x4.  The
// stage is then written to the slot by bulk copies (shared -> global).
#pragma once
#include "mma_pass.cuh"

namespace sqb {

template <int N> struct IntC { static constexpr int value = N; };

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
}
// max(|a|, |b|, |c|)
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ void stsm_x4(uint32_t saddr, const uint32_t (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(saddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void ldsm_x2(uint32_t (&r)[2], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(saddr));
}
__device__ __forceinline__ void stsm_x2(uint32_t saddr, uint32_t r0, uint32_t r1) {
  asm volatile("stmatrix.sync.aligned.m8n8.x2.shared.b16 [%0], {%1, %2};" ::"r"(saddr), "r"(r0), "r"(r1) : "memory");
}
__device__ __forceinline__ void st_v8(float* p, float a, float b, float c, float d, float e, float f, float g, float h) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d), "f"(e), "f"(f), "f"(g), "f"(h) : "memory");
}
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes) : "memory");
}
// One copy of a box of a tensor map (64- or 128-byte rows of a slot's codes, swizzled in shared memory: mma_pass.cuh); x = 0 always.
struct alignas(64) TileMap { unsigned char bytes[128]; };      // a CUtensorMap, encoded by the host (tile_map.h)
__device__ __forceinline__ void tile_g2s(void* dst, const TileMap* map, int row, int slot, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(0), "r"(row), "r"(slot), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tile_s2g(const TileMap* map, int row, int slot, const void* src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
               ::"l"(map), "r"(0), "r"(row), "r"(slot), "r"(smem_u32(src)) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the bulk stores of this thread have read their shared-memory source (which may then be reused or released)
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

__device__ __forceinline__ uint32_t bf2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// x = p1 + p2 + p3 exactly, each a bf16 (x finite; pieces that underflow are dropped, far below the rounding of the sum)
__device__ __forceinline__ void split3(float x, float& p1, float& p2, float& p3) {
  p1 = __bfloat162float(__float2bfloat16_rn(x));
  const float r1 = x - p1;
  p2 = __bfloat162float(__float2bfloat16_rn(r1));
  p3 = __bfloat162float(__float2bfloat16_rn(r1 - p2));
}

// x / s + mb for a pair of values, rounded to an integer by the addition of mb: r = RN(1 / s), ns = -s.  With the
// reciprocal correctly rounded and an exact residual, q0 + residual r is the IEEE quotient (Markstein; checked for every
// fp16 divisor by tests/div_h16_check.c), so the integer is rint(div_rn(x, s)) without a branch.  A scale that
// overflowed to infinity comes as r = s = 0 and gives 0, as the division does.
__device__ __forceinline__ float2 div_round2(float2 x, float2 r, float2 ns, float mb) {
  const float2 q0 = __fmul2_rn(x, r);
  return __fadd2_rn(__ffma2_rn(__ffma2_rn(q0, ns, x), r, q0), make_float2(mb, mb));
}

// Columns are taken 32 at a time (a HALF: one 32-byte span of 8-bit codes, 16 bytes of 4-bit codes): four N-blocks, whose
// column order is the order in which a fragment register holds the codes.  First column of N-block p of half h for
// accumulator column pair t; the pair is (col, col + 1).
template <int BITS>
__host__ __device__ __forceinline__ int fold_col(int h, int p, int t) {
  if (BITS == 8) return 32 * h + (p >> 1) * 16 + 4 * t + (p & 1) * 2;
  return 32 * h + 8 * t + 2 * p;
}

// The B operand of the fold: for every (half, N-block) the thread's register: the key codes of slots (2t, 2t + 1), t = lane
// % 4, at the column of accumulator column lane / 4, as a bf16 pair.  KBf[(half * 32 + lane) * 4 + N-block], so that a
// thread's four registers of a half are one 128-bit read; built by the CTA's threads, one (half, lane) pair each.
// kbt: buffered keys [8][DK] int8 (slots 0..6 valid), kcur: the key appended by this token (its rounded codes).
template <int BITS, int DK = 128>
__device__ __forceinline__ void build_key_frags(uint32_t* KBf, const int8_t* kbt, const int8_t* kcur, int tid) {
  if (tid >= DK) return;
  const int h = tid >> 5, l = tid & 31, n = l >> 2, s0 = 2 * (l & 3);
  const int8_t* r0 = kbt + s0 * DK + (n & 1);
  const int8_t* r1 = (s0 + 1 == 7 ? kcur : kbt + (s0 + 1) * DK) + (n & 1);
  uint32_t w[4];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const int col = fold_col<BITS>(h, p, n >> 1);
    w[p] = bf2(static_cast<float>(r0[col]), static_cast<float>(r1[col]));
  }
  *reinterpret_cast<uint4*>(KBf + tid * 4) = make_uint4(w[0], w[1], w[2], w[3]);
}

// KDA: the fold's right factor is the buffered key times its per-channel decay ratio, an fp32 value:
//     Kd_i[k] = (code_i[k] ks_i) exp(gnew[k] - G_i[k])          (slot 7: this token's key, ratio 1)
// cut into three bf16 pieces like L.  Three planes of fragments, KBf[p * PLANE + x], x as in build_key_frags.
// gbt: the slot's buffered log decays [8][128] fp32; ga: gnew [128]; ksf: key scales of slots 0..6, [7] = this token's.
template <int BITS>
__device__ __forceinline__ void build_key_frags_kda(uint32_t* KBf, const int8_t* kbt, const int8_t* kcur, const float* gbt,
                                                    const float* ga, const float* ksf, int tid) {
  constexpr int PLANE = 512;
  const int h = tid >> 5, l = tid & 31, n = l >> 2, s0 = 2 * (l & 3);
  uint32_t w[3][4];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const int col = fold_col<BITS>(h, p, n >> 1) + (n & 1);
    const float g = ga[col];
    const float k0 = (static_cast<float>(kbt[s0 * 128 + col]) * ksf[s0]) * expf(g - gbt[s0 * 128 + col]);
    const float k1 = s0 + 1 == 7 ? static_cast<float>(kcur[col]) * ksf[7]
                                 : (static_cast<float>(kbt[(s0 + 1) * 128 + col]) * ksf[s0 + 1]) * expf(g - gbt[(s0 + 1) * 128 + col]);
    float a1, a2, a3, b1, b2, b3;
    split3(k0, a1, a2, a3);
    split3(k1, b1, b2, b3);
    w[0][p] = bf2(a1, b1); w[1][p] = bf2(a2, b2); w[2][p] = bf2(a3, b3);
  }
#pragma unroll
  for (int i = 0; i < 3; i++) *reinterpret_cast<uint4*>(KBf + i * PLANE + tid * 4) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// One A fragment register triple: L of one row at slots 2t, 2t + 1 in three bf16 pieces.  ub: the head's buffered values
// of that row (slots DV apart), uq: this token's rounded value; VDEC: no decay and no key scale in L.
template <int DV, bool VDEC>
__device__ __forceinline__ void fold_left(const int8_t* ub, float uq, const float* tb, const float* ksf, int t, uint32_t& A1,
                                          uint32_t& A2, uint32_t& A3) {
  float p1[2], p2[2], p3[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int s = 2 * t + e;
    float L = uq;
    if (s < 7) L = tb[s] * (static_cast<float>(ub[s * DV]) * tb[8 + s]);
    split3(VDEC ? L : L * ksf[s], p1[e], p2[e], p3[e]);
  }
  A1 = bf2(p1[0], p1[1]); A2 = bf2(p2[0], p2[1]); A3 = bf2(p3[0], p3[1]);
}

// The values of NH halves (32 columns each) of two rows from half h0 on, advanced across the buffer, as accumulators
// acc[half][N-block][row pair].  m: the two rows' codes as fragment registers (8-bit: (row a, row b) x two words; 4-bit: (row
// a, row b)); sc: their scales by group; A1 .. A3: the A fragments of L (fold_left); al2 / ae: the decay (VDEC: per channel).
template <int BITS, int UPG, int NH, bool VDEC>
__device__ __forceinline__ void fold_acc(const uint32_t (&m)[NH][4], const float (&sc)[2][UPG == 1 ? NH : 1], const uint32_t (&A1)[2],
                                         const uint32_t (&A2)[2], const uint32_t (&A3)[2], const uint32_t* KBf, int h0, int lane,
                                         float2 al2, const float* ae, float (&acc)[NH][4][4]) {
  [[maybe_unused]] const int t = lane & 3;
  // ---- start values: (code * scale) * decay; code * scale is exact in fp32, so this rounds once, as the reference's
  // two multiplications do ----
#pragma unroll
  for (int h = 0; h < NH; h++) {
    const float s0 = sc[0][UPG == 1 ? h : 0], s1 = sc[1][UPG == 1 ? h : 0];
    auto decay_of = [&](int p) -> float2 {         // of N-block p's column pair: per head, or (KDA) per key channel
      if constexpr (VDEC) return *reinterpret_cast<const float2*>(ae + fold_col<BITS>(h0 + h, p, t));
      else return al2;
    };
    if constexpr (BITS == 8) {
      // byte u = code + 128 lands in bits 8..15 of 2^23's mantissa: the float is 2^23 + 256 u, and
      // fma(that, scale / 256, -(2^23 + 2^15) scale / 256) is code * scale with every intermediate exact
      const float q0 = s0 * 0.00390625f, q1 = s1 * 0.00390625f;
      const float2 m0 = make_float2(q0, q0), m1 = make_float2(q1, q1);
      const float2 c0 = make_float2(-8421376.0f * q0, -8421376.0f * q0), c1 = make_float2(-8421376.0f * q1, -8421376.0f * q1);
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const uint32_t wa = m[h][2 * (p >> 1)] ^ 0x80808080u, wb = m[h][2 * (p >> 1) + 1] ^ 0x80808080u;
        float2 a, c;
        if (p & 1) {
          a = make_float2(__uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7424)), __uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7434)));
          c = make_float2(__uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7424)), __uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7434)));
        } else {
          a = make_float2(__uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7404)), __uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7414)));
          c = make_float2(__uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7404)), __uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7414)));
        }
        a = __fmul2_rn(__ffma2_rn(a, m0, c0), decay_of(p));
        c = __fmul2_rn(__ffma2_rn(c, m1, c1), decay_of(p));
        acc[h][p][0] = a.x; acc[h][p][1] = a.y; acc[h][p][2] = c.x; acc[h][p][3] = c.y;
      }
    } else {
      // nibble n of a word is masked IN PLACE into 2^23's mantissa (n <= 4; nibbles 5, 6, 7 from the word shifted down
      // by 20): the float is 2^23 + u 16^e, minus (2^23 + 8 16^e) gives (u - 8) 16^e exactly, and the power of
      // sixteen goes into the scale.  Byte i of a word holds the pair (e, e') = (0,1), (2,3), (4,0), (1,2).
      constexpr float E0[4] = {1.0f, 256.0f, 65536.0f, 16.0f}, E1[4] = {16.0f, 4096.0f, 1.0f, 256.0f};
      const uint32_t w0 = m[h][0], w1 = m[h][1], w0s = w0 >> 20, w1s = w1 >> 20;
      const uint32_t K = 0x4B000000u;
      const float2 a[4] = {make_float2(nib_f<0x0000000Fu>(w0, K), nib_f<0x000000F0u>(w0, K)),
                           make_float2(nib_f<0x00000F00u>(w0, K), nib_f<0x0000F000u>(w0, K)),
                           make_float2(nib_f<0x000F0000u>(w0, K), nib_f<0x0000000Fu>(w0s, K)),
                           make_float2(nib_f<0x000000F0u>(w0s, K), nib_f<0x00000F00u>(w0s, K))};
      const float2 c[4] = {make_float2(nib_f<0x0000000Fu>(w1, K), nib_f<0x000000F0u>(w1, K)),
                           make_float2(nib_f<0x00000F00u>(w1, K), nib_f<0x0000F000u>(w1, K)),
                           make_float2(nib_f<0x000F0000u>(w1, K), nib_f<0x0000000Fu>(w1s, K)),
                           make_float2(nib_f<0x000000F0u>(w1s, K), nib_f<0x00000F00u>(w1s, K))};
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const float2 bias = make_float2(-(8388608.0f + 8.0f * E0[p]), -(8388608.0f + 8.0f * E1[p]));
        const float2 f0 = make_float2(s0 / E0[p], s0 / E1[p]), f1 = make_float2(s1 / E0[p], s1 / E1[p]);   // powers of two: exact
        const float2 av = __fmul2_rn(__fmul2_rn(__fadd2_rn(a[p], bias), f0), decay_of(p));
        const float2 cv = __fmul2_rn(__fmul2_rn(__fadd2_rn(c[p], bias), f1), decay_of(p));
        acc[h][p][0] = av.x; acc[h][p][1] = av.y; acc[h][p][2] = cv.x; acc[h][p][3] = cv.y;
      }
    }
  }
  // ---- the eight buffer slots ----
#pragma unroll
  for (int h = 0; h < NH; h++) {
    const uint32_t* kb = KBf + ((h0 + h) * 32 + lane) * 4;
    const uint4 k1 = *reinterpret_cast<const uint4*>(kb);
    const uint32_t r1[4] = {k1.x, k1.y, k1.z, k1.w};
    if constexpr (VDEC) {
      const uint4 k2 = *reinterpret_cast<const uint4*>(kb + 512), k3 = *reinterpret_cast<const uint4*>(kb + 1024);
      const uint32_t r2[4] = {k2.x, k2.y, k2.z, k2.w}, r3[4] = {k3.x, k3.y, k3.z, k3.w};
#pragma unroll
      for (int p = 0; p < 4; p++) {
        mma_bf16(acc[h][p], A1[0], A1[1], A1[0], A1[1], r1[p], r2[p]);      // p1 r1 + p1 r2
        mma_bf16(acc[h][p], A2[0], A2[1], A1[0], A1[1], r1[p], r3[p]);      // p2 r1 + p1 r3
        mma_bf16(acc[h][p], A2[0], A2[1], A3[0], A3[1], r2[p], r1[p]);      // p2 r2 + p3 r1
      }
    } else {
#pragma unroll
      for (int p = 0; p < 4; p++) mma_bf16(acc[h][p], A1[0], A1[1], A2[0], A2[1], r1[p], r1[p]);
#pragma unroll
      for (int p = 0; p < 4; p++) mma_bf16_k8(acc[h][p], A3[0], A3[1], r1[p]);
    }
  }
}
// The fresh scales of the two rows' groups and the rounded codes, in the layout fold_acc took them.  Returns the scale that
// lane t of the quad owns: row t & 1 of group t >> 1 (one group: lanes 2 and 3 hold copies).
template <int BITS, int UPG, int NH>
__device__ __forceinline__ float fold_round(const float (&acc)[NH][4][4], int lane, uint32_t (&o)[NH][4]) {
  constexpr int NS = UPG == 1 ? NH : 1;
  constexpr float QMAX = BITS == 4 ? 7.0f : 127.0f, MB = BITS == 4 ? MAGIC + 8.0f : MAGIC;
  const int t = lane & 3;
  // ---- fresh scales: absolute maxima over (row, group), index 2 group + row, over the quad ----
  float mx[2 * NS];
#pragma unroll
  for (int r = 0; r < 2; r++) {
#pragma unroll
    for (int s = 0; s < NS; s++) {
      float v = 0.f;
#pragma unroll
      for (int h = 0; h < NH / NS; h++) {
#pragma unroll
        for (int p = 0; p < 4; p++) v = max3_abs(v, acc[s * (NH / NS) + h][p][2 * r], acc[s * (NH / NS) + h][p][2 * r + 1]);
      }
      mx[2 * s + r] = v;
    }
  }
  float am;                                        // lane t of the quad: index t (two maxima: t & 1)
  if constexpr (NS == 2) {
    const bool up = (t & 2) != 0;
    const float x0 = __shfl_xor_sync(0xffffffffu, up ? mx[0] : mx[2], 2), x1 = __shfl_xor_sync(0xffffffffu, up ? mx[1] : mx[3], 2);
    mx[0] = fmaxf(up ? mx[2] : mx[0], x0);
    mx[1] = fmaxf(up ? mx[3] : mx[1], x1);
  }
  am = fmaxf((t & 1) ? mx[1] : mx[0], __shfl_xor_sync(0xffffffffu, (t & 1) ? mx[0] : mx[1], 1));
  if constexpr (NS == 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
  const float s_own = fp16_scale(am, QMAX);
  const bool fin = s_own <= 65504.0f;
  const float r_own = fin ? __frcp_rn(s_own) : 0.f, n_own = fin ? -s_own : 0.f;
  const bool tiny = __any_sync(0xffffffffu, s_own < FP16_MIN_NORMAL);
  float rc[2][NS], ns[2][NS];
#pragma unroll
  for (int s = 0; s < NS; s++) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      rc[r][s] = __shfl_sync(0xffffffffu, r_own, (lane & 28) + 2 * s + r);
      ns[r][s] = __shfl_sync(0xffffffffu, n_own, (lane & 28) + 2 * s + r);
    }
  }
  // ---- round ----
  float tv[NH][4][4];
#pragma unroll
  for (int h = 0; h < NH; h++) {
    const int s = UPG == 1 ? h : 0;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const float2 a = div_round2(make_float2(acc[h][p][0], acc[h][p][1]), make_float2(rc[0][s], rc[0][s]), make_float2(ns[0][s], ns[0][s]), MB);
      const float2 c = div_round2(make_float2(acc[h][p][2], acc[h][p][3]), make_float2(rc[1][s], rc[1][s]), make_float2(ns[1][s], ns[1][s]), MB);
      tv[h][p][0] = a.x; tv[h][p][1] = a.y; tv[h][p][2] = c.x; tv[h][p][3] = c.y;
    }
  }
  // only a scale in fp16's subnormal range (rounded far from absmax / qmax) lets a quotient round beyond qmax
  if (tiny) {
#pragma unroll
    for (int h = 0; h < NH; h++) {
#pragma unroll
      for (int p = 0; p < 4; p++) {
#pragma unroll
        for (int e = 0; e < 4; e++) tv[h][p][e] = fminf(fmaxf(tv[h][p][e], MB - QMAX), MB + QMAX);
      }
    }
  }
  // ---- repack into the fragment registers ----
  auto two = [](uint32_t a, uint32_t c) { return __byte_perm(a, c, 0x0040); };   // bytes (a, c)
  auto u = [](float f) { return __float_as_uint(f); };
#pragma unroll
  for (int h = 0; h < NH; h++) {
    const auto& v = tv[h];
    if constexpr (BITS == 8) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int p = i & 2, e = (i & 1) * 2;
        o[h][i] = __byte_perm(two(u(v[p][e]), u(v[p][e + 1])), two(u(v[p + 1][e]), u(v[p + 1][e + 1])), 0x5410);
      }
    } else {
      // a candidate's low 4 bits are code + 8 and the next 4 are zero, so lo + 16 hi has the packed byte at the bottom
      auto by = [](float lo, float hi) { return __float_as_uint(lo) + (__float_as_uint(hi) << 4); };
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int e = 2 * i;
        o[h][i] = __byte_perm(two(by(v[0][e], v[0][e + 1]), by(v[1][e], v[1][e + 1])),
                              two(by(v[2][e], v[2][e + 1]), by(v[3][e], v[3][e + 1])), 0x5410);
      }
    }
  }
  return s_own;
}

// Folds the 32 rows of warp w (two row blocks) of a stage.
//   st_addr / scs: the stage's codes and scales [row][NG] in shared memory, both rewritten in place.  The codes lie as the tensor-map
//   copy swizzles them (mma_pass.cuh: block bb = rows 32 w + 16 bb .., a thread's rows g and g + 8 of it)
//   ubt: the stage's buffered values [heads][8][DV] int8 (slots 0..6); udq: this token's rounded values [heads][DV]
//   tab: per head of the stage 8 floats dec_i (dec_7 unused), 8 floats value scales, then alpha; ksf: key scales [8]
// VDEC (KDA): decays per key channel: the start value is (code scale) ae[k], ae = exp(gnew); L carries no decay and no
// key scale (both are in the key fragments, three bf16 planes: build_key_frags_kda), and a product L Kd is taken as
// p1 r1 + p1 r2 + p2 r1 + p1 r3 + p2 r2 + p3 r1 (the three terms left out are below 2^-24 of it).
// READ: nothing is rounded or written back; the accumulators, i.e. the state advanced across the buffer, go to
// out [stage rows][DK] fp32 instead.  A thread of a quad has four adjacent columns of a row (8-bit: the quad stores 64 bytes at a
// time) or eight (4-bit): a whole 32-byte sector, stored as one where out allows.  As two 16-byte stores each writes half a
// sector, and the read-out is bound by the sectors it writes: 256 rows of 32 heads 149 us, 116 us as one.
//
// Bound by instruction issue (with its share of the step around it).  Two halves (64 columns, 32 values of a thread) are
// taken at once: independent chains for the scheduler, and the 2 or 4 fresh scales of a quad (rows x groups) are
// reduced by a transposing butterfly, computed by ONE lane each and exchanged.  Rounding is a branch-free exact division
// (div_round2).  One span at a time with a verified reciprocal the token that folds took a seventh longer (256 rows of 32 heads, 8-bit,
// with the step kernel of then: 141 us, 123 so).
template <int BITS, int UPG, int DV, bool VDEC = false, bool READ = false>
__device__ __forceinline__ void fold_stage_mma(uint32_t st_addr, unsigned short* scs, const int8_t* ubt, const float* udq,
                                               const float* tab, const float* ksf, const uint32_t* KBf, int w, int lane,
                                               const float* ae = nullptr, float* out = nullptr) {
  constexpr int DK = 128, NHALF = DK / 32, NG = NHALF / UPG, ROWB = DK * BITS / 8, TABW = 20;
  constexpr int DR = 8;                                // rows between a thread's two rows of a block
  static_assert(UPG == 1 || UPG == 2, "a scale group is one or two halves");
  const int g = lane >> 2, t = lane & 3;
  const uint32_t lrow = tile_lrow<BITS>(st_addr, w, lane, 0);
  const int hh = (32 * w) / DV;                        // head of the warp's rows within the stage
  const float* tb = tab + hh * TABW;
  const float2 al2 = make_float2(tb[16], tb[16]);
  [[maybe_unused]] const bool sectors = (reinterpret_cast<uintptr_t>(out) & 31) == 0;     // out on a 32-byte boundary: st_v8
  auto block = [&](int bb) {
    const int row0 = 32 * w + 16 * bb + g;             // stage rows row0, row0 + DR
    uint32_t A1[2], A2[2], A3[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int rv = row0 % DV + DR * r;
      fold_left<DV, VDEC>(ubt + hh * 8 * DV + rv, udq[hh * DV + rv], tb, ksf, t, A1[r], A2[r], A3[r]);
    }
    unsigned short* srow = scs + row0 * NG;
    // NH halves from half h0 on
    auto chunk = [&](auto nh, int h0) {
      constexpr int NH = decltype(nh)::value, NS = UPG == 1 ? NH : 1;      // halves; scale groups among them
      const uint32_t addr = (lrow + bb * 16 * ROWB) ^ ((BITS == 8 ? 32 : 16) * h0);         // chunks of half h0 on
      const int g0 = h0 / UPG;
      uint32_t m[NH][4];                               // 8-bit: (row, row + 1) x two 16-byte pieces; 4-bit: (row, row + 1)
      if constexpr (BITS == 8) {
#pragma unroll
        for (int h = 0; h < NH; h++) ldsm_x4(m[h], addr ^ (32 * h));
      } else {
        uint32_t x[4];
        ldsm_x4(x, addr);
        m[0][0] = x[0]; m[0][1] = x[1]; m[1][0] = x[2]; m[1][1] = x[3];
      }
      float sc[2][NS];
#pragma unroll
      for (int s = 0; s < NS; s++) { sc[0][s] = h2f(srow[g0 + s]); sc[1][s] = h2f(srow[DR * NG + g0 + s]); }
      float acc[NH][4][4];
      fold_acc<BITS, UPG, NH, VDEC>(m, sc, A1, A2, A3, KBf, h0, lane, al2, ae, acc);
      if constexpr (READ) {
        float* o0 = out + (long long)row0 * DK;
#pragma unroll
        for (int h = 0; h < NH; h++) {
#pragma unroll
          for (int r = 0; r < 2; r++) {
            float* p0 = o0 + r * DR * DK + fold_col<BITS>(h0 + h, 0, t);
            const auto& v = acc[h];
            if (BITS == 4 && sectors) {
              st_v8(p0, v[0][2 * r], v[0][2 * r + 1], v[1][2 * r], v[1][2 * r + 1], v[2][2 * r], v[2][2 * r + 1], v[3][2 * r], v[3][2 * r + 1]);
            } else {
              *reinterpret_cast<float4*>(p0) = make_float4(v[0][2 * r], v[0][2 * r + 1], v[1][2 * r], v[1][2 * r + 1]);
              *reinterpret_cast<float4*>(p0 + (BITS == 8 ? 16 : 4)) = make_float4(v[2][2 * r], v[2][2 * r + 1], v[3][2 * r], v[3][2 * r + 1]);
            }
          }
        }
        return;
      }
      uint32_t o[NH][4];
      const float s_own = fold_round<BITS, UPG, NH>(acc, lane, o);
      if (NS == 2 || t < 2) srow[(t & 1) * DR * NG + g0 + (NS == 2 ? t >> 1 : 0)] = f2h(s_own);   // (the old scales are in registers by now)
      if constexpr (BITS == 8) {
#pragma unroll
        for (int h = 0; h < NH; h++) stsm_x4(addr ^ (32 * h), o[h]);
      } else {
        const uint32_t x[4] = {o[0][0], o[0][1], o[1][0], o[1][1]};
        stsm_x4(addr, x);
      }
    };
#pragma unroll 1
    for (int h0 = 0; h0 + 2 <= NHALF; h0 += 2) chunk(IntC<2>(), h0);
  };
#pragma unroll 1
  for (int bb = 0; bb < 2; bb++) block(bb);
}

// The same fold for 4-bit codes scaled along v in groups of 32 rows (one scale per column and group).  Warp w owns
// group w of the stage (the warp's 32 rows), so a column's absolute maximum over the group is a
// reduction inside the warp.  The row is walked in four chunks of 32 columns (16 bytes: one ldmatrix.x2 per 16-row
// block); a thread holds 8 columns of 4 rows per chunk.  The reduction is a transposing butterfly over the eight lanes of
// one t, after which lane (i, t) computes the fresh scale of ONE column (the i-th of its eight) and the lanes exchange them.
//   scs: the stage's scales [4][128] fp16, rewritten in place; the other arguments as fold_stage_mma.
template <int DV>
__device__ __forceinline__ void fold_stage_mma_v4(uint32_t st_addr, unsigned short* scs, const int8_t* ubt, const float* udq,
                                                  const float* tab, const float* ksf, const uint32_t* KBf, int w, int lane) {
  constexpr int ROWB = 64, TABW = 20;
  constexpr float QMAX = 7.0f, MB = MAGIC + 8.0f;
  const int i = lane >> 2, t = lane & 3;
  const uint32_t lrow = tile_addr<4>(st_addr, 32 * w + (lane & 15), 0);
  const int hh = (32 * w) / DV;                        // the warp's 32 rows lie in one head
  const float* tb = tab + hh * TABW;
  const float2 al2 = make_float2(tb[16], tb[16]);
  // ---- A fragments: L of the thread's four rows (fragment rows i, i + 8 of blocks 0, 1) at slots 2t, 2t + 1 ----
  uint32_t A1[2][2], A2[2][2], A3[2][2];
#pragma unroll
  for (int bb = 0; bb < 2; bb++) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int rv0 = (32 * w + 16 * bb + i + 8 * r) % DV;
      fold_left<DV, false>(ubt + hh * 8 * DV + rv0, udq[hh * DV + rv0], tb, ksf, t, A1[bb][r], A2[bb][r], A3[bb][r]);
    }
  }
  constexpr float E0[4] = {1.0f, 256.0f, 65536.0f, 16.0f}, E1[4] = {16.0f, 4096.0f, 1.0f, 256.0f};   // see fold_stage_mma
#pragma unroll 1
  for (int c4 = 0; c4 < 4; c4++) {
    uint32_t wd[2][2];                                 // [block][fragment row i / i + 8]: 8 nibbles = this thread's 8 columns
    ldsm_x2(wd[0], lrow ^ (16 * c4));
    ldsm_x2(wd[1], (lrow ^ (16 * c4)) + 16 * ROWB);
    unsigned short* scol = scs + w * 128 + 32 * c4 + 8 * t;                  // the thread's 8 column scales
    const uint4 sw = *reinterpret_cast<const uint4*>(scol);
    const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sw.x)), s23 = __half22float2(*reinterpret_cast<const __half2*>(&sw.y));
    const float2 s45 = __half22float2(*reinterpret_cast<const __half2*>(&sw.z)), s67 = __half22float2(*reinterpret_cast<const __half2*>(&sw.w));
    const float2 so[4] = {s01, s23, s45, s67};
    float acc[2][4][4];
    // ---- start values: (code * scale) * alpha ----
#pragma unroll
    for (int bb = 0; bb < 2; bb++) {
      const uint32_t w0 = wd[bb][0], w1 = wd[bb][1], w0s = w0 >> 20, w1s = w1 >> 20;
      const uint32_t K = 0x4B000000u;
      float2 a[4], c[4];
      a[0] = make_float2(nib_f<0x0000000Fu>(w0, K), nib_f<0x000000F0u>(w0, K));
      a[1] = make_float2(nib_f<0x00000F00u>(w0, K), nib_f<0x0000F000u>(w0, K));
      a[2] = make_float2(nib_f<0x000F0000u>(w0, K), nib_f<0x0000000Fu>(w0s, K));
      a[3] = make_float2(nib_f<0x000000F0u>(w0s, K), nib_f<0x00000F00u>(w0s, K));
      c[0] = make_float2(nib_f<0x0000000Fu>(w1, K), nib_f<0x000000F0u>(w1, K));
      c[1] = make_float2(nib_f<0x00000F00u>(w1, K), nib_f<0x0000F000u>(w1, K));
      c[2] = make_float2(nib_f<0x000F0000u>(w1, K), nib_f<0x0000000Fu>(w1s, K));
      c[3] = make_float2(nib_f<0x000000F0u>(w1s, K), nib_f<0x00000F00u>(w1s, K));
#pragma unroll
      for (int b4 = 0; b4 < 4; b4++) {
        const float2 f = make_float2(so[b4].x / E0[b4], so[b4].y / E1[b4]);     // powers of two: exact
        const float2 bias = make_float2(-(8388608.0f + 8.0f * E0[b4]), -(8388608.0f + 8.0f * E1[b4]));
        const float2 av = __fmul2_rn(__fmul2_rn(__fadd2_rn(a[b4], bias), f), al2);
        const float2 cv = __fmul2_rn(__fmul2_rn(__fadd2_rn(c[b4], bias), f), al2);
        acc[bb][b4][0] = av.x; acc[bb][b4][1] = av.y; acc[bb][b4][2] = cv.x; acc[bb][b4][3] = cv.y;
      }
    }
    // ---- the eight buffer slots ----
    const uint4 k4 = *reinterpret_cast<const uint4*>(KBf + (c4 * 32 + lane) * 4);
    const uint32_t kw[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
    for (int bb = 0; bb < 2; bb++) {
#pragma unroll
      for (int q = 0; q < 4; q++) mma_bf16(acc[bb][q], A1[bb][0], A1[bb][1], A2[bb][0], A2[bb][1], kw[q], kw[q]);
#pragma unroll
      for (int q = 0; q < 4; q++) mma_bf16_k8(acc[bb][q], A3[bb][0], A3[bb][1], kw[q]);
    }
    // ---- fresh scales: a column's absolute maximum over the group's 32 rows ----
    float cm[8];
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
      for (int e = 0; e < 2; e++)
        cm[2 * q + e] = fmaxf(max3_abs(acc[0][q][e], acc[0][q][2 + e], acc[1][q][e]), fabsf(acc[1][q][2 + e]));
    }
    // transposing butterfly over the eight lanes of one t: lane (i, t) ends up with column i of the thread's eight
#pragma unroll
    for (int hw = 4; hw >= 1; hw >>= 1) {
      const bool up = (i & hw) != 0;
#pragma unroll
      for (int x = 0; x < hw; x++) {
        const float other = __shfl_xor_sync(0xffffffffu, up ? cm[x] : cm[x + hw], 4 * hw);
        cm[x] = fmaxf(up ? cm[x + hw] : cm[x], other);
      }
    }
    const float sc_mine = fp16_scale(cm[0], QMAX);
    const bool fin = sc_mine <= 65504.0f;
    const float rc_mine = fin ? __frcp_rn(sc_mine) : 0.f, ns_mine = fin ? -sc_mine : 0.f;
    const bool tiny = __any_sync(0xffffffffu, sc_mine < FP16_MIN_NORMAL);
    __syncwarp();                                      // every lane has read the chunk's old scales
    scol[i] = f2h(sc_mine);
    float2 rn[4], sn[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      rn[q] = make_float2(__shfl_sync(0xffffffffu, rc_mine, 8 * q + t), __shfl_sync(0xffffffffu, rc_mine, 8 * q + 4 + t));
      sn[q] = make_float2(__shfl_sync(0xffffffffu, ns_mine, 8 * q + t), __shfl_sync(0xffffffffu, ns_mine, 8 * q + 4 + t));
    }
    // ---- round (one scale and reciprocal per column) and repack ----
    uint32_t o[2][2];
#pragma unroll
    for (int bb = 0; bb < 2; bb++) {
      float tv[4][4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float2 a = div_round2(make_float2(acc[bb][q][0], acc[bb][q][1]), rn[q], sn[q], MB);
        const float2 c = div_round2(make_float2(acc[bb][q][2], acc[bb][q][3]), rn[q], sn[q], MB);
        tv[q][0] = a.x; tv[q][1] = a.y; tv[q][2] = c.x; tv[q][3] = c.y;
      }
      if (tiny) {                    // only a scale in fp16's subnormal range lets a quotient pass qmax
#pragma unroll
        for (int b4 = 0; b4 < 4; b4++) {
#pragma unroll
          for (int e = 0; e < 4; e++) tv[b4][e] = fminf(fmaxf(tv[b4][e], MB - QMAX), MB + QMAX);
        }
      }
      auto two = [](uint32_t a, uint32_t c) { return __byte_perm(a, c, 0x0040); };
      auto by = [](float lo, float hi) { return __float_as_uint(lo) + (__float_as_uint(hi) << 4); };
      o[bb][0] = __byte_perm(two(by(tv[0][0], tv[0][1]), by(tv[1][0], tv[1][1])), two(by(tv[2][0], tv[2][1]), by(tv[3][0], tv[3][1])), 0x5410);
      o[bb][1] = __byte_perm(two(by(tv[0][2], tv[0][3]), by(tv[1][2], tv[1][3])), two(by(tv[2][2], tv[2][3]), by(tv[3][2], tv[3][3])), 0x5410);
    }
    __syncwarp();                                      // every lane has read the chunk's codes
    stsm_x2(lrow ^ (16 * c4), o[0][0], o[0][1]);
    stsm_x2((lrow ^ (16 * c4)) + 16 * ROWB, o[1][0], o[1][1]);
  }
}

// The same for 8-bit codes scaled along v: a chunk is 32 columns = 32 bytes of
// a row, one ldmatrix.x4 per 16-row block; a thread holds columns 4t .. 4t + 3 and 16 + 4t .. 16 + 4t + 3 of the chunk
// (N-block q: half q >> 1, byte pair q & 1) of four rows.
template <int DV>
__device__ __forceinline__ void fold_stage_mma_v8(uint32_t st_addr, unsigned short* scs, const int8_t* ubt, const float* udq,
                                                  const float* tab, const float* ksf, const uint32_t* KBf, int w, int lane) {
  constexpr int TABW = 20;
  constexpr float QMAX = 127.0f, MB = MAGIC;
  const int i = lane >> 2, t = lane & 3;
  const uint32_t lrow = tile_lrow<8>(st_addr, w, lane, 0);
  const int hh = (32 * w) / DV;
  const float* tb = tab + hh * TABW;
  const float2 al2 = make_float2(tb[16], tb[16]);
  uint32_t A1[2][2], A2[2][2], A3[2][2];
#pragma unroll
  for (int bb = 0; bb < 2; bb++) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int rv0 = (32 * w + 16 * bb + i + 8 * r) % DV;
      fold_left<DV, false>(ubt + hh * 8 * DV + rv0, udq[hh * DV + rv0], tb, ksf, t, A1[bb][r], A2[bb][r], A3[bb][r]);
    }
  }
#pragma unroll 1
  for (int c4 = 0; c4 < 4; c4++) {
    uint32_t m[2][4];
    ldsm_x4(m[0], lrow ^ (32 * c4));
    ldsm_x4(m[1], (lrow ^ (32 * c4)) + 16 * 128);
    // the thread's 8 column scales: columns 4t .. 4t + 3 and 16 + 4t .. 16 + 4t + 3 of the chunk
    unsigned short* scol = scs + w * 128 + 32 * c4 + 4 * t;
    const uint2 swa = *reinterpret_cast<const uint2*>(scol), swb = *reinterpret_cast<const uint2*>(scol + 16);
    const float2 so[4] = {__half22float2(*reinterpret_cast<const __half2*>(&swa.x)), __half22float2(*reinterpret_cast<const __half2*>(&swa.y)),
                          __half22float2(*reinterpret_cast<const __half2*>(&swb.x)), __half22float2(*reinterpret_cast<const __half2*>(&swb.y))};
    float acc[2][4][4];
    // ---- start values: (code * scale) * alpha (fold_stage_mma's exact byte-in-mantissa product, one scale per column) ----
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 mq = make_float2(so[q].x * 0.00390625f, so[q].y * 0.00390625f);
      const float2 cq = make_float2(-8421376.0f * mq.x, -8421376.0f * mq.y);
#pragma unroll
      for (int bb = 0; bb < 2; bb++) {
        const uint32_t wa = m[bb][2 * (q >> 1)] ^ 0x80808080u, wb = m[bb][2 * (q >> 1) + 1] ^ 0x80808080u;
        float2 a, c;
        if (q & 1) {
          a = make_float2(__uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7424)), __uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7434)));
          c = make_float2(__uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7424)), __uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7434)));
        } else {
          a = make_float2(__uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7404)), __uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7414)));
          c = make_float2(__uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7404)), __uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7414)));
        }
        a = __fmul2_rn(__ffma2_rn(a, mq, cq), al2);
        c = __fmul2_rn(__ffma2_rn(c, mq, cq), al2);
        acc[bb][q][0] = a.x; acc[bb][q][1] = a.y; acc[bb][q][2] = c.x; acc[bb][q][3] = c.y;
      }
    }
    // ---- the eight buffer slots ----
    const uint4 k4 = *reinterpret_cast<const uint4*>(KBf + (c4 * 32 + lane) * 4);
    const uint32_t kw[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
    for (int bb = 0; bb < 2; bb++) {
#pragma unroll
      for (int q = 0; q < 4; q++) mma_bf16(acc[bb][q], A1[bb][0], A1[bb][1], A2[bb][0], A2[bb][1], kw[q], kw[q]);
#pragma unroll
      for (int q = 0; q < 4; q++) mma_bf16_k8(acc[bb][q], A3[bb][0], A3[bb][1], kw[q]);
    }
    // ---- fresh scales: a column's absolute maximum over the group's 32 rows ----
    float cm[8];
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
      for (int e = 0; e < 2; e++)
        cm[2 * q + e] = fmaxf(max3_abs(acc[0][q][e], acc[0][q][2 + e], acc[1][q][e]), fabsf(acc[1][q][2 + e]));
    }
    // transposing butterfly over the eight lanes of one t: lane (i, t) ends up with column i of the thread's eight
#pragma unroll
    for (int hw = 4; hw >= 1; hw >>= 1) {
      const bool up = (i & hw) != 0;
#pragma unroll
      for (int x = 0; x < hw; x++) {
        const float other = __shfl_xor_sync(0xffffffffu, up ? cm[x] : cm[x + hw], 4 * hw);
        cm[x] = fmaxf(up ? cm[x + hw] : cm[x], other);
      }
    }
    const float sc_mine = fp16_scale(cm[0], QMAX);
    const bool fin = sc_mine <= 65504.0f;
    const float rc_mine = fin ? __frcp_rn(sc_mine) : 0.f, ns_mine = fin ? -sc_mine : 0.f;
    const bool tiny = __any_sync(0xffffffffu, sc_mine < FP16_MIN_NORMAL);
    __syncwarp();                                      // every lane has read the chunk's old scales
    scol[(i >> 2) * 16 + (i & 3)] = f2h(sc_mine);      // column i of the thread's eight: (q, e) = (i >> 1, i & 1)
    float2 rn[4], sn[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      rn[q] = make_float2(__shfl_sync(0xffffffffu, rc_mine, 8 * q + t), __shfl_sync(0xffffffffu, rc_mine, 8 * q + 4 + t));
      sn[q] = make_float2(__shfl_sync(0xffffffffu, ns_mine, 8 * q + t), __shfl_sync(0xffffffffu, ns_mine, 8 * q + 4 + t));
    }
    // ---- round (one scale and reciprocal per column) and repack ----
#pragma unroll
    for (int bb = 0; bb < 2; bb++) {
      float tv[4][4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float2 a = div_round2(make_float2(acc[bb][q][0], acc[bb][q][1]), rn[q], sn[q], MB);
        const float2 c = div_round2(make_float2(acc[bb][q][2], acc[bb][q][3]), rn[q], sn[q], MB);
        tv[q][0] = a.x; tv[q][1] = a.y; tv[q][2] = c.x; tv[q][3] = c.y;
      }
      if (tiny) {                    // only a scale in fp16's subnormal range lets a quotient pass qmax
#pragma unroll
        for (int q = 0; q < 4; q++) {
#pragma unroll
          for (int e = 0; e < 4; e++) tv[q][e] = fminf(fmaxf(tv[q][e], MB - QMAX), MB + QMAX);
        }
      }
      auto two = [](uint32_t a, uint32_t c) { return __byte_perm(a, c, 0x0040); };
      auto u = [](float f) { return __float_as_uint(f); };
      uint32_t o[4];
      o[0] = __byte_perm(two(u(tv[0][0]), u(tv[0][1])), two(u(tv[1][0]), u(tv[1][1])), 0x5410);
      o[1] = __byte_perm(two(u(tv[0][2]), u(tv[0][3])), two(u(tv[1][2]), u(tv[1][3])), 0x5410);
      o[2] = __byte_perm(two(u(tv[2][0]), u(tv[2][1])), two(u(tv[3][0]), u(tv[3][1])), 0x5410);
      o[3] = __byte_perm(two(u(tv[2][2]), u(tv[2][3])), two(u(tv[3][2]), u(tv[3][3])), 0x5410);
      __syncwarp();                                    // every lane has read the block's codes of this chunk
      stsm_x4((lrow ^ (32 * c4)) + bb * 16 * 128, o);
    }
  }
}

}  // namespace sqb
