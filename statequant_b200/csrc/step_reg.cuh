// The fused decode step with the state held in REGISTERS: bf16 states of d_k 128, and 4- / 8-bit states of d_k 128 or 96 scaled
// along k (groups of 64 / 32, the last one of 96 columns short); decays per head (Gated DeltaNet, Mamba2), int8 buffer of 8,
// q / k per key head.
//
// One CTA per batch row and head, a thread per state row: a head of d_v 128 or 192, or two heads of d_v 64 (of one key head).  Warp w owns rows 32 w .. 32 w + 31 = two blocks of 16; lane (g, t) = (lane / 4, lane % 4) loads rows g and g + 8 of
// a block, columns 32 j + 8 t .. + 7 of every unit j of 32 columns: one load each (16 bytes of bf16, 8 of int8, 4 of int4),
// all requested before anything waits.  A loaded word is a register of a matrix instruction's A fragment as it stands (the
// order of the columns along the contraction is free as long as B follows it) and, on the token that folds, part of a C
// fragment as well: the state is read once, never passes through shared memory and goes back by stores of the registers it
// came into.
//
// Read-out, bf16: q and k are cut into three bf16 pieces each (8 + 8 + 8 mantissa bits: exact), the columns of B; every
// product is exact; 16 columns at a time are summed from zero by the tensor core, the eight sums in an fp32 tree.  Columns 0, 1, 2 are
// the pieces of q, 4, 5, 6 those of k, so that the thread pair t = 0, 1 holds the parts of q and t = 2, 3 those of k.  The vectors
// are scaled below 2^-15 for this, so that 128 products with states up to the format's maximum do not overflow.
// Integer states: the byte digits of mma_pass.cuh, exact integer sums.
// Fold: fold_mma.cuh's (three bf16 pieces of L against the int8 key codes), accumulators started at decay * state.
//
// HBM-bound by intent (a CTA's whole state is in flight at once); small grids are bound by the serial chain idx -> state and
// prologue -> read-out -> append, which is why q and k are taken as they come and their norms applied to the finished sums.
// Measured per layer and token, generic kernel -> this one (the generic kernel's CTA goes through six block reductions before
// its state pass and holds 12 warps per SM): bf16, 96 rows of 32 heads of 128 x 128, 120 -> 29.6 us (18 us at the copy rate);
// 4-bit, 64 rows of 30 heads of 96 x 192, a slot in eight folding, 103 -> 25.2 us.  Against the tensor-core kernel: sqb200.cu.
//
// Not taken, and left to the kernels that had them: integer states scaled along v (a column's scale would have to go into the
// vectors, a set of fragments per scale group), decays per key channel (fragments per buffer slot), other key groups than those
// of the presets, and d_k 96 with bf16 states or Mamba2.
#pragma once
#include "launchers.h"
#include "step_tma.cuh"
#include "fold_mma.cuh"

namespace sqb {

// Threads per SM: bf16 holds 64 words of state per thread (128 registers); integer states of d_k 128 come here in grids of up
// to four CTAs per SM, and need the registers more than the residency; those of d_k 96 in grids of any size (80 registers:
// 852 us a pass against 955 us with 112).  What the caps cost (ptxas): 96-wide instances spill 4 .. 56 bytes (4 .. 64
// loaded), bf16 ones up to 20 (36), integer ones of d_k 128 nothing.  (No lambda in this kernel captures by reference what another part
// of it keeps in registers: one that did cost the bf16 instances 20 bytes of spills and 9 % of their time.)
constexpr int reg_min_ctas(int bits, int dk, int threads) { return (bits == 16 || dk == 128 ? 512 : 768) / threads; }

// N words of a lane's slice of a unit: 4 (bf16), 2 (int8) or 1 (int4)
template <int N>
__device__ __forceinline__ void ld_words(uint32_t* r, const uint8_t* p) {
  if constexpr (N == 4) { const uint4 v = *reinterpret_cast<const uint4*>(p); r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w; }
  else if constexpr (N == 2) { const uint2 v = *reinterpret_cast<const uint2*>(p); r[0] = v.x; r[1] = v.y; }
  else r[0] = *reinterpret_cast<const uint32_t*>(p);
}
template <int N>
__device__ __forceinline__ void st_words(uint8_t* p, const uint32_t* r) {
  if constexpr (N == 4) *reinterpret_cast<uint4*>(p) = make_uint4(r[0], r[1], r[2], r[3]);
  else if constexpr (N == 2) *reinterpret_cast<uint2*>(p) = make_uint2(r[0], r[1]);
  else *reinterpret_cast<uint32_t*>(p) = r[0];
}

// the NG scales of a row as packed words: one load where the row's scales are an aligned 4 or 8 bytes
template <int NG>
__device__ __forceinline__ void ld_scales(uint32_t* r, const unsigned short* p) {
  if constexpr (NG == 4) { const uint2 v = *reinterpret_cast<const uint2*>(p); r[0] = v.x; r[1] = v.y; }
  else if constexpr (NG == 2) r[0] = *reinterpret_cast<const uint32_t*>(p);
  else {
    r[0] = p[0];
    if constexpr (NG > 1) r[0] |= static_cast<uint32_t>(p[1]) << 16;
    if constexpr (NG > 2) r[1] = p[2];
  }
}
__device__ __forceinline__ float scale_of(const uint32_t* r, int i) { return h2f(static_cast<unsigned short>(r[i >> 1] >> (16 * (i & 1)))); }

// The gates of value head h (one lane per head calls it): g, beta | dt, gcur, exp(gcur), exp(g), gcur + g, D into o[0 .. 6].
// In two steps, so that the loads of a warp are in flight before their first use.
struct GateRaw { uint32_t r[4]; float gcur; };
template <int KIND>
__device__ __forceinline__ GateRaw gates_load(const StepArgs& A, int b, int h, const float* GCseq) {
  GateRaw w;
  w.r[0] = w.r[1] = w.r[2] = w.r[3] = 0u;
  if (KIND == K_GDN) {
    if (A.gate) {
      w.r[0] = ld1_raw(A.a + (long long)b * A.sa, A.dt_ab, h); w.r[1] = ld1_raw(A.dt_bias, A.dt_dtb, h);
      w.r[2] = ld1_raw(A.A_log, A.dt_alog, h);                 w.r[3] = ld1_raw(A.b + (long long)b * A.sb, A.dt_ab, h);
    } else {
      w.r[0] = ld1_raw(A.g + (long long)b * A.sg, A.dt_g, h);  w.r[1] = ld1_raw(A.beta + (long long)b * A.sbeta, A.dt_g, h);
    }
  } else {
    w.r[0] = ld1_raw(A.g + (long long)b * A.sg, A.dt_g, h);
    if (A.dt_bias) w.r[1] = ld1_raw(A.dt_bias, A.dt_dtb, h);
    w.r[2] = ld1_raw(A.A_log, A.dt_alog, h);
    if (A.beta) w.r[3] = ld1_raw(A.beta, A.dt_beta, h);
  }
  w.gcur = GCseq[h];
  return w;
}
template <int KIND>
__device__ __forceinline__ void gates_finish(const StepArgs& A, const GateRaw& w, float* o) {
  float g, bt, Dv = 0.f;
  if (KIND == K_GDN) {
    if (A.gate) {
      const float x = cvt_raw(w.r[0], A.dt_ab) + cvt_raw(w.r[1], A.dt_dtb);
      const float sp = x <= 20.0f ? logf(1.0f + expf(x)) : x;
      g = -expf(cvt_raw(w.r[2], A.dt_alog)) * sp;
      bt = __fdiv_rn(1.0f, 1.0f + expf(-cvt_raw(w.r[3], A.dt_ab)));
    } else {
      g = cvt_raw(w.r[0], A.dt_g);
      bt = cvt_raw(w.r[1], A.dt_g);
    }
  } else {
    float dtv = cvt_raw(w.r[0], A.dt_g);
    if (A.dt_bias) dtv = dtv + cvt_raw(w.r[1], A.dt_dtb);
    if (A.dt_softplus) dtv = dtv <= 20.0f ? logf(1.0f + expf(dtv)) : dtv;
    if (A.dt_clamp) dtv = fminf(fmaxf(dtv, A.dt_min), A.dt_max);
    g = __fmul_rn(cvt_raw(w.r[2], A.dt_alog), dtv);
    bt = dtv;
    if (A.beta) Dv = cvt_raw(w.r[3], A.dt_beta);
  }
  o[0] = g; o[1] = bt; o[2] = w.gcur; o[3] = expf(w.gcur); o[4] = expf(g); o[5] = w.gcur + g; o[6] = Dv;
}

// the sum of a hi + mid + lo triple whose lower parts may be 0 * inf: a hi part that is not finite stands alone
__device__ __forceinline__ float add_parts(float hi, float lo) { return fabsf(hi) <= 3.402823466e38f ? hi + lo : hi; }

// The fold of NH units, from unit h0 on, of a block's rows g and g + 8 (words w0, w1; scales sc by group): fresh codes to Sx (the
// lane's place in row g of the block) and scales to SCx.
template <int BITS, int UPG, int NH, int NG, int ROWB>
__device__ __forceinline__ void reg_fold_chunk(const uint32_t* w0, const uint32_t* w1, const float (&sc)[2][UPG == 1 ? NH : 1],
                                               const uint32_t (&A1)[2], const uint32_t (&A2)[2], const uint32_t (&A3)[2],
                                               const uint32_t* KBf, int h0, int lane, float2 al2, uint8_t* Sx, unsigned short* SCx) {
  constexpr int NS = UPG == 1 ? NH : 1, WPU = BITS / 4;
  const int t = lane & 3;
  uint32_t m[NH][4], o[NH][4];
  float acc[NH][4][4];
#pragma unroll
  for (int n = 0; n < NH; n++) {
#pragma unroll
    for (int p = 0; p < WPU; p++) { m[n][2 * p] = w0[n * WPU + p]; m[n][2 * p + 1] = w1[n * WPU + p]; }
  }
  fold_acc<BITS, UPG, NH, false>(m, sc, A1, A2, A3, KBf, h0, lane, al2, nullptr, acc);
  const float s_own = fold_round<BITS, UPG, NH>(acc, lane, o);
  if (NS == 2 || t < 2) SCx[8 * (t & 1) * NG + h0 / UPG + (NS == 2 ? t >> 1 : 0)] = f2h(s_own);
#pragma unroll
  for (int n = 0; n < NH; n++) {
    uint32_t a[WPU], c[WPU];
#pragma unroll
    for (int p = 0; p < WPU; p++) { a[p] = o[n][2 * p]; c[p] = o[n][2 * p + 1]; }
    st_words<WPU>(Sx + 4 * BITS * (h0 + n), a);
    st_words<WPU>(Sx + 8 * ROWB + 4 * BITS * (h0 + n), c);
  }
}

template <int KIND, int BITS, int DK, int DV, int HPS, bool BIO>
__global__ void __launch_bounds__(HPS * DV, reg_min_ctas(BITS, DK, HPS * DV)) step_reg_kernel(const __grid_constant__ StepArgs A) {
  dependency_wait();
  dependency_release();
  constexpr int NT = HPS * DV, M = 8, WPH = DV / 32, NU = DK / 32, CW = 4, ROWB = DK * BITS / 8;
  constexpr int WPU = BITS / 4, UPG = BITS == 4 ? 2 : 1, NG = BITS == 16 ? 1 : (NU + UPG - 1) / UPG;
  constexpr bool TWO = KIND != K_M2, QUANT = BITS != 16;
  constexpr int TOP = QUANT ? 29 : -16;                    // q and k lie below 2^(TOP + 1); the byte digits want 2^30
  constexpr float UPF = QUANT ? 1.0f : 35184372088832.0f;  // 2^(29 - TOP)
  __shared__ __align__(16) uint2 Bf[QUANT ? 1 : 2 * NU * 32];          // bf16: B fragments of the state pass (bf16 pieces)
  __shared__ __align__(16) uint32_t Bf8[2 * 4 * 32];       // B fragments of byte codes (byte digits): key tile, int8 state
  __shared__ __align__(16) uint32_t Bf4[BITS == 4 ? 2 * 4 * 32 : 1];   // B fragments of nibble codes
  __shared__ __align__(16) uint32_t KBf[DK * 4];           // key fragments of the fold
  __shared__ __align__(16) uint32_t Lp[NT * 12];          // the fold's L: per row three pieces of eight bf16
  __shared__ __align__(16) int8_t kbt[M * DK];
  __shared__ __align__(16) int8_t kcur[DK];
  __shared__ __align__(16) float hd[HPS * HD_W];
  __shared__ float2 dcu[HPS * M], dqk[M];
  __shared__ float gbs[HPS * M], ksf[M], tab[HPS * 20], red[NT / 32], misc[12];

  const int dt_qk = BIO ? static_cast<int>(DT_BF16) : A.dt_qk, dt_v = BIO ? static_cast<int>(DT_BF16) : A.dt_v,
            dt_out = BIO ? static_cast<int>(DT_BF16) : A.dt_out;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int b = blockIdx.x, h0 = blockIdx.y * HPS, hk = h0 / A.gqa_full;
  const bool first = h0 == hk * A.gqa_full;                // the CTA that appends the key head's key
  const int osz = dt_size(dt_out);
  // Roles: warp 0 makes the fragments of q and k; in a CTA of six warps of q only, and warp 4 those of k (everybody waits for the
  // longest of them: 96 x 192, int4 k/64, 64 rows of 30 heads 24.9 -> 20.5 us; in a CTA of four warps another warp's work would have to
  // move for it, and a small grid loses 4 %); warp 1 the gates, warp 2 the decays, warp 3 the norms and the key.
  constexpr int NVEC = NT > 128 ? 1 : 2;
  const bool makes = warp == 0 || (NVEC == 1 && warp == 4);
  const int vec0 = warp == 0 ? 0 : 1;
  // q and k leave before the slot index is known
  Raw4 rqk[2];
#pragma unroll
  for (int v = 0; v < 2; v++) { rqk[v].v = make_uint4(0u, 0u, 0u, 0u); rqk[v].vec = false; }
  const bool has_col = lane * CW < DK;                     // four columns per lane
  if (has_col && (makes || warp == 3)) {
    const uint8_t *q = A.q + (long long)b * A.sq, *k = A.k + (long long)b * A.sk;
    rqk[0] = ld4_raw<BIO>(NVEC == 1 && warp == 4 ? k : q, dt_qk, (long long)hk * DK + lane * CW);
    if (NVEC == 2 || warp == 3) rqk[1] = ld4_raw<BIO>(k, dt_qk, (long long)hk * DK + lane * CW);
  }
  long long seq = b;
  if (A.idx != nullptr) {
    seq = A.idx[b];
    if (seq <= 0) {
      uint8_t* orow = A.out + (long long)b * A.so + (long long)h0 * DV * osz;
      for (int v = tid; v < HPS * DV; v += NT) stf(orow, dt_out, v, 0.0f);
      return;
    }
  }
  int* NPseq = reinterpret_cast<int*>(A.NPTR + seq * A.sN);
  uint8_t* KBh = A.KB + seq * A.sKB + (long long)hk * M * DK;
  uint8_t* UBseq = A.UB + seq * A.sUB;
  unsigned short* KBSh = reinterpret_cast<unsigned short*>(A.KBS + seq * A.sKBS) + hk * M;
  unsigned short* UBSseq = reinterpret_cast<unsigned short*>(A.UBS + seq * A.sUBS);
  float* GBseq = reinterpret_cast<float*>(A.GB + seq * A.sGB);
  float* GCseq = reinterpret_cast<float*>(A.GCUR + seq * A.sGC);

  // ---- every fetch: a role's small ones first (they head the serial chains), then the state, then the buffered values --
  uint2 kw[NU];                                            // fragments' warps: slot g of the key tile, its 8 columns of every unit
  float ksl = 0.f;
  GateRaw gr;
  int nraw = 0;
  float gb0 = 0.f, gc0 = 0.f;
  unsigned short us0 = 0;
  if (makes) {
#pragma unroll
    for (int u = 0; u < NU; u++) kw[u] = *reinterpret_cast<const uint2*>(KBh + g * DK + 32 * u + 8 * t);
    ksl = h2f(KBSh[g]);
  } else if (warp == 1) {
    gr.r[0] = gr.r[1] = gr.r[2] = gr.r[3] = 0u; gr.gcur = 0.f;
    if (lane < HPS) gr = gates_load<KIND>(A, b, h0 + lane, GCseq);
  } else if (warp == 2) {
    nraw = NPseq[h0];                                      // the heads of a slot advance together
    if (lane < HPS * M) {
      gb0 = GBseq[(long long)h0 * M + lane]; gc0 = GCseq[h0 + lane / M];
      us0 = UBSseq[h0 * M + lane];
    }
  }
  const int hw = warp / WPH, h = h0 + hw, rv0 = (warp % WPH) * 32;       // this warp's head and its first row in it
  const long long row0 = (long long)h * DV + rv0 + g;      // row g of the warp's first block
  uint8_t* Srow = A.S + seq * A.sS + row0 * ROWB + BITS * t;
  uint32_t sw[2][2][NU * WPU];                             // [block][row g, row g + 8][unit, word]
  uint32_t scr[2][2][(NG + 1) / 2];                        // their scales, two to a word
  unsigned short* SCrow = nullptr;
  if (QUANT) SCrow = reinterpret_cast<unsigned short*>(A.SC + seq * A.sSC) + row0 * NG;
#pragma unroll
  for (int x = 0; x < 2; x++) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
#pragma unroll
      for (int u = 0; u < NU; u++) ld_words<WPU>(&sw[x][r][u * WPU], Srow + (16 * x + 8 * r) * ROWB + 4 * BITS * u);
      if constexpr (QUANT) {
        ld_scales<NG>(scr[x][r], SCrow + (16 * x + 8 * r) * NG);
      }
    }
  }
  const int rv = rv0 + 8 * t + g;                          // the row this lane finishes: block t / 2, half t % 2
  const uint32_t rvt = ld1_raw(A.v + (long long)b * A.sv, dt_v, (long long)h * DV + rv);
  int8_t ub[M - 1];
#pragma unroll
  for (int i = 0; i < M - 1; i++) ub[i] = static_cast<int8_t>(UBseq[((long long)h * M + i) * DV + rv]);

  // ---- prologue, by role ----------------------------------------------------------------------------------------
  uint32_t kword = 0;                                      // warp 3: the key as it goes into the buffer
  float kscale = 0.f;
  if (makes) {
    // q and k as they come, scaled by powers of two (integer states: 30-bit fixed point, mma_pass.cuh); what their norms make
    // of the results, warp 3 finds out meanwhile and every row applies at the end.  (Mamba2 reads the state against q only.)
    float x[NVEC][CW], mx[NVEC], d = 0.f;
    FxScale fx[NVEC];
#pragma unroll
    for (int v = 0; v < NVEC; v++) {
      cvt4_raw<BIO>(rqk[v], dt_qk, x[v]);
      mx[v] = 0.f;
#pragma unroll
      for (int j = 0; j < CW; j++) mx[v] = fmaxf(mx[v], fabsf(x[v][j]));
    }
#pragma unroll
    for (int v = 0; v < NVEC; v++) {
      mx[v] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx[v])));
      fx[v] = fx_scale<TOP>(mx[v]);
    }
#pragma unroll
    for (int j = 0; j < CW; j++) {
      if (NVEC == 2 && KIND == K_M2) d += x[NVEC - 1][j] * x[0][j];        // C . B as it is
#pragma unroll
      for (int v = 0; v < NVEC; v++) x[v][j] = (x[v][j] * fx[v].m1) * fx[v].m2;
      if (NVEC == 2 && KIND != K_M2) d += x[NVEC - 1][j] * x[0][j];        // (the vectors' norms still missing, so not to overflow or vanish)
    }
    // bf16: the state pass's fragments: lane l's columns 4 l .. 4 l + 3 are step l / 8 * 2 + l % 2, thread (l % 8) / 2
    if constexpr (!QUANT) {
#pragma unroll
      for (int v = 0; v < NVEC; v++) {
        uint2* bw = Bf + (2 * (lane >> 3) + (lane & 1)) * 32 + ((lane & 7) >> 1) + 16 * (vec0 + v);
        const bool on = TWO || vec0 + v == 0;
        float p[3][CW];
#pragma unroll
        for (int j = 0; j < CW; j++) split3(on ? x[v][j] : 0.f, p[0][j], p[1][j], p[2][j]);
#pragma unroll
        for (int s = 0; s < 3; s++) bw[s * 4] = make_uint2(bf2(p[s][0], p[s][1]), bf2(p[s][2], p[s][3]));
        bw[12] = make_uint2(0u, 0u);
      }
    }
    // the buffered keys against them: integer digits (mma_pass.cuh), the key codes straight from the loads
#pragma unroll
    for (int v = 0; v < NVEC; v++) {
      const int vec = vec0 + v;
      uint32_t y[CW];
#pragma unroll
      for (int j = 0; j < CW; j++) y[j] = TWO || vec == 0 ? byte_digits(x[v][j] * UPF) : 0u;
      const uint32_t t0 = __byte_perm(y[0], y[1], 0x5140), t1 = __byte_perm(y[2], y[3], 0x5140);
      const uint32_t t2 = __byte_perm(y[0], y[1], 0x7362), t3 = __byte_perm(y[2], y[3], 0x7362);
      const uint32_t W[4] = {__byte_perm(t0, t1, 0x5410), __byte_perm(t0, t1, 0x7632), __byte_perm(t2, t3, 0x5410),
                             __byte_perm(t2, t3, 0x7632)};                 // W[s]: digit s of the four columns
#pragma unroll
      for (int s = 0; s < 4; s++) Bf8[(2 * (lane >> 3) + (lane & 1)) * 32 + (vec * 4 + 3 - s) * 4 + ((lane & 7) >> 1)] = W[s];
      if constexpr (BITS == 4) put_b_words<4>(Bf4, lane, vec, y[0], y[1], y[2], y[3]);
    }
    if (NVEC == 2) d = warp_sum(d);
    if (lane == 0) {
      if (NVEC == 2) misc[0] = d;
#pragma unroll
      for (int v = 0; v < NVEC; v++) { misc[4 + 2 * (vec0 + v)] = fx[v].i1; misc[5 + 2 * (vec0 + v)] = fx[v].i2; }
    }
    if (vec0 == 0) {
#pragma unroll
      for (int u = 0; u < NU; u++) *reinterpret_cast<uint2*>(kbt + g * DK + 32 * u + 8 * t) = kw[u];
      if (t == 0) ksf[g] = ksl;
    }
    __syncwarp();
    // (fragment rows 8 .. 15 are empty; one vector a warp: the other's columns may not be written yet, and are not looked at)
    int acc[4] = {MAGIC_I, MAGIC_I, 0, 0};
#pragma unroll
    for (int u = 0; u < NU; u++)
      mma_i8<false>(acc, kw[u].x, 0u, kw[u].y, 0u, Bf8[(2 * u) * 32 + lane], Bf8[(2 * u + 1) * 32 + lane]);
    const float wa = (t & 1) ? 256.0f : 16777216.0f, wb = (t & 1) ? 1.0f : 65536.0f;
    float T = fmaf((__int_as_float(acc[0]) - 12582912.0f) * ksl, wa, ((__int_as_float(acc[1]) - 12582912.0f) * ksl) * wb);
    T += __shfl_xor_sync(0xffffffffu, T, 1);
    T *= 1.0f / UPF;                                       // (in the unit of the state's sums)
    if (!(t & 1) && (NVEC == 2 || (t >> 1) == vec0)) reinterpret_cast<float*>(dqk + g)[t >> 1] = T;
  } else if (warp == 1) {
    if (lane < HPS) gates_finish<KIND>(A, gr, hd + lane * HD_W);
  } else if (warp == 2) {
    const int n0 = nraw & (M - 1);
    if (lane == 0) misc[1] = __int_as_float(n0);
    if (lane < HPS * M) {
      // dead entries may hold anything: they are selected away
      dcu[lane] = (lane & (M - 1)) < n0 ? make_float2(expf(gc0 - gb0), h2f(us0)) : make_float2(0.f, 0.f);
      gbs[lane] = gb0;
    }
  } else if (warp == 3) {
    // the norms, and the key as it goes into the buffer (one vector a warp: k . q as well)
    static_assert(NVEC == 2 || KIND != K_M2, "C . B is summed by the warp that has both");
    float kr[CW];
    cvt4_raw<BIO>(rqk[1], dt_qk, kr);
    if (KIND != K_M2) {
      float qr[CW], s0 = 0.f, s1 = 0.f;
      cvt4_raw<BIO>(rqk[0], dt_qk, qr);
#pragma unroll
      for (int j = 0; j < CW; j++) { s0 += qr[j] * qr[j]; s1 += kr[j] * kr[j]; }
      s0 = warp_sum(s0);
      s1 = warp_sum(s1);
      const float nk = __fsqrt_rn(s1 + 1e-6f), rn = __fdiv_rn(A.scale, __fsqrt_rn(s0 + 1e-6f));
      if (lane == 0) { misc[8] = rn; misc[9] = __fdiv_rn(1.0f, nk); }
      div_norm(kr, nk);
      if constexpr (NVEC == 1) {
        float d = 0.f;
#pragma unroll
        for (int j = 0; j < CW; j++) d += kr[j] * (qr[j] * rn);
        d = warp_sum(d);
        if (lane == 0) misc[0] = d;
      }
    }
    float mx = 0.f;
#pragma unroll
    for (int j = 0; j < CW; j++) mx = fmaxf(mx, fabsf(kr[j]));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    kscale = fp16_scale(mx, 127.0f);
    float cc[CW];
    round4(kr, kscale, cc);
#pragma unroll
    for (int j = 0; j < CW; j++) kword |= (static_cast<uint32_t>(static_cast<int>(cc[j])) & 0xFFu) << (8 * j);
    if (has_col) *reinterpret_cast<uint32_t*>(kcur + lane * 4) = kword;
    if (lane == 0) misc[2] = kscale;
  }
  __syncthreads();
  // back to the vectors' own size and, but for Mamba2, over the norm: powers of two (exact) and one factor per vector (with the
  // first power, so that no step between lies beyond the sum and the result: states near the largest float)
  const float iq1 = KIND == K_M2 ? misc[4] : misc[4] * misc[8], iq2 = misc[5];
  const float ik1 = KIND == K_M2 ? misc[6] : misc[6] * misc[9], ik2 = misc[7];
  const float kq = KIND == K_M2 || NVEC == 1 ? misc[0] : (((misc[0] * iq1) * iq2) * ik1) * ik2;
  const int n0 = __float_as_int(misc[1]);                  // live buffer entries of this slot
  const bool full = n0 == M - 1;                           // this token fills the buffer: fold after the read-out
  if (warp == 3 && first) {
    if (has_col) *reinterpret_cast<uint32_t*>(KBh + (long long)n0 * DK + lane * 4) = kword;
    if (lane == 0) KBSh[n0] = f2h(kscale);
  }

  // ---- read-out ---------------------------------------------------------------------------------------------------
  float y[2];                                              // block x: this thread pair's vector, half t % 2
  if constexpr (!QUANT) {
#pragma unroll
    for (int x = 0; x < 2; x++) {
      float2 s01[NU], s23[NU];
#pragma unroll
      for (int u = 0; u < NU; u++) {
        const uint2 b0 = Bf[(2 * u) * 32 + lane], b1 = Bf[(2 * u + 1) * 32 + lane];
        const uint32_t *wa = &sw[x][0][u * WPU], *wc = &sw[x][1][u * WPU];
        float e[4] = {0.f, 0.f, 0.f, 0.f}, f[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(e, wa[0], wc[0], wa[1], wc[1], b0.x, b0.y);
        mma_bf16(f, wa[2], wc[2], wa[3], wc[3], b1.x, b1.y);
        s01[u] = __fadd2_rn(make_float2(e[0], e[1]), make_float2(f[0], f[1]));
        s23[u] = __fadd2_rn(make_float2(e[2], e[3]), make_float2(f[2], f[3]));
      }
#pragma unroll
      for (int n = NU / 2; n > 0; n >>= 1) {
#pragma unroll
        for (int u = 0; u < n; u++) { s01[u] = __fadd2_rn(s01[u], s01[u + n]); s23[u] = __fadd2_rn(s23[u], s23[u + n]); }
      }
      // t even: (hi, mid); t odd: (lo, -).  The even lane of a pair ends up with row g, the odd one with row g + 8.
      const float v0 = (t & 1) ? s01[0].x : add_parts(s01[0].x, s01[0].y), v1 = (t & 1) ? s23[0].x : add_parts(s23[0].x, s23[0].y);
      const float own = (t & 1) ? v1 : v0, recv = __shfl_xor_sync(0xffffffffu, (t & 1) ? v0 : v1, 1);
      y[x] = (t & 1) ? add_parts(recv, own) : add_parts(own, recv);
    }
  } else {
    uint32_t bf[2 * NU];
#pragma unroll
    for (int r = 0; r < 2 * NU; r++) bf[r] = (BITS == 4 ? Bf4 : Bf8)[r * 32 + lane];
    int ci[NG][2];                                         // start values: nibbles carry an offset of 8 (mma_pass.cuh)
#pragma unroll
    for (int i = 0; i < NG; i++) {
      int d[4] = {0, 0, 0, 0};
      if constexpr (BITS == 4) {
#pragma unroll
        for (int u = i * UPG; u < (i + 1) * UPG && u < NU; u++)
          mma_i8<true>(d, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, bf[2 * u], bf[2 * u + 1]);
      }
      ci[i][0] = MAGIC_I - 8 * d[0];
      ci[i][1] = MAGIC_I - 8 * d[1];
    }
#pragma unroll
    for (int x = 0; x < 2; x++) {
      float2 p01 = make_float2(0.f, 0.f), p23 = p01;
#pragma unroll
      for (int i = 0; i < NG; i++) {
        int acc[4] = {ci[i][0], ci[i][1], ci[i][0], ci[i][1]};
#pragma unroll
        for (int u = i * UPG; u < (i + 1) * UPG && u < NU; u++) {
          const uint32_t *wa = &sw[x][0][u * WPU], *wc = &sw[x][1][u * WPU];
          if constexpr (BITS == 8)
            mma_i8<false>(acc, wa[0], wc[0], wa[1], wc[1], bf[2 * u], bf[2 * u + 1]);
          else
            mma_i8<true>(acc, wa[0] & 0x0F0F0F0Fu, wc[0] & 0x0F0F0F0Fu, (wa[0] >> 4) & 0x0F0F0F0Fu, (wc[0] >> 4) & 0x0F0F0F0Fu,
                         bf[2 * u], bf[2 * u + 1]);
        }
        const float sa = scale_of(scr[x][0], i), sc = scale_of(scr[x][1], i);
        const float2 nm = make_float2(-12582912.0f, -12582912.0f);
        p01 = __ffma2_rn(__fadd2_rn(make_float2(__int_as_float(acc[0]), __int_as_float(acc[1])), nm), make_float2(sa, sa), p01);
        p23 = __ffma2_rn(__fadd2_rn(make_float2(__int_as_float(acc[2]), __int_as_float(acc[3])), nm), make_float2(sc, sc), p23);
      }
      const float p[4] = {p01.x, p01.y, p23.x, p23.y};
      y[x] = join_digits(p, t);
    }
  }
  float tq, tk;
  {
    const float recv = __shfl_xor_sync(0xffffffffu, t < 2 ? y[1] : y[0], 2);
    tq = t < 2 ? y[0] : recv;
    tk = t < 2 ? recv : y[1];
  }
  const float4 hda = *reinterpret_cast<const float4*>(hd + hw * HD_W), hdb = *reinterpret_cast<const float4*>(hd + hw * HD_W + 4);
  const float vt = cvt_raw(rvt, dt_v);
  tq = hda.w * tq;
  tk = hda.w * tk;
#pragma unroll
  for (int i = 0; i < M - 1; i++) {
    if (i < n0) {                                          // uniform; dead entries may hold garbage
      const float2 du = dcu[hw * M + i], dd = dqk[i];
      const float xb = static_cast<float>(ub[i]) * du.y;
      tq = fmaf(xb, du.x * dd.x, tq);
      if (TWO) tk = fmaf(xb, du.x * dd.y, tk);
    }
  }
  tq = (tq * iq1) * iq2;
  tk = (tk * ik1) * ik2;
  float u, o;
  if (KIND == K_GDN) {
    u = hda.y * fmaf(-hdb.x, tk, vt);
    o = fmaf(kq, u, hdb.x * tq);
  } else {
    u = hda.y * vt;                                        // dt
    o = fmaf(kq, u, hdb.x * tq);
    if (A.beta) o = fmaf(hdb.z, vt, o);
  }
  stf(A.out + (long long)b * A.so + (long long)h * DV * osz, dt_out, rv, o);
  // largest |u| of the head (non-negative floats order like their bit patterns; a NaN ends up as the maximum)
  const float um = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(u))));
  if (lane == 0) red[warp] = um;
  __syncthreads();

  // ---- append at slot n0 ---------------------------------------------------------------------------------------------
  float umax = red[hw * WPH];
#pragma unroll
  for (int w = 1; w < WPH; w++) umax = fmaxf(umax, red[hw * WPH + w]);
  const float usc = fp16_scale(umax, 127.0f);
  float cc = fmaf(u, rcp_approx(usc), MAGIC) - MAGIC;
  const float rem = fmaf(-cc, usc, u);
  if (!(fabsf(rem) < usc * 0.49998474f) || usc < FP16_MIN_NORMAL) cc = rq_exact(u, usc, 127.0f);
  UBseq[((long long)h * M + n0) * DV + rv] = static_cast<uint8_t>(static_cast<int>(cc));
  if (rv == 0) {
    UBSseq[h * M + n0] = f2h(usc);
    GBseq[(long long)h * M + n0] = hdb.y;
    GCseq[h] = full ? 0.f : hdb.y;
    NPseq[h] = full ? 0 : n0 + 1;
  }
  if (!full) return;

  // ---- fold ------------------------------------------------------------------------------------------------------
  if (tid < HPS * M) {                                     // per head: decays and value scales of the slots
    const int i = tid & (M - 1), hq = tid / M;
    const float gnew = hd[hq * HD_W + 5];
    tab[hq * 20 + i] = i == M - 1 ? 1.0f : expf(gnew - gbs[tid]);
    tab[hq * 20 + 8 + i] = dcu[tid].y;
    if (i == 0) tab[hq * 20 + 16] = expf(gnew);
  }
  build_key_frags<4, DK>(KBf, kbt, kcur, tid);             // (columns in the order of the state's words)
  __syncthreads();
  {
    // this lane's row of L, in pieces: slot pairs as bf16 words
    const float* tb = tab + hw * 20;
    uint32_t* lw = Lp + (warp * 32 + 8 * t + g) * 12;
#pragma unroll
    for (int s = 0; s < M; s += 2) {
      const float L0 = tb[s] * (static_cast<float>(ub[s]) * tb[8 + s]);
      const float L1 = s + 1 == M - 1 ? cc * usc : tb[s + 1] * (static_cast<float>(ub[s + 1 < M - 1 ? s + 1 : 0]) * tb[9 + s]);
      float p[3], q[3];
      split3(L0 * ksf[s], p[0], p[1], p[2]);
      split3(L1 * (s + 1 == M - 1 ? misc[2] : ksf[s + 1]), q[0], q[1], q[2]);
#pragma unroll
      for (int j = 0; j < 3; j++) lw[4 * j + (s >> 1)] = bf2(p[j], q[j]);
    }
    __syncwarp();
    const float2 al2 = make_float2(tb[16], tb[16]);
    if constexpr (!QUANT) {
#pragma unroll
      for (int x = 0; x < 2; x++) {
        uint32_t A1[2], A2[2], A3[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const uint32_t* l = Lp + (warp * 32 + 16 * x + 8 * r + g) * 12 + t;
          A1[r] = l[0]; A2[r] = l[4]; A3[r] = l[8];
        }
#pragma unroll
        for (int un = 0; un < NU; un++) {
          const uint4 kf = *reinterpret_cast<const uint4*>(KBf + (un * 32 + lane) * 4);
          const uint32_t kb[4] = {kf.x, kf.y, kf.z, kf.w};
          uint32_t a[4], c[4];
#pragma unroll
          for (int p = 0; p < 4; p++) {                    // the two rows' words of one column pair
            const uint32_t wa = sw[x][0][un * WPU + p], wc = sw[x][1][un * WPU + p];
            const float2 fa = __fmul2_rn(make_float2(__uint_as_float(wa << 16), __uint_as_float(wa & 0xFFFF0000u)), al2);
            const float2 fc = __fmul2_rn(make_float2(__uint_as_float(wc << 16), __uint_as_float(wc & 0xFFFF0000u)), al2);
            float acc[4] = {fa.x, fa.y, fc.x, fc.y};
            mma_bf16(acc, A1[0], A1[1], A2[0], A2[1], kb[p], kb[p]);
            mma_bf16_k8(acc, A3[0], A3[1], kb[p]);
            a[p] = bf2(acc[0], acc[1]);
            c[p] = bf2(acc[2], acc[3]);
          }
          st_words<WPU>(Srow + 16 * x * ROWB + 4 * BITS * un, a);
          st_words<WPU>(Srow + (16 * x + 8) * ROWB + 4 * BITS * un, c);
        }
      }
    } else {
      // A loop over the blocks that moves the state's registers up behind it: unrolled, the fold was half of the kernel's code, and a
      // token that folds now and then waits for instructions (1 row of 32 heads, int4 k/64: 6.2 -> 5.6 us).  A block's two halves stay
      // side by side: each on its own in the loop, 37 rows of 8 heads with a slot in eight folding take 7.6 us a layer instead of 7.3.
#pragma unroll 1
      for (int x = 0; x < 2; x++) {
        uint32_t A1[2], A2[2], A3[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const uint32_t* l = Lp + (warp * 32 + 16 * x + 8 * r + g) * 12 + t;
          A1[r] = l[0]; A2[r] = l[4]; A3[r] = l[8];
        }
        constexpr int NH2 = NU - 2;
        float s0[2][UPG == 1 ? 2 : 1], s1[2][UPG == 1 ? NH2 : 1];
#pragma unroll
        for (int r = 0; r < 2; r++) {
#pragma unroll
          for (int i = 0; i < (UPG == 1 ? 2 : 1); i++) s0[r][i] = scale_of(scr[0][r], i);
#pragma unroll
          for (int i = 0; i < (UPG == 1 ? NH2 : 1); i++) s1[r][i] = scale_of(scr[0][r], (UPG == 1 ? 2 : 1) + i);
        }
        uint8_t* Sx = Srow + 16 * x * ROWB;
        unsigned short* SCx = SCrow + 16 * x * NG;
        reg_fold_chunk<BITS, UPG, 2, NG, ROWB>(sw[0][0], sw[0][1], s0, A1, A2, A3, KBf, 0, lane, al2, Sx, SCx);
        reg_fold_chunk<BITS, UPG, NH2, NG, ROWB>(sw[0][0] + 2 * WPU, sw[0][1] + 2 * WPU, s1, A1, A2, A3, KBf, 2, lane, al2, Sx, SCx);
#pragma unroll
        for (int r = 0; r < 2; r++) {
#pragma unroll
          for (int p = 0; p < NU * WPU; p++) sw[0][r][p] = sw[1][r][p];
#pragma unroll
          for (int p = 0; p < (NG + 1) / 2; p++) scr[0][r][p] = scr[1][r][p];
        }
      }
    }
  }
}

template <int KIND, int BITS, int DK, int DV, int HPS>
int launch_reg_one(const StepArgs& a, cudaStream_t stream) {
  StepArgs b = a;
  b.gqa_full = a.HV / a.HK;
  const dim3 grid(static_cast<unsigned>(a.rows), static_cast<unsigned>(a.HV / HPS));
  const bool bio = bf16_io(a);              // takes the kernel with those element types compiled in
  auto kern = bio ? step_reg_kernel<KIND, BITS, DK, DV, HPS, true> : step_reg_kernel<KIND, BITS, DK, DV, HPS, false>;
  static Residency residency[2];
  const bool early = enters_early(static_cast<long long>(grid.x) * grid.y, residency[bio].ctas(kern, HPS * DV, 0), false);
  const cudaError_t e = early ? launch_pdl(kern, grid, HPS * DV, 0, stream, b) : launch_plain(kern, grid, HPS * DV, 0, stream, b);
  return e == cudaSuccess ? 0 : -(1000 + static_cast<int>(e));
}

}  // namespace sqb
