// Host side of the fold launch (see fold_kernel.cuh and launchers.h for the return convention).
#include <atomic>
#include "launchers.h"
#include "fold_kernel.cuh"
#include "tile_map.h"
#include "slot_io.cuh"

namespace sqb {
namespace {

template <bool VDEC, int BITS, bool AXK, int LPR, int MODE>
int launch_fold_mode(const StepArgs& a, cudaStream_t stream, float* out) {
  auto kern = fold_kernel<VDEC, BITS, AXK, LPR, MODE>;
  const SmemF plan = smemf_plan(VDEC, BITS, AXK, a.group, a.DK, a.DV, a.M, a.qbuf);
  if (plan.total > 220 * 1024) return 1;
  static SmemLimit limit;                   // per instantiation
  {
    cudaError_t e = limit.ensure(kern, plan.total);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
  }
  static thread_local int sms[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int& nsm = sms[dev & 63];
  if (!nsm) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (!nsm) return 1;
  FoldArgs f;
  f.S = a.S; f.SC = a.SC; f.KB = a.KB; f.KBS = a.KBS; f.UB = a.UB; f.UBS = a.UBS; f.GB = a.GB; f.GCUR = a.GCUR; f.NPTR = a.NPTR;
  f.sS = a.sS; f.sSC = a.sSC; f.sKB = a.sKB; f.sKBS = a.sKBS; f.sUB = a.sUB; f.sUBS = a.sUBS; f.sGB = a.sGB; f.sGC = a.sGC; f.sN = a.sN;
  f.idx = a.idx; f.group = a.group; f.qbuf = a.qbuf; f.M = a.M; f.HV = a.HV; f.HK = a.HK; f.DV = a.DV; f.rows = a.rows;
  f.status = a.status;
  f.out = out;
  const long long pairs = static_cast<long long>(a.rows) * a.HV;
  int per_sm = (220 * 1024) / (plan.total + 1024);
  if (per_sm > 4) per_sm = 4;
  if (per_sm < 1) per_sm = 1;
  const long long wave = static_cast<long long>(nsm) * per_sm;
  const dim3 grid(static_cast<unsigned>(pairs < wave ? pairs : wave));
  // Which of this kernel and its neighbours on the stream may overlap (us per layer-step of the two-launch paths; launches as in
  // stream order / this kernel let in early (launch_pdl) / the next kernel let in early (release) / both).  CTAs let in early
  // take the SMs that are free first.  That pays while no CTA has more than two pairs: int8 k/32, 4 rows of 32 heads 8.5 / 7.7 /
  // 8.3 / 8.0, 16 rows 12.1 / 11.8 / 12.3 / 12.8; int4 k/64, 24 rows 9.8 / 9.1 / 10.3 / 10.5; d_v 192, 16 rows 24.4 / 24.2 / 29.9
  // / 32.8.  A longer grid ends up bunched, its first CTAs, with a pair more, on the same SMs: int8 k/32, 256 rows with every
  // slot due 51.5 / 58.8 / 50.9 / 58.0; d_k 64, 64 rows 15.4 / 14.8 / 15.6 / 15.9.  Decays per channel (KDA: the step kernel behind it
  // has the longest prologue) gain from the release at any size, 4 rows 10.9 / 11.4 / 10.1 / 10.1, 64 rows 37.2 / 43.1 / 36.7 / 39.7.
  // The read-out, with a slot write behind it: 64 rows of 32 heads 73 / 74 / 79 / 80 us a pair of calls.
  TileMap map{};
  if (MODE != FOLD_ANY) {
    if (const int e = tile_map(map, a, BITS)) return -1000 - e;
  }
  const bool early = out == nullptr && !VDEC && pairs <= 2 * wave;
  f.release = out == nullptr && VDEC;
  const cudaError_t e = early ? launch_pdl(kern, grid, NT, plan.total, stream, f, map, plan) : launch_plain(kern, grid, NT, plan.total, stream, f, map, plan);
  if (e != cudaSuccess) return -1000 - static_cast<int>(e);
  return 0;
}

template <bool VDEC, int BITS, bool AXK, int LPR>
int launch_fold_one(const StepArgs& a, cudaStream_t stream, float* out) {
  if constexpr (!VDEC && AXK && LPR == 8) {
    if (a.DV == 128 && a.M == 8 && a.qbuf && a.group == (BITS == 8 ? 32 : 64) && tile_map_ok(a))
      return out != nullptr ? launch_fold_mode<VDEC, BITS, AXK, LPR, READ_TENS>(a, stream, out)
                            : launch_fold_mode<VDEC, BITS, AXK, LPR, FOLD_TENS>(a, stream, out);
  }
  return launch_fold_mode<VDEC, BITS, AXK, LPR, FOLD_ANY>(a, stream, out);
}

template <bool VDEC>
int launch_fold_kind(const StepArgs& a, int bits, bool axk, cudaStream_t stream, float* out) {
  const bool d128 = a.DK == 128;
  if (bits == 4) {
    if (axk) return d128 ? launch_fold_one<VDEC, 4, true, 8>(a, stream, out) : launch_fold_one<VDEC, 4, true, 4>(a, stream, out);
    return d128 ? launch_fold_one<VDEC, 4, false, 8>(a, stream, out) : launch_fold_one<VDEC, 4, false, 4>(a, stream, out);
  }
  if (axk) return d128 ? launch_fold_one<VDEC, 8, true, 8>(a, stream, out) : launch_fold_one<VDEC, 8, true, 4>(a, stream, out);
  return d128 ? launch_fold_one<VDEC, 8, false, 8>(a, stream, out) : launch_fold_one<VDEC, 8, false, 4>(a, stream, out);
}

}  // namespace

int launch_fold(int kind, const StepArgs& a, int bits, bool axk, cudaStream_t stream) {
  return kind == K_KDA ? launch_fold_kind<true>(a, bits, axk, stream, nullptr) : launch_fold_kind<false>(a, bits, axk, stream, nullptr);
}

int launch_read(int kind, const StepArgs& a, int bits, bool axk, float* out, cudaStream_t stream) {
  return kind == K_KDA ? launch_fold_kind<true>(a, bits, axk, stream, out) : launch_fold_kind<false>(a, bits, axk, stream, out);
}

namespace {
template <int BITS, bool AXK, int LPR>
int launch_write_one(int kind, const StepArgs& a, const float* X, cudaStream_t stream) {
  WriteArgs w;
  w.S = a.S; w.SC = a.SC; w.GCUR = a.GCUR; w.NPTR = a.NPTR;
  w.sS = a.sS; w.sSC = a.sSC; w.sGC = a.sGC; w.sN = a.sN;
  w.idx = a.idx; w.X = X; w.group = a.group; w.HV = a.HV; w.DV = a.DV; w.rows = a.rows;
  w.nptr = a.HV > 4 ? a.HV : 4;
  w.gc_width = kind == K_KDA ? a.DK : 1;
  const long long ctas = static_cast<long long>(a.rows) * a.HV;
  if (ctas > 2147483647LL) return 1;
  const cudaError_t e = launch_pdl(slot_write_kernel<BITS, AXK, LPR>, dim3(static_cast<unsigned>(ctas)), NT, 0, stream, w);
  if (e != cudaSuccess) return -1000 - static_cast<int>(e);
  return 0;
}
}  // namespace

int launch_write(int kind, const StepArgs& a, int bits, bool axk, const float* X, cudaStream_t stream) {
  const bool d128 = a.DK == 128;
  if (bits == 4) {
    if (axk) return d128 ? launch_write_one<4, true, 8>(kind, a, X, stream) : launch_write_one<4, true, 4>(kind, a, X, stream);
    return d128 ? launch_write_one<4, false, 8>(kind, a, X, stream) : launch_write_one<4, false, 4>(kind, a, X, stream);
  }
  if (axk) return d128 ? launch_write_one<8, true, 8>(kind, a, X, stream) : launch_write_one<8, true, 4>(kind, a, X, stream);
  return d128 ? launch_write_one<8, false, 8>(kind, a, X, stream) : launch_write_one<8, false, 4>(kind, a, X, stream);
}

}  // namespace sqb
