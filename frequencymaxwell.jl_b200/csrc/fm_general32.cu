// Launchers of the general-length passes on FP32 storage (fm_general32.cuh), in either arithmetic.
#include <algorithm>

#include "fm_general32.h"

namespace fm {

template <typename K>
static void gen_allow_smem(K kern, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

static unsigned gen_blocks(long long work) {
  return (unsigned)std::max<long long>(1, std::min<long long>((work + 255) / 256, 148LL * 32));
}

template <typename R, int M, int DIR>
static cudaError_t gen_axis_M(const Dims& d, int axis, const void* in, void* out, const GenAxis& ax, const int* act,
                              cudaStream_t st) {
  using T = cplx<R>;
  using P_ = Plan<M, R>;
  constexpr int PW = 32 / P_::TP;
  constexpr int W = 8;
  const long long pencils = d.n / ax.n * 3 * d.nb;
  const long long warps = (pencils + PW - 1) / PW;
  const unsigned blocks = (unsigned)((warps + W - 1) / W);
  const size_t smem = (size_t)(2 * M + W * PW * PencilStride<M, T, P_::TP, true>::v) * sizeof(T);
  gen_allow_smem(k_gen_axis<R, M, DIR>, smem);
  k_gen_axis<R, M, DIR><<<blocks, W * 32, smem, st>>>(d, axis, (const float2*)in, (float2*)out, ax, act);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_gen_axis(const Dims& d, int axis, int dir, const void* in, void* out, const GenAxis& ax,
                            const int* act, cudaStream_t st) {
#define FM_GEN_AXIS(MM)                                                               \
  case MM:                                                                            \
    return dir < 0 ? gen_axis_M<R, MM, -1>(d, axis, in, out, ax, act, st)          \
                   : gen_axis_M<R, MM, +1>(d, axis, in, out, ax, act, st);
  switch (ax.m) {
    FM_GEN_AXIS(8)
    FM_GEN_AXIS(16)
    FM_GEN_AXIS(32)
    FM_GEN_AXIS(64)
    FM_GEN_AXIS(128)
    FM_GEN_AXIS(256)
    FM_GEN_AXIS(512)
    default:
      return cudaErrorNotSupported;
  }
#undef FM_GEN_AXIS
}

template <typename R>
cudaError_t launch_gen_pre(const Dims& d, int pro, const void* in, const void* V, const double* rs, const GenRamps& rp,
                           void* out, const int* act, cudaStream_t st, VecTab vt) {
  const unsigned bl = gen_blocks(3 * d.n * d.nb);
  if (pro == PRO_COPY)
    k_gen_pre<R, PRO_COPY><<<bl, 256, 0, st>>>(d, (const float2*)in, (const float2*)V, rs, rp, (float2*)out, act, vt);
  else if (pro == PRO_V)
    k_gen_pre<R, PRO_V><<<bl, 256, 0, st>>>(d, (const float2*)in, (const float2*)V, rs, rp, (float2*)out, act, vt);
  else
    k_gen_pre<R, PRO_V_SCALE><<<bl, 256, 0, st>>>(d, (const float2*)in, (const float2*)V, rs, rp, (float2*)out, act,
                                                     vt);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_gen_kspace(const Dims& d, int mode, void* f, const GreenParams& gp, const int* act, cudaStream_t st) {
  const unsigned bl = gen_blocks(d.n * d.nb);
  if (mode == ZMODE_CURL) k_gen_kspace<R, ZMODE_CURL><<<bl, 256, 0, st>>>(d, (float2*)f, gp, act);
  else k_gen_kspace<R, ZMODE_ONE><<<bl, 256, 0, st>>>(d, (float2*)f, gp, act);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_gen_post(const Dims& d, int epi, const void* in, const void* V, const void* xv, const void* bv,
                            const double* rs, const EpiParams& ep, const GenRamps& rp, void* out, const int* act,
                            cudaStream_t st, VecTab vt) {
  const unsigned bl = gen_blocks(3 * d.n * d.nb);
#define FM_GEN_POST(EE)                                                                                          \
  k_gen_post<R, EE><<<bl, 256, 0, st>>>(d, (const float2*)in, (const float2*)V, (const float2*)xv, (const float2*)bv, rs, ep, rp, \
                                           (float2*)out, act, vt)
  switch (epi) {
    case EPI_STORE: FM_GEN_POST(EPI_STORE); break;
    case EPI_OP: FM_GEN_POST(EPI_OP); break;
    case EPI_PREC_OP: FM_GEN_POST(EPI_PREC_OP); break;
    case EPI_PREC_RES: FM_GEN_POST(EPI_PREC_RES); break;
    default: return cudaErrorInvalidValue;
  }
#undef FM_GEN_POST
  return cudaGetLastError();
}

#define FM_GEN_INST(R)                                                                                              \
  template cudaError_t launch_gen_axis<R>(const Dims&, int, int, const void*, void*, const GenAxis&, const int*,    \
                                          cudaStream_t);                                                            \
  template cudaError_t launch_gen_pre<R>(const Dims&, int, const void*, const void*, const double*, const GenRamps&, \
                                         void*, const int*, cudaStream_t, VecTab);                                  \
  template cudaError_t launch_gen_kspace<R>(const Dims&, int, void*, const GreenParams&, const int*, cudaStream_t); \
  template cudaError_t launch_gen_post<R>(const Dims&, int, const void*, const void*, const void*, const void*,     \
                                          const double*, const EpiParams&, const GenRamps&, void*, const int*,      \
                                          cudaStream_t, VecTab);
FM_GEN_INST(float)
FM_GEN_INST(double)
#undef FM_GEN_INST

}  // namespace fm
