// Launcher bodies of the passes for general axis lengths (fm_generic.cuh); included once per storage / arithmetic pair.
#pragma once
#include "fm_generic.h"

namespace fm {

template <typename K>
static void blue_allow_smem(K kern, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

#define FM_BLUE_SWITCH(CALL)                \
  switch (ax.m) {                           \
    case 8: return CALL(8);                 \
    case 16: return CALL(16);               \
    case 32: return CALL(32);               \
    case 64: return CALL(64);               \
    case 128: return CALL(128);             \
    case 256: return CALL(256);             \
    case 512: return CALL(512);             \
    default: return cudaErrorNotSupported;  \
  }

// grid and shared memory of the row passes
template <typename R, int M>
struct BlueRows {
  static constexpr int TP = BluePlan<M, R>::TP, PW = 32 / TP;
  static unsigned blocks(const Dims& d) {
    return (unsigned)(((long long)d.ny * d.nz * d.nb + BX_WARPS * PW - 1) / (BX_WARPS * PW));
  }
  static constexpr size_t smem =
      (size_t)(M + BX_WARPS * PW * BluePlan<M, R>::STRIDE) * sizeof(cplx<R>);
};

template <typename S, typename R, int M>
static cudaError_t bxf_M(const Dims& d, int pro, const void* in, const void* V, const double* rs, const BlueAxis& ax,
                         const void* f, void* out, const int* act, cudaStream_t st, VecTab vt) {
  using C = BlueRows<R, M>;
  blue_allow_smem(k_bxf<S, R, M>, C::smem);
  k_bxf<S, R, M><<<C::blocks(d), 32 * BX_WARPS, C::smem, st>>>(d, pro, (const cplx<S>*)in, (const cplx<S>*)V, rs, ax,
                                                               (const cplx<R>*)f, (cplx<S>*)out, act, vt);
  return cudaGetLastError();
}

template <typename S, typename R, int M, int EPI>
static cudaError_t bxi_M(const Dims& d, const void* in, const void* V, const void* xv, const void* bv, const double* rs,
                         const EpiParams& ep, const BlueAxis& ax, const void* f, void* out, const int* act,
                         cudaStream_t st, VecTab vt) {
  using C = BlueRows<R, M>;
  using TS = cplx<S>;
  blue_allow_smem(k_bxi<S, R, M, EPI>, C::smem);
  k_bxi<S, R, M, EPI><<<C::blocks(d), 32 * BX_WARPS, C::smem, st>>>(d, (const TS*)in, (const TS*)V, (const TS*)xv,
                                                                    (const TS*)bv, rs, ep, ax, (const cplx<R>*)f,
                                                                    (TS*)out, act, vt);
  return cudaGetLastError();
}

template <typename S, typename R, int M, int DIR>
static cudaError_t by_M(const Dims& d, const void* in, const BlueAxis& ax, const void* f, void* out, const int* act,
                        cudaStream_t st) {
  using C = BlueTile<R, M, false>;
  const size_t smem = C::smem(ax.n);
  const unsigned blocks = (unsigned)((long long)((d.nx + C::XT - 1) / C::XT) * d.nz * 3 * d.nb);
  blue_allow_smem(k_by<S, R, M, DIR>, smem);
  k_by<S, R, M, DIR><<<blocks, 32 * C::W, smem, st>>>(d, (const cplx<S>*)in, (cplx<S>*)out, ax, (const cplx<R>*)f,
                                                      act);
  return cudaGetLastError();
}

template <typename S, typename R, int M, int MODE>
static cudaError_t bz_M(const Dims& d, const void* in, const GreenParams& gp, const BlueAxis& ax, const void* f,
                        void* out, const int* act, cudaStream_t st) {
  using C = BlueTile<R, M, true>;
  const size_t smem = C::smem(3 * ax.n);
  const unsigned blocks = (unsigned)((long long)((d.nx + C::XT - 1) / C::XT) * d.ny * d.nb);
  blue_allow_smem(k_bz<S, R, M, MODE>, smem);
  k_bz<S, R, M, MODE><<<blocks, 32 * C::W, smem, st>>>(d, (const cplx<S>*)in, gp, ax, (const cplx<R>*)f, (cplx<S>*)out,
                                                       act);
  return cudaGetLastError();
}

template <typename S, typename R>
cudaError_t launch_bxf(const Dims& d, int pro, const void* in, const void* V, const double* rs, const BlueAxis& ax,
                       const void* f, void* out, const int* act, cudaStream_t st, VecTab vt) {
#define BX(MM) bxf_M<S, R, MM>(d, pro, in, V, rs, ax, f, out, act, st, vt)
  FM_BLUE_SWITCH(BX)
#undef BX
}

template <typename S, typename R>
cudaError_t launch_bxi(const Dims& d, int epi, const void* in, const void* V, const void* xv, const void* bv,
                       const double* rs, const EpiParams& ep, const BlueAxis& ax, const void* f, void* out,
                       const int* act, cudaStream_t st, VecTab vt) {
#define BI(MM, EE) bxi_M<S, R, MM, EE>(d, in, V, xv, bv, rs, ep, ax, f, out, act, st, vt)
#define BI0(MM) BI(MM, EPI_STORE)
#define BI1(MM) BI(MM, EPI_OP)
#define BI2(MM) BI(MM, EPI_PREC_OP)
#define BI3(MM) BI(MM, EPI_PREC_RES)
  if (epi == EPI_STORE) { FM_BLUE_SWITCH(BI0) }
  if (epi == EPI_OP) { FM_BLUE_SWITCH(BI1) }
  if (epi == EPI_PREC_OP) { FM_BLUE_SWITCH(BI2) }
  FM_BLUE_SWITCH(BI3)
#undef BI
#undef BI0
#undef BI1
#undef BI2
#undef BI3
}

template <typename S, typename R>
cudaError_t launch_by(const Dims& d, int dir, const void* in, const BlueAxis& ax, const void* f, void* out,
                      const int* act, cudaStream_t st) {
#define BYF(MM) by_M<S, R, MM, -1>(d, in, ax, f, out, act, st)
#define BYI(MM) by_M<S, R, MM, +1>(d, in, ax, f, out, act, st)
  if (dir < 0) { FM_BLUE_SWITCH(BYF) }
  FM_BLUE_SWITCH(BYI)
#undef BYF
#undef BYI
}

template <typename S, typename R>
cudaError_t launch_bz(const Dims& d, int mode, const void* in, const GreenParams& gp, const BlueAxis& ax,
                      const void* f, void* out, const int* act, cudaStream_t st) {
#define BZO(MM) bz_M<S, R, MM, ZMODE_ONE>(d, in, gp, ax, f, out, act, st)
#define BZC(MM) bz_M<S, R, MM, ZMODE_CURL>(d, in, gp, ax, f, out, act, st)
  if (mode == ZMODE_ONE) { FM_BLUE_SWITCH(BZO) }
  if (mode == ZMODE_CURL) { FM_BLUE_SWITCH(BZC) }
  return cudaErrorInvalidValue;
#undef BZO
#undef BZC
}

#define FM_BLUE_INST(S, R)                                                                                           \
  template cudaError_t launch_bxf<S, R>(const Dims&, int, const void*, const void*, const double*, const BlueAxis&,  \
                                        const void*, void*, const int*, cudaStream_t, VecTab);                       \
  template cudaError_t launch_bxi<S, R>(const Dims&, int, const void*, const void*, const void*, const void*,        \
                                        const double*, const EpiParams&, const BlueAxis&, const void*, void*,        \
                                        const int*, cudaStream_t, VecTab);                                           \
  template cudaError_t launch_by<S, R>(const Dims&, int, const void*, const BlueAxis&, const void*, void*,           \
                                       const int*, cudaStream_t);                                                    \
  template cudaError_t launch_bz<S, R>(const Dims&, int, const void*, const GreenParams&, const BlueAxis&,           \
                                       const void*, void*, const int*, cudaStream_t);

}  // namespace fm
