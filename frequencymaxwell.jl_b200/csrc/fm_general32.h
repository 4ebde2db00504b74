// Host-side launchers of the general-length passes on FP32 storage (fm_general32.cuh); R: arithmetic.
#pragma once
#include <cuda_runtime.h>

#include "fm_general32.cuh"

namespace fm {

// axis lengths that run the FFT directly; the others run Bluestein's algorithm (blue_axis_tables)
inline bool gen_axis_plain(int n) { return n >= 8 && n <= 512 && (n & (n - 1)) == 0; }

template <typename R>
cudaError_t launch_gen_axis(const Dims& d, int axis, int dir, const void* in, void* out, const GenAxis& ax,
                            const int* act, cudaStream_t st);
template <typename R>
cudaError_t launch_gen_pre(const Dims& d, int pro, const void* in, const void* V, const double* rs, const GenRamps& rp,
                           void* out, const int* act, cudaStream_t st, VecTab vt = VecTab{});
template <typename R>
cudaError_t launch_gen_kspace(const Dims& d, int mode, void* f, const GreenParams& gp, const int* act, cudaStream_t st);
template <typename R>
cudaError_t launch_gen_post(const Dims& d, int epi, const void* in, const void* V, const void* xv, const void* bv,
                            const double* rs, const EpiParams& ep, const GenRamps& rp, void* out, const int* act,
                            cudaStream_t st, VecTab vt = VecTab{});

}  // namespace fm
