// Host-side launchers and tables of the passes for general axis lengths (fm_generic.cuh).
#pragma once
#include <cuda_runtime.h>

#include <complex>
#include <vector>

#include "fm_generic.cuh"

namespace fm {

// Axis lengths without a fused pass that these passes take: any n in [1, 256], by Bluestein's algorithm with a
// power-of-two FFT of length >= max(8, 2n - 1).
constexpr int BLUE_AXIS_MAX = 256;
inline bool blue_axis_supported(int n) { return n >= 1 && n <= BLUE_AXIS_MAX; }
inline int blue_fft_length(int n) {
  int m = 8;
  while (m < 2 * n - 1) m <<= 1;
  return m;
}

// FP64 host tables of one axis: the chirps of both directions and the transformed convolution kernels (BlueAxis).
// The stage twiddles of length m: twiddles16(512), and by the arithmetic type's radix split below that,
// twiddles<R>(m).
struct BlueAxisTables {
  int n = 0, m = 0;
  std::vector<std::complex<double>> chirp[2], kern[2];
};
BlueAxisTables blue_axis_tables(int n);

// The same arguments as launch_xf, launch_xi, launch_y and launch_zg, with the axis tables in place of the twiddles and
// f = c_n [* ramp] in place of the ramp.
template <typename S, typename R>
cudaError_t launch_bxf(const Dims& d, int pro, const void* in, const void* V, const double* rs, const BlueAxis& ax,
                       const void* f, void* out, const int* act, cudaStream_t st, VecTab vt);
template <typename S, typename R>
cudaError_t launch_bxi(const Dims& d, int epi, const void* in, const void* V, const void* xv, const void* bv,
                       const double* rs, const EpiParams& ep, const BlueAxis& ax, const void* f, void* out,
                       const int* act, cudaStream_t st, VecTab vt);
template <typename S, typename R>
cudaError_t launch_by(const Dims& d, int dir, const void* in, const BlueAxis& ax, const void* f, void* out,
                      const int* act, cudaStream_t st);
template <typename S, typename R>
cudaError_t launch_bz(const Dims& d, int mode, const void* in, const GreenParams& gp, const BlueAxis& ax,
                      const void* f, void* out, const int* act, cudaStream_t st);

}  // namespace fm
