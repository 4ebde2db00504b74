// Host-side construction of the FFT stage-twiddle tables and sub-pixel ramps (FP64, then cast to the
// arithmetic type of the kernels).
#pragma once
#include <cmath>
#include <complex>
#include <vector>

#include "fm_fft.cuh"

namespace fm {

using cd_t = std::complex<double>;

// Stage-twiddle table of one radix order (see fft_stage): entry (ns-1) + (q-1)*ns + k
// = exp(-2 pi i k q / (ns*R)) for each stage after the first.
inline void stage_table(std::vector<cd_t>& t, size_t off, const std::vector<int>& radices) {
  int ns = 1;
  for (size_t s = 0; s < radices.size(); ++s) {
    const int R = radices[s];
    if (s > 0)
      for (int q = 1; q < R; ++q)
        for (int k = 0; k < ns; ++k) {
          const double a = -2.0 * M_PI * (double)k * (double)q / ((double)ns * R);
          t[off + (ns - 1) + (size_t)(q - 1) * ns + k] = cd_t(std::cos(a), std::sin(a));
        }
    ns *= R;
  }
}

template <int L, typename R>
inline std::vector<int> radices_of() {
  using P_ = Plan<L, R>;
  std::vector<int> r{P_::R0};
  if (P_::R1) r.push_back(P_::R1);
  if (P_::R2) r.push_back(P_::R2);
  return r;
}

// radices of Plan<L, R>, and of the plans of sixteen values a lane (Plan16; empty for other lengths)
template <typename R>
inline std::vector<int> radices(int L) {
  switch (L) {
    case 8: return radices_of<8, R>();
    case 16: return radices_of<16, R>();
    case 32: return radices_of<32, R>();
    case 64: return radices_of<64, R>();
    case 128: return radices_of<128, R>();
    case 256: return radices_of<256, R>();
    case 512: return radices_of<512, R>();
    case 96: return radices_of<96, R>();
    default: return {};
  }
}
inline std::vector<int> radices16(int L) {
  return L == 64 ? std::vector<int>{16, 4} : L == 128 ? std::vector<int>{16, 8} : L == 256 ? std::vector<int>{16, 16}
         : L == 512 ? std::vector<int>{16, 8, 4} : std::vector<int>{};
}
// of the y tiles (YTilePlan: Plan but for FP64 storage at 256)
template <typename S, typename R>
inline std::vector<int> ytile_radices(int L) {
  return std::is_same<S, double>::value && L == 256 ? radices16(L) : radices<R>(L);
}

// [forward-order table | reversed-order table] of an FFT of length L
inline std::vector<cd_t> twiddle_pair(int L, const std::vector<int>& r) {
  if (r.empty()) return {};
  std::vector<cd_t> t(2 * (size_t)L, cd_t(1.0, 0.0));
  stage_table(t, 0, r);
  stage_table(t, L, std::vector<int>(r.rbegin(), r.rend()));
  return t;
}
template <typename R>
inline std::vector<cd_t> twiddles(int L) { return twiddle_pair(L, radices<R>(L)); }
inline std::vector<cd_t> twiddles16(int L) { return twiddle_pair(L, radices16(L)); }
template <typename S, typename R>
inline std::vector<cd_t> ytile_twiddles(int L) { return twiddle_pair(L, ytile_radices<S, R>(L)); }

// exp(sgn * 2 pi i * idx * s / L)
inline std::vector<cd_t> ramp(int L, double s, double sgn) {
  std::vector<cd_t> t(L);
  for (int k = 0; k < L; ++k) {
    double a = sgn * 2.0 * M_PI * (double)k * s / (double)L;
    t[k] = cd_t(std::cos(a), std::sin(a));
  }
  return t;
}

}  // namespace fm
