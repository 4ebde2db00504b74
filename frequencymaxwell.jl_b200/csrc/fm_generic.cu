// Host tables of the passes for general axis lengths (fm_generic.cuh).
#include <cmath>

#include "fm_generic.h"

namespace fm {

BlueAxisTables blue_axis_tables(int n) {
  BlueAxisTables t;
  t.n = n;
  t.m = blue_fft_length(n);
  const int m = t.m;
  for (int dir = 0; dir < 2; ++dir) {
    const double sg = dir == 0 ? -1.0 : 1.0;
    t.chirp[dir].resize(n);
    for (int k = 0; k < n; ++k) {
      // c_k = exp(sg i pi k^2 / n), with k^2 reduced mod 2n so the angle stays small
      const long long q = ((long long)k * k) % (2LL * n);
      const double a = sg * M_PI * (double)q / (double)n;
      t.chirp[dir][k] = std::complex<double>(std::cos(a), std::sin(a));
    }
    // b (length m): conj(c_j) at j and at m - j (j < n), zero elsewhere; kern = DFT_m(b) / m
    std::vector<std::complex<double>> b(m, 0.0);
    for (int j = 0; j < n; ++j) {
      b[j] = std::conj(t.chirp[dir][j]);
      if (j > 0) b[m - j] = std::conj(t.chirp[dir][j]);
    }
    t.kern[dir].assign(m, 0.0);
    for (int k = 0; k < m; ++k) {
      std::complex<double> s = 0.0;
      for (int j = 0; j < m; ++j) {
        if (b[j] == 0.0) continue;
        const long long q = ((long long)j * k) % m;
        const double a = -2.0 * M_PI * (double)q / (double)m;
        s += b[j] * std::complex<double>(std::cos(a), std::sin(a));
      }
      t.kern[dir][k] = s / (double)m;
    }
  }
  return t;
}

}  // namespace fm
