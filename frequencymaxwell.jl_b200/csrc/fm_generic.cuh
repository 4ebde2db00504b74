// Axis passes for lengths without a fused pass (odd lengths, other non-powers of two, e.g. the 201 x 201 x 197 padded
// grid of the reference's two-beam example).  They take the places of k_xf, k_y, k_zg and k_xi (fm_passes.cuh) axis by
// axis, so a grid pays for Bluestein's algorithm only on the axes that need it, and the two sub-pixel-shifted branches
// of a z-only boundary share the x and y passes.
//
// A length N runs Bluestein's algorithm (L. Bluestein, "A linear filtering approach to the computation of the discrete
// Fourier transform", 1970): with c_n = exp(DIR i pi n^2 / N),
//    X_k = c_k * sum_n (x_n c_n) conj(c_{k-n}),
// a circular convolution evaluated with a power-of-two FFT of length M >= 2N - 1.  N <= M/2, so the upper half of the
// first transform's input is zero and the upper half of the second one's output is not needed.
//
// About 160 FP64 instructions per value and transform at N = 201 (M = 512): bound by the FP64 pipe, not by HBM.  The
// strided passes stage the tile of a CTA in shared memory so that global rows are read and written coalesced.
// Measured on the 201 x 201 x 197 grid in FP64: one operator application 6.2 ms, against 14.8 ms as nine plain passes
// per branch with strided accesses (prologue, three DFTs, Green, three DFTs, epilogue).
#pragma once
#include "fm_passes.cuh"

namespace fm {

// Tables of one axis (arithmetic type R, device pointers).
struct BlueAxis {
  int n = 0;                  // axis length (0: the axis has fused passes)
  int m = 0;                  // FFT length, a power of two >= 2n - 1
  const void* tw = nullptr;   // [forward-order | reversed-order] stage twiddles of length m (fm_tables.h)
  const void* chirp[2] = {nullptr, nullptr};  // [forward, inverse]: n values c_k = exp(-/+ i pi k^2 / n)
  const void* kern[2] = {nullptr, nullptr};   // [forward, inverse]: m values FFT_m(conj(c) wrapped) / m
};

// FFT of length M inside the transform.  At 512 the sixteen-value plan's padding keeps the strided writes off each
// other's banks (201 x 201 x 197, k_bxf: 606 -> 529 us in FP64, 418 -> 315 in FP32); at 256 eight values a lane and twice
// the warps are faster (100 points, FP64: 56 us against 64)
template <int M, typename R> struct BluePlan : Plan<M, R> {
  static constexpr bool IS16 = false;
  static constexpr int STRIDE = PencilStride<M, cplx<R>, Plan<M, R>::TP, true>::v;
};
template <typename R> struct BluePlan<512, R> : Plan16<512> {
  static constexpr bool IS16 = true;
};

// One transform of a pencil: v[e] holds x_i at i = lay_idx<R0>(t, e) < N (zero elsewhere) and returns X_i there.
template <typename P_, typename T>
__device__ __forceinline__ void blue_dft(T (&v)[P_::E], T* sm, const T* tw, const T* ch, const T* kk, int N, int t) {
  constexpr int M = P_::L, E = P_::E, R0 = P_::R0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = lay_idx<M, E, R0>(t, e);
    if (e % R0 < R0 / 2 && i < N) v[e] = cmul(v[e], ch[i]);
  }
  if constexpr (P_::IS16) fft16_fwd<-1, P_, true>(v, sm, tw, t);
  else fft_fwd_plan<-1, P_, true>(v, sm, tw, t);
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = cmul(v[e], kk[lay_idx<M, E, P_::RL>(t, e)]);
  __syncwarp();
  if constexpr (P_::IS16) fft16_rev<+1, P_>(v, sm, tw + M, t);
  else fft_rev_plan<+1, P_>(v, sm, tw + M, t);
  __syncwarp();
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = lay_idx<M, E, R0>(t, e);
    if (e % R0 < R0 / 2 && i < N) v[e] = cmul(v[e], ch[i]);
  }
}

// ---- x rows ------------------------------------------------------------------------------------------------------
constexpr int BX_WARPS = 4;

// forward: out = DFT_x(in [.* V [* rs[b]]] [* rampx])   (PRO_COPY / PRO_V / PRO_V_SCALE as in k_xf)
template <typename S, typename R, int M>
__global__ void __launch_bounds__(32 * BX_WARPS) k_bxf(Dims d, int pro, const cplx<S>* __restrict__ in,
                                                       const cplx<S>* __restrict__ V,
                                                       const double* __restrict__ rhs_scale, BlueAxis ax,
                                                       const cplx<R>* __restrict__ rampx, cplx<S>* __restrict__ out,
                                                       const int* __restrict__ active, VecTab vt) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP, R0 = P_::R0;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + 2 * M;
  load_table(tw, (const T*)ax.tw, 2 * M);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  const int N = ax.n;
  const long long plane = (long long)d.ny * d.nz, rows = plane * d.nb;
  const long long row = ((long long)blockIdx.x * BX_WARPS + wic) * PW + p;
  if (row >= rows) return;  // whole pencils leave
  const int b = (int)(row / plane);
  if (active && !active[b]) return;
  const long long yz = row - (long long)b * plane;
  T* sm = warp_smem<T, P_::STRIDE>(ex, wic, PW, p);
  const T* ch = (const T*)ax.chirp[0];
  const T* kk = (const T*)ax.kern[0];
  const R s = pro == PRO_V_SCALE ? (R)rhs_scale[b] : R(1);
  const cplx<S>* inb = vt.in ? (const cplx<S>*)vt.in[b] : in + (long long)b * 3 * d.n;
  const cplx<S>* Vrow = V + b * d.vstride + yz * N;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const long long base = ((long long)(c + 3 * b) * plane + yz) * N;
    const long long rbase = ((long long)c * plane + yz) * N;
    T v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<M, E, R0>(t, e);
      T a = czero<T>();
      if (e % R0 < R0 / 2 && x < N) {
        a = cv<T>(inb[rbase + x]);
        if (pro != PRO_COPY) a = cmul(a, cv<T>(Vrow[x]));
        if (pro == PRO_V_SCALE) a = cscale(a, s);
        if (rampx) a = cmul(a, rampx[x]);
      }
      v[e] = a;
    }
    blue_dft<P_>(v, sm, tw, ch, kk, N, t);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<M, E, R0>(t, e);
      if (e % R0 < R0 / 2 && x < N) out[base + x] = cv<cplx<S>>(v[e]);
    }
  }
}

// inverse and epilogue: g = DFT_x^{-1}(in) [* conj(rampx)] [+ ep.gadd], then EPI (fm_passes.cuh, epi_element)
template <typename S, typename R, int M, int EPI>
__global__ void __launch_bounds__(32 * BX_WARPS) k_bxi(Dims d, const cplx<S>* __restrict__ in,
                                                       const cplx<S>* __restrict__ V, const cplx<S>* __restrict__ xv,
                                                       const cplx<S>* __restrict__ bv,
                                                       const double* __restrict__ rhs_scale, EpiParams ep, BlueAxis ax,
                                                       const cplx<R>* __restrict__ rampx, cplx<S>* __restrict__ out,
                                                       const int* __restrict__ active, VecTab vt) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP, R0 = P_::R0;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + 2 * M;
  load_table(tw, (const T*)ax.tw, 2 * M);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  const int N = ax.n;
  const long long plane = (long long)d.ny * d.nz, rows = plane * d.nb;
  const long long row = ((long long)blockIdx.x * BX_WARPS + wic) * PW + p;
  if (row >= rows) return;
  const int b = (int)(row / plane);
  if (active && !active[b]) return;
  const long long yz = row - (long long)b * plane;
  T* sm = warp_smem<T, P_::STRIDE>(ex, wic, PW, p);
  const T* ch = (const T*)ax.chirp[1];
  const T* kk = (const T*)ax.kern[1];
  const R ie = (EPI == EPI_PREC_OP || EPI == EPI_PREC_RES) ? (ep.inv_eps_b ? (R)ep.inv_eps_b[b] : (R)ep.inv_eps) : R(0);
  const T shf = (EPI == EPI_PREC_OP && ep.shift_b) ? mk((R)ep.shift_b[b].x, (R)ep.shift_b[b].y) : czero<T>();
  const R s = rhs_scale ? (R)rhs_scale[b] : R(1);
  const T al = mk((R)ep.alpha_re, (R)ep.alpha_im), be = mk((R)ep.beta_re, (R)ep.beta_im);
  const cplx<S>* xvb = vt.in ? (const cplx<S>*)vt.in[b] : xv + (long long)b * 3 * d.n;
  cplx<S>* outb = vt.out ? (cplx<S>*)vt.out[b] : out + (long long)b * 3 * d.n;
  const cplx<S>* bvb = bv + (long long)b * 3 * d.n;
  const cplx<S>* Vrow = V + b * d.vstride + yz * N;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const long long base = ((long long)(c + 3 * b) * plane + yz) * N;
    const long long rbase = ((long long)c * plane + yz) * N;
    T v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<M, E, R0>(t, e);
      v[e] = e % R0 < R0 / 2 && x < N ? cv<T>(in[base + x]) : czero<T>();
    }
    blue_dft<P_>(v, sm, tw, ch, kk, N, t);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<M, E, R0>(t, e);
      if (e % R0 < R0 / 2 && x < N) {
        const long long ix = rbase + x;
        T g = v[e];
        if (rampx) g = cmul(g, cconj(rampx[x]));
        if (ep.gadd) g = cadd(g, cv<T>(reinterpret_cast<const cplx<S>*>(ep.gadd)[(long long)b * 3 * d.n + ix]));
        outb[ix] = cv<cplx<S>>(epi_element<EPI, S, T, R>(g, ix, xvb, bvb, outb, Vrow + x, ie, s, al, be, ep, shf));
      }
    }
  }
}

// ---- y and z pencils ---------------------------------------------------------------------------------------------
// A CTA takes XT x-consecutive pencils and stages them in shared memory in the arithmetic type (rows of XT values,
// pencil slots swizzled with the row so that the lanes of a pencil, on consecutive rows, hit distinct banks).  Rows are
// 128 bytes, and 64 at M = 512: there several CTAs of four warps share an SM, and one's loads overlap another's
// transforms, where a CTA of eight would be alone (up to 166 KB of shared memory in the z pass).
template <typename R, int M>
struct BlueTile {
  using T = cplx<R>;
  static constexpr int TP = BluePlan<M, R>::TP, PW = 32 / TP;
  static constexpr int XT = (M == 512 ? 64 : 128) / (int)sizeof(T);
  static constexpr int W = XT / PW > 0 ? (XT / PW < 8 ? XT / PW : 8) : 1;
  static constexpr int ROUNDS = (XT + W * PW - 1) / (W * PW);
  static constexpr int SH = XT * (int)sizeof(T) == 128 ? 0 : 1;
  static constexpr int STRIDE = BluePlan<M, R>::STRIDE;
  __device__ static __forceinline__ int at(int r, int g) { return r * XT + (g ^ ((r >> SH) & (XT - 1))); }
  static size_t smem(int n, int comps) {
    return (size_t)(2 * M + W * PW * STRIDE + comps * n * XT) * sizeof(T);
  }
};

template <typename S, typename R, int M, int DIR>
__global__ void __launch_bounds__(32 * BlueTile<R, M>::W) k_by(Dims d, const cplx<S>* in, cplx<S>* out,
                                                                      BlueAxis ax, const cplx<R>* __restrict__ rampy,
                                                                      const int* __restrict__ active) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  using C = BlueTile<R, M>;
  constexpr int E = P_::E, TP = P_::TP, R0 = P_::R0, XT = C::XT;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + 2 * M;
  T* tile = ex + C::W * C::PW * C::STRIDE;
  const int xtiles = (d.nx + XT - 1) / XT;
  const int x0 = (int)(blockIdx.x % xtiles) * XT;
  const long long zcb = blockIdx.x / xtiles;  // z + nz*(c + 3b)
  const int b = (int)(zcb / (3LL * d.nz));
  if (active && !active[b]) return;
  const int N = ax.n, w = min(XT, d.nx - x0);
  const long long base = zcb * (long long)N * d.nx + x0;
  load_table(tw, (const T*)ax.tw, 2 * M);
  for (int i = threadIdx.x; i < N * XT; i += blockDim.x) {
    const int g = i % XT, r = i / XT;
    T a = czero<T>();
    if (g < w) {
      a = cv<T>(in[base + (long long)r * d.nx + g]);
      if (DIR < 0 && rampy) a = cmul(a, rampy[r]);
    }
    tile[C::at(r, g)] = a;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  T* sm = warp_smem<T, C::STRIDE>(ex, wic, C::PW, p);
  const T* ch = (const T*)ax.chirp[DIR < 0 ? 0 : 1];
  const T* kk = (const T*)ax.kern[DIR < 0 ? 0 : 1];
#pragma unroll 1
  for (int rd = 0; rd < C::ROUNDS; ++rd) {
    const int g = (rd * C::W + wic) * C::PW + p;
    T v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int y = lay_idx<M, E, R0>(t, e);
      v[e] = e % R0 < R0 / 2 && y < N ? tile[C::at(y, g)] : czero<T>();
    }
    blue_dft<P_>(v, sm, tw, ch, kk, N, t);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int y = lay_idx<M, E, R0>(t, e);
      if (e % R0 < R0 / 2 && y < N) tile[C::at(y, g)] = v[e];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N * XT; i += blockDim.x) {
    const int g = i % XT, r = i / XT;
    if (g < w) {
      T a = tile[C::at(r, g)];
      if (DIR > 0 && rampy) a = cmul(a, cconj(rampy[r]));
      out[base + (long long)r * d.nx + g] = cv<cplx<S>>(a);
    }
  }
}

// z pass: forward DFT of the three components, the Green of one branch (ZMODE_ONE) or the curl (ZMODE_CURL) per bin,
// inverse DFT; gp.accumulate adds the result to out.
template <typename S, typename R, int M, int MODE>
__global__ void __launch_bounds__(32 * BlueTile<R, M>::W) k_bz(Dims d, const cplx<S>* __restrict__ in,
                                                                     GreenParams gp, BlueAxis ax,
                                                                     const cplx<R>* __restrict__ rz,
                                                                     cplx<S>* __restrict__ out,
                                                                     const int* __restrict__ active) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  using C = BlueTile<R, M>;
  constexpr int E = P_::E, TP = P_::TP, R0 = P_::R0, XT = C::XT;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + 2 * M;
  T* tile = ex + C::W * C::PW * C::STRIDE;
  const int xtiles = (d.nx + XT - 1) / XT;
  const int x0 = (int)(blockIdx.x % xtiles) * XT;
  const long long yb = blockIdx.x / xtiles;
  const int y = (int)(yb % d.ny), b = (int)(yb / d.ny);
  if (active && !active[b]) return;
  const int N = ax.n, w = min(XT, d.nx - x0);
  const long long plane = (long long)d.nx * d.ny;
  const long long base = (long long)b * 3 * d.n + (long long)y * d.nx + x0;
  load_table(tw, (const T*)ax.tw, 2 * M);
  for (int i = threadIdx.x; i < 3 * N * XT; i += blockDim.x) {
    const int g = i % XT, r = i / XT, c = r / N, z = r - c * N;
    T a = czero<T>();
    if (g < w) {
      a = cv<T>(in[base + (long long)r * plane + g]);  // components follow each other every N planes
      if (MODE == ZMODE_ONE && rz) a = cmul(a, rz[z]);
    }
    tile[C::at(r, g)] = a;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  T* sm = warp_smem<T, C::STRIDE>(ex, wic, C::PW, p);
  const GreenBin<R> gb(gp, b);
#pragma unroll 1
  for (int rd = 0; rd < C::ROUNDS; ++rd) {
    const int g = (rd * C::W + wic) * C::PW + p, x = x0 + g;
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      const T* ch = (const T*)ax.chirp[dir];
      const T* kk = (const T*)ax.kern[dir];
#pragma unroll 1
      for (int c = 0; c < 3; ++c) {
        T v[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int z = lay_idx<M, E, R0>(t, e);
          v[e] = e % R0 < R0 / 2 && z < N ? tile[C::at(c * N + z, g)] : czero<T>();
        }
        blue_dft<P_>(v, sm, tw, ch, kk, N, t);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int z = lay_idx<M, E, R0>(t, e);
          if (e % R0 < R0 / 2 && z < N) tile[C::at(c * N + z, g)] = v[e];
        }
      }
      __syncwarp();
      if (dir == 0) {
        const R kx = MODE == ZMODE_CURL ? (R)gp.dk[0] * kidx_curl<R>(x, d.nx)
                                        : (R)gp.dk[0] * (kidx_green<R>(x, d.nx) + (R)gp.shift[0]);
        const R ky = MODE == ZMODE_CURL ? (R)gp.dk[1] * kidx_curl<R>(y, d.ny)
                                        : (R)gp.dk[1] * (kidx_green<R>(y, d.ny) + (R)gp.shift[1]);
        for (int k = t; k < N; k += TP) {
          const R kz = MODE == ZMODE_CURL ? (R)gp.dk[2] * kidx_curl<R>(k, N)
                                          : (R)gp.dk[2] * (kidx_green<R>(k, N) + (R)gp.shift[2]);
          T& e1 = tile[C::at(k, g)];
          T& e2 = tile[C::at(N + k, g)];
          T& e3 = tile[C::at(2 * N + k, g)];
          if constexpr (MODE == ZMODE_CURL) gb.curl(e1, e2, e3, kx, ky, kz);
          else gb.green(e1, e2, e3, kx, ky, kz);
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * N * XT; i += blockDim.x) {
    const int g = i % XT, r = i / XT, z = r % N;
    if (g < w) {
      T a = tile[C::at(r, g)];
      if (MODE == ZMODE_ONE && rz) a = cmul(a, cconj(rz[z]));
      cplx<S>* o = out + base + (long long)r * plane + g;
      if (gp.accumulate) a = cadd(a, cv<T>(*o));
      *o = cv<cplx<S>>(a);
    }
  }
}

}  // namespace fm
