// Axis passes of the dyadic-Green convolution and of the spectral curl.
//
// Field layout (column-major like the reference): element (x, y, z, c, b) of a
// batch of 3-component fields sits at x + nx*(y + ny*(z + nz*(c + 3*b))).
// One Green application G_avg(V.*x) runs as five passes, each reading and
// writing the batch once:
//   XF  x-rows   : psi = V.*x (prologue) -> forward FFT along x
//   YF  y-pencils: forward FFT along y
//   ZG  z-pencils: forward FFT along z -> 3x3 dyadic Green -> inverse FFT along z
//                  (both sub-pixel-shifted branches of the reference's average are
//                   produced by ONE length-2L transform of the zero-padded pencil)
//   YI  y-pencils: inverse FFT along y
//   XI  x-rows   : inverse FFT along x -> epilogue (operator / preconditioner / residual)
// Every pass keeps a pencil in registers (see fm_fft.cuh); warps are independent.
#pragma once
#include "fm_fft.cuh"

namespace fm {

// storage <-> compute conversion (identity when the types match)
template <typename To, typename From>
__device__ __forceinline__ To cv(From a) {
  if constexpr (std::is_same<To, From>::value) return a;
  else return mk((typename RealOf<To>::R)a.x, (typename RealOf<To>::R)a.y);
}

struct Dims {
  int nx, ny, nz, nb;
  long long n;           // nx*ny*nz
  long long vstride = 0; // potential of RHS b at V + b*vstride (0: one potential shared by all RHS)
  int row_threads = 256; // launch shape (tuning): threads per block of the x and y row passes (128 or 256)
  int tma_ctas = 0;      // launch shape (tuning): persistent CTAs per SM of the TMA passes (0: occupancy limit)
};

// Optional per-RHS vector pointers (RHS b's field starts at tab[b]); null -> contiguous batch.
struct VecTab {
  const void* const* in = nullptr;   // XF input / XI operator input x
  void* const* out = nullptr;        // XI output
};

// Warp-local exchange buffers: each warp owns PW pencils of STRIDE elements.
template <typename T, int STRIDE>
__device__ __forceinline__ T* warp_smem(T* base, int warp_in_cta, int pencils_per_warp, int p) {
  return base + ((size_t)warp_in_cta * pencils_per_warp + p) * STRIDE;
}

// Starts bringing n consecutive values at p to L2 (lanes t of TP, one 128-byte line each at a time).  The row passes ask
// for the operands of their epilogue and of the next component this way before a transform: a load would need
// registers until then, and after the transform's synchronisations it would wait for HBM.
// Only for batches beyond PREFETCH_BYTES a field: smaller ones are in L2 already, and the instructions cost as much as
// they save.  k_xi with and without them, FP64: 1.6 MB a field 1.04, 12.6 MB 0.99-1.00, 25 MB 0.88, 50 MB 0.83, 100 MB and
// more 0.87-0.97; FP32: 12.6 MB 1.00, 21 MB 0.99, 25 MB 0.88, 50 MB 0.83 (64^3 in batches, 96^3, 128^3).
constexpr long long PREFETCH_BYTES = 24ll << 20;
// (AHEAD of the row passes: compiled in for those alone, since the code costs small fields 5-14 % of k_xi even where it is
// skipped: 64^3 15.4 us, 17.5 with it)
template <typename TS>
inline bool prefetch_pays(const Dims& d) {
  return 3 * d.n * d.nb * (long long)sizeof(TS) > PREFETCH_BYTES;
}
template <int TP, typename TS>
__device__ __forceinline__ void prefetch_row(const TS* p, int n, int t) {
  constexpr int PER = 128 / (int)sizeof(TS);
  for (int i = t * PER; i < n; i += TP * PER) prefetch_l2(p + i);
}

// Twiddle tables per FFT length are stored as [forward-order stage table (L) |
// reversed-order stage table (L)] (see fft_stage).

template <typename T>
__device__ __forceinline__ void load_table(T* dst, const T* src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

// ---------------------------------------------------------------------------
// XF: prologue + forward FFT along x.  One warp = P rows (y,z,b); a thread
// handles all 3 components of its row so V is loaded once.
// PRO: 0 copy, 1 multiply by V, 2 multiply by V and by a per-RHS real scale.
// ---------------------------------------------------------------------------
enum { PRO_COPY = 0, PRO_V = 1, PRO_V_SCALE = 2 };

// CTAs of 256 threads per SM that a row pass is compiled for, by its length.  At 256 one CTA an SM (no bound on the
// registers) ran the FP32-storage passes of 256^3 at 2.6 (k_xf) and 1.6 TB/s (k_xi); two and three run them at
// 3.9 and 3.2; k_xf with three spills (3.5).  At 512 (16 values a lane) two fit, k_xf with V in FP64 only by spilling 224
// to 248 bytes a thread.
constexpr int row_ctas(int L, int small, int at256) { return L == 96 ? 1 : L <= 128 ? small : L == 256 ? at256 : 2; }

template <typename S, typename R, int L, int PRO, bool AHEAD>
__global__ void __launch_bounds__(256, row_ctas(L, 2, 2)) k_xf(Dims d, const cplx<S>* __restrict__ in, const cplx<S>* __restrict__ V,
                                            const double* __restrict__ rhs_scale, const cplx<R>* __restrict__ twx,
                                            const cplx<R>* __restrict__ rampx, cplx<S>* __restrict__ out,
                                            const int* __restrict__ active, VecTab vt) {
  using T = cplx<R>;
  using TS = cplx<S>;
  using P_ = RowPlan<L, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + L;
  load_table(tw, twx, L);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  const long long rows = (long long)d.ny * d.nz * d.nb;
  const long long row = ((long long)blockIdx.x * (blockDim.x >> 5) + wic) * PW + p;
  // whole pencils leave; where ny*nz*nb is no multiple of PW the last warp goes on with some of its lanes, so what
  // follows has no shuffles (__syncwarp does not wait for lanes that have left)
  if (row >= rows) return;
  const int b = (int)(row / ((long long)d.ny * d.nz));
  if (active && !active[b]) return;
  const long long yz = row - (long long)b * d.ny * d.nz;
  T* sm = warp_smem<T, P_::STRIDE>(ex, wic, PW, p);
  // V is held across the three components, except at the long lengths: there the registers it would take decide how
  // many CTAs fit on an SM, and it is read per component (an L1 hit after the first)
  constexpr bool HOLD = PRO != PRO_COPY && L <= 128;
  const cplx<S>* Vrow = V + b * d.vstride + yz * L;
  T vrow[HOLD ? E : 1];
  if constexpr (HOLD) {
#pragma unroll
    for (int e = 0; e < E; ++e) vrow[e] = cv<T>(Vrow[lay_idx<L, E, P_::R0>(t, e)]);
  }
  R s = R(1);
  if constexpr (PRO == PRO_V_SCALE) s = (R)rhs_scale[b];
  const cplx<S>* inb = vt.in ? (const cplx<S>*)vt.in[b] : in + (long long)b * 3 * d.n;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const long long base = ((long long)(c + 3 * b) * d.ny * d.nz + yz) * L;
    const long long rbase = ((long long)c * d.ny * d.nz + yz) * L;
    T v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<L, E, P_::R0>(t, e);
      T a = cv<T>(inb[rbase + x]);
      if constexpr (HOLD) a = cmul(a, vrow[e]);
      else if constexpr (PRO != PRO_COPY) a = cmul(a, cv<T>(Vrow[x]));
      if constexpr (PRO == PRO_V_SCALE) a = cscale(a, s);
      if (rampx) a = cmul(a, rampx[x]);
      v[e] = a;
    }
    if (AHEAD && c < 2) prefetch_row<TP>(inb + rbase + (long long)d.ny * d.nz * L, L, t);
    long_fwd<-1, P_>(v, sm, tw, t);
#pragma unroll
    for (int e = 0; e < E; ++e) out[base + lay_idx<L, E, P_::RL>(t, e)] = cv<TS>(v[e]);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Y pass (forward DIR=-1 or inverse DIR=+1), plain.  One warp = P consecutive
// x columns at fixed (z, c, b); lane = t*P + p so consecutive lanes read
// consecutive x.
// ---------------------------------------------------------------------------
// STG (one pencil per warp only): the CTA's warps (YG_WARPS) take x-consecutive pencils of one (z, c, b) plane
// and the CTA stages the L x W block in shared memory with coalesced rows of W consecutive x values; the pencil
// slot is XOR-swizzled with bits 2.. of the row.  The launcher uses it when nx is a multiple of the warps per CTA.
constexpr int YG_WARPS = 4;
template <typename S, typename R, int L, int DIR, bool STG = false>
__global__ void __launch_bounds__(256) k_y(Dims d, const cplx<S>* __restrict__ in, const cplx<R>* __restrict__ twy,
                                           const cplx<R>* __restrict__ rampy, cplx<S>* __restrict__ out,
                                           const int* __restrict__ active) {
  using T = cplx<R>;
  using TS = cplx<S>;
  using P_ = Plan<L, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP;
  static_assert(!STG || PW == 1, "the staged y pass takes one pencil per warp");
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + L;
  load_table(tw, twy + (DIR < 0 ? 0 : L), L);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane % PW, t = lane / PW;
  const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + wic;
  const int xg = (d.nx + PW - 1) / PW;
  const long long total = (long long)xg * d.nz * 3 * d.nb;
  if (gw >= total) return;
  const int xl = (int)(gw % xg) * PW + p, x = min(xl, d.nx - 1);  // a ragged last group repeats the last column
  const long long zcb = gw / xg;  // z + nz*(c + 3b)
  const int b = (int)(zcb / (3LL * d.nz));
  if (active && !active[b]) return;
  const long long base = zcb * (long long)d.ny * d.nx + x;
  T* sm = warp_smem<T, PencilStride<L, T, TP, false>::v>(ex, wic, PW, p);
  constexpr int W = STG ? YG_WARPS : 1;
  static_assert(!STG || W == 4, "the swizzle assumes 4 pencils per row");
  auto tix = [](int r, int g) { return r * W + (g ^ ((r >> 2) & (W - 1))); };
  TS* tile = reinterpret_cast<TS*>(ex + (size_t)(blockDim.x >> 5) * PW * PencilStride<L, T, TP, false>::v);
  const long long cbase = base - wic;  // the CTA's first pencil
  if constexpr (STG) {
    for (int i = threadIdx.x; i < L * W; i += blockDim.x) {
      const int g = i % W, r = i / W;
      tile[tix(r, g)] = in[cbase + (long long)r * d.nx + g];
    }
    __syncthreads();
  }
  auto ld = [&](int y) -> T {
    if constexpr (STG) return cv<T>(tile[tix(y, wic)]);
    else return cv<T>(in[base + (long long)y * d.nx]);
  };
  auto st = [&](int y, T a) {
    if constexpr (STG) tile[tix(y, wic)] = cv<TS>(a);
    else if (xl < d.nx) out[base + (long long)y * d.nx] = cv<TS>(a);
  };
  T v[E];
  if constexpr (DIR < 0) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int y = lay_idx<L, E, P_::R0>(t, e);
      T a = ld(y);
      if (rampy) a = cmul(a, rampy[y]);
      v[e] = a;
    }
    fft_fwd_plan<-1, P_>(v, sm, tw, t);
#pragma unroll
    for (int e = 0; e < E; ++e) st(lay_idx<L, E, P_::RL>(t, e), v[e]);
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = ld(lay_idx<L, E, P_::RL>(t, e));
    fft_rev_plan<+1, P_>(v, sm, tw, t);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int y = lay_idx<L, E, P_::R0>(t, e);
      T a = v[e];
      if (rampy) a = cmul(a, cconj(rampy[y]));
      st(y, a);
    }
  }
  if constexpr (STG) {
    __syncthreads();
    for (int i = threadIdx.x; i < L * W; i += blockDim.x) {
      const int g = i % W, r = i / W;
      out[cbase + (long long)r * d.nx + g] = tile[tix(r, g)];
    }
  }
}

// ---------------------------------------------------------------------------
// Z pass with the dyadic Green (or the curl) between forward and inverse FFT.
// MODE_AVG2 : the reference's average of the +s and -s shifted Green functions
//             (s = 1/4 on z).  The pencil psi(z), z < L, is multiplied by
//             exp(-i*pi*z/(2L)), zero-padded to 2L and transformed; bin 2k holds
//             the +s spectrum at k and bin 2k-1 the -s spectrum at k (mod L).
//             After the Green product per bin, the length-2L inverse transform,
//             restricted to z < L and multiplied by exp(+i*pi*z/(2L)), is
//             L*(o_plus + o_minus) up to the constant folded into `scale`.
// MODE_ONE  : one branch with shift sz (0 when z is periodic), ramp table rz.
// MODE_CURL : ik x E with the curl k-index, complex scale folded in.
// ---------------------------------------------------------------------------
enum { ZMODE_AVG2 = 0, ZMODE_ONE = 1, ZMODE_CURL = 2 };

struct GreenParams {
  double dk[3];      // 2*pi/(N_d*res_d) / k_ref
  double shift[3];   // sub-pixel shift of this branch per axis (x, y used in all modes)
  double ksq_re, ksq_im;  // k_square / k_ref^2
  double scale_re, scale_im;  // folded normalisation (and curl factor)
  int curl_index;    // 1 -> curl index formula for odd sizes
  const double* ksq_im_b = nullptr;  // per-RHS imaginary part of k_square (null: ksq_im for all)
  int accumulate = 0;                // 1: add the result to out (second branch of a split average)
};

template <typename R>
__device__ __forceinline__ R kidx_green(int i, int n) {
  const int h = n >> 1;
  return (R)(((i + h) % n) - h);
}
template <typename R>
__device__ __forceinline__ R kidx_curl(int i, int n) {
  return (R)(i < (n >> 1) ? i : i - n);
}

// The per-bin 3x3 operators between the forward and inverse z transforms, on the components (e1, e2, e3) at k.
template <typename R>
struct GreenBin {
  using T = cplx<R>;
  R ksr, ksi;
  T sc, iks;  // folded normalisation; 1/k_square
  __device__ __forceinline__ GreenBin(const GreenParams& gp, int b) {
    ksr = (R)gp.ksq_re;
    ksi = gp.ksq_im_b ? (R)gp.ksq_im_b[b] : (R)gp.ksq_im;
    sc = mk((R)gp.scale_re, (R)gp.scale_im);
    const R kden = ksr * ksr + ksi * ksi;
    iks = mk(ksr / kden, -ksi / kden);
  }
  // (E - k (k.E)/k_square) / (|k|^2 - k_square)
  __device__ __forceinline__ void green(T& e1, T& e2, T& e3, R kx, R ky, R kz) const {
    const T kE = cmul(cadd(cadd(cscale(e1, kx), cscale(e2, ky)), cscale(e3, kz)), iks);
    const R dr = kx * kx + ky * ky + kz * kz - ksr, di = -ksi;
    const R dd = dr * dr + di * di;
    const R rdd = R(1) / dd;  // one division for both parts of 1 / (k^2 - ks)
    const T f = cmul(sc, mk(dr * rdd, -di * rdd));
    e1 = cmul(csub(e1, cscale(kE, kx)), f);
    e2 = cmul(csub(e2, cscale(kE, ky)), f);
    e3 = cmul(csub(e3, cscale(kE, kz)), f);
  }
  // The same with every fused multiply-add written out, in the order in which the compiler forms them for k_zg, so that
  // k_zreg returns the same bits (DD: which square is fused; in k_zg's FP32 average di's).  The scale is real here.
  template <bool DD>
  __device__ __forceinline__ void green_fixed(T& e1, T& e2, T& e3, R kx, R ky, R kz) const {
    const T k = mk(fma(e3.x, kz, fma(e1.x, kx, e2.x * ky)), fma(e3.y, kz, fma(e1.y, kx, e2.y * ky)));
    const T kE = mk(fma(k.x, iks.x, -(k.y * iks.y)), fma(k.x, iks.y, k.y * iks.x));
    const R dr = fma(kz, kz, fma(kx, kx, ky * ky)) - ksr, di = -ksi;
    const R rdd = R(1) / (DD ? fma(di, di, dr * dr) : fma(dr, dr, di * di));
    const T f = mk(sc.x * (dr * rdd), sc.x * (-di * rdd));
    auto out = [&](T e, R c) {
      const T a = mk(fma(-kE.x, c, e.x), fma(-kE.y, c, e.y));
      return mk(fma(a.x, f.x, -(a.y * f.y)), fma(a.x, f.y, a.y * f.x));
    };
    e1 = out(e1, kx);
    e2 = out(e2, ky);
    e3 = out(e3, kz);
  }
  // i k x E
  __device__ __forceinline__ void curl(T& e1, T& e2, T& e3, R kx, R ky, R kz) const {
    const T isc = cmul_i<1>(sc);
    const T c1 = csub(cscale(e3, ky), cscale(e2, kz));
    const T c2 = csub(cscale(e1, kz), cscale(e3, kx));
    const T c3 = csub(cscale(e2, kx), cscale(e1, ky));
    e1 = cmul(c1, isc);
    e2 = cmul(c2, isc);
    e3 = cmul(c3, isc);
  }
};

// wave number of z bin m (MODE_AVG2: bin 2k is the +s spectrum at k, bin 2k - 1 the -s spectrum)
template <int MODE, int L, typename R>
__device__ __forceinline__ R z_wavenumber(const GreenParams& gp, int m) {
  if constexpr (MODE == ZMODE_AVG2) {
    if ((m & 1) == 0) return (R)gp.dk[2] * (kidx_green<R>(m >> 1, L) + (R)gp.shift[2]);
    return (R)gp.dk[2] * (kidx_green<R>(((m + 1) >> 1) % L, L) - (R)gp.shift[2]);
  } else if constexpr (MODE == ZMODE_ONE) {
    return (R)gp.dk[2] * (kidx_green<R>(m, L) + (R)gp.shift[2]);
  } else {
    return (R)gp.dk[2] * kidx_curl<R>(m, L);
  }
}

constexpr int ZG_WARPS = 4;  // warps per CTA of the register z pass

// STG (one pencil per warp only): the CTA's warps take x-consecutive pencils at the same (y, b), and the CTA stages
// the 3 x L x W column block in shared memory with coalesced loads and stores (rows of W consecutive x values)
// instead of each lane reading one value per z-plane.  The launcher uses it when nx is a multiple of the warps
// per CTA, so every CTA's warps share (y, b) and leave together.
template <typename S, typename R, int L, int MODE, bool STG = false>
__global__ void __launch_bounds__(256) k_zg(Dims d, const cplx<S>* __restrict__ in, GreenParams gp,
                                            const cplx<R>* __restrict__ twz, const cplx<R>* __restrict__ rz,
                                            cplx<S>* __restrict__ out, const int* __restrict__ active) {
  using T = cplx<R>;
  using TS = cplx<S>;
  constexpr int LF = (MODE == ZMODE_AVG2) ? 2 * L : L;
  using P_ = Plan<LF, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP;
  static_assert(!STG || PW == 1, "the staged z pass takes one pencil per warp");
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* twr = tw + LF;
  T* rtab = twr + LF;
  T* ex = rtab + L;
  load_table(tw, twz, 2 * LF);
  if (rz) load_table(rtab, rz, L);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane % PW, t = lane / PW;
  const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + wic;
  const int xg = (d.nx + PW - 1) / PW;
  const long long total = (long long)xg * d.ny * d.nb;
  if (gw >= total) return;
  const int xl = (int)(gw % xg) * PW + p, x = min(xl, d.nx - 1);  // a ragged last group repeats the last column
  const long long yb = gw / xg;
  const int y = (int)(yb % d.ny);
  const int b = (int)(yb / d.ny);
  if (active && !active[b]) return;
  const long long plane = (long long)d.nx * d.ny;
  const long long base0 = (long long)b * 3 * d.n + (long long)y * d.nx + x;
  T* sm = warp_smem<T, PencilStride<LF, T, TP, false>::v>(ex, wic, PW, p);
  // staged block: row r = (c, z) holds the W pencils' values; the pencil slot is XOR-swizzled with bits 2.. of r,
  // so 16 consecutive rows of one pencil fall in 16 distinct 8-byte bank slots
  constexpr int W = STG ? ZG_WARPS : 1;
  static_assert(!STG || W == 4, "the swizzle assumes 4 pencils per row");
  auto tix = [](int r, int g) { return r * W + (g ^ ((r >> 2) & (W - 1))); };
  TS* tile = reinterpret_cast<TS*>(ex + (size_t)(blockDim.x >> 5) * PW * PencilStride<LF, T, TP, false>::v);
  const long long cbase = base0 - wic;  // the CTA's first pencil (x - wic)
  if constexpr (STG) {
    for (int i = threadIdx.x; i < 3 * L * W; i += blockDim.x) {
      const int g = i % W, r = i / W, c = r / L, z = r - c * L;
      tile[tix(r, g)] = in[cbase + (long long)c * d.n + (long long)z * plane + g];
    }
    __syncthreads();
  }

  T v[3][E];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int z = lay_idx<LF, E, P_::R0>(t, e);
      T a = czero<T>();
      if (MODE != ZMODE_AVG2 || z < L) {
        if constexpr (STG) a = cv<T>(tile[tix(c * L + z, wic)]);
        else a = cv<T>(in[base0 + (long long)c * d.n + (long long)z * plane]);
        if (MODE != ZMODE_CURL && rz) a = cmul(a, rtab[z]);
      }
      v[c][e] = a;
    }
    fft_fwd_plan<-1, P_, MODE == ZMODE_AVG2>(v[c], sm, tw, t);
    __syncwarp();
  }

  // per-bin 3x3 operator
  {
    int kxi = x, kyi = y;
    R kx, ky;
    if (MODE == ZMODE_CURL) {
      kx = (R)gp.dk[0] * kidx_curl<R>(kxi, d.nx);
      ky = (R)gp.dk[1] * kidx_curl<R>(kyi, d.ny);
    } else {
      kx = (R)gp.dk[0] * (kidx_green<R>(kxi, d.nx) + (R)gp.shift[0]);
      ky = (R)gp.dk[1] * (kidx_green<R>(kyi, d.ny) + (R)gp.shift[1]);
    }
    const R ksr = (R)gp.ksq_re, ksi = gp.ksq_im_b ? (R)gp.ksq_im_b[b] : (R)gp.ksq_im;
    const T sc = mk((R)gp.scale_re, (R)gp.scale_im);
    // 1/k_square
    const R kden = ksr * ksr + ksi * ksi;
    const T iks = mk(ksr / kden, -ksi / kden);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int m = lay_idx<LF, E, P_::RL>(t, e);
      R kz;
      if constexpr (MODE == ZMODE_AVG2) {
        if ((m & 1) == 0) kz = (R)gp.dk[2] * (kidx_green<R>(m >> 1, L) + (R)gp.shift[2]);
        else kz = (R)gp.dk[2] * (kidx_green<R>(((m + 1) >> 1) % L, L) - (R)gp.shift[2]);
      } else if constexpr (MODE == ZMODE_ONE) {
        kz = (R)gp.dk[2] * (kidx_green<R>(m, L) + (R)gp.shift[2]);
      } else {
        kz = (R)gp.dk[2] * kidx_curl<R>(m, L);
      }
      T e1 = v[0][e], e2 = v[1][e], e3 = v[2][e];
      if constexpr (MODE == ZMODE_CURL) {
        // (ik x E) * sc
        T c1 = csub(cscale(e3, ky), cscale(e2, kz));
        T c2 = csub(cscale(e1, kz), cscale(e3, kx));
        T c3 = csub(cscale(e2, kx), cscale(e1, ky));
        const T isc = cmul_i<1>(sc);
        v[0][e] = cmul(c1, isc);
        v[1][e] = cmul(c2, isc);
        v[2][e] = cmul(c3, isc);
      } else {
        T kE = cadd(cadd(cscale(e1, kx), cscale(e2, ky)), cscale(e3, kz));
        kE = cmul(kE, iks);
        const R k2 = kx * kx + ky * ky + kz * kz;
        const R dr = k2 - ksr, di = -ksi;
        const R dd = dr * dr + di * di;
        const R rdd = R(1) / dd;  // one division for both parts of 1 / (k^2 - ks)
        const T f = cmul(sc, mk(dr * rdd, -di * rdd));
        v[0][e] = cmul(csub(e1, cscale(kE, kx)), f);
        v[1][e] = cmul(csub(e2, cscale(kE, ky)), f);
        v[2][e] = cmul(csub(e3, cscale(kE, kz)), f);
      }
    }
  }

#pragma unroll
  for (int c = 0; c < 3; ++c) {
    fft_rev_plan<+1, P_>(v[c], sm, twr, t);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int z = lay_idx<LF, E, P_::R0>(t, e);
      if (MODE != ZMODE_AVG2 || z < L) {
        T a = v[c][e];
        if (MODE != ZMODE_CURL && rz) a = cmul(a, cconj(rtab[z]));
        if constexpr (STG) {
          tile[tix(c * L + z, wic)] = cv<TS>(a);
        } else if (xl < d.nx) {
          const long long o = base0 + (long long)c * d.n + (long long)z * plane;
          if (gp.accumulate) a = cadd(a, cv<T>(out[o]));
          out[o] = cv<TS>(a);
        }
      }
    }
  }
  if constexpr (STG) {
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * L * W; i += blockDim.x) {
      const int g = i % W, r = i / W, c = r / L, z = r - c * L;
      const long long o = cbase + (long long)c * d.n + (long long)z * plane + g;
      TS a = tile[tix(r, g)];
      if (gp.accumulate) {
        const T s2 = cadd(cv<T>(a), cv<T>(out[o]));
        a = cv<TS>(s2);
      }
      out[o] = a;
    }
  }
}

// ---------------------------------------------------------------------------
// XI: inverse FFT along x + epilogue (g += gadd first when given).
//   EPI_STORE    out = g
//   EPI_OP       out = beta*out + alpha*(x - g)                 (CBSLinearOperator)
//   EPI_PREC_OP  out = (i/eps)*V*(xs - g)                       (M^{-1} A x)
//   EPI_PREC_RES out = (i/eps)*V*(bb - xs + g)                  (M^{-1}(b - A x))
// xs = x * rhs_scale[b] when rhs_scale is given.
// ---------------------------------------------------------------------------
enum { EPI_STORE = 0, EPI_OP = 1, EPI_PREC_OP = 2, EPI_PREC_RES = 3 };

struct EpiParams {
  double alpha_re, alpha_im, beta_re, beta_im;
  double inv_eps;  // 1/eps_imag (scaled units)
  const double* inv_eps_b = nullptr;  // per-RHS 1/eps_imag (null: inv_eps for all)
  const double2* shift_b = nullptr;   // EPI_PREC_OP: per-RHS shift theta, out = M^{-1}A x - theta x
  const void* gadd = nullptr;         // storage-typed batch added to g before the epilogue (second branch of a
                                      // two-branch average), element (x, y, z, c, b) at the contiguous batch index
};

// The epilogue on one element: g = G_avg(psi) there, ix its index within RHS b's field, vp its potential value.
template <int EPI, typename S, typename T, typename R>
__device__ __forceinline__ T epi_element(T g, long long ix, const cplx<S>* xvb, const cplx<S>* bvb, const cplx<S>* outb,
                                         const cplx<S>* vp, R ie, R s, T al, T be, const EpiParams& ep, T shf) {
  if constexpr (EPI == EPI_STORE) {
    return g;
  } else if constexpr (EPI == EPI_OP) {
    T xx = cv<T>(xvb[ix]);
    T a = cmul(al, csub(xx, g));
    if (ep.beta_re != 0.0 || ep.beta_im != 0.0) a = cadd(a, cmul(be, cv<T>(outb[ix])));
    return a;
  } else if constexpr (EPI == EPI_PREC_OP) {
    const T vv = cv<T>(*vp);
    const T gam = mk(-vv.y * ie, vv.x * ie);  // (i/eps) * V
    T xx = cscale(cv<T>(xvb[ix]), s);
    T r = cmul(gam, csub(xx, g));
    if (ep.shift_b) r = csub(r, cmul(shf, xx));
    return r;
  } else {
    const T vv = cv<T>(*vp);
    const T gam = mk(-vv.y * ie, vv.x * ie);
    T xx = cscale(cv<T>(xvb[ix]), s);
    return cmul(gam, cadd(csub(cv<T>(bvb[ix]), xx), g));
  }
}

template <typename S, typename R, int L, int EPI, bool AHEAD>
__global__ void __launch_bounds__(256, row_ctas(L, 3, 3)) k_xi(Dims d, const cplx<S>* __restrict__ in, const cplx<S>* __restrict__ V,
                                            const cplx<S>* __restrict__ xv, const cplx<S>* __restrict__ bv,
                                            const double* __restrict__ rhs_scale, EpiParams ep,
                                            const cplx<R>* __restrict__ twx, const cplx<R>* __restrict__ rampx,
                                            cplx<S>* __restrict__ out, const int* __restrict__ active, VecTab vt) {
  using T = cplx<R>;
  using TS = cplx<S>;
  using P_ = RowPlan<L, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + L;
  load_table(tw, twx + L, L);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  const long long rows = (long long)d.ny * d.nz * d.nb;
  const long long row = ((long long)blockIdx.x * (blockDim.x >> 5) + wic) * PW + p;
  if (row >= rows) return;
  const int b = (int)(row / ((long long)d.ny * d.nz));
  if (active && !active[b]) return;
  const long long yz = row - (long long)b * d.ny * d.nz;
  T* sm = warp_smem<T, P_::STRIDE>(ex, wic, PW, p);
  // (i/eps) V is formed per component from V (an L1 hit after the first component) rather than held across
  // the three components: the registers it would take decide how many CTAs fit on an SM
  const R ie = (EPI == EPI_PREC_OP || EPI == EPI_PREC_RES) ? (ep.inv_eps_b ? (R)ep.inv_eps_b[b] : (R)ep.inv_eps) : R(0);
  const cplx<S>* Vrow = V + b * d.vstride + yz * L;
  const T shf = (EPI == EPI_PREC_OP && ep.shift_b) ? mk((R)ep.shift_b[b].x, (R)ep.shift_b[b].y) : czero<T>();
  R s = R(1);
  if (rhs_scale) s = (R)rhs_scale[b];
  const T al = mk((R)ep.alpha_re, (R)ep.alpha_im), be = mk((R)ep.beta_re, (R)ep.beta_im);
  const cplx<S>* xvb = vt.in ? (const cplx<S>*)vt.in[b] : xv + (long long)b * 3 * d.n;
  cplx<S>* outb = vt.out ? (cplx<S>*)vt.out[b] : out + (long long)b * 3 * d.n;
  const cplx<S>* bvb = bv + (long long)b * 3 * d.n;
  const long long cstride = (long long)d.ny * d.nz * L;  // from one component's row to the next one's
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const long long base = ((long long)(c + 3 * b) * d.ny * d.nz + yz) * L;
    const long long rbase = ((long long)c * d.ny * d.nz + yz) * L;
    T v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = cv<T>(in[base + lay_idx<L, E, P_::RL>(t, e)]);
    if constexpr (AHEAD) {
      if constexpr (EPI != EPI_STORE) prefetch_row<TP>(xvb + rbase, L, t);
      if constexpr (EPI == EPI_PREC_RES) prefetch_row<TP>(bvb + rbase, L, t);
      if ((EPI == EPI_PREC_OP || EPI == EPI_PREC_RES) && c == 0) prefetch_row<TP>(Vrow, L, t);
      if (c < 2) prefetch_row<TP>(in + base + cstride, L, t);
    }
    long_rev<+1, P_>(v, sm, tw, t);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<L, E, P_::R0>(t, e);
      const long long ix = rbase + x;
      T g = v[e];
      if (rampx) g = cmul(g, cconj(rampx[x]));
      if (ep.gadd) g = cadd(g, cv<T>(reinterpret_cast<const cplx<S>*>(ep.gadd)[(long long)b * 3 * d.n + ix]));
      const T r = epi_element<EPI, S, T, R>(g, ix, xvb, bvb, outb, Vrow + x, ie, s, al, be, ep, shf);
      outb[ix] = cv<TS>(r);
    }
    __syncwarp();
  }
}

// XI with EPI_PREC_OP followed, on the same rows, by the XF pass (PRO_V) of the next operator application:
//   out  = (i/eps) V (x - g) - theta x          (this application's result, as k_xi stores it)
//   out2 = FFT_x(V .* out)                      (what k_xf would write from the stored out)
// Each row's result is still in registers in the R0 layout that the forward transform takes, so the next
// application's x pass neither reads `out` nor V again.  The forward input is the stored (storage-typed) value,
// so out2 equals k_xf's output bit for bit.  Contiguous batches and no x ramp (the z-only and periodic plans).
template <typename S, typename R, int L, bool AHEAD>
__global__ void __launch_bounds__(256, row_ctas(L, 3, 3)) k_xi_xf(Dims d, const cplx<S>* __restrict__ in,
                                                                          const cplx<S>* __restrict__ V,
                                                                          const cplx<S>* __restrict__ xv,
                                                                          EpiParams ep,
                                                                          const cplx<R>* __restrict__ twx,
                                                                          cplx<S>* __restrict__ out,
                                                                          cplx<S>* __restrict__ out2,
                                                                          const int* __restrict__ active) {
  using T = cplx<R>;
  using TS = cplx<S>;
  using P_ = RowPlan<L, R>;
  constexpr int E = P_::E, TP = P_::TP, PW = 32 / TP;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* twf = reinterpret_cast<T*>(smraw);  // forward-order stage twiddles
  T* twr = twf + L;                      // reversed-order stage twiddles
  T* ex = twr + L;
  load_table(twf, twx, 2 * L);
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  const long long rows = (long long)d.ny * d.nz * d.nb;
  const long long row = ((long long)blockIdx.x * (blockDim.x >> 5) + wic) * PW + p;
  if (row >= rows) return;  // as in k_xf
  const int b = (int)(row / ((long long)d.ny * d.nz));
  if (active && !active[b]) return;
  const long long yz = row - (long long)b * d.ny * d.nz;
  T* sm = warp_smem<T, P_::STRIDE>(ex, wic, PW, p);
  const R ie = ep.inv_eps_b ? (R)ep.inv_eps_b[b] : (R)ep.inv_eps;
  const cplx<S>* Vrow = V + b * d.vstride + yz * L;
  const T shf = ep.shift_b ? mk((R)ep.shift_b[b].x, (R)ep.shift_b[b].y) : czero<T>();
  const T al = mk((R)ep.alpha_re, (R)ep.alpha_im), be = mk((R)ep.beta_re, (R)ep.beta_im);
  const cplx<S>* xvb = xv + (long long)b * 3 * d.n;
  cplx<S>* outb = out + (long long)b * 3 * d.n;
  const long long cstride = (long long)d.ny * d.nz * L;  // from one component's row to the next one's
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const long long base = ((long long)(c + 3 * b) * d.ny * d.nz + yz) * L;
    const long long rbase = ((long long)c * d.ny * d.nz + yz) * L;
    T v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = cv<T>(in[base + lay_idx<L, E, P_::RL>(t, e)]);
    if constexpr (AHEAD) {
      prefetch_row<TP>(xvb + rbase, L, t);
      if (c == 0) prefetch_row<TP>(Vrow, L, t);
      if (c < 2) prefetch_row<TP>(in + base + cstride, L, t);
    }
    long_rev<+1, P_>(v, sm, twr, t);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = lay_idx<L, E, P_::R0>(t, e);
      const long long ix = rbase + x;
      const T r = epi_element<EPI_PREC_OP, S, T, R>(v[e], ix, xvb, nullptr, outb, Vrow + x, ie, R(1), al, be, ep, shf);
      const TS rs = cv<TS>(r);
      outb[ix] = rs;
      v[e] = cmul(cv<T>(rs), cv<T>(Vrow[x]));  // PRO_V of the next application on the stored value
    }
    __syncwarp();
    long_fwd<-1, P_>(v, sm, twf, t);
#pragma unroll
    for (int e = 0; e < E; ++e) out2[base + lay_idx<L, E, P_::RL>(t, e)] = cv<TS>(v[e]);
    __syncwarp();
  }
}

}  // namespace fm
