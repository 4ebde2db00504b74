// Axis passes on FP64 storage for lengths without a fused pass (odd lengths, other non-powers of two, e.g. the
// 201 x 201 x 197 padded grid of the reference's two-beam example; FP32 storage: fm_general32.cuh).  They take the places of k_xf, k_y, k_zg and k_xi (fm_passes.cuh) axis by
// axis, so a grid pays for Bluestein's algorithm only on the axes that need it, and the two sub-pixel-shifted branches
// of a z-only boundary share the x and y passes.
//
// A length N runs Bluestein's algorithm (L. Bluestein, "A linear filtering approach to the computation of the discrete
// Fourier transform", 1970): with c_n = exp(DIR i pi n^2 / N),
//    X_k = c_k * sum_n (x_n c_n) conj(c_{k-n}),
// a circular convolution evaluated with a power-of-two FFT of length M >= 2N - 1.  N <= M/2, so the upper half of the
// first transform's input is zero and the upper half of the second one's output is not needed.  What stands between
// the forward and the inverse transform of an axis is diagonal in k, and the two directions' c_k are conjugates of
// modulus one, so the factor c_k of the forward result and c_k of the inverse input cancel: both are left out, and a
// pass multiplies once, by c_n times the axis's ramp (forward) or the conjugate of that (inverse).
//
// Bound by latency: registers and shared memory hold 8 (z) to 16 (x) warps an SM, which wait for their loads and for the
// exchanges.  On the 201 x 201 x 197 grid the FP64 pipe is 26-41 % busy (about 150 FP64 instructions per value and
// transform at N = 201, M = 512), shared memory and L1 55-78 %, DRAM 7-24 %.  The strided passes stage the tile of a CTA in
// shared memory so that global rows are read and written coalesced.  One operator application there takes 5.4 ms, against
// 14.8 ms as nine plain passes per branch with strided accesses (prologue, three DFTs, Green, three DFTs, epilogue).
#pragma once
#include "fm_passes.cuh"

namespace fm {

// Tables of one axis (arithmetic type R, device pointers).
struct BlueAxis {
  int n = 0;                  // axis length (0: the axis has fused passes)
  int m = 0;                  // FFT length, a power of two >= 2n - 1
  const void* tw = nullptr;   // forward-order stage twiddles of length m (fm_tables.h)
  const void* chirp = nullptr;                // n values c_k = exp(-i pi k^2 / n): the factor of an axis without a ramp
  const void* kern[2] = {nullptr, nullptr};   // [forward, inverse]: m values FFT_m(conj(c) wrapped) / m
};

// FFT of length M inside the transform.  At 512 the sixteen-value plan's padding keeps the strided writes off each
// other's banks (201 x 201 x 197, k_bxf: 606 -> 529 us); at 256 eight values a lane and twice the warps are faster
// (100 points: 56 us against 64)
template <int M, typename R> struct BluePlan : Plan<M, R> {
  static constexpr bool IS16 = false;
  static constexpr int STRIDE = PencilStride<M, cplx<R>, Plan<M, R>::TP, true>::v;
};
template <typename R> struct BluePlan<512, R> : Plan16<512> {
  static constexpr bool IS16 = true;
};

// v from the layout of the last radix to the order of the elements (v[i] at t + TP*i), in which every plan here starts
// (R0 = E): a renaming of registers, so the inverse transform runs the same radix order and table as the forward one.
template <typename P_, typename T>
__device__ __forceinline__ void blue_order(T (&v)[P_::E]) {
  static_assert(P_::R0 == P_::E, "the first radix takes all values of a lane");
  constexpr int E = P_::E, RL = P_::RL;
  T w[E];
#pragma unroll
  for (int e = 0; e < E; ++e) w[e / RL + (e % RL) * (E / RL)] = v[e];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = w[e];
}

// The convolution of one pencil: v[i], i < E/2, holds x_n c_n at n = t + TP*i (zero from N on), and returns X_n / c_n.
template <typename P_, typename T>
__device__ __forceinline__ void blue_conv(T (&v)[P_::E], T* sm, const T* tw, const T* kk, int t) {
  constexpr int E = P_::E, TP = P_::TP;
  if constexpr (P_::IS16) fft16_fwd<-1, P_, true>(v, sm, tw, t);
  else fft_fwd_plan<-1, P_, true>(v, sm, tw, t);
  blue_order<P_>(v);
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = cmul(v[e], kk[t + TP * e]);
  __syncwarp();
  if constexpr (P_::IS16) fft16_fwd<+1, P_>(v, sm, tw, t);
  else fft_fwd_plan<+1, P_>(v, sm, tw, t);
  blue_order<P_>(v);
  __syncwarp();
}

// ---- x rows ------------------------------------------------------------------------------------------------------
constexpr int BX_WARPS = 4;  // four CTAs an SM, 128 registers (k_bxi at 512 points: 591 us, 811 with 172 registers)

// forward: out = DFT_x(in [.* V [* rs[b]]] [* ramp]) / c_k   (PRO_COPY / PRO_V / PRO_V_SCALE as in k_xf); f: c_n [* ramp]
template <typename S, typename R, int M>
__global__ void __launch_bounds__(32 * BX_WARPS, 4) k_bxf(Dims d, int pro, const cplx<S>* __restrict__ in,
                                                       const cplx<S>* __restrict__ V,
                                                       const double* __restrict__ rhs_scale, BlueAxis ax,
                                                       const cplx<R>* __restrict__ f, cplx<S>* __restrict__ out,
                                                       const int* __restrict__ active, VecTab vt) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  constexpr int H = P_::E / 2, TP = P_::TP, PW = 32 / TP;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + M;
  load_table(tw, (const T*)ax.tw, M);
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
  const T* kk = (const T*)ax.kern[0];
  const R s = pro == PRO_V_SCALE ? (R)rhs_scale[b] : R(1);
  const cplx<S>* inb = vt.in ? (const cplx<S>*)vt.in[b] : in + (long long)b * 3 * d.n;
  const cplx<S>* Vrow = V + b * d.vstride + yz * N;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const long long base = ((long long)(c + 3 * b) * plane + yz) * N;
    const long long rbase = ((long long)c * plane + yz) * N;
    T v[P_::E];
#pragma unroll
    for (int e = 0; e < H; ++e) {
      const int x = t + TP * e;
      T a = czero<T>();
      if (x < N) {
        a = cv<T>(inb[rbase + x]);
        if (pro != PRO_COPY) a = cmul(a, cv<T>(Vrow[x]));
        if (pro == PRO_V_SCALE) a = cscale(a, s);
        a = cmul(a, f[x]);
      }
      v[e] = a;
    }
    blue_conv<P_>(v, sm, tw, kk, t);
#pragma unroll
    for (int e = 0; e < H; ++e)
      if (t + TP * e < N) out[base + t + TP * e] = cv<cplx<S>>(v[e]);
  }
}

// inverse and epilogue: g = DFT_x^{-1}(in c_k) [* conj(ramp)] [+ ep.gadd], then EPI (fm_passes.cuh, epi_element)
template <typename S, typename R, int M, int EPI>
__global__ void __launch_bounds__(32 * BX_WARPS, 4) k_bxi(Dims d, const cplx<S>* __restrict__ in,
                                                       const cplx<S>* __restrict__ V, const cplx<S>* __restrict__ xv,
                                                       const cplx<S>* __restrict__ bv,
                                                       const double* __restrict__ rhs_scale, EpiParams ep, BlueAxis ax,
                                                       const cplx<R>* __restrict__ f, cplx<S>* __restrict__ out,
                                                       const int* __restrict__ active, VecTab vt) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  constexpr int H = P_::E / 2, TP = P_::TP, PW = 32 / TP;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + M;
  load_table(tw, (const T*)ax.tw, M);
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
    T v[P_::E];
#pragma unroll
    for (int e = 0; e < H; ++e) v[e] = t + TP * e < N ? cv<T>(in[base + t + TP * e]) : czero<T>();
    blue_conv<P_>(v, sm, tw, kk, t);
#pragma unroll
    for (int e = 0; e < H; ++e) {
      const int x = t + TP * e;
      if (x < N) {
        const long long ix = rbase + x;
        T g = cmul(v[e], cconj(f[x]));
        if (ep.gadd) g = cadd(g, cv<T>(reinterpret_cast<const cplx<S>*>(ep.gadd)[(long long)b * 3 * d.n + ix]));
        outb[ix] = cv<cplx<S>>(epi_element<EPI, S, T, R>(g, ix, xvb, bvb, outb, Vrow + x, ie, s, al, be, ep, shf));
      }
    }
  }
}

// ---- y and z pencils ---------------------------------------------------------------------------------------------
// A CTA takes XT x-consecutive pencils and stages them in shared memory in the arithmetic type, pencil after pencil:
// the lanes of a pencil read consecutive slots at constant offsets.  Global rows are 128 bytes; at M = 512 64 in the y
// pass and 32 in the z pass, which holds three components: narrow tiles let several CTAs share an SM, and one's loads
// overlap another's transforms (z pass of 201 x 201 x 197, one branch: 1558 us at 64 bytes, 1425 at 32; the rows that neighbouring CTAs split meet in L2).
template <typename R, int M, bool Z>
struct BlueTile {
  using T = cplx<R>;
  static constexpr int TP = BluePlan<M, R>::TP, PW = 32 / TP;
  static constexpr int XT = (M < 512 ? 128 : Z ? 32 : 64) / (int)sizeof(T);
  static constexpr int W = XT / PW > 0 ? (XT / PW < 8 ? XT / PW : 8) : 1;
  static constexpr int ROUNDS = (XT + W * PW - 1) / (W * PW);
  static constexpr int STRIDE = BluePlan<M, R>::STRIDE;
  // slots per pencil: a residue that puts the XT pencils of a wavefront's rows on disjoint slots in the copies
  __host__ __device__ static constexpr int pencil(int rows) {
    constexpr int units = 128 / (int)sizeof(T), want = units / XT > 0 ? units / XT : 1;
    return rows + ((want - rows % units) % units + units) % units;
  }
  static size_t smem(int rows) { return (size_t)(M + W * PW * STRIDE + XT * pencil(rows)) * sizeof(T); }
};

// DIR = -1: DFT_y(in * f) / c_k; +1: DFT_y^{-1}(in c_k) * conj(f); f: c_n [* ramp].  In place or not.
template <typename S, typename R, int M, int DIR>
__global__ void __launch_bounds__(32 * BlueTile<R, M, false>::W) k_by(Dims d, const cplx<S>* in, cplx<S>* out, BlueAxis ax,
                                                               const cplx<R>* __restrict__ f,
                                                               const int* __restrict__ active) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  using C = BlueTile<R, M, false>;
  constexpr int H = P_::E / 2, TP = P_::TP, XT = C::XT;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + M;
  T* tile = ex + C::W * C::PW * C::STRIDE;
  const int xtiles = (d.nx + XT - 1) / XT;
  const int x0 = (int)(blockIdx.x % xtiles) * XT;
  const long long zcb = blockIdx.x / xtiles;  // z + nz*(c + 3b)
  const int b = (int)(zcb / (3LL * d.nz));
  if (active && !active[b]) return;
  const int N = ax.n, w = min(XT, d.nx - x0), PS = C::pencil(N);
  const long long base = zcb * (long long)N * d.nx + x0;
  load_table(tw, (const T*)ax.tw, M);
  for (int i = threadIdx.x; i < N * XT; i += blockDim.x) {
    const int g = i % XT, r = i / XT;
    T a = czero<T>();
    if (g < w) {
      a = cv<T>(in[base + (long long)r * d.nx + g]);
      if (DIR < 0) a = cmul(a, f[r]);
    }
    tile[g * PS + r] = a;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  T* sm = warp_smem<T, C::STRIDE>(ex, wic, C::PW, p);
  const T* kk = (const T*)ax.kern[DIR < 0 ? 0 : 1];
#pragma unroll 1
  for (int rd = 0; rd < C::ROUNDS; ++rd) {
    T* pen = tile + ((rd * C::W + wic) * C::PW + p) * PS + t;
    T v[P_::E];
#pragma unroll
    for (int e = 0; e < H; ++e) v[e] = t + TP * e < N ? pen[TP * e] : czero<T>();
    blue_conv<P_>(v, sm, tw, kk, t);
#pragma unroll
    for (int e = 0; e < H; ++e)
      if (t + TP * e < N) pen[TP * e] = v[e];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N * XT; i += blockDim.x) {
    const int g = i % XT, r = i / XT;
    if (g < w) {
      T a = tile[g * PS + r];
      if (DIR > 0) a = cmul(a, cconj(f[r]));
      out[base + (long long)r * d.nx + g] = cv<cplx<S>>(a);
    }
  }
}

// z pass: forward DFT of the three components, the Green of one branch (ZMODE_ONE) or the curl (ZMODE_CURL) per bin,
// inverse DFT; f: c_n [* the branch's ramp]; gp.accumulate adds the result to out.
template <typename S, typename R, int M, int MODE>
__global__ void __launch_bounds__(32 * BlueTile<R, M, true>::W) k_bz(Dims d, const cplx<S>* __restrict__ in, GreenParams gp,
                                                               BlueAxis ax, const cplx<R>* __restrict__ f,
                                                               cplx<S>* __restrict__ out,
                                                               const int* __restrict__ active) {
  using T = cplx<R>;
  using P_ = BluePlan<M, R>;
  using C = BlueTile<R, M, true>;
  constexpr int H = P_::E / 2, TP = P_::TP, XT = C::XT;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* tw = reinterpret_cast<T*>(smraw);
  T* ex = tw + M;
  T* tile = ex + C::W * C::PW * C::STRIDE;
  const int xtiles = (d.nx + XT - 1) / XT;
  const int x0 = (int)(blockIdx.x % xtiles) * XT;
  const long long yb = blockIdx.x / xtiles;
  const int y = (int)(yb % d.ny), b = (int)(yb / d.ny);
  if (active && !active[b]) return;
  const int N = ax.n, w = min(XT, d.nx - x0), PS = C::pencil(3 * N);
  const long long plane = (long long)d.nx * d.ny;
  const long long base = (long long)b * 3 * d.n + (long long)y * d.nx + x0;
  load_table(tw, (const T*)ax.tw, M);
#pragma unroll 1
  for (int c = 0; c < 3; ++c)
#pragma unroll 4
    for (int i = threadIdx.x; i < N * XT; i += blockDim.x) {
      const int g = i % XT, z = i / XT;
      T a = czero<T>();
      if (g < w) {
        const long long o = base + c * d.n + z * plane + g;
        if (gp.accumulate) prefetch_l2(out + o);  // wanted after the transforms
        a = cmul(cv<T>(in[o]), f[z]);
      }
      tile[g * PS + c * N + z] = a;
    }
  __syncthreads();
  const int lane = threadIdx.x & 31, wic = threadIdx.x >> 5;
  const int p = lane / TP, t = lane % TP;
  T* sm = warp_smem<T, C::STRIDE>(ex, wic, C::PW, p);
  const GreenBin<R> gb(gp, b);
#pragma unroll 1
  for (int rd = 0; rd < C::ROUNDS; ++rd) {
    const int g = (rd * C::W + wic) * C::PW + p, x = x0 + g;
    T* pen = tile + g * PS + t;
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      const T* kk = (const T*)ax.kern[dir];
#pragma unroll 1
      for (int c = 0; c < 3; ++c) {
        T v[P_::E];
#pragma unroll
        for (int e = 0; e < H; ++e) v[e] = t + TP * e < N ? pen[c * N + TP * e] : czero<T>();
        blue_conv<P_>(v, sm, tw, kk, t);
#pragma unroll
        for (int e = 0; e < H; ++e)
          if (t + TP * e < N) pen[c * N + TP * e] = v[e];
      }
      __syncwarp();
      if (dir == 0) {
        const R kx = MODE == ZMODE_CURL ? (R)gp.dk[0] * kidx_curl<R>(x, d.nx)
                                        : (R)gp.dk[0] * (kidx_green<R>(x, d.nx) + (R)gp.shift[0]);
        const R ky = MODE == ZMODE_CURL ? (R)gp.dk[1] * kidx_curl<R>(y, d.ny)
                                        : (R)gp.dk[1] * (kidx_green<R>(y, d.ny) + (R)gp.shift[1]);
        for (int k = 0; t + k < N; k += TP) {
          const R kz = MODE == ZMODE_CURL ? (R)gp.dk[2] * kidx_curl<R>(t + k, N)
                                          : (R)gp.dk[2] * (kidx_green<R>(t + k, N) + (R)gp.shift[2]);
          if constexpr (MODE == ZMODE_CURL) gb.curl(pen[k], pen[N + k], pen[2 * N + k], kx, ky, kz);
          else gb.green(pen[k], pen[N + k], pen[2 * N + k], kx, ky, kz);
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int c = 0; c < 3; ++c)
#pragma unroll 4
    for (int i = threadIdx.x; i < N * XT; i += blockDim.x) {
      const int g = i % XT, z = i / XT;
      if (g < w) {
        T a = cmul(tile[g * PS + c * N + z], cconj(f[z]));
        cplx<S>* o = out + base + c * d.n + z * plane + g;
        if (gp.accumulate) a = cadd(a, cv<T>(*o));
        *o = cv<cplx<S>>(a);
      }
    }
}

}  // namespace fm
