// TMA-staged versions of the strided passes (y pencils; z pencils with the dyadic Green or the curl).
// Same arithmetic as k_y / k_zg in fm_passes.cuh; the data path goes through swizzled shared-memory
// tiles loaded and stored by the tensor memory accelerator (see fm_tma.cuh).
//
// Pipeline: a persistent CTA walks its tiles i = blockIdx.x, blockIdx.x + gridDim.x, ... (tiles of
// inactive right-hand sides skipped).  Thread 0 keeps NST loads in flight: after it has stored tile i
// from stage s (and the store has read the stage) it issues the load of tile i + NST into stage s.
// Every consumer warp waits on the stage's "full" barrier; each warp arrives on the stage's "done"
// barrier after writing its pencils back, and thread 0 waits on "done" before storing.
//
// Tensor-map x coordinates count 8-byte words: a tile row is ROWB/8 words (128, 64 or 32 bytes) whatever the
// storage type, so tile xt starts at word xt*ROWB/8, a multiple of 16 bytes.
#pragma once
#include "fm_passes.cuh"
#include "fm_tma.cuh"

namespace fm {

// Shared-memory carve-up shared by the host launcher and the kernels.
template <int TILE_BYTES, int NST, int EXB, int TABB>
struct TmaSmem {
  static constexpr int tiles = 0;                                 // 1024-aligned
  static constexpr int ex = NST * TILE_BYTES;                     // exchange buffers
  static constexpr int tab = ex + ((EXB + 15) / 16) * 16;         // twiddles / ramps
  static constexpr int bars = tab + ((TABB + 15) / 16) * 16;      // 2*NST mbarriers
  static constexpr int total = bars + 2 * NST * 8 + 1024;         // + alignment slack
};

template <typename S, typename R, int L>
struct YTmaCfg {
  using T = cplx<R>;
  using TS = cplx<S>;
  using P = YTilePlan<L, S, R>;
  // bytes of a tile row: at 512 points two stages of whole lines leave no room for a second CTA; at 256 points and FP32
  // storage 64-byte rows run more CTAs an SM (k_y_tma 256^3: 223 us, 395 with 128), in FP64 storage whole lines are better
  // (5.9 TB/s, 5.2 with 64)
  static constexpr int ROWB = L == 512 || (L == 256 && sizeof(S) == 4) ? 64 : 128;
  static constexpr int TX = ROWB / (int)sizeof(TS);
  static constexpr int PW = 32 / P::TP;
  static constexpr int CW = (TX / PW) < 4 ? (TX / PW) : 4;
  static constexpr int ROUNDS = TX / (CW * PW);
  static constexpr int TILE = L * ROWB;
  static constexpr int NST = L <= 128 ? 3 : 2;  // three stages leave room for three CTAs per SM
  static constexpr int STRIDE = P::STRIDE;
  using SM = TmaSmem<TILE, NST, CW * PW * STRIDE * (int)sizeof(T), L * (int)sizeof(T)>;
  static constexpr int THREADS = CW * 32;
};

// next tile of this CTA at or after `tile` whose right-hand side is active (ntiles if none)
__device__ __forceinline__ long long next_active(long long tile, long long ntiles, long long per_rhs,
                                                 const int* __restrict__ active) {
  while (tile < ntiles && active && !active[(int)(tile / per_rhs)]) tile += gridDim.x;
  return tile;
}

template <typename S, typename R, int L, int DIR>
__global__ void __launch_bounds__(YTmaCfg<S, R, L>::THREADS)
    k_y_tma(Dims d, const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out,
            const cplx<R>* __restrict__ twy, const cplx<R>* __restrict__ rampy, const int* __restrict__ active,
            int* __restrict__ err) {
  using C = YTmaCfg<S, R, L>;
  using T = typename C::T;
  using TS = typename C::TS;
  using P_ = typename C::P;
  constexpr int E = P_::E, TP = P_::TP, PW = C::PW, CW = C::CW, NST = C::NST, TX = C::TX;
  constexpr int BOX = L > 256 ? 256 : L;
  extern __shared__ unsigned char smraw_[];
  unsigned char* sm0 = (unsigned char*)(((uintptr_t)smraw_ + 1023) & ~(uintptr_t)1023);
  unsigned char* tiles = sm0 + C::SM::tiles;
  T* ex = reinterpret_cast<T*>(sm0 + C::SM::ex);
  T* tw = reinterpret_cast<T*>(sm0 + C::SM::tab);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm0 + C::SM::bars);
  uint64_t* done = full + NST;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int xtiles = d.nx / TX;
  const long long per_rhs = (long long)xtiles * d.nz * 3;
  const long long ntiles = per_rhs * d.nb;
  load_table(tw, twy + (DIR < 0 ? 0 : L), L);
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(full + s, 1);
      mbar_init(done + s, CW);
    }
    fence_barrier_init();
  }
  __syncthreads();
  auto issue = [&](long long tile, int s) {
    const int xt = (int)(tile % xtiles);
    const int zcb = (int)(tile / xtiles);
    mbar_expect_tx(full + s, C::TILE);
    for (int k = 0; k < L / BOX; ++k)
      tma_load_3d(tiles + s * C::TILE + k * BOX * C::ROWB, &tm_in, full + s, xt * (C::ROWB / 8), k * BOX, zcb);
  };
  long long ld = next_active(blockIdx.x, ntiles, per_rhs, active);  // load cursor (thread 0)
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST && ld < ntiles; ++s) {
      issue(ld, s);
      ld = next_active(ld + gridDim.x, ntiles, per_rhs, active);
    }
  }
  const int p = lane / TP, t = lane % TP;  // t-fastest: consecutive rows across lanes
  T* sm = ex + (warp * PW + p) * C::STRIDE;
  int it = 0;
  bool ok = true;
  for (long long tile = next_active(blockIdx.x, ntiles, per_rhs, active); tile < ntiles;
       tile = next_active(tile + gridDim.x, ntiles, per_rhs, active)) {
    const int xt = (int)(tile % xtiles);
    const int zcb = (int)(tile / xtiles);
    const int s = it % NST;
    const uint32_t ph = (it / NST) & 1;
    if (!mbar_wait(full + s, ph, err, 13)) { ok = false; break; }
    unsigned char* tl = tiles + s * C::TILE;
#pragma unroll 1
    for (int rd = 0; rd < C::ROUNDS; ++rd) {
      const int xl = rd * CW * PW + warp * PW + p;
      T v[E];
      if constexpr (DIR < 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int y = lay_idx<L, E, P_::R0>(t, e);
          T a = cv<T>(*tile_at<TS, C::ROWB>(tl, y, xl));
          if (rampy) a = cmul(a, rampy[y]);
          v[e] = a;
        }
        long_fwd<-1, P_>(v, sm, tw, t);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < E; ++e) *tile_at<TS, C::ROWB>(tl, lay_idx<L, E, P_::RL>(t, e), xl) = cv<TS>(v[e]);
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = cv<T>(*tile_at<TS, C::ROWB>(tl, lay_idx<L, E, P_::RL>(t, e), xl));
        long_rev<+1, P_>(v, sm, tw, t);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int y = lay_idx<L, E, P_::R0>(t, e);
          T a = v[e];
          if (rampy) a = cmul(a, cconj(rampy[y]));
          *tile_at<TS, C::ROWB>(tl, y, xl) = cv<TS>(a);
        }
      }
      __syncwarp();
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(done + s);
    if (threadIdx.x == 0) {
      if (!mbar_wait(done + s, ph, err, 14)) { ok = false; break; }
      for (int k = 0; k < L / BOX; ++k) tma_store_3d(&tm_out, tl + k * BOX * C::ROWB, xt * (C::ROWB / 8), k * BOX, zcb);
      bulk_commit();
      bulk_wait_read0();
      if (ld < ntiles) {
        issue(ld, s);
        ld = next_active(ld + gridDim.x, ntiles, per_rhs, active);
      }
    }
    ++it;
  }
  if (threadIdx.x == 0) {
    if (!ok) {
      // drain the loads this thread issued but nobody consumed (bounded waits)
      for (int k = 0; k < NST; ++k) mbar_wait(full + ((it + k) % NST), ((it + k) / NST) & 1, err, 15);
    }
    bulk_wait0();
  }
}

// ---------------------------------------------------------------------------
// z pass: tile = TX x-pencils (128-byte rows) x Lz x 3 components at fixed (y, b).
// ---------------------------------------------------------------------------
template <typename S, typename R, int L, int MODE>
struct ZTmaCfg {
  using T = cplx<R>;
  using TS = cplx<S>;
  static constexpr int LF = (MODE == ZMODE_AVG2) ? 2 * L : L;
  using P = Plan<LF, R>;
  static constexpr int TX = 128 / (int)sizeof(TS);
  static constexpr int PW = 32 / P::TP;
  static constexpr int CW = (TX / PW) < 8 ? (TX / PW) : 8;
  static constexpr int ROUNDS = TX / (CW * PW);
  static constexpr int TILE = 3 * L * 128;
  static constexpr int NST = TILE <= 32768 ? 3 : 2;
  static constexpr int STRIDE = PencilStride<LF, T, P::TP, true>::v;
  // exchange buffers per pencil: the three components of a length-256 transform run stage by stage together
  // (their exchanges overlap), each with its own buffer; shorter transforms run one component at a time
  static constexpr int NCX = LF >= 256 ? 3 : 1;
  using SM = TmaSmem<TILE, NST, CW * PW * NCX * STRIDE * (int)sizeof(T), (2 * LF + L) * (int)sizeof(T)>;
  static constexpr int THREADS = CW * 32;
};

template <typename S, typename R, int L, int MODE>
__global__ void __launch_bounds__(ZTmaCfg<S, R, L, MODE>::THREADS)
    k_zg_tma(Dims d, const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out,
             GreenParams gp, const cplx<R>* __restrict__ twz, const cplx<R>* __restrict__ rz,
             const int* __restrict__ active, int* __restrict__ err) {
  using C = ZTmaCfg<S, R, L, MODE>;
  using T = typename C::T;
  using TS = typename C::TS;
  using P_ = typename C::P;
  constexpr int LF = C::LF, E = P_::E, TP = P_::TP, PW = C::PW, CW = C::CW, NST = C::NST, TX = C::TX;
  extern __shared__ unsigned char smraw_[];
  unsigned char* sm0 = (unsigned char*)(((uintptr_t)smraw_ + 1023) & ~(uintptr_t)1023);
  unsigned char* tiles = sm0 + C::SM::tiles;
  T* ex = reinterpret_cast<T*>(sm0 + C::SM::ex);
  T* tw = reinterpret_cast<T*>(sm0 + C::SM::tab);
  T* twr = tw + LF;
  T* rtab = twr + LF;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm0 + C::SM::bars);
  uint64_t* done = full + NST;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int xtiles = d.nx / TX;
  const long long per_rhs = (long long)xtiles * d.ny;
  const long long ntiles = per_rhs * d.nb;
  load_table(tw, twz, 2 * LF);
  if (rz) load_table(rtab, rz, L);
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(full + s, 1);
      mbar_init(done + s, CW);
    }
    fence_barrier_init();
  }
  __syncthreads();
  auto issue = [&](long long tile, int s) {
    const int xt = (int)(tile % xtiles);
    const long long yb = tile / xtiles;
    mbar_expect_tx(full + s, C::TILE);
    tma_load_4d(tiles + s * C::TILE, &tm_in, full + s, xt * 16, (int)(yb % d.ny), 0, 3 * (int)(yb / d.ny));
  };
  long long ld = next_active(blockIdx.x, ntiles, per_rhs, active);
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST && ld < ntiles; ++s) {
      issue(ld, s);
      ld = next_active(ld + gridDim.x, ntiles, per_rhs, active);
    }
  }
  const int p = lane / TP, t = lane % TP;
  constexpr int NCX = C::NCX, SMS = C::STRIDE;
  T* sm = ex + (warp * PW + p) * NCX * SMS;
  const R ksr = (R)gp.ksq_re;
  const T sc = mk((R)gp.scale_re, (R)gp.scale_im);
  int it = 0;
  bool ok = true;
  for (long long tile = next_active(blockIdx.x, ntiles, per_rhs, active); tile < ntiles;
       tile = next_active(tile + gridDim.x, ntiles, per_rhs, active)) {
    const int xt = (int)(tile % xtiles);
    const long long yb = tile / xtiles;
    const int y = (int)(yb % d.ny), b = (int)(yb / d.ny);
    const int s = it % NST;
    const uint32_t ph = (it / NST) & 1;
    if (!mbar_wait(full + s, ph, err, 23)) { ok = false; break; }
    unsigned char* tl = tiles + s * C::TILE;
    const R ksi = gp.ksq_im_b ? (R)gp.ksq_im_b[b] : (R)gp.ksq_im;
    const R kden = ksr * ksr + ksi * ksi;
    const T iks = mk(ksr / kden, -ksi / kden);
#pragma unroll 1
    for (int rd = 0; rd < C::ROUNDS; ++rd) {
      const int xl = rd * CW * PW + warp * PW + p;
      const int x = xt * TX + xl;
      T v[3][E];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int z = lay_idx<LF, E, P_::R0>(t, e);
          T a = czero<T>();
          if (MODE != ZMODE_AVG2 || z < L) {
            a = cv<T>(*tile_at<TS>(tl, c * L + z, xl));
            if (MODE != ZMODE_CURL && rz) a = cmul(a, rtab[z]);
          }
          v[c][e] = a;
        }
        if constexpr (NCX == 1) {
          fft_fwd_plan<-1, P_>(v[c], sm, tw, t);
          __syncwarp();
        }
      }
      if constexpr (NCX == 3) {
        fft_fwd_plan_n<-1, P_, 3, SMS>(v, sm, tw, t);
        __syncwarp();
      }
      R kx, ky;
      if (MODE == ZMODE_CURL) {
        kx = (R)gp.dk[0] * kidx_curl<R>(x, d.nx);
        ky = (R)gp.dk[1] * kidx_curl<R>(y, d.ny);
      } else {
        kx = (R)gp.dk[0] * (kidx_green<R>(x, d.nx) + (R)gp.shift[0]);
        ky = (R)gp.dk[1] * (kidx_green<R>(y, d.ny) + (R)gp.shift[1]);
      }
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
          const T isc = cmul_i<1>(sc);
          v[0][e] = cmul(csub(cscale(e3, ky), cscale(e2, kz)), isc);
          v[1][e] = cmul(csub(cscale(e1, kz), cscale(e3, kx)), isc);
          v[2][e] = cmul(csub(cscale(e2, kx), cscale(e1, ky)), isc);
        } else {
          T kE = cmul(cadd(cadd(cscale(e1, kx), cscale(e2, ky)), cscale(e3, kz)), iks);
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
      if constexpr (NCX == 3) {
        fft_rev_plan_n<+1, P_, 3, SMS>(v, sm, twr, t);
        __syncwarp();
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if constexpr (NCX == 1) {
          fft_rev_plan<+1, P_>(v[c], sm, twr, t);
          __syncwarp();
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int z = lay_idx<LF, E, P_::R0>(t, e);
          if (MODE != ZMODE_AVG2 || z < L) {
            T a = v[c][e];
            if (MODE != ZMODE_CURL && rz) a = cmul(a, cconj(rtab[z]));
            *tile_at<TS>(tl, c * L + z, xl) = cv<TS>(a);
          }
        }
      }
      __syncwarp();
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(done + s);
    if (threadIdx.x == 0) {
      if (!mbar_wait(done + s, ph, err, 24)) { ok = false; break; }
      tma_store_4d(&tm_out, tl, xt * 16, y, 0, 3 * b);
      bulk_commit();
      bulk_wait_read0();
      if (ld < ntiles) {
        issue(ld, s);
        ld = next_active(ld + gridDim.x, ntiles, per_rhs, active);
      }
    }
    ++it;
  }
  if (threadIdx.x == 0) {
    if (!ok) {
      for (int k = 0; k < NST; ++k) mbar_wait(full + ((it + k) % NST), ((it + k) / NST) & 1, err, 25);
    }
    bulk_wait0();
  }
}

// ---------------------------------------------------------------------------
// z pass in sixteen values a lane and component, for L = 64, 128, 256, 512 (zreg_mode): all three components stay in
// registers from the forward transform through the Green product to the inverse one.  BR = 2 is the averaged Green function
// (shift 1/4 on z): the two shifted branches run as two transforms of length L on neighbouring lane groups; branch s
// multiplies by exp(-/+ 2 pi i z/(4L)), and the groups add their results at the end (a shuffle; for L = 512, where a
// branch fills a warp, through shared memory).  BR = 1 is one branch with its ramp rz (none when z has no shift).
// ZR_PAD is the average as one transform of length 2 L of the zero-padded pencil (z_wavenumber): FP32 storage at 256
// points, whose results have its radices (zreg_mode; 256^3: 943 us, 1170 in k_zg, 829 as two branches).
//
// What bounds it is shared memory: per value and branch one exchange (two at L = 512) each way, where the length-2L
// transform in eight values a lane exchanges twice on twice the values.  In FP64 192 of 255 registers hold the values,
// so an SM has eight warps at most, in CTAs of one tile each (one branch of FP64 storage: shared memory holds four to six);
// one CTA's copies overlap the others' transforms.  The rest of the registers is too few for the compiler: in FP64 it
// spills 56 to 320 bytes a thread (128 points, both branches: 120 stored, 208 loaded).
// ---------------------------------------------------------------------------
enum { ZR_NONE = 0, ZR_ONE = 1, ZR_TWO = 2, ZR_PAD = 3 };

template <typename S, typename R, int L, int MODE>
struct ZRegCfg {
  using T = cplx<R>;
  using TS = cplx<S>;
  static constexpr int BR = MODE == ZR_TWO ? 2 : 1, LF = MODE == ZR_PAD ? 2 * L : L;
  using P = Plan16<LF>;
  static constexpr bool F64 = sizeof(R) == 8;
  // bytes of a tile row: what lets a CTA's lane groups take whole rows, and the SM its CTAs
  static constexpr int ROWB = LF <= 128 ? (F64 && sizeof(TS) == 16 ? 128 : 64)
                              : LF == 256 ? (F64 || BR == 1 ? 64 : 32) : 32;
  static constexpr int TX = ROWB / (int)sizeof(TS);  // pencils of a tile
  static constexpr int WMAX = TX * BR * P::TP / 32;  // warps that one round of the tile keeps busy
  static constexpr int W = WMAX < 4 ? WMAX : 4, THREADS = 32 * W;
  static constexpr int GROUPS = THREADS / (BR * P::TP);  // pencils in flight
  static constexpr int ROUNDS = TX / GROUPS;
  static_assert(W >= 1 && TX % GROUPS == 0 && ROUNDS >= 1, "tile rows hold whole rounds");
  static constexpr int BZ = L > 256 ? 256 : L;  // z extent of one copy
  static constexpr int TILE = 3 * L * ROWB;
  static constexpr int EXB = BR * GROUPS * P::STRIDE * (int)sizeof(T);
  using SM = TmaSmem<TILE, 1, EXB, (2 * LF + L) * (int)sizeof(T)>;
  // CTAs per SM: what 255 (FP32 arithmetic: 168) registers a thread and the 228 KB of shared memory hold
  static constexpr int BYREG = (F64 ? 8 : 12) / W, BYMEM = 233472 / (SM::total + 1024);
  static constexpr int CTAS = BYREG < BYMEM ? BYREG : BYMEM;
  static_assert(CTAS >= 2, "one CTA's copies overlap another's transforms");
  // element (component 0, z = t < TP, pencil x) of the tile: rows of ROWB bytes, swizzled by the copy in 16-byte chunks
  static __device__ __forceinline__ unsigned char* at(unsigned char* tile, int t, int x) {
    const int byte = x * (int)sizeof(TS);
    const int sw = ROWB == 128 ? (t & 7) : ROWB == 64 ? ((t >> 1) & 3) : ((t >> 2) & 1);
    return tile + t * ROWB + (((byte >> 4) ^ sw) << 4) + (byte & 15);
  }
  // at L = 64 (TP = 4) the rows t + 4e alternate between the halves of the swizzle's 8 rows: the odd ones have this
  // bit of the address flipped
  static constexpr int FLIP = P::TP == 4 ? ROWB / 2 : 0;
  // byte offset of component c and z = t + e*TP from there (multiples of 8 rows, which the swizzle repeats over, but
  // for FLIP)
  static constexpr int off(int c, int e) {
    return ((e * P::TP / BZ) * (3 * BZ) + c * BZ + (e * P::TP) % BZ) * ROWB;
  }
};

template <typename S, typename R, int L, int MODE>
__global__ void __launch_bounds__(ZRegCfg<S, R, L, MODE>::THREADS, ZRegCfg<S, R, L, MODE>::CTAS)
    k_zreg(Dims d, const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out, GreenParams gp,
           const cplx<R>* __restrict__ twz, const cplx<R>* __restrict__ rz, const int* __restrict__ active,
           int* __restrict__ err) {
  using C = ZRegCfg<S, R, L, MODE>;
  using T = typename C::T;
  using TS = typename C::TS;
  using P_ = typename C::P;
  constexpr int TP = P_::TP, BR = C::BR, LF = C::LF;
  constexpr int EL = MODE == ZR_PAD ? 8 : 16;  // values of a lane that the pencil has (the padding has the others)
  static_assert(P_::R0 == 16, "value e of a lane is z = t + e TP");
  // at 512 points and FP32 storage each branch is rounded to storage before their sum (zreg_mode)
  constexpr bool ROUND = BR == 2 && sizeof(TS) < sizeof(T);
  // the multiply-adds as in k_zg (GreenBin::green_fixed): FP32 storage, and one branch, which is faster with them (128^3,
  // FP64, two right-hand sides: 150 us, 174 with the compiler's; the average is not: 645 and 634 us for six)
  constexpr bool FIXED = sizeof(TS) == 8 || MODE == ZR_ONE;
  extern __shared__ unsigned char smraw_[];
  unsigned char* sm0 = (unsigned char*)(((uintptr_t)smraw_ + 1023) & ~(uintptr_t)1023);
  unsigned char* tl = sm0 + C::SM::tiles;
  T* ex = reinterpret_cast<T*>(sm0 + C::SM::ex);
  T* tw = reinterpret_cast<T*>(sm0 + C::SM::tab);
  T* twr = tw + LF;
  T* rtab = twr + LF;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm0 + C::SM::bars);
  const int xtiles = d.nx / C::TX;
  const long long per_rhs = (long long)xtiles * d.ny;
  const long long ntiles = per_rhs * d.nb;
  load_table(tw, twz, 2 * LF);
  if (rz) load_table(rtab, rz, L);
  if (threadIdx.x == 0) {
    mbar_init(full, 1);
    fence_barrier_init();
  }
  __syncthreads();
  auto issue = [&](long long tile) {
    const int xt = (int)(tile % xtiles);
    const long long yb = tile / xtiles;
    mbar_expect_tx(full, C::TILE);
    for (int k = 0; k < L / C::BZ; ++k)
      tma_load_4d(tl + k * 3 * C::BZ * C::ROWB, &tm_in, full, xt * (C::ROWB / 8), (int)(yb % d.ny), k * C::BZ,
                  3 * (int)(yb / d.ny));
  };
  long long tile = next_active(blockIdx.x, ntiles, per_rhs, active);
  if (threadIdx.x == 0 && tile < ntiles) issue(tile);
  // lane group of this thread: TP lanes of one branch of one pencil, the branches of a pencil side by side
  const int grp = threadIdx.x / TP, t = threadIdx.x % TP;
  const int br = BR == 2 ? grp & 1 : 0, pen = grp / BR;
  const R sg = br ? R(-1) : R(1);
  T* sm = ex + grp * P_::STRIDE;
  uint32_t ph = 0;
  for (; tile < ntiles; ph ^= 1) {
    const int xt = (int)(tile % xtiles);
    const long long yb = tile / xtiles;
    const int y = (int)(yb % d.ny), b = (int)(yb / d.ny);
    const bool ok = mbar_wait(full, ph, err, 33);
    if (__syncthreads_or(!ok)) break;  // timed out
    const GreenBin<R> gb(gp, b);
    const R ky = (R)gp.dk[1] * (kidx_green<R>(y, d.ny) + (R)gp.shift[1]);
#pragma unroll 1
    for (int rd = 0; rd < C::ROUNDS; ++rd) {
      const int xl = rd * C::GROUPS + pen;
      unsigned char* const tp0 = C::at(tl, t, xl);
      unsigned char* const tp1 = tl + ((tp0 - tl) ^ C::FLIP);
      // one component at a time between synchronisations, so that only the transform in hand needs temporaries
      T v[3][16];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int e = 0; e < EL; ++e) {
          T a = cv<T>(*reinterpret_cast<TS*>((e & 1 ? tp1 : tp0) + C::off(c, e)));
          if (MODE != ZR_ONE || rz) {
            T r = rtab[t + e * TP];
            r.y *= sg;
            a = FIXED ? cmul_fixed(a, r) : cmul(a, r);
          }
          v[c][e] = a;
        }
        fft16_fwd<-1, P_, MODE == ZR_PAD>(v[c], sm, tw, t);
        __syncwarp();
      }
      const R kx = (R)gp.dk[0] * (kidx_green<R>(xt * C::TX + xl, d.nx) + (R)gp.shift[0]);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int m = lay_idx<LF, 16, P_::RL>(t, e);
        R kz;
        if constexpr (MODE == ZR_PAD) kz = z_wavenumber<ZMODE_AVG2, L, R>(gp, m);
        else kz = (R)gp.dk[2] * (kidx_green<R>(m, L) + sg * (R)gp.shift[2]);
        if constexpr (FIXED) gb.template green_fixed<MODE == ZR_PAD && !C::F64>(v[0][e], v[1][e], v[2][e], kx, ky, kz);
        else gb.green(v[0][e], v[1][e], v[2][e], kx, ky, kz);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        fft16_rev<+1, P_>(v[c], sm, twr, t);
        if (MODE != ZR_ONE || rz) {
#pragma unroll
          for (int e = 0; e < EL; ++e) {
            T r = rtab[t + e * TP];
            r.y *= -sg;
            v[c][e] = FIXED ? cmul_fixed(v[c][e], r) : cmul(v[c][e], r);
          }
        }
        if constexpr (ROUND) {
#pragma unroll
          for (int e = 0; e < 16; ++e) v[c][e] = cv<T>(cv<TS>(v[c][e]));
        }
        if constexpr (BR == 1) {
#pragma unroll
          for (int e = 0; e < EL; ++e) *reinterpret_cast<TS*>((e & 1 ? tp1 : tp0) + C::off(c, e)) = cv<TS>(v[c][e]);
        } else {
          // sum of the branches: each group keeps half of the values and takes the partner's share of them.  By now
          // both groups of the pencil have read the tile (the exchanges synchronise them): the result may go into it.
          if constexpr (TP < 32) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const T send = br ? v[c][e] : v[c][e + 8], keep = br ? v[c][e + 8] : v[c][e];
              v[c][e] = mk(keep.x + __shfl_xor_sync(0xffffffffu, send.x, TP),
                           keep.y + __shfl_xor_sync(0xffffffffu, send.y, TP));
            }
          } else {
            T* other = ex + (grp ^ 1) * P_::STRIDE;
#pragma unroll
            for (int e = 0; e < 8; ++e) sm[t + 32 * e] = br ? v[c][e] : v[c][e + 8];
            named_bar(1 + pen, 64);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[c][e] = cadd(br ? v[c][e + 8] : v[c][e], other[t + 32 * e]);
            named_bar(1 + pen, 64);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e)
            *reinterpret_cast<TS*>((e & 1 ? tp1 : tp0) + C::off(c, e) + br * (C::off(0, 8) - C::off(0, 0))) =
                cv<TS>(v[c][e]);
        }
        __syncwarp();
      }
    }
    fence_proxy_async();
    __syncthreads();
    const long long next = next_active(tile + gridDim.x, ntiles, per_rhs, active);
    if (threadIdx.x == 0) {
      for (int k = 0; k < L / C::BZ; ++k)
        tma_store_4d(&tm_out, tl + k * 3 * C::BZ * C::ROWB, xt * (C::ROWB / 8), y, k * C::BZ, 3 * b);
      bulk_commit();
      bulk_wait_read0();
      if (next < ntiles) issue(next);
    }
    tile = next;
  }
  if (threadIdx.x == 0) {
    if (tile < ntiles) mbar_wait(full, ph, err, 34);  // timed out: once more (bounded) for the load in flight
    bulk_wait0();
  }
}

}  // namespace fm
