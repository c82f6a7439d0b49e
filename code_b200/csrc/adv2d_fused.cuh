// adv2d_fused.cuh -- the depth-averaged momentum advection of one micro step (uv_advect.F90:94-300
// with split = HALFSPLIT) as ONE kernel for both momentum components. Included by kernels_inst.cuh.
//
// uv_advect builds the advected quantity and the face transports of the U (or V) control volumes
// from U, V, DU, DV (uv_advect.F90:94-110 / :204-220) and runs do_advection (advection.F90:
// 362-702) on them: u/2, v, u/2 split sweeps whose flux divergences sum to UEx (VEx). Done as
// separate launches that is six passes over the 2D state per component. Here a block owns an
// FX x FY tile, stages U, V, DU, DV over the tile plus the halo the three sweeps need (4 cells in
// x for two u/2 sweeps, 2 in y for the v sweep) in shared memory, runs u/2 on the tile+halo, v on
// the tile widened in x, u/2 on the tile, and writes UEx once. Every flux and update is the
// expression of the split-sweep kernels (face_flux_s, fv_update) in the same order, so FP64
// results equal the three-sweep sequence bit for bit. The u sweeps pass face fluxes between
// neighbouring cells by warp shuffles (the two warps of a region row overlap by one column), the v
// sweep through shared memory; each thread's own cells keep their depth and flux-divergence sum
// in registers across the three sweeps.
#pragma once
#include "kernels.cuh"

namespace gb {

// launches of fewer large tiles than this take the small ones (two large tiles per SM)
constexpr long long TILE2D_SMALL = 296;
// A block of RW x FTY threads (lane x <-> region column) owns FX x FY cells of a staged region of
// RW x RH, i in [-4, FX+3], j in [-2, FY+1]. Two sizes: 56 x 16 own cells (64 x 8 threads, two own
// rows each) where the domain gives every SM work, and 24 x 8 (32 x 8 threads, one own row each)
// below, where the time is the latency of one block: a thread's chain of divisions and logarithms
// then runs once instead of twice, for 1.9 times the halo work on SMs that would idle. Whole step with one
// and two own rows per thread: 128 x 96 FP64 379 against 464 us, 80 x 96 x 12 FP64 563 against 640,
// 259 x 251 x 17 mixed 671 against 682, 300 x 300 x 12 FP64 1204 against 1242, mixed 720 against 708.
template <int RW_, int FTY_, int RPT_>
struct Tile2d {
  static constexpr int RW = RW_, FTY = FTY_, RPT = RPT_;  // RPT: own rows per thread
  static constexpr int FX = RW - 8, FY = RPT * FTY, RH = FY + 4, FT = RW * FTY;
};
using TileLarge = Tile2d<64, 8, 2>;
using TileSmall = Tile2d<32, 8, 1>;

// k*(a*s - b*s)*c as single rounded operations in this order: the volume and flux differences of
// the cell updates. FP64: the plain operations (the FP64 build contracts nothing); FP32: explicit
// intrinsics, so that the result does not depend on which products the compiler contracts.
template <class T>
__device__ __forceinline__ T diff_scaled(T k, T a, T b, T s, T c) {
  if constexpr (sizeof(T) == 4) return __fmul_rn(__fmul_rn(k, __fsub_rn(__fmul_rn(a, s), __fmul_rn(b, s))), c);
  else return k * (a * s - b * s) * c;
}
template <class T>
__device__ __forceinline__ T add_r(T a, T b) {
  if constexpr (sizeof(T) == 4) return __fadd_rn(a, b);
  else return a + b;
}

template <class T, class TL>
struct Adv2dSmem {
  static constexpr int RH = TL::RH, RW = TL::RW;
  T F0[RH][RW];   // advected quantity; reused for the field after the v sweep
  T F1[RH][RW];   // after the first u/2 sweep
  T Di[RH][RW];   // staged control-volume depth (the sweeps carry their rows' updated depths in registers)
  T Ua[RH][RW], DUa[RH][RW], Va[RH][RW], DVa[RH][RW];  // face transports / depths
  T FL[RH][RW];   // face fluxes of the v sweep
  T Q[RH][RW];    // bottom friction: the other component's velocity V/DV (DIR 0) or U/DU (DIR 1)
  uint8_t mfu[RH][RW], mfv[RH][RW], mpu[RH][RW], mpv[RH][RW];
};

// The FP64 form of the log-law drag (bf_law_f32), the expressions of k_bottom_friction in its order.
__device__ __forceinline__ void bf_law_f64(double zb, double zb0, double HH, double uloc, double vloc, double kappa,
                                           double avmmol, int runtype, double& zn, double& rr, double& r) {
  double x = kappa / log((zb + 0.5 * HH) / zb);
  rr = x * x;
  zn = zb;
  if (runtype == 1) {
    const double fricvel = sqrt(rr * (uloc * uloc + vloc * vloc));
    zn = fmin(HH, zb0 + 0.1 * avmmol / fmax(avmmol, fricvel));
    rr = (zn + 0.5 * HH) / zn;
    x = kappa / log(rr);
    rr = x * x;
  }
  r = rr * sqrt(uloc * uloc + vloc * vloc);
}
// velocity quotient, four-point mean and maximum of the bottom friction in its arithmetic
template <class T, class TI>
__device__ __forceinline__ T bf_quot(TI a, TI b) {
  if constexpr (sizeof(T) == 4) return __fdividef(float(a), float(b));
  else return a / b;
}
template <class T>
__device__ __forceinline__ T bf_mean(T a, T b, T c, T e) {
  if constexpr (sizeof(T) == 4) return __fmul_rn(0.25f, __fadd_rn(__fadd_rn(__fadd_rn(a, b), c), e));
  else return 0.25 * (a + b + c + e);
}
template <class T>
__device__ __forceinline__ T bf_max(T a, T b) {
  if constexpr (sizeof(T) == 4) return fmaxf(a, b);
  else return fmax(a, b);
}

// DIR 0: UEx on the U grid (fadv = U/DU, faces between U points); DIR 1: VEx on the V grid.
// TI: the storage type of U, V, DU, DV and Ex (FP64 state arrays, or the FP32 working copies of
// the mixed-precision micro step)
template <class TL, class T, int S, int DIR, class TI>
__device__ __forceinline__ void uvadv2d_tile(const Dev& d, T dt, const TI* __restrict__ U, const TI* __restrict__ V,
                                             const TI* __restrict__ DU, const TI* __restrict__ DV,
                                             const uint8_t* __restrict__ mflux_u,
                                             const uint8_t* __restrict__ mflux_v,
                                             const uint8_t* __restrict__ mupd_u, const uint8_t* __restrict__ mupd_v,
                                             TI* __restrict__ Ex, const Bf2Args<TI>& bf) {
  constexpr int FX = TL::FX, FY = TL::FY, RW = TL::RW, RH = TL::RH, FTY = TL::FTY, RPT = TL::RPT;
  extern __shared__ unsigned char smem_raw[];
  Adv2dSmem<T, TL>& sm = *reinterpret_cast<Adv2dSmem<T, TL>*>(smem_raw);
  const int ni = d.ni(), nj = d.nj();
  const long long sj = d.sj;
  const int ii0 = blockIdx.x * FX, jj0 = blockIdx.y * FY;
  constexpr int sub = (S == UPSTREAM) ? 0 : 1;
  const T half = T(0.5), one = T(1), zero = T(0);
  const T dxu = T(d.dx), dyu = T(d.dy), ard1 = T(d.ard1);
  // ---- stage: region cell (r, q) <-> array (jj0-2+r, ii0-4+q); thread (q, ty) takes column q
  const int q = threadIdx.x, ty = threadIdx.y;
  const int ii = ii0 - 4 + q;
  const bool iin = ii >= 0 && ii < ni;
  // SB region rows of a thread at a time, their loads issued together: small tiles (few blocks per SM, a
  // block's latency is the time) stage every row in one go, large ones (32 registers per thread) one
  constexpr int SB = RW == 32 ? (RH + FTY - 1) / FTY : 1;
  for (int rb = ty; rb < RH; rb += SB * FTY) {
    TI u0[SB], v0[SB], du0[SB], dv0[SB], u1[SB], v1[SB], du1[SB], dv1[SB];
    uint8_t a[SB], b[SB], c2[SB], e2[SB];
    bool in[SB], ok[SB];
#pragma unroll
    for (int m = 0; m < SB; ++m) {
      const int r = rb + m * FTY, jj = jj0 - 2 + r;
      in[m] = r < RH && iin && jj >= 0 && jj < nj;
      ok[m] = in[m] && (DIR == 0 ? (ii <= ni - 2) : (jj <= nj - 2));  // the next U (V) point exists
      const long long c = (long long)jj * sj + ii, cn = DIR == 0 ? c + 1 : c + sj;
      u0[m] = v0[m] = du0[m] = dv0[m] = u1[m] = v1[m] = du1[m] = dv1[m] = TI(0);
      a[m] = b[m] = c2[m] = e2[m] = 0;
      if (in[m]) {
        a[m] = mflux_u[c];
        b[m] = mflux_v[c];
        c2[m] = mupd_u[c];
        e2[m] = mupd_v[c];
        u0[m] = U[c];
        v0[m] = V[c];
        du0[m] = DU[c];
        dv0[m] = DV[c];
      }
      if (ok[m]) {
        u1[m] = U[cn];
        v1[m] = V[cn];
        du1[m] = DU[cn];
        dv1[m] = DV[cn];
      }
    }
#pragma unroll
    for (int m = 0; m < SB; ++m) {
      const int r = rb + m * FTY;
      if (SB > 1 && r >= RH) break;
      T f0 = zero, ua = zero, dua = zero, va = zero, dva = zero, dio = zero, oq = zero;
      if (in[m]) {
        if (bf.r) oq = DIR == 0 ? bf_quot<T>(v0[m], dv0[m]) : bf_quot<T>(u0[m], du0[m]);
        dio = T(DIR == 0 ? du0[m] : dv0[m]);
      }
      if (ok[m]) {
        // FP32 working copies: the approximate division (2 ulp); FP64 arrays: the reference's quotient
        if constexpr (sizeof(T) == 4 && sizeof(TI) == 4)
          f0 = DIR == 0 ? __fdividef(u0[m], du0[m]) : __fdividef(v0[m], dv0[m]);
        else
          f0 = T(DIR == 0 ? u0[m] / du0[m] : v0[m] / dv0[m]);
        ua = T(0.5 * (u0[m] + u1[m]));
        va = T(0.5 * (v0[m] + v1[m]));
        dua = T(0.5 * (du0[m] + du1[m]));
        dva = T(0.5 * (dv0[m] + dv1[m]));
      }
      sm.F0[r][q] = f0;
      sm.Q[r][q] = oq;
      sm.Ua[r][q] = ua;
      sm.DUa[r][q] = dua;
      sm.Va[r][q] = va;
      sm.DVa[r][q] = dva;
      sm.Di[r][q] = dio;
      sm.mfu[r][q] = a[m];
      sm.mfv[r][q] = b[m];
      sm.mpu[r][q] = c2[m];
      sm.mpv[r][q] = e2[m];
    }
  }
  __syncthreads();
  // ---- the sweeps. A thread takes region column qc of the rows below; the two warps of a row
  // overlap by one column (warp 0: qc = 0..31, warp 1: qc = 31..62; warp 1's copy of column 31,
  // `dup`, updates and stores nothing), so that the left face flux of every cell a u sweep updates
  // is the flux of the lane before it (a warp shuffle, no shared-memory round trip or barrier).
  // The own rows of a thread, r = 2 + ty + FTY*m (m < RPT), are the same in all three sweeps: their
  // depths and flux-divergence sums stay in registers.
  const int qc = q - (q >> 5);
  const bool dup = q == 32;
  const int iic = ii0 - 4 + qc;
  const bool qown = qc >= 4 && qc < FX + 4 && !dup;  // own cells q in [4, FX+4)
  T di[RPT], acc[RPT] = {};
  // ---- sweep 1: u/2 on rows r in [0, RH), cells q in [2, RW-2), faces q in [1, RW-3]
  {
    const T dti = half * dt, cdx = dti / dxu;
    const bool fok = qc >= 1 && qc <= RW - 3 && iic >= sub && iic <= ni - 2 - sub;  // face between qc, qc+1
    const bool cok = iic >= 1 + sub && iic <= ni - 2 - sub;
    const bool upd = qc >= 2 && qc < RW - 2 && !dup;
#pragma unroll
    for (int m = 0; m <= RPT; ++m) {
      // the own rows, then the halo rows 0, 1, RH-2, RH-1 (thread rows 0..3)
      const int r = m < RPT ? 2 + ty + FTY * m : (ty < 2 ? ty : RH - 4 + ty);
      if (m == RPT && ty >= 4) continue;
      T fl = zero;
      if (fok)
        fl = face_flux_s<T, S>(sm.Ua[r][qc], sm.DUa[r][qc], sm.F0[r][qc - 1], sm.F0[r][qc], sm.F0[r][qc + 1],
                               sm.F0[r][qc + 2], sm.mfu[r][qc - 1] != 0, sm.mfu[r][qc] != 0,
                               sm.mfu[r][qc + 1] != 0, dti, cdx, zero, false, dxu);
      const T flm = __shfl_up_sync(0xffffffffu, fl, 1);  // the face between qc-1 and qc
      if (upd) {
        const T fio = sm.F0[r][qc];
        T fnew = fio;
        T Dio = sm.Di[r][qc];
        if (cok && sm.mpu[r][qc]) {
          const T dD = diff_scaled<T>(dti, sm.Ua[r][qc], sm.Ua[r][qc - 1], dyu, ard1);
          const T Dn = Dio - dD;
          const T advn = diff_scaled<T>(half, fl, flm, dyu, ard1);
          fnew = fv_update<T>(Dio, dD, Dn, fio, dt, advn);
          Dio = Dn;
          if (m < RPT && qown) acc[m] = add_r<T>(acc[m], advn);
        }
        if (m < RPT) di[m] = Dio;
        sm.F1[r][qc] = fnew;
      }
    }
    __syncthreads();
  }
  // ---- sweep 2: v on columns q in [2, RW-2), cells r in [2, RH-2), faces r in [1, RH-3]
  {
    const T dti = one * dt, cdy = dti / dyu;
    const bool col = qc >= 2 && qc < RW - 2 && !dup;
    if (col)
      for (int r = 1 + ty; r <= RH - 3; r += FTY) {
        const int fa = jj0 - 2 + r;  // face between r and r+1
        T fl = zero;
        if (fa >= sub && fa <= nj - 2 - sub)
          fl = face_flux_s<T, S>(sm.Va[r][qc], sm.DVa[r][qc], sm.F1[r - 1][qc], sm.F1[r][qc], sm.F1[r + 1][qc],
                                 sm.F1[r + 2][qc], sm.mfv[r - 1][qc] != 0, sm.mfv[r][qc] != 0,
                                 sm.mfv[r + 1][qc] != 0, dti, cdy, zero, false, dyu);
        sm.FL[r][qc] = fl;
      }
    __syncthreads();
    if (col) {
#pragma unroll
      for (int m = 0; m < RPT; ++m) {
        const int r = 2 + ty + FTY * m;
        const int jj = jj0 - 2 + r;
        const T fio = sm.F1[r][qc];
        T fnew = fio;
        if (jj >= 1 + sub && jj <= nj - 2 - sub && sm.mpv[r][qc]) {
          const T Dio = di[m];
          const T dD = diff_scaled<T>(dti, sm.Va[r][qc], sm.Va[r - 1][qc], dxu, ard1);
          const T Dn = Dio - dD;
          const T advn = diff_scaled<T>(one, sm.FL[r][qc], sm.FL[r - 1][qc], dxu, ard1);
          fnew = fv_update<T>(Dio, dD, Dn, fio, dt, advn);
          if (qown) acc[m] = add_r<T>(acc[m], advn);
        }
        sm.F0[r][qc] = fnew;  // the field after v (F0 is no longer needed)
      }
    }
    __syncthreads();
  }
  // ---- sweep 3: u/2 on the own rows, own cells q in [4, RW-4), faces q in [3, RW-5]
  {
    const T dti = half * dt, cdx = dti / dxu;
    const bool fok = qc >= 3 && qc <= RW - 5 && iic >= sub && iic <= ni - 2 - sub;
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
      const int r = 2 + ty + FTY * m;
      T fl = zero;
      if (fok)
        fl = face_flux_s<T, S>(sm.Ua[r][qc], sm.DUa[r][qc], sm.F0[r][qc - 1], sm.F0[r][qc], sm.F0[r][qc + 1],
                               sm.F0[r][qc + 2], sm.mfu[r][qc - 1] != 0, sm.mfu[r][qc] != 0,
                               sm.mfu[r][qc + 1] != 0, dti, cdx, zero, false, dxu);
      const T flm = __shfl_up_sync(0xffffffffu, fl, 1);
      if (qown) {
        const int jj = jj0 - 2 + r;
        T a = acc[m];
        if (iic >= 1 + sub && iic <= ni - 2 - sub && jj < nj && sm.mpu[r][qc]) {
          const T advn = diff_scaled<T>(half, fl, flm, dyu, ard1);
          a = add_r<T>(a, advn);
        }
        if (iic < ni && jj < nj) Ex[(long long)jj * sj + iic] = (TI)a;
      }
    }
  }
  // ---- the bottom friction of the own points (bottom_friction.F90:48-150)
  if (bf.r && qown) {
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
      const int r = 2 + ty + FTY * m;
      const int jj = jj0 - 2 + r;
      if (iic >= ni || jj >= nj) continue;
      const long long c = (long long)jj * sj + iic;
      const int i = iic + d.imin - HALO, j = jj + d.jmin - HALO;
      const bool in = i >= d.imin && i <= d.imax && j >= d.jmin && j <= d.jmax;
      T uloc, vloc, HHl;
      if (DIR == 0) {
        if (!(i <= d.imax + HALO - 1 && bf.mask_at(c) > 0)) continue;
        vloc = in ? bf_mean<T>(sm.Q[r][qc], sm.Q[r][qc + 1], sm.Q[r - 1][qc], sm.Q[r - 1][qc + 1]) : zero;
        uloc = bf_quot<T>(U[c], DU[c]);
        HHl = bf_max<T>(T(bf.min_depth), T(DU[c]));
      } else {
        if (!(j <= d.jmax + HALO - 1 && bf.mask_at(c) > 0)) continue;
        if (in)
          uloc = bf_mean<T>(sm.Q[r][qc], sm.Q[r][qc - 1], sm.Q[r + 1][qc], sm.Q[r + 1][qc - 1]);
        else
          uloc = (i <= d.imax + HALO - 1 && bf.au_at(c) > 0) ? sm.Q[r][qc] : zero;
        vloc = bf_quot<T>(V[c], DV[c]);
        HHl = bf_max<T>(T(bf.min_depth), T(DV[c]));
      }
      T zn, rr, rv;
      if constexpr (sizeof(T) == 4) {
        const BfLaw b = bf_law_f32(float(bf.zb[c]), float(bf.zb0[c]), HHl, uloc, vloc, float(bf.kappa), float(bf.avmmol),
                                   bf.runtype);
        zn = b.zn;
        rr = b.rr;
        rv = b.r;
      } else {
        bf_law_f64(bf.zb[c], bf.zb0 ? bf.zb0[c] : 0.0, HHl, uloc, vloc, bf.kappa, bf.avmmol, bf.runtype, zn, rr, rv);
      }
      if (bf.runtype == 1) bf.zb[c] = (TI)zn;
      bf.rr[c] = (TI)rr;
      bf.r[c] = (TI)rv;
    }
  }
}

// Threads per SM the registers are held to. FP32 working copies in large tiles: 2048 (32 registers, no
// spills; the shared memory holds them): the issue-bound sweeps then have 64 warps to choose from
// instead of 48. FP64 arrays: 1024 (2048x2048, 20 micro steps: 20.6 ms; 27.1 at 512). Small tiles: 512, as
// they run one or two to an SM and 1024 spilled (128x96: 467 against 512 us).
template <class TI, class TL>
constexpr int adv2d_threads() { return TL::RW == 32 ? 512 : sizeof(TI) == 4 ? 2048 : 1024; }

// Both components in one launch (blockIdx.z = 0: UEx on the U grid, 1: VEx on the V grid): one grid,
// one tail.
struct Adv2dMasks {
  const uint8_t *mflux_u, *mflux_v, *mupd_u, *mupd_v;
};
template <class TL, class T, int S, class TI>
__global__ void __launch_bounds__(TL::FT, adv2d_threads<TI, TL>() / TL::FT)
    k_uvadv2d_both(Dev d, T dt, const TI* __restrict__ U, const TI* __restrict__ V, const TI* __restrict__ DU,
                   const TI* __restrict__ DV, Adv2dMasks mu, Adv2dMasks mv, TI* __restrict__ UEx, TI* __restrict__ VEx,
                   Bf2Args<TI> bfu, Bf2Args<TI> bfv) {
  chain_sync();
  if (blockIdx.z == 0)
    uvadv2d_tile<TL, T, S, 0, TI>(d, dt, U, V, DU, DV, mu.mflux_u, mu.mflux_v, mu.mupd_u, mu.mupd_v, UEx, bfu);
  else
    uvadv2d_tile<TL, T, S, 1, TI>(d, dt, U, V, DU, DV, mv.mflux_u, mv.mflux_v, mv.mupd_u, mv.mupd_v, VEx, bfv);
}

// T: arithmetic, TI: the 2D fields (FP64 state arrays or FP32 working copies)
template <class T, class TI>
int run_uvadv2d(const Dev& d, cudaStream_t s, T dt, int scheme, const TI* U, const TI* V, const TI* DU, const TI* DV,
                const uint8_t* const* mu, const uint8_t* const* mv, TI* UEx, TI* VEx, const Bf2Args<TI>* bfu,
                const Bf2Args<TI>* bfv) {
  return dispatch_scheme(scheme, [&](auto sc) {
    constexpr int S = decltype(sc)::value;
    auto go = [&](auto tile) -> int {
      using TL = decltype(tile);
      auto kern = k_uvadv2d_both<TL, T, S, TI>;
      const size_t smem = sizeof(Adv2dSmem<T, TL>);
      if (smem > 48 * 1024)
        if (const int e = allow_smem(kern, smem)) return e;
      const dim3 grd((d.ni() + TL::FX - 1) / TL::FX, (d.nj() + TL::FY - 1) / TL::FY, 2);
      return launch_chained(kern, grd, dim3(TL::RW, TL::FTY, 1), smem, s, d, dt, U, V, DU, DV,
                            Adv2dMasks{mu[0], mu[1], mu[2], mu[3]}, Adv2dMasks{mv[0], mv[1], mv[2], mv[3]}, UEx, VEx,
                            bfu ? *bfu : Bf2Args<TI>{}, bfv ? *bfv : Bf2Args<TI>{});
    };
    const long long large = 2LL * ((d.ni() + TileLarge::FX - 1) / TileLarge::FX) *
                            ((d.nj() + TileLarge::FY - 1) / TileLarge::FY);
    if (large < TILE2D_SMALL) return go(TileSmall());
    return go(TileLarge());
  });
}

}  // namespace gb
