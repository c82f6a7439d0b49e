// adv_fused.cuh -- the horizontal split sweeps of one HALFSPLIT advection (advection_3d.F90:439-537,
// u/2 v/2 w v/2 u/2) as two launches instead of four: k_adv_uv runs u/2 then v/2, k_adv_vu runs v/2
// then u/2. Included by kernels_inst.cuh.
//
// What bounds it: run one by one, the four sweeps move 26 words per cell for a momentum component
// (field, transports, heights and flux sum in and out of HBM at every sweep) and 28 for a tracer
// pair; here the field between the two sweeps of a launch stays in registers, so a launch reads
// the field, the transports (and, second launch, heights and flux sum) once and writes the field,
// the heights and the flux sum once. What is left is instruction issue: the limiter of each face.
//
// Split of the work: a warp owns a strip of lanes along i, N cells a lane, and marches along j over
// a segment of rows of one level. In k_adv_uv the row that enters the window at j+2 is swept along i
// first (stencil neighbours and the right face flux by warp shuffles; the outermost lanes of the warp
// only supply them), then the four rows j-1..j+2 in registers give the flux of face j and the update
// of row j; the row segment's first four steps only fill the window (rows = 64: 6% more row sweeps). In
// k_adv_vu the v sweep of row j is followed by the u sweep of the same row. No barrier and no shared-memory
// exchange: each thread stages the inputs of its next rows in its own slots of a shared-memory ring by cp.async. Every face flux and cell update is the expression of the
// one-sweep kernels (sweeps_vec.cuh), so the results equal theirs bit for bit.
//
// Outer lanes and rows read cells that another warp updates, so no array a launch writes may be one
// it reads there: the field, the heights and the carried errors go to other arrays than they come
// from (the flux sum, which only a cell's owner touches, is updated in place).
//
// MOM (momentum advection of integrate_3d, uv_advect_3d.F90:62-460): U and V are the 3D transports
// uu, vv; the advected velocity uu/hun (vv/hvn), and the transports of the U (V) control volumes, means
// of neighbouring ones, are formed here instead of in a set-up pass that wrote eight 3D arrays.
#pragma once
#include "sweeps_vec.cuh"

namespace gb {

// Warps per block: consecutive levels of one strip and row segment, which read the same masks and column
// heights; an odd level is the only one whose block runs half empty, and those blocks come first, among
// full ones. (Four consecutive row segments per block left three warps of four idle in domains of up to 64
// rows: 1100x48x50 FP64 step of ten micro steps 1934 -> 1411 us. Four levels per block: the same there, but
// up to three idle warps, 64x250x30 FP64 606 against 576 us; one level: 1024x1024x40 FP64 tracer 2711 against
// 2671 us.)
constexpr int AW = 2;

// Blocks per SM the registers are held to (16 warps in FP32, 20 in FP64): the sweeps are bound by issue and by
// the fixed latency of dependent instructions, so warps count more than registers (2048x2048x50 mixed step,
// u/v passes: 8.1 ms at 16 warps, 8.8 unbounded; 1024x1024x50 FP64: 7.2 ms unbounded, 5.9 at 20 warps, 8.0 at 24)
template <class R>
constexpr int adv_blocks() { return sizeof(R) == 4 ? 8 : 10; }

// Cells a lane owns and lanes that only supply neighbours: a u sweep reads two cells to either side.
// The second launch's v sweep must be complete on the right outer cells; with MOM = 1 each of those
// takes the transport of the cell after it. Outer lanes cost 2 of 32 with two or four cells per lane, 4 (MOM = 1
// in the second launch: 5) with one.
template <int N>
struct LaneSplit {
  static constexpr int LH = N >= 2 ? 1 : 2;
  static constexpr int rh_uv = N >= 2 ? 1 : 2;
  template <int MOM>
  static constexpr int rh_vu() { return N >= 4 ? 1 : N == 2 ? (MOM == 1 ? 2 : 1) : (MOM == 1 ? 3 : 2); }
};

// Constants and level strides of a launch (strides 0: 2D arrays of column values).
template <class R>
struct AdvC {
  SweepC<R> u, v;             // u.skdu / v.skdu: face depths, u.skdi: heights read
  const R *U, *DU, *V, *DV;   // transports and face depths (MOM: uu, face depth, vv, face depth)
  const R* Di_src;            // heights before the launch
  R* Di_dst;                  // heights after it (may be null in k_adv_vu)
  R* adv;                     // flux-divergence sum (may be null)
  const uint8_t* flags;       // the grid's masks (ADV_FU ..), a byte per cell
  uint8_t *code_u, *code_v;   // limiter branches (REC)
};

// per-lane asynchronous copy of a vector of B bytes (4, 8 or 16), `bytes` of it read, the rest zero
template <int B>
__device__ __forceinline__ void cp_lane(unsigned smem, const void* gmem, int bytes) {
  if constexpr (B == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
  else if constexpr (B == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}

// Masks of an advection grid in one byte per cell: flux and update masks of the u and the v sweep.
__device__ __forceinline__ bool flag(uint32_t w, int m, int bit) { return ((w >> (8 * m)) & bit) != 0; }
// flag bytes of N cells as one word (byte m = cell c0+m); N = 1, 2 or 4
template <int N>
__device__ __forceinline__ uint32_t ld_mask_n(const uint8_t* p, bool full, int navail) {
  if constexpr (N == 1) return navail > 0 ? *p : 0u;
  else return ld_mask_w<N>(p, full, navail);
}
template <int N>
__device__ __forceinline__ void st_codes_n(uint8_t* p, bool full, int navail, const uint8_t (&v)[N]) {
  if constexpr (N == 1) {
    if (navail > 0) *p = v[0];
  } else {
    st_codes<N>(p, full, navail, v);
  }
}

// Fluxes of one face for NF fields with the same transport and masks: face_flux_s for each. FP32
// without branch codes: its values, formed from the differences of neighbouring cells (the face's
// and the upwind one), which adjacent faces share; the sign of the limited correction follows the
// flow.
template <class R, int S, bool REC, int NF>
__device__ __forceinline__ void face_fluxes(const SweepC<R>& C, bool use_AH, R Uf, R DUf, const R (&fm1)[NF],
                                            const R (&f0)[NF], const R (&f1)[NF], const R (&f2)[NF], bool mm1, bool m0,
                                            bool mp1, R (&fl)[NF], uint8_t* code) {
  if constexpr (sizeof(R) == 4 && !REC) {
    const bool pos = Uf > 0.f;
    const bool lim = pos ? mm1 : mp1;
    const float cfl = fdiv_fast(fabsf(Uf) * C.cdx, DUf);
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      float fu = pos ? f0[n] : f1[n];
      if constexpr (S == P2_PDM) {
        const float d0 = f1[n] - f0[n];
        const float ds = pos ? f0[n] - fm1[n] : f2[n] - f1[n];
        const Pdm32 p = pdm32(cfl, fabsf(ds), fabsf(d0));
        const float m = copysignf(fminf(fminf(p.v1, p.v2), fabsf(d0)), d0);
        const float val = fu + (pos ? m : -m);
        fu = (lim && d0 * ds > 0.f) ? val : fu;
      } else if constexpr (S != UPSTREAM) {
        const float val = recon_s<float, S>(cfl, pos ? fm1[n] : f2[n], fu, pos ? f1[n] : f0[n]);
        fu = lim ? val : fu;
      }
      float x = Uf * fu;
      if (use_AH) x = x - C.AH * DUf * (f1[n] - f0[n]) / C.dxf;
      fl[n] = m0 ? x : 0.f;
    }
  } else {
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      uint8_t c = 0;
      fl[n] = face_flux_s<R, S, REC>(Uf, DUf, fm1[n], f0[n], f1[n], f2[n], mm1, m0, mp1, C.dti, C.cdx, C.AH, use_AH,
                                     C.dxf, &c);
      if (REC && n == 0) *code = c;
    }
  }
}

// u sweep of one row held by the lanes of a warp: f (in and out), D (heights, in and out), the
// flux divergence `add` of updated cells (0 elsewhere), lo the packed carried errors. fw: the flags of
// the lane's cells, zero outside the row; fok / uok: bit m set where face c0+m-1 / cell c0+m is in the
// sweep's range.
template <class R, int S, bool REC, int NF, int N, bool LO>
__device__ __forceinline__ void u_row(const SweepC<R>& C, bool use_AH, R (&f)[NF][N], R (&D)[N], const R (&U)[N],
                                      const R (&DU)[N], uint32_t fw, unsigned fok, unsigned uok,
                                      R (&add)[NF][N], LoVec<N> (&lo)[NF], uint8_t (&cd)[N]) {
  constexpr unsigned FULL = 0xffffffffu;
  R e[NF][N + 3];  // cells c0-2 .. c0+N
#pragma unroll
  for (int n = 0; n < NF; ++n) {
    e[n][0] = N >= 2 ? __shfl_up_sync(FULL, f[n][N >= 2 ? N - 2 : 0], 1) : __shfl_up_sync(FULL, f[n][0], 2);
    e[n][1] = __shfl_up_sync(FULL, f[n][N - 1], 1);
#pragma unroll
    for (int m = 0; m < N; ++m) e[n][m + 2] = f[n][m];
    e[n][N + 2] = __shfl_down_sync(FULL, f[n][0], 1);
  }
  R Uv[N + 1], DUv[N];  // faces c0-1 .. c0+N-1 (depths: up to c0+N-2)
  Uv[0] = __shfl_up_sync(FULL, U[N - 1], 1);
  DUv[0] = __shfl_up_sync(FULL, DU[N - 1], 1);
#pragma unroll
  for (int m = 0; m < N; ++m) Uv[m + 1] = U[m];
#pragma unroll
  for (int m = 1; m < N; ++m) DUv[m] = DU[m - 1];
  bool mf[N + 2];  // flux masks of cells c0-2 .. c0+N-1
  if constexpr (N >= 2) {
    const uint32_t lw = __shfl_up_sync(FULL, fw, 1);
    mf[0] = flag(lw, N - 2, ADV_FU);
    mf[1] = flag(lw, N - 1, ADV_FU);
  } else {
    mf[0] = flag(__shfl_up_sync(FULL, fw, 2), 0, ADV_FU);
    mf[1] = flag(__shfl_up_sync(FULL, fw, 1), 0, ADV_FU);
  }
#pragma unroll
  for (int m = 0; m < N; ++m) mf[m + 2] = flag(fw, m, ADV_FU);
  R fl[NF][N + 1];
  uint8_t cl[N + 1];
#pragma unroll
  for (int m = 0; m < N; ++m) {
    R a[NF], b[NF], c[NF], g[NF], x[NF];
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      a[n] = e[n][m];
      b[n] = e[n][m + 1];
      c[n] = e[n][m + 2];
      g[n] = e[n][m + 3];
    }
    cl[m] = 0;
    face_fluxes<R, S, REC, NF>(C, use_AH, Uv[m], DUv[m], a, b, c, g, mf[m], ((fok >> m) & 1u) && mf[m + 1], mf[m + 2],
                               x, &cl[m]);
#pragma unroll
    for (int n = 0; n < NF; ++n) fl[n][m] = x[n];
  }
#pragma unroll
  for (int n = 0; n < NF; ++n) fl[n][N] = __shfl_down_sync(FULL, fl[n][0], 1);
  if constexpr (REC) {
    cl[N] = (uint8_t)__shfl_down_sync(FULL, (uint32_t)cl[0], 1);
#pragma unroll
    for (int m = 0; m < N; ++m) cd[m] = cl[m + 1];  // face c0+m, stored at its left cell
  }
  float sl[NF][N];
  if constexpr (LO) {
#pragma unroll
    for (int n = 0; n < NF; ++n) lo_unpack<N>(lo[n], sl[n]);
  }
#pragma unroll
  for (int m = 0; m < N; ++m) {
    const bool upd = ((uok >> m) & 1u) && flag(fw, m, ADV_PU);
    const R dD = cell_dD<R>(C, Uv[m + 1], Uv[m]);
    const R Dn = D[m] - dD;
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      const R advn = cell_advn<R>(C, fl[n][m + 1], fl[n][m]);
      if constexpr (LO) {
        float s = sl[n][m];
        const R v = fv_update_lo<R>(D[m], dD, Dn, f[n][m], C.dt, advn, s);
        if (upd) sl[n][m] = s;
        f[n][m] = upd ? v : f[n][m];
      } else if constexpr (sizeof(R) == 8) {
        if (upd) f[n][m] = fv_update<R>(D[m], dD, Dn, f[n][m], C.dt, advn);
      } else {
        const R v = fv_update<R>(D[m], dD, Dn, f[n][m], C.dt, advn);
        f[n][m] = upd ? v : f[n][m];
      }
      add[n][m] = upd ? advn : R(0);
    }
    D[m] = upd ? Dn : D[m];
  }
  if constexpr (LO) {
#pragma unroll
    for (int n = 0; n < NF; ++n) lo[n] = lo_pack<N>(sl[n]);
  }
}

// v sweep of row j from the window w (rows j-1..j+2 of each field): the flux of face j into fl, and
// the update of the row's cells from the faces below (flo, Vp) and above (fl, Vc).
template <class R, int S, bool REC, int NF, int N>
__device__ __forceinline__ void v_face(const SweepC<R>& C, bool use_AH, const R (&w)[NF][4][N], const R (&Vc)[N],
                                       const R (&DVc)[N], uint32_t w0, uint32_t w1, uint32_t w2, bool valid,
                                       R (&fl)[NF][N], uint8_t (&cd)[N]) {
#pragma unroll
  for (int m = 0; m < N; ++m) {
    R a[NF], b[NF], c[NF], g[NF], x[NF];
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      a[n] = w[n][0][m];
      b[n] = w[n][1][m];
      c[n] = w[n][2][m];
      g[n] = w[n][3][m];
    }
    cd[m] = 0;
    face_fluxes<R, S, REC, NF>(C, use_AH, Vc[m], DVc[m], a, b, c, g, flag(w0, m, ADV_FV),
                               valid && flag(w1, m, ADV_FV), flag(w2, m, ADV_FV), x, &cd[m]);
#pragma unroll
    for (int n = 0; n < NF; ++n) fl[n][m] = x[n];
  }
}
template <class R, int S, int NF, int N, bool LO>
__device__ __forceinline__ void v_update(const SweepC<R>& C, R (&f)[NF][N], R (&D)[N], const R (&Vc)[N], const R (&Vp)[N],
                                         const R (&fl)[NF][N], const R (&flo)[NF][N], uint32_t fw, bool jin,
                                         R (&add)[NF][N], LoVec<N> (&lo)[NF]) {
  float sl[NF][N];
  if constexpr (LO) {
#pragma unroll
    for (int n = 0; n < NF; ++n) lo_unpack<N>(lo[n], sl[n]);
  }
#pragma unroll
  for (int m = 0; m < N; ++m) {
    const bool upd = jin && flag(fw, m, ADV_PV);
    const R dD = cell_dD<R>(C, Vc[m], Vp[m]);
    const R Dn = D[m] - dD;
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      const R advn = cell_advn<R>(C, fl[n][m], flo[n][m]);
      if constexpr (LO) {
        float s = sl[n][m];
        const R v = fv_update_lo<R>(D[m], dD, Dn, f[n][m], C.dt, advn, s);
        if (upd) sl[n][m] = s;
        f[n][m] = upd ? v : f[n][m];
      } else if constexpr (sizeof(R) == 8) {
        if (upd) f[n][m] = fv_update<R>(D[m], dD, Dn, f[n][m], C.dt, advn);
      } else {
        const R v = fv_update<R>(D[m], dD, Dn, f[n][m], C.dt, advn);
        f[n][m] = upd ? v : f[n][m];
      }
      add[n][m] = upd ? advn : R(0);
    }
    D[m] = upd ? Dn : D[m];
  }
  if constexpr (LO) {
#pragma unroll
    for (int n = 0; n < NF; ++n) lo[n] = lo_pack<N>(sl[n]);
  }
}

// The tracer fields of a launch: src -> dst, carried errors lo_src -> lo_dst (LO)
template <class R, int NF>
struct AdvF {
  const R* src[NF];
  R* dst[NF];
  const __half* lo_src[NF];
  __half* lo_dst[NF];
};

// Geometry of a warp: its strip, level and row segment. Rows outside the domain (and, through zero
// bytes, lanes outside the row) only reach faces that the sweeps leave out, so their addresses are
// clamped to the first and last row. In-plane offsets are 32-bit.
#define GB_ADV_LANES(OWN_, LH_)                                                                  \
  const int lane = threadIdx.x;                                                                  \
  const int tid = threadIdx.y * 32 + lane;                                                       \
  const int ni = d.ni(), nj = d.nj();                                                            \
  const int c0 = (blockIdx.x * (OWN_) + lane - (LH_)) * N;                                       \
  const int j0 = blockIdx.y * rows, kz = nk - (int)(gridDim.z - blockIdx.z) * AW + (int)threadIdx.y; \
  if (kz < 0) return; /* whole warp (no barrier in these kernels) */                           \
  const int j1 = min(j0 + rows, nj);                                                             \
  const bool act = c0 >= 0 && c0 < ni;                                                           \
  const int navail = act ? ni - c0 : 0;                                                          \
  const bool full = navail >= N;                                                                 \
  const int nav = full ? N : navail;                                                             \
  const int vbytes = nav * (int)sizeof(R);                                                       \
  const bool own = act && lane >= (LH_) && lane < (LH_) + (OWN_);                                \
  const unsigned cc = act ? c0 : 0; /* a valid column for the lanes outside the row */          \
  const unsigned sj = (unsigned)d.sj;                                                            \
  const long long lev = (long long)kz * d.sk;                                                    \
  const R *const Ul = C.U + lev, *const Vl = C.V + lev;                                          \
  const R *const DUl = C.DU + kz * C.u.skdu, *const DVl = C.DV + kz * C.v.skdu,                  \
          *const Dil = C.Di_src + kz * C.u.skdi;                                                 \
  auto off = [&](int j) -> unsigned { return (unsigned)min(max(j, 0), nj - 1) * sj + cc; };      \
  const bool use_AH = C.u.AH > R(0);                                                             \
  unsigned fok = 0, uok = 0; /* faces c0+m-1 and cells c0+m in the u sweep's range */           \
  _Pragma("unroll") for (int m = 0; m < N; ++m) {                                                \
    const int fa = c0 + m - 1, c = c0 + m;                                                       \
    if (fa >= sub && fa <= ni - 2 - sub) fok |= 1u << m;                                         \
    if (c >= 1 + sub && c <= ni - 2 - sub) uok |= 1u << m;                                       \
  }                                                                                              \
  constexpr unsigned ARR = 32 * AW * VB, STG = NA * ARR;                                         \
  const unsigned sb = (unsigned)__cvta_generic_to_shared(&sbuf[0][0][tid]);                      \
  const unsigned sl0 = (unsigned)__cvta_generic_to_shared(&slo[0][0][tid]);                      \
  auto put = [&](int st, int q, const R* p) { cp_lane<VB>(sb + st * STG + q * ARR, p, vbytes); }; \
  auto put_lo = [&](int st, int n, const __half* p) {                                            \
    if constexpr (N > 1) cp_lane<2 * N>(sl0 + (st * NF + n) * (32 * AW * 2 * N), p, nav * 2);    \
  };                                                                                             \
  auto get = [&](int st, int q, R (&v)[N]) { lds_vec<R, N>(sbuf[st][q][tid], v); };              \
  auto frow = [&](int j) -> uint32_t { return ld_mask_n<N>(C.flags + off(j), full, navail); };

// value of the cell to the right of each of the lane's cells
template <class R, int N>
__device__ __forceinline__ void right_of(const R (&v)[N], R (&r)[N]) {
#pragma unroll
  for (int m = 0; m + 1 < N; ++m) r[m] = v[m + 1];
  r[N - 1] = __shfl_down_sync(0xffffffffu, v[0], 1);
}

template <class R, int S, bool REC, int NF, int N, bool LO, int MOM>
__global__ void __launch_bounds__(32 * AW, adv_blocks<R>()) k_adv_uv(Dev d, AdvC<R> C, AdvF<R, NF> F, int nk, int rows) {
  chain_sync();
  constexpr int VB = N * (int)sizeof(R);
  constexpr int LH = LaneSplit<N>::LH, OWN = 32 - LH - LaneSplit<N>::rh_uv;
  constexpr int sub = (S == UPSTREAM) ? 0 : 1;
  // slots: the fields (MOM: uu or vv) of row j+2; U of row j+2 (MOM 1: none, MOM 2: uu of row j+3);
  // DU, Di of row j+2; V of row j (MOM 2: none), DV of row j; the carried errors of row j+2
  constexpr int XU = NF, XDU = XU + 1, XDI = XU + 2, XV = XU + 3, XDV = XU + 4, NA = NF + 5;
  __shared__ VecPack<R, N> sbuf[VST][NA][32 * AW];
  __shared__ LoVec<N> slo[LO ? VST : 1][NF][32 * AW];
  GB_ADV_LANES(OWN, LH)
  auto issue = [&](int j, int st) {
    if (j < j1) {
      const unsigned r = off(j + 2), q = off(j);
      if constexpr (MOM == 0) {
#pragma unroll
        for (int n = 0; n < NF; ++n) put(st, n, F.src[n] + lev + r);
        put(st, XU, Ul + r);
      } else if constexpr (MOM == 1) {
        put(st, 0, Ul + r);
      } else {
        put(st, 0, Vl + r);
        put(st, XU, Ul + off(j + 3));
      }
      put(st, XDU, DUl + r);
      put(st, XDI, Dil + r);
      if constexpr (MOM != 2) put(st, XV, Vl + q);
      put(st, XDV, DVl + q);
      if constexpr (LO) {
#pragma unroll
        for (int n = 0; n < NF; ++n) put_lo(st, n, F.lo_src[n] + lev + r);
      }
    }
    cp_async_commit();
  };
  R w[NF][4][N], fl_old[NF][N], Vp[N];
  R D1[N], D2[N], D3[N];                 // heights after the u sweep of rows j, j+1, j+2
  R a1[NF][N], a2[NF][N], a3[NF][N];     // its flux divergences (with adv)
  LoVec<N> l1[NF], l2[NF], l3[NF];       // carried errors after it (LO)
  R x1[MOM == 2 ? N : 1], x2[MOM == 2 ? N : 1], x3[MOM == 2 ? N : 1];  // MOM 2: vv of rows j, j+1, j+2
  R un[MOM == 2 ? N : 1];                // MOM 2: uu of row j+2 (read one row ahead)
#pragma unroll
  for (int m = 0; m < N; ++m) {
    Vp[m] = D1[m] = D2[m] = D3[m] = R(0);
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      fl_old[n][m] = a1[n][m] = a2[n][m] = a3[n][m] = R(0);
#pragma unroll
      for (int q = 0; q < 4; ++q) w[n][q][m] = R(0);
    }
  }
#pragma unroll
  for (int n = 0; n < NF; ++n) l1[n] = l2[n] = l3[n] = LoVec<N>{};
  if constexpr (MOM == 2) {
#pragma unroll
    for (int m = 0; m < N; ++m) x1[m] = x2[m] = x3[m] = R(0);
    ld_row<R, N>(Ul + off(j0 - 2), full, navail, un);  // the first row entering
  }
  const int jb = j0 - 4;
#pragma unroll
  for (int q = 0; q < VST - 1; ++q) issue(jb + q, q);
  // flags of rows j-1 .. j+2, and of row j+3 a step ahead
  uint32_t g0 = frow(jb - 1), g1 = frow(jb), g2 = frow(jb + 1), g3 = frow(jb + 2);
  int st = 0;
  for (int j = jb; j < j1; ++j) {
    issue(j + VST - 1, st == 0 ? VST - 1 : st - 1);
    const int jr = j + 2;
    const uint32_t gn = frow(j + 3);
    LoVec<N> lq[NF];
    if constexpr (LO && N == 1) {  // two bytes: below the smallest asynchronous copy
#pragma unroll
      for (int n = 0; n < NF; ++n)
        lq[n] = __half_as_ushort(F.lo_src[n][lev + off(jr)]);
    }
    cp_async_wait<VST - 1>();
    // ---- the row entering the window: the u sweep of row jr
    R f[NF][N], U[N], DU[N];
    get(st, XDU, DU);
#pragma unroll
    for (int m = 0; m < N; ++m) {
      D1[m] = D2[m];
      D2[m] = D3[m];
    }
    get(st, XDI, D3);
    if constexpr (MOM == 0) {
#pragma unroll
      for (int n = 0; n < NF; ++n) get(st, n, f[n]);
      get(st, XU, U);
    } else {
      // uv_advect_3d.F90:76-98 (U grid, MOM 1) / :267-289 (V grid, MOM 2); no values in the last
      // column (row), whose faces and cells are outside the sweeps
      R x[N];
      get(st, 0, x);
      const bool rowok = MOM == 1 || jr < nj - 1;
#pragma unroll
      for (int m = 0; m < N; ++m) f[0][m] = (rowok && c0 + m >= 0 && c0 + m < (MOM == 1 ? ni - 1 : ni)) ? x[m] / D3[m] : R(0);
      if constexpr (MOM == 1) {
        R xr[N];
        right_of<R, N>(x, xr);
#pragma unroll
        for (int m = 0; m < N; ++m) U[m] = R(0.5) * (x[m] + xr[m]);
      } else {
        R uq[N];
        get(st, XU, uq);
#pragma unroll
        for (int m = 0; m < N; ++m) {
          U[m] = R(0.5) * (un[m] + uq[m]);
          un[m] = uq[m];
          x1[m] = x2[m];
          x2[m] = x3[m];
          x3[m] = x[m];
        }
      }
    }
    if constexpr (LO && N > 1) {
#pragma unroll
      for (int n = 0; n < NF; ++n) lq[n] = slo[st][n][tid];
    }
    R add[NF][N];
    uint8_t cd[N];
    u_row<R, S, REC, NF, N, LO>(C.u, use_AH, f, D3, U, DU, g3, fok, uok, add, lq, cd);
    if (REC && own && jr >= j0 && jr < j1) st_codes_n<N>(C.code_u + lev + off(jr), full, navail, cd);
#pragma unroll
    for (int n = 0; n < NF; ++n) {
#pragma unroll
      for (int m = 0; m < N; ++m) {
        w[n][0][m] = w[n][1][m];
        w[n][1][m] = w[n][2][m];
        w[n][2][m] = w[n][3][m];
        w[n][3][m] = f[n][m];
        a1[n][m] = a2[n][m];
        a2[n][m] = a3[n][m];
        a3[n][m] = add[n][m];
      }
      l1[n] = l2[n];
      l2[n] = l3[n];
      l3[n] = lq[n];
    }
    if (j >= j0 - 1) {
      // ---- the v sweep of row j
      R Vc[N], DVc[N], fl[NF][N];
      if constexpr (MOM == 2) {
#pragma unroll
        for (int m = 0; m < N; ++m) Vc[m] = R(0.5) * (x1[m] + x2[m]);
      } else {
        get(st, XV, Vc);
        if constexpr (MOM == 1) {
          R xr[N];
          right_of<R, N>(Vc, xr);
#pragma unroll
          for (int m = 0; m < N; ++m) Vc[m] = R(0.5) * (Vc[m] + xr[m]);
        }
      }
      get(st, XDV, DVc);
      const bool fvalid = j >= sub && j <= nj - 2 - sub;
      v_face<R, S, REC, NF, N>(C.v, use_AH, w, Vc, DVc, g0, g1, g2, fvalid, fl, cd);
      if (j >= j0) {
        const bool jin = j >= 1 + sub && j <= nj - 2 - sub;
        R fo[NF][N], addv[NF][N];
#pragma unroll
        for (int n = 0; n < NF; ++n)
#pragma unroll
          for (int m = 0; m < N; ++m) fo[n][m] = w[n][1][m];
        v_update<R, S, NF, N, LO>(C.v, fo, D1, Vc, Vp, fl, fl_old, g1, jin, addv, l1);
        if (own) {
          const long long p = lev + off(j);
          if (REC) st_codes_n<N>(C.code_v + p, full, navail, cd);
#pragma unroll
          for (int n = 0; n < NF; ++n) {
            st_row<R, N>(F.dst[n] + p, full, navail, fo[n]);
            if constexpr (LO) {
              float sl[N];
              lo_unpack<N>(l1[n], sl);
              st_lo<N>(F.lo_dst[n] + p, full, navail, sl);
            }
          }
          st_row<R, N>(C.Di_dst + p, full, navail, D1);
          if (NF == 1 && C.adv) {
            R ad[N];
#pragma unroll
            for (int m = 0; m < N; ++m) ad[m] = (R(0) + a1[0][m]) + addv[0][m];
            st_row<R, N>(C.adv + p, full, navail, ad);
          }
        }
      }
#pragma unroll
      for (int n = 0; n < NF; ++n)
#pragma unroll
        for (int m = 0; m < N; ++m) fl_old[n][m] = fl[n][m];
#pragma unroll
      for (int m = 0; m < N; ++m) Vp[m] = Vc[m];
    }
    g0 = g1;
    g1 = g2;
    g2 = g3;
    g3 = gn;
    st = st == VST - 1 ? 0 : st + 1;
  }
  cp_async_wait<0>();
}

template <class R, int S, bool REC, int NF, int N, bool LO, int MOM>
__global__ void __launch_bounds__(32 * AW, adv_blocks<R>()) k_adv_vu(Dev d, AdvC<R> C, AdvF<R, NF> F, int nk, int rows) {
  chain_sync();
  constexpr int VB = N * (int)sizeof(R);
  constexpr int LH = LaneSplit<N>::LH, OWN = 32 - LH - LaneSplit<N>::template rh_vu<MOM>();
  constexpr int sub = (S == UPSTREAM) ? 0 : 1;
  // slots: the fields of row j+2; V and DV of row j (MOM 2: vv of row j+1); U, DU, Di of row j (MOM
  // 2: uu of row j+1), the flux sum (one field) and the carried errors of row j
  constexpr int XV = NF, XDV = XV + 1, XU = XV + 2, XDU = XV + 3, XDI = XV + 4, XAD = XV + 5, NA = NF + (NF == 1 ? 6 : 5);
  __shared__ VecPack<R, N> sbuf[VST][NA][32 * AW];
  __shared__ LoVec<N> slo[LO ? VST : 1][NF][32 * AW];
  GB_ADV_LANES(OWN, LH)
  auto issue = [&](int j, int st) {
    if (j < j1) {
      const unsigned q = off(j), r2 = off(j + 2);
#pragma unroll
      for (int n = 0; n < NF; ++n) put(st, n, F.src[n] + lev + r2);
      if (j >= j0 - 1) {
        const unsigned r1 = MOM == 2 ? off(j + 1) : q;
        put(st, XV, Vl + r1);
        put(st, XDV, DVl + q);
        if (j >= j0) {
          put(st, XU, Ul + r1);
          put(st, XDU, DUl + q);
          put(st, XDI, Dil + q);
          if (NF == 1 && C.adv) put(st, XAD, C.adv + lev + q);
          if constexpr (LO) {
#pragma unroll
            for (int n = 0; n < NF; ++n) put_lo(st, n, F.lo_src[n] + lev + q);
          }
        }
      }
    }
    cp_async_commit();
  };
  R w[NF][4][N], fl_old[NF][N], Vp[N];
  R un[MOM == 2 ? N : 1], vn[MOM == 2 ? N : 1];  // MOM 2: uu and vv of row j (read one row ahead)
#pragma unroll
  for (int m = 0; m < N; ++m) {
    Vp[m] = R(0);
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      fl_old[n][m] = R(0);
#pragma unroll
      for (int q = 0; q < 4; ++q) w[n][q][m] = R(0);
    }
  }
  if constexpr (MOM == 2) {
    ld_row<R, N>(Ul + off(j0), full, navail, un);
    ld_row<R, N>(Vl + off(j0 - 1), full, navail, vn);
  }
  const int jb = j0 - 4;
#pragma unroll
  for (int q = 0; q < VST - 1; ++q) issue(jb + q, q);
  // flags of rows j-1, j, j+1, and of row j+2 a step ahead
  uint32_t g0 = frow(j0 - 2), g1 = frow(j0 - 1), g2 = frow(j0);
  int st = 0;
  for (int j = jb; j < j1; ++j) {
    issue(j + VST - 1, st == 0 ? VST - 1 : st - 1);
    cp_async_wait<VST - 1>();
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      R x[N];
      get(st, n, x);
#pragma unroll
      for (int m = 0; m < N; ++m) {
        w[n][0][m] = w[n][1][m];
        w[n][1][m] = w[n][2][m];
        w[n][2][m] = w[n][3][m];
        w[n][3][m] = x[m];
      }
    }
    if (j >= j0 - 1) {
      const uint32_t gn = frow(j + 2);
      // ---- the v sweep of row j (all lanes)
      R Vc[N], DVc[N], fl[NF][N];
      uint8_t cd[N];
      get(st, XV, Vc);
      get(st, XDV, DVc);
      if constexpr (MOM == 1) {
        R xr[N];
        right_of<R, N>(Vc, xr);
#pragma unroll
        for (int m = 0; m < N; ++m) Vc[m] = R(0.5) * (Vc[m] + xr[m]);
      } else if constexpr (MOM == 2) {
#pragma unroll
        for (int m = 0; m < N; ++m) {
          const R x = Vc[m];
          Vc[m] = R(0.5) * (vn[m] + x);
          vn[m] = x;
        }
      }
      v_face<R, S, REC, NF, N>(C.v, use_AH, w, Vc, DVc, g0, g1, g2, j >= sub && j <= nj - 2 - sub, fl, cd);
      if (j >= j0) {
        const long long p = lev + off(j);
        if (REC && own) st_codes_n<N>(C.code_v + p, full, navail, cd);
        R f[NF][N], D[N], addv[NF][N], addu[NF][N], U[N], DU[N];
        LoVec<N> lq[NF];
#pragma unroll
        for (int n = 0; n < NF; ++n) {
#pragma unroll
          for (int m = 0; m < N; ++m) f[n][m] = w[n][1][m];
          if constexpr (LO && N > 1) lq[n] = slo[st][n][tid];
          if constexpr (LO && N == 1) lq[n] = __half_as_ushort(F.lo_src[n][p]);
        }
        get(st, XDI, D);
        v_update<R, S, NF, N, LO>(C.v, f, D, Vc, Vp, fl, fl_old, g1, j >= 1 + sub && j <= nj - 2 - sub, addv, lq);
        // ---- the u sweep of row j
        get(st, XU, U);
        get(st, XDU, DU);
        if constexpr (MOM == 1) {
          R xr[N];
          right_of<R, N>(U, xr);
#pragma unroll
          for (int m = 0; m < N; ++m) U[m] = R(0.5) * (U[m] + xr[m]);
        } else if constexpr (MOM == 2) {
#pragma unroll
          for (int m = 0; m < N; ++m) {
            const R x = U[m];
            U[m] = R(0.5) * (un[m] + x);
            un[m] = x;
          }
        }
        u_row<R, S, REC, NF, N, LO>(C.u, use_AH, f, D, U, DU, g1, fok, uok, addu, lq, cd);
        if (own) {
          if (REC) st_codes_n<N>(C.code_u + p, full, navail, cd);
#pragma unroll
          for (int n = 0; n < NF; ++n) {
            if (F.dst[n]) st_row<R, N>(F.dst[n] + p, full, navail, f[n]);
            if constexpr (LO) {
              float sl[N];
              lo_unpack<N>(lq[n], sl);
              st_lo<N>(F.lo_dst[n] + p, full, navail, sl);
            }
          }
          if (C.Di_dst) st_row<R, N>(C.Di_dst + p, full, navail, D);
          if (NF == 1 && C.adv) {
            R ad[N];
            get(st, XAD, ad);
#pragma unroll
            for (int m = 0; m < N; ++m) ad[m] = (ad[m] + addv[0][m]) + addu[0][m];
            st_row<R, N>(C.adv + p, full, navail, ad);
          }
        }
      }
#pragma unroll
      for (int n = 0; n < NF; ++n)
#pragma unroll
        for (int m = 0; m < N; ++m) fl_old[n][m] = fl[n][m];
#pragma unroll
      for (int m = 0; m < N; ++m) Vp[m] = Vc[m];
      g0 = g1;
      g1 = g2;
      g2 = gn;
    }
    st = st == VST - 1 ? 0 : st + 1;
  }
  cp_async_wait<0>();
}
#undef GB_ADV_LANES
}  // namespace gb
