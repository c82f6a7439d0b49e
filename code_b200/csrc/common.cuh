// common.cuh -- shared device-side definitions of the B200 hot-path library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/getm_b200.h"

namespace gb {

constexpr int HALO = 2;

// Index space of one context as the kernels see it (value copy of getm_domain).
struct Dev {
  int imin, imax, jmin, jmax, kmax;
  long long sj, sk;
  double dx, dy, ard1;
  // haloed extents
  __host__ __device__ int ni() const { return imax - imin + 1 + 2 * HALO; }
  __host__ __device__ int nj() const { return jmax - jmin + 1 + 2 * HALO; }
  // offset of (i,j) relative to the origin (imin-2, jmin-2)
  __host__ __device__ long long ix(int i, int j) const {
    return (long long)(i - (imin - HALO)) + (long long)(j - (jmin - HALO)) * sj;
  }
};

inline Dev to_dev(const getm_domain& d) {
  Dev v;
  v.imin = d.imin; v.imax = d.imax; v.jmin = d.jmin; v.jmax = d.jmax; v.kmax = d.kmax;
  v.sj = d.sj; v.sk = d.sk; v.dx = d.dx; v.dy = d.dy; v.ard1 = d.ard1;
  return v;
}

// Programmatic dependent launch for the chains of kernels of a step: a kernel launched by
// launch_chained is set up while its predecessor in the stream still runs, and every one of its
// threads calls chain_sync() before it touches memory, which waits until that one, and with it every
// kernel before, has completed with its writes visible. No kernel lets its successor start early: the
// waiting blocks would take its place on the SMs (barotropic 128 x 96, 20 micro steps: 783 us with plain
// launches, 617 with the successor released at the start, 556 released by completion; 2048x2048x50
// mixed step 33.3, 34.8, 33.1 ms). A kernel launched the plain way passes through chain_sync().
__device__ __forceinline__ void chain_sync() { cudaGridDependencySynchronize(); }
template <class... P, class... A>
inline int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// Levels that the column solvers hold in shared memory at most (getm_tridiagonal_columns, the mode-split
// state): the limit of the entry points.
constexpr int KMAX_COLUMNS = 199;

// Before a launch of more than 48 KB of dynamic shared memory. The limit belongs to the device's function,
// which all contexts and host threads share: `most` is the same for every launch of a kernel, since a
// limit set to one launch's own size could be lowered by another thread before that launch.
template <class K>
inline int allow_smem(K* kernel, size_t most) {
  return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// Scheme ids (advection.F90:60-62)
enum : int { NOADV = 0, UPSTREAM = 1, UPSTREAM_2DH = 2, P2 = 3, SUPERBEE = 4, MUSCL = 5, P2_PDM = 6 };

__host__ __device__ inline bool is_split_scheme(int s) {
  return s == UPSTREAM || s == P2 || s == SUPERBEE || s == MUSCL || s == P2_PDM;
}

// Reference-exact min/max (Fortran MIN/MAX on ordered operands).
template <class R>
__device__ __forceinline__ R rmin(R a, R b) { return (b < a) ? b : a; }
template <class R>
__device__ __forceinline__ R rmax(R a, R b) { return (b > a) ? b : a; }

// a / b as a times the approximate reciprocal of b: the bits of __fdividef (2 ulp) for every b from 2^-126
// to 2^126, subnormal a and quotients included, so tracers at the low end of FP32 keep their
// increments. __fdividef also scales its operands for a subnormal b, two or three instructions more
// for each of the sweeps' two or three divisions per face and cell (701x555x33 tracer step 492 against
// 462 us, 2048x2048x50 mixed step 33.85 against 32.8 ms); here such a b counts as zero. The divisors
// are layer heights and Courant numbers + 1e-10, far above 2^-126 wherever a cell is updated.
__device__ __forceinline__ float fdiv_fast(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return __fmul_rn(a, r);
}

// advection.F90:854-879 adv_interfacial_reconstruction_p2
template <class R>
__device__ __forceinline__ R recon_p2(R cfl, R fu, R deltafu, R deltaf) {
  const R one6th = R(1) / R(6);
  R x = one6th * (R(1) - R(2) * cfl);
  return fu + R(0.5) * (R(1) - cfl) * ((R(0.5) + x) * deltaf + (R(0.5) - x) * deltafu);
}

// advection.F90:785-845 adv_interfacial_reconstruction. Same expression order as the
// reference so that an FP64 build without contraction reproduces it bit for bit.
template <class R>
__device__ __forceinline__ R recon(int scheme, R cfl, R fuu, R fu, R fd) {
  const R one6th = R(1) / R(6);
  R deltaf = fd - fu;
  R deltafu = fu - fuu;
  if (deltaf * deltafu > R(0)) {
    R ratio = deltafu / deltaf;
    R limiter;
    if (scheme == SUPERBEE) {
      limiter = rmax(rmin(R(2) * ratio, R(1)), rmin(ratio, R(2)));
    } else if (scheme == P2_PDM) {
      R x = one6th * (R(1) - R(2) * cfl);
      limiter = (R(0.5) + x) + (R(0.5) - x) * ratio;
      limiter = rmin(rmin(R(2) * ratio / (cfl + R(1.e-10)), limiter), R(2) / (R(1) - cfl));
    } else if (scheme == MUSCL) {
      limiter = rmin(rmin(R(2) * ratio, R(0.5) * (R(1) + ratio)), R(2));
    } else if (scheme == P2) {
      return recon_p2(cfl, fu, deltafu, deltaf);
    } else {
      return fu;
    }
    return fu + R(0.5) * limiter * (R(1) - cfl) * deltaf;
  }
  if (scheme == P2) return recon_p2(cfl, fu, deltafu, deltaf);
  return fu;
}

// FP32 log-law bottom drag of one velocity point (bottom_friction.F90:86-103 / :121-138), shared by
// every FP32 form of the bottom friction so that they give the same bits: from the roughness zb,
// the point's depth HH and the velocity components, the drag coefficient rr and r = rr*|u|; with
// runtype 1 the roughness is first renewed from the friction velocity (zn, which the caller
// stores). Every operation is explicitly rounded (no dependence on multiply-add contraction); the
// divisions outside the logarithm's argument are the approximate ones (2 ulp).
struct BfLaw {
  float zn, rr, r;
};
__device__ __forceinline__ BfLaw bf_law_f32(float zb, float zb0, float HH, float uloc, float vloc, float kappa,
                                            float avmmol, int runtype) {
  const float h = 0.5f;
  const float sp = __fadd_rn(__fmul_rn(uloc, uloc), __fmul_rn(vloc, vloc));
  float x = __fdividef(kappa, logf(__fdiv_rn(__fadd_rn(zb, __fmul_rn(h, HH)), zb)));
  float rr = __fmul_rn(x, x);
  BfLaw o;
  o.zn = zb;
  if (runtype == 1) {
    const float fricvel = __fsqrt_rn(__fmul_rn(rr, sp));
    const float zn = fminf(HH, __fadd_rn(zb0, __fdividef(__fmul_rn(0.1f, avmmol), fmaxf(avmmol, fricvel))));
    o.zn = zn;
    x = __fdividef(kappa, logf(__fdiv_rn(__fadd_rn(zn, __fmul_rn(h, HH)), zn)));
    rr = __fmul_rn(x, x);
  }
  o.rr = rr;
  o.r = __fmul_rn(rr, __fsqrt_rn(sp));
  return o;
}

}  // namespace gb
