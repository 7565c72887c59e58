// Kernels of the explicit residual-and-update path, compiled once per arithmetic mode.
//
// Included by kernels_exact.cu (TY_KNS = kexact, TY_FAST = 0, compiled with -fmad=false:
// every FP64 operation separately rounded, in Typhon's order) and kernels_fast.cu
// (TY_KNS = kfast, TY_FAST = 1, fused multiply-add and precomputed weights).
//
// Typhon routines restated (file:line of the Fortran reference):
//   k_prim          SOURCE/EQNS/calc_varprim_ns.f90:43-54
//   k_ghost_prim    SOURCE/MGRID/calcboco_connect_per_match.f90:56-78 (periodic copy),
//                   SOURCE/MGRID/calcboco_ust_sym.f90 (symmetry mirror)
//   k_grad          SOURCE/MGRID/calc_gradient.f90:67-196 + SOURCE/MATH/MATRIX.f90:79-111
//   k_ghost_grad    SOURCE/MGRID/calcboco_gen.f90:78-84 (connections only)
//   recon           SOURCE/EQNS/hres_ns_musclfast.f90, hres_ns_muscl.f90, hres_ns_muscluns.f90,
//                   tvdgrad{fst,str,uns}_{scal,vect}.f90, SOURCE/MGRID/LIMITER.f90
//   k_barth         SOURCE/MGRID/postlimit_barth.f90:42-223
//   flux_*          SOURCE/EQNS/calc_flux_hllc.f90:61-171, calc_roe_states.f90:35-53,
//                   calc_flux_rusanov.f90:57-83; Roe: new (Roe 1981 + Harten fix)
//   k_gather        SOURCE/MAIN/flux_to_res.f90:47-144 (colour-ordered sums, as a gather)
//   k_rk_update     SOURCE/MAIN/treelevel_rungekutta.f90:60-113, SOURCE/ZONE/update_field.f90:38
//   k_timestep      SOURCE/EQNS/calc_ns_timestep.f90:52-103
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>
#include <utility>

#include "../../include/typhon_gpu.h"
#include "devmesh.hpp"
#include "fastmath.cuh"

#ifndef TY_KNS
#error "define TY_KNS and TY_FAST before including kernels.cuh"
#endif

namespace tyk {
namespace TY_KNS {

constexpr bool kFast = TY_FAST;
constexpr int kBlock = 256;

// Programmatic dependent launch: a kernel launched by launch_pdl is set up while its predecessor
// on the stream drains, and may start before it has finished; pdl_wait() returns when it has,
// and its writes are visible (at once in a kernel launched normally).  Every kernel so launched
// calls it before it touches anything that a kernel writes (mesh tables copied at creation may
// be read earlier), so completion is transitive along the stream.  Their parameters carry no
// __restrict__: a compiler may take such data as constant and read it ahead of the wait.  The gap
// between the short kernels of a Runge-Kutta stage shrinks from 2.7 to 0.2 us.  No kernel calls
// launch_dependents: blocks of the next kernel then fill the SMs that have room first and stay
// there, which doubled the 8,192-cell vortex's step (75 -> 150 us).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline void launch_pdl(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t st, A&&... a) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, std::forward<A>(a)...);
}

__device__ __forceinline__ double d3(const double* a, int ld, int i, int k) { return a[k * (size_t)ld + i]; }

// Rotational periodicity (calcboco_connect_per_match.f90:56-78, transvec_per): the velocity
// (q[2..4]) of a state taken from the partner of periodic face f, rotated into f's frame.
__device__ __forceinline__ void rot_to_face(const DevMesh& m, int f, double* q) {
  if (!m.frot) return;
  const size_t lf = m.ldf;
  double R[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) R[k] = m.frot[k * lf + f];
  const double x = q[2], y = q[3], z = q[4];
  q[2] = R[0] * x + R[1] * y + R[2] * z;
  q[3] = R[3] * x + R[4] * y + R[5] * z;
  q[4] = R[6] * x + R[7] * y + R[8] * z;
}

// ---------------------------------------------------------------------------
// Limiters (LIMITER.f90).  Scalars (rho, p) pass through the array forms, vector
// components through the scalar forms, as tvdgrad*_scal / tvdgrad*_vect call them.
__device__ __forceinline__ double sgn1(double x) { return signbit(x) ? -1.0 : 1.0; }

__device__ double lim_scalar_form(int lim, double x1, double x2) {
  switch (lim) {
    case TY_LIM_MINMOD: {
      double s = 0.5 * (sgn1(x1) + sgn1(x2));
      return s * fmin(fabs(x1), fabs(x2));
    }
    case TY_LIM_ALBADA: {
      double s = x1 * x2;
      if (s <= 0.0) return 0.0;
      return s * (x1 + x2) / (x1 * x1 + x2 * x2);
    }
    case TY_LIM_VLEER: {
      double s = x1 * x2;
      if (s <= 0.0) return 0.0;
      return 2.0 * s / (x1 + x2);
    }
    case TY_LIM_SUPERBEE: {
      double r = 0.0;
      if (x1 > 0.0 && x2 > 0.0) r = fmax(fmin(2.0 * x1, x2), fmin(2.0 * x2, x1));
      if (x1 < 0.0 && x2 < 0.0) r = fmin(fmax(2.0 * x1, x2), fmax(2.0 * x2, x1));
      return r;
    }
    case TY_LIM_KIM3: {
      double r = 0.0;
      if (x1 > 0.0 && x2 > 0.0) { r = (2.0 * x1 + x2) / 3.0; r = fmin(fmin(2.0 * x1, 2.0 * x2), r); }
      if (x1 < 0.0 && x2 < 0.0) { r = (2.0 * x1 + x2) / 3.0; r = fmax(fmax(2.0 * x1, 2.0 * x2), r); }
      return r;
    }
    case TY_LIM_LIM03: {
      double eta = (x1 * x1 + x2 * x2) / 0.01 / 0.01;
      double r = 0.0;
      if (eta < 1.0) r = (2.0 * x2 + x1) / 3.0;
      else if (x1 > 0.0 && x2 > 0.0) { r = (2.0 * x2 + x1) / 3.0; r = fmin(fmin(1.6 * x2, 2.0 * x1), r); }
      else if (x1 < 0.0 && x2 < 0.0) { r = (2.0 * x2 + x1) / 3.0; r = fmax(fmax(1.6 * x2, 2.0 * x1), r); }
      else if (x1 < 0.0 && x2 > 0.0) { r = (2.0 * x2 + x1) / 3.0; r = fmax(0.0, fmin(-0.5 * x1, r)); }
      else if (x1 > 0.0 && x2 < 0.0) { r = (2.0 * x2 + x1) / 3.0; r = fmin(0.0, fmax(-0.5 * x1, r)); }
      return r;
    }
  }
  return 0.0;
}
__device__ double lim_array_form(int lim, double x1, double x2) {
  switch (lim) {
    case TY_LIM_MINMOD:
      if (x1 > 0.0 && x2 > 0.0) return fmin(x1, x2);
      if (x1 < 0.0 && x2 < 0.0) return fmax(x1, x2);
      return 0.0;
    case TY_LIM_ALBADA:
      if ((x1 > 0.0 && x2 > 0.0) || (x1 < 0.0 && x2 < 0.0)) return x1 * x2 * (x1 + x2) / (x1 * x1 + x2 * x2);
      return 0.0;
    case TY_LIM_VLEER:
      if ((x1 > 0.0 && x2 > 0.0) || (x1 < 0.0 && x2 < 0.0)) return 2.0 * x1 * x2 / (x1 + x2);
      return 0.0;
    default:
      return lim_scalar_form(lim, x1, x2);
  }
}
// slope limiter of the MUSCL variants: lim(2g - LR, LR) for FAST/str, lim(g, LR) for UNS;
// KIM3 takes its arguments swapped
__device__ __forceinline__ double apply_lim(int lim, bool uns, bool arrayform, double g, double LR) {
  double a = uns ? g : 2.0 * g - LR, b = LR;
  if (lim == TY_LIM_KIM3) { double t = a; a = b; b = t; }
  return arrayform ? lim_array_form(lim, a, b) : lim_scalar_form(lim, a, b);
}

// ---------------------------------------------------------------------------
// cons -> prim (calc_varprim_ns.f90:43-54)
__device__ __forceinline__ void cons_to_prim(double gamma, const double c[5], double q[5]) {
  const double g1 = gamma - 1.0;
  double rho = c[0];
  double vx, vy, vz;
  if constexpr (kFast) {
    const double ir = rcp_nr(rho);
    vx = c[2] * ir; vy = c[3] * ir; vz = c[4] * ir;
  } else {
    vx = c[2] / rho; vy = c[3] / rho; vz = c[4] / rho;
  }
  double ec = 0.5 * rho * (vx * vx + vy * vy + vz * vz);
  q[0] = rho;
  q[1] = g1 * (c[1] - ec);
  q[2] = vx; q[3] = vy; q[4] = vz;
}

__global__ void k_prim(DevMesh m, const double* cons, double* prim, double gamma) {
  pdl_wait();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  double u[5], q[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) u[v] = cons[v * (size_t)m.ldc + c];
  cons_to_prim(gamma, u, q);
#pragma unroll
  for (int v = 0; v < 5; ++v) prim[v * (size_t)m.ldc + c] = q[v];
}

// x^1.5: 0 for x = 0 (and below the normal numbers, whose result underflows), where the root's
// reciprocal is infinite; NaN for x < 0
template <class T>
__device__ __forceinline__ T pow15_nr(T x) {
  const T r = x * x * rsqrt_nr(x);
  return ((unsigned)__double2hiint(value(x)) << 1) < (2u << 20) ? T(0.0) : r;
}

// calc_viscosity (SOURCE/EQNS/EQNS.f90:225-265): nu rho, or Sutherland with AIR's constants
__device__ __forceinline__ double viscosity(const SpatOpts& o, double rho, double T) {
  if (o.visc_law == TY_VISC_KINEMATIC) return o.visc_kin * rho;
  const double mu0 = 0.0000168, T0 = 273.00, S = 110.50;
  if constexpr (kFast) {
    const double x = T * (1.0 / T0);
    return mu0 * (T0 + S) * pow15_nr(x) * rcp_nr(T + S);
  }
  return mu0 * pow(T / T0, 1.5) * (T0 + S) / (T + S);
}

// far-field ghost state (new), kind fixed by the free-stream normal velocity (see ty_bc)
__device__ __forceinline__ void farfield_state(const SpatOpts& o, double nx, double ny, double nz, const double* q,
                                               double* out) {
  const double* qi = o.farfield;
  const double vn = qi[2] * nx + qi[3] * ny + qi[4] * nz;
  const double c = sqrt(o.gamma * qi[1] / qi[0]);
  if (vn <= -c) {
#pragma unroll
    for (int v = 0; v < 5; ++v) out[v] = qi[v];
  } else if (vn < -1e-8 * c) {
    out[0] = qi[0]; out[1] = q[1]; out[2] = qi[2]; out[3] = qi[3]; out[4] = qi[4];
  } else if (vn < c) {
    out[0] = q[0]; out[1] = qi[1]; out[2] = q[2]; out[3] = q[3]; out[4] = q[4];
  } else {
#pragma unroll
    for (int v = 0; v < 5; ++v) out[v] = q[v];
  }
}

// inlet / outlet states from the inside state qi (setboco_ns_inlet_sub.f90:64-96,
// setboco_ns_outlet_sub.f90:31-60, setboco_ns_inlet_sup.f90:75-101, setboco_ns_outlet_sup.f90)
// with the isentropic relations of EQNS.f90:139-219 (pi_ti_mach_dir2nspri,
// pi_ti_ps_dir2nspri, nspri2pi_ti_mach_dir), in their operation order
__device__ void inout_state(const DevMesh& m, const SpatOpts& o, int f, int kind, const double* qi, double* qo) {
  if (kind == TY_BC_OUTLET_SUP) {
#pragma unroll
    for (int v = 0; v < 5; ++v) qo[v] = qi[v];
    return;
  }
  const double g = o.gamma, r = o.rgas, g1 = g - 1.0;
  const size_t lf = m.ldf;
  const double* D = m.fbcd + f;
  if (kind == TY_BC_INLET_SUP) {
    const double dx = D[3 * lf], dy = D[4 * lf], dz = D[5 * lf];
    const double dn = sqrt(dx * dx + dy * dy + dz * dz);
    const double mach = D[2 * lf];
    const double fm = 1.0 / (1.0 + .5 * g1 * (mach * mach));
    const double ts = D[lf] * fm;
    const double a = sqrt(g * r * ts);
    qo[1] = D[0] * pow(fm, g / g1);
    qo[0] = qo[1] / (r * ts);
    const double va = mach * a;
    qo[2] = va * (dx / dn); qo[3] = va * (dy / dn); qo[4] = va * (dz / dn);
    return;
  }
  double pi, ti, ps, ux, uy, uz;
  if (kind == TY_BC_INLET_SUB) {
    pi = D[0]; ti = D[lf]; ps = qi[1];
    const double dx = D[2 * lf], dy = D[3 * lf], dz = D[4 * lf];
    const double dn = sqrt(dx * dx + dy * dy + dz * dz);
    ux = dx / dn; uy = dy / dn; uz = dz / dn;
  } else {  // TY_BC_OUTLET_SUB: totals and direction of the inside state
    double fmv = qi[2] * qi[2] + qi[3] * qi[3] + qi[4] * qi[4];
    const double n = sqrt(fmv);
    ux = qi[2] / n; uy = qi[3] / n; uz = qi[4] / n;
    fmv = fmv / (g * qi[1]) * qi[0];
    fmv = 1.0 + 0.5 * g1 * fmv;
    pi = qi[1] * pow(fmv, g / g1);
    ti = qi[1] / r / qi[0] * fmv;
    ps = D[0];
  }
  double fm = pow(pi / ps, g1 / g);
  if (fm < 1.0) fm = 1.0;  // Typhon: "Bad ratio Pi/P : truncated to 1."
  qo[1] = ps;
  qo[0] = ps / (r * ti) * fm;
  const double va = sqrt((fm - 1.0) * 2.0 / g1) * sqrt(g * ps / qo[0]);
  qo[2] = va * ux; qo[3] = va * uy; qo[4] = va * uz;
}

// ghost states: periodic copy, symmetry mirror (velocity reflected across the face),
// adiabatic moving wall (setboco_ns_flux.f90, cell-state mode: pressure copied, temperature
// of the cell minus lflux d / conduct with lflux = 0, velocity reflected about the wall's)
__global__ void k_ghost_prim(DevMesh m, double* prim, SpatOpts o) {
  pdl_wait();
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m.ng) return;
  const int g = m.nci + k, src = m.gsrc[k], f = m.gface[k];
  const size_t ld = m.ldc;
  const int kind = m.fbc[f];
  double vx = prim[2 * ld + src], vy = prim[3 * ld + src], vz = prim[4 * ld + src];
  if (kind == TY_BC_FARFIELD || kind >= TY_BC_INLET_SUB) {
    double q[5], out[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) q[v] = prim[v * ld + src];
    if (kind == TY_BC_FARFIELD)
      farfield_state(o, d3(m.fn, m.ldf, f, 0), d3(m.fn, m.ldf, f, 1), d3(m.fn, m.ldf, f, 2), q, out);
    else
      inout_state(m, o, f, kind, q, out);
#pragma unroll
    for (int v = 0; v < 5; ++v) prim[v * ld + g] = out[v];
    return;
  }
  if (kind == TY_BC_WALL || kind == TY_BC_NOSLIP) {
    const double r = o.rgas, lflux = 0.0;
    const double rho = prim[src], p = prim[ld + src];
    if constexpr (kFast) {  // lflux = 0: the wall's temperature is the cell's, its density too
      prim[ld + g] = p;
      prim[g] = rho;
      prim[2 * ld + g] = fma(2.0, d3(m.fwall, m.ldf, f, 0), -vx);
      prim[3 * ld + g] = fma(2.0, d3(m.fwall, m.ldf, f, 1), -vy);
      prim[4 * ld + g] = fma(2.0, d3(m.fwall, m.ldf, f, 2), -vz);
      return;
    }
    const double mu = viscosity(o, rho, p / (r * rho));
    const double cp = o.gamma / (o.gamma - 1.0) * r;
    const double conduct = mu * cp / o.prandtl;
    const double temp = p / (rho * r) - lflux * m.gdist[k] / conduct;
    prim[ld + g] = p;
    prim[g] = p / (r * temp);
    prim[2 * ld + g] = (2.0 * d3(m.fwall, m.ldf, f, 0)) - vx;
    prim[3 * ld + g] = (2.0 * d3(m.fwall, m.ldf, f, 1)) - vy;
    prim[4 * ld + g] = (2.0 * d3(m.fwall, m.ldf, f, 2)) - vz;
    return;
  }
  prim[g] = prim[src];
  prim[ld + g] = prim[ld + src];
  if (kind == TY_BC_PERIODIC && m.frot) {
    double q[5] = {0.0, 0.0, vx, vy, vz};
    rot_to_face(m, f, q);
    vx = q[2]; vy = q[3]; vz = q[4];
  }
  if (kind == TY_BC_SYMMETRY) {
    double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
    double wx = vx - 0.0, wy = vy - 0.0, wz = vz - 0.0;
    double dn = 2.0 * (wx * nx + wy * ny + wz * nz);
    vx = vx - dn * nx; vy = vy - dn * ny; vz = vz - dn * nz;
  }
  prim[2 * ld + g] = vx;
  prim[3 * ld + g] = vy;
  prim[4 * ld + g] = vz;
}

// Comparisons of doubles run on the FP64 pipe (a minimum is a comparison and a select); on bit
// patterns they run on the integer pipe.
__device__ __forceinline__ long long order_key(double x) {  // orders like x
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double min_bits(double a, double b) { return order_key(a) < order_key(b) ? a : b; }
__device__ __forceinline__ double max_bits(double a, double b) { return order_key(a) < order_key(b) ? b : a; }
__device__ __forceinline__ bool is_nan(double x) {  // of the quiet NaNs that arithmetic makes
  return ((unsigned)__double2hiint(x) << 1) > (0x7ffu << 21);
}
__device__ __forceinline__ bool is_neg(double x) { return __double2hiint(x) < 0; }  // sign bit
// x without the sign (fabs of a stored value is an FP64 instruction)
__device__ __forceinline__ double abs_bits(double x) {
  return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}

__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }

// x == 0 on the integer pipe (on the 32-bit halves: the compiler turns a test of the 64-bit
// pattern back into an FP64 comparison)
__device__ __forceinline__ bool is_zero(double x) {
  return (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) == 0u;
}

// |x| as an FP32 number, truncated (relative error below 2^-23) on the integer pipe, when x lies
// in [2^-60, 2^60); ok is cleared otherwise.
__device__ __forceinline__ float trunc32(double x, bool& ok) {
  const int hi = __double2hiint(x) & 0x7fffffff;
  ok = ok && (unsigned)(hi - ((1023 - 60) << 20)) < (unsigned)(120 << 20);
  return __uint_as_float(__funnelshift_l((unsigned)__double2loint(x), (unsigned)hi, 3) - ((1023u - 127u) << 23));
}

// Exact mode: double arithmetic issued as F64 (fastmath.cuh: the same rounded values, and at
// -fmad=false nothing is contracted); the fast mode's compiler contracts plain doubles itself.
using X64 = typename std::conditional<kFast, double, F64>::type;

// a / b correctly rounded for several a and one b: with y = 1/b correctly rounded, q0 = a y
// corrected once by its residual is within an ulp of a/b, and corrected again it is the
// correctly rounded quotient (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34 (1990): q + (a - b q) y with exact residual).
// Five fused multiply-adds where an IEEE division issues about ten FP64 instructions.  Exponents are
// limited so that no residual leaves the normal range; zeros keep their sign (q0); anything else sets
// `bad` and is divided by div_ieee.
struct Divisor {
  F64 b, y;
  bool ok;
};
__device__ __forceinline__ Divisor divisor(double b) {
  return {b, 1.0 / b, ((unsigned)(__double2hiint(b) >> 20) & 0x7ffu) - 823u <= 400u};
}
__device__ __forceinline__ F64 quotient(F64 a, const Divisor& d, bool& bad) {
  const unsigned hi = (unsigned)__double2hiint(a.v);
  const bool zero = ((hi << 1) | (unsigned)__double2loint(a.v)) == 0u;
  bad = bad || !d.ok || (!zero && ((hi >> 20) & 0x7ffu) - 323u > 1400u);
  const F64 q0 = a * d.y, q1 = fma(fma(-d.b, q0, a), d.y, q0), q2 = fma(fma(-d.b, q1, a), d.y, q1);
  return zero ? q0.v : q2.v;
}
__device__ __noinline__ double div_ieee(double a, double b) { return a / b; }
__device__ __forceinline__ F64 quotient(F64 a, const Divisor& d) {
  bool bad = false;
  F64 q = quotient(a, d, bad);
  if (bad) q = div_ieee(a.v, d.b.v);
  return q;
}

// A cell's face list read ahead of its use (and of the wait): one trip to L2 less.
__device__ __forceinline__ void face_list(const DevMesh& m, int c, int es[kMaxSlot]) {
#pragma unroll
  for (int sl = 0; sl < kMaxSlot; ++sl) es[sl] = sl < m.nslot ? m.cf[sl * (size_t)m.nci + c] : -1;
}

// ---------------------------------------------------------------------------
// least-squares gradient: b_c = sum_f (q(fc2) - q(fc1)) d_f over the cell's faces in colour
// order, then the Cholesky solve (exact) or, in fast mode, the precomputed A^-1 d weights.
// The solve divides by three numbers, ten times each: their reciprocals once and quotient().
// 87,880 tetrahedra: 95 us with IEEE divisions, 60 us.
__device__ __noinline__ double3 cholesky_ieee(double x1, double x2, double x3, double L11, double L21, double L31,
                                              double L22, double L32, double L33) {
  x1 = x1 / L11;
  x2 = x2 - L21 * x1;
  x2 = x2 / L22;
  x3 = x3 - L31 * x1;
  x3 = x3 - L32 * x2;
  x3 = x3 / L33;
  x3 = x3 / L33;
  x2 = x2 - L32 * x3;
  x2 = x2 / L22;
  x1 = x1 - L21 * x2;
  x1 = x1 - L31 * x3;
  x1 = x1 / L11;
  return make_double3(x1, x2, x3);
}

__global__ void __launch_bounds__(kBlock) k_grad(DevMesh m, DevState s) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  int es[kMaxSlot];
  face_list(m, c, es);
  pdl_wait();
  const size_t ld = m.ldc, n = m.nci;
  X64 b[15];
#pragma unroll
  for (int k = 0; k < 15; ++k) b[k] = 0.0;
  const double* __restrict__ prim = s.prim;
#pragma unroll
  for (int sl = 0; sl < kMaxSlot; ++sl) {
    const int e = es[sl];
    if (e < 0) break;
    const int f = e >> 1;
    const int i1 = m.fc1[f], i2 = m.fc2[f];
    const int side = kFast ? e & 1 : 0;
    const double* w = kFast ? m.lsqw : m.dcg;
    const X64 wx = d3(w, m.ldf, f, 3 * side), wy = d3(w, m.ldf, f, 3 * side + 1), wz = d3(w, m.ldf, f, 3 * side + 2);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const X64 dsca = X64(prim[v * ld + i2]) - X64(prim[v * ld + i1]);
      b[3 * v] = b[3 * v] + dsca * wx;
      b[3 * v + 1] = b[3 * v + 1] + dsca * wy;
      b[3 * v + 2] = b[3 * v + 2] + dsca * wz;
    }
  }
  if constexpr (!kFast) {
    const F64 L21 = m.lsq[n + c], L31 = m.lsq[2 * n + c], L32 = m.lsq[4 * n + c];
    const Divisor L11 = divisor(m.lsq[c]), L22 = divisor(m.lsq[3 * n + c]), L33 = divisor(m.lsq[5 * n + c]);
    // cholesky_solve (MATRIX.f90:79-111), column per variable
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      bool bad = false;
      const F64 y1 = quotient(b[3 * v], L11, bad);
      const F64 y2 = quotient(b[3 * v + 1] - L21 * y1, L22, bad);
      const F64 y3 = quotient((b[3 * v + 2] - L31 * y1) - L32 * y2, L33, bad);
      const F64 x3 = quotient(y3, L33, bad);
      const F64 x2 = quotient(y2 - L32 * x3, L22, bad);
      const F64 x1 = quotient((y1 - L21 * x2) - L31 * x3, L11, bad);
      double3 x = make_double3(x1.v, x2.v, x3.v);
      if (bad)
        x = cholesky_ieee(value(b[3 * v]), value(b[3 * v + 1]), value(b[3 * v + 2]), L11.b.v, L21.v, L31.v, L22.b.v, L32.v,
                          L33.b.v);
      s.grad[3 * v * ld + c] = x.x;
      s.grad[(3 * v + 1) * ld + c] = x.y;
      s.grad[(3 * v + 2) * ld + c] = x.z;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 15; ++k) s.grad[k * ld + c] = value(b[k]);
  }
}

__global__ void k_ghost_grad(DevMesh m, double* grad) {
  pdl_wait();
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m.ng) return;
  const int f = m.gface[k];
  if (m.fbc[f] != TY_BC_PERIODIC) return;
  const int g = m.nci + k, src = m.gsrc[k];
  const size_t ld = m.ldc;
  if (!m.frot) {
#pragma unroll
    for (int v = 0; v < 15; ++v) grad[v * ld + g] = grad[v * ld + src];
    return;
  }
  // rotational periodicity: the scalar gradients are vectors, R g (transvec_per); the velocity
  // gradient G(i,j) = du_i/dx_j becomes G R^T (transten_per -> t3d_rot, TENSOR3.f90:328-340)
  const size_t lf = m.ldf;
  double R[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) R[q] = m.frot[q * lf + f];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double x = grad[(3 * q) * ld + src], y = grad[(3 * q + 1) * ld + src], z = grad[(3 * q + 2) * ld + src];
    grad[(3 * q) * ld + g] = R[0] * x + R[1] * y + R[2] * z;
    grad[(3 * q + 1) * ld + g] = R[3] * x + R[4] * y + R[5] * z;
    grad[(3 * q + 2) * ld + g] = R[6] * x + R[7] * y + R[8] * z;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double G0 = grad[(6 + 3 * i) * ld + src], G1 = grad[(7 + 3 * i) * ld + src], G2 = grad[(8 + 3 * i) * ld + src];
#pragma unroll
    for (int j = 0; j < 3; ++j) grad[(6 + 3 * i + j) * ld + g] = G0 * R[3 * j] + G1 * R[3 * j + 1] + G2 * R[3 * j + 2];
  }
}

// ---------------------------------------------------------------------------
// High-order face state on one side of face f (side 0: cell fc1 "L", side 1: cell fc2 "R").
// LR: (q(fc2) - q(fc1)) / |C_L C_R|, the same for both sides (slopes_lr).
__device__ __forceinline__ void slopes_lr(const DevMesh& m, const DevState& s, int f, X64 LR[5]) {
  const int icl = m.fc1[f], icr = m.fc2[f];
  if constexpr (kFast) {
    const double id = rcp_nr(m.dLR[f]);
#pragma unroll
    for (int v = 0; v < 5; ++v) LR[v] = (s.prim[v * (size_t)m.ldc + icr] - s.prim[v * (size_t)m.ldc + icl]) * id;
  } else {
    const Divisor d = divisor(m.dLR[f]);
#pragma unroll
    for (int v = 0; v < 5; ++v)
      LR[v] = value(quotient(F64(s.prim[v * (size_t)m.ldc + icr]) - F64(s.prim[v * (size_t)m.ldc + icl]), d));
  }
}

__device__ __forceinline__ void recon(const DevMesh& m, const DevState& s, const SpatOpts& o, int f, int side,
                                      const X64 LR[5], double q[5]) {
  const size_t ld = m.ldc;
  const int c = side ? m.fc2[f] : m.fc1[f];
  const double* __restrict__ prim = s.prim;
#pragma unroll
  for (int v = 0; v < 5; ++v) q[v] = prim[v * ld + c];
  if (o.highres == TY_HRES_NONE) return;
  const double* __restrict__ gr = s.grad;
  const X64 ux = d3(m.uLR, m.ldf, f, 0), uy = d3(m.uLR, m.ldf, f, 1), uz = d3(m.uLR, m.ldf, f, 2);
  if (o.highres == TY_HRES_MUSCLFAST) {
    const double k = side ? m.kRF[f] : m.kLF[f];
    // scalars (tvdgradfst_scal.f90:35-57)
#pragma unroll
    for (int sv = 0; sv < 2; ++sv) {
      double sg;
      if (o.limiter == TY_LIM_NONE) {
        sg = value(LR[sv]);
      } else {
        X64 g = X64(gr[(3 * sv) * ld + c]) * ux + X64(gr[(3 * sv + 1) * ld + c]) * uy + X64(gr[(3 * sv + 2) * ld + c]) * uz;
        sg = apply_lim(o.limiter, false, true, value(g), value(LR[sv]));
      }
      q[sv] = q[sv] + sg * k;
    }
    // velocity (tvdgradfst_vect.f90:36-58)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double sg;
      if (o.limiter == TY_LIM_NONE) {
        sg = value(LR[2 + i]);
      } else {
        X64 g = X64(gr[(6 + 3 * i) * ld + c]) * ux + X64(gr[(7 + 3 * i) * ld + c]) * uy + X64(gr[(8 + 3 * i) * ld + c]) * uz;
        sg = apply_lim(o.limiter, false, false, value(g), value(LR[2 + i]));
      }
      q[2 + i] = q[2 + i] + k * sg;
    }
    return;
  }
  // MUSCL / MUSCL-UNS (tvdgradstr_*.f90, tvdgraduns_*.f90)
  const bool uns = o.highres == TY_HRES_MUSCLUNS;
  const double* CF = side ? m.RF : m.LF;
  const X64 cx = d3(CF, m.ldf, f, 0), cy = d3(CF, m.ldf, f, 1), cz = d3(CF, m.ldf, f, 2);
#pragma unroll
  for (int sv = 0; sv < 2; ++sv) {
    X64 gx = gr[(3 * sv) * ld + c], gy = gr[(3 * sv + 1) * ld + c], gz = gr[(3 * sv + 2) * ld + c];
    const X64 g = gx * ux + gy * uy + gz * uz;
    const X64 sg = o.limiter == TY_LIM_NONE ? LR[sv] - g : X64(apply_lim(o.limiter, uns, true, value(g), value(LR[sv]))) - g;
    gx = gx + sg * ux; gy = gy + sg * uy; gz = gz + sg * uz;
    q[sv] = value(X64(q[sv]) + (gx * cx + gy * cy + gz * cz));
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const X64 T0 = gr[(6 + 3 * i) * ld + c], T1 = gr[(7 + 3 * i) * ld + c], T2 = gr[(8 + 3 * i) * ld + c];
    const X64 g = T0 * ux + T1 * uy + T2 * uz, lr = LR[2 + i];
    const X64 sg = o.limiter == TY_LIM_NONE ? lr - g : X64(apply_lim(o.limiter, uns, false, value(g), value(lr))) - g;
    const X64 t0 = T0 + sg * ux, t1 = T1 + sg * uy, t2 = T2 + sg * uz;
    q[2 + i] = value(X64(q[2 + i]) + (t0 * cx + t1 * cy + t2 * cz));
  }
}

// one side of a face by itself
__device__ void recon(const DevMesh& m, const DevState& s, const SpatOpts& o, int f, int side, double q[5]) {
  X64 LR[5];
  if (o.highres != TY_HRES_NONE) slopes_lr(m, s, f, LR);
  recon(m, s, o, f, side, LR, q);
}

// moving adiabatic wall, face-state mode (setboco_ns_flux.f90): the right state takes the left
// state's pressure as its density, its pressure, and the velocity reflected about the wall's
__device__ __forceinline__ void wall_state(const DevMesh& m, int f, const double* QL, double* QR) {
  QR[0] = m.fbc[f] == TY_BC_NOSLIP ? QL[0] : QL[1];  // TY_BC_NOSLIP: the inside density (new)
  QR[1] = QL[1];
  QR[2] = (2.0 * d3(m.fwall, m.ldf, f, 0)) - QL[2];
  QR[3] = (2.0 * d3(m.fwall, m.ldf, f, 1)) - QL[3];
  QR[4] = (2.0 * d3(m.fwall, m.ldf, f, 2)) - QL[4];
}

// velocity mirrored across the face plane (calcboco_ust_sym.f90, face-state mode)
__device__ __forceinline__ void mirror(const DevMesh& m, int f, double q[5]) {
  double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  double wx = q[2] - 0.0, wy = q[3] - 0.0, wz = q[4] - 0.0;
  double dn = 2.0 * (wx * nx + wy * ny + wz * nz);
  q[2] = q[2] - dn * nx; q[3] = q[3] - dn * ny; q[4] = q[4] - dn * nz;
}

// ---------------------------------------------------------------------------
// Riemann fluxes per unit area, F = (mass, energy, momentum x, y, z)

// Outer wave speeds of the HLL family (calc_flux_hllc.f90:64-124, calc_flux_hlle.f90:64-120):
// beta = 1 (HLLC, HLLE, K) or sqrt((g-1)/(2g)) (B, KB variants); the kinetic variants take the
// EFM estimates c (m kinw + kind), m = vn/c -+ f1 beta, c = a/f1, kinw = (1 -+ erf m)/2,
// kind = -+ f2 exp(-m^2).  Standard HLLE speeds are clamped to 0, the kinetic ones are not.
__device__ __forceinline__ void hll_speeds(const SpatOpts& o, double vnl, double vnr, double al, double ar, double vm,
                                           double am, double& sl, double& sr) {
  const double beta = o.hll_beta;
  if (o.hll_kin) {
    const double f1 = o.hll_f1, f2 = o.hll_f2;
    const double cl = al / f1, cr = ar / f1;
    const double modml = vnl / cl - f1 * beta, modmr = vnr / cr + f1 * beta;
    const double kinwl = 0.5 * (1.0 - erf(modml)), kinwr = 0.5 * (1.0 + erf(modmr));
    const double kindl = -f2 * exp(-modml * modml), kindr = +f2 * exp(-modmr * modmr);
    sl = fmin(cl * (modml * kinwl + kindl), vm - am);
    sr = fmax(cr * (modmr * kinwr + kindr), vm + am);
  } else if (o.hll_family == 2) {
    sl = fmin(fmin(0.0, vnl - beta * al), vm - am);
    sr = fmax(fmax(0.0, vnr + beta * ar), vm + am);
  } else {
    sl = fmin(vnl - beta * al, vm - am);
    sr = fmax(vnr + beta * ar, vm + am);
  }
}

// calc_flux_hlle.f90:83-150 (beta = 1), the Roe average of calc_roe_states.f90:37-53
__device__ void flux_hlle(const SpatOpts& o, const double* L, const double* R, double nx, double ny, double nz,
                          double* F) {
  const double g = o.gamma;
  const double ig1 = 1.0 / (g - 1.0);
  const double gig1 = g / (g - 1.0);
  double t1 = sqrt(R[0] / L[0]);
  double roe_rho = L[0] * t1;
  double kl0 = 1.0 / (1.0 + t1);
  double kr0 = t1 * kl0;
  double rux = kl0 * L[2] + kr0 * R[2], ruy = kl0 * L[3] + kr0 * R[3], ruz = kl0 * L[4] + kr0 * R[4];
  double sqL = L[2] * L[2] + L[3] * L[3] + L[4] * L[4];
  double sqR = R[2] * R[2] + R[3] * R[3] + R[4] * R[4];
  double h1 = gig1 * L[1] / L[0] + 0.5 * sqL;
  double h2 = gig1 * R[1] / R[0] + 0.5 * sqR;
  h1 = kl0 * h1 + kr0 * h2;
  double roe_p = (h1 - 0.5 * (rux * rux + ruy * ruy + ruz * ruz)) * roe_rho / gig1;
  double vnl = L[2] * nx + L[3] * ny + L[4] * nz;
  double vnr = R[2] * nx + R[3] * ny + R[4] * nz;
  double al = sqrt(g * L[1] / L[0]);
  double ar = sqrt(g * R[1] / R[0]);
  double vm = rux * nx + ruy * ny + ruz * nz;
  double am = sqrt(g * roe_p / roe_rho);
  double rel = ig1 * L[1] + .5 * L[0] * sqL;
  double rer = ig1 * R[1] + .5 * R[0] * sqR;
  double sl, sr;
  hll_speeds(o, vnl, vnr, al, ar, vm, am, sl, sr);
  double iks = 1.0 / (sr - sl);
  double kl = sr * iks, kr = -sl * iks, ku = sl * sr * iks;
  double wl = kl * vnl - ku, wr = kr * vnr + ku;
  F[0] = wl * L[0] + wr * R[0];
  F[1] = wl * rel + wr * rer + (kl * vnl * L[1] + kr * vnr * R[1]);
  double ml = wl * L[0], mr = wr * R[0], pp = kl * L[1] + kr * R[1];
  F[2] = ml * L[2] + mr * R[2] + pp * nx;
  F[3] = ml * L[3] + mr * R[3] + pp * ny;
  F[4] = ml * L[4] + mr * R[4] + pp * nz;
}
// calc_flux_ausmm.f90:62-118: AUSM-M, van Leer's Mach and pressure splittings (no Jacobian)
__device__ void flux_ausmm(double g, const double* L, const double* R, double nx, double ny, double nz, double* F) {
  const double gig1 = g / (g - 1.0);
  const double al = sqrt(g * L[1] / L[0]);
  const double ar = sqrt(g * R[1] / R[0]);
  const double mnl = (L[2] * nx + L[3] * ny + L[4] * nz) / al;
  const double mnr = (R[2] * nx + R[3] * ny + R[4] * nz) / ar;
  double mp, pp, mm, pm;
  if (mnl >= 1.0) { mp = mnl; pp = 1.0; }
  else if (mnl <= -1.0) { mp = 0.0; pp = 0.0; }
  else { mp = .25 * ((mnl + 1.0) * (mnl + 1.0)); pp = mp * (2.0 - mnl); }
  if (mnr <= -1.0) { mm = mnr; pm = 1.0; }
  else if (mnr >= 1.0) { mm = 0.0; pm = 0.0; }
  else { mm = -(.25 * ((mnr - 1.0) * (mnr - 1.0))); pm = -mm * (2.0 + mnr); }
  const double ms = mp + mm;
  const double wl = al * fmax(0.0, ms), wr = ar * fmin(0.0, ms);
  const double rhl = gig1 * L[1] + .5 * L[0] * (L[2] * L[2] + L[3] * L[3] + L[4] * L[4]);
  const double rhr = gig1 * R[1] + .5 * R[0] * (R[2] * R[2] + R[3] * R[3] + R[4] * R[4]);
  F[0] = wl * L[0] + wr * R[0];
  F[1] = wl * rhl + wr * rhr;
  const double ml = wl * L[0], mr = wr * R[0], pf = pp * L[1] + pm * R[1];
  F[2] = ml * L[2] + mr * R[2] + pf * nx;
  F[3] = ml * L[3] + mr * R[3] + pf * ny;
  F[4] = ml * L[4] + mr * R[4] + pf * nz;
}
__device__ void flux_hllc(const SpatOpts& o, const double* L, const double* R, double nx, double ny, double nz,
                          double* F) {
  const double g = o.gamma;
  const double ig1 = 1.0 / (g - 1.0);
  const double gig1 = g / (g - 1.0);
  // calc_roe_states.f90:37-53
  double t1 = sqrt(R[0] / L[0]);
  double roe_rho = L[0] * t1;
  double kl = 1.0 / (1.0 + t1);
  double kr = t1 * kl;
  double rux = kl * L[2] + kr * R[2], ruy = kl * L[3] + kr * R[3], ruz = kl * L[4] + kr * R[4];
  double sqL = L[2] * L[2] + L[3] * L[3] + L[4] * L[4];
  double sqR = R[2] * R[2] + R[3] * R[3] + R[4] * R[4];
  double h1 = gig1 * L[1] / L[0] + 0.5 * sqL;
  double h2 = gig1 * R[1] / R[0] + 0.5 * sqR;
  h1 = kl * h1 + kr * h2;
  double roe_p = (h1 - 0.5 * (rux * rux + ruy * ruy + ruz * ruz)) * roe_rho / gig1;
  // calc_flux_hllc.f90:86-171 (beta = 1)
  double vnl = L[2] * nx + L[3] * ny + L[4] * nz;
  double vnr = R[2] * nx + R[3] * ny + R[4] * nz;
  double al = sqrt(g * L[1] / L[0]);
  double ar = sqrt(g * R[1] / R[0]);
  double vm = rux * nx + ruy * ny + ruz * nz;
  double am = sqrt(g * roe_p / roe_rho);
  double rel = ig1 * L[1] + 0.5 * L[0] * sqL;
  double rer = ig1 * R[1] + 0.5 * R[0] * sqR;
  double sl, sr;
  hll_speeds(o, vnl, vnr, al, ar, vm, am, sl, sr);
  if (sl >= 0.0) {
    F[0] = vnl * L[0];
    F[1] = vnl * (rel + L[1]);
    double m0 = vnl * L[0];
    F[2] = m0 * L[2] + L[1] * nx; F[3] = m0 * L[3] + L[1] * ny; F[4] = m0 * L[4] + L[1] * nz;
  } else if (sr <= 0.0) {
    F[0] = vnr * R[0];
    F[1] = vnr * (rer + R[1]);
    double m0 = vnr * R[0];
    F[2] = m0 * R[2] + R[1] * nx; F[3] = m0 * R[3] + R[1] * ny; F[4] = m0 * R[4] + R[1] * nz;
  } else {
    double rqL = L[0] * (sl - vnl);
    double rqR = R[0] * (sr - vnr);
    double Sst = (rqR * vnr - rqL * vnl - R[1] + L[1]) / (rqR - rqL);
    double iks, rst, pst, rest, rvx, rvy, rvz;
    if (Sst >= 0.0) {
      iks = 1.0 / (sl - Sst);
      rst = rqL * iks;
      pst = L[1] - rqL * (vnl - Sst);
      double dp = pst - L[1];
      rvx = iks * ((rqL * L[2]) + dp * nx); rvy = iks * ((rqL * L[3]) + dp * ny); rvz = iks * ((rqL * L[4]) + dp * nz);
      rest = iks * (rel * (sl - vnl) - L[1] * vnl + pst * Sst);
    } else {
      iks = 1.0 / (sr - Sst);
      rst = rqR * iks;
      pst = R[1] - rqR * (vnr - Sst);
      double dp = pst - R[1];
      rvx = iks * ((rqR * R[2]) + dp * nx); rvy = iks * ((rqR * R[3]) + dp * ny); rvz = iks * ((rqR * R[4]) + dp * nz);
      rest = iks * (rer * (sr - vnr) - R[1] * vnr + pst * Sst);
    }
    F[0] = Sst * rst;
    F[1] = Sst * (rest + pst);
    F[2] = (Sst * rvx) + (pst * nx); F[3] = (Sst * rvy) + (pst * ny); F[4] = (Sst * rvz) + (pst * nz);
  }
}

__device__ void flux_rusanov(double g, const double* L, const double* R, double nx, double ny, double nz, double* F) {
  const double ig1 = 1.0 / (g - 1.0);
  double vnl = L[2] * nx + L[3] * ny + L[4] * nz;
  double vnr = R[2] * nx + R[3] * ny + R[4] * nz;
  double al = sqrt(g * L[1] / L[0]);
  double ar = sqrt(g * R[1] / R[0]);
  double ray = fmax(fabs(vnl) + al, fabs(vnr) + ar);
  double rel = ig1 * L[1] + 0.5 * L[0] * (L[2] * L[2] + L[3] * L[3] + L[4] * L[4]);
  double rer = ig1 * R[1] + 0.5 * R[0] * (R[2] * R[2] + R[3] * R[3] + R[4] * R[4]);
  F[0] = 0.5 * ((vnl + ray) * L[0] + (vnr - ray) * R[0]);
  F[1] = 0.5 * ((vnl + ray) * rel + (vnr - ray) * rer + vnl * L[1] + vnr * R[1]);
  double a = (vnl + ray) * L[0], b = (vnr - ray) * R[0], pp = L[1] + R[1];
  F[2] = 0.5 * ((a * L[2] + b * R[2]) + pp * nx);
  F[3] = 0.5 * ((a * L[3] + b * R[3]) + pp * ny);
  F[4] = 0.5 * ((a * L[4] + b * R[4]) + pp * nz);
}

// Harten's fix of a wave speed below delta: a call, taken by few faces
__device__ __noinline__ double harten(double l, double delta) { return (l * l + delta * delta) / (2.0 * delta); }

// Roe flux-difference splitting with Harten's entropy fix (new: Typhon has no Roe flux).  The oracle's
// operations in its order, as F64; the three divisions by a^2 share its reciprocal, comparisons are of
// bit patterns.  Limited states and flux of 175,760 faces: 111 -> 92 us.
__device__ void flux_roe(const SpatOpts& o, const double* Ls, const double* Rs, double nxs, double nys, double nzs,
                         double* F) {
  F64 L[5], R[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) { L[v] = Ls[v]; R[v] = Rs[v]; }
  const F64 nx = nxs, ny = nys, nz = nzs, half = 0.5;
  const F64 ig1 = o.ig1, gig1 = o.gdg1;
  F64 t1 = sqrt(Rs[0] / Ls[0]);
  F64 rroe = L[0] * t1;
  F64 kl = 1.0 / (F64(1.0) + t1).v, kr = t1 * kl;
  F64 ux = kl * L[2] + kr * R[2], uy = kl * L[3] + kr * R[3], uz = kl * L[4] + kr * R[4];
  F64 sqL = L[2] * L[2] + L[3] * L[3] + L[4] * L[4];
  F64 sqR = R[2] * R[2] + R[3] * R[3] + R[4] * R[4];
  F64 hl = F64((gig1 * L[1]).v / Ls[0]) + half * sqL;
  F64 hr = F64((gig1 * R[1]).v / Rs[0]) + half * sqR;
  F64 hroe = kl * hl + kr * hr;
  F64 q2 = ux * ux + uy * uy + uz * uz, hq2 = half * q2;
  F64 a2 = F64(o.gamma - 1.0) * (hroe - hq2);
  F64 a = sqrt(a2.v);
  F64 vn = ux * nx + uy * ny + uz * nz;
  F64 vnl = L[2] * nx + L[3] * ny + L[4] * nz;
  F64 vnr = R[2] * nx + R[3] * ny + R[4] * nz;
  F64 rel = ig1 * L[1] + half * L[0] * sqL;
  F64 rer = ig1 * R[1] + half * R[0] * sqR;
  F64 drho = R[0] - L[0], dp = R[1] - L[1], dvn = vnr - vnl;
  F64 dux = R[2] - L[2], duy = R[3] - L[3], duz = R[4] - L[4];
  const Divisor d = divisor(a2.v), dd = {a2 + a2, d.y * half, d.ok};
  const F64 rad = rroe * a * dvn;
  F64 al1 = quotient(dp - rad, dd);
  F64 al5 = quotient(dp + rad, dd);
  F64 al2 = drho - quotient(dp, d);
  F64 dutx = dux - dvn * nx, duty = duy - dvn * ny, dutz = duz - dvn * nz;
  F64 l1 = abs_bits((vn - a).v), l5 = abs_bits((vn + a).v), l2 = abs_bits(vn.v);
  F64 delta = F64(o.entropy_fix) * a;
  if (dbits(l1.v) < dbits(delta.v)) l1 = harten(l1.v, delta.v);  // positive doubles order like their bits
  if (dbits(l5.v) < dbits(delta.v)) l5 = harten(l5.v, delta.v);
  F64 w1 = l1 * al1, w2 = l2 * al2, w5 = l5 * al5, ws = l2 * rroe;
  F64 d_mass = w1 + w2 + w5;
  const F64 anx = a * nx, any = a * ny, anz = a * nz, avn = a * vn;
  F64 dmx = w1 * (ux - anx) + w2 * ux + w5 * (ux + anx) + ws * dutx;
  F64 dmy = w1 * (uy - any) + w2 * uy + w5 * (uy + any) + ws * duty;
  F64 dmz = w1 * (uz - anz) + w2 * uz + w5 * (uz + anz) + ws * dutz;
  F64 d_ener = w1 * (hroe - avn) + w2 * hq2 + w5 * (hroe + avn) + ws * ((ux * dux + uy * duy + uz * duz) - vn * dvn);
  F64 ml = vnl * L[0], mr = vnr * R[0];
  F[0] = (half * (ml + mr - d_mass)).v;
  F[1] = (half * (vnl * (rel + L[1]) + vnr * (rer + R[1]) - d_ener)).v;
  F[2] = (half * ((ml * L[2] + L[1] * nx) + (mr * R[2] + R[1] * nx) - dmx)).v;
  F[3] = (half * ((ml * L[3] + L[1] * ny) + (mr * R[3] + R[1] * ny) - dmy)).v;
  F[4] = (half * ((ml * L[4] + L[1] * nz) + (mr * R[4] + R[1] * nz) - dmz)).v;
}

// ===========================================================================
// Fast mode.  Same mathematics, fewer FP64 operations: on GB300 the FP64 pipe (about 2
// DFMA per SM per clock, a division or square root costing about ten) bounds this path,
// so reciprocals, reconstruction weights and geometric factors are precomputed once
// (HBM-resident) and the per-stage work avoids divisions.

#if TY_FAST
// Roe weights and reciprocal densities from one reciprocal square root: with y = 1/sqrt(rho_L
// rho_R), rroe = sqrt(rho_L rho_R) = rho_L rho_R y, kl = rho_L / (rho_L + rroe), kr = rroe /
// (rho_L + rroe), 1/rho_L = y^2 rho_R, 1/rho_R = y^2 rho_L.
struct RoeAvg {
  F64 rroe, kl, kr, TL, TR;  // TL = p_L / rho_L
};
__device__ __forceinline__ RoeAvg roe_avg(const F64* L, const F64* R) {
  RoeAvg r;
  const F64 P = L[0] * R[0], y = rsqrt_nr(P), y2 = y * y;
  r.rroe = P * y;
  const F64 inv = rcp_nr(L[0] + r.rroe);
  r.kl = L[0] * inv;
  r.kr = r.rroe * inv;
  r.TL = L[1] * (y2 * R[0]);
  r.TR = R[1] * (y2 * L[0]);
  return r;
}

// The acoustic waves of the Roe flux with Harten's fix, any regime: sum = w1 + w5 and
// wa = (w5 - w1) a.  A call, taken by supersonic faces and those inside the fix.
__device__ __noinline__ double2 roe_acoustic(double vn, double a, double ra, double dp, double Q, double eps, double ieps) {
  const double h = 0.5 * ra * ra, rad = Q * a;
  const double al1 = (dp - rad) * h, al5 = (dp + rad) * h, delta = eps * a;
  double l1 = fabs(vn - a), l5 = fabs(vn + a);
  const double hd = 0.5 * ra * ieps;  // 1 / (2 delta)
  if (l1 < delta) l1 = (l1 * l1 + delta * delta) * hd;
  if (l5 < delta) l5 = (l5 * l5 + delta * delta) * hd;
  const double w1 = l1 * al1, w5 = l5 * al5;
  return make_double2(w1 + w5, (w5 - w1) * a);
}

// Roe flux times S: no division, one reciprocal and two reciprocal square roots by
// Newton-Raphson steps (fastmath.cuh).  The same flux as flux_roe, regrouped so that the
// central and dissipative parts share their products (u~ = u_L + k_r du, du = u_R - u_L):
//   2 F_mass = M = m_L + m_R - d                       (m = rho u.n, d = w1 + w2 + w5)
//   2 F_mom  = M u_L + (m_R - ws - d k_r) du + c_n n,  c_n = p_L + p_R - (w5 - w1) a + ws du.n
//   2 F_ener = m_L H_L + m_R H_R - d_ener              (rho u.n (rho E + p) = m H)
// Where |u~.n| <= (1 - eps) a (subsonic, outside the entropy fix) the acoustic waves add up to
//   w1 + w5 = dp/a + vn Q/a,  (w5 - w1) a = a Q + vn dp/a,  Q = rroe du.n,
// without their strengths: 105 FP64 operations a face instead of 127, all of them DFMA (F64,
// fastmath.cuh).  The face kernel of TGV 64^3x5 on GB300: 585 -> 507 us regrouped -> 456 us as F64
// (FP64 pipe 96 % busy).
__device__ void flux_roe_fast(const SpatOpts& o, const F64* L, const F64* R, F64 nx, F64 ny, F64 nz,
                              F64 S, F64* F) {
  const F64 gig2 = 2.0 * o.gig1, hg1 = 0.5 * (o.gamma - 1.0);
  const RoeAvg r = roe_avg(L, R);
  const F64 dx = R[2] - L[2], dy = R[3] - L[3], dz = R[4] - L[4];
  const F64 ux = fma(r.kr, dx, L[2]), uy = fma(r.kr, dy, L[3]), uz = fma(r.kr, dz, L[4]);
  // twice the enthalpies, and |u|^2 of the average
  const F64 hl = fma(gig2, r.TL, fma(L[2], L[2], fma(L[3], L[3], L[4] * L[4])));
  const F64 hr = fma(gig2, r.TR, fma(R[2], R[2], fma(R[3], R[3], R[4] * R[4])));
  const F64 h = fma(r.kl, hl, r.kr * hr);
  const F64 q2 = fma(ux, ux, fma(uy, uy, uz * uz));
  const F64 a2 = hg1 * (h - q2);
  const F64 ra = rsqrt_nr(a2), a = a2 * ra;
  const F64 vnl = fma(L[2], nx, fma(L[3], ny, L[4] * nz)), vnr = fma(R[2], nx, fma(R[3], ny, R[4] * nz));
  const F64 dvn = vnr - vnl, vn = fma(r.kr, dvn, vnl), dp = R[1] - L[1], drho = R[0] - L[0];
  const F64 p1 = dp * ra, Q = r.rroe * dvn, l2 = abs_bits(vn.v);
  F64 sum, wa;
  if (__double_as_longlong(l2.v) <= __double_as_longlong((F64(o.roe_sub) * a).v)) {
    sum = fma(vn, Q * ra, p1);
    wa = fma(a, Q, vn * p1);
  } else {
    const double2 w = roe_acoustic(vn.v, a.v, ra.v, dp.v, Q.v, o.entropy_fix, o.inv_entropy_fix);
    sum = w.x;
    wa = w.y;
  }
  const F64 w2 = l2 * fma(-p1, ra, drho), ws = l2 * r.rroe, d = sum + w2;
  const F64 ml = vnl * L[0], mr = vnr * R[0];
  const F64 M = ml + mr - d, hs = F64(0.5) * S;
  const F64 B = hs * fma(-d, r.kr, mr - ws);
  const F64 cn = hs * (fma(ws, dvn, L[1] + R[1]) - wa);
  const F64 F0 = hs * M;
  F[0] = F0;
  F[2] = fma(F0, L[2], fma(B, dx, cn * nx));
  F[3] = fma(F0, L[3], fma(B, dy, cn * ny));
  F[4] = fma(F0, L[4], fma(B, dz, cn * nz));
  const F64 X = fma(-vn, dvn, fma(ux, dx, fma(uy, dy, uz * dz)));
  const F64 Y = fma(wa, vn, ws * X);
  const F64 d2 = fma(sum, h, fma(w2, q2, Y + Y));  // twice d_ener
  F[1] = (F64(0.5) * hs) * (fma(ml, hl, mr * hr) - d2);
}

// mass and energy flux and pressure term of a supersonic face, times S (a call: see product_less)
__device__ __noinline__ double3 hllc_supersonic(double S, double vq, double q0, double re, double p) {
  return make_double3(S * (vq * q0), (S * vq) * (re + p), S * p);
}

// HLLC times S (calc_flux_hllc.f90) without divisions: Roe weights and both 1/rho from one
// reciprocal square root, the average sound speed from
//   a~^2 = g (k_l p_l/rho_l + k_r p_r/rho_r) + (g - 1)/2 k_l k_r |u_R - u_L|^2
// (the kinetic energies of the enthalpies cancel against |u~|^2, which is not formed), only the
// upwind side's energy, comparisons on bit patterns.  The face kernel of 370,440 tetrahedra:
// 208 -> 137 us.
__device__ void flux_hllc_fast(const SpatOpts& o, const F64* L, const F64* R, F64 nx, F64 ny, F64 nz,
                               F64 S, F64* F) {
  const F64 g = o.gamma;
  const RoeAvg r = roe_avg(L, R);
  const F64 dx = R[2] - L[2], dy = R[3] - L[3], dz = R[4] - L[4];
  const F64 dd = fma(dx, dx, fma(dy, dy, dz * dz));
  const F64 vnl = fma(L[2], nx, fma(L[3], ny, L[4] * nz)), vnr = fma(R[2], nx, fma(R[3], ny, R[4] * nz));
  const F64 vm = fma(r.kr, vnr - vnl, vnl);
  const F64 al = sqrt_nr(g * r.TL), ar = sqrt_nr(g * r.TR);
  const F64 am = sqrt_nr(fma(g, fma(r.kl, r.TL, r.kr * r.TR), F64(0.5 * (o.gamma - 1.0)) * (r.kl * r.kr * dd)));
  F64 sl, sr;
  if (o.hll_kin) {
    hll_speeds(o, vnl.v, vnr.v, al.v, ar.v, vm.v, am.v, sl.v, sr.v);
  } else {
    sl = min_bits(fma(F64(-o.hll_beta), al, vnl).v, (vm - am).v);
    sr = max_bits(fma(F64(o.hll_beta), ar, vnr).v, (vm + am).v);
  }
  const F64 dl = sl - vnl, dr = sr - vnr;
  const F64 rql = L[0] * dl, rqr = R[0] * dr;
  const F64 Sst = (fma(rqr, vnr, fma(-rql, vnl, L[1])) - R[1]) * rcp_nr(rqr - rql);
  // the side whose state gives the flux, and its wave speed
  const bool supl = !is_neg(sl.v), supr = !supl && (is_neg(sr.v) || __double2hiint(sr.v) == 0);
  const bool left = supl || (!supr && !is_neg(Sst.v));
  const F64 q0 = left ? L[0] : R[0], p = left ? L[1] : R[1];
  const F64 qx = left ? L[2] : R[2], qy = left ? L[3] : R[3], qz = left ? L[4] : R[4];
  const F64 vq = left ? vnl : vnr, ds = left ? dl : dr, rq = left ? rql : rqr, sq = left ? sl : sr;
  const F64 re = fma(F64(o.ig1), p, (F64(0.5) * q0) * fma(qx, qx, fma(qy, qy, qz * qz)));
  F64 m0, E, c;
  if (supl || supr) {
    const double3 w = hllc_supersonic(S.v, vq.v, q0.v, re.v, p.v);
    m0 = w.x; E = w.y; c = w.z;
  } else {
    const F64 i = rcp_nr(sq - Sst), dp = rq * (Sst - vq), pst = p + dp;
    const F64 w = S * Sst, wi = w * i;
    m0 = wi * rq;
    E = w * fma(i, fma(re, ds, fma(pst, Sst, -p * vq)), pst);
    c = fma(wi, dp, S * pst);
  }
  F[0] = m0;
  F[1] = E;
  F[2] = fma(m0, qx, c * nx);
  F[3] = fma(m0, qy, c * ny);
  F[4] = fma(m0, qz, c * nz);
}

// fmax of numbers that are not negative, on their bit patterns; a NaN of either sign loses
__device__ __forceinline__ double fmax_bits(double a, double b) {
  const long long ka = is_nan(a) ? -1ll : dbits(a), kb = is_nan(b) ? -1ll : dbits(b);
  return ka < kb ? b : a;
}

// Rusanov times S (calc_flux_rusanov.f90:57-83) without divisions.  The root of a negative pressure is
// NaN, and a face of two such states too; beside an ordinary state it has no say (fmax), as in the
// exact mode.
__device__ void flux_rusanov_fast(const SpatOpts& o, const F64* L, const F64* R, F64 nx, F64 ny, F64 nz,
                                  F64 S, F64* F) {
  const F64 TL = L[1] * rcp_nr(L[0]), TR = R[1] * rcp_nr(R[0]);
  const F64 vnl = fma(L[2], nx, fma(L[3], ny, L[4] * nz)), vnr = fma(R[2], nx, fma(R[3], ny, R[4] * nz));
  const F64 cl = F64(abs_bits(vnl.v)) + root_nr(F64(o.gamma) * TL), cr = F64(abs_bits(vnr.v)) + root_nr(F64(o.gamma) * TR);
  const F64 ray = fmax_bits(cl.v, cr.v), hs = F64(0.5) * S;
  const F64 el = fma(F64(o.ig1), TL, F64(0.5) * fma(L[2], L[2], fma(L[3], L[3], L[4] * L[4])));
  const F64 er = fma(F64(o.ig1), TR, F64(0.5) * fma(R[2], R[2], fma(R[3], R[3], R[4] * R[4])));
  const F64 A = hs * ((vnl + ray) * L[0]), B = hs * ((vnr - ray) * R[0]), pp = hs * (L[1] + R[1]);
  F[0] = A + B;
  F[1] = fma(A, el, fma(B, er, hs * fma(vnl, L[1], vnr * R[1])));
  F[2] = fma(A, L[2], fma(B, R[2], pp * nx));
  F[3] = fma(A, L[3], fma(B, R[3], pp * ny));
  F[4] = fma(A, L[4], fma(B, R[4], pp * nz));
}
#endif

// Laminar viscous flux added to F (per unit area), calc_flux_viscous_cell.f90:71-144, on the
// cell states and cell gradients of the face's two cells (integration_ns_ust.f90:139-159).
// Face gradients: CELL-AVERAGE a.grad_R + b.grad_L, or FULL with the compact correction along
// C_L C_R (interpface_gradient_vect.f90:59-81, interpface_gradn_scal.f90:60-90, theta = 1).
// On adiabatic-wall faces the conduction term is added back (ns_bocoflux.f90:60-108).
__device__ void add_viscous(const DevMesh& m, const DevState& s, const SpatOpts& o, int f, double* F) {
  const size_t ld = m.ldc, lf = m.ldf;
  const int icl = m.fc1[f], icr = m.fc2[f];
  const double* __restrict__ q = s.prim;
  const double* __restrict__ gr = s.grad;
  const double r = o.rgas;
  const double cp = o.gamma * r / (o.gamma - 1.0);
  const double dHL = m.vgeo[f], dHR = m.vgeo[lf + f];
  const double wx = m.vgeo[2 * lf + f], wy = m.vgeo[3 * lf + f], wz = m.vgeo[4 * lf + f];
  const double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  const double vL[3] = {q[2 * ld + icl], q[3 * ld + icl], q[4 * ld + icl]};
  const double vR[3] = {q[2 * ld + icr], q[3 * ld + icr], q[4 * ld + icr]};
  double velH[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) velH[i] = dHR * vL[i] + dHL * vR[i];
  const double rL = q[icl], rR = q[icr], pL = q[ld + icl], pR = q[ld + icr];
  const double TL = pL / (rL * r), TR = pR / (rR * r);
  const double TH = dHR * TL + dHL * TR;
  const double rhoH = dHR * rL + dHL * rR;
  const double aL = 1.0 / (rL * r), bL = pL / ((rL * rL) * r);
  const double aR = 1.0 / (rR * r), bR = pR / ((rR * rR) * r);
  double gT[3];  // dHL gradT_R + dHR gradT_L
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double gTL = aL * gr[(3 + k) * ld + icl] - bL * gr[k * ld + icl];
    const double gTR = aR * gr[(3 + k) * ld + icr] - bR * gr[k * ld + icr];
    gT[k] = dHL * gTR + dHR * gTL;
  }
  const double mu = viscosity(o, rhoH, TH);
  double G[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      G[i][j] = dHL * gr[(6 + 3 * i + j) * ld + icr] + dHR * gr[(6 + 3 * i + j) * ld + icl];
  double gTH;
  if (o.viscous == TY_VISC_CELLFULL) {
    const double dLR2 = wx * wx + wy * wy + wz * wz;
    const double it = 1.0 / dLR2;
    const double ex = it * wx, ey = it * wy, ez = it * wz;
    double Fav[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) Fav[i] = vR[i] - vL[i] - (G[i][0] * wx + G[i][1] * wy + G[i][2] * wz);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      G[i][0] = G[i][0] + Fav[i] * ex;
      G[i][1] = G[i][1] + Fav[i] * ey;
      G[i][2] = G[i][2] + Fav[i] * ez;
    }
    const double pscal = (wx * nx + wy * ny + wz * nz) / dLR2;
    const double Fcomp = pscal * (TR - TL);
    const double tp = 1.0 * pscal;
    const double vix = nx - tp * wx, viy = ny - tp * wy, viz = nz - tp * wz;
    gTH = 1.0 * Fcomp + (gT[0] * vix + gT[1] * viy + gT[2] * viz);
  } else {
    gTH = gT[0] * nx + gT[1] * ny + gT[2] * nz;
  }
  double Sg[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Sg[i][j] = G[i][j] + G[j][i];
  const double addvisc = -(2.0 / 3.0) * (G[0][0] + G[1][1] + G[2][2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) Sg[i][i] = Sg[i][i] + addvisc;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Sg[i][j] = mu * Sg[i][j];
  const double snx = Sg[0][0] * nx + Sg[0][1] * ny + Sg[0][2] * nz;
  const double sny = Sg[1][0] * nx + Sg[1][1] * ny + Sg[1][2] * nz;
  const double snz = Sg[2][0] * nx + Sg[2][1] * ny + Sg[2][2] * nz;
  const double svn = snx * velH[0] + sny * velH[1] + snz * velH[2];
  F[2] = F[2] - snx;
  F[3] = F[3] - sny;
  F[4] = F[4] - snz;
  F[1] = F[1] - svn;
  const double conduct = mu * cp / o.prandtl;
  F[1] = F[1] - conduct * gTH;
  if (f >= m.nfi && (m.fbc[f] == TY_BC_WALL || m.fbc[f] == TY_BC_NOSLIP)) F[1] = F[1] + conduct * gTH + 0.0;
}

#if TY_FAST
// add_viscous times S: the same flux with theta = p/rho = r T in place of T (the gas constant
// cancels between the conductivity mu cp / Pr and grad T), the temperature gradient contracted
// with its normal before it is formed, Sutherland's (T/T0)^1.5 as x^2 / sqrt(x), and the
// reciprocals by Newton-Raphson.  550 -> 215 FP64 operations a face with HLLC (plate of 87,500
// cells: the face kernel 175 -> 72 us on GB300).
__device__ void add_viscous_fast(const DevMesh& m, const DevState& s, const SpatOpts& o, int f, F64 S, F64* F) {
  const size_t ld = m.ldc, lf = m.ldf;
  const int icl = m.fc1[f], icr = m.fc2[f];
  const double* __restrict__ q = s.prim;
  const double* __restrict__ gl = s.grad + icl;
  const double* __restrict__ gr = s.grad + icr;
  const F64 hl = m.vgeo[f], hr = m.vgeo[lf + f];
  const F64 nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  const F64 rL = q[icl], rR = q[icr], pL = q[ld + icl], pR = q[ld + icr];
  const F64 iL = rcp_nr(rL), iR = rcp_nr(rR), tL = pL * iL, tR = pR * iR;
  const F64 tH = fma(hr, tL, hl * tR);
  F64 mu;
  if (o.visc_law == TY_VISC_KINEMATIC) {
    mu = F64(o.visc_kin) * fma(hr, rL, hl * rR);
  } else {  // mu0 (T/T0)^1.5 (T0 + S) / (T + S), T = tH / r
    const double T0 = 273.00, S0 = 110.50;
    const F64 T = tH * F64(o.irgas), x = T * F64(1.0 / T0);
    mu = F64(0.0000168 * (T0 + S0)) * pow15_nr(x) * rcp_nr(T + F64(S0));
  }
  // velocity gradient at the face (CELL-AVERAGE), G n and G^T n and the divergence
  F64 vL[3], vR[3], G[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    vL[i] = q[(2 + i) * ld + icl];
    vR[i] = q[(2 + i) * ld + icr];
#pragma unroll
    for (int j = 0; j < 3; ++j) G[i][j] = fma(hl, F64(gr[(6 + 3 * i + j) * ld]), hr * F64(gl[(6 + 3 * i + j) * ld]));
  }
  F64 mx = nx, my = ny, mz = nz, comp = 0.0;  // direction of grad theta, and the compact part
  if (o.viscous == TY_VISC_CELLFULL) {           // compact correction along C_L C_R
    const F64 wx = m.vgeo[2 * lf + f], wy = m.vgeo[3 * lf + f], wz = m.vgeo[4 * lf + f];
    const F64 it = rcp_nr(fma(wx, wx, fma(wy, wy, wz * wz)));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const F64 c = it * (vR[i] - vL[i] - fma(G[i][0], wx, fma(G[i][1], wy, G[i][2] * wz)));
      G[i][0] = fma(c, wx, G[i][0]);
      G[i][1] = fma(c, wy, G[i][1]);
      G[i][2] = fma(c, wz, G[i][2]);
    }
    const F64 ps = it * fma(wx, nx, fma(wy, ny, wz * nz));
    comp = ps * (tR - tL);
    mx = fma(-ps, wx, nx); my = fma(-ps, wy, ny); mz = fma(-ps, wz, nz);
  }
  const F64 mS = S * mu, div = F64(2.0 / 3.0) * (G[0][0] + G[1][1] + G[2][2]);
  const F64 n[3] = {nx, ny, nz};
  F64 work = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // (G + G^T) n - 2/3 div n
    F64 t = fma(G[i][0], nx, fma(G[i][1], ny, G[i][2] * nz));
    t = fma(G[0][i], nx, fma(G[1][i], ny, fma(G[2][i], nz, fma(-div, n[i], t))));
    t = t * mS;
    F[2 + i] = F[2 + i] - t;
    work = fma(t, fma(hr, vL[i], hl * vR[i]), work);
  }
  F[1] = F[1] - work;
  if (f >= m.nfi && (m.fbc[f] == TY_BC_WALL || m.fbc[f] == TY_BC_NOSLIP)) return;  // adiabatic
  // grad theta . m of each side: (grad p - theta grad rho) . m / rho
  const F64 gpl = fma(F64(gl[3 * ld]), mx, fma(F64(gl[4 * ld]), my, F64(gl[5 * ld]) * mz));
  const F64 grl = fma(F64(gl[0]), mx, fma(F64(gl[ld]), my, F64(gl[2 * ld]) * mz));
  const F64 gpr = fma(F64(gr[3 * ld]), mx, fma(F64(gr[4 * ld]), my, F64(gr[5 * ld]) * mz));
  const F64 grr = fma(F64(gr[0]), mx, fma(F64(gr[ld]), my, F64(gr[2 * ld]) * mz));
  const F64 tl = iL * fma(-tL, grl, gpl), tr = iR * fma(-tR, grr, gpr);
  F[1] = fma(-(mS * F64(o.gig1 * o.iprandtl)), fma(hl, tr, fma(hr, tl, comp)), F[1]);
}
#endif

#if TY_FAST
__device__ __forceinline__ void face_flux(const DevMesh& m, const DevState& s, const SpatOpts& o, int f,
                                          const double* QL, const double* QR, double* __restrict__ flux) {
  const double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  const double S = m.fs[f];
  F64 L[5], R[5], Fx[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) { L[v] = QL[v]; R[v] = QR[v]; }
  if (o.scheme == TY_SCH_ROE) {
    flux_roe_fast(o, L, R, nx, ny, nz, S, Fx);
  } else if (o.hll_family == 1) {
    flux_hllc_fast(o, L, R, nx, ny, nz, S, Fx);
  } else if (o.scheme == TY_SCH_RUSANOV) {
    flux_rusanov_fast(o, L, R, nx, ny, nz, S, Fx);
  } else {
    double F[5];
    if (o.hll_family == 2) flux_hlle(o, QL, QR, nx, ny, nz, F);
    else flux_ausmm(o.gamma, QL, QR, nx, ny, nz, F);
#pragma unroll
    for (int v = 0; v < 5; ++v) Fx[v] = S * F[v];
  }
  if (o.viscous != TY_VISC_NONE) add_viscous_fast(m, s, o, f, S, Fx);
#pragma unroll
  for (int v = 0; v < 5; ++v) flux[v * (size_t)m.ldf + f] = Fx[v].v;
}
#else
__device__ __forceinline__ void face_flux(const DevMesh& m, const DevState& s, const SpatOpts& o, int f,
                                          const double* QL, const double* QR, double* __restrict__ flux) {
  const double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  double F[5];
  if (o.hll_family == 1) flux_hllc(o, QL, QR, nx, ny, nz, F);
  else if (o.scheme == TY_SCH_RUSANOV) flux_rusanov(o.gamma, QL, QR, nx, ny, nz, F);
  else if (o.hll_family == 2) flux_hlle(o, QL, QR, nx, ny, nz, F);
  else if (o.scheme == TY_SCH_AUSMM) flux_ausmm(o.gamma, QL, QR, nx, ny, nz, F);
  else flux_roe(o, QL, QR, nx, ny, nz, F);
  if (o.viscous != TY_VISC_NONE) add_viscous(m, s, o, f, F);
  const double S = m.fs[f];
#pragma unroll
  for (int v = 0; v < 5; ++v) flux[v * (size_t)m.ldf + f] = S * F[v];
}
#endif

// fused face states + flux (no post-limiter)
__global__ void __launch_bounds__(kBlock) k_face_flux(DevMesh m, DevState s, SpatOpts o) {
  pdl_wait();
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  double QL[5], QR[5];
  X64 LR[5];
  if (o.highres != TY_HRES_NONE) slopes_lr(m, s, f, LR);
  recon(m, s, o, f, 0, LR, QL);
  const int kind = f < m.nfi ? TY_BC_INTERIOR : m.fbc[f];
  if (kind == TY_BC_PERIODIC) {
    recon(m, s, o, m.part[f], 0, QR);  // cell_r(face) = cell_l(partner face)
    rot_to_face(m, f, QR);
  } else if (kind == TY_BC_WALL || kind == TY_BC_NOSLIP) {
    wall_state(m, f, QL, QR);
  } else if (kind == TY_BC_FARFIELD) {
    farfield_state(o, d3(m.fn, m.ldf, f, 0), d3(m.fn, m.ldf, f, 1), d3(m.fn, m.ldf, f, 2), QL, QR);
  } else if (kind >= TY_BC_INLET_SUB) {
    inout_state(m, o, f, kind, QL, QR);
  } else if (kind == TY_BC_SYMMETRY) {
#pragma unroll
    for (int v = 0; v < 5; ++v) QR[v] = QL[v];
    mirror(m, f, QR);
  } else {
    recon(m, s, o, f, 1, LR, QR);
  }
  face_flux(m, s, o, f, QL, QR, s.flux);
}

// post-limiter path, 1: unlimited face states.  Both sides share the slopes (q(fc2) - q(fc1)) / |C_L C_R|,
// five quotients by one divisor where each side divided for itself: 175,760 faces 102 -> 70 us.
__global__ void __launch_bounds__(kBlock) k_face_states(DevMesh m, DevState s, SpatOpts o) {
  pdl_wait();
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  double Q[5];
  X64 LR[5];
  if (o.highres != TY_HRES_NONE) slopes_lr(m, s, f, LR);
  recon(m, s, o, f, 0, LR, Q);
#pragma unroll
  for (int v = 0; v < 5; ++v) s.cl[v * (size_t)m.ldf + f] = Q[v];
  recon(m, s, o, f, 1, LR, Q);
#pragma unroll
  for (int v = 0; v < 5; ++v) s.cr[v * (size_t)m.ldf + f] = Q[v];
}

// klim n/d < klim bn/bd as the limiter computes them (a NaN counts as 0): the call taken where the
// FP32 comparison of k_barth does not decide
__device__ __noinline__ bool ratio_less(double klim, double n, double d, double bn, double bd) {
  return fmax(klim * (n / d), 0.0) < fmax(klim * (bn / bd), 0.0);
}

// post-limiter path, 2: Barth-type ratio of each interior cell (postlimit_barth.f90:60-80,
// 140-170): min(1, max(klim LR/den, 0)) over faces and variables of a group.  A face whose
// increment is exactly zero imposes no constraint.  Division and product round monotonically, so
// the fraction that is smallest gives the minimum: fractions are compared in FP32, truncated and
// cross-multiplied (exactly, ratio_less, where they are within 1e-6 or out of FP32's range), and one
// division per group is left of one per face and variable.  87,880 tetrahedra: 62 -> 19 us.
__global__ void __launch_bounds__(kBlock) k_barth(DevMesh m, DevState s, double klim) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  int es[kMaxSlot];
  face_list(m, c, es);
  pdl_wait();
  const size_t ld = m.ldc, lf = m.ldf;
  X64 qc[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) qc[v] = s.prim[v * ld + c];
  // smallest fraction so far, 1 / klim at first (klim is 1 or 1/2)
  double bn[3] = {1.0, 1.0, 1.0}, bd[3] = {klim, klim, klim};
  float fn[3] = {1.0f, 1.0f, 1.0f}, fd[3] = {(float)klim, (float)klim, (float)klim};
  bool zero[3] = {false, false, false}, far[3] = {false, false, false};
#pragma unroll
  for (int sl = 0; sl < kMaxSlot; ++sl) {
    const int e = es[sl];
    if (e < 0) break;
    const int f = e >> 1, side = e & 1;
    const int nb = side ? m.fc1[f] : m.fc2[f];
    const double* qf = side ? s.cr : s.cl;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const int k = v < 2 ? v : 2;
      const double n = value(X64(s.prim[v * ld + nb]) - qc[v]);  // = +-(q(fc2) - q(fc1)) seen from c
      const double d = value(X64(qf[v * lf + f]) - qc[v]);
      if (is_zero(d)) continue;
      if (is_zero(n) || (__double2hiint(n) ^ __double2hiint(d)) < 0) {  // n/d <= 0
        zero[k] = true;
        continue;
      }
      bool ok = !far[k];
      const float gn = trunc32(n, ok), gd = trunc32(d, ok);
      const float x = gn * fd[k], y = fn[k] * gd;
      bool less = x < y;
      if (!ok || fabsf(x - y) <= 9.6e-7f * y) less = ratio_less(klim, n, d, bn[k], bd[k]);
      if (less) {
        bn[k] = abs_bits(n);
        bd[k] = abs_bits(d);
        bool in = true;
        fn[k] = trunc32(n, in); fd[k] = trunc32(d, in);
        far[k] = !in;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) s.ratio[k * ld + c] = zero[k] ? 0.0 : fmin(1.0, fmax(klim * (bn[k] / bd[k]), 0.0));
}

// post-limiter path, 3: limited states + flux
__global__ void __launch_bounds__(kBlock) k_face_flux_lim(DevMesh m, DevState s, SpatOpts o) {
  pdl_wait();
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const size_t ld = m.ldc, lf = m.ldf;
  double QL[5], QR[5];
  auto limited = [&](int face, int side, double* Q) {
    int c = side ? m.fc2[face] : m.fc1[face];
    const double* qf = side ? s.cr : s.cl;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const X64 qc = s.prim[v * ld + c], rr = s.ratio[(v < 2 ? v : 2) * ld + c];
      Q[v] = value(qc + rr * (X64(qf[v * lf + face]) - qc));
    }
  };
  limited(f, 0, QL);
  const int kind = f < m.nfi ? TY_BC_INTERIOR : m.fbc[f];
  if (kind == TY_BC_PERIODIC) {
    limited(m.part[f], 0, QR);
    rot_to_face(m, f, QR);
  } else if (kind == TY_BC_WALL || kind == TY_BC_NOSLIP) {
    wall_state(m, f, QL, QR);
  } else if (kind == TY_BC_FARFIELD) {
    farfield_state(o, d3(m.fn, m.ldf, f, 0), d3(m.fn, m.ldf, f, 1), d3(m.fn, m.ldf, f, 2), QL, QR);
  } else if (kind >= TY_BC_INLET_SUB) {
    inout_state(m, o, f, kind, QL, QR);
  } else if (kind == TY_BC_SYMMETRY) {
#pragma unroll
    for (int v = 0; v < 5; ++v) QR[v] = QL[v];
    mirror(m, f, QR);
  } else {
    limited(f, 1, QR);
  }
  face_flux(m, s, o, f, QL, QR, s.flux);
}


#if TY_FAST
// |a| b < |c| d of positive products, as bit patterns.  A call, so that the multiplications are not
// if-converted into the callers (a predicated-off FP64 instruction occupies the pipe as well), and a
// short one: the registers of a division, with its own call, are the callers' too (FORM 0 of the
// kernel below: 51 -> 69, its launch 10 % slower).
__device__ __noinline__ bool product_less(double a, double b, double c, double d) {
  return dbits(fabs(a) * b) < dbits(d * fabs(c));
}

// The same where a, b, c or d is out of the FP32 comparison's range: scaled where c or b is so small that
// a product could be subnormal.
constexpr int kTiny = (1023 - 400) << 20;  // upper word of 2^-400
__device__ __noinline__ bool product_less_far(double a, double b, double c, double d) {
  a = fabs(a);
  c = fabs(c);
  if (__double2hiint(c) < kTiny || __double2hiint(b) < kTiny) {
    a *= 0x1p600;
    b *= 0x1p600;
    c *= 0x1p600;
    d *= 0x1p600;
  }
  return dbits(a * b) < dbits(d * c);
}

// klim n / d where d is below 2^-400 and may have no normal reciprocal (a call for the same reasons)
__device__ __noinline__ double barth_ratio(double klim, double n, double d) {
  return klim * (n * 0x1p600) * rcp_nr(d * 0x1p600);
}

// van Albada's phi(a, b) = a b (a + b) / (a^2 + b^2) where a b > 0, else 0, sum = a + b given.
// Products below 2^-1000 count as 0 (the reciprocal's seed flushes subnormal numbers).
__device__ __forceinline__ double albada_fast(double a, double b, double sum) {
  const double ab = a * b;
  if (__double2hiint(ab) < (23 << 20)) return 0.0;
  return ab * sum * rcp_nr(fma(a, a, b * b));
}

// Fused cell kernel: neighbour differences, face increments, Barth-type ratio and the limited
// face states, written once per face side (cl for the fc1 side, cr for the fc2 side).
//
// One thread per cell and variable: a warp holds 32 cells of one variable, a block the five
// variables of its cells.  GB300 issues one FP64 warp instruction per 64 clocks and SM quarter
// and everything here but the velocities' common ratio is per variable, so five short chains
// replace one long one: small meshes occupy five times as many SM quarters, and the differences
// and increments of the (at most NS) faces fit in registers at full occupancy.  The lists and
// tables are read by five warps of one block, from L1 after the first.
//
// FORM 0 (MUSCL / MUSCL-UNS without limiter): D_i = sum_j M_ij dq_j from the cell's matrix
//   (DevMesh::mtab).
// FORM 1 (van Albada) and FORM 2 (the other limiters, none included): the least-squares
//   gradient G, then per face, with the slot table of DevMesh::stab (outward vectors),
//     D = G . w + phi(a, dq) k,  a = 2 G . d - dq (MUSCL, MUSCL-FAST) or G . d (MUSCL-UNS),
//   the slopes scaled by the distance |d| (the limiters are homogeneous of degree one; LIM03,
//   which is not, gets them unscaled, and its table has k for them: a division by 1/|d| here took
//   two steps on 729,000 hexahedra from 24.7 to 27.0 ms).
//
// The ratio min_f max(klim dq/D, 0) is kept as a fraction n/d.  A candidate is compared with it
// in FP32 on truncated operands, which decides all but comparisons closer than 2^-20, and those
// are redone with the FP64 products: the same winner as an FP64 comparison without its two
// multiplications per face.  An increment of exactly zero imposes no constraint.
//
// copy_ghosts: every boundary face is a translational periodic one; the ghosts' states are
// copies of their source cells', written here by the one cell that reads them, and
// k_ghost_prim is not launched.
//
// Bound by the FP64 pipe (82 % busy at 30 operations per thread in FORM 0 with the ratio).
// Comparisons of doubles, |x| and predicated-off arithmetic run on that pipe too, so tests are
// made on bit patterns and rare FP64 work sits behind a call.  Microseconds per launch on GB300,
// one thread per cell (differences staged in shared memory) -> one thread per cell and variable:
// 1,310,720 tetrahedra FORM 0 + ratio 628 -> 350; 370,440 tetrahedra FORM 1 460 -> 283; 87,500
// prisms and tetrahedra FORM 1 133 -> 78; 163,840 tetrahedra FORM 1 213 -> 127.
constexpr int kCellVars = 5;

template <int NS, int FORM>
__global__ void __launch_bounds__(32 * kCellVars) k_cell_fast(DevMesh m, DevState s, SpatOpts o, double klim,
                                                              bool copy_ghosts) {
  __shared__ double sr[3][32];
  const int c0 = blockIdx.x * 32 + threadIdx.x, v = threadIdx.y;
  const bool on = c0 < m.nci;
  const int c = on ? c0 : m.nci - 1;
  const size_t ld = m.ldc, lf = m.ldf, n = m.nci;
  int es[NS], nbs[NS];
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) es[sl] = sl < m.nslot ? m.cf[sl * n + c] : -1;
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) nbs[sl] = es[sl] >= 0 ? m.cfn[sl * n + c] : c;
  // the slot tables may be one launch old: their loads must not move above the wait
  const double *mtab = m.mtab, *stab = m.stab;
  pdl_wait();
  asm volatile("" : "+l"(mtab), "+l"(stab));
  double* __restrict__ prim = s.prim + v * ld;
  const double qc = prim[c];
  double dq[NS];
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) {
    const bool ghost = copy_ghosts && nbs[sl] >= m.nci;
    const double q = prim[ghost ? m.gsrc[nbs[sl] - m.nci] : nbs[sl]];
    if (ghost && on) prim[nbs[sl]] = q;
    dq[sl] = q - qc;  // 0 on an unused slot
  }
  double D[NS];
  if constexpr (FORM == 0) {
    const double* M = mtab + c;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      double d = 0.0;
      if (es[i] >= 0) {
#pragma unroll
        for (int j = 0; j < NS; ++j)
          if (j < m.nslot) d = fma(__ldg(M + ((size_t)i * m.nslot + j) * n), dq[j], d);
      }
      D[i] = d;
    }
  } else {
    const double* T = stab + c;
    const bool uns = o.highres == TY_HRES_MUSCLUNS, fst = o.highres == TY_HRES_MUSCLFAST;
    double gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      if (es[i] < 0) continue;
      const double* t = T + (size_t)(kSlotTab * i) * n;
      gx = fma(dq[i], __ldg(t), gx);
      gy = fma(dq[i], __ldg(t + n), gy);
      gz = fma(dq[i], __ldg(t + 2 * n), gz);
    }
    if (on) {
      double* g = s.grad + 3 * v * ld + c;
      g[0] = gx; g[ld] = gy; g[2 * ld] = gz;
    }
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      D[i] = 0.0;
      if (es[i] < 0) continue;
      const double* t = T + (size_t)(kSlotTab * i + 3) * n;
      const double k = __ldg(t + 6 * n), b = dq[i];
      double phi = b;
      if (FORM == 1 || o.limiter != TY_LIM_NONE) {
        const double g = fma(gx, __ldg(t), fma(gy, __ldg(t + n), gz * __ldg(t + 2 * n)));  // G . d, twice it unless UNS
        if constexpr (FORM == 1) {
          phi = uns ? albada_fast(g, b, g + b) : albada_fast(g - b, b, g);
        } else if (o.limiter == TY_LIM_LIM03) {
          const double id = __ldg(t + 7 * n);
          phi = apply_lim(o.limiter, uns, v < 2, (uns ? g : 0.5 * g) * id, b * id);
          D[i] = fst ? 0.0 : fma(gx, __ldg(t + 3 * n), fma(gy, __ldg(t + 4 * n), gz * __ldg(t + 5 * n)));
          D[i] = fma(phi, k, D[i]);
          continue;
        } else {
          phi = apply_lim(o.limiter, uns, v < 2, uns ? g : 0.5 * g, b);
        }
      }
      D[i] = fst ? phi * k : fma(gx, __ldg(t + 3 * n), fma(gy, __ldg(t + 4 * n), fma(gz, __ldg(t + 5 * n), phi * k)));
    }
  }
  double r = 1.0;
  if (o.postlim != TY_POSTLIM_NONE) {
    double bn = 1.0, bd = klim;
    float fn = 1.0f, fd = o.postlim == TY_POSTLIM_SUPERBARTH ? 1.0f : 0.5f;
    bool zero = false, far = false;  // far: the fraction is outside the FP32 comparison's range
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      if (es[i] < 0 || is_zero(D[i])) continue;
      if (is_zero(dq[i]) || (__double2hiint(dq[i]) ^ __double2hiint(D[i])) < 0) {  // dq/D <= 0
        zero = true;
        continue;
      }
      bool ok = !far;
      const float fq = trunc32(dq[i], ok), fD = trunc32(D[i], ok);
      const float x = fq * fd, y = fn * fD;
      bool less = x < y;
      if (!ok) less = product_less_far(dq[i], bd, D[i], bn);
      else if (fabsf(x - y) <= 9.6e-7f * y) less = product_less(dq[i], bd, D[i], bn);
      if (less) {
        bn = abs_bits(dq[i]);
        bd = abs_bits(D[i]);
        bool in = true;
        fn = trunc32(dq[i], in); fd = trunc32(D[i], in);
        far = !in;
      }
    }
    // the fraction starts at 1: min(1, klim n/d), as bit patterns (positive doubles order alike; a NaN
    // of either sign orders above 1 when unsigned).  The reciprocal's seed flushes subnormal numbers.
    r = klim * bn * rcp_nr(bd);
    if (__double2hiint(bd) < kTiny) r = barth_ratio(klim, bn, bd);
    if ((unsigned long long)dbits(r) > (unsigned long long)dbits(1.0)) r = 1.0;
    if (zero) r = 0.0;
    if (v >= 2) sr[v - 2][threadIdx.x] = r;
    __syncthreads();
    if (v >= 2) {  // the three velocity components share the smallest ratio (compared as bit patterns)
      const double a = sr[0][threadIdx.x], b = sr[1][threadIdx.x], d = sr[2][threadIdx.x];
      r = dbits(a) < dbits(b) ? a : b;
      r = dbits(d) < dbits(r) ? d : r;
    }
    if (on && v < 3) s.ratio[v * ld + c] = r;
  }
  if (!on) return;
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) {
    if (es[sl] < 0) continue;
    double* out = (es[sl] & 1) ? s.cr : s.cl;
    out[v * lf + (es[sl] >> 1)] = fma(r, D[sl], qc);
  }
}

template <int NS>
void cell_fast_ns(const DevMesh& m, const DevState& s, const SpatOpts& o, double klim, bool copy_ghosts, bool matrix,
                  cudaStream_t st) {
  const dim3 b(32, kCellVars);
  const unsigned g = (unsigned)((m.nci + 31) / 32);
  if (matrix) launch_pdl(k_cell_fast<NS, 0>, g, b, st, m, s, o, klim, copy_ghosts);
  else if (o.limiter == TY_LIM_ALBADA) launch_pdl(k_cell_fast<NS, 1>, g, b, st, m, s, o, klim, copy_ghosts);
  else launch_pdl(k_cell_fast<NS, 2>, g, b, st, m, s, o, klim, copy_ghosts);
}

// want_grad: the caller reads s.grad (a viscous flux, the adjoint); the matrix form has none.
// NS is the mesh's largest number of faces per cell (3 triangles, 4 quadrangles and tetrahedra,
// 5 pyramids and prisms, 6 hexahedra), so that no unrolled slot is idle on a uniform mesh.
void cell_fast(const DevMesh& m, const DevState& s, const SpatOpts& o, bool want_grad, bool copy_ghosts,
               cudaStream_t st) {
  const double klim = o.postlim == TY_POSTLIM_SUPERBARTH ? 1.0 : 0.5;
  const bool matrix = m.mtab && !want_grad;
  if (m.nslot <= 3) cell_fast_ns<3>(m, s, o, klim, copy_ghosts, matrix, st);
  else if (m.nslot == 4) cell_fast_ns<4>(m, s, o, klim, copy_ghosts, matrix, st);
  else if (m.nslot == 5) cell_fast_ns<5>(m, s, o, klim, copy_ghosts, matrix, st);
  else if (m.nslot == 6) cell_fast_ns<6>(m, s, o, klim, copy_ghosts, matrix, st);
  else cell_fast_ns<kMaxSlot>(m, s, o, klim, copy_ghosts, matrix, st);
}
#endif

#if TY_FAST
// DevMesh::mtab of every interior cell: M_ij = (+-A^-1 d_j) . w_i + k_i [i == j] over the
// cell's gather-list faces i, j (w, k: the reconstruction weights recw of face i on the cell's
// side; the least-squares weight's sign flipped for the fc2 side, as k_cell_fast does);
// zero outside the cell's faces
__global__ void k_build_mtab(DevMesh m, double* __restrict__ mt) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  const size_t n = m.nci, lf = m.ldf;
  const int ns = m.nslot;
  for (int i = 0; i < ns; ++i) {
    const int ei = m.cf[i * n + c];
    for (int j = 0; j < ns; ++j) {
      const int ej = m.cf[j * n + c];
      double v = 0.0;
      if (ei >= 0 && ej >= 0) {
        const int fi = ei >> 1, si = ei & 1, fj = ej >> 1, sj = ej & 1;
        const double sg = sj ? -1.0 : 1.0;
        for (int k = 0; k < 3; ++k) v += sg * m.lsqw[(3 * sj + k) * lf + fj] * m.recw[(4 * si + k) * lf + fi];
        if (i == j) v += m.recw[(4 * si + 3) * lf + fi];
      }
      mt[((size_t)i * ns + j) * n + c] = v;
    }
  }
}

// DevMesh::stab of every interior cell and slot: the least-squares weight +-A^-1 d (3), the
// vector to the neighbour (3; doubled unless MUSCL-UNS, whose limiter takes G . d itself), the
// reconstruction weight CF - (u . CF) u (3; 0 for MUSCL-FAST), the slope's factor (u . CF)/|d|
// or, MUSCL-FAST, |F - C|/dLR (lim03: without the divisor), and 1/dLR, all seen from the cell outwards
__global__ void k_build_stab(DevMesh m, int highres, bool lim03, double* __restrict__ T) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  const size_t n = m.nci, lf = m.ldf;
  for (int i = 0; i < m.nslot; ++i) {
    double* t = T + (size_t)(kSlotTab * i) * n + c;
    const int e = m.cf[i * n + c];
    if (e < 0) {
      for (int k = 0; k < kSlotTab; ++k) t[k * n] = 0.0;
      continue;
    }
    const int f = e >> 1, side = e & 1;
    const double sg = side ? -1.0 : 1.0, two = highres == TY_HRES_MUSCLUNS ? 1.0 : 2.0;
    for (int k = 0; k < 3; ++k) {
      t[k * n] = sg * m.lsqw[(3 * side + k) * lf + f];
      t[(3 + k) * n] = two * sg * (m.uLR[k * lf + f] * m.dLR[f]);
      t[(6 + k) * n] = m.recw[(4 * side + k) * lf + f];
    }
    if (highres == TY_HRES_MUSCLFAST) t[9 * n] = (side ? -m.kRF[f] : m.kLF[f]) * (lim03 ? 1.0 : m.invdLR[f]);
    else t[9 * n] = m.recw[(4 * side + 3) * lf + f] * (lim03 ? m.dLR[f] : 1.0);
    t[10 * n] = m.invdLR[f];
  }
}

cudaError_t build_stab(const DevMesh& m, int highres, bool lim03, double* stab, cudaStream_t st) {
  k_build_stab<<<(unsigned)((m.nci + kBlock - 1) / kBlock), kBlock, 0, st>>>(m, highres, lim03, stab);
  return cudaGetLastError();
}

cudaError_t build_mtab(const DevMesh& m, double* mtab, cudaStream_t st) {
  k_build_mtab<<<(unsigned)((m.nci + kBlock - 1) / kBlock), kBlock, 0, st>>>(m, mtab);
  return cudaGetLastError();
}
#endif

// face fluxes from the limited states of k_cell_fast
// PDL: launched by launch_pdl.  The wait costs the kernel 3 to 8 % wherever it stands (Roe at 2.6M
// faces 456 -> 495 us, HLLC at 0.74M 134 -> 144, 12,416 faces 5.9 -> 6.2) and saves the 2.5 us gap.
// So does reading the boundary kind ahead of the state: the order of these loads stays as it is.
template <bool PDL>
__global__ void __launch_bounds__(kBlock) k_face_flux_fast(DevMesh m, DevState s, SpatOpts o) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const size_t lf = m.ldf;
  if constexpr (PDL) pdl_wait();
  double QL[5], QR[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) QL[v] = s.cl[v * lf + f];
  const int kind = f < m.nfi ? TY_BC_INTERIOR : m.fbc[f];
  if (kind == TY_BC_PERIODIC) {
    const int p = m.part[f];
#pragma unroll
    for (int v = 0; v < 5; ++v) QR[v] = s.cl[v * lf + p];
    rot_to_face(m, f, QR);
  } else if (kind == TY_BC_WALL || kind == TY_BC_NOSLIP) {
    wall_state(m, f, QL, QR);
  } else if (kind == TY_BC_FARFIELD) {
    farfield_state(o, d3(m.fn, m.ldf, f, 0), d3(m.fn, m.ldf, f, 1), d3(m.fn, m.ldf, f, 2), QL, QR);
  } else if (kind >= TY_BC_INLET_SUB) {
    inout_state(m, o, f, kind, QL, QR);
  } else if (kind == TY_BC_SYMMETRY) {
#pragma unroll
    for (int v = 0; v < 5; ++v) QR[v] = QL[v];
    mirror(m, f, QR);
  } else {
#pragma unroll
    for (int v = 0; v < 5; ++v) QR[v] = s.cr[v * lf + f];
  }
  face_flux(m, s, o, f, QL, QR, s.flux);
}

// ---------------------------------------------------------------------------
// residual R_c = dt/V_c * sum(+-F S), in the colour order of flux_to_res.  The sign is put on the
// flux's bits (R - F is R + (-F), bit for bit), so that one sum per flux is issued: a branch on
// the side issued both, one of them predicated off.
template <class T>
__device__ __forceinline__ void gather_residual(const DevMesh& m, const DevState& s, const int es[kMaxSlot], T R[5]) {
#pragma unroll
  for (int v = 0; v < 5; ++v) R[v] = 0.0;
  const double* __restrict__ F = s.flux;
  const size_t lf = m.ldf;
#pragma unroll
  for (int sl = 0; sl < kMaxSlot; ++sl) {
    const int e = es[sl];
    if (e < 0) break;
    const double* f = F + (e >> 1);
    const int sign = (~e & 1) << 31;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double x = f[v * lf];
      R[v] = R[v] + T(__hiloint2double(__double2hiint(x) ^ sign, __double2loint(x)));
    }
  }
}

__device__ __forceinline__ double load_dt(double dt, const unsigned long long* dtbits) {
  return dtbits ? __longlong_as_double((long long)*dtbits) : dt;
}

__global__ void __launch_bounds__(kBlock) k_gather(DevMesh m, DevState s, double dt, const unsigned long long* dtbits,
                                                   double* out, int ld) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  using T = typename std::conditional<kFast, F64, double>::type;
  T R[5];
  int es[kMaxSlot];
  face_list(m, c, es);
  pdl_wait();
  gather_residual(m, s, es, R);
  const double coef = kFast ? load_dt(dt, dtbits) * m.invV[c] : load_dt(dt, dtbits) / m.cvol[c];
#pragma unroll
  for (int v = 0; v < 5; ++v) out[v * (size_t)ld + c] = value(T(coef) * R[v]);
}

// per-cell stability time step; returns false for negative or NaN internal energy
__device__ __forceinline__ bool cell_dt(const DevMesh& m, double gamma, double cfl, int c, const double u[5], double& dt) {
  const double gg1 = gamma * (gamma - 1.0);
  double d;
  if constexpr (kFast) d = cfl * m.geo2[c];
  else d = cfl * 2.0 * m.cvol[c] / m.sumS[c];
  if constexpr (kFast) {
    const double irho = rcp_nr(u[0]);
    const double rv2 = u[2] * u[2] + u[3] * u[3] + u[4] * u[4];
    const double a2 = (u[1] - 0.5 * rv2 * irho) * gg1 * irho;
    if (!(a2 > 0.0)) return false;
    dt = d * rcp_nr(sqrt_nr(rv2) * irho + sqrt_nr(a2));
    return true;
  }
  double irho = 1.0 / u[0];
  double rv2 = u[2] * u[2] + u[3] * u[3] + u[4] * u[4];
  double a2 = (u[1] - 0.5 * rv2 * irho) * gg1 * irho;
  if (!(a2 > 0.0)) return false;
  dt = d / (sqrt(rv2) * irho + sqrt(a2));
  return true;
}

constexpr unsigned long long kMaxDtBits = 0x7fefffffffffffffull;  // largest finite double

// block minimum of positive doubles through their bit patterns (order-independent, exact)
__device__ __forceinline__ void block_min_dt(double dt, unsigned long long* dtbits) {
  __shared__ unsigned long long smin[kBlock / 32];
  unsigned long long b = (unsigned long long)__double_as_longlong(dt);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long t = __shfl_down_sync(0xffffffffu, b, o);
    b = t < b ? t : b;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) smin[w] = b;
  __syncthreads();
  if (w == 0) {
    b = lane < (int)(blockDim.x >> 5) ? smin[lane] : ~0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long t = __shfl_down_sync(0xffffffffu, b, o);
      b = t < b ? t : b;
    }
    if (lane == 0) atomicMin(dtbits, b);
  }
}

__device__ __forceinline__ void flag_error(int* err, int code, int cell) {
  if (atomicCAS(err, 0, code) == 0) err[1] = cell;
}

__global__ void __launch_bounds__(kBlock) k_timestep(DevMesh m, const double* cons, double gamma,
                                                      double cfl, unsigned long long* dtbits, int* err) {
  pdl_wait();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  double dt = __longlong_as_double(0x7fefffffffffffffll);  // largest finite double
  if (c < m.nci) {
    double u[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) u[v] = cons[v * (size_t)m.ldc + c];
    double d;
    if (cell_dt(m, gamma, cfl, c, u, d)) {
      dt = d;
      if (!(d > 0.0)) flag_error(err, TY_ERR_NANDT, c);
    } else {
      flag_error(err, TY_ERR_NEGENERGY, c);
    }
  }
  block_min_dt(dt, dtbits);
}

#if TY_FAST
// a > 0 (infinity included, NaN not) on the bit pattern
__device__ __forceinline__ bool positive_bits(double a) {
  return (unsigned long long)(__double_as_longlong(a) - 1) < 0x7ff0000000000000ull;
}

// Runge-Kutta update at the end of a stage, one kernel per shape of the plan: INIT the first
// non-zero term of the final combination, FINAL the last stage.  A run-time plan in one kernel
// issued both sides of its choices (a predicated-off FP64 instruction occupies the pipe too);
// dt/V is folded into the coefficients, zero coefficients do no work, 1/rho serves the
// primitive variables and the next time step.  TGV 64^3x5 on GB300: 194 -> 118 us per launch
// (152 us for the last stage, with the next time step).
template <bool INIT, bool FINAL>
__global__ void __launch_bounds__(kBlock) k_rk_update(DevMesh m, DevState s, RkStagePlan plan, double gamma, double dt,
                                                       const unsigned long long* dtbits, unsigned long long* dtbits_next,
                                                       unsigned long long* dtbits_reset, double cfl) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  int es[kMaxSlot];
  face_list(m, min(c, m.nci - 1), es);
  pdl_wait();
  double dtc = __longlong_as_double(0x7fefffffffffffffll);
  if (c < m.nci) {
    const size_t ld = m.ldc;
    F64 R[5], u0[5], next[5];
    gather_residual(m, s, es, R);
    const F64 rs = F64(plan.dtloc ? plan.dtloc[c] : load_dt(dt, dtbits)) * F64(m.invV[c]);
#pragma unroll
    for (int v = 0; v < 5; ++v) u0[v] = s.u0[v * ld + c];
    for (int k = 0; k < plan.nops; ++k) {
      const RkOp op = plan.ops[k];
      const F64 oc = F64(op.c) * rs;
      double* part = s.pk[op.target] + c;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const F64 val = fma(oc, R[v], op.from_u0 ? u0[v] : F64(part[v * ld]));
        if (op.is_next) next[v] = val;
        else part[v * ld] = val.v;
      }
    }
    if (FINAL || plan.has_acc) {
      const F64 ca = F64(plan.c_acc) * rs;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const F64 a = INIT ? ca * R[v] : fma(ca, R[v], F64(s.acc[v * ld + c]));
        if constexpr (FINAL) next[v] = u0[v] + a;
        if (!FINAL || plan.store_acc) s.acc[v * ld + c] = a.v;
      }
    }
    const F64 ir = rcp_nr(next[0]);
    const F64 vx = next[2] * ir, vy = next[3] * ir, vz = next[4] * ir;
    const F64 v2 = fma(vx, vx, fma(vy, vy, vz * vz));
    const F64 p = F64(gamma - 1.0) * fma(F64(-0.5) * next[0], v2, next[1]);
    if constexpr (FINAL) {
#pragma unroll
      for (int v = 0; v < 5; ++v) s.u0[v * ld + c] = next[v].v;
    }
    s.prim[c] = next[0].v;
    s.prim[ld + c] = p.v;
    s.prim[2 * ld + c] = vx.v;
    s.prim[3 * ld + c] = vy.v;
    s.prim[4 * ld + c] = vz.v;
    if (FINAL && dtbits_next) {
      const F64 a2 = F64(gamma) * p * ir;
      if (positive_bits(a2.v)) {
        const F64 d = F64(cfl * m.geo2[c]) * rcp_nr(sqrt_nr(v2) + sqrt_nr(a2));
        dtc = d.v;
        if (!positive_bits(dtc)) flag_error(s.err, TY_ERR_NANDT, c);
      } else {
        flag_error(s.err, TY_ERR_NEGENERGY, c);
      }
    }
  }
  if (FINAL && dtbits_next) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *dtbits_reset = kMaxDtBits;
    block_min_dt(dtc, dtbits_next);
  }
}
#else
// Runge-Kutta update at the end of a stage.  Applies the plan's partial sums, the final
// combination, and derives the primitive variables of the new state (and its time step
// after the last stage when dtbits_next is given).
__global__ void __launch_bounds__(kBlock) k_rk_update(DevMesh m, DevState s, RkStagePlan plan, double gamma, double dt,
                                                       const unsigned long long* dtbits, unsigned long long* dtbits_next,
                                                       unsigned long long* dtbits_reset, double cfl) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  int es[kMaxSlot];
  face_list(m, min(c, m.nci - 1), es);
  pdl_wait();
  const bool active = c < m.nci;
  double dtc = __longlong_as_double(0x7fefffffffffffffll);
  if (active) {
    const size_t ld = m.ldc;
    double R[5];
    gather_residual(m, s, es, R);
    const double dtv = plan.dtloc ? plan.dtloc[c] : load_dt(dt, dtbits);
    const double coef = dtv / m.cvol[c];  // R = (dt/V) R first, as flux_to_res does
#pragma unroll
    for (int v = 0; v < 5; ++v) R[v] = coef * R[v];
    double u0[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) u0[v] = s.u0[v * ld + c];
    double next[5];
    bool have_next = false;
    for (int k = 0; k < plan.nops; ++k) {
      const RkOp op = plan.ops[k];
      double* part = s.pk[op.target];
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        double base = op.from_u0 ? u0[v] : part[v * ld + c];
        double val = base + op.c * R[v];
        if (op.is_next) next[v] = val;
        else part[v * ld + c] = val;
      }
      if (op.is_next) have_next = true;
    }
    if (plan.has_acc) {
      const double ca = plan.c_acc;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        double a = plan.acc_init ? ca * R[v] : s.acc[v * ld + c] + ca * R[v];
        if (plan.final_stage) next[v] = u0[v] + a;
        if (!plan.final_stage || plan.store_acc) s.acc[v * ld + c] = a;
      }
      if (plan.final_stage) have_next = true;
    }
    if (have_next) {
      if (plan.final_stage) {
#pragma unroll
        for (int v = 0; v < 5; ++v) s.u0[v * ld + c] = next[v];
      }
      double q[5];
      cons_to_prim(gamma, next, q);
#pragma unroll
      for (int v = 0; v < 5; ++v) s.prim[v * ld + c] = q[v];
      if (dtbits_next) {
        double d;
        if (cell_dt(m, gamma, cfl, c, next, d)) {
          dtc = d;
          if (!(d > 0.0)) flag_error(s.err, TY_ERR_NANDT, c);
        } else {
          flag_error(s.err, TY_ERR_NEGENERGY, c);
        }
      }
    }
  }
  if (dtbits_next) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *dtbits_reset = kMaxDtBits;
    block_min_dt(dtc, dtbits_next);
  }
}
#endif

// ---------------------------------------------------------------------------
// launch sequences
inline unsigned nblk(int n) { return (unsigned)((n + kBlock - 1) / kBlock); }
// Blocks of the stage kernels: four warps, one per SM quarter, so that a small mesh spreads over
// as many quarters as it has warps (8,192 cells: face kernel 8.7 -> 5.9 us, update 5.1-6.8 ->
// 4.2-5.3 us against blocks of 256; no difference on large meshes).
constexpr int kStage = 128;
constexpr int kPdlFaces = 1 << 17;  // see k_face_flux_fast: the wait costs more than the gap beyond
inline unsigned sblk(int n) { return (unsigned)((n + kStage - 1) / kStage); }

cudaError_t prim_from(const DevMesh& m, const DevState& s, const SpatOpts& o, const double* cons,
                      cudaStream_t st, Prof* pr) {
  if (m.nci > 0)
    pr->launch(K_PRIM, st, [&] { launch_pdl(k_prim, sblk(m.nci), kStage, st, m, cons, s.prim, o.gamma); });
  return cudaGetLastError();
}

// everything between the primitive variables of a stage state and the face fluxes
cudaError_t residual_faces(const DevMesh& m, const DevState& s, const SpatOpts& o, cudaStream_t st, Prof* pr) {
  const bool cell_kernel = kFast && o.highres != TY_HRES_NONE;
  if (m.ng > 0 && !(cell_kernel && m.ghost_copy))
    pr->launch(K_GHOST_PRIM, st, [&] { launch_pdl(k_ghost_prim, sblk(m.ng), kStage, st, m, s.prim, o); });
#if TY_FAST
  if (cell_kernel) {
    pr->launch(K_CELL_FAST, st, [&] { cell_fast(m, s, o, o.viscous != TY_VISC_NONE, m.ghost_copy, st); });
    if (o.viscous != TY_VISC_NONE && m.ng > 0)
      pr->launch(K_GHOST_GRAD, st, [&] { launch_pdl(k_ghost_grad, sblk(m.ng), kStage, st, m, s.grad); });
    pr->launch(K_FACE_FLUX_FAST, st, [&] {
      if (m.nf <= kPdlFaces) launch_pdl(k_face_flux_fast<true>, sblk(m.nf), kStage, st, m, s, o);
      else k_face_flux_fast<false><<<sblk(m.nf), kStage, 0, st>>>(m, s, o);
    });
    return cudaGetLastError();
  }
#endif
  if (o.gradmeth != TY_GRAD_NONE) {
    pr->launch(K_GRAD, st, [&] { launch_pdl(k_grad, sblk(m.nci), kStage, st, m, s); });
    if (m.ng > 0)
      pr->launch(K_GHOST_GRAD, st, [&] { launch_pdl(k_ghost_grad, sblk(m.ng), kStage, st, m, s.grad); });
  }
  if (o.postlim != TY_POSTLIM_NONE) {
    pr->launch(K_FACE_STATES, st, [&] { launch_pdl(k_face_states, sblk(m.nf), kStage, st, m, s, o); });
    const double klim = o.postlim == TY_POSTLIM_BARTH ? 0.5 : 1.0;
    pr->launch(K_BARTH, st, [&] { launch_pdl(k_barth, sblk(m.nci), kStage, st, m, s, klim); });
    pr->launch(K_FACE_FLUX_LIM, st, [&] { launch_pdl(k_face_flux_lim, sblk(m.nf), kStage, st, m, s, o); });
  } else {
    pr->launch(K_FACE_FLUX, st, [&] { launch_pdl(k_face_flux, sblk(m.nf), kStage, st, m, s, o); });
  }
  return cudaGetLastError();
}

cudaError_t residual_gather(const DevMesh& m, const DevState& s, double dt, const unsigned long long* dtbits,
                            double* out, int ld, cudaStream_t st, Prof* pr) {
  pr->launch(K_GATHER, st, [&] { launch_pdl(k_gather, sblk(m.nci), kStage, st, m, s, dt, dtbits, out, ld); });
  return cudaGetLastError();
}

cudaError_t rk_update(const DevMesh& m, const DevState& s, const SpatOpts& o, const RkStagePlan& plan, double dt,
                      const unsigned long long* dtbits, unsigned long long* dtbits_next,
                      unsigned long long* dtbits_reset, double cfl, cudaStream_t st, Prof* pr) {
  pr->launch(K_RK_UPDATE, st, [&] {
#if TY_FAST
    auto* k = plan.final_stage ? (plan.acc_init ? k_rk_update<true, true> : k_rk_update<false, true>)
                               : (plan.acc_init ? k_rk_update<true, false> : k_rk_update<false, false>);
    launch_pdl(k, sblk(m.nci), kStage, st, m, s, plan, o.gamma, dt, dtbits, dtbits_next, dtbits_reset, cfl);
#else
    launch_pdl(k_rk_update, sblk(m.nci), kStage, st, m, s, plan, o.gamma, dt, dtbits, dtbits_next, dtbits_reset, cfl);
#endif
  });
  return cudaGetLastError();
}

cudaError_t timestep(const DevMesh& m, const DevState& s, const SpatOpts& o, const double* cons, double cfl,
                     unsigned long long* dtbits, cudaStream_t st, Prof* pr) {
  pr->launch(K_TIMESTEP, st, [&] {
    launch_pdl(k_timestep, sblk(m.nci), kStage, st, m, cons, o.gamma, cfl, dtbits, s.err);
  });
  return cudaGetLastError();
}

// One stage of the ghost-row bookkeeping (GhostRk): one thread per ghost cell, [5][ng] arrays
// (gres [nstage][5][ng]), the operation order of the oracle's Runge-Kutta loop over all cells.
__global__ void k_ghost_rows(DevMesh m, const double* __restrict__ flux, GhostRk r, double gamma,
                             double* __restrict__ gcons, double* __restrict__ gres, double* __restrict__ gprim) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= m.ng) return;
  const size_t ng = m.ng;
  const int f = m.gface[g];
  double U[5], Q[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) U[v] = gcons[v * ng + g];
  for (int s = 0; s < r.stage; ++s)
#pragma unroll
    for (int v = 0; v < 5; ++v) U[v] = U[v] + r.cs[s] * gres[(s * 5 + v) * ng + g];
  cons_to_prim(gamma, U, Q);
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    gprim[v * ng + g] = Q[v];
    gres[(r.stage * 5 + v) * ng + g] = flux[v * (size_t)m.ldf + f];
  }
  if (r.stage == r.nstage - 1) {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      double a = r.cf[0] * gres[v * ng + g];
      for (int s = 1; s < r.nstage; ++s) a = a + r.cf[s] * gres[(s * 5 + v) * ng + g];
      gcons[v * ng + g] = gcons[v * ng + g] + a;
    }
  }
}

cudaError_t ghost_rows(const DevMesh& m, const DevState& s, const SpatOpts& o, const GhostRk& r, double* gcons,
                       double* gres, double* gprim, cudaStream_t st) {
  if (m.ng > 0) k_ghost_rows<<<nblk(m.ng), kBlock, 0, st>>>(m, s.flux, r, o.gamma, gcons, gres, gprim);
  return cudaGetLastError();
}

// Typhon layout (rho[n], rhoE[n], rhou as (x,y,z)[n]) <-> SoA u0, on the device
__global__ void k_unpack_state(DevMesh m, const double* __restrict__ stage, double* __restrict__ u0) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  const size_t n = m.nci, ld = m.ldc;
  u0[c] = stage[c];
  u0[ld + c] = stage[n + c];
#pragma unroll
  for (int k = 0; k < 3; ++k) u0[(2 + k) * ld + c] = stage[2 * n + 3 * (size_t)c + k];
}
__global__ void k_pack_state(DevMesh m, const double* __restrict__ u0, double* __restrict__ stage) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  const size_t n = m.nci, ld = m.ldc;
  stage[c] = u0[c];
  stage[n + c] = u0[ld + c];
#pragma unroll
  for (int k = 0; k < 3; ++k) stage[2 * n + 3 * (size_t)c + k] = u0[(2 + k) * ld + c];
}
cudaError_t unpack_state(const DevMesh& m, const DevState& s, cudaStream_t st) {
  k_unpack_state<<<nblk(m.nci), kBlock, 0, st>>>(m, s.stage, s.u0);
  return cudaGetLastError();
}
cudaError_t pack_state(const DevMesh& m, const DevState& s, cudaStream_t st) {
  k_pack_state<<<nblk(m.nci), kBlock, 0, st>>>(m, s.u0, s.stage);
  return cudaGetLastError();
}

}  // namespace TY_KNS
}  // namespace tyk
