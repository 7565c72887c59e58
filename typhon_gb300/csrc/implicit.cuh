// Kernels of the implicit step, instantiated once per arithmetic mode after kernels.cuh.
//
// Assembly follows Typhon's order of operations so that the exact mode reproduces the CPU
// restatement bit for bit:
//   flux Jacobians       calc_jacflux.f90:49-77, calc_jac_hll.f90:46-57 (HLLC, Roe),
//                        calc_jac_rusanov.f90 (Rusanov), viscous diagonal
//                        calc_flux_viscous_cell.f90:149-158, symmetry ns_bocojacobian.f90:47-85
//                        (and, new, the far-field and no-slip wall ghost dependences folded in
//                        the same way),
//                        surface scaling flux_to_res.f90:74-80
//   BDLU blocks          build_implicit_bdlu.f90:44-83 (diagonal contributions of a cell
//                        summed in ascending face order, as the face loop there does)
//   mat-vec              SPMAT_BDLU.f90:139-157 (y = A x), :240-262 (y = z - A x)
// Reductions (dot products, norms) use a fixed two-level tree: deterministic from run to run,
// but not Typhon's sequential sum, so the Krylov iterates agree with the CPU restatement to
// rounding, not bitwise.
#pragma once
#include <algorithm>
#include <type_traits>

#include "implicit.hpp"

namespace tyk {
namespace TY_KNS {

// quotient and root of the Jacobians: IEEE in exact mode, Newton-Raphson (fastmath.cuh) in fast mode
__device__ __forceinline__ double jac_div(double a, double b) {
  if constexpr (kFast) return a * rcp_nr(b);
  return a / b;
}
__device__ __forceinline__ double jac_sqrt(double a) {
  if constexpr (kFast) return root_nr(a);
  return sqrt(a);
}

// Jacobian of the physical flux along n, row-major (calc_jacflux.f90:49-77); q = (rho, p, u)
__device__ void jacflux(double g, double ig1, const double* q, double nx, double ny, double nz, double vn, double* J) {
  const double g1 = g - 1.0;
  const double u[3] = {q[2], q[3], q[4]}, t[3] = {nx, ny, nz};
  const double v2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  const double en = jac_div(ig1 * q[1], q[0]) + .5 * v2;
  J[0] = 0.0; J[1] = 0.0; J[2] = t[0]; J[3] = t[1]; J[4] = t[2];
  J[5] = vn * (g1 * v2 - g * en);
  J[6] = vn * g;
  const double c23 = g * en - .5 * g1 * v2;
#pragma unroll
  for (int k = 0; k < 3; ++k) J[7 + k] = c23 * t[k] - g1 * vn * u[k];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    J[(2 + k) * 5] = .5 * g1 * v2 * t[k] - vn * u[k];
    J[(2 + k) * 5 + 1] = g1 * t[k];
  }
  const double gn[3] = {g1 * t[0], g1 * t[1], g1 * t[2]};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) J[(2 + i) * 5 + 2 + j] = u[i] * t[j] - gn[i] * u[j];
  J[12] = J[12] + vn;
  J[18] = J[18] + vn;
  J[24] = J[24] + vn;
}

// Left and right flux Jacobians of one face, per unit surface
__device__ void face_jacobians(const SpatOpts& o, const double* L, const double* R, double nx, double ny, double nz,
                               double* JL, double* JR) {
  const double g = o.gamma;
  const double vnl = L[2] * nx + L[3] * ny + L[4] * nz;
  const double vnr = R[2] * nx + R[3] * ny + R[4] * nz;
  const double al = jac_sqrt(jac_div(g * L[1], L[0])), ar = jac_sqrt(jac_div(g * R[1], R[0]));
  jacflux(g, o.ig1, L, nx, ny, nz, vnl, JL);
  jacflux(g, o.ig1, R, nx, ny, nz, vnr, JR);
  if (o.scheme == TY_SCH_RUSANOV) {  // calc_jac_rusanov.f90: (A_L + ray I)/2, (A_R - ray I)/2
    const double ray = fmax(fabs(vnl) + al, fabs(vnr) + ar);
#pragma unroll
    for (int i = 0; i < 5; ++i) { JL[i * 6] = JL[i * 6] + ray; JR[i * 6] = JR[i * 6] - ray; }
#pragma unroll
    for (int k = 0; k < 25; ++k) { JL[k] = .5 * JL[k]; JR[k] = .5 * JR[k]; }
    return;
  }
  double sl, sr;
  if (o.hll_family != 0) {  // the HLLC / HLLE family's wave speeds (calc_flux_hllc.f90:86-124, calc_flux_hlle.f90:83-120)
    const double gig1 = o.gdg1;
    double t1 = jac_sqrt(jac_div(R[0], L[0]));
    double roe_rho = L[0] * t1;
    double kl = jac_div(1.0, 1.0 + t1);
    double kr = t1 * kl;
    double rux = kl * L[2] + kr * R[2], ruy = kl * L[3] + kr * R[3], ruz = kl * L[4] + kr * R[4];
    double sqL = L[2] * L[2] + L[3] * L[3] + L[4] * L[4];
    double sqR = R[2] * R[2] + R[3] * R[3] + R[4] * R[4];
    double h1 = jac_div(gig1 * L[1], L[0]) + 0.5 * sqL;
    double h2 = jac_div(gig1 * R[1], R[0]) + 0.5 * sqR;
    h1 = kl * h1 + kr * h2;
    double roe_p = jac_div((h1 - 0.5 * (rux * rux + ruy * ruy + ruz * ruz)) * roe_rho, gig1);
    double vm = rux * nx + ruy * ny + ruz * nz;
    double am = jac_sqrt(jac_div(g * roe_p, roe_rho));
    hll_speeds(o, vnl, vnr, al, ar, vm, am, sl, sr);
    if (o.hll_family == 1) {  // calc_flux_hllc.f90 passes min(sl, 0), max(sr, 0) to calc_jac_hll
      sl = fmin(sl, 0.0);
      sr = fmax(sr, 0.0);
    }
  } else {  // Roe flux: HLL Jacobian with Einfeldt's speeds from the Roe average (new)
    double t1 = jac_sqrt(jac_div(R[0], L[0]));
    double kl = jac_div(1.0, 1.0 + t1), kr = t1 * kl;
    double ux = kl * L[2] + kr * R[2], uy = kl * L[3] + kr * R[3], uz = kl * L[4] + kr * R[4];
    double hl = jac_div(o.gdg1 * L[1], L[0]) + 0.5 * (L[2] * L[2] + L[3] * L[3] + L[4] * L[4]);
    double hr = jac_div(o.gdg1 * R[1], R[0]) + 0.5 * (R[2] * R[2] + R[3] * R[3] + R[4] * R[4]);
    double am = jac_sqrt((g - 1.0) * (kl * hl + kr * hr - 0.5 * (ux * ux + uy * uy + uz * uz)));
    double vm = ux * nx + uy * ny + uz * nz;
    sl = fmin(fmin(vnl - al, vm - am), 0.0);
    sr = fmax(fmax(vnr + ar, vm + am), 0.0);
  }
#pragma unroll
  for (int i = 0; i < 5; ++i) { JL[i * 6] = JL[i * 6] - sl; JR[i * 6] = JR[i * 6] - sr; }
  const double cl = jac_div(sr, sr - sl), cr = jac_div(-sl, sr - sl);
#pragma unroll
  for (int k = 0; k < 25; ++k) { JL[k] = cl * JL[k]; JR[k] = cr * JR[k]; }
}

// d(ghost conservative state)/d(inside conservative state) of a far-field face (new), rows
// and columns (rho, rhoE, rhou, rhov, rhow); false when the ghost does not depend on the inside
__device__ bool farfield_jacobian(const SpatOpts& o, double nx, double ny, double nz, const double* q, double* M) {
  const double* qi = o.farfield;
  const double vn = qi[2] * nx + qi[3] * ny + qi[4] * nz;
  const double c = sqrt(o.gamma * qi[1] / qi[0]);
#pragma unroll
  for (int k = 0; k < 25; ++k) M[k] = 0.0;
  if (vn <= -c) return false;
  const double u2 = q[2] * q[2] + q[3] * q[3] + q[4] * q[4];
  if (vn < -1e-8 * c) {
    M[5] = 0.5 * u2; M[6] = 1.0; M[7] = -q[2]; M[8] = -q[3]; M[9] = -q[4];
  } else if (vn < c) {
    M[0] = 1.0;
    M[5] = -0.5 * u2; M[7] = q[2]; M[8] = q[3]; M[9] = q[4];
    M[12] = 1.0; M[18] = 1.0; M[24] = 1.0;
  } else {
#pragma unroll
    for (int i = 0; i < 5; ++i) M[i * 6] = 1.0;
  }
  return true;
}

// face states exactly as the flux kernels of the residual build them
__device__ void implicit_face_states(const DevMesh& m, const DevState& s, const SpatOpts& o, int src, int f,
                                     double* QL, double* QR) {
  const size_t ld = m.ldc, lf = m.ldf;
  auto side_state = [&](int face, int side, double* Q) {
    if (src == 0) {
      recon(m, s, o, face, side, Q);
    } else if (src == 1) {
      const int c = side ? m.fc2[face] : m.fc1[face];
      const double* qf = side ? s.cr : s.cl;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        double qc = s.prim[v * ld + c];
        double rr = s.ratio[(v < 2 ? v : 2) * ld + c];
        Q[v] = qc + rr * (qf[v * lf + face] - qc);
      }
    } else {
      const double* qf = side ? s.cr : s.cl;
#pragma unroll
      for (int v = 0; v < 5; ++v) Q[v] = qf[v * lf + face];
    }
  };
  side_state(f, 0, QL);
  const int kind = f < m.nfi ? TY_BC_INTERIOR : m.fbc[f];
  if (kind == TY_BC_PERIODIC) {
    side_state(m.part[f], 0, QR);
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
    side_state(f, 1, QR);
  }
}

// J dt / V of build_implicit_bdlu.f90:51-55: two roundings per entry in exact mode (the 25
// quotients by V through its reciprocal), a product with the per-cell quotient dt / V in fast mode
__device__ __forceinline__ void scaled_block(const double* J, double dt, double V, double* U) {
  if constexpr (kFast) {
    const double q = dt / V;
#pragma unroll
    for (int k = 0; k < 25; ++k) U[k] = J[k] * q;
  } else {
    const Divisor d = divisor(V);
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 25; ++k) U[k] = value(quotient(F64(J[k]) * F64(dt), d, bad));
    if (bad) {
#pragma unroll
      for (int k = 0; k < 25; ++k) U[k] = div_ieee(J[k] * dt, V);
    }
  }
}

__device__ __forceinline__ double imp_dt(const ImpState& im, const ImpArgs& a, int c) {
  return a.local_dt ? im.dtloc[c] : __longlong_as_double((long long)*a.dtg);
}

// per-cell stability time step of the implicit step (calc_ns_timestep.f90:52-103), its global
// minimum through the bit patterns, and the error word for a negative or NaN energy
__global__ void __launch_bounds__(kBlock) k_imp_dtloc(DevMesh m, const double* __restrict__ cons, double gamma,
                                                       double cfl, double* __restrict__ dtloc,
                                                       unsigned long long* dtbits, int* err) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  double dt = __longlong_as_double(0x7fefffffffffffffll);
  if (c < m.nci) {
    double u[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) u[v] = cons[v * (size_t)m.ldc + c];
    double d;
    if (cell_dt(m, gamma, cfl, c, u, d)) {
      dt = d;
      dtloc[c] = d;
      if (!(d > 0.0)) flag_error(err, TY_ERR_NANDT, c);
    } else {
      dtloc[c] = 0.0;
      flag_error(err, TY_ERR_NEGENERGY, c);
    }
  }
  block_min_dt(dt, dtbits);
}

__device__ __forceinline__ void store_block(double* dst, const double* J) {
  double2* d2 = reinterpret_cast<double2*>(dst);
#pragma unroll
  for (int k = 0; k < 12; ++k) d2[k] = make_double2(J[2 * k], J[2 * k + 1]);
  dst[24] = J[24];
}
__device__ __forceinline__ void load_block(const double* src, double* J) {
  const double2* s2 = reinterpret_cast<const double2*>(src);
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    double2 t = __ldg(s2 + k);
    J[2 * k] = t.x;
    J[2 * k + 1] = t.y;
  }
  J[24] = __ldg(src + 24);
}
__device__ __forceinline__ void store_block32(float* dst, const double* J) {
  float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
  for (int k = 0; k < 6; ++k)
    d4[k] = make_float4((float)J[4 * k], (float)J[4 * k + 1], (float)J[4 * k + 2], (float)J[4 * k + 3]);
  d4[6] = make_float4((float)J[24], 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void store_block32f(float* dst, const float* J) {
  float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
  for (int k = 0; k < 6; ++k) d4[k] = make_float4(J[4 * k], J[4 * k + 1], J[4 * k + 2], J[4 * k + 3]);
  d4[6] = make_float4(J[24], 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void load_block32(const float* src, float* J) {
  const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    float4 t = __ldg(s4 + k);
    J[4 * k] = t.x;
    if (4 * k + 1 < 25) J[4 * k + 1] = t.y;
    if (4 * k + 2 < 25) J[4 * k + 2] = t.z;
    if (4 * k + 3 < 25) J[4 * k + 3] = t.w;
  }
}

// Face Jacobians: inviscid, + viscous diagonal, symmetry mirror, times S; then the
// off-diagonal blocks of interior faces (build_implicit_bdlu.f90:54-58)
__global__ void __launch_bounds__(128) k_imp_face(DevMesh m, DevState s, SpatOpts o, ImpState im, ImpArgs a) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  double QL[5], QR[5];
  implicit_face_states(m, s, o, a.src, f, QL, QR);
  const double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  double JL[25], JR[25];
  face_jacobians(o, QL, QR, nx, ny, nz, JL, JR);
  if (o.viscous != TY_VISC_NONE) {
    const size_t ld = m.ldc, lf = m.ldf;
    const int icl = m.fc1[f], icr = m.fc2[f];
    const double r = o.rgas;
    const double dHL = m.vgeo[f], dHR = m.vgeo[lf + f];
    const double wx = m.vgeo[2 * lf + f], wy = m.vgeo[3 * lf + f], wz = m.vgeo[4 * lf + f];
    const double rL = s.prim[icl], rR = s.prim[icr], pL = s.prim[ld + icl], pR = s.prim[ld + icr];
    const double TL = jac_div(pL, rL * r), TR = jac_div(pR, rR * r);
    const double TH = dHR * TL + dHL * TR;
    const double rhoH = dHR * rL + dHL * rR;
    const double mu = viscosity(o, rhoH, TH);
    const double id = jac_div(jac_div(mu, dHR * rL + dHL * rR), jac_sqrt(wx * wx + wy * wy + wz * wz));
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      JR[i * 6] = JR[i * 6] - id;
      JL[i * 6] = JL[i * 6] + id;
    }
  }
  const int bkind = f >= m.nfi ? m.fbc[f] : TY_BC_INTERIOR;
  bool fold = false;
  double M[25];
  if (bkind == TY_BC_SYMMETRY) {
    const double nn[3] = {nx, ny, nz};
#pragma unroll
    for (int k = 0; k < 25; ++k) M[k] = 0.0;
#pragma unroll
    for (int i = 0; i < 5; ++i) M[i * 6] = 1.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) M[(2 + i) * 5 + 2 + j] = M[(2 + i) * 5 + 2 + j] - 2.0 * (nn[i] * nn[j]);
    fold = true;
  } else if (bkind == TY_BC_FARFIELD) {
    fold = farfield_jacobian(o, nx, ny, nz, QL, M);
  } else if (bkind == TY_BC_OUTLET_SUP) {  // ns_bocojacobian.f90: dQr/dQl = I
#pragma unroll
    for (int k = 0; k < 25; ++k) M[k] = 0.0;
#pragma unroll
    for (int i = 0; i < 5; ++i) M[i * 6] = 1.0;
    fold = true;
  } else if (bkind == TY_BC_NOSLIP) {  // new: d(2 rho u_w - m, rho E + 2 rho |u_w|^2 - 2 u_w.m)/dU
    const double w[3] = {d3(m.fwall, m.ldf, f, 0), d3(m.fwall, m.ldf, f, 1), d3(m.fwall, m.ldf, f, 2)};
#pragma unroll
    for (int k = 0; k < 25; ++k) M[k] = 0.0;
    M[0] = 1.0;
    M[5] = 2.0 * (w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    M[6] = 1.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) M[7 + j] = -2.0 * w[j];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      M[(2 + i) * 5] = 2.0 * w[i];
      M[(2 + i) * 5 + 2 + i] = -1.0;
    }
    fold = true;
  }
  if (fold) {
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k) t = t + JR[i * 5 + k] * M[k * 5 + j];
        JL[i * 5 + j] = JL[i * 5 + j] + t;
      }
#pragma unroll
    for (int k = 0; k < 25; ++k) JR[k] = 0.0;
  }
  const double S = m.fs[f];
#pragma unroll
  for (int k = 0; k < 25; ++k) { JL[k] = S * JL[k]; JR[k] = S * JR[k]; }
  store_block(im.jacL + (size_t)f * kBlk, JL);
  store_block(im.jacR + (size_t)f * kBlk, JR);
  if (f < m.nfi) {
    const int c1 = m.fc1[f], c2 = m.fc2[f];
    const double dt1 = imp_dt(im, a, c1), dt2 = imp_dt(im, a, c2);
    double U[25];
    scaled_block(JR, dt1, m.cvol[c1], U);
    if (a.want64) store_block(im.upper + (size_t)f * kBlk, U);
    if (a.want32) store_block32(im.upper32 + (size_t)f * kBlk32, U);
    scaled_block(JL, -dt2, m.cvol[c2], U);
    if (a.want64) store_block(im.lower + (size_t)f * kBlk, U);
    if (a.want32) store_block32(im.lower32 + (size_t)f * kBlk32, U);
  }
}

// 5x5 inverse by Gauss-Jordan elimination with partial pivoting; false if singular
template <class T>
__device__ bool inv5(const T* A, T* X) {
  T a[25];
#pragma unroll
  for (int k = 0; k < 25; ++k) { a[k] = A[k]; X[k] = T(0); }
#pragma unroll
  for (int i = 0; i < 5; ++i) X[i * 6] = T(1);
#pragma unroll
  for (int col = 0; col < 5; ++col) {
    int p = col;
    T best = fabs(a[col * 5 + col]);
#pragma unroll
    for (int r = col + 1; r < 5; ++r) {
      T v = fabs(a[r * 5 + col]);
      if (v > best) { best = v; p = r; }
    }
    if (!(best > T(0))) return false;
    // row swap with compile-time indices only (selects), so that a and X stay in registers
#pragma unroll
    for (int r = col + 1; r < 5; ++r) {
      const bool sw = r == p;
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const T ta = a[col * 5 + k], tx = X[col * 5 + k];
        a[col * 5 + k] = sw ? a[r * 5 + k] : ta;
        a[r * 5 + k] = sw ? ta : a[r * 5 + k];
        X[col * 5 + k] = sw ? X[r * 5 + k] : tx;
        X[r * 5 + k] = sw ? tx : X[r * 5 + k];
      }
    }
    const T ip = T(1) / a[col * 5 + col];
#pragma unroll
    for (int k = 0; k < 5; ++k) { a[col * 5 + k] *= ip; X[col * 5 + k] *= ip; }
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      if (r == col) continue;
      const T fct = a[r * 5 + col];
#pragma unroll
      for (int k = 0; k < 5; ++k) { a[r * 5 + k] -= fct * a[col * 5 + k]; X[r * 5 + k] -= fct * X[col * 5 + k]; }
    }
  }
  return true;
}

// Diagonal block of each interior cell: identity, then the cell's faces in ascending order
// (build_implicit_bdlu.f90:52-58, 71-73); optional block-Jacobi inverse
__global__ void __launch_bounds__(128) k_imp_diag(DevMesh m, ImpState im, ImpArgs a, int want_inv, int* err) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  double D[25];
#pragma unroll
  for (int k = 0; k < 25; ++k) D[k] = 0.0;
#pragma unroll
  for (int i = 0; i < 5; ++i) D[i * 6] = 1.0;
  const double dt = imp_dt(im, a, c), V = m.cvol[c];
  for (int sl = 0; sl < m.nslot; ++sl) {
    const int e = im.cfo[sl * (size_t)m.nci + c];
    if (e < 0) break;
    const int f = e >> 1;
    double J[25];
    load_block(((e & 1) ? im.jacR : im.jacL) + (size_t)f * kBlk, J);
    double U[25];
    scaled_block(J, (e & 1) ? -dt : dt, V, U);
#pragma unroll
    for (int k = 0; k < 25; ++k) D[k] = value(X64(D[k]) + X64(U[k]));
  }
  if (a.want64) store_block(im.diag + (size_t)c * kBlk, D);
  if (a.want32) store_block32(im.diag32 + (size_t)c * kBlk32, D);
  if (want_inv && !a.want64) {  // mixed solve: only the FP32 inverse is used, so invert in FP32
    float Df[25], Xf[25];
#pragma unroll
    for (int k = 0; k < 25; ++k) Df[k] = (float)D[k];
    if (!inv5(Df, Xf)) {
      flag_error(err, TY_ERR_STATE, c);
#pragma unroll
      for (int k = 0; k < 25; ++k) Xf[k] = 0.f;
#pragma unroll
      for (int i = 0; i < 5; ++i) Xf[i * 6] = 1.f;
    }
    store_block32f(im.dinv32 + (size_t)c * kBlk32, Xf);
  } else if (want_inv) {
    double X[25];
    if (!inv5(D, X)) {
      flag_error(err, TY_ERR_STATE, c);
#pragma unroll
      for (int k = 0; k < 25; ++k) X[k] = 0.0;
#pragma unroll
      for (int i = 0; i < 5; ++i) X[i * 6] = 1.0;
    }
    if (a.want64) store_block(im.dinv + (size_t)c * kBlk, X);
    if (a.want32) store_block32(im.dinv32 + (size_t)c * kBlk32, X);
  }
}

// right-hand side: the residual with per-cell dt (flux_to_res.f90:90-144), packed per cell
__global__ void __launch_bounds__(kBlock) k_imp_rhs(DevMesh m, DevState s, ImpState im, ImpArgs a,
                                                     double* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  double R[5];
  int es[kMaxSlot];
  face_list(m, c, es);
  gather_residual(m, s, es, R);
  const double coef = imp_dt(im, a, c) / m.cvol[c];
#pragma unroll
  for (int v = 0; v < 5; ++v) out[5 * (size_t)c + v] = coef * R[v];
}

__device__ __forceinline__ void mv5(const double* A, const double* x, double* t) {
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) s = s + A[i * 5 + j] * x[j];
    t[i] = s;
  }
}

// ---- 5x5 blocks of 32 cells through shared memory ----
// A thread that reads its own block, 16 bytes at a time, makes each warp request touch 32 lines
// (208- or 112-byte strides): the first-level cache, not HBM, then bounds the mat-vec.  Instead
// the warp copies 32 blocks together (PIECES consecutive lanes one block, asynchronously, one
// block list ahead of the arithmetic) and every thread reads its block back from shared memory,
// where both strides are free of bank conflicts.
template <int PIECES>  // 16-byte pieces of a block: 13 (26 doubles) or 7 (28 floats)
__device__ __forceinline__ void fetch_blocks(const void* mine, char* stage) {
  constexpr int PB = 32 / PIECES;  // blocks per request
  const int lane = threadIdx.x & 31, q = lane / PIECES, piece = lane - q * PIECES;
#pragma unroll
  for (int r = 0; r < 32; r += PB) {
    const int b = r + q;
    const unsigned long long p = __shfl_sync(0xffffffffu, (unsigned long long)mine, b & 31);
    if (q < PB && b < 32 && p != 0)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(stage + (b * PIECES + piece) * 16)),
                   "l"((const char*)p + piece * 16)
                   : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// y = A x (z == null) or y = z - A x: diagonal block first, then the cell's interior faces in
// ascending order.  Boundary faces multiply the (zero) ghost unknowns and are skipped.
// F32: y = S A x with FP32 blocks and FP32 x, FP32 accumulation, FP64 result.  The FP64 fast mode
// accumulates every product into the row's sum (25 multiply-adds a block instead of 30 operations).
// A slot's list entries are read one list ahead of its fetch.  GB300, us per product, own loads ->
// staged -> entries ahead: 250,000 cells FP32 40.5 -> 35.6 -> 32.4, 320,000 FP64 (fast) 108 -> 90 -> 79
// (the floors: 23 us of HBM traffic, 28 with the 64-byte granules that 112-byte blocks touch; 65 us of
// FP64 multiply-adds).
// FP64 in the fast mode only: the exact mode's rounded products are k_imp_matvec_row's.
constexpr int kMvThreads = 128;
template <bool F32>
__global__ void __launch_bounds__(kMvThreads) k_imp_matvec(DevMesh m, ImpState im, const void* __restrict__ xp,
                                                            const double* __restrict__ z, double* __restrict__ y) {
  static_assert(F32 || kFast, "sums of fused products");
  using T = typename std::conditional<F32, float, double>::type;
  constexpr int PIECES = F32 ? 7 : 13, kBytes = 32 * PIECES * 16, kStride = F32 ? kBlk32 : kBlk;
  extern __shared__ __align__(16) char stages[];  // [warps][2][32 blocks]
  const T* __restrict__ x = (const T*)xp;
  const T* up = F32 ? (const T*)im.upper32 : (const T*)im.upper;
  const T* lo = F32 ? (const T*)im.lower32 : (const T*)im.lower;
  const T* dg = F32 ? (const T*)im.diag32 : (const T*)im.diag;
  char* mine = stages + (threadIdx.x >> 5) * (2 * kBytes);
  const int lane = threadIdx.x & 31, c0 = blockIdx.x * kMvThreads + threadIdx.x;
  const bool on = c0 < m.nci;
  const int c = on ? c0 : m.nci - 1;
  const size_t n = m.nci;
  // entry of a slot: its block and neighbour, null past the cell's interior faces
  const T* A = nullptr;
  int nb = c;
  bool more = on;
  int ne = m.nslot > 0 ? im.cfo[c] : -1, nn = m.nslot > 0 ? im.cfon[c] : c;  // the next slot's, one list ahead
  auto entry = [&](int sl) {
    const int e = more && sl < m.nslot ? ne : -1;
    more = e >= 0 && (e >> 1) < m.nfi;
    A = more ? ((e & 1) ? lo : up) + (size_t)(e >> 1) * kStride : nullptr;
    nb = more ? nn : c;
    if (sl + 1 < m.nslot) {
      ne = im.cfo[(sl + 1) * n + c];
      nn = im.cfon[(sl + 1) * n + c];
    }
  };
  fetch_blocks<PIECES>(on ? dg + (size_t)c * kStride : nullptr, mine);
  T xv[5], yv[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) xv[v] = x[5 * (size_t)c + v];
  bool have = on;
  for (int s = 0; s <= m.nslot; ++s) {  // block list 0: the diagonal; s: slot s - 1
    const bool cur = have;
    T xn[5];
    entry(s);  // the next list's block and x while this one is on its way
    have = A != nullptr;
    const bool any = __any_sync(0xffffffffu, have);
    if (any) {
      fetch_blocks<PIECES>(A, mine + ((s + 1) & 1) * kBytes);
#pragma unroll
      for (int v = 0; v < 5; ++v) xn[v] = x[5 * (size_t)nb + v];
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    if (cur) {
      const T* B = (const T*)(mine + (s & 1) * kBytes + lane * PIECES * 16);
      T a[28];
      if constexpr (F32) {
#pragma unroll
        for (int k = 0; k < 7; ++k) {
          const float4 t = reinterpret_cast<const float4*>(B)[k];
          a[4 * k] = t.x; a[4 * k + 1] = t.y; a[4 * k + 2] = t.z; a[4 * k + 3] = t.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 13; ++k) {
          const double2 t = reinterpret_cast<const double2*>(B)[k];
          a[2 * k] = t.x; a[2 * k + 1] = t.y;
        }
      }
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        T q = s == 0 ? T(0) : yv[i];
        if (!F32 && s == 0 && z) q = (T)z[5 * (size_t)c + i];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          if constexpr (F32) q = fmaf(a[i * 5 + j], xv[j], q);
          else q = fma(a[i * 5 + j], z ? -xv[j] : xv[j], q);
        }
        yv[i] = q;
      }
    }
    if (!any) break;
    __syncwarp();  // the stage is free for the list after next
#pragma unroll
    for (int v = 0; v < 5; ++v) xv[v] = xn[v];
  }
  if (!on) return;
  // S A x (the row scale is all ones outside the flexible GMRES)
#pragma unroll
  for (int v = 0; v < 5; ++v) y[5 * (size_t)c + v] = !F32 && z ? (double)yv[v] : (double)yv[v] * im.rs[v];
}

// The same with one thread per row (five consecutive threads a cell, 32 cells a block): chains a
// fifth as long, so that small meshes fill the SM quarters' FP64 pipes better; the order within
// a row is the same.
constexpr int kRowCells = 32;
__global__ void __launch_bounds__(5 * kRowCells) k_imp_matvec_row(DevMesh m, ImpState im, const double* __restrict__ x,
                                                               const double* __restrict__ z, double* __restrict__ y) {
  const int lc = threadIdx.x / 5, i = threadIdx.x - 5 * lc;
  const int c = blockIdx.x * kRowCells + lc;
  if (c >= m.nci) return;
  const size_t n = m.nci;
  int e = m.nslot > 0 ? im.cfo[c] : -1, nb = e >= 0 ? im.cfon[c] : 0;
  X64 acc = z ? z[5 * (size_t)c + i] : 0.0;
  // the row's product with a block is added (y = A x) or subtracted
  auto row = [&](const double* __restrict__ A, const double* __restrict__ v, bool first) {
    X64 a[5], q[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) { a[j] = __ldg(A + 5 * i + j); q[j] = v[j]; }
    X64 s = 0.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) s = s + a[j] * q[j];
    acc = z ? acc - s : (first ? s : acc + s);
  };
  row(im.diag + (size_t)c * kBlk, x + 5 * (size_t)c, true);
  for (int sl = 0; sl < m.nslot; ++sl) {
    if (e < 0 || (e >> 1) >= m.nfi) break;
    const double* A = ((e & 1) ? im.lower : im.upper) + (size_t)(e >> 1) * kBlk;
    const double* v = x + 5 * (size_t)nb;
    if (sl + 1 < m.nslot) {  // the next face's entries while this block is on its way
      e = im.cfo[(sl + 1) * n + c];
      nb = e >= 0 ? im.cfon[(sl + 1) * n + c] : 0;
    }
    row(A, v, false);
  }
  // S A x (the row scale is all ones outside the flexible GMRES)
  y[5 * (size_t)c + i] = value(z ? acc : acc * X64(im.rs[i]));
}

// z = D^-1 S^-1 v, the block-Jacobi preconditioner of the flexible GMRES on its row-scaled
// system (S D)^-1: FP64 (v, dinv, z) or FP32 (v or v32, dinv32, z32)
__global__ void __launch_bounds__(128) k_imp_precond(DevMesh m, ImpState im, const double* __restrict__ v,
                                                      const float* __restrict__ v32, double* __restrict__ z,
                                                      float* __restrict__ z32) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  if (z) {
    double A[25], vv[5], t[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) vv[k] = v[5 * (size_t)c + k] * im.rsi[k];
    load_block(im.dinv + (size_t)c * kBlk, A);
    mv5(A, vv, t);
#pragma unroll
    for (int k = 0; k < 5; ++k) z[5 * (size_t)c + k] = t[k];
  } else {
    float A[28], vf[5];
    load_block32(im.dinv32 + (size_t)c * kBlk32, A);
#pragma unroll
    for (int k = 0; k < 5; ++k)
      vf[k] = v32 ? v32[5 * (size_t)c + k] * (float)im.rsi[k] : (float)(v[5 * (size_t)c + k] * im.rsi[k]);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 5; ++j) s = fmaf(A[i * 5 + j], vf[j], s);
      z32[5 * (size_t)c + i] = s;
    }
  }
}

// initial guess of bdlu_gmres.f90:77-82: x = b / diag(i, i)
__global__ void __launch_bounds__(kBlock) k_imp_x0(DevMesh m, ImpState im, const double* __restrict__ b,
                                                    double* __restrict__ x) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
#pragma unroll
  for (int k = 0; k < 5; ++k) x[5 * (size_t)c + k] = b[5 * (size_t)c + k] / im.diag[(size_t)c * kBlk + k * 6];
}

// ---- deterministic reductions: fixed grid, block tree, then one block over the partials ----
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[kRedThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  v = threadIdx.x < kRedThreads / 32 ? sh[threadIdx.x] : 0.0;
  if (wid == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;  // valid in thread 0
}

inline unsigned red_grid(size_t n) {
  size_t g = (n + (size_t)kRedThreads * 4 - 1) / ((size_t)kRedThreads * 4);
  if (g < 1) g = 1;
  if (g > (size_t)kRedBlocks) g = kRedBlocks;
  return (unsigned)g;
}

// kind 0: sum a*b, kind 1: sum |a|
__global__ void __launch_bounds__(kRedThreads) k_red_part(const double* __restrict__ a, const double* __restrict__ b,
                                                           size_t n, int kind, double* __restrict__ part) {
  double s = 0.0;
  for (size_t i = blockIdx.x * (size_t)kRedThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kRedThreads)
    s += kind == 0 ? a[i] * b[i] : fabs(a[i]);
  s = block_sum(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// out[k] = sum of part[k * stride + 0 .. nb-1], one block per k
__global__ void __launch_bounds__(kRedThreads) k_red_final(const double* __restrict__ part, int nb, size_t stride,
                                                            double* __restrict__ out) {
  const double* p = part + blockIdx.x * stride;
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += kRedThreads) s += p[i];
  s = block_sum(s);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// ---- BiCGSTAB of bdlu_bicgstab.f90:52-75, scalars kept on the device: sc[0] rho1, sc[1] rho0,
// sc[2] alpha, sc[3] omega (of the previous iteration), sc[4] r2.v, sc[5] t.s, sc[6] t.t,
// sc[7] err.  Each kernel derives the step's alpha, beta, omega from them itself.
// p = r1 (first iteration) or r1 + beta (p - omega v), beta = (rho1/rho0)(alpha/omega)
__global__ void k_bicg_p(const double* __restrict__ r1, const double* __restrict__ v, double* __restrict__ p,
                         const double* __restrict__ sc, int first, size_t n) {
  const double beta = first ? 0.0 : (sc[0] / sc[1]) * (sc[2] / sc[3]);
  const double om = sc[3];
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (first) p[i] = r1[i];
    else {
      const double q = p[i] - om * v[i];
      p[i] = r1[i] + beta * q;
    }
  }
}
// s = r1 - alpha v, alpha = rho1 / (r2.v)
__global__ void k_bicg_s(const double* __restrict__ r1, const double* __restrict__ v, double* __restrict__ s,
                         const double* __restrict__ sc, size_t n) {
  const double alpha = sc[0] / sc[4];
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    s[i] = r1[i] - alpha * v[i];
}
// partial sums of t.s and t.t
__global__ void __launch_bounds__(kRedThreads) k_bicg_ts(const double* __restrict__ t, const double* __restrict__ s,
                                                          size_t n, double* __restrict__ part) {
  double a = 0.0, b = 0.0;
  for (size_t i = blockIdx.x * (size_t)kRedThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kRedThreads) {
    a += t[i] * s[i];
    b += t[i] * t[i];
  }
  a = block_sum(a);
  b = block_sum(b);
  if (threadIdx.x == 0) { part[blockIdx.x] = a; part[kRedBlocks + blockIdx.x] = b; }
}
// omega = (t.s)/(t.t); err partials of |alpha p + omega s|; x += alpha p + omega s; r1 = s - omega t
__global__ void __launch_bounds__(kRedThreads) k_bicg_update(double* __restrict__ x, double* __restrict__ r1,
                                                              const double* __restrict__ p,
                                                              const double* __restrict__ s,
                                                              const double* __restrict__ t,
                                                              const double* __restrict__ sc, size_t n,
                                                              double* __restrict__ part) {
  const double alpha = sc[0] / sc[4], omega = sc[5] / sc[6];
  double e = 0.0;
  for (size_t i = blockIdx.x * (size_t)kRedThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kRedThreads) {
    const double ap = alpha * p[i], os = omega * s[i];
    e += fabs(ap + os);
    x[i] = x[i] + ap + os;
    r1[i] = s[i] - omega * t[i];
  }
  e = block_sum(e);
  if (threadIdx.x == 0) part[blockIdx.x] = e;
}
// end of an iteration: rho0 = rho1, alpha and omega kept for the next beta
__global__ void k_bicg_shift(double* sc) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    const double alpha = sc[0] / sc[4], omega = sc[5] / sc[6];
    sc[1] = sc[0];
    sc[2] = alpha;
    sc[3] = omega;
  }
}

// ---- modified Gram-Schmidt of one Krylov vector in one cooperative launch ----
// bdlu_gmres.f90:100-118 takes h_i = w . v_i, w -= h_i v_i one vector after the other: jk + 1
// dependent reductions.  The same h solves (I + L) h = V^T w with L_ij = v_i . v_j (j < i), so the
// kernel measures V^T w at once, solves the triangle, subtracts V h in the order of i, and
// measures V^T w and w . w again for the next row of L and h_{jk+1} (the low-synchronisation
// form of modified Gram-Schmidt of Swirydowicz, Langou, Ananthan, Yang and Thomas, Numer. Linear
// Algebra Appl. 28, 2021: two reductions a vector, the same loss of orthogonality).
// The grid is resident and every thread keeps its K entries of w in registers (K = 0: in
// memory).  No barrier: a block publishes its sums in slots of its own (prefilled by the column
// before with a NaN pattern that no arithmetic produces) and every block reads all slots, waiting (bounded) for
// those still empty, five polls in flight per lane; nothing else travels between blocks.  GB300, 122,825 unknowns, restart 30, us a
// vector on average: 142 in 2 (jk + 1) launches, 105 with the reductions one after the other in one
// launch, 35 so (60 with 128 threads a block, 37 with 512), 33 with several polls in flight.  The memset before and the copy after each
// launch cost 8 us a vector more: the column before empties the slots (a later column has as many
// blocks or fewer), and the sums go to pinned memory.
constexpr int kMgsThreads = 256;
constexpr unsigned long long kMgsEmpty = ~0ull;
constexpr int kMgsSpins = 1 << 22;

template <int K>
__global__ void __launch_bounds__(kMgsThreads) k_mgs_column(double* w, double* V, size_t n, int jk, double* L,
                                                            double* slots, double* next, double* out, unsigned* err) {
  constexpr int KR = K > 0 ? K : 1, kWarps = kMgsThreads / 32;
  extern __shared__ double acc[];  // [jk + 1][kMgsThreads] per-thread sums
  __shared__ double h[kMaxKrylov + 1];
  __shared__ volatile int late;  // a wait of this block ran out (about three seconds): its others end too
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, g = gridDim.x;
  const size_t first = blockIdx.x * (size_t)kMgsThreads + t, stride = g * (size_t)kMgsThreads;
  double W[KR];
  if (t == 0) late = 0;
  // this block's slots of the next column's exchanges (read by nobody until the next launch)
  if (jk < kMaxKrylov)
    for (int i = t; i < 2 * jk + 3; i += kMgsThreads)
      reinterpret_cast<unsigned long long*>(next)[(size_t)i * g + blockIdx.x] = kMgsEmpty;
  if constexpr (K > 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) W[k] = first + k * stride < n ? w[first + k * stride] : 0.0;
  }
  // this thread's products of w with the vectors 0 .. jk-1 (and with itself) into acc
  auto products = [&](bool self) {
    for (int i = 0; i < jk; i += 4) {
      double s[4] = {0.0, 0.0, 0.0, 0.0};
      const double* v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = V + (size_t)min(i + q, jk - 1) * n;
      if constexpr (K > 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (i + q < jk) {
#pragma unroll
            for (int k = 0; k < K; ++k)
              s[q] = fma(W[k], first + k * stride < n ? v[q][first + k * stride] : 0.0, s[q]);
          }
        }
      } else {
        for (size_t k = first; k < n; k += stride) {
          const double wk = w[k];
#pragma unroll
          for (int q = 0; q < 4; ++q) s[q] = fma(wk, v[q][k], s[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + q < jk) acc[(i + q) * kMgsThreads + t] = s[q];
    }
    if (self) {
      double s = 0.0;
      if constexpr (K > 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) s = fma(W[k], W[k], s);
      } else {
        for (size_t k = first; k < n; k += stride) s = fma(w[k], w[k], s);
      }
      acc[jk * kMgsThreads + t] = s;
    }
    __syncthreads();
  };
  // the grid's sums of acc rows 0 .. count-1 into h; every block adds the blocks' sums in block
  // order.  False after the limit.
  auto exchange = [&](int count, double* sl) -> bool {
    for (int i = wid; i < count; i += kWarps) {
      const double* a = acc + i * kMgsThreads;
      double s = a[lane];
#pragma unroll
      for (int j = 32; j < kMgsThreads; j += 32) s += a[lane + j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) {
        unsigned long long b = (unsigned long long)__double_as_longlong(s);
        if (b == kMgsEmpty) b = 0x7fffffffffffffffull;
        asm volatile("st.relaxed.gpu.u64 [%0], %1;" ::"l"(sl + (size_t)i * g + blockIdx.x), "l"(b) : "memory");
      }
    }
    for (int i = wid; i < count; i += kWarps) {
      double s = 0.0;
      auto poll = [&](int q) {
        unsigned long long b;
        asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(b) : "l"(sl + (size_t)i * g + q) : "memory");
        return b;
      };
      constexpr int kBatch = 5;  // polls in flight per lane: 160 blocks
      for (int q = lane; q < g; q += 32 * kBatch) {
        unsigned long long b[kBatch];
#pragma unroll
        for (int d = 0; d < kBatch; ++d) b[d] = q + 32 * d < g ? poll(q + 32 * d) : 0ull;
#pragma unroll
        for (int d = 0; d < kBatch; ++d) {
          if (q + 32 * d >= g) break;
          for (int spins = 0; b[d] == kMgsEmpty && spins < kMgsSpins && !late; ++spins) b[d] = poll(q + 32 * d);
          if (b[d] == kMgsEmpty) late = 1;
          s += __longlong_as_double((long long)b[d]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) h[i] = s;
    }
    __syncthreads();
    return late == 0;  // set at most once: nothing resets it
  };
  products(false);
  if (!exchange(jk, slots)) {
    if (t == 0) *err = 1u;
    return;
  }
  if (wid == 0) {  // (I + L) h = V^T w, by columns; two entries per lane
    double d0 = lane < jk ? h[lane] : 0.0, d1 = lane + 32 < jk ? h[lane + 32] : 0.0;
    for (int i = 0; i < jk; ++i) {
      const double hi = __shfl_sync(0xffffffffu, i < 32 ? d0 : d1, i & 31);
      if (lane > i && lane < jk) d0 = fma(-__ldcg(L + lane * kMaxKrylov + i), hi, d0);
      if (lane + 32 > i && lane + 32 < jk) d1 = fma(-__ldcg(L + (lane + 32) * kMaxKrylov + i), hi, d1);
    }
    __syncwarp();
    if (lane < jk) h[lane] = d0;
    if (lane + 32 < jk) h[lane + 32] = d1;
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int i = t; i < jk; i += kMgsThreads) out[i] = h[i];
  if constexpr (K > 0) {
#pragma unroll 4
    for (int i = 0; i < jk; ++i) {
      const double c = -h[i];
      const double* v = V + (size_t)i * n + first;
#pragma unroll
      for (int k = 0; k < K; ++k) W[k] = fma(c, first + k * stride < n ? v[k * stride] : 0.0, W[k]);
    }
  } else {
    for (size_t k = first; k < n; k += stride) {
      double x = w[k];
#pragma unroll 4
      for (int i = 0; i < jk; ++i) x = fma(-h[i], V[(size_t)i * n + k], x);
      w[k] = x;
    }
  }
  __syncthreads();  // h is read before the second exchange writes it
  products(true);
  if (!exchange(jk + 1, slots + (size_t)jk * g)) {
    if (t == 0) *err = 1u;
    return;
  }
  const double f = 1.0 / sqrt(h[jk]);
  if (blockIdx.x == 0) {
    for (int i = t; i < jk; i += kMgsThreads) L[jk * kMaxKrylov + i] = h[i] * f;
    if (t == 0) out[jk] = h[jk];
  }
  double* vn = V + (size_t)jk * n;
  if constexpr (K > 0) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (first + k * stride < n) vn[first + k * stride] = f * W[k];
  } else {
    for (size_t k = first; k < n; k += stride) vn[k] = f * w[k];
  }
}

// Krylov basis pass of the flexible GMRES (basis vector i at V + i ldv):
//   project: out_i = V_i . src (i < nv), out_nv = src . src
//   extend:  v = (src - sum_{i<nv} c_i V_i) s is stored as V_nv (rounded to the basis' type), then
//            out_i = V_i . v (i < nv), out_nv = v . v, of the stored values
// An FP64 basis is swept in FP64; an FP32 basis (mixed-precision solve) in FP32 arithmetic with
// FP64 block sums.  The first form projects A z_j on the basis; the second forms the next basis
// vector and the new column of the basis' Gram matrix in the same sweep, so one iteration reads
// the basis twice and synchronises with the host once.  Each block reduces its sums once, writes
// one partial per output, and the last block to finish adds the partials in block order: one
// launch, the same result for the same grid.

// The end of a sweep: acc [nout][T] per-thread sums -> one partial per output and block -> out.
template <int T>
__device__ __forceinline__ void finish_sums(const double* acc, int nout, double* __restrict__ part,
                                            unsigned* __restrict__ done, double* __restrict__ out) {
  __shared__ bool last;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for (int i = wid; wid < T / 32 && i < nout; i += T / 32) {
    double x = 0.0;
#pragma unroll
    for (int q = 0; q < T / 32; ++q) x += acc[(size_t)i * T + q * 32 + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) part[(size_t)i * kRedBlocks + blockIdx.x] = x;
  }
  __threadfence();
  __syncthreads();
  if (t == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = wid; wid < T / 32 && i < nout; i += T / 32) {
    const double* p = part + (size_t)i * kRedBlocks;
    double x = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32) x += __ldcg(p + b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) out[i] = x;
  }
  if (t == 0) *done = 0u;  // ready for the next launch on the stream
}

// ---- bulk copies into shared memory (TMA) with their completion barrier ----
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(b))
               : "memory");
}
// waits for the phase of the given parity; false after the limit, about two seconds
constexpr long long kWaitClocks = 4000000000ll;
__device__ __forceinline__ bool mbar_try(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile("{.reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
               : "=r"(ok)
               : "r"(smem_addr(b)), "r"(parity)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity) {
  if (mbar_try(b, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try(b, parity))
    if (clock64() - t0 > kWaitClocks) return false;
  return true;
}

// The FP64 sweep.  Bound by the FP64 pipe (nv + 1 multiply-adds a row, 2 nv + 2 when it extends):
// compiled per form and per even J >= nv (predicated-off slots occupy the pipe), one block per SM whose
// tiles of T rows of the nv + 1 vectors are brought to shared memory by a last warp's bulk copies
// several tiles ahead, so that neither registers nor occupancy limit the loads in flight.  T: 15 warps
// compute up to J = 16, so that with the producer every SM quarter has four (a row's sum of nv
// dependent multiply-adds leaves two warps a quarter short of the pipe; 16 + 1 warps leave 96 registers
// a thread, too few at J = 14 and 16); 8 beyond, whose rows take more shared memory.
// One block per SM also because a block's reduction costs (nv + 1) (T/32 + 5) additions and the last
// block adds a partial per block: 15 us of a 66 us sweep when eight blocks per SM did.  The vectors are
// padded to 16 bytes (ldv a multiple of 2, src at least ldv long).  GB300, us, project on 15 / extend
// from 14 vectors:
//   rows                  200,000   1,250,000   5,000,000
//   loads to registers    21 / 27    56 / 81    159 / 263
//   8 computing warps     16 / 21    52 / 78    174 / 278
//   15                    17 / 20    49 / 76    152 / 261
// 24 vectors of 1,412,500 rows 121 / 317 (the compiler spread the loads out) -> 79 / 146.
template <int J>
constexpr int kSweepThreads = J <= 16 ? 480 : 256;
template <int J>
constexpr int kSweepStages = std::min(8, 212000 / ((J + 1) * kSweepThreads<J> * (int)sizeof(double)));

template <int J, bool EXTEND>
__global__ void __launch_bounds__(kSweepThreads<J> + 32) k_basis_pass(double* V, size_t ldv, int nv,
                                                               const double* __restrict__ c,
                                                               const double* __restrict__ src,
                                                               const double* __restrict__ sp, size_t n,
                                                               double* __restrict__ part, unsigned* __restrict__ done,
                                                               double* __restrict__ out, unsigned* err) {
  constexpr int T = kSweepThreads<J>, S = kSweepStages<J>;
  extern __shared__ __align__(16) double buf[];  // [S][J + 1][T]: the vectors 0 .. nv-1, then src
  __shared__ __align__(8) unsigned long long full[S], empty[S];
  __shared__ double cl[J];
  const int t = threadIdx.x;
  if (EXTEND && t < J) cl[t] = t < nv ? -c[t] : 0.0;
  const double sc = EXTEND ? *sp : 1.0;
  const int tiles = (int)((n + T - 1) / T), mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  auto load = [&](int i) {  // this block's tile i into its stage (one thread)
    const size_t k0 = (size_t)(blockIdx.x + i * gridDim.x) * T;
    const unsigned bytes = (unsigned)(min((size_t)T, ldv - k0) * sizeof(double));
    double* d = buf + (size_t)(i % S) * (J + 1) * T;
    unsigned long long* b = &full[i % S];
    mbar_expect(b, bytes * (nv + 1));
    for (int v = 0; v < nv; ++v) bulk_load(d + v * T, V + v * ldv + k0, bytes, b);
    bulk_load(d + J * T, src + k0, bytes, b);
  };
  if (t == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], T / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (nv < J && t < T) {  // the padding slot of an odd nv
    for (int i = 0; i < S; ++i) buf[(size_t)i * (J + 1) * T + nv * T + t] = 0.0;
    if (nv + 1 < J)
      for (int i = 0; i < S; ++i) buf[(size_t)i * (J + 1) * T + (nv + 1) * T + t] = 0.0;
  }
  __syncthreads();
  bool ok = true;
  int issued = 0;
  if (t == T)  // the producer: one thread of the last warp
    for (; issued < mine; ++issued) {
      if (issued >= S && !mbar_wait(&empty[issued % S], (issued / S - 1) & 1)) {
        ok = false;
        break;
      }
      load(issued);
    }
  double* vout = V + (size_t)nv * ldv;
  double ad[J], cr[EXTEND && J <= 20 ? J : 1], xx = 0.0;
#pragma unroll
  for (int i = 0; i < J; ++i) {
    ad[i] = 0.0;
    if (EXTEND && J <= 20) cr[i] = cl[i];
  }
  for (int i = 0; i < (t < T ? mine : 0); ++i) {
    const int st = i % S;
    if (!__all_sync(0xffffffffu, mbar_wait(&full[st], (i / S) & 1))) {
      ok = false;
      break;
    }
    const double* d = buf + (size_t)st * (J + 1) * T + t;
    const size_t k = (size_t)(blockIdx.x + i * gridDim.x) * T + t;
    if (k < n) {
      double x = d[J * T], b[J];
#pragma unroll
      for (int v = 0; v < J; ++v) b[v] = d[v * T];
      if constexpr (EXTEND) {
#pragma unroll
        for (int v = 0; v < J; ++v) x = fma(J <= 20 ? cr[v] : cl[v], b[v], x);
        x = x * sc;
        vout[k] = x;
      }
#pragma unroll
      for (int v = 0; v < J; ++v) ad[v] = fma(b[v], x, ad[v]);
      xx = fma(x, x, xx);
    }
    __syncwarp();
    if ((t & 31) == 0) mbar_arrive(&empty[st]);
  }
  // every copy has been waited for: the stages become the per-thread sums
  if (__syncthreads_or(!ok)) {  // or a wait ran out: the copies still on their way first
    if (t == T)
      for (int i = issued > S ? issued - S : 0; i < issued; ++i) mbar_wait(&full[i % S], (i / S) & 1);
    if (t == 0) *err = 1u;
    __syncthreads();
  }
  if (t < T) {
#pragma unroll
    for (int i = 0; i < J; ++i) buf[i * T + t] = ad[i];
    buf[nv * T + t] = xx;
  }
  __syncthreads();
  finish_sums<T>(buf, nv + 1, part, done, out);
}

template <int J>
__global__ void __launch_bounds__(kCgsThreads) k_basis_pass32(float* V, size_t ldv, int nv, const double* __restrict__ c,
                                                             const double* __restrict__ src,
                                                             const double* __restrict__ sp, int extend, size_t n,
                                                             double* __restrict__ part, unsigned* __restrict__ done,
                                                             double* __restrict__ out) {
  __shared__ double cl[J];
  __shared__ double acc[J + 1][kCgsThreads];
  const int t = threadIdx.x;
  if (t < J) cl[t] = (extend && t < nv) ? c[t] : 0.0;
#pragma unroll
  for (int i = 0; i <= J; ++i) acc[i][t] = 0.0;
  const double sc = extend ? *sp : 1.0;
  __syncthreads();
  float* vout = V + (size_t)nv * ldv;
  {
    // FP32 basis: FP32 arithmetic per row (GB300 issues FP32 at about 60x its FP64 rate),
    // per-thread sums in FP32 registers over the thread's rows, FP64 from the block sums on
    float cf[J], af[J];
#pragma unroll
    for (int i = 0; i < J; ++i) {
      cf[i] = (float)cl[i];
      af[i] = 0.f;
    }
    const float sf = (float)sc;
    float xx = 0.f;
    // R rows per trip (R x nv independent 4-byte loads in flight) for the short bases
    constexpr int R = J <= 8 ? 4 : (J <= 16 ? 2 : 1);
    const size_t stride = (size_t)gridDim.x * kCgsThreads;
    for (size_t k0 = blockIdx.x * (size_t)kCgsThreads + t; k0 < n; k0 += R * stride) {
      float v[R][J], x[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const size_t k = k0 + r * stride;
        const bool ok = k < n;
        const float* pv = V + k;
#pragma unroll
        for (int i = 0; i < J; ++i) {
          v[r][i] = (ok && i < nv) ? *pv : 0.f;
          pv += ldv;
        }
        x[r] = ok ? (float)src[k] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (extend) {
#pragma unroll
          for (int i = 0; i < J; ++i)
            if (i < nv) x[r] = fmaf(-cf[i], v[r][i], x[r]);
          x[r] = x[r] * sf;
          if (k0 + r * stride < n) vout[k0 + r * stride] = x[r];
        }
#pragma unroll
        for (int i = 0; i < J; ++i)
          if (i < nv) af[i] = fmaf(v[r][i], x[r], af[i]);
        xx = fmaf(x[r], x[r], xx);
      }
    }
#pragma unroll
    for (int i = 0; i < J; ++i)
      if (i < nv) acc[i][t] = (double)af[i];
    acc[nv][t] = (double)xx;
  }
  __syncthreads();
  finish_sums<kCgsThreads>(&acc[0][0], nv + 1, part, done, out);
}

__global__ void k_scale(const double* __restrict__ w, double s, double* __restrict__ v, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    v[i] = s * w[i];
}

// x = x + y_j V_j over j (descending order when asked, as bdlu_gmres.f90:176-187 does)
__global__ void k_axpy_multi(double* __restrict__ x, const double* __restrict__ V, const float* __restrict__ V32,
                             size_t ldv, int j, const double* __restrict__ y, int descending, size_t n) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    double xk = x[k];
    for (int q = 0; q < j; ++q) {
      const int i = descending ? j - 1 - q : q;
      const double vi = V ? V[i * ldv + k] : (double)V32[i * ldv + k];
      xk = xk + y[i] * vi;
    }
    x[k] = xk;
  }
}

// U += x (update_field.f90:38) on the resident state; partial sums of |x| per variable
__global__ void __launch_bounds__(kRedThreads) k_imp_update(DevMesh m, double* __restrict__ u0,
                                                             const double* __restrict__ x, double* __restrict__ part) {
  double s[6] = {0, 0, 0, 0, 0, 0};
  for (int c = blockIdx.x * kRedThreads + threadIdx.x; c < m.nci; c += gridDim.x * kRedThreads) {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double d = x[5 * (size_t)c + v];
      u0[v * (size_t)m.ldc + c] = u0[v * (size_t)m.ldc + c] + d;
      s[v] += fabs(d);
    }
    const double mx = x[5 * (size_t)c + 2], my = x[5 * (size_t)c + 3], mz = x[5 * (size_t)c + 4];
    s[5] += sqrt(mx * mx + my * my + mz * mz);
  }
#pragma unroll
  for (int v = 0; v < 6; ++v) {
    double t = block_sum(s[v]);
    if (threadIdx.x == 0) part[(size_t)v * kRedBlocks + blockIdx.x] = t;
  }
}

// unscaled residual norms per variable: sum (b_c V_c / dt_c)^2
__global__ void __launch_bounds__(kRedThreads) k_imp_resnorm(DevMesh m, ImpState im, ImpArgs a,
                                                              const double* __restrict__ b, double* __restrict__ part) {
  double s[5] = {0, 0, 0, 0, 0};
  for (int c = blockIdx.x * kRedThreads + threadIdx.x; c < m.nci; c += gridDim.x * kRedThreads) {
    const double k = m.cvol[c] / imp_dt(im, a, c);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double r = b[5 * (size_t)c + v] * k;
      s[v] += r * r;
    }
  }
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    double t = block_sum(s[v]);
    if (threadIdx.x == 0) part[(size_t)v * kRedBlocks + blockIdx.x] = t;
  }
}

// Jacobian-free products: the perturbed state U + eps z (SoA), then w = z - (R(U + eps z) - R(U)) / eps
__global__ void k_imp_perturb(DevMesh m, const double* __restrict__ u0, const double* __restrict__ z, double eps,
                              double* __restrict__ up) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
#pragma unroll
  for (int v = 0; v < 5; ++v) up[v * (size_t)m.ldc + c] = u0[v * (size_t)m.ldc + c] + eps * z[5 * (size_t)c + v];
}
// w = rs (z - (rp - r0) inv_eps) per packed entry (rs of its variable i mod 5); rp null: w = rs z
__global__ void k_imp_fd(const double* __restrict__ z, const float* __restrict__ z32, const double* __restrict__ rp,
                         const double* __restrict__ r0, double inv_eps, Row5 rs, double* __restrict__ w, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double zi = z ? z[i] : (double)z32[i];
    const double d = rp ? zi - (rp[i] - (r0 ? r0[i] : 0.0)) * inv_eps : zi;
    w[i] = d * rs.v[i % 5];
  }
}

// ---------------------------------------------------------------------------
// launchers
inline unsigned grid_of(size_t n, int b) { return (unsigned)((n + b - 1) / b); }

cudaError_t imp_dtloc(const DevMesh& m, const DevState& s, const SpatOpts& o, const ImpState& im, double cfl,
                      unsigned long long* dtbits, cudaStream_t st) {
  k_imp_dtloc<<<nblk(m.nci), kBlock, 0, st>>>(m, s.u0, o.gamma, cfl, im.dtloc, dtbits, s.err);
  return cudaGetLastError();
}

cudaError_t imp_assemble(const DevMesh& m, const DevState& s, const SpatOpts& o, const ImpState& im,
                         const ImpArgs& a, cudaStream_t st, Prof* pr) {
  pr->launch(K_IMP_FACE, st, [&] { k_imp_face<<<grid_of(m.nf, 128), 128, 0, st>>>(m, s, o, im, a); });
  pr->launch(K_IMP_DIAG, st, [&] { k_imp_diag<<<grid_of(m.nci, 128), 128, 0, st>>>(m, im, a, 1, s.err); });
  return cudaGetLastError();
}

cudaError_t imp_rhs(const DevMesh& m, const DevState& s, const ImpState& im, const ImpArgs& a, double* out,
                    cudaStream_t st) {
  k_imp_rhs<<<nblk(m.nci), kBlock, 0, st>>>(m, s, im, a, out);
  return cudaGetLastError();
}

template <bool F32>
void mv_staged(const DevMesh& m, const ImpState& im, const void* x, const double* z, double* y, cudaStream_t st) {
  constexpr int bytes = kMvThreads / 32 * 2 * 32 * (F32 ? 7 : 13) * 16;
  cudaFuncSetAttribute(k_imp_matvec<F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  k_imp_matvec<F32><<<grid_of(m.nci, kMvThreads), kMvThreads, bytes, st>>>(m, im, x, z, y);
}

// FP64: a row per thread in the exact mode, whose longer chains it shortens at every size, and up to
// 40,000 cells in the fast mode, where above that its narrower loads cost more than its shorter chains
// gain.  GB300, us per product, cell (staged) / row form, tetrahedra:
//   cells     1,080       5,000       13,720      24,565      40,000      69,120      135,000     320,000    1,080,000
//   fast   12.2 /  9.1 12.2 / 10.1 12.3 / 10.6 16.3 / 16.3 20.4 / 20.5 26.8 / 32.7 41.1 / 51.1 83.8 / 110  252 / 346
//   exact  18.3 / 10.1 18.3 / 11.4 18.3 / 14.1 28.6 / 20.4 38.8 / 28.6 49.8 / 43.5 81.2 / 74.3  182 / 167  582 / 539
constexpr int kRowFormCells = 40000;
inline void matvec_launch(const DevMesh& m, const ImpState& im, const double* x, const double* z, double* y,
                          cudaStream_t st) {
  if constexpr (kFast) {
    if (m.nci > kRowFormCells) return mv_staged<false>(m, im, x, z, y, st);
  }
  k_imp_matvec_row<<<grid_of(m.nci, kRowCells), 5 * kRowCells, 0, st>>>(m, im, x, z, y);
}

cudaError_t imp_matvec(const DevMesh& m, const ImpState& im, const double* x, const double* z, double* y,
                       cudaStream_t st, Prof* pr) {
  pr->launch(K_IMP_MATVEC, st, [&] { matvec_launch(m, im, x, z, y, st); });
  return cudaGetLastError();
}

cudaError_t imp_matvec32(const DevMesh& m, const ImpState& im, const float* z, double* y, cudaStream_t st,
                         Prof* pr) {
  pr->launch(K_IMP_MATVEC, st, [&] { mv_staged<true>(m, im, z, nullptr, y, st); });
  return cudaGetLastError();
}

cudaError_t imp_precond(const DevMesh& m, const ImpState& im, const double* v, const float* v32, double* z,
                        float* z32, cudaStream_t st, Prof* pr) {
  pr->launch(K_IMP_PRECOND, st,
             [&] { k_imp_precond<<<grid_of(m.nci, 128), 128, 0, st>>>(m, im, v, v32, z, z32); });
  return cudaGetLastError();
}

cudaError_t imp_x0_diag(const DevMesh& m, const ImpState& im, const double* b, double* x, cudaStream_t st) {
  k_imp_x0<<<nblk(m.nci), kBlock, 0, st>>>(m, im, b, x);
  return cudaGetLastError();
}

cudaError_t imp_dot(const double* a, const double* b, size_t n, double* part, double* out, cudaStream_t st) {
  const unsigned g = red_grid(n);
  k_red_part<<<g, kRedThreads, 0, st>>>(a, b, n, 0, part);
  k_red_final<<<1, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, out);
  return cudaGetLastError();
}

// update_field.f90:45-60's residual terms of an explicit step: per block the sums over its
// interior cells of |acc_rho|, |acc_rhoE| and |acc_m| (acc: the step's combination of stage
// residuals, [5][ld])
__global__ void __launch_bounds__(kRedThreads) k_res_l1(int nci, const double* __restrict__ acc, size_t ld,
                                                         double* __restrict__ part) {
  double a = 0.0, b = 0.0, q = 0.0;
  for (int c = blockIdx.x * kRedThreads + threadIdx.x; c < nci; c += gridDim.x * kRedThreads) {
    a += fabs(acc[c]);
    b += fabs(acc[ld + c]);
    const double mx = acc[2 * ld + c], my = acc[3 * ld + c], mz = acc[4 * ld + c];
    q += sqrt(mx * mx + my * my + mz * mz);
  }
  a = block_sum(a);
  b = block_sum(b);
  q = block_sum(q);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a;
    part[kRedBlocks + blockIdx.x] = b;
    part[2 * kRedBlocks + blockIdx.x] = q;
  }
}

cudaError_t res_l1(int nci, const double* acc, size_t ld, double* part, double* out, cudaStream_t st) {
  const unsigned g = red_grid((size_t)nci);
  k_res_l1<<<g, kRedThreads, 0, st>>>(nci, acc, ld, part);
  k_red_final<<<3, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, out);
  return cudaGetLastError();
}

cudaError_t imp_asum(const double* a, size_t n, double* part, double* out, cudaStream_t st) {
  const unsigned g = red_grid(n);
  k_red_part<<<g, kRedThreads, 0, st>>>(a, nullptr, n, 1, part);
  k_red_final<<<1, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, out);
  return cudaGetLastError();
}

template <int K>
cudaError_t mgs_launch(double* w, double* V, size_t n, int jk, double* L, double* part, double* out, unsigned* err,
                       int sms, cudaStream_t st) {
  const size_t lists = (size_t)(jk + 1) * kMgsThreads * sizeof(double);
  // the limit of the longest column, whatever this one needs: the attribute is the function's, and
  // another thread's launch may stand between this call and the launch below
  cudaError_t e = cudaFuncSetAttribute(k_mgs_column<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (kMaxKrylov + 1) * kMgsThreads * (int)sizeof(double));
  if (e != cudaSuccess) return e;
  int blocks = sms;
  if (K > 0) {
    blocks = (int)std::min<size_t>(sms, (n + kMgsThreads * K - 1) / (kMgsThreads * K));
  } else {  // long vectors in memory: as many blocks as are resident, within the slots
    int per = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mgs_column<K>, kMgsThreads, lists);
    if (e != cudaSuccess) return e;
    blocks = std::min(sms * std::max(per, 1), kRedBlocks / 2);
  }
  double *slots = part + (jk & 1 ? 0 : kMgsSlots), *next = part + (jk & 1 ? kMgsSlots : 0);
  if (jk == 1 && (e = cudaMemsetAsync(slots, 0xff, (size_t)3 * blocks * sizeof(double), st)) != cudaSuccess) return e;
  void* args[] = {&w, &V, &n, &jk, &L, &slots, &next, &out, &err};
  return cudaLaunchCooperativeKernel((const void*)k_mgs_column<K>, dim3((unsigned)blocks), dim3(kMgsThreads), args, lists,
                                     st);
}

// One block per SM with the fewest register entries per thread that cover the vector (152 x 256 x
// 16 = 622,592 unknowns on GB300); beyond that w stays in memory.
cudaError_t imp_mgs_column(double* w, double* V, size_t n, int jk, double* L, double* part, double* out, unsigned* err,
                           cudaStream_t st) {
  if (jk < 1 || jk > kMaxKrylov) return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  sms = std::min(sms, kRedBlocks / 2);
  const size_t row = (size_t)sms * kMgsThreads;
  if (n <= row) return mgs_launch<1>(w, V, n, jk, L, part, out, err, sms, st);
  if (n <= 2 * row) return mgs_launch<2>(w, V, n, jk, L, part, out, err, sms, st);
  if (n <= 4 * row) return mgs_launch<4>(w, V, n, jk, L, part, out, err, sms, st);
  if (n <= 8 * row) return mgs_launch<8>(w, V, n, jk, L, part, out, err, sms, st);
  if (n <= 16 * row) return mgs_launch<16>(w, V, n, jk, L, part, out, err, sms, st);
  return mgs_launch<0>(w, V, n, jk, L, part, out, err, sms, st);
}

// Blocks of a sweep: a fixed function of n and the device, so that sums repeat from run to run.
inline unsigned sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (unsigned)std::max(1, std::min(sms, kRedBlocks));
}

template <int J>
cudaError_t basis_launch_j(double* V, size_t ldv, int nv, const double* c, const double* src, const double* sp,
                           int extend, size_t n, double* part, unsigned* done, double* out, unsigned* err,
                           cudaStream_t st) {
  const unsigned g = (unsigned)std::max<size_t>(1, std::min<size_t>((n + kSweepThreads<J> - 1) / kSweepThreads<J>, sm_count()));
  const size_t sums = (size_t)kSweepStages<J> * (J + 1) * kSweepThreads<J> * sizeof(double);
  auto* k = extend ? k_basis_pass<J, true> : k_basis_pass<J, false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sums);
  if (e != cudaSuccess) return e;
  k<<<g, kSweepThreads<J> + 32, sums, st>>>(V, ldv, nv, c, src, sp, n, part, done, out, err);
  return cudaGetLastError();
}

// the smallest even J >= nv
template <int J = 2>
cudaError_t basis_launch(double* V, size_t ldv, int nv, const double* c, const double* src, const double* sp, int extend,
                         size_t n, double* part, unsigned* done, double* out, unsigned* err, cudaStream_t st) {
  if constexpr (J < kMaxCgs) {
    if (nv > J) return basis_launch<J + 2>(V, ldv, nv, c, src, sp, extend, n, part, done, out, err, st);
  }
  return basis_launch_j<J>(V, ldv, nv, c, src, sp, extend, n, part, done, out, err, st);
}

// an FP32 sweep, bound by HBM, takes 8, 16 or 32 slots and every resident block
template <int J>
cudaError_t basis_launch32_j(float* V, size_t ldv, int nv, const double* c, const double* src, const double* sp,
                             int extend, size_t n, double* part, unsigned* done, double* out, cudaStream_t st) {
  static const unsigned cap = [] {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_basis_pass32<J>, kCgsThreads, 0);
    return (unsigned)std::min<long>((long)sm_count() * std::max(per, 1), kRedBlocks);
  }();
  const size_t g = std::max<size_t>(1, std::min<size_t>((n + kCgsThreads - 1) / kCgsThreads, cap));
  k_basis_pass32<J><<<(unsigned)g, kCgsThreads, 0, st>>>(V, ldv, nv, c, src, sp, extend, n, part, done, out);
  return cudaGetLastError();
}
inline cudaError_t basis_launch32(float* V, size_t ldv, int nv, const double* c, const double* src, const double* sp,
                                  int extend, size_t n, double* part, unsigned* done, double* out, cudaStream_t st) {
  if (nv <= 8) return basis_launch32_j<8>(V, ldv, nv, c, src, sp, extend, n, part, done, out, st);
  if (nv <= 16) return basis_launch32_j<16>(V, ldv, nv, c, src, sp, extend, n, part, done, out, st);
  return basis_launch32_j<kMaxCgs>(V, ldv, nv, c, src, sp, extend, n, part, done, out, st);
}

cudaError_t imp_basis_pass(double* V, float* V32, size_t ldv, int nv, const double* c, const double* src,
                           const double* sp, int extend, size_t n, double* part, unsigned* done, double* out,
                           unsigned* err, cudaStream_t st, Prof* pr) {
  if (nv < 0 || nv > kMaxCgs) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  pr->launch(K_IMP_ORTHO, st, [&] {
    e = V32 ? basis_launch32(V32, ldv, nv, c, src, sp, extend, n, part, done, out, st)
            : basis_launch(V, ldv, nv, c, src, sp, extend, n, part, done, out, err, st);
  });
  return e;
}

cudaError_t imp_bicgstab_iter(const DevMesh& m, const ImpState& im, double* x, double* r1, const double* r2,
                              double* p, double* v, double* s, double* t, int first, double* part, double* sc,
                              cudaStream_t st, Prof* pr) {
  const size_t n = 5 * (size_t)m.nci;
  const unsigned gv = (unsigned)std::min<size_t>(grid_of(n, 256), 4 * kRedBlocks);
  const unsigned g = red_grid(n);
  k_red_part<<<g, kRedThreads, 0, st>>>(r1, r2, n, 0, part);                // rho1 = r1.r2
  k_red_final<<<1, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, sc + 0);
  k_bicg_p<<<gv, 256, 0, st>>>(r1, v, p, sc, first, n);
  pr->launch(K_IMP_MATVEC, st, [&] { matvec_launch(m, im, p, nullptr, v, st); });
  k_red_part<<<g, kRedThreads, 0, st>>>(r2, v, n, 0, part);                 // r2.v
  k_red_final<<<1, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, sc + 4);
  k_bicg_s<<<gv, 256, 0, st>>>(r1, v, s, sc, n);
  pr->launch(K_IMP_MATVEC, st, [&] { matvec_launch(m, im, s, nullptr, t, st); });
  k_bicg_ts<<<g, kRedThreads, 0, st>>>(t, s, n, part);
  k_red_final<<<2, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, sc + 5);
  k_bicg_update<<<g, kRedThreads, 0, st>>>(x, r1, p, s, t, sc, n, part);
  k_red_final<<<1, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, sc + 7);
  k_bicg_shift<<<1, 32, 0, st>>>(sc);
  return cudaGetLastError();
}

cudaError_t imp_scale(const double* w, double s, double* v, size_t n, cudaStream_t st) {
  k_scale<<<std::min<size_t>(grid_of(n, 256), 4 * kRedBlocks), 256, 0, st>>>(w, s, v, n);
  return cudaGetLastError();
}

cudaError_t imp_axpy_multi(double* x, const double* V, const float* V32, size_t ldv, int j, const double* y,
                           int descending, size_t n, cudaStream_t st) {
  k_axpy_multi<<<std::min<size_t>(grid_of(n, 256), 4 * kRedBlocks), 256, 0, st>>>(x, V, V32, ldv, j, y,
                                                                                 descending, n);
  return cudaGetLastError();
}

cudaError_t imp_update_state(const DevMesh& m, DevState& s, const double* x, double* part, double* out,
                             cudaStream_t st) {
  const unsigned g = red_grid(m.nci);
  k_imp_update<<<g, kRedThreads, 0, st>>>(m, s.u0, x, part);
  k_red_final<<<6, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, out);
  return cudaGetLastError();
}

cudaError_t imp_perturb(const DevMesh& m, const double* u0, const double* z, double eps, double* up,
                        cudaStream_t st) {
  k_imp_perturb<<<nblk(m.nci), kBlock, 0, st>>>(m, u0, z, eps, up);
  return cudaGetLastError();
}

cudaError_t imp_fd_combine(const double* z, const float* z32, const double* rp, const double* r0, double inv_eps,
                           Row5 rs, double* w, size_t n, cudaStream_t st) {
  k_imp_fd<<<std::min<size_t>(grid_of(n, 256), 4 * kRedBlocks), 256, 0, st>>>(z, z32, rp, r0, inv_eps, rs, w, n);
  return cudaGetLastError();
}

__global__ void k_to_f32(const double* __restrict__ x, float* __restrict__ y, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = (float)x[i];
}
cudaError_t imp_to_f32(const double* x, float* y, size_t n, cudaStream_t st) {
  k_to_f32<<<std::min<size_t>(grid_of(n, 256), 4 * kRedBlocks), 256, 0, st>>>(x, y, n);
  return cudaGetLastError();
}

cudaError_t imp_res_norms(const DevMesh& m, const ImpState& im, const ImpArgs& a, const double* b, double* part,
                          double* out, cudaStream_t st) {
  const unsigned g = red_grid(m.nci);
  k_imp_resnorm<<<g, kRedThreads, 0, st>>>(m, im, a, b, part);
  k_red_final<<<5, kRedThreads, 0, st>>>(part, (int)g, kRedBlocks, out);
  return cudaGetLastError();
}

}  // namespace TY_KNS
}  // namespace tyk
