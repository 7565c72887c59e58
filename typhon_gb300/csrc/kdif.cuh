// Heat-conduction (KDIF) kernels, instantiated once per arithmetic mode after kernels.cuh.
//
// Face flux per unit surface (calc_kdif_flux.f90:106-137, theta = 1) with the face
// conductivity of the two cells, then times S; imposed-flux walls replace it
// (kdif_bocoflux.f90) and have no Jacobian.  The residual gathers the face fluxes in
// colour order (flux_to_res.f90); the diagonal of the symmetrised implicit matrix
// diag(V/dt) A is V/dt - sum_f J_R S over the cell's faces in ascending face order, its
// off-diagonal J_R S, as the oracle assembles them.  Conjugate gradients keep their scalars
// on the device: the FP64 solve runs in launches of up to 1,000 iterations of one cooperative kernel.
#pragma once
#include "implicit.hpp"
#include "kdif.hpp"

namespace tyk {
namespace TY_KNS {

__global__ void __launch_bounds__(kBlock) k_kdif_ghost(DevMesh m, KdifState k) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= m.ng) return;
  const int f = m.gface[g];
  k.T[m.nci + g] = k.fkind[f] == TY_KBC_ISOTHERMAL ? k.fval[f] : k.T[m.gsrc[g]];
}

// least-squares gradient of T (the 5-variable k_grad restricted to one scalar)
__global__ void __launch_bounds__(kBlock) k_kdif_grad(DevMesh m, KdifState k) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  double b0 = 0.0, b1 = 0.0, b2 = 0.0;
  for (int sl = 0; sl < m.nslot; ++sl) {
    const int e = m.cf[sl * (size_t)m.nci + c];
    if (e < 0) break;
    const int f = e >> 1;
    const double dsca = k.T[m.fc2[f]] - k.T[m.fc1[f]];
    if constexpr (kFast) {
      const int side = e & 1;
      b0 = fma(dsca, d3(m.lsqw, m.ldf, f, 3 * side), b0);
      b1 = fma(dsca, d3(m.lsqw, m.ldf, f, 3 * side + 1), b1);
      b2 = fma(dsca, d3(m.lsqw, m.ldf, f, 3 * side + 2), b2);
    } else {
      b0 = b0 + dsca * d3(m.dcg, m.ldf, f, 0);
      b1 = b1 + dsca * d3(m.dcg, m.ldf, f, 1);
      b2 = b2 + dsca * d3(m.dcg, m.ldf, f, 2);
    }
  }
  if constexpr (!kFast) {  // cholesky_solve (MATRIX.f90:79-111)
    const size_t n = m.nci;
    const double L11 = m.lsq[c], L21 = m.lsq[n + c], L31 = m.lsq[2 * n + c];
    const double L22 = m.lsq[3 * n + c], L32 = m.lsq[4 * n + c], L33 = m.lsq[5 * n + c];
    double x1 = b0, x2 = b1, x3 = b2;
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
    b0 = x1; b1 = x2; b2 = x3;
  }
  const size_t ld = m.ldc;
  k.grad[c] = b0;
  k.grad[ld + c] = b1;
  k.grad[2 * ld + c] = b2;
}

__global__ void __launch_bounds__(kBlock) k_kdif_face(DevMesh m, KdifState k) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const size_t lf = m.ldf, ld = m.ldc;
  const int icl = m.fc1[f], icr = m.fc2[f];
  const double dHL = k.kgeo[f], dHR = k.kgeo[lf + f];
  const double vx = k.kgeo[2 * lf + f], vy = k.kgeo[3 * lf + f], vz = k.kgeo[4 * lf + f];
  const double dn = k.kgeo[5 * lf + f], dl2 = k.kgeo[6 * lf + f];
  const double nx = d3(m.fn, m.ldf, f, 0), ny = d3(m.fn, m.ldf, f, 1), nz = d3(m.fn, m.ldf, f, 2);
  const double kl = k.k[icl], kr = k.k[icr];
  const double kH = kl == kr ? kl : 1.0 / (dHL / kl + dHR / kr);
  const double TL = k.T[icl], TR = k.T[icr];
  double Fl;
  if (k.scheme == TY_KDIF_COMPACT) {
    Fl = -kH * (TR - TL) * dn / dl2;
  } else {
    const double gx = dHL * k.grad[icr] + dHR * k.grad[icl];
    const double gy = dHL * k.grad[ld + icr] + dHR * k.grad[ld + icl];
    const double gz = dHL * k.grad[2 * ld + icr] + dHR * k.grad[2 * ld + icl];
    if (k.scheme == TY_KDIF_CELLAVG) {
      Fl = -kH * (gx * nx + gy * ny + gz * nz);
    } else {
      const double pscal = dn / dl2;
      const double Fcomp = pscal * (TR - TL);
      const double tp = 1.0 * pscal;
      const double wx = nx - tp * vx, wy = ny - tp * vy, wz = nz - tp * vz;
      const double Favg = gx * wx + gy * wy + gz * wz;
      Fl = -kH * (1.0 * Fcomp + Favg);
    }
  }
  double jR = -kH * dn / (k.cp * dl2);
  if (f >= m.nfi && k.fkind[f] == TY_KBC_FLUX) {
    Fl = -k.fval[f];
    jR = 0.0;
  }
  const double S = m.fs[f];
  k.flux[f] = S * Fl;
  k.jac[f] = S * jR;
}

// flux balance sum(+-F S) in colour order; optionally dt/V times it into R
__global__ void __launch_bounds__(kBlock) k_kdif_gather(DevMesh m, KdifState k, double dt, double* __restrict__ R) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  double s = 0.0;
  for (int sl = 0; sl < m.nslot; ++sl) {
    const int e = m.cf[sl * (size_t)m.nci + c];
    if (e < 0) break;
    const double F = k.flux[e >> 1];
    s = (e & 1) ? s + F : s - F;
  }
  k.bal[c] = s;
  if (R) R[c] = dt / m.cvol[c] * s;
}

__global__ void __launch_bounds__(kBlock) k_kdif_diag(DevMesh m, KdifState k, double dt, int want32) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  double d = m.cvol[c] / dt;
  for (int sl = 0; sl < m.nslot; ++sl) {
    const int e = k.cfo[sl * (size_t)m.nci + c];
    if (e < 0) break;
    d = d - k.jac[e >> 1];
  }
  k.diag[c] = d;
  if (want32) k.diag32[c] = (float)d;
}

__global__ void k_kdif_jac32(KdifState k, int nf) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) k.jac32[f] = (float)k.jac[f];
}

// y = S x: diagonal, then the cell's interior faces in ascending order; optional partial x.y
template <class V>
__global__ void __launch_bounds__(kRedThreads) k_kdif_mv(DevMesh m, KdifState k, const V* __restrict__ x,
                                                          V* __restrict__ y, const V* __restrict__ dg,
                                                          const V* __restrict__ off, double* __restrict__ part) {
  double acc = 0.0;
  for (int c = blockIdx.x * kRedThreads + threadIdx.x; c < m.nci; c += gridDim.x * kRedThreads) {
    V s = dg[c] * x[c];
    for (int sl = 0; sl < m.nslot; ++sl) {
      const int e = k.cfo[sl * (size_t)m.nci + c];
      if (e < 0) break;
      const int f = e >> 1;
      if (f >= m.nfi) break;
      s = s + off[f] * x[k.cfon[sl * (size_t)m.nci + c]];
    }
    y[c] = s;
    acc += (double)x[c] * (double)s;
  }
  if (part) {
    acc = block_sum(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
  }
}

// CG start: x = 0, z = r / diag, p = z; partial r.z and r.r
template <class V>
__global__ void __launch_bounds__(kRedThreads) k_kdif_cg0(int n, V* x, const V* r, V* z, V* p, const V* dg,
                                                           double* part) {
  double rz = 0.0, rr = 0.0;
  for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads) {
    const V zi = r[i] / dg[i];
    x[i] = V(0);
    z[i] = zi;
    p[i] = zi;
    rz += (double)r[i] * (double)zi;
    rr += (double)r[i] * (double)r[i];
  }
  rz = block_sum(rz);
  if (threadIdx.x == 0) part[blockIdx.x] = rz;
  rr = block_sum(rr);
  if (threadIdx.x == 0) part[kRedBlocks + blockIdx.x] = rr;
}

// x += alpha p, r -= alpha q, z = r / diag; partial r.z and r.r (alpha = scal[0] / scal[1])
template <class V>
__global__ void __launch_bounds__(kRedThreads) k_kdif_cg1(int n, V* x, V* r, V* z, const V* p, const V* q,
                                                           const V* dg, const double* scal, double* part) {
  const double alpha = scal[0] / scal[1];
  double rz = 0.0, rr = 0.0;
  for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads) {
    x[i] = x[i] + V(alpha) * p[i];
    const V ri = r[i] - V(alpha) * q[i];
    r[i] = ri;
    const V zi = ri / dg[i];
    z[i] = zi;
    rz += (double)ri * (double)zi;
    rr += (double)ri * (double)ri;
  }
  rz = block_sum(rz);
  if (threadIdx.x == 0) part[blockIdx.x] = rz;
  rr = block_sum(rr);
  if (threadIdx.x == 0) part[kRedBlocks + blockIdx.x] = rr;
}

// p = z + beta p, beta = scal[2] / scal[0]; then scal[0] = scal[2]
template <class V>
__global__ void k_kdif_cg2(int n, const V* z, V* p, const double* scal) {
  const double beta = scal[2] / scal[0];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    p[i] = z[i] + V(beta) * p[i];
}

// scalar finals: mode 0 start (scal[0] = rz, scal[3] = scal[4] = rr), mode 1 p.q (scal[1]),
// mode 2 update (scal[2] = rz', scal[4] = rr), mode 3 (after cg2) scal[0] = scal[2]
__global__ void __launch_bounds__(kRedThreads) k_kdif_final(const double* part, int nb, int mode, double* scal) {
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < nb; i += kRedThreads) {
    a += part[i];
    if (mode != 1) b += part[kRedBlocks + i];
  }
  a = block_sum(a);
  b = block_sum(b);
  if (threadIdx.x == 0) {
    if (mode == 0) { scal[0] = a; scal[3] = b; scal[4] = b; }
    else if (mode == 1) scal[1] = a;
    else { scal[2] = a; scal[4] = b; }
  }
}
__global__ void k_kdif_shift(double* scal) { scal[0] = scal[2]; }

// r = bal - S x (FP64), r32 = r (the refinement residual)
__global__ void __launch_bounds__(kRedThreads) k_kdif_res64(DevMesh m, KdifState k, double* part) {
  double rr = 0.0;
  for (int c = blockIdx.x * kRedThreads + threadIdx.x; c < m.nci; c += gridDim.x * kRedThreads) {
    double s = k.diag[c] * k.x[c];
    for (int sl = 0; sl < m.nslot; ++sl) {
      const int e = k.cfo[sl * (size_t)m.nci + c];
      if (e < 0) break;
      const int f = e >> 1;
      if (f >= m.nfi) break;
      s = s + k.jac[f] * k.x[k.cfon[sl * (size_t)m.nci + c]];
    }
    const double r = k.bal[c] - s;
    k.r[c] = r;
    k.r32[c] = (float)r;
    rr += r * r;
  }
  rr = block_sum(rr);
  if (threadIdx.x == 0) part[blockIdx.x] = rr;
}
__global__ void __launch_bounds__(kRedThreads) k_kdif_final1(const double* part, int nb, double* out) {
  double a = 0.0;
  for (int i = threadIdx.x; i < nb; i += kRedThreads) a += part[i];
  a = block_sum(a);
  if (threadIdx.x == 0) *out = a;
}
__global__ void k_kdif_refine(int n, double* x, const float* d) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] = x[i] + (double)d[i];
}
__global__ void k_kdif_update_T(DevMesh m, KdifState k) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  k.T[c] = k.T[c] + k.x[c] / k.cp;
}

// ---- fused conjugate gradients in one persistent kernel ----
// Chronopoulos and Gear's arrangement of Jacobi-preconditioned CG: with u = D^-1 r, w = S u,
// and p and s = S p carried by recurrences, the inner products of an iteration, gamma = r.u,
// delta = w.u (and r.r when the residual is checked), come from the same iterate:
//   p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = r / diag;  barrier
//   w = S u; gamma, delta;  barrier;  beta = gamma / gamma_old,
//   alpha = gamma / (delta - beta (gamma / alpha_old))
// One cooperative launch runs up to pcg_chunk() iterations: the grid is resident, every thread
// owns up to K cells whose r, p, s and w stay in registers, only u travels through L2 (z), and
// the scalars are recomputed by every block from the blocks' partial sums, in block order
// (deterministic).  Separate launches cost 9 us of reduction tails and gaps each, whatever the
// mesh.  On GB300, us per iteration: 13,182 cells 26.5 -> 8.0, 750,000 cells 51 -> 30 (FP64 pipe:
// 17 operations per cell, 20 us), 2,058,000 cells (vectors in memory, K = 0) 104 -> 79.
constexpr int kPcgThreads = 512;
constexpr int kPcgPart = 3;  // partial sums per block: gamma, delta, r.r
constexpr int kPcgBlocks = 4 * 160;

// Barrier over a resident grid: `goal` arrivals in total.  Bounded: false after about two
// seconds (the caller leaves the kernel and the host sees the error word).
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned goal) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
    unsigned v = 0;
    int spins = 0;
    do {
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
    } while (v < goal && ++spins < (1 << 22));
    ok = v >= goal;
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// Sums of the N per-thread values over the grid, valid in thread 0.  FP64 instructions are
// scarce (one per 64 clocks, SM quarter and warp), so no warp does what one can do: the values
// meet in shared memory, 128 threads per value add them down to 128, one warp per value to one;
// the blocks' sums meet in part and every block adds them in block order.  False when the
// barrier ran out.
template <int N>
__device__ __forceinline__ bool grid_sum(const double (&v)[N], double* tot, double* part, unsigned* count, unsigned goal) {
  __shared__ double sh[N][kPcgThreads];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nt = blockDim.x;
#pragma unroll
  for (int q = 0; q < N; ++q) sh[q][t] = v[q];
  __syncthreads();
  if (nt > 128) {
    const int q = t >> 7, i = t & 127;
    if (q < N) {
      double a = sh[q][i];
      for (int j = i + 128; j < nt; j += 128) a += sh[q][j];
      sh[q][i] = a;
    }
    __syncthreads();
    if (nt < 128 * N) {  // fewer groups of 128 threads than values
      for (int r = nt >> 7; r < N; ++r) {
        if (t < 128) {
          double a = sh[r][t];
          for (int j = t + 128; j < nt; j += 128) a += sh[r][j];
          sh[r][t] = a;
        }
      }
      __syncthreads();
    }
  }
  if (wid < N) {
    double a = sh[wid][lane];
#pragma unroll
    for (int i = 32; i < 128; i += 32) a += sh[wid][lane + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) part[wid * kPcgBlocks + blockIdx.x] = a;
  }
  if (!grid_barrier(count, goal)) return false;
  if (wid < N) {
    double a = 0.0;
    for (int i = lane; i < (int)gridDim.x; i += 32) a += __ldcg(part + wid * kPcgBlocks + i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) tot[wid] = a;
  }
  __syncthreads();
  return true;
}

template <int K>
__global__ void __launch_bounds__(kPcgThreads, K > 0 ? 1 : 2) k_kdif_pcg(int n, int ns, KdifState k, PcgArgs a) {
  constexpr int KR = K > 0 ? K : 1;
  double R[KR], P[KR], Q[KR], W[KR];  // r, p, s = S p and w = S u of this thread's cells
  const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const int cells = K > 0 ? K : (n - first + stride - 1) / stride;
  unsigned goal = 0;
  bool a32 = a.a32 != 0;
  int it = a.it0, done = 0, switched = 0;
  double alpha = 0.0, beta = 0.0, gamma = 0.0, b2, rr = 0.0;
  // neighbour lists of this thread's cells, [j][slot][thread]: read every iteration, and the
  // address of the gather that the FP64 chain waits for
  extern __shared__ int nbs[];
#define TY_EACH_CELL                      \
  _Pragma("unroll") for (int j = 0; j < cells; ++j) { \
    const int i = first + j * stride;     \
    const int q = K > 0 ? j : 0;          \
    (void)q;                              \
    if (i < n) {
#define TY_END_CELL \
    }               \
  }
  double* gr = k.r;
  double* gp = k.p;
  double* gs = k.s;
  double* gw = k.q;
  // u (already in z, visible to every block) -> w and this thread's sums; one copy per precision
  // of the conductances (a conversion, even predicated off, occupies the FP64 pipe)
  auto product_of = [&](auto* cond, double (&v)[kPcgPart], bool want_rr) {
    F64 g = 0.0, dl = 0.0;
    TY_EACH_CELL
      const F64 uc = __ldcg(k.z + i);
      F64 w = F64(__ldg(k.ell_m + i)) * uc;
      for (int s0 = 0; s0 < ns; s0 += 4) {  // four gathers in flight before the first is used
        F64 c[4], zn[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const int sl = s0 + d < ns ? s0 + d : ns - 1;
          const size_t e = (size_t)sl * n + i;
          const int nb = K > 0 ? nbs[(j * ns + sl) * blockDim.x + threadIdx.x] : __ldg(k.ell_nb + e);
          c[d] = (double)__ldg(cond + e);
          zn[d] = __ldcg(k.z + nb);
        }
#pragma unroll
        for (int d = 0; d < 4; ++d)
          if (s0 + d < ns) w = fma(c[d], uc - zn[d], w);
      }
      const F64 r = K > 0 ? R[q] : gr[i];
      if (K > 0) W[q] = w.v; else gw[i] = w.v;
      g = fma(r, uc, g);
      dl = fma(w, uc, dl);
    TY_END_CELL
    v[0] = g.v;
    v[1] = dl.v;
    v[2] = 0.0;
    if (want_rr) {  // every `check` iterations only
      TY_EACH_CELL
        const double r = K > 0 ? R[q] : gr[i];
        v[2] = fma(r, r, v[2]);
      TY_END_CELL
    }
  };
  auto product = [&](double (&v)[kPcgPart], bool want_rr) {
    if (a32) product_of(k.ell_a32, v, want_rr);
    else product_of(k.ell_a, v, want_rr);
  };
  double v[kPcgPart];
  // Scalars of the next step: sh[0..2] the sums, sh[3] alpha, sh[4] beta.  IEEE divisions (a
  // reciprocal's seed flushes the subnormal numbers that gamma may fall to), two of the three
  // side by side in one warp: gamma / gamma_old and gamma / alpha_old.  gamma = 0: r = 0, reached
  // exactly by a few cells before the residual is due for a check; every block sees it and stops.
  __shared__ double sh[5];
  auto scalars = [&](bool first_step) {
    if (threadIdx.x < 32) {
      const double g = sh[0], q = first_step ? 0.0 : g / (threadIdx.x == 0 ? gamma : alpha);
      const double ga = __shfl_sync(0xffffffffu, q, 1);
      if (threadIdx.x == 0) {
        const double den = sh[1] - q * ga;
        if (den == 0.0 && fabs(g) < 0x1p-1022) sh[0] = 0.0;  // both underflowed
        sh[3] = g / den;
        sh[4] = q;
      }
    }
    __syncthreads();
    gamma = sh[0];
    alpha = sh[3];
    beta = sh[4];
  };
  // the iteration's start from the residual in R (or r): u, w, the sums and the first step
  auto restart = [&]() -> bool {
    TY_EACH_CELL
      const double r = K > 0 ? R[q] : gr[i];
      k.z[i] = r * __ldg(k.dinv + i);
    TY_END_CELL
    if (!grid_barrier(k.count, goal += gridDim.x)) return false;
    product(v, true);
    if (!grid_sum(v, sh, k.part, k.count, goal += gridDim.x)) return false;
    scalars(true);
    return true;
  };
  if (K > 0) {
    TY_EACH_CELL
      for (int sl = 0; sl < ns; ++sl)
        nbs[(j * ns + sl) * blockDim.x + threadIdx.x] = __ldg(k.ell_nb + (size_t)sl * n + i);
    TY_END_CELL
  }
  if (a.start) {
    TY_EACH_CELL
      k.x[i] = 0.0;
      const double b = k.bal[i];
      if (K > 0) { R[q] = b; P[q] = 0.0; Q[q] = 0.0; }
      else { gr[i] = b; gp[i] = 0.0; gs[i] = 0.0; }
    TY_END_CELL
    if (!restart()) { if (threadIdx.x == 0) k.count[1] = 1u; return; }
    b2 = rr = sh[2];
    if (!(b2 > 0.0) || gamma == 0.0) done = 1;  // zero right-hand side
  } else {
    alpha = k.scal[kPcgAlpha]; beta = k.scal[kPcgBeta]; gamma = k.scal[kPcgGamma]; b2 = k.scal[kPcgB2];
    if (K > 0) {
      TY_EACH_CELL
        R[q] = gr[i]; P[q] = gp[i]; Q[q] = gs[i]; W[q] = gw[i];
      TY_END_CELL
    }
  }
  while (!done && it < a.it1) {
    TY_EACH_CELL
      const double u = __ldcg(k.z + i), w = K > 0 ? W[q] : gw[i];
      const double p = fma(beta, K > 0 ? P[q] : gp[i], u), s = fma(beta, K > 0 ? Q[q] : gs[i], w);
      const double r = fma(-alpha, s, K > 0 ? R[q] : gr[i]);
      k.x[i] = fma(alpha, p, k.x[i]);
      k.z[i] = (F64(r) * F64(__ldg(k.dinv + i))).v;
      if (K > 0) { P[q] = p; Q[q] = s; R[q] = r; }
      else { gp[i] = p; gs[i] = s; gr[i] = r; }
    TY_END_CELL
    ++it;
    const bool check = it % a.check == 0 || it == a.max_it;
    if (!grid_barrier(k.count, goal += gridDim.x)) { if (threadIdx.x == 0) k.count[1] = 1u; return; }
    product(v, check);
    if (!grid_sum(v, sh, k.part, k.count, goal += gridDim.x)) { if (threadIdx.x == 0) k.count[1] = 1u; return; }
    scalars(false);
    if (check || gamma == 0.0) {
      rr = sh[2];  // 0 where it was not summed: r = 0
      const double rel = sqrt(rr / b2);
      if (a32 && rel < a.sw) {
        // restart on the FP64 conductances from the true residual r = b - S x (continuing the
        // old directions on the changed operator loses their conjugacy: on a stiff system the
        // iteration stagnates)
        a32 = false;
        switched = 1;
        TY_EACH_CELL
          k.z[i] = k.x[i];
        TY_END_CELL
        bool ok = grid_barrier(k.count, goal += gridDim.x);
        if (ok) {
          double sum[kPcgPart];
          product(sum, false);  // w = S x
          TY_EACH_CELL
            const double r = k.bal[i] - (K > 0 ? W[q] : gw[i]);
            if (K > 0) { R[q] = r; P[q] = 0.0; Q[q] = 0.0; }
            else { gr[i] = r; gp[i] = 0.0; gs[i] = 0.0; }
          TY_END_CELL
          ok = grid_barrier(k.count, goal += gridDim.x) && restart();
        }
        if (!ok) { if (threadIdx.x == 0) k.count[1] = 1u; return; }
        rr = sh[2];
        done = gamma == 0.0;
      } else if (!a32 && (rel < a.tol || gamma == 0.0)) {
        done = 1;
      }
    }
  }
  if (K > 0 && !done) {
    TY_EACH_CELL
      gr[i] = R[q]; gp[i] = P[q]; gs[i] = Q[q]; gw[i] = W[q];
    TY_END_CELL
  }
#undef TY_EACH_CELL
#undef TY_END_CELL
  if (first == 0) {
    k.scal[kPcgAlpha] = alpha; k.scal[kPcgBeta] = beta; k.scal[kPcgGamma] = gamma; k.scal[kPcgB2] = b2;
    k.scal[kPcgRR] = rr; k.scal[kPcgIt] = it; k.scal[kPcgDone] = done;
    k.scal[kPcgA32] = a32 ? 1.0 : 0.0; k.scal[kPcgSwitched] = switched;
  }
}

// the symmetrised matrix in difference form (kdif.hpp) and the Jacobi inverse
__global__ void __launch_bounds__(kBlock) k_kdif_ell(DevMesh m, KdifState k, double dt) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nci) return;
  const size_t n = m.nci;
  double mc = m.cvol[c] / dt, d = mc;
  for (int sl = 0; sl < m.nslot; ++sl) {
    const int e = k.cfo[sl * n + c];
    double a = 0.0;
    int nb = c;
    if (e >= 0) {
      const int f = e >> 1;
      if (f >= m.nfi) mc = mc - k.jac[f];
      else { a = -k.jac[f]; nb = k.cfon[sl * n + c]; }
      d = d - k.jac[f];
    }
    k.ell_a[sl * n + c] = a;
    k.ell_a32[sl * n + c] = (float)a;
    k.ell_nb[sl * n + c] = nb;
  }
  k.ell_m[c] = mc;
  k.dinv[c] = 1.0 / d;
}

// ---- launchers ----
cudaError_t kdif_ell_build(const DevMesh& m, const KdifState& k, double dt, cudaStream_t st) {
  k_kdif_ell<<<nblk(m.nci), kBlock, 0, st>>>(m, k, dt);
  return cudaGetLastError();
}
template <int K>
cudaError_t pcg_launch(int n, int ns, const KdifState& k, const PcgArgs& a, int threads, cudaStream_t st) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t lists = (size_t)K * ns * threads * sizeof(int);
  // the limit of the largest lists, whatever these need: the attribute is the function's, and another
  // thread's launch on another mesh may stand between this call and the launch below
  cudaError_t e = cudaFuncSetAttribute(k_kdif_pcg<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       K * kMaxSlot * kPcgThreads * (int)sizeof(int));
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_kdif_pcg<K>, threads, lists);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorCooperativeLaunchTooLarge;
  const int want = (n + threads * std::max(K, 1) - 1) / (threads * std::max(K, 1));
  const int grid = std::max(1, std::min(want, std::min(K > 0 ? sms : sms * per, kPcgBlocks)));
  int nn = n, nns = ns;
  KdifState kk = k;
  PcgArgs aa = a;
  void* args[] = {&nn, &nns, &kk, &aa};
  if ((e = cudaMemsetAsync(k.count, 0, 2 * sizeof(unsigned), st)) != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel((const void*)k_kdif_pcg<K>, dim3(grid), dim3(threads), args, lists, st);
}

// One block of up to 512 threads per SM and K cells per thread, K the smallest of the list that
// covers the mesh (152 x 512 x 12 = 934,000 cells on GB300), with the block cut to 128 or 256
// threads where that already spreads the mesh over every SM; beyond that the vectors stay in
// memory and the grid takes as many blocks as are resident.
cudaError_t kdif_pcg(const DevMesh& m, const KdifState& k, const PcgArgs& a, cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long n = m.nci;
  if (n <= 128L * sms) return pcg_launch<1>(m.nci, m.nslot, k, a, 128, st);
  if (n <= 256L * sms) return pcg_launch<1>(m.nci, m.nslot, k, a, 256, st);
  const long per = (n + 512L * sms - 1) / (512L * sms);
  if (per <= 1) return pcg_launch<1>(m.nci, m.nslot, k, a, 512, st);
  if (per <= 2) return pcg_launch<2>(m.nci, m.nslot, k, a, 512, st);
  if (per <= 4) return pcg_launch<4>(m.nci, m.nslot, k, a, 512, st);
  if (per <= 6) return pcg_launch<6>(m.nci, m.nslot, k, a, 512, st);
  if (per <= 8) return pcg_launch<8>(m.nci, m.nslot, k, a, 512, st);
  if (per <= 10) return pcg_launch<10>(m.nci, m.nslot, k, a, 512, st);
  if (per <= 12) return pcg_launch<12>(m.nci, m.nslot, k, a, 512, st);
  return pcg_launch<0>(m.nci, m.nslot, k, a, 512, st);
}

cudaError_t kdif_residual(const DevMesh& m, const KdifState& k, double dt, cudaStream_t st) {
  if (m.ng > 0) k_kdif_ghost<<<nblk(m.ng), kBlock, 0, st>>>(m, k);
  if (k.scheme != TY_KDIF_COMPACT) k_kdif_grad<<<nblk(m.nci), kBlock, 0, st>>>(m, k);
  k_kdif_face<<<nblk(m.nf), kBlock, 0, st>>>(m, k);
  k_kdif_gather<<<nblk(m.nci), kBlock, 0, st>>>(m, k, dt, nullptr);
  return cudaGetLastError();
}
cudaError_t kdif_assemble(const DevMesh& m, const KdifState& k, double dt, int want32, cudaStream_t st) {
  k_kdif_diag<<<nblk(m.nci), kBlock, 0, st>>>(m, k, dt, want32);
  if (want32) k_kdif_jac32<<<std::min<unsigned>(nblk(m.nf), 4 * kRedBlocks), kBlock, 0, st>>>(k, m.nf);
  return cudaGetLastError();
}
cudaError_t kdif_matvec(const DevMesh& m, const KdifState& k, const double* x, double* y, cudaStream_t st) {
  k_kdif_mv<double><<<red_grid(m.nci), kRedThreads, 0, st>>>(m, k, x, y, k.diag, k.jac, nullptr);
  return cudaGetLastError();
}
// CG on S x = r (FP64: r = bal; FP32: r32 = refinement residual), scalars in k.scal
cudaError_t kdif_cg_start(const DevMesh& m, const KdifState& k, int f32, cudaStream_t st) {
  const unsigned g = red_grid(m.nci);
  if (f32) k_kdif_cg0<float><<<g, kRedThreads, 0, st>>>(m.nci, k.x32, k.r32, k.z32, k.p32, k.diag32, k.part);
  else {
    cudaMemcpyAsync(k.r, k.bal, m.nci * sizeof(double), cudaMemcpyDeviceToDevice, st);
    k_kdif_cg0<double><<<g, kRedThreads, 0, st>>>(m.nci, k.x, k.r, k.z, k.p, k.diag, k.part);
  }
  k_kdif_final<<<1, kRedThreads, 0, st>>>(k.part, (int)g, 0, k.scal);
  return cudaGetLastError();
}
cudaError_t kdif_cg_iter(const DevMesh& m, const KdifState& k, int f32, cudaStream_t st) {
  const unsigned g = red_grid(m.nci);
  const unsigned g2 = std::min<unsigned>(nblk(m.nci), 4 * kRedBlocks);
  if (f32) {
    k_kdif_mv<float><<<g, kRedThreads, 0, st>>>(m, k, k.p32, k.q32, k.diag32, k.jac32, k.part);
    k_kdif_final<<<1, kRedThreads, 0, st>>>(k.part, (int)g, 1, k.scal);
    k_kdif_cg1<float><<<g, kRedThreads, 0, st>>>(m.nci, k.x32, k.r32, k.z32, k.p32, k.q32, k.diag32, k.scal, k.part);
    k_kdif_final<<<1, kRedThreads, 0, st>>>(k.part, (int)g, 2, k.scal);
    k_kdif_cg2<float><<<g2, kBlock, 0, st>>>(m.nci, k.z32, k.p32, k.scal);
  } else {
    k_kdif_mv<double><<<g, kRedThreads, 0, st>>>(m, k, k.p, k.q, k.diag, k.jac, k.part);
    k_kdif_final<<<1, kRedThreads, 0, st>>>(k.part, (int)g, 1, k.scal);
    k_kdif_cg1<double><<<g, kRedThreads, 0, st>>>(m.nci, k.x, k.r, k.z, k.p, k.q, k.diag, k.scal, k.part);
    k_kdif_final<<<1, kRedThreads, 0, st>>>(k.part, (int)g, 2, k.scal);
    k_kdif_cg2<double><<<g2, kBlock, 0, st>>>(m.nci, k.z, k.p, k.scal);
  }
  k_kdif_shift<<<1, 1, 0, st>>>(k.scal);
  return cudaGetLastError();
}
cudaError_t kdif_residual64(const DevMesh& m, const KdifState& k, cudaStream_t st) {
  const unsigned g = red_grid(m.nci);
  k_kdif_res64<<<g, kRedThreads, 0, st>>>(m, k, k.part);
  k_kdif_final1<<<1, kRedThreads, 0, st>>>(k.part, (int)g, k.scal + 5);
  return cudaGetLastError();
}
cudaError_t kdif_refine(const DevMesh& m, const KdifState& k, cudaStream_t st) {
  k_kdif_refine<<<std::min<unsigned>(nblk(m.nci), 4 * kRedBlocks), kBlock, 0, st>>>(m.nci, k.x, k.x32);
  return cudaGetLastError();
}
cudaError_t kdif_update_T(const DevMesh& m, const KdifState& k, cudaStream_t st) {
  k_kdif_update_T<<<nblk(m.nci), kBlock, 0, st>>>(m, k);
  return cudaGetLastError();
}

}  // namespace TY_KNS
}  // namespace tyk
