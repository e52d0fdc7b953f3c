// mpm_f64.cu — the all-FP64 substep on the GPU, for precision studies.
//
// FP64 particle state and FP64 grid, the reference's substep
// (crates/molla-solvers/src/mpm.rs:2476-2551): p2g (mpm.wgsl:495-628),
// grid_update (:1013-1058), g2p (:1242-1353), plasticity (:1366-1479), with its
// two-sided Jacobi SVD (:349-468) run in FP64 to a tight tolerance.  It measures
// how far the FP32 and FP32 + FP64-SVD modes drift from an all-FP64 run of the
// same step on the same device.
//
// Three launches a substep:
//   k64_grid      acc -> velocity; clears acc, but for a call's last substep,
//                 whose sums are read by the totals
//   k64_particle  g2p, plasticity, the particle's stress and scatter record
//                 (the return mapping's SVD serves the next p2g, which in the
//                 reference runs its own on the F rebuilt from it), and a push
//                 onto its base cell's list
//   k64_p2g       one lane per (cell, x-slab): adds the records of the cell's
//                 particles in registers, then 36 atomics
// A call opens with k64_particle<false>, which only makes the records.
//
// What bounds it: FP64 arithmetic and latency in k64_particle (a Jacobi sweep
// is a serial chain of square roots), latency of the list walk in k64_p2g.  With
// a thread per particle issuing 108 global atomics, its own SVD there, and
// separate g2p and plasticity kernels a call of 100 substeps of 132,651
// particles on a 64^3 grid took 18.9 ms; it takes 7.5.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "mpm_device.cuh"
#include "mpm_f64.cuh"
#include "mpm_kernels.cuh"

namespace mpm {

namespace {

constexpr uint32_t kFault = 2u;  // mpm.wgsl:229

__device__ __forceinline__ bool fin(double x) { return isfinite(x); }

__device__ __forceinline__ double det3d(const double* a) {
  return a[0] * (a[4] * a[8] - a[7] * a[5]) - a[3] * (a[1] * a[8] - a[7] * a[2]) + a[6] * (a[1] * a[5] - a[4] * a[2]);
}

// o = u diag(d) v^T, column-major 3x3.
__device__ __forceinline__ void sandwich64(const double* u, const double* d, const double* v, double* o) {
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) o[3 * c + r] = u[r] * d[0] * v[c] + u[3 + r] * d[1] * v[3 + c] + u[6 + r] * d[2] * v[6 + c];
}

// One FP64 Jacobi rotation of the (P, Q) pair of the symmetric a[3][3]: t =
// sgn(d) e / (|d| + sqrt(d^2 + e^2)) with d = a_qq - a_pp, e = 2 a_pq (the
// reference's 1 / (theta + sgn(theta) sqrt(1 + theta^2))), square roots and
// reciprocals from Newton-refined seeds (nr_rsqrt).
template <int P, int Q>
__device__ __forceinline__ void rot64(double (&a)[3][3], double* v, double tol, double& max_off) {
  constexpr int K = 3 - P - Q;
  const double apq = a[P][Q];
  max_off = fmax(max_off, fabs(apq));
  if (fabs(apq) < tol) return;
  double d = a[Q][Q] - a[P][P], e = 2.0 * apq;
  // t takes d and e to a common factor: a power of two keeps the squares of a
  // blown-up F's inside nr_rsqrt's range (an infinite one leaves a NaN)
  const double m = fmax(fabs(d), fabs(e));
  if (m > 1.0e40) {
    const double k = scalbn(1.0, -ilogb(m));
    d *= k;
    e *= k;
  }
  const double r2 = d * d + e * e;
  const double ri = nr_rsqrt(fabs(d) + r2 * nr_rsqrt(r2));
  const double t = (d >= 0.0 ? e : -e) * (ri * ri);
  const double c = nr_rsqrt(fma(t, t, 1.0));
  const double s = t * c;
  a[P][P] -= t * apq;
  a[Q][Q] += t * apq;
  a[P][Q] = a[Q][P] = 0.0;
  const double akp = a[P][K], akq = a[Q][K];
  a[P][K] = a[K][P] = c * akp - s * akq;
  a[Q][K] = a[K][Q] = s * akp + c * akq;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double vp = v[3 * P + k], vq = v[3 * Q + k];
    v[3 * P + k] = c * vp - s * vq;
    v[3 * Q + k] = s * vp + c * vq;
  }
}

// Two-sided Jacobi SVD of F (column-major) on A = F^T F, cyclic over
// (0,1), (0,2), (1,2), with the reference's sign fixes, all in FP64.  u, v
// column-major; s may carry one negative sign.
__device__ __forceinline__ void svd_ref64(const double* f, double* u, double* s, double* v, double tol, int sweeps) {
  double a[3][3];  // a[col][row]
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) a[c][r] = f[3 * r] * f[3 * c] + f[3 * r + 1] * f[3 * c + 1] + f[3 * r + 2] * f[3 * c + 2];
#pragma unroll
  for (int i = 0; i < 9; ++i) v[i] = (i % 4 == 0) ? 1.0 : 0.0;
#pragma unroll 1
  for (int sw = 0; sw < sweeps; ++sw) {
    double max_off = 0.0;
    rot64<0, 1>(a, v, tol, max_off);
    rot64<0, 2>(a, v, tol, max_off);
    rot64<1, 2>(a, v, tol, max_off);
    if (max_off < tol) break;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double m[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) m[r] = f[r] * v[3 * i] + f[3 + r] * v[3 * i + 1] + f[6 + r] * v[3 * i + 2];
    const double q = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
    const bool zero = q <= 1.0e-24;  // a NaN takes the other branch and reaches s
    double ri = zero ? 0.0 : nr_rsqrt(q);
    s[i] = q * ri;
    if (q > 1.0e96) {  // beyond nr_rsqrt; an overflow reaches s
      s[i] = sqrt(q);
      ri = 1.0 / s[i];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) u[3 * i + r] = zero ? (i == r ? 1.0 : 0.0) : m[r] * ri;
  }
  if (det3d(u) < 0.0) {
    int mi = 0;
    if (s[1] < s[mi]) mi = 1;
    if (s[2] < (mi ? s[1] : s[0])) mi = 2;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double sg = i == mi ? -1.0 : 1.0;
#pragma unroll
      for (int r = 0; r < 3; ++r) u[3 * i + r] *= sg;
      s[i] *= sg;
    }
  }
  if (det3d(v) < 0.0) {
    int mi = 0;
    if (fabs(s[1]) < fabs(s[0])) mi = 1;
    if (fabs(s[2]) < (mi ? fabs(s[1]) : fabs(s[0]))) mi = 2;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double sg = i == mi ? -1.0 : 1.0;
#pragma unroll
      for (int r = 0; r < 3; ++r) v[3 * i + r] *= sg;
      s[i] *= sg;
    }
  }
}

__device__ __forceinline__ void weights64(double fx, double* w) {
  w[0] = 0.5 * (1.5 - fx) * (1.5 - fx);
  w[1] = 0.75 - (fx - 1.0) * (fx - 1.0);
  w[2] = 0.5 * (fx - 0.5) * (fx - 0.5);
}

__device__ __forceinline__ bool latched(const State64& st) { return *(volatile const uint32_t*)st.status != 0u; }

// The scatter record of a particle, in the FP32 path's deposit form (16
// doubles: m, q, Bd, fx: node (i, j, k) of its stencil receives w (m, q + i Bdx
// + j Bdy + k Bdz)), from its position, velocity, C and the SVD of its F; pushed
// onto its base cell's list, or, when the base cell lies outside the grid,
// deposited node by node.  A position off by more than 1e9 cells (or
// NaN) deposits nothing.
__device__ __forceinline__ void record64(const Scene64& sc, const State64& st, int i, const double* x, const double* vel,
                                         const double* C, const double* u, const double* s, double jp, const Mat64& md,
                                         uint32_t* __restrict__ n_cells) {
  double h = 1.0;
  if (md.rheo == 1) h = exp(fmin(fmax(-md.hardening * jp, -3.0), 3.0));
  else if (md.rheo == 0) h = exp(fmin(fmax(jp, -3.0), 3.0));
  double scl[3], tau[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) scl[k] = fmin(fmax(s[k], 0.1), 10.0);
  const double J = scl[0] * scl[1] * scl[2];
  const double m = st.mass[i];
#pragma unroll
  for (int k = 0; k < 3; ++k) tau[k] = 2.0 * md.mu * h * (scl[k] - 1.0) * scl[k] + md.lam * h * (J - 1.0) * J;
  // 4/dx^2 S d with d = (i - fx) dx: inv_dx is the reference's 1/dx rounded to
  // FP32, so that inv_dx dx is 1 to 6e-8 only (exactly for powers of two)
  const double k4 = -sc.dt * st.vol[i] * 4.0 * sc.inv_dx * (sc.inv_dx * sc.dx);
  double Bd[9];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r)
      Bd[3 * c + r] = m * sc.dx * C[3 * c + r] +
                      k4 * (u[r] * tau[0] * u[c] + u[3 + r] * tau[1] * u[3 + c] + u[6 + r] * tau[2] * u[6 + c]);
  int base[3];
  double fx[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double xp = (x[a] - sc.o[a]) * sc.inv_dx;
    if (!(fabs(xp) < 1.0e9)) return;
    const double bf = floor(xp - 0.5);
    base[a] = (int)bf - sc.win[a];
    fx[a] = xp - bf;
  }
  double q[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) q[r] = m * vel[r] - fx[0] * Bd[r] - fx[1] * Bd[3 + r] - fx[2] * Bd[6 + r];
  const int n = sc.n;
  if ((unsigned)base[0] < (unsigned)n && (unsigned)base[1] < (unsigned)n && (unsigned)base[2] < (unsigned)n) {
    double2* rec = reinterpret_cast<double2*>(st.rec + 16 * (size_t)i);
    rec[0] = make_double2(m, q[0]);
    rec[1] = make_double2(q[1], q[2]);
    rec[2] = make_double2(Bd[0], Bd[1]);
    rec[3] = make_double2(Bd[2], Bd[3]);
    rec[4] = make_double2(Bd[4], Bd[5]);
    rec[5] = make_double2(Bd[6], Bd[7]);
    rec[6] = make_double2(Bd[8], fx[0]);
    rec[7] = make_double2(fx[1], fx[2]);
    const uint32_t cell = (uint32_t)base[0] + (uint32_t)n * ((uint32_t)base[1] + (uint32_t)n * (uint32_t)base[2]);
    const int old = atomicExch(&st.head[cell], i);
    st.next[i] = old;
    if (old < 0) st.cells[atomicAdd(n_cells, 1u)] = cell;
    return;
  }
  double w[3][3];
  for (int a = 0; a < 3; ++a) weights64(fx[a], w[a]);
#pragma unroll 1
  for (int k = 0; k < 27; ++k) {
    const int a = k % 3, b = (k / 3) % 3, c = k / 9;
    const int ix = base[0] + a, iy = base[1] + b, iz = base[2] + c;
    if ((unsigned)ix >= (unsigned)n || (unsigned)iy >= (unsigned)n || (unsigned)iz >= (unsigned)n) continue;
    const double wt = w[0][a] * w[1][b] * w[2][c];
    double* g = reinterpret_cast<double*>(st.acc + ((size_t)ix + (size_t)n * ((size_t)iy + (size_t)n * (size_t)iz)));
    atomicAdd(g, wt * m);
    for (int r = 0; r < 3; ++r) atomicAdd(g + 1 + r, wt * (q[r] + a * Bd[r] + b * Bd[3 + r] + c * Bd[6 + r]));
  }
}

// P2G of the listed cells: ten cells x three x-slabs a warp (the slab lanes of
// a cell adjacent, so that they share the record's loads).  Empties the lists.
__global__ void __launch_bounds__(128) k64_p2g(Scene64 sc, State64 st, int par) {
  launch_next();
  wait_previous();
  if (latched(st)) return;
  const int lane = threadIdx.x & 31, slab = lane % 3;
  const uint32_t count = st.n_cells[par];
  const int n = sc.n;
  const uint32_t warps = gridDim.x * (blockDim.x / 32);
  for (uint32_t w = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); w * 10u < count; w += warps) {
    const uint32_t g = w * 10u + (uint32_t)lane / 3u;
    const bool mine = lane < 30 && g < count;
    const uint32_t cell = mine ? st.cells[g] : 0u;
    int j = mine ? st.head[cell] : -1;
    __syncwarp();
    if (mine && slab == 0) st.head[cell] = -1;
    double acc[9][4];
#pragma unroll
    for (int q = 0; q < 9; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.0;
    const double fs = (double)slab;
    while (j >= 0) {
      const double2* r = reinterpret_cast<const double2*>(st.rec + 16 * (size_t)j);
      j = st.next[j];
      const double2 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3], r4 = r[4], r5 = r[5], r6 = r[6], r7 = r[7];
      double wx[3], wy[3], wz[3];
      weights64(r6.y, wx);
      weights64(r7.x, wy);
      weights64(r7.y, wz);
      const double wi = slab == 0 ? wx[0] : (slab == 1 ? wx[1] : wx[2]);
      double qj[3] = {r0.y + fs * r2.x, r1.x + fs * r2.y, r1.y + fs * r3.x};
#pragma unroll
      for (int jj = 0; jj < 3; ++jj) {
        if (jj) {
          qj[0] += r3.y;
          qj[1] += r4.x;
          qj[2] += r4.y;
        }
        const double wij = wi * wy[jj];
        double qk[3] = {qj[0], qj[1], qj[2]};
#pragma unroll
        for (int kk = 0; kk < 3; ++kk) {
          if (kk) {
            qk[0] += r5.x;
            qk[1] += r5.y;
            qk[2] += r6.x;
          }
          const double wt = wij * wz[kk];
          acc[3 * jj + kk][0] += wt * r0.x;
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[3 * jj + kk][1 + c] += wt * qk[c];
        }
      }
    }
    const uint32_t un = (uint32_t)n;
    const int ix = (int)(cell % un) + slab, iy = (int)((cell / un) % un), iz = (int)(cell / un / un);
    const bool put = mine && ix < n;
#pragma unroll
    for (int jj = 0; jj < 3; ++jj)
#pragma unroll
      for (int kk = 0; kk < 3; ++kk) {
        if (!put || iy + jj >= n || iz + kk >= n) continue;
        double* g = reinterpret_cast<double*>(st.acc + ((size_t)ix + (size_t)n * ((size_t)(iy + jj) + (size_t)n * (size_t)(iz + kk))));
#pragma unroll
        for (int c = 0; c < 4; ++c) atomicAdd(g + c, acc[3 * jj + kk][c]);
      }
  }
}

// Grid update; clears the sums (`last`: not) and the cell count of the next p2g.
__global__ void __launch_bounds__(256) k64_grid(Scene64 sc, State64 st, int par, int last) {
  launch_next();
  wait_previous();
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t n3 = (size_t)sc.n * sc.n * sc.n;
  if (c >= n3 || latched(st)) return;
  if (c == 0) {
    atomicAdd(st.status + 1, 1u);
    st.n_cells[par ^ 1] = 0u;
  }
  const double4 a = st.acc[c];
  // A node nothing was deposited to is read by no particle with a weight other
  // than zero, and its old velocity is finite: set_particles clears it, and a
  // velocity that is not finite faults the particle that deposited there in the
  // same substep, after which nothing moves.
  if (a.x == 0.0 && a.y == 0.0 && a.z == 0.0 && a.w == 0.0) return;
  if (!last) st.acc[c] = make_double4(0.0, 0.0, 0.0, 0.0);
  const double m = a.x;
  if (m <= 1.0e-9 || !(m == m)) {
    st.gvel[c] = make_double4(0.0, 0.0, 0.0, 0.0);
    return;
  }
  double vv[3] = {a.y / m, a.z / m, a.w / m};
  vv[1] = vv[1] + sc.dt * sc.gy;
  const int n = sc.n, pad = sc.pad;
  const int ix = (int)(c % n), iy = (int)((c / n) % n), iz = (int)(c / ((size_t)n * n));
  const double f = sc.friction;
  if (sc.sticky) {
    if (ix < pad || ix >= n - pad || iy < pad || iy >= n - pad || iz < pad || iz >= n - pad) vv[0] = vv[1] = vv[2] = 0.0;
  } else {
    if (ix < pad) { vv[0] = fmax(vv[0], 0.0); vv[1] *= f; vv[2] *= f; }
    if (ix >= n - pad) { vv[0] = fmin(vv[0], 0.0); vv[1] *= f; vv[2] *= f; }
    if (iy < pad) { vv[1] = fmax(vv[1], 0.0); vv[0] *= f; vv[2] *= f; }
    if (iy >= n - pad) { vv[1] = fmin(vv[1], 0.0); vv[0] *= f; vv[2] *= f; }
    if (iz < pad) { vv[2] = fmax(vv[2], 0.0); vv[0] *= f; vv[1] *= f; }
    if (iz >= n - pad) { vv[2] = fmin(vv[2], 0.0); vv[0] *= f; vv[1] *= f; }
  }
  st.gvel[c] = make_double4(vv[0], vv[1], vv[2], 0.0);
}

// GATHER: g2p, plasticity and the record for the next p2g (into the lists of
// parity `par`; a call's last substep makes none); otherwise the record of the
// state as it is.
// Four blocks an SM (128 registers, 116 bytes spilled) beat three at 168: 43 -> 37
// us for 132,651 particles, which are 2.3 waves of the latter.
template <bool GATHER>
__global__ void __launch_bounds__(128, 4) k64_particle(Scene64 sc, State64 st, int par, int last) {
  launch_next();
  wait_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= st.n || latched(st)) return;
  double* pos = st.pos + 3 * (size_t)i;
  double* vel = st.vel + 3 * (size_t)i;
  double* Cp = st.C + 9 * (size_t)i;
  double* Fp = st.F + 9 * (size_t)i;
  const Mat64& md = sc.mat[st.mat[i] < (uint32_t)sc.n_mat ? st.mat[i] : 0];
  double x[3], v[3], C[9], F[9], jp = st.jp[i], u[9], s[3], V[9];
#pragma unroll
  for (int a = 0; a < 3; ++a) x[a] = pos[a];
#pragma unroll
  for (int k = 0; k < 9; ++k) F[k] = Fp[k];
  if constexpr (!GATHER) {
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = vel[a];
#pragma unroll
    for (int k = 0; k < 9; ++k) C[k] = Cp[k];
    svd_ref64(F, u, s, V, sc.tol, sc.sweeps);
  } else {
    bool ok = fin(jp);
    double xp[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      xp[a] = (x[a] - sc.o[a]) * sc.inv_dx;
      ok = ok && fin(x[a]) && fin(xp[a]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) ok = ok && fin(F[k]);
    if (!ok) {
      atomicOr(st.status, kFault);
      return;
    }
    int at[3][3];  // node coordinates, clamped; out-of-grid nodes weigh nothing
    double w[3][3], wd[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double bf = floor(xp[a] - 0.5);
      const int base = (int)bf - sc.win[a];
      const double fx = xp[a] - bf;
      weights64(fx, w[a]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const bool in = (unsigned)(base + k) < (unsigned)sc.n;
        at[a][k] = in ? base + k : 0;
        if (!in) w[a][k] = 0.0;
        wd[a][k] = w[a][k] * (((double)k - fx) * sc.dx);
      }
    }
    // separable sums: v = sum w gv, G = sum (w gv) d^T
    double vn[3] = {0.0, 0.0, 0.0}, G[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (int kz = 0; kz < 3; ++kz) {
      double s0[3] = {0, 0, 0}, sx[3] = {0, 0, 0}, sy[3] = {0, 0, 0};
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        const double4* row = st.gvel + (size_t)sc.n * ((size_t)at[1][ky] + (size_t)sc.n * (size_t)at[2][kz]);
        double r0[3] = {0, 0, 0}, rx[3] = {0, 0, 0};
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const double4 g = row[at[0][kx]];
          const double gv[3] = {g.x, g.y, g.z};
#pragma unroll
          for (int r = 0; r < 3; ++r) {
            r0[r] += w[0][kx] * gv[r];
            rx[r] += wd[0][kx] * gv[r];
          }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          s0[r] += w[1][ky] * r0[r];
          sx[r] += w[1][ky] * rx[r];
          sy[r] += wd[1][ky] * r0[r];
        }
      }
      const double wz = kz == 0 ? w[2][0] : (kz == 1 ? w[2][1] : w[2][2]);
      const double wdz = kz == 0 ? wd[2][0] : (kz == 1 ? wd[2][1] : wd[2][2]);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        vn[r] += wz * s0[r];
        G[r] += wz * sx[r];
        G[3 + r] += wz * sy[r];
        G[6 + r] += wdz * s0[r];
      }
    }
    const double scale = 4.0 * sc.inv_dx * sc.inv_dx;
#pragma unroll
    for (int k = 0; k < 9; ++k) C[k] = scale * G[k];
    if (md.rheo == 2) {
      const double vd = exp(-fmax(md.vdamp, 0.0) * sc.dt), ad = exp(-fmax(md.adamp, 0.0) * sc.dt);
#pragma unroll
      for (int r = 0; r < 3; ++r) vn[r] *= vd;
#pragma unroll
      for (int k = 0; k < 9; ++k) C[k] *= ad;
    }
    double np[3];
    bool ok2 = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      np[a] = x[a] + sc.dt * vn[a];
      ok2 = ok2 && fin(np[a]) && fin(vn[a]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) ok2 = ok2 && fin(C[k]);
    double Fn[9];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) acc += ((r == k ? 1.0 : 0.0) + sc.dt * C[3 * k + r]) * F[3 * c + k];
        Fn[3 * c + r] = acc;
        ok2 = ok2 && fin(acc);
      }
    if (!ok2) {
      atomicOr(st.status, kFault);
      return;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[a] = (np[a] < sc.lo[a] || np[a] > sc.hi[a]) ? 0.0 : vn[a];
      x[a] = fmin(fmax(np[a], sc.lo[a]), sc.hi[a]);
      pos[a] = x[a];
      vel[a] = v[a];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) Cp[k] = C[k];
    // ---- plasticity (mpm.wgsl:1366-1479); a fault here leaves the g2p state ----
    svd_ref64(Fn, u, s, V, sc.tol, sc.sweeps);
    bool ok3 = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) ok3 = ok3 && fin(s[k]);
#pragma unroll
    for (int k = 0; k < 9; ++k) ok3 = ok3 && fin(u[k]) && fin(V[k]);
    double ns[3] = {s[0], s[1], s[2]}, dq = 0.0, jp_new = 0.0;
    bool replace = false;
    if (md.rheo == 1) {
#pragma unroll
      for (int a = 0; a < 3; ++a) ns[a] = fmin(fmax(s[a], 1.0 - md.theta_c), 1.0 + md.theta_s);
      const double det_old = fmax(s[0] * s[1] * s[2], 1.0e-6), det_new = fmax(ns[0] * ns[1] * ns[2], 1.0e-6);
      replace = true;
      jp_new = jp + (log(det_old) - log(det_new));
      ok3 = ok3 && fin(jp_new);
      jp_new = fmin(fmax(jp_new, -5.0), 5.0);
    } else if (md.rheo == 2) {
      replace = true;
    } else {
      double eps[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) eps[a] = log(fmax(s[a], 1.0e-6));
      const double tr = eps[0] + eps[1] + eps[2], mean = tr / 3.0;
      const double dev[3] = {eps[0] - mean, eps[1] - mean, eps[2] - mean};
      const double dn = sqrt(dev[0] * dev[0] + dev[1] * dev[1] + dev[2] * dev[2]);
      if (tr > 0.0) {
        ns[0] = ns[1] = ns[2] = 1.0;
        dq = sqrt(eps[0] * eps[0] + eps[1] * eps[1] + eps[2] * eps[2]);
      } else if (dn != 0.0) {
        const double fy = dn + md.kappa * tr * md.dp_alpha;
        if (fy > 0.0) {
          const double rc = fmax(0.0, -md.dp_alpha * md.kappa * tr);
#pragma unroll
          for (int a = 0; a < 3; ++a) ns[a] = exp(dev[a] * (rc / dn) + mean);
          dq = fy;
        }
      }
    }
    ok3 = ok3 && fin(ns[0]) && fin(ns[1]) && fin(ns[2]) && fin(dq) && fin(jp + dq);
    if (!ok3) {
#pragma unroll
      for (int k = 0; k < 9; ++k) Fp[k] = Fn[k];
      atomicOr(st.status, kFault);
      return;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) s[a] = fmin(fmax(ns[a], 0.05), 20.0);
    sandwich64(u, s, V, F);
#pragma unroll
    for (int k = 0; k < 9; ++k) Fp[k] = F[k];
    jp = replace ? jp_new : fmin(fmax(jp + dq, 0.0), 5.0);
    st.jp[i] = jp;
  }
  if (!last) record64(sc, st, i, x, v, C, u, s, jp, md, st.n_cells + par);
}

// Grid totals of a P2G: out[0] mass, out[1..3] momentum.
__global__ void k64_totals(size_t n3, const double4* __restrict__ g, double* out) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n3; c += (size_t)gridDim.x * blockDim.x) {
    const double4 a = g[c];
    acc[0] += a.x;
    acc[1] += a.y;
    acc[2] += a.z;
    acc[3] += a.w;
  }
  for (int k = 0; k < 4; ++k) {
    double x = acc[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&out[k], x);
  }
}

}  // namespace

cudaError_t launch_step64(const Scene64& sc, const State64& st, uint32_t substeps, cudaStream_t s,
                          uint64_t* launches) {
  const size_t n3 = (size_t)sc.n * sc.n * sc.n;
  const int pb = (st.n + 127) / 128, gb = (int)((n3 + 255) / 256);
  // forty cells a block; about as many blocks as stay resident
  const int cb = std::min((st.n + 39) / 40, 148 * 8);
  if (!substeps) return cudaSuccess;
  cudaMemsetAsync(st.head, 0xff, n3 * sizeof(int), s);
  cudaMemsetAsync(st.n_cells, 0, 2 * sizeof(uint32_t), s);
  cudaMemsetAsync(st.acc, 0, n3 * sizeof(double4), s);
  cudaError_t e = cudaGetLastError();
  if (st.n && e == cudaSuccess) {
    e = launch_dependent(k64_particle<false>, pb, 128, 0, s, sc, st, 0, 0);
    ++*launches;
  }
  for (uint32_t k = 0; k < substeps && e == cudaSuccess; ++k) {
    const int par = (int)(k & 1u), last = k + 1 == substeps ? 1 : 0;
    if (st.n) e = launch_dependent(k64_p2g, cb, 128, 0, s, sc, st, par);
    if (e == cudaSuccess) e = launch_dependent(k64_grid, gb, 256, 0, s, sc, st, par, last);
    if (st.n && e == cudaSuccess) e = launch_dependent(k64_particle<true>, pb, 128, 0, s, sc, st, par ^ 1, last);
    *launches += st.n ? 3 : 1;
  }
  return e;
}

cudaError_t launch_totals64(const Scene64& sc, const State64& st, double* out4, cudaStream_t s) {
  cudaMemsetAsync(out4, 0, 4 * sizeof(double), s);
  k64_totals<<<592, 256, 0, s>>>((size_t)sc.n * sc.n * sc.n, st.acc, out4);
  return cudaGetLastError();
}

}  // namespace mpm
