// elastic3d_adjoint.cu -- hand-written discrete adjoint of the 3D SSG-CPML
// moment-tensor step (src/Elastic3D_SSG_Tensor.py:166-345) and point-force
// step (src/Elastic3D_SSG_CPML.py:144-309, the same stencils) for gradients of
// a seismogram misfit with respect to rho, lambda and mu.  No reference
// counterpart.
//
// Forward step it (the oracle's velocity3d / stress3d order):
//   inject   sigma_ab[src] += w(it) * (-M_ab)
//   V   vx += dt/rho      (Dx+ sxx' + Dz- sxz' + Dy- sxy')     vx cells
//       vy += dt/rho_y    (Dx- sxy' + Dy+ syy' + Dz- syz')     vy cells
//       vz += dt/rho_4    (Dx- sxz' + Dy- syz' + Dz+ szz')     vz cells
//   S   sxx += dt*(lpm e0 + lhx (e2 + e1)), syy, szz likewise, e = D- v   normal cells
//       sxy += m_xy (Dy+ vx' + Dx+ vy') dt, sxz += m_xz (Dz+ vx' + Dx+ vz') dt,
//       syz += m_yz (Dy+ vz' + Dz+ vy') dt
//   record data[it] = field[rec]
// with D+ f = sum c_m (f[+m+1] - f[-m]), D- f = sum c_m (f[+m] - f[-m-1]) along
// one axis, divided by the spacing, and d' = d/kappa + psi_new on the CPML
// cells.  The adjoint of step it runs the phases in reverse: receivers, the
// stress phase's mids (CPML recursion reversed) and lambda/mu gradients, the
// gather of the transposed stencils into the velocity adjoints, then the same
// for the velocity phase.  Forward values come from sw3d_record snapshots:
// slot k is the state of step it after its source injection, slot k+1 holds
// the velocities after the velocity phase of step it.
#include "sw_device.cuh"

namespace sw {

template <typename T>
struct A3 {
  T* f[9];          // adjoint of vx vy vz sxx syy szz sxy sxz syz
  T* mem[3];        // adjoint memory variables, slab layout of P3::mem
  T* tmp[9];        // mid fields (nx, ny, nz)
  T* grad[8];       // per-cell sums: G_vx G_vy G_vz (densities), G_lpm G_lhx (normal), G_xy G_xz G_yz (shear)
  const T* res;     // receiver residual (nt, nrec)
  const T* snap0;   // slot k
  const T* snap1;   // slot k+1
};

constexpr int B3Z = 32;
constexpr int B3Y = 8;
// Resident blocks per SM the float kernels are compiled for: one thread per
// cell waits on its loads (104 x 96 x 80, order 2, stress / velocity mid us: the
// compiler's own count 90 / 74, 4 blocks 78 / 74, 6 70 / 68, 8 74 / 68).
#define SW_ADJ3_MINB (sizeof(T) == 4 ? 6 : 1)

// stencil along one axis (stride st), forward (D+) or backward (D-)
template <typename T, int N, bool FWD>
__device__ __forceinline__ T d3(const T* f, long long idx, long long st, const T* c) {
  T v = 0;
#pragma unroll
  for (int m = 0; m < N; ++m)
    v += FWD ? c[m] * (f[idx + (m + 1) * st] - f[idx - m * st]) : c[m] * (f[idx + m * st] - f[idx - (m + 1) * st]);
  return v;
}

// transposed stencil of a mid field M along one axis at coordinate x of n
template <typename T, int N, bool FWD>
__device__ __forceinline__ T d3t(const T* M, long long idx, long long st, int x, int n, const T* c) {
  T v = 0;
#pragma unroll
  for (int m = 0; m < N; ++m) {
    const int a = FWD ? x - m - 1 : x - m, b = FWD ? x + m : x + m + 1;
    const T ma = (a >= 0 && a < n) ? M[idx + (long long)(a - x) * st] : (T)0;
    const T mb = (b >= 0 && b < n) ? M[idx + (long long)(b - x) * st] : (T)0;
    v += c[m] * (ma - mb);
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T pml_fwd3(T d, T psi_old, T b, T a, T kk) {
  const T psi = b * psi_old + a * d;
  return div_v(d, kk) + psi;
}
template <typename T>
__device__ __forceinline__ T pml_adj3(T dbar, T* psibar, T b, T a, T kk) {
  const T tot = *psibar + dbar;
  *psibar = b * tot;
  return dbar / kk + a * tot;
}

// CPML of one derivative of component `comp` along axis AX at cell (i, j, k):
// forward value from the snapshot's psi, adjoint through the adjoint psi.
template <typename T, int AX>
struct Cpml3 {
  long long off;  // element offset of psi within the axis's component array
  bool on;
  T b, a, kk;
};

template <typename T, int AX>
__device__ __forceinline__ Cpml3<T, AX> cpml3(const P3<T>& p, int comp, bool half, bool pred, int i, int j, int k) {
  Cpml3<T, AX> r{};
  const int n = AX == 0 ? p.nx : AX == 1 ? p.ny : p.nz;
  const int x = AX == 0 ? i : AX == 1 ? j : k;
  const int s = slab_index(x, n, p.lo[AX], p.hi[AX]);
  r.on = pred && s >= 0;
  if (!r.on) return r;
  const T* cf = p.cf[AX];
  r.b = cf[(half ? CBH : CB) * n + x];
  r.a = cf[(half ? CAH : CA) * n + x];
  r.kk = cf[(half ? CKH : CK) * n + x];
  if (AX == 0) r.off = comp * p.mcomp[0] + ((long long)s * p.ny + j) * p.nz + k;
  else if (AX == 1) r.off = comp * p.mcomp[1] + ((long long)i * p.sn[1] + s) * p.nz + k;
  else r.off = comp * p.mcomp[2] + ((long long)i * p.ny + j) * p.sn[2] + s;
  return r;
}

// snapshot memory variables of axis AX
template <typename T, int AX>
__device__ __forceinline__ const T* snap_mem(const P3<T>& p, const T* snap) {
  const long long nc = (long long)p.nx * p.ny * p.nz;
  const long long base = 9 * nc + (AX >= 1 ? 6 * p.mcomp[0] : 0) + (AX >= 2 ? 6 * p.mcomp[1] : 0);
  return snap + base;
}

#define CELL3                                                   \
  const int k = blockIdx.x * B3Z + threadIdx.x;                 \
  const int j = blockIdx.y * B3Y + threadIdx.y;                 \
  const int i = blockIdx.z;                                     \
  const int nx = p.nx, ny = p.ny, nz = p.nz;                    \
  if (j >= ny || k >= nz) return;                               \
  const long long sx = (long long)ny * nz, sy = nz;             \
  const long long idx = i * sx + (long long)j * nz + k;         \
  T c[N];                                                       \
  _Pragma("unroll") for (int m = 0; m < N; ++m) c[m] = p.c[m];  \
  const uint8_t fx = p.fl[0][i], fy = p.fl[1][j], fz = p.fl[2][k];

// The nearest cell whose taps all lie inside the grid.  The mid kernels form
// their nine derivatives there before they look at any range: all tap loads
// are in flight together and the quotients by the spacings form one group (a
// cell outside a component's range never uses that component's derivatives).
// What bounded these kernels was 18 IEEE divisions a cell, one after another
// behind the loads of its own component: 104 x 96 x 80, order 2, stress /
// velocity mid 104 / 111 -> 90 / 74 us.
#define INNER3                                                                                  \
  const long long in = min(max(i, N), nx - 1 - N) * sx + (long long)min(max(j, N), ny - 1 - N) * nz + \
                       min(max(k, N), nz - 1 - N);

template <typename T>
__global__ void k3a_record(const __grid_constant__ P3<T> p, const __grid_constant__ A3<T> a, int it) {
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < p.nrec) atomicAdd(a.f[p.rec_field] + p.rec_idx[r], a.res[(long long)it * p.nrec + r]);
}

// ---- stress phase ---------------------------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(B3Z * B3Y, SW_ADJ3_MINB)
k3a_stress_mid(const __grid_constant__ P3<T> p, const __grid_constant__ A3<T> a) {
  CELL3
  INNER3
  const long long nc = (long long)nx * ny * nz;
  const T* vx = a.snap1;
  const T* vy = a.snap1 + nc;
  const T* vz = a.snap1 + 2 * nc;
  const T* m0 = snap_mem<T, 0>(p, a.snap0);
  const T* m1 = snap_mem<T, 1>(p, a.snap0);
  const T* m2 = snap_mem<T, 2>(p, a.snap0);
  const T dt = p.dt;
  // the nine derivatives before their ranges are looked at (INNER3)
  const T hd[9] = {p.dx, p.dy, p.dz, p.dx, p.dy, p.dx, p.dz, p.dy, p.dz};
  const T hr[9] = {p.rd[0], p.rd[1], p.rd[2], p.rd[0], p.rd[1], p.rd[0], p.rd[2], p.rd[1], p.rd[2]};
  T dv[9] = {d3<T, N, false>(vx, in, sx, c), d3<T, N, false>(vy, in, sy, c), d3<T, N, false>(vz, in, 1, c),
             d3<T, N, true>(vy, in, sx, c),  d3<T, N, true>(vx, in, sy, c),  d3<T, N, true>(vz, in, sx, c),
             d3<T, N, true>(vx, in, 1, c),   d3<T, N, true>(vz, in, sy, c),  d3<T, N, true>(vy, in, 1, c)};
  divc_group<9>(dv, hd, hr, p.fast_div);
  T out[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const T u0 = ldg(p.mu + in), ux = ldg(p.mu + in + sx), uy = ldg(p.mu + in + sy), uz = ldg(p.mu + in + 1);
  // normal stresses: i, j, k in [N+1, n-N)
  if (i >= N + 1 && i < nx - N && j >= N + 1 && j < ny - N && k >= N + 1 && k < nz - N) {
    const T lhx = (T)0.5 * (ldg(p.lam + idx) + ldg(p.lam + idx + sx));
    const T mhx = (T)0.5 * (u0 + ux);
    const T lpm = lhx + (T)2 * mhx;
    const bool P = ((fx | fy | fz) & 1) != 0;
    auto cx = cpml3<T, 0>(p, 3, false, P, i, j, k);
    auto cy = cpml3<T, 1>(p, 3, false, P, i, j, k);
    auto cz = cpml3<T, 2>(p, 3, false, P, i, j, k);
    T e0 = dv[0], e1 = dv[1], e2 = dv[2];
    if (cx.on) e0 = pml_fwd3(e0, m0[cx.off], cx.b, cx.a, cx.kk);
    if (cy.on) e1 = pml_fwd3(e1, m1[cy.off], cy.b, cy.a, cy.kk);
    if (cz.on) e2 = pml_fwd3(e2, m2[cz.off], cz.b, cz.a, cz.kk);
    const T bx = a.f[3][idx], by = a.f[4][idx], bz = a.f[5][idx];
    a.grad[3][idx] += dt * (bx * e0 + by * e1 + bz * e2);
    a.grad[4][idx] += dt * (bx * (e2 + e1) + by * (e0 + e2) + bz * (e0 + e1));
    T g0 = dt * (lpm * bx + lhx * by + lhx * bz);
    T g1 = dt * (lhx * bx + lpm * by + lhx * bz);
    T g2 = dt * (lhx * bx + lhx * by + lpm * bz);
    if (cx.on) g0 = pml_adj3(g0, a.mem[0] + cx.off, cx.b, cx.a, cx.kk);
    if (cy.on) g1 = pml_adj3(g1, a.mem[1] + cy.off, cy.b, cy.a, cy.kk);
    if (cz.on) g2 = pml_adj3(g2, a.mem[2] + cz.off, cz.b, cz.a, cz.kk);
    out[0] = g0;
    out[1] = g1;
    out[2] = g2;
  }
  // sxy: i, j in [N+1, n-N), k in [N, nz-N)
  if (i >= N + 1 && i < nx - N && j >= N + 1 && j < ny - N && k >= N && k < nz - N) {
    const T m4 = (T)0.25 * (uy + u0 + u0 + ux);
    const bool P = (fx & 2) || (fy & 2) || (fz & 1);
    auto cx = cpml3<T, 0>(p, 4, true, P, i, j, k);
    auto cy = cpml3<T, 1>(p, 4, true, P, i, j, k);
    T f0 = dv[3], f1 = dv[4];
    if (cx.on) f0 = pml_fwd3(f0, m0[cx.off], cx.b, cx.a, cx.kk);
    if (cy.on) f1 = pml_fwd3(f1, m1[cy.off], cy.b, cy.a, cy.kk);
    const T b = a.f[6][idx];
    a.grad[5][idx] += dt * b * (f1 + f0);
    T g = m4 * dt * b, g0 = g, g1 = g;
    if (cx.on) g0 = pml_adj3(g0, a.mem[0] + cx.off, cx.b, cx.a, cx.kk);
    if (cy.on) g1 = pml_adj3(g1, a.mem[1] + cy.off, cy.b, cy.a, cy.kk);
    out[3] = g0;
    out[4] = g1;
  }
  // sxz: i in [N, nx-N-1), j in [N, ny-N), k in [N, nz-N-1)
  if (i >= N && i < nx - N - 1 && j >= N && j < ny - N && k >= N && k < nz - N - 1) {
    const T m4 = (T)0.25 * (u0 + ux + u0 + uy);
    const bool P = (fx & 2) || (fy & 1) || (fz & 2);
    auto cx = cpml3<T, 0>(p, 5, true, P, i, j, k);
    auto cz = cpml3<T, 2>(p, 4, true, P, i, j, k);
    T h0 = dv[5], h1 = dv[6];
    if (cx.on) h0 = pml_fwd3(h0, m0[cx.off], cx.b, cx.a, cx.kk);
    if (cz.on) h1 = pml_fwd3(h1, m2[cz.off], cz.b, cz.a, cz.kk);
    const T b = a.f[7][idx];
    a.grad[6][idx] += dt * b * (h1 + h0);
    T g = m4 * dt * b, g0 = g, g1 = g;
    if (cx.on) g0 = pml_adj3(g0, a.mem[0] + cx.off, cx.b, cx.a, cx.kk);
    if (cz.on) g1 = pml_adj3(g1, a.mem[2] + cz.off, cz.b, cz.a, cz.kk);
    out[5] = g0;
    out[6] = g1;
  }
  // syz: i in [N, nx-N), j in [N, ny-N-1), k in [N, nz-N-1)
  if (i >= N && i < nx - N && j >= N && j < ny - N - 1 && k >= N && k < nz - N - 1) {
    const T m4 = (T)0.25 * (uy + u0 + uz + u0);
    const bool P = (fx & 1) || (fy & 2) || (fz & 2);
    auto cy = cpml3<T, 1>(p, 5, true, P, i, j, k);
    auto cz = cpml3<T, 2>(p, 5, true, P, i, j, k);
    T q0 = dv[7], q1 = dv[8];
    if (cy.on) q0 = pml_fwd3(q0, m1[cy.off], cy.b, cy.a, cy.kk);
    if (cz.on) q1 = pml_fwd3(q1, m2[cz.off], cz.b, cz.a, cz.kk);
    const T b = a.f[8][idx];
    a.grad[7][idx] += dt * b * (q0 + q1);
    T g = m4 * dt * b, g0 = g, g1 = g;
    if (cy.on) g0 = pml_adj3(g0, a.mem[1] + cy.off, cy.b, cy.a, cy.kk);
    if (cz.on) g1 = pml_adj3(g1, a.mem[2] + cz.off, cz.b, cz.a, cz.kk);
    out[7] = g0;
    out[8] = g1;
  }
  divc_group<9>(out, hd, hr, p.fast_div);
#pragma unroll
  for (int q = 0; q < 9; ++q) a.tmp[q][idx] = out[q];
}

// vx_bar += D-x^T t0 + D+y^T t4 + D+z^T t6; vy_bar += D-y^T t1 + D+x^T t3 + D+z^T t8;
// vz_bar += D-z^T t2 + D+x^T t5 + D+y^T t7
template <typename T, int N>
__global__ void __launch_bounds__(B3Z * B3Y, SW_ADJ3_MINB)
k3a_vel_gather(const __grid_constant__ P3<T> p, const __grid_constant__ A3<T> a) {
  CELL3
  (void)fx; (void)fy; (void)fz;
  a.f[0][idx] += d3t<T, N, false>(a.tmp[0], idx, sx, i, nx, c) + d3t<T, N, true>(a.tmp[4], idx, sy, j, ny, c) +
                 d3t<T, N, true>(a.tmp[6], idx, 1, k, nz, c);
  a.f[1][idx] += d3t<T, N, false>(a.tmp[1], idx, sy, j, ny, c) + d3t<T, N, true>(a.tmp[3], idx, sx, i, nx, c) +
                 d3t<T, N, true>(a.tmp[8], idx, 1, k, nz, c);
  a.f[2][idx] += d3t<T, N, false>(a.tmp[2], idx, 1, k, nz, c) + d3t<T, N, true>(a.tmp[5], idx, sx, i, nx, c) +
                 d3t<T, N, true>(a.tmp[7], idx, sy, j, ny, c);
}

// ---- velocity phase -------------------------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(B3Z * B3Y, SW_ADJ3_MINB)
k3a_vel_mid(const __grid_constant__ P3<T> p, const __grid_constant__ A3<T> a) {
  CELL3
  INNER3
  const long long nc = (long long)nx * ny * nz;
  const T* sxx = a.snap0 + 3 * nc;
  const T* syy = a.snap0 + 4 * nc;
  const T* szz = a.snap0 + 5 * nc;
  const T* sxy = a.snap0 + 6 * nc;
  const T* sxz = a.snap0 + 7 * nc;
  const T* syz = a.snap0 + 8 * nc;
  const T* m0 = snap_mem<T, 0>(p, a.snap0);
  const T* m1 = snap_mem<T, 1>(p, a.snap0);
  const T* m2 = snap_mem<T, 2>(p, a.snap0);
  const T dt = p.dt;
  const T* rho = p.rho;
  const T hd[9] = {p.dx, p.dy, p.dz, p.dx, p.dy, p.dz, p.dx, p.dy, p.dz};
  const T hr[9] = {p.rd[0], p.rd[1], p.rd[2], p.rd[0], p.rd[1], p.rd[2], p.rd[0], p.rd[1], p.rd[2]};
  T dv[9] = {d3<T, N, true>(sxx, in, sx, c),  d3<T, N, false>(sxy, in, sy, c), d3<T, N, false>(sxz, in, 1, c),
             d3<T, N, false>(sxy, in, sx, c), d3<T, N, true>(syy, in, sy, c),  d3<T, N, false>(syz, in, 1, c),
             d3<T, N, false>(sxz, in, sx, c), d3<T, N, false>(syz, in, sy, c), d3<T, N, true>(szz, in, 1, c)};
  divc_group<9>(dv, hd, hr, p.fast_div);
  T out[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const T r00 = ldg(rho + in), r01 = ldg(rho + in + sy), r11 = ldg(rho + in + sx + sy), r10 = ldg(rho + in + sx);
  // vx: i in [N, nx-N-1), j in [N+1, ny-N), k in [N+1, nz-N)
  if (i >= N && i < nx - N - 1 && j >= N + 1 && j < ny - N && k >= N + 1 && k < nz - N) {
    const bool P = (fx & 2) || (fy & 1) || (fz & 1);
    auto cx = cpml3<T, 0>(p, 0, true, P, i, j, k);
    auto cy = cpml3<T, 1>(p, 0, false, P, i, j, k);
    auto cz = cpml3<T, 2>(p, 0, false, P, i, j, k);
    T d0 = dv[0], d1 = dv[1], d2 = dv[2];
    if (cx.on) d0 = pml_fwd3(d0, m0[cx.off], cx.b, cx.a, cx.kk);
    if (cy.on) d1 = pml_fwd3(d1, m1[cy.off], cy.b, cy.a, cy.kk);
    if (cz.on) d2 = pml_fwd3(d2, m2[cz.off], cz.b, cz.a, cz.kk);
    const T vb = a.f[0][idx];
    a.grad[0][idx] += vb * (d0 + d2 + d1) * dt;
    T g = vb * dt / r00, g0 = g, g1 = g, g2 = g;
    if (cx.on) g0 = pml_adj3(g0, a.mem[0] + cx.off, cx.b, cx.a, cx.kk);
    if (cy.on) g1 = pml_adj3(g1, a.mem[1] + cy.off, cy.b, cy.a, cy.kk);
    if (cz.on) g2 = pml_adj3(g2, a.mem[2] + cz.off, cz.b, cz.a, cz.kk);
    out[0] = g0;
    out[1] = g1;
    out[2] = g2;
  }
  // vy: i in [N+1, nx-N), j in [N, ny-N-1), k in [N+1, nz-N)
  if (i >= N + 1 && i < nx - N && j >= N && j < ny - N - 1 && k >= N + 1 && k < nz - N) {
    const T rhy = (T)0.5 * (r00 + r01);
    const bool P = (fx & 1) || (fy & 2) || (fz & 1);
    auto cx = cpml3<T, 0>(p, 1, false, P, i, j, k);
    auto cy = cpml3<T, 1>(p, 1, true, P, i, j, k);
    auto cz = cpml3<T, 2>(p, 1, false, P, i, j, k);
    T d0 = dv[3], d1 = dv[4], d2 = dv[5];
    if (cx.on) d0 = pml_fwd3(d0, m0[cx.off], cx.b, cx.a, cx.kk);
    if (cy.on) d1 = pml_fwd3(d1, m1[cy.off], cy.b, cy.a, cy.kk);
    if (cz.on) d2 = pml_fwd3(d2, m2[cz.off], cz.b, cz.a, cz.kk);
    const T vb = a.f[1][idx];
    a.grad[1][idx] += vb * (d0 + d1 + d2) * dt;
    T g = vb * dt / rhy, g0 = g, g1 = g, g2 = g;
    if (cx.on) g0 = pml_adj3(g0, a.mem[0] + cx.off, cx.b, cx.a, cx.kk);
    if (cy.on) g1 = pml_adj3(g1, a.mem[1] + cy.off, cy.b, cy.a, cy.kk);
    if (cz.on) g2 = pml_adj3(g2, a.mem[2] + cz.off, cz.b, cz.a, cz.kk);
    out[3] = g0;
    out[4] = g1;
    out[5] = g2;
  }
  // vz: i in [N+1, nx-N), j in [N+1, ny-N), k in [N, nz-N-1)
  if (i >= N + 1 && i < nx - N && j >= N + 1 && j < ny - N && k >= N && k < nz - N - 1) {
    const T r4 = (T)0.25 * (r00 + r01 + r11 + r10);
    const bool P = (fx & 1) || (fy & 1) || (fz & 2);
    auto cx = cpml3<T, 0>(p, 2, false, P, i, j, k);
    auto cy = cpml3<T, 1>(p, 2, false, P, i, j, k);
    auto cz = cpml3<T, 2>(p, 2, true, P, i, j, k);
    T d0 = dv[6], d1 = dv[7], d2 = dv[8];
    if (cx.on) d0 = pml_fwd3(d0, m0[cx.off], cx.b, cx.a, cx.kk);
    if (cy.on) d1 = pml_fwd3(d1, m1[cy.off], cy.b, cy.a, cy.kk);
    if (cz.on) d2 = pml_fwd3(d2, m2[cz.off], cz.b, cz.a, cz.kk);
    const T vb = a.f[2][idx];
    a.grad[2][idx] += vb * (d0 + d1 + d2) * dt;
    T g = vb * dt / r4, g0 = g, g1 = g, g2 = g;
    if (cx.on) g0 = pml_adj3(g0, a.mem[0] + cx.off, cx.b, cx.a, cx.kk);
    if (cy.on) g1 = pml_adj3(g1, a.mem[1] + cy.off, cy.b, cy.a, cy.kk);
    if (cz.on) g2 = pml_adj3(g2, a.mem[2] + cz.off, cz.b, cz.a, cz.kk);
    out[6] = g0;
    out[7] = g1;
    out[8] = g2;
  }
  divc_group<9>(out, hd, hr, p.fast_div);
#pragma unroll
  for (int q = 0; q < 9; ++q) a.tmp[q][idx] = out[q];
}

// sxx_bar += D+x^T t0; syy_bar += D+y^T t4; szz_bar += D+z^T t8;
// sxy_bar += D-y^T t1 + D-x^T t3; sxz_bar += D-z^T t2 + D-x^T t6; syz_bar += D-z^T t5 + D-y^T t7
template <typename T, int N>
__global__ void __launch_bounds__(B3Z * B3Y, SW_ADJ3_MINB)
k3a_str_gather(const __grid_constant__ P3<T> p, const __grid_constant__ A3<T> a) {
  CELL3
  (void)fx; (void)fy; (void)fz;
  a.f[3][idx] += d3t<T, N, true>(a.tmp[0], idx, sx, i, nx, c);
  a.f[4][idx] += d3t<T, N, true>(a.tmp[4], idx, sy, j, ny, c);
  a.f[5][idx] += d3t<T, N, true>(a.tmp[8], idx, 1, k, nz, c);
  a.f[6][idx] += d3t<T, N, false>(a.tmp[1], idx, sy, j, ny, c) + d3t<T, N, false>(a.tmp[3], idx, sx, i, nx, c);
  a.f[7][idx] += d3t<T, N, false>(a.tmp[2], idx, 1, k, nz, c) + d3t<T, N, false>(a.tmp[6], idx, sx, i, nx, c);
  a.f[8][idx] += d3t<T, N, false>(a.tmp[5], idx, 1, k, nz, c) + d3t<T, N, false>(a.tmp[7], idx, sy, j, ny, c);
}

#undef CELL3
#undef INNER3

// The point force (Elastic3D_SSG_CPML.py:245) adds t/rho[src], t = dt*w(it),
// to vz after the velocity phase; its adjoint leaves vz_bar as it is and adds
// -t*vz_bar/rho^2 to d misfit / d rho[src], kept as t*vz_bar in grad[0] (the
// slot whose coefficient is 1/rho of the same cell).  vz_bar here is the
// adjoint after the stress phase's gather.
template <typename T>
__global__ void k3a_force(const __grid_constant__ P3<T> p, const __grid_constant__ A3<T> a, int it) {
  const long long s = ((long long)p.si * p.ny + p.sj) * p.nz + p.sk;
  a.grad[0][s] += (p.dt * p.wav[it]) * a.f[2][s];
}

template <typename T, int N>
static cudaError_t adj3_step(const P3<T>& p, const A3<T>& a, int it, cudaStream_t st) {
  dim3 block(B3Z, B3Y);
  dim3 grid((p.nz + B3Z - 1) / B3Z, (p.ny + B3Y - 1) / B3Y, p.nx);
  if (p.nrec > 0) k3a_record<T><<<(p.nrec + 255) / 256, 256, 0, st>>>(p, a, it);
  k3a_stress_mid<T, N><<<grid, block, 0, st>>>(p, a);
  k3a_vel_gather<T, N><<<grid, block, 0, st>>>(p, a);
  if (p.src_kind == SW_SRC_FORCE) k3a_force<T><<<1, 1, 0, st>>>(p, a, it);
  k3a_vel_mid<T, N><<<grid, block, 0, st>>>(p, a);
  k3a_str_gather<T, N><<<grid, block, 0, st>>>(p, a);
  return cudaGetLastError();
}

template <typename T>
cudaError_t sw3_adjoint_step(const P3<T>& p, const A3<T>& a, int order, int it, cudaStream_t st) {
  switch (order) {
    case 1: return adj3_step<T, 1>(p, a, it, st);
    case 2: return adj3_step<T, 2>(p, a, it, st);
    case 3: return adj3_step<T, 3>(p, a, it, st);
    case 4: return adj3_step<T, 4>(p, a, it, st);
    default: return cudaErrorInvalidValue;
  }
}

template cudaError_t sw3_adjoint_step<float>(const P3<float>&, const A3<float>&, int, int, cudaStream_t);
template cudaError_t sw3_adjoint_step<double>(const P3<double>&, const A3<double>&, int, int, cudaStream_t);

}  // namespace sw
