// elastic3d_cpml.cu -- 3D SSG-CPML time step, one thread per cell, any order and
// type: float64, single steps of grids the staged kernels do not take, and the
// sizes and orders where it is the faster path (Elastic3D_SSG_Tensor.update_SSG,
// src/Elastic3D_SSG_Tensor.py:166-345; Elastic3D_SSG_CPML.update_SSG,
// src/Elastic3D_SSG_CPML.py:144-309).
//
//   k3_velocity  vx, vy, vz (+ point force)          reference :194-243 / :163-245
//   k3_stress    sxx syy szz, sxy, sxz, syz (+ receivers, + next step's
//                moment-tensor injection)              reference :245-310 / :246-309
//
// A cell is a chain of loads, a quotient group and a store per component, so
// what counts is how many cells are in flight: one thread per cell at 48 to 64
// warps per SM, taps from L1 and L2, against the form before it, which streamed
// x planes through per-thread register queues at 16 to 32 warps.  Measured (us
// per step, register queues at their best -> this): float64 order 2
// 128 x 120 x 112 327 -> 232, 60 x 60 x 64 58 -> 37, 200^3 1152 -> 859, order 4
// 520 -> 250; float 200^3 order 2 759 -> 573, order 3 814 -> 615, order 4 895 ->
// 636.  CPML memory variables are stored only on their slabs
// (sw_pml_axis.lo/hi): outside a slab the reference's update is the identity
// (a = 0, kappa = 1).
#include "sw_device.cuh"

namespace sw {

constexpr int T3Z = 32;
constexpr int T3Y = 8;
// Resident blocks per SM the kernels are compiled for (us per step with 5, 6,
// 8 blocks: float 200^3 order 2 638, 590, 573, order 3 623, 625, 615, order 4
// 657, 636, 669; float64 128 x 120 x 112 order 2 with 4, 5, 6, 8 252, 234, 232, 238)
#define SW_C3_MINB (sizeof(T) == 4 && N <= 3 ? 8 : 6)

template <typename T, int N, bool FWD>
__device__ __forceinline__ T d3c(const T* f, long long idx, long long st, const T* c) {
  T v = 0;
#pragma unroll
  for (int m = 0; m < N; ++m)
    v += FWD ? c[m] * (ldg(f + idx + (m + 1) * st) - ldg(f + idx - m * st))
             : c[m] * (ldg(f + idx + m * st) - ldg(f + idx - (m + 1) * st));
  return v;
}

// CPML correction of derivative d along axis AX (memory variable component
// comp, integer or half point) where the cell lies in the axis's slab
template <typename T, int AX, bool HALF>
__device__ __forceinline__ void cpml3c(const P3<T>& p, int comp, int s, int i, int j, int k, T& d) {
  const int n = AX == 0 ? p.nx : AX == 1 ? p.ny : p.nz, x = AX == 0 ? i : AX == 1 ? j : k;
  const T* cf = p.cf[AX] + (HALF ? CBH : CB) * n + x;
  const long long off = AX == 0   ? ((long long)s * p.ny + j) * p.nz + k
                        : AX == 1 ? ((long long)i * p.sn[1] + s) * p.nz + k
                                  : ((long long)i * p.ny + j) * p.sn[2] + s;
  T* m = p.mem[AX] + comp * p.mcomp[AX] + off;
  const T psi = cf[0] * (*m) + cf[n] * d;
  *m = psi;
  d = div_v(d, cf[2 * n]) + psi;
}

// LONG: the launch's first plane is x0 (each_slice), else N.  (As an argument of
// one kernel for both it cost the float kernels, which are at their register
// limit, 1 to 4% at 200^3.)
template <typename T, int N, bool TENSOR, bool LONG>
__global__ void __launch_bounds__(T3Z * T3Y, SW_C3_MINB)
k3_velocity(const __grid_constant__ P3<T> p, int it, int force_here, int x0) {
  const int k = blockIdx.x * T3Z + threadIdx.x;
  const int j = blockIdx.y * T3Y + threadIdx.y;
  const int i = blockIdx.z + (LONG ? x0 : N);
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  if (j < N || j >= ny - N || k < N || k >= nz - N) return;
  const long long sx = (long long)ny * nz, sy = nz;
  const long long idx = (long long)i * sx + (long long)j * nz + k;
  T c[N];
#pragma unroll
  for (int m = 0; m < N; ++m) c[m] = p.c[m];
  const T dt = p.dt;
  const T *sxx = p.f[3], *syy = p.f[4], *szz = p.f[5], *sxy = p.f[6], *sxz = p.f[7], *syz = p.f[8], *rho = p.rho;
  const int xi = slab_index(i, nx, p.lo[0], p.hi[0]), yj = slab_index(j, ny, p.lo[1], p.hi[1]),
            zk = slab_index(k, nz, p.lo[2], p.hi[2]);
  const uint8_t fx = p.fl[0][i], fy = p.fl[1][j], fz = p.fl[2][k];
  // vx: x half; i in [N, nx-N-1), j in [N+1, ny-N), k in [N+1, nz-N)
  if (i < nx - N - 1 && j >= N + 1 && k >= N + 1) {
    T a = d3c<T, N, true>(sxx, idx, sx, c), b = d3c<T, N, false>(sxy, idx, sy, c), d = d3c<T, N, false>(sxz, idx, 1, c);
    spacings<T, 0, 1, 2>(p, a, b, d);
    if ((fx & 2) || (fy & 1) || (fz & 1)) {
      if (xi >= 0) cpml3c<T, 0, true>(p, 0, xi, i, j, k, a);
      if (yj >= 0) cpml3c<T, 1, false>(p, 0, yj, i, j, k, b);
      if (zk >= 0) cpml3c<T, 2, false>(p, 0, zk, i, j, k, d);
    }
    T t = (a + d + b) * dt;
    p.f[0][idx] = p.f[0][idx] + div_v(t, ldg(rho + idx));
  }
  // vy: y half; i in [N+1, nx-N), j in [N, ny-N-1), k in [N+1, nz-N)
  if (i >= N + 1 && j < ny - N - 1 && k >= N + 1) {
    T a = d3c<T, N, false>(sxy, idx, sx, c), b = d3c<T, N, true>(syy, idx, sy, c), d = d3c<T, N, false>(syz, idx, 1, c);
    spacings<T, 0, 1, 2>(p, a, b, d);
    if ((fx & 1) || (fy & 2) || (fz & 1)) {
      if (xi >= 0) cpml3c<T, 0, false>(p, 1, xi, i, j, k, a);
      if (yj >= 0) cpml3c<T, 1, true>(p, 1, yj, i, j, k, b);
      if (zk >= 0) cpml3c<T, 2, false>(p, 1, zk, i, j, k, d);
    }
    T t = (a + b + d) * dt;
    p.f[1][idx] = p.f[1][idx] + div_v(t, (T)0.5 * (ldg(rho + idx) + ldg(rho + idx + sy)));
  }
  // vz: z half; i in [N+1, nx-N), j in [N+1, ny-N), k in [N, nz-N-1), then the
  // point force (Elastic3D_SSG_CPML.py:245)
  const bool upd = i >= N + 1 && j >= N + 1 && k < nz - N - 1;
  const bool src = force_here && i == p.si && j == p.sj && k == p.sk;
  if (upd || src) {
    T v = p.f[2][idx];
    if (upd) {
      T a = d3c<T, N, false>(sxz, idx, sx, c), b = d3c<T, N, false>(syz, idx, sy, c), d = d3c<T, N, true>(szz, idx, 1, c);
      spacings<T, 0, 1, 2>(p, a, b, d);
      if ((fx & 1) || (fy & 1) || (fz & 2)) {
        if (xi >= 0) cpml3c<T, 0, false>(p, 2, xi, i, j, k, a);
        if (yj >= 0) cpml3c<T, 1, false>(p, 2, yj, i, j, k, b);
        if (zk >= 0) cpml3c<T, 2, true>(p, 2, zk, i, j, k, d);
      }
      T t = (TENSOR ? (a + b + d) : (d + a + b)) * dt;
      v = v + div_v(t, (T)0.25 * (ldg(rho + idx) + ldg(rho + idx + sy) + ldg(rho + idx + sx + sy) + ldg(rho + idx + sx)));
    }
    if (src) {
      T t = dt * p.wav[it];
      v = v + div_v(t, ldg(rho + idx));
    }
    p.f[2][idx] = v;
  }
}

template <typename T, int N, bool LONG>
__global__ void __launch_bounds__(T3Z * T3Y, SW_C3_MINB)
k3_stress(const __grid_constant__ P3<T> p, int it, int inject_next, int x0) {
  {
    const long long b = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
    const long long n = (long long)gridDim.x * gridDim.y * gridDim.z * (T3Z * T3Y);
    for (long long r = b * (T3Z * T3Y) + threadIdx.y * T3Z + threadIdx.x; r < p.nrec; r += n)
      store_rec(p.rec_data, p.rec_f64, (long long)it * p.nrec + r, p.f[p.rec_field][p.rec_idx[r]]);
  }
  const int k = blockIdx.x * T3Z + threadIdx.x;
  const int j = blockIdx.y * T3Y + threadIdx.y;
  const int i = blockIdx.z + (LONG ? x0 : N);
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  if (j < N || j >= ny - N || k < N || k >= nz - N) return;
  const long long sx = (long long)ny * nz, sy = nz;
  const long long idx = (long long)i * sx + (long long)j * nz + k;
  T c[N];
#pragma unroll
  for (int m = 0; m < N; ++m) c[m] = p.c[m];
  const T dt = p.dt;
  const T *vx = p.f[0], *vy = p.f[1], *vz = p.f[2], *lam = p.lam, *mu = p.mu;
  const int xi = slab_index(i, nx, p.lo[0], p.hi[0]), yj = slab_index(j, ny, p.lo[1], p.hi[1]),
            zk = slab_index(k, nz, p.lo[2], p.hi[2]);
  const uint8_t fx = p.fl[0][i], fy = p.fl[1][j], fz = p.fl[2][k];
  const bool src = inject_next && i == p.si && j == p.sj && k == p.sk;
  const T wn = src ? p.wav[it + 1] : (T)0;
  // normal stresses: i, j, k in [N+1, n-N)
  const bool un = i >= N + 1 && j >= N + 1 && k >= N + 1;
  if (un || src) {
    T sa = p.f[3][idx], sb = p.f[4][idx], sc = p.f[5][idx];
    if (un) {
      T a = d3c<T, N, false>(vx, idx, sx, c), b = d3c<T, N, false>(vy, idx, sy, c), d = d3c<T, N, false>(vz, idx, 1, c);
      spacings<T, 0, 1, 2>(p, a, b, d);
      if ((fx | fy | fz) & 1) {
        if (xi >= 0) cpml3c<T, 0, false>(p, 3, xi, i, j, k, a);
        if (yj >= 0) cpml3c<T, 1, false>(p, 3, yj, i, j, k, b);
        if (zk >= 0) cpml3c<T, 2, false>(p, 3, zk, i, j, k, d);
      }
      const T lhx = (T)0.5 * (ldg(lam + idx) + ldg(lam + idx + sx));
      const T mhx = (T)0.5 * (ldg(mu + idx) + ldg(mu + idx + sx));
      const T lpm = lhx + (T)2 * mhx;
      sa = sa + (lpm * a + lhx * (d + b)) * dt;
      sb = sb + (lpm * b + lhx * (a + d)) * dt;
      sc = sc + (lpm * d + lhx * (a + b)) * dt;
    }
    if (src) {
      sa = sa + wn * p.mneg[0];
      sb = sb + wn * p.mneg[1];
      sc = sc + wn * p.mneg[2];
    }
    p.f[3][idx] = sa;
    p.f[4][idx] = sb;
    p.f[5][idx] = sc;
  }
  // sxy: i, j in [N+1, n-N), k in [N, nz-N)
  const bool uxy = i >= N + 1 && j >= N + 1;
  if (uxy || src) {
    T s = p.f[6][idx];
    if (uxy) {
      T a = d3c<T, N, true>(vy, idx, sx, c), b = d3c<T, N, true>(vx, idx, sy, c);
      spacings<T, 0, 1>(p, a, b);
      if ((fx & 2) || (fy & 2) || (fz & 1)) {
        if (xi >= 0) cpml3c<T, 0, true>(p, 4, xi, i, j, k, a);
        if (yj >= 0) cpml3c<T, 1, true>(p, 4, yj, i, j, k, b);
      }
      const T m4 = (T)0.25 * (ldg(mu + idx + sy) + ldg(mu + idx) + ldg(mu + idx) + ldg(mu + idx + sx));
      s = s + m4 * (b + a) * dt;
    }
    if (src) s = s + wn * p.mneg[3];
    p.f[6][idx] = s;
  }
  // sxz: i in [N, nx-N-1), j in [N, ny-N), k in [N, nz-N-1)
  const bool uxz = i < nx - N - 1 && k < nz - N - 1;
  if (uxz || src) {
    T s = p.f[7][idx];
    if (uxz) {
      T a = d3c<T, N, true>(vz, idx, sx, c), b = d3c<T, N, true>(vx, idx, 1, c);
      spacings<T, 0, 2>(p, a, b);
      if ((fx & 2) || (fy & 1) || (fz & 2)) {
        if (xi >= 0) cpml3c<T, 0, true>(p, 5, xi, i, j, k, a);
        if (zk >= 0) cpml3c<T, 2, true>(p, 4, zk, i, j, k, b);
      }
      const T m4 = (T)0.25 * (ldg(mu + idx) + ldg(mu + idx + sx) + ldg(mu + idx) + ldg(mu + idx + sy));
      s = s + m4 * (b + a) * dt;
    }
    if (src) s = s + wn * p.mneg[4];
    p.f[7][idx] = s;
  }
  // syz: i in [N, nx-N), j in [N, ny-N-1), k in [N, nz-N-1)
  const bool uyz = j < ny - N - 1 && k < nz - N - 1;
  if (uyz || src) {
    T s = p.f[8][idx];
    if (uyz) {
      T a = d3c<T, N, true>(vz, idx, sy, c), b = d3c<T, N, true>(vy, idx, 1, c);
      spacings<T, 1, 2>(p, a, b);
      if ((fx & 1) || (fy & 2) || (fz & 2)) {
        if (yj >= 0) cpml3c<T, 1, true>(p, 5, yj, i, j, k, a);
        if (zk >= 0) cpml3c<T, 2, true>(p, 5, zk, i, j, k, b);
      }
      const T m4 = (T)0.25 * (ldg(mu + idx + sy) + ldg(mu + idx) + ldg(mu + idx + 1) + ldg(mu + idx));
      s = s + m4 * (a + b) * dt;
    }
    if (src) s = s + wn * p.mneg[5];
    p.f[8][idx] = s;
  }
}

// ---------------------------------------------------------------------------
// Elastic3D_SSG_Tensor.py:186-193: sigma_ab[src] += w * (-M_ab)
template <typename T>
__global__ void k3_moment_inject(const __grid_constant__ P3<T> p, int it) {
  const long long s = ((long long)p.si * p.ny + p.sj) * p.nz + p.sk;
  const T w = p.wav[it];
#pragma unroll
  for (int a = 0; a < 6; ++a) p.f[3 + a][s] = p.f[3 + a][s] + w * p.mneg[a];
}

// vz[src] += dt*w/rho[src] for a source cell outside the velocity pass
template <typename T>
__global__ void k3_force_inject(const __grid_constant__ P3<T> p, int it) {
  const long long s = ((long long)p.si * p.ny + p.sj) * p.nz + p.sk;
  T t = p.dt * p.wav[it];
  t = div_v(t, p.rho[s]);
  p.f[2][s] = p.f[2][s] + t;
}

// receivers of a field written by the stress pass
template <typename T>
__global__ void k3_gather(const __grid_constant__ P3<T> p, int it) {
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < p.nrec) store_rec(p.rec_data, p.rec_f64, (long long)it * p.nrec + r, p.f[p.rec_field][p.rec_idx[r]]);
}

// ---------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------
// One x plane per blockIdx.z; the planes N .. nx-N-1 in launches of at most
// SW_GRID_Z planes, the limit of a grid's z extent.  The planes of a pass do not
// read what it writes.
template <typename T, int N, typename F>
static void each_slice(const P3<T>& p, F launch) {
  for (int x0 = N; x0 < p.nx - N; x0 += SW_GRID_Z) {
    const int planes = x0 + SW_GRID_Z < p.nx - N ? SW_GRID_Z : p.nx - N - x0;
    launch(dim3((p.nz + T3Z - 1) / T3Z, (p.ny + T3Y - 1) / T3Y, planes), x0);
  }
}

template <typename T, int N>
static void launch3_velocity(const P3<T>& p, int it, bool tensor, bool force_here, cudaStream_t st) {
  each_slice<T, N>(p, [&](dim3 grid, int x0) {
    const bool slices = p.nx - 2 * N > SW_GRID_Z;
    auto kern = tensor ? (slices ? k3_velocity<T, N, true, true> : k3_velocity<T, N, true, false>)
                       : (slices ? k3_velocity<T, N, false, true> : k3_velocity<T, N, false, false>);
    kern<<<grid, dim3(T3Z, T3Y), 0, st>>>(p, it, !tensor && force_here ? 1 : 0, x0);
  });
}

template <typename T, int N>
static void launch3_stress(const P3<T>& p, int it, bool inject_next, cudaStream_t st) {
  P3<T> q = p;
  each_slice<T, N>(p, [&](dim3 grid, int x0) {
    auto kern = p.nx - 2 * N > SW_GRID_Z ? k3_stress<T, N, true> : k3_stress<T, N, false>;
    kern<<<grid, dim3(T3Z, T3Y), 0, st>>>(q, it, inject_next ? 1 : 0, x0);
    q.nrec = 0;  // recorded by the first launch
  });
}

#define SW_ORDER_SWITCH(order, CALL)            \
  switch (order) {                              \
    case 1: { constexpr int NN = 1; CALL; break; } \
    case 2: { constexpr int NN = 2; CALL; break; } \
    case 3: { constexpr int NN = 3; CALL; break; } \
    case 4: { constexpr int NN = 4; CALL; break; } \
    case 5: { constexpr int NN = 5; CALL; break; } \
    case 6: { constexpr int NN = 6; CALL; break; } \
    case 7: { constexpr int NN = 7; CALL; break; } \
    case 8: { constexpr int NN = 8; CALL; break; } \
    default: return cudaErrorInvalidValue;      \
  }

// velocity pass of one step (force_here: the point force is added in-kernel)
template <typename T>
cudaError_t sw3_velocity(const P3<T>& p, int order, int it, bool tensor, bool force_here, cudaStream_t st) {
  SW_ORDER_SWITCH(order, (launch3_velocity<T, NN>(p, it, tensor, force_here, st)));
  return cudaGetLastError();
}

// stress pass of one step; p.nrec > 0 gathers receivers of a velocity field,
// inject_next adds the moment-tensor source of step it+1 at the end.
template <typename T>
cudaError_t sw3_stress(const P3<T>& p, int order, int it, bool inject_next, cudaStream_t st) {
  SW_ORDER_SWITCH(order, (launch3_stress<T, NN>(p, it, inject_next, st)));
  return cudaGetLastError();
}

template <typename T>
cudaError_t sw3_moment_inject(const P3<T>& p, int it, cudaStream_t st) {
  k3_moment_inject<T><<<1, 1, 0, st>>>(p, it);
  return cudaGetLastError();
}
template <typename T>
cudaError_t sw3_force_inject(const P3<T>& p, int it, cudaStream_t st) {
  k3_force_inject<T><<<1, 1, 0, st>>>(p, it);
  return cudaGetLastError();
}
// free-surface hook (Elastic3D_SSG_Tensor.py:160-163): szz = 0 on the z layer kz
template <typename T>
__global__ void k3_aea(T* szz, long long nxy, int nz, int kz) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c < nxy) szz[c * nz + kz] = (T)0;
}
template <typename T>
cudaError_t sw3_aea(const P3<T>& p, int kz, cudaStream_t st) {
  const long long nxy = (long long)p.nx * p.ny;
  k3_aea<T><<<(unsigned)((nxy + 255) / 256), 256, 0, st>>>(p.f[5], nxy, p.nz, kz);
  return cudaGetLastError();
}
template <typename T>
cudaError_t sw3_gather(const P3<T>& p, int it, cudaStream_t st) {
  if (p.nrec <= 0) return cudaSuccess;
  k3_gather<T><<<(p.nrec + 255) / 256, 256, 0, st>>>(p, it);
  return cudaGetLastError();
}

template cudaError_t sw3_velocity<float>(const P3<float>&, int, int, bool, bool, cudaStream_t);
template cudaError_t sw3_velocity<double>(const P3<double>&, int, int, bool, bool, cudaStream_t);
template cudaError_t sw3_stress<float>(const P3<float>&, int, int, bool, cudaStream_t);
template cudaError_t sw3_stress<double>(const P3<double>&, int, int, bool, cudaStream_t);
template cudaError_t sw3_moment_inject<float>(const P3<float>&, int, cudaStream_t);
template cudaError_t sw3_moment_inject<double>(const P3<double>&, int, cudaStream_t);
template cudaError_t sw3_force_inject<float>(const P3<float>&, int, cudaStream_t);
template cudaError_t sw3_force_inject<double>(const P3<double>&, int, cudaStream_t);
template cudaError_t sw3_aea<float>(const P3<float>&, int, cudaStream_t);
template cudaError_t sw3_aea<double>(const P3<double>&, int, cudaStream_t);
template cudaError_t sw3_gather<float>(const P3<float>&, int, cudaStream_t);
template cudaError_t sw3_gather<double>(const P3<double>&, int, cudaStream_t);

}  // namespace sw
