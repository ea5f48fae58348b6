// elastic3d_spml.cu -- 3D staggered-grid kernels with the split-field PML of
// src/Elastic3D_SSG_SPML.py:160-393 (update_SSG_SPML).
//
// Inside the PML predicate each component is advanced as split parts
//   psi_d <- ((1 - dt/2 d) psi_d + dt * term_d) / (1 + dt/2 d)
// and the field is set to their sum; outside it the plain update is used.
// The 24 split fields live only on the PML shell (split[24][scomp], cells
// ordered by shell_index); a cell whose axis predicates are all clear never
// touches them.  One thread per cell, block 32 (z) x 8 (y), one x plane per
// blockIdx.z.
#include "sw_device.cuh"

namespace sw {

// Resident blocks per SM the kernels are compiled for: one thread per cell
// waits on its loads (us per step with 4, 5, 6, 8 blocks: float 200^3 order 2
// 874, 780, 729, 622, order 4 897, 830, 812, 718; 100^3 order 4 107, 106, 107,
// 102).  Double with the compiler's own count, 2, 3, 4, 5: 160 x 150 x 101 order
// 2 569, 569, 466, 392, 355, order 8 935, 524, 423, 377, 360 (its own 139
// registers left one block on an SM); 60 x 60 x 61 order 3 43, 43, 38, 38, 38,
// order 8 62, 39, 40, 33, 37.
#define SW_KS_MINB (sizeof(T) == 4 ? 8 : 5)
constexpr int TSZ = 32;
constexpr int TSY = 8;

template <typename T, int N>
__device__ __forceinline__ T d_fm(const T* f, long long idx, long long s, const T* c) {
  T v = 0;
#pragma unroll
  for (int m = 0; m < N; ++m) v += c[m] * (ldg(f + idx + (m + 1) * s) - ldg(f + idx - m * s));
  return v;
}
template <typename T, int N>
__device__ __forceinline__ T d_bm(const T* f, long long idx, long long s, const T* c) {
  T v = 0;
#pragma unroll
  for (int m = 0; m < N; ++m) v += c[m] * (ldg(f + idx + m * s) - ldg(f + idx - (m + 1) * s));
  return v;
}

// one axis of a split update: w = 1 - dt/2 d, the divisor and its reciprocal
template <typename T>
struct Damp {
  T w, d, y;
};
template <typename T>
__device__ __forceinline__ Damp<T> damp_of(T damp, T hdt) {
  const T d = (T)1 + hdt * damp;
  return Damp<T>{(T)1 - hdt * damp, d, (T)1 / d};
}
// the parts' quotients as one group (div_v's bits)
template <typename T, int K>
__device__ __forceinline__ void split_quotients(T (&x)[K], const Damp<T> (&a)[K]) {
  T d[K], y[K];
  bool ok = true;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    d[k] = a[k].d;
    y[k] = a[k].y;
    ok = ok && mk2_divisor(d[k]);
  }
  cell_quotients<K>(x, d, y, ok);
}
// LONG: the launch's first plane is x0, else 0 (an argument of one kernel for
// both costs the float kernels up to 5%)
template <typename T, int N, bool LONG>
__global__ void __launch_bounds__(TSZ * TSY, SW_KS_MINB)
ks_velocity(const __grid_constant__ P3<T> p, int it, int src_here, int x0) {
  const int k = blockIdx.x * TSZ + threadIdx.x;
  const int j = blockIdx.y * TSY + threadIdx.y;
  const int i = blockIdx.z + (LONG ? x0 : 0);
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  if (j >= ny || k >= nz) return;
  const long long sx = (long long)ny * nz, sy = nz;
  const long long idx = (long long)i * sx + (long long)j * nz + k;
  const long long G = p.scomp;
  const T dt = p.dt;
  const T hdt = (T)0.5 * dt;
  T c[N];
#pragma unroll
  for (int m = 0; m < N; ++m) c[m] = p.c[m];
  const T *sxx = p.f[3], *syy = p.f[4], *szz = p.f[5], *sxy = p.f[6], *sxz = p.f[7], *syz = p.f[8];
  T *vx = p.f[0], *vy = p.f[1], *vz = p.f[2];
  T* sp = p.split;
  const T *rho = p.rho, *dpx = p.dmp[0], *dpy = p.dmp[1], *dpz = p.dmp[2];
  const uint8_t fx = p.fl[0][i], fy = p.fl[1][j], fz = p.fl[2][k];
  // every flagged index lies in its axis's slabs (checked when the plan is made)
  const long long sh = (fx | fy | fz) ? shell_index(p, i, j, k) : 0;

  // vx :182-205
  if (i >= N && i < nx - N - 1 && j >= N + 1 && j < ny - N && k >= N + 1 && k < nz - N) {
    T dsxxdx = d_fm<T, N>(sxx, idx, sx, c), dsxydy = d_bm<T, N>(sxy, idx, sy, c), dsxzdz = d_bm<T, N>(sxz, idx, 1, c);
    spacings<T, 0, 1, 2>(p, dsxxdx, dsxydy, dsxzdz);
    const T rh = ldg(rho + idx);
    const T ro = (T)1 / rh;
    if ((fx & 2) || (fy & 1) || (fz & 1)) {
      const Damp<T> x = damp_of(dpx[nx + i], hdt), y = damp_of(dpy[j], hdt), z = damp_of(dpz[k], hdt);
      T qa[3] = {x.w * sp[PVX_X * G + sh] + dsxxdx * dt * ro,
          y.w * sp[PVX_Y * G + sh] + dsxydy * dt * ro,
          z.w * sp[PVX_Z * G + sh] + dsxzdz * dt * ro};
      split_quotients<T, 3>(qa, {x, y, z});
      const T a = qa[0], b = qa[1], cc = qa[2];
      sp[PVX_X * G + sh] = a;
      sp[PVX_Y * G + sh] = b;
      sp[PVX_Z * G + sh] = cc;
      vx[idx] = a + b + cc;
    } else {
      vx[idx] = vx[idx] + (dsxxdx + dsxydy + dsxzdz) * dt * ro;
    }
  }
  // vy :209-233
  if (i >= N + 1 && i < nx - N && j >= N && j < ny - N - 1 && k >= N + 1 && k < nz - N) {
    const T rhy = (T)0.5 * (ldg(rho + idx) + ldg(rho + idx + sy));
    const T ro = (T)1 / rhy;
    T dsxydx = d_bm<T, N>(sxy, idx, sx, c), dsyydy = d_fm<T, N>(syy, idx, sy, c), dsyzdz = d_bm<T, N>(syz, idx, 1, c);
    spacings<T, 0, 1, 2>(p, dsxydx, dsyydy, dsyzdz);
    if ((fx & 1) || (fy & 2) || (fz & 1)) {
      const Damp<T> x = damp_of(dpx[i], hdt), y = damp_of(dpy[ny + j], hdt), z = damp_of(dpz[k], hdt);
      T qa[3] = {x.w * sp[PVY_X * G + sh] + dt * dsxydx * ro,
          y.w * sp[PVY_Y * G + sh] + dt * dsyydy * ro,
          z.w * sp[PVY_Z * G + sh] + dt * dsyzdz * ro};
      split_quotients<T, 3>(qa, {x, y, z});
      const T a = qa[0], b = qa[1], cc = qa[2];
      sp[PVY_X * G + sh] = a;
      sp[PVY_Y * G + sh] = b;
      sp[PVY_Z * G + sh] = cc;
      vy[idx] = a + b + cc;
    } else {
      vy[idx] = vy[idx] + (dsxydx + dsyydy + dsyzdz) * dt * ro;
    }
  }
  // vz :235-259, then the source :294
  const bool upd = i >= N + 1 && i < nx - N && j >= N + 1 && j < ny - N && k >= N && k < nz - N - 1;
  const bool src = src_here && i == p.si && j == p.sj && k == p.sk;
  if (upd || src) {
    T v = vz[idx];
    if (upd) {
      const T r4 = (T)0.25 * (ldg(rho + idx) + ldg(rho + idx + sy) + ldg(rho + idx + sx + sy) + ldg(rho + idx + sx));
      const T ro = (T)1 / r4;
      T dsxzdx = d_bm<T, N>(sxz, idx, sx, c), dsyzdy = d_bm<T, N>(syz, idx, sy, c), dszzdz = d_fm<T, N>(szz, idx, 1, c);
      spacings<T, 0, 1, 2>(p, dsxzdx, dsyzdy, dszzdz);
      if ((fx & 1) || (fy & 1) || (fz & 2)) {
        const Damp<T> x = damp_of(dpx[i], hdt), y = damp_of(dpy[j], hdt), z = damp_of(dpz[nz + k], hdt);
        T qa[3] = {x.w * sp[PVZ_X * G + sh] + dt * dsxzdx * ro,
            y.w * sp[PVZ_Y * G + sh] + dt * dsyzdy * ro,
            z.w * sp[PVZ_Z * G + sh] + dt * dszzdz * ro};
        split_quotients<T, 3>(qa, {x, y, z});
        const T a = qa[0], b = qa[1], cc = qa[2];
        sp[PVZ_X * G + sh] = a;
        sp[PVZ_Y * G + sh] = b;
        sp[PVZ_Z * G + sh] = cc;
        v = a + b + cc;
      } else {
        v = v + (dsxzdx + dsyzdy + dszzdz) * dt * ro;
      }
    }
    if (src) {
      T t = dt * p.wav[it];
      t = div_v(t, ldg(rho + idx));
      v = v + t;
    }
    vz[idx] = v;
  }
}

template <typename T, int N, bool LONG>
__global__ void __launch_bounds__(TSZ * TSY, SW_KS_MINB)
ks_stress(const __grid_constant__ P3<T> p, int it, int x0) {
  {
    const long long b = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
    const long long r = b * (TSZ * TSY) + threadIdx.y * TSZ + threadIdx.x;
    if (r < p.nrec) store_rec(p.rec_data, p.rec_f64, (long long)it * p.nrec + r, p.f[p.rec_field][p.rec_idx[r]]);
  }
  const int k = blockIdx.x * TSZ + threadIdx.x;
  const int j = blockIdx.y * TSY + threadIdx.y;
  const int i = blockIdx.z + (LONG ? x0 : 0);
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  if (j >= ny || k >= nz) return;
  const long long sx = (long long)ny * nz, sy = nz;
  const long long idx = (long long)i * sx + (long long)j * nz + k;
  const long long G = p.scomp;
  const T dt = p.dt;
  const T hdt = (T)0.5 * dt;
  T c[N];
#pragma unroll
  for (int m = 0; m < N; ++m) c[m] = p.c[m];
  const T *vx = p.f[0], *vy = p.f[1], *vz = p.f[2];
  T *sxx = p.f[3], *syy = p.f[4], *szz = p.f[5], *sxy = p.f[6], *sxz = p.f[7], *syz = p.f[8];
  T* sp = p.split;
  const T *lam = p.lam, *mu = p.mu, *dpx = p.dmp[0], *dpy = p.dmp[1], *dpz = p.dmp[2];
  const uint8_t fx = p.fl[0][i], fy = p.fl[1][j], fz = p.fl[2][k];
  // every flagged index lies in its axis's slabs (checked when the plan is made)
  const long long sh = (fx | fy | fz) ? shell_index(p, i, j, k) : 0;

  // normal stresses :296-333
  if (i >= N + 1 && i < nx - N && j >= N + 1 && j < ny - N && k >= N + 1 && k < nz - N) {
    const T lm = ldg(lam + idx), u = ldg(mu + idx);
    const T l2m = lm + (T)2 * u;
    T dvxdx = d_bm<T, N>(vx, idx, sx, c), dvydy = d_bm<T, N>(vy, idx, sy, c), dvzdz = d_bm<T, N>(vz, idx, 1, c);
    spacings<T, 0, 1, 2>(p, dvxdx, dvydy, dvzdz);
    if ((fx | fy | fz) & 1) {
      const Damp<T> x = damp_of(dpx[i], hdt), y = damp_of(dpy[j], hdt), z = damp_of(dpz[k], hdt);
      T qxx[3] = {x.w * sp[PSXX_X * G + sh] + dt * l2m * dvxdx,
          y.w * sp[PSXX_Y * G + sh] + dt * lm * dvydy,
          z.w * sp[PSXX_Z * G + sh] + dt * lm * dvzdz};
      split_quotients<T, 3>(qxx, {x, y, z});
      const T xx = qxx[0], xy = qxx[1], xz = qxx[2];
      T qyx[3] = {x.w * sp[PSYY_X * G + sh] + dt * lm * dvxdx,
          y.w * sp[PSYY_Y * G + sh] + dt * l2m * dvydy,
          z.w * sp[PSYY_Z * G + sh] + dt * lm * dvzdz};
      split_quotients<T, 3>(qyx, {x, y, z});
      const T yx = qyx[0], yy = qyx[1], yz = qyx[2];
      T qzx[3] = {x.w * sp[PSZZ_X * G + sh] + dt * lm * dvxdx,
          y.w * sp[PSZZ_Y * G + sh] + dt * lm * dvydy,
          z.w * sp[PSZZ_Z * G + sh] + dt * l2m * dvzdz};
      split_quotients<T, 3>(qzx, {x, y, z});
      const T zx = qzx[0], zy = qzx[1], zz = qzx[2];
      sp[PSXX_X * G + sh] = xx; sp[PSXX_Y * G + sh] = xy; sp[PSXX_Z * G + sh] = xz;
      sp[PSYY_X * G + sh] = yx; sp[PSYY_Y * G + sh] = yy; sp[PSYY_Z * G + sh] = yz;
      sp[PSZZ_X * G + sh] = zx; sp[PSZZ_Y * G + sh] = zy; sp[PSZZ_Z * G + sh] = zz;
      sxx[idx] = xx + xy + xz;
      syy[idx] = yx + yy + yz;
      szz[idx] = zx + zy + zz;
    } else {
      sxx[idx] = sxx[idx] + (l2m * dvxdx + lm * (dvzdz + dvydy)) * dt;
      syy[idx] = syy[idx] + (l2m * dvydy + lm * (dvxdx + dvzdz)) * dt;
      szz[idx] = szz[idx] + (l2m * dvzdz + lm * (dvxdx + dvydy)) * dt;
    }
  }
  // sxy :334-350
  if (i >= N + 1 && i < nx - N && j >= N + 1 && j < ny - N && k >= N && k < nz - N) {
    const T m4 = (T)0.25 * (ldg(mu + idx + sy) + ldg(mu + idx) + ldg(mu + idx) + ldg(mu + idx + sx));
    T dvydx = d_fm<T, N>(vy, idx, sx, c), dvxdy = d_fm<T, N>(vx, idx, sy, c);
    spacings<T, 0, 1>(p, dvydx, dvxdy);
    if ((fx & 2) || (fy & 2) || (fz & 1)) {
      const Damp<T> x = damp_of(dpx[nx + i], hdt), y = damp_of(dpy[ny + j], hdt);
      T qa[2] = {x.w * sp[PSXY_X * G + sh] + dt * m4 * dvydx,
          y.w * sp[PSXY_Y * G + sh] + dt * m4 * dvxdy};
      split_quotients<T, 2>(qa, {x, y});
      const T a = qa[0], b = qa[1];
      sp[PSXY_X * G + sh] = a;
      sp[PSXY_Y * G + sh] = b;
      sxy[idx] = a + b;
    } else {
      sxy[idx] = sxy[idx] + m4 * (dvxdy + dvydx) * dt;
    }
  }
  // sxz :352-371
  if (i >= N && i < nx - N - 1 && j >= N && j < ny - N && k >= N && k < nz - N - 1) {
    const T m4 = (T)0.25 * (ldg(mu + idx) + ldg(mu + idx + sx) + ldg(mu + idx) + ldg(mu + idx + sy));
    T dvzdx = d_fm<T, N>(vz, idx, sx, c), dvxdz = d_fm<T, N>(vx, idx, 1, c);
    spacings<T, 0, 2>(p, dvzdx, dvxdz);
    if ((fx & 2) || (fy & 1) || (fz & 2)) {
      const Damp<T> x = damp_of(dpx[nx + i], hdt), z = damp_of(dpz[nz + k], hdt);
      T qa[2] = {x.w * sp[PSXZ_X * G + sh] + dt * m4 * dvzdx,
          z.w * sp[PSXZ_Z * G + sh] + dt * m4 * dvxdz};
      split_quotients<T, 2>(qa, {x, z});
      const T a = qa[0], b = qa[1];
      sp[PSXZ_X * G + sh] = a;
      sp[PSXZ_Z * G + sh] = b;
      sxz[idx] = a + b;
    } else {
      sxz[idx] = sxz[idx] + m4 * (dvxdz + dvzdx) * dt;
    }
  }
  // syz :373-391
  if (i >= N && i < nx - N && j >= N && j < ny - N - 1 && k >= N && k < nz - N - 1) {
    const T m4 = (T)0.25 * (ldg(mu + idx + sy) + ldg(mu + idx) + ldg(mu + idx + 1) + ldg(mu + idx));
    T dvzdy = d_fm<T, N>(vz, idx, sy, c), dvydz = d_fm<T, N>(vy, idx, 1, c);
    spacings<T, 1, 2>(p, dvzdy, dvydz);
    if ((fx & 1) || (fy & 2) || (fz & 2)) {
      const Damp<T> y = damp_of(dpy[ny + j], hdt), z = damp_of(dpz[nz + k], hdt);
      T qa[2] = {y.w * sp[PSYZ_Y * G + sh] + dt * m4 * dvzdy,
          z.w * sp[PSYZ_Z * G + sh] + dt * m4 * dvydz};
      split_quotients<T, 2>(qa, {y, z});
      const T a = qa[0], b = qa[1];
      sp[PSYZ_Y * G + sh] = a;
      sp[PSYZ_Z * G + sh] = b;
      syz[idx] = a + b;
    } else {
      syz[idx] = syz[idx] + m4 * (dvydz + dvzdy) * dt;
    }
  }
}

template <typename T, int N>
static cudaError_t launch_spml(const P3<T>& p, int it, bool gather_in_stress, cudaStream_t st) {
  dim3 block(TSZ, TSY);
  // launches of at most SW_GRID_Z planes, the limit of a grid's z extent
  auto grid = [&](int x0) {
    return dim3((p.nz + TSZ - 1) / TSZ, (p.ny + TSY - 1) / TSY, x0 + SW_GRID_Z < p.nx ? SW_GRID_Z : p.nx - x0);
  };
  const bool slices = p.nx > SW_GRID_Z;
  auto velocity = slices ? ks_velocity<T, N, true> : ks_velocity<T, N, false>;
  auto stress = slices ? ks_stress<T, N, true> : ks_stress<T, N, false>;
  for (int x0 = 0; x0 < p.nx; x0 += SW_GRID_Z)
    velocity<<<grid(x0), block, 0, st>>>(p, it, p.src_kind != SW_SRC_NONE ? 1 : 0, x0);
  P3<T> q = p;
  if (!gather_in_stress) q.nrec = 0;
  for (int x0 = 0; x0 < p.nx; x0 += SW_GRID_Z) {
    stress<<<grid(x0), block, 0, st>>>(q, it, x0);
    q.nrec = 0;  // recorded by the first launch
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t sw3_spml_step(const P3<T>& p, int order, int it, bool gather_in_stress, cudaStream_t st) {
  switch (order) {
    case 1: return launch_spml<T, 1>(p, it, gather_in_stress, st);
    case 2: return launch_spml<T, 2>(p, it, gather_in_stress, st);
    case 3: return launch_spml<T, 3>(p, it, gather_in_stress, st);
    case 4: return launch_spml<T, 4>(p, it, gather_in_stress, st);
    case 5: return launch_spml<T, 5>(p, it, gather_in_stress, st);
    case 6: return launch_spml<T, 6>(p, it, gather_in_stress, st);
    case 7: return launch_spml<T, 7>(p, it, gather_in_stress, st);
    case 8: return launch_spml<T, 8>(p, it, gather_in_stress, st);
    default: return cudaErrorInvalidValue;
  }
}

template cudaError_t sw3_spml_step<float>(const P3<float>&, int, int, bool, cudaStream_t);
template cudaError_t sw3_spml_step<double>(const P3<double>&, int, int, bool, cudaStream_t);

}  // namespace sw
