// elastic2d_resident.cu -- 2D SSG_VS / SSG_SV time loops that stay on the chip
// (src/Elastic2D_CPML.py:128-275): one cooperative launch runs all steps.
// (Waves of a batch's shots side by side in one launch measured 0.98-1.03x the
// batch's own two launches per step, so batches keep those.)
//
// What bounds the two-launch step is not memory but the chain of one short
// kernel after another: at 400 x 400 each of the two launches takes 6.2 us
// (latency of its dependent loads and of a cold instruction cache) for 0.7 us
// worth of HBM traffic.  Here a shot's grid is cut into one tile per block, one
// block per SM; a tile's wavefields, material coefficients and CPML memory
// variables live in shared memory for the whole run and only the N-cell rims
// travel, through L2.  Per step two exchanges are needed (velocities, then
// stresses).  A rim value travels as one 8-byte packet {value, tag} (a double
// as two), written and polled with single 8-byte accesses, so a packet
// validates itself: no fence, no flag and no grid barrier, one L2 trip per
// exchange.  A tile computes its rim cells first and sends them while it
// computes the inner ones.
//
// Packets of the velocity phase and of the stress phase have a buffer each.
// A tile overwrites its neighbour's velocity buffer of step t only after it
// has received that neighbour's stress rim of step t-1 (and the other way
// round), which the neighbour sent after it had read that buffer: two buffers
// are enough.  Tags count phases from 1; the inbox is zeroed before every
// launch, on its stream.
//
// Measured on B200 (us per step of 300, order 2, two launches per step from a
// graph -> on the chip): 60 x 64 8.6 -> 3.9, 200^2 9.2 -> 4.1, 400^2 10.9 -> 5.3,
// 700 x 400 14.8 -> 7.9, 1000 x 420 18.9 -> 9.9; float64 121 x 90 11.5 -> 4.1.
// What is left: two exchanges of about 1.2 us, instruction issue (about 190
// warp instructions per 32 cells and phase, more in the slabs and where
// numerators are below 2^-100).  640 threads: 96 registers and no spills, 20
// warps; 512, 768 and 1024 threads measured 7-16% slower at 400^2.
//
// Every cell runs the expressions of vel2_cell / str2_cell (elastic2d.cu) in
// their order, so all paths give the same bits.
#include <algorithm>

#include "sw_device.cuh"
#include "sw_resident2d.cuh"
#include "sw_stencil2d.cuh"
#include "sw_tma.cuh"

namespace sw {

namespace {

// the two values of a rim cell: one 8-byte packet {value, tag} each (float) or
// two packets {half, tag} each (double), adjacent in the buffer
template <typename T>
struct Rim;
template <>
struct Rim<float> {
  static constexpr int WORDS = 2;
  static __device__ __forceinline__ void send(uint64_t* at, float a, float b, uint32_t tag) {
    const uint64_t t = (uint64_t)tag << 32;
    const uint64_t wa = t | __float_as_uint(a), wb = t | __float_as_uint(b);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(at), "l"(wa) : "memory");
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(at + 1), "l"(wb) : "memory");
  }
  static __device__ __forceinline__ bool poll(const uint64_t* at, uint32_t tag, float* a, float* b) {
    uint64_t wa, wb;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(wa) : "l"(at) : "memory");
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(wb) : "l"(at + 1) : "memory");
    *a = __uint_as_float((uint32_t)wa);
    *b = __uint_as_float((uint32_t)wb);
    return (uint32_t)(wa >> 32) == tag && (uint32_t)(wb >> 32) == tag;
  }
};
template <>
struct Rim<double> {
  static constexpr int WORDS = 4;
  static __device__ __forceinline__ void send(uint64_t* at, double a, double b, uint32_t tag) {
    const uint64_t t = (uint64_t)tag << 32;
    const uint64_t ba = (uint64_t)__double_as_longlong(a), bb = (uint64_t)__double_as_longlong(b);
    const uint64_t w[4] = {t | (ba & 0xffffffffull), t | (ba >> 32), t | (bb & 0xffffffffull), t | (bb >> 32)};
#pragma unroll
    for (int q = 0; q < 4; ++q) asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(at + q), "l"(w[q]) : "memory");
  }
  static __device__ __forceinline__ bool poll(const uint64_t* at, uint32_t tag, double* a, double* b) {
    uint64_t w[4];
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w[q]) : "l"(at + q) : "memory");
      ok = ok && (uint32_t)(w[q] >> 32) == tag;
    }
    *a = __longlong_as_double((long long)((w[1] << 32) | (w[0] & 0xffffffffull)));
    *b = __longlong_as_double((long long)((w[3] << 32) | (w[2] & 0xffffffffull)));
    return ok;
  }
};

// q / d for 0 <= q < 2^16, 0 < d < 2^16 and r = 1.f / d: the nearest integer
// below (q + 0.5) / d, whose distance from an integer is at least 1/(2d),
// far above the rounding error of the product
__device__ __forceinline__ int small_div(int q, float r) { return (int)(((float)q + 0.5f) * r); }

// 2N taps at shared-memory stride ST, sum_m c_m (t[N+m] - t[N-1-m]); FWD: the
// forward difference (taps -N+1 .. N), else the backward one (-N .. N-1)
template <typename T, int N, bool FWD, int ST>
__device__ __forceinline__ T sdiff(const T* f, const T (&c)[N]) {
  T v = 0;
#pragma unroll
  for (int m = 0; m < N; ++m) v += c[m] * (f[(FWD ? m + 1 : m) * ST] - f[-(FWD ? m : m + 1) * ST]);
  return v;
}

// divc_group for sums of taps: they are never -0 (they start from +0), so the
// spacings' correction needs no zero test (same bits)
__device__ __forceinline__ void spacing4(float (&x)[4], const float (&d)[2], const float (&r)[2], bool fast) {
  RangeAcc acc;
#pragma unroll
  for (int k = 0; k < 4; ++k) acc.add(x[k]);
  if (fast && acc.ok()) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = mk_core(x[k], d[k & 1], r[k & 1]);
  } else if (fast && acc.below_huge()) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = mk_div_any(x[k], d[k & 1], r[k & 1]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = div_c(x[k], d[k & 1], r[k & 1], 0);
  }
}
__device__ __forceinline__ void spacing4(double (&x)[4], const double (&d)[2], const double (&r)[2], bool fast) {
  RangeAccT<double> acc;
#pragma unroll
  for (int k = 0; k < 4; ++k) acc.add(x[k]);
  if (fast && acc.ok()) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = mk2_core(x[k], d[k & 1], r[k & 1]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = div_v(x[k], d[k & 1]);
  }
}
// The tiles' agreement at the end of a run: every tile keeps its new state, or
// none does.  w[0] counts the tiles that are through, w[1] is the decision, made
// once by the first of: the last tile to get there (keep), a tile whose rims
// did not come or that gave up waiting here (drop).  stop: see Res2.  Not
// inlined, and all of it in here: with anything more in the kernel's body the
// step loop is scheduled worse (400 x 400 5.01 -> 5.25 us per step).
enum : uint32_t { RUN_OPEN = 0, RUN_KEEP = 1, RUN_DROP = 2 };
__device__ __noinline__ int run_settle(uint64_t* word, bool through, int stop) {
  const uint32_t tiles = gridDim.x;
  through = through && (int)blockIdx.x != stop;
  uint32_t* const w = reinterpret_cast<uint32_t*>(word);
  uint32_t want = RUN_DROP;
  if (through) {
    want = RUN_KEEP;
    if (atomicAdd(w, 1u) != tiles - 1) {
      uint64_t t0 = 0;
      for (uint32_t n = 0;; ++n) {
        uint32_t d;
        asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(d) : "l"(w + 1) : "memory");
        if (d != RUN_OPEN) return d == RUN_KEEP;
        if ((n & 255) == 255) {
          const uint64_t t = global_ns();
          if (t0 == 0) t0 = t;
          else if (t - t0 > SW_WAIT_NS) break;
        }
      }
      want = RUN_DROP;
    }
  }
  const uint32_t was = atomicCAS(w + 1, RUN_OPEN, want);
  return (was == RUN_OPEN ? want : was) == RUN_KEEP;
}

// a cell's word: which components are updated, where the CPML corrects their
// derivatives (velocity phase: vx by x, by z, vz by x, by z; stress phase:
// normal by x, by z, shear by x, by z), source cell, row of the free-surface hook
enum : uint32_t {
  W_UX = 1u, W_UZ = 2u, W_UN = 4u, W_US = 8u, W_SRC = 16u, W_AEA = 32u,
  W_V = 1u << 8, W_S = 1u << 12  // first of four bits each
};

}  // namespace

template <typename T, int N, int SCHEME, int BZ, int NT>
__global__ void __launch_bounds__(NT, 1)
k2r_run(const __grid_constant__ Res2<T> rs, int it0, int nsteps, int aea) {
  constexpr bool VS = SCHEME == SW2D_SSG_VS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int n_own;

  // this block's tile
  const P2<T>& p = rs.shot;
  const int tiles_x = rs.tx, tiles_z = rs.tz;
  const int tile = blockIdx.x;
  const int tix = tile / tiles_z, tiz = tile % tiles_z;
  const int nx = p.nx, nz = p.nz;
  const int i0 = res2_cut_x(nx, p.lo[0], p.hi[0], tix, tiles_x), i1 = res2_cut_x(nx, p.lo[0], p.hi[0], tix + 1, tiles_x);
  const int j0 = res2_cut_z(nz, tiz, tiles_z), j1 = res2_cut_z(nz, tiz + 1, tiles_z);
  const int bx = i1 - i0, bz = j1 - j0, nc = bx * bz;
  const int tid = threadIdx.x;
  // neighbours: bit 0 x-lo, 1 x-hi, 2 z-lo, 3 z-hi
  const int sides = (tix > 0 ? 1 : 0) | (tix + 1 < tiles_x ? 2 : 0) | (tiz > 0 ? 4 : 0) | (tiz + 1 < tiles_z ? 8 : 0);

  // shared-memory layout (res2_smem in sw_resident2d.cuh)
  // A row holds its five fields side by side and a row of the material block
  // its seven coefficients, at fixed strides: every tap of a cell is at an
  // immediate offset from one address.
  constexpr int P = BZ + 2 * N, RS = 5 * P, MS = 7 * BZ;
  const int sxl = max(0, min(i1, p.lo[0]) - i0), sxh = max(0, i1 - max(i0, nx - p.hi[0]));  // slab rows: leading, trailing
  const int szl = max(0, min(j1, p.lo[1]) - j0), szh = max(0, j1 - max(j0, nz - p.hi[1]));
  const int nsx = sxl + sxh, nsz = szl + szh;
  T* const F = reinterpret_cast<T*>(smem_raw);  // [bx + 2N][vx vz sxx szz sxz][P], rims included
  // [bx][7][BZ]: rho of vx, of vz, their reciprocals, lam, lam + 2 mu, mu of sxz
  T* const M = F + (bx + 2 * N) * RS;
  T* const px = M + bx * MS;                    // [4][nsx][bz]
  T* const pz = px + 4 * nsx * bz;              // [4][bx][nsz]
  T* const cx = pz + 4 * bx * nsz;              // [8][bx]: b a kappa 1/kappa at integer, at half points
  T* const cz = cx + 8 * bx;                    // [8][bz]
  int2* const own = reinterpret_cast<int2*>(smem_raw + res2_align16((size_t)((unsigned char*)(cz + 8 * bz) - smem_raw)));
  uint32_t* const word = reinterpret_cast<uint32_t*>(own + SW_RES_RECV);  // [bx][BZ]

  T c[N];
#pragma unroll
  for (int m = 0; m < N; ++m) c[m] = p.c[m];
  const T dt = p.dt;
  const T hd[2] = {p.dx, p.dz}, hr[2] = {p.rd[0], p.rd[1]};
  // float: the spacings' correction is verified; double: mk2_core's range
  const bool fast = sizeof(T) == 4 ? (p.fast_div & 1) != 0 : mk2_divisor(hd[0]) && mk2_divisor(hd[1]);
  bool mk2 = true;  // every density and kappa of the tile is in mk2_core's range
  const float rbz = 1.f / (float)bz;

  // A warp updates 32 consecutive columns of a row (a unit): its shared-memory
  // accesses are free of bank conflicts and what depends on the row is uniform.
  // The rim rows come first, so that their packets leave early.
  const int lane = tid & 31, wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
  constexpr int cols = BZ / 32;
  const int units = bx * cols;
  auto unit_row = [&](int u) {
    const int r = cols == 1 ? u : u / cols;
    return r < N ? r : (r < 2 * N ? bx - 2 * N + r : r - N);
  };
  auto unit_col = [&](int u) { return (cols == 1 ? 0 : (u % cols) * 32) + lane; };

  // ---- load the tile -------------------------------------------------------
  if (tid == 0) n_own = 0;
  for (int q = tid; q < 8 * bx; q += NT) {
    const int row = q / bx, src = row < 4 ? min(row, 2) : min(row - 1, 5);  // rows 3 and 7: 1/kappa
    const T v = p.cf[0][src * nx + i0 + q % bx];
    cx[q] = (row & 3) == 3 ? (T)1 / v : v;
    if ((row & 3) == 3) mk2 = mk2 && mk2_divisor(v);
  }
  for (int q = tid; q < 8 * bz; q += NT) {
    const int row = q / bz, src = row < 4 ? min(row, 2) : min(row - 1, 5);
    const T v = p.cf[1][src * nz + j0 + q % bz];
    cz[q] = (row & 3) == 3 ? (T)1 / v : v;
    if ((row & 3) == 3) mk2 = mk2 && mk2_divisor(v);
  }
  const bool moment = p.src_kind == SW_SRC_MOMENT;
  {
    // the stresses come with their rims; the first step's free-surface hook
    // and moment source precede it
    const T w = moment ? p.wav[it0] : (T)0;
    for (int q = tid; q < (bx + 2 * N) * P; q += NT) {
      const int r = q / P, s = q % P;
      const int i = i0 + r - N, j = j0 + s - N;
      const bool cross = (r >= N && r < N + bx) || (s >= N && s < N + bz);
      const bool in = cross && i >= 0 && i < nx && j >= 0 && j < nz;
      const bool mine = r >= N && r < N + bx && s >= N && s < N + bz;
      const long long g = (long long)i * nz + j;
      T v[5];
#pragma unroll
      for (int f = 0; f < 5; ++f) v[f] = (f >= 2 ? in : mine) ? p.f[f][g] : (T)0;
      if (aea && in && i == N) v[2] = (T)0;
      if (moment && in && i == p.si && j == p.sk) {
        v[2] = v[2] + w * p.mneg[0];
        v[3] = v[3] + w * p.mneg[1];
        v[4] = v[4] + w * p.mneg[2];
      }
#pragma unroll
      for (int f = 0; f < 5; ++f) F[r * RS + f * P + s] = v[f];
    }
  }
  const bool force = p.src_kind == SW_SRC_FORCE;
  for (int q = tid; q < nc; q += NT) {
    const int li = q / bz, lj = q % bz, i = i0 + li, j = j0 + lj;
    const bool in_i = i >= N + 1 && i < nx - N, in_j = j >= N + 1 && j < nz - N;
    const bool b_i = i >= N && i < nx - N - 1, b_j = j >= N && j < nz - N - 1;
    const bool ux = (VS ? in_i : b_i) && in_j, uz = (VS ? b_i : in_i) && b_j;
    const bool un = (VS ? b_i : in_i) && in_j, us = in_i && (VS ? b_j : in_j);
    const int fx = p.fl[0][i], fz = p.fl[1][j];
    const bool sx = li < sxl || li >= bx - sxh, sz = lj < szl || lj >= bz - szh;
    // vx and the shear stress sit at integer x points in VS, at half points in
    // SV, vz and the normal stresses the other way round; vx and the normal
    // stresses at integer z points, vz and the shear stress at half points
    const bool px0 = ux && ((fx & (VS ? 1 : 2)) || (fz & 1)), px1 = uz && ((fx & (VS ? 2 : 1)) || (fz & 2));
    const bool pn = un && ((fx & (VS ? 2 : 1)) || (fz & 1)), pq = us && ((fx & (VS ? 1 : 2)) || (fz & 2));
    uint32_t w = (ux ? W_UX : 0u) | (uz ? W_UZ : 0u) | (un ? W_UN : 0u) | (us ? W_US : 0u);
    w |= (px0 && sx ? W_V : 0u) | (px0 && sz ? 2 * W_V : 0u) | (px1 && sx ? 4 * W_V : 0u) | (px1 && sz ? 8 * W_V : 0u);
    w |= (pn && sx ? W_S : 0u) | (pn && sz ? 2 * W_S : 0u) | (pq && sx ? 4 * W_S : 0u) | (pq && sz ? 8 * W_S : 0u);
    if (p.src_kind != SW_SRC_NONE && i == p.si && j == p.sk) w |= W_SRC;
    if (aea && i == N) w |= W_AEA;
    word[li * BZ + lj] = w;
    const int ip = min(i + 1, nx - 1), jp = min(j + 1, nz - 1);
    const long long g00 = (long long)i * nz + j, g01 = (long long)i * nz + jp, g10 = (long long)ip * nz + j,
                    g11 = (long long)ip * nz + jp;
    const T r00 = p.rho[g00], r01 = p.rho[g01], r10 = p.rho[g10], r11 = p.rho[g11];
    const T l0 = p.lam[g00], u0 = p.mu[g00];
    T rx, rz, lm, lpm, ms;
    if (VS) {
      rx = r00;
      rz = (T)0.25 * (r00 + r01 + r11 + r10);
      lm = (T)0.5 * (l0 + p.lam[g10]);
      const T mh = (T)0.5 * (u0 + p.mu[g10]);
      lpm = lm + (T)2 * mh;
      ms = (T)0.5 * (p.mu[g01] + u0);
    } else {
      rx = (r00 + r10) / (T)2;
      rz = (T)0.5 * (r00 + r01);
      lm = l0;
      lpm = l0 + (T)2 * u0;
      ms = (T)0.25 * (p.mu[g01] + u0 + p.mu[g11] + p.mu[g10]);
    }
    mk2 = mk2 && mk2_divisor(rx) && mk2_divisor(rz);
    const T m[7] = {rx, rz, (T)1 / rx, (T)1 / rz, lm, lpm, ms};
#pragma unroll
    for (int f = 0; f < 7; ++f) M[li * MS + f * BZ + lj] = m[f];
  }
  for (int q = tid; q < 4 * nsx * bz; q += NT) {
    const int cm = q / (nsx * bz), r = (q / bz) % nsx, lj = q % bz;
    const int li = r < sxl ? r : bx - nsx + r;
    px[q] = *mx(p, cm, slab_index(i0 + li, nx, p.lo[0], p.hi[0]), j0 + lj);
  }
  for (int q = tid; q < 4 * bx * nsz; q += NT) {
    const int cm = q / (bx * nsz), li = (q / nsz) % bx, s = q % nsz;
    const int lj = s < szl ? s : bz - nsz + s;
    pz[q] = *mz(p, cm, i0 + li, slab_index(j0 + lj, nz, p.lo[1], p.hi[1]));
  }
  mk2 = __syncthreads_and(mk2) != 0;
  // this tile's receivers; a table that overflows is scanned in every step
  const int nrec = p.nrec;
  auto local_of = [&](long long g) {
    const int i = (int)(g / nz), j = (int)(g % nz);
    return i >= i0 && i < i1 && j >= j0 && j < j1 ? (i - i0 + N) * RS + (j - j0 + N) : -1;
  };
  for (int r = tid; r < nrec; r += NT) {
    const int o = local_of(p.rec_idx[r]);
    if (o >= 0) {
      const int at = atomicAdd(&n_own, 1);
      if (at < SW_RES_RECV) own[at] = make_int2(r, o);
    }
  }
  __syncthreads();
  const int n_rec = n_own;

  // rim cells received: N rows of bz on the x sides (lo, hi), then bx rows of
  // N on the z sides (lo, hi)
  const int nrim = 2 * N * (bx + bz);
  constexpr int W = Rim<T>::WORDS;
  auto buffer = [&](int t, int phase) { return rs.inbox + ((long long)t * 2 + phase) * rs.stride; };
  const int bz_lo = j0 - res2_cut_z(nz, max(tiz - 1, 0), tiles_z);  // columns of the z neighbours
  const int bz_hi = res2_cut_z(nz, min(tiz + 2, tiles_z), tiles_z) - j1;
  // Send new values where a neighbour's rim needs them.  The rows of the x rims
  // go out whole, as their warp has computed them; the columns of the z rims
  // after the phase, 32 of their cells to a warp.  The stress phase's first
  // value is sxx for the x sides, szz for the z sides.
  auto send_row = [&](int phase, int li, int lj, T a, T b, uint32_t tag) {
    if ((sides & 1) && li < N)  // the lower x neighbour's hi rim
      Rim<T>::send(buffer(tile - tiles_z, phase) + (N * bz + li * bz + lj) * W, a, b, tag);
    if ((sides & 2) && li >= bx - N)
      Rim<T>::send(buffer(tile + tiles_z, phase) + ((li - (bx - N)) * bz + lj) * W, a, b, tag);
  };
  auto send_columns = [&](int phase, uint32_t tag) {
    for (int q = tid; q < 2 * N * bx; q += NT) {
      const int hi = q >= N * bx, e = q - hi * N * bx, li = e / N, c = e % N;
      if (!(sides & (hi ? 8 : 4))) continue;
      const T* f = F + (li + N) * RS + N + (hi ? bz - N + c : c);
      // the upper z neighbour's lo rim, or the lower one's hi rim
      uint64_t* to = hi ? buffer(tile + 1, phase) + (2 * N * bz_hi + e) * W
                        : buffer(tile - 1, phase) + (2 * N * bz_lo + N * bx + e) * W;
      Rim<T>::send(to, f[(phase ? 3 : 0) * P], f[(phase ? 4 : 1) * P], tag);
    }
  };
  // poll this tile's rim packets of a phase into the rims of its fields;
  // false once a packet has not come for SW_WAIT_NS
  auto receive = [&](int phase, uint32_t tag) {
    const uint64_t* b = buffer(tile, phase);
    for (int q = tid; q < nrim; q += NT) {
      int side, off;
      if (q < 2 * N * bz) {
        const int r = small_div(q, rbz);
        side = r < N ? 0 : 1;
        off = (r < N ? r : r + bx) * RS + N + (q - r * bz);
      } else {
        int e = q - 2 * N * bz;
        side = e < N * bx ? 2 : 3;
        if (side == 3) e -= N * bx;
        const int li = e / N, s = e % N;
        off = (li + N) * RS + (side == 2 ? s : s + N + bz);
      }
      if (!((sides >> side) & 1)) continue;
      T va, vb;
      uint64_t t0 = 0;
      for (uint32_t n = 0; !Rim<T>::poll(b + q * W, tag, &va, &vb); ++n)
        if ((n & 255) == 255) {  // the timer is far slower to read than a packet
          const uint64_t t = global_ns();
          if (t0 == 0) t0 = t;
          else if (t - t0 > SW_WAIT_NS) return false;
        }
      const int fa = phase == 0 ? 0 : (side < 2 ? 2 : 3), fb = phase == 0 ? 1 : 4;
      F[fa * P + off] = va;
      F[fb * P + off] = vb;
    }
    return true;
  };
  // CPML correction of a cell's derivatives sd (x, z of the first component,
  // x, z of the second; memory variables cm and cm + 1 of each axis), as pml2
  // gives it; on: the four bits of the cell's word; hx: the first component
  // sits at half x points (the second at integer ones, or the other way
  // round); the first sits at integer, the second at half z points
  auto correct = [&](uint32_t on, int li, int lj, int cm, bool hx, T(&sd)[4]) {
    if (on & 5u) {
      const int xr = li < sxl ? li : li - (bx - nsx);
      const T* t0 = cx + (hx ? 4 : 0) * bx + li;
      const T* t1 = cx + (hx ? 0 : 4) * bx + li;
      T* m0 = px + (cm * nsx + xr) * bz + lj;
      T* m1 = m0 + nsx * bz;
      T x[2] = {on & 1u ? sd[0] : (T)0, on & 4u ? sd[2] : (T)0};
      const T n0 = t0[0] * *m0 + t0[bx] * sd[0], n1 = t1[0] * *m1 + t1[bx] * sd[2];
      const T kd[2] = {t0[2 * bx], t1[2 * bx]}, ky[2] = {t0[3 * bx], t1[3 * bx]};
      cell_quotients<2>(x, kd, ky, mk2);
      if (on & 1u) {
        *m0 = n0;
        sd[0] = x[0] + n0;
      }
      if (on & 4u) {
        *m1 = n1;
        sd[2] = x[1] + n1;
      }
    }
    if (on & 10u) {
      const int zr = lj < szl ? lj : lj - (bz - nsz);
      const T* t = cz + lj;
      T* m0 = pz + (cm * bx + li) * nsz + zr;
      T* m1 = m0 + bx * nsz;
      T x[2] = {on & 2u ? sd[1] : (T)0, on & 8u ? sd[3] : (T)0};
      const T n0 = t[0] * *m0 + t[bz] * sd[1], n1 = t[4 * bz] * *m1 + t[5 * bz] * sd[3];
      const T kd[2] = {t[2 * bz], t[6 * bz]}, ky[2] = {t[3 * bz], t[7 * bz]};
      cell_quotients<2>(x, kd, ky, mk2);
      if (on & 2u) {
        *m0 = n0;
        sd[1] = x[0] + n0;
      }
      if (on & 8u) {
        *m1 = n1;
        sd[3] = x[1] + n1;
      }
    }
  };

  bool ok = true;
  for (int s = 0; s < nsteps; ++s) {
    const int it = it0 + s;
    // ---- velocities (vel2_cell) ---------------------------------------------
    const uint32_t tv = 2 * s + 1, ts = 2 * s + 2;
    for (int u = wid; u < units; u += NT / 32) {
      const int li = unit_row(u), lj = unit_col(u);
      if (lj >= bz) continue;
      T* const f = F + (li + N) * RS + lj + N;
      const T* const m = M + li * MS + lj;
      const uint32_t w = word[li * BZ + lj];
      const bool ux = w & W_UX, uz = w & W_UZ;
      T sd[4];
      sd[0] = sdiff<T, N, !VS, RS>(f + 2 * P, c);    // sxx along x
      sd[1] = sdiff<T, N, false, 1>(f + 4 * P, c);   // sxz along z
      sd[2] = sdiff<T, N, VS, RS>(f + 4 * P, c);     // sxz along x
      sd[3] = sdiff<T, N, true, 1>(f + 3 * P, c);    // szz along z
      if (!ux) sd[0] = sd[1] = (T)0;
      if (!uz) sd[2] = sd[3] = (T)0;
      spacing4(sd, hd, hr, fast);
      if (w & (15 * W_V)) correct((w / W_V) & 15u, li, lj, 0, !VS, sd);
      const T rd[2] = {m[0], m[BZ]}, ry[2] = {m[2 * BZ], m[3 * BZ]};
      T tq[2] = {(sd[0] + sd[1]) * dt, (sd[3] + sd[2]) * dt};
      cell_quotients<2>(tq, rd, ry, mk2);
      T a = f[0], b = f[P];
      if (ux) a = a + tq[0];
      if (uz) b = b + tq[1];
      if ((w & W_SRC) && force) {
        T t = dt * p.wav[it];
        t = div_v(t, ldg(p.rho + (long long)p.si * nz + p.sk));
        if (VS) b = b + t;
        else a = a + t;
      }
      f[0] = a;
      f[P] = b;
      if (li < N || li >= bx - N) send_row(0, li, lj, a, b, tv);
    }
    __syncthreads();
    send_columns(0, tv);
    if (!receive(0, tv)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }

    // ---- receivers: the velocities are final ---------------------------------
    if (nrec > 0) {
      const T* rf = F + p.rec_field * P;
      if (n_rec <= SW_RES_RECV) {
        for (int r = tid; r < n_rec; r += NT)
          store_rec(p.rec_data, p.rec_f64, (long long)it * nrec + own[r].x, rf[own[r].y]);
      } else {
        for (int r = tid; r < nrec; r += NT) {
          const int o = local_of(p.rec_idx[r]);
          if (o >= 0) store_rec(p.rec_data, p.rec_f64, (long long)it * nrec + r, rf[o]);
        }
      }
    }

    // ---- stresses (str2_cell), then the next step's hook and source ----------
    const bool last = s == nsteps - 1;
    for (int u = wid; u < units; u += NT / 32) {
      const int li = unit_row(u), lj = unit_col(u);
      if (lj >= bz) continue;
      T* const f = F + (li + N) * RS + lj + N;
      const T* const m = M + li * MS + lj;
      const uint32_t w = word[li * BZ + lj];
      const bool un = w & W_UN, us = w & W_US;
      T sd[4];
      sd[0] = sdiff<T, N, VS, RS>(f, c);            // vx along x
      sd[1] = sdiff<T, N, false, 1>(f + P, c);      // vz along z
      sd[2] = sdiff<T, N, !VS, RS>(f + P, c);       // vz along x
      sd[3] = sdiff<T, N, true, 1>(f, c);           // vx along z
      if (!un) sd[0] = sd[1] = (T)0;
      if (!us) sd[2] = sd[3] = (T)0;
      spacing4(sd, hd, hr, fast);
      if (w & (15 * W_S)) correct((w / W_S) & 15u, li, lj, 2, VS, sd);
      T a = f[2 * P], b = f[3 * P], d = f[4 * P];
      const T lm = m[4 * BZ], lpm = m[5 * BZ], ms = m[6 * BZ];
      if (un) {
        a = a + (lpm * sd[0] + lm * sd[1]) * dt;
        b = b + (lpm * sd[1] + lm * sd[0]) * dt;
      }
      if (us) d = d + ms * (sd[3] + sd[2]) * dt;
      if ((w & (W_SRC | W_AEA)) && !last) {
        if (w & W_AEA) a = (T)0;
        if (moment && (w & W_SRC)) {
          const T wv = p.wav[it + 1];
          a = a + wv * p.mneg[0];
          b = b + wv * p.mneg[1];
          d = d + wv * p.mneg[2];
        }
      }
      f[2 * P] = a;
      f[3 * P] = b;
      f[4 * P] = d;
      if (!last && (li < N || li >= bx - N)) send_row(1, li, lj, a, d, ts);
    }
    if (!last) {
      __syncthreads();
      send_columns(1, ts);
      if (!receive(1, ts)) ok = false;
    }
    if (__syncthreads_or(!ok)) { ok = false; break; }
  }

  __shared__ int keep;
  if (tid == 0) keep = run_settle(rs.inbox + 2LL * gridDim.x * rs.stride, ok, rs.stop_tile);
  __syncthreads();
  if (keep == 0) {  // somewhere a rim never came: every tile leaves the caller's arrays as they were
    if (tid == 0) atomicOr(rs.err, 4);
    return;
  }
  for (int q = tid; q < nc; q += NT) {
    const int li = q / bz, lj = q % bz;
    const long long g = (long long)(i0 + li) * nz + j0 + lj;
#pragma unroll
    for (int f = 0; f < 5; ++f) p.f[f][g] = F[(li + N) * RS + f * P + lj + N];
  }
  for (int q = tid; q < 4 * nsx * bz; q += NT) {
    const int cm = q / (nsx * bz), r = (q / bz) % nsx, lj = q % bz;
    const int li = r < sxl ? r : bx - nsx + r;
    *mx(p, cm, slab_index(i0 + li, nx, p.lo[0], p.hi[0]), j0 + lj) = px[q];
  }
  for (int q = tid; q < 4 * bx * nsz; q += NT) {
    const int cm = q / (bx * nsz), li = (q / nsz) % bx, s = q % nsz;
    const int lj = s < szl ? s : bz - nsz + s;
    *mz(p, cm, i0 + li, slab_index(j0 + lj, nz, p.lo[1], p.hi[1])) = pz[q];
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

// Shot p cut into tx x tz tiles: the largest shared memory of a tile (0 when a
// side would be too short), its work per step in warp units, the 8-byte words
// of its rim buffer.
template <typename T>
size_t tile_smem(const P2<T>& p, int N, int tx, int tz, long long* work, int* words, int* width) {
  const int lim = std::max(2 * N, SW_RES_MIN);
  int bx = 0, bz = 0, nsx = 0, nsz = 0, wx = 0;
  for (int a = 0; a < tx; ++a) {
    const int i0 = res2_cut_x(p.nx, p.lo[0], p.hi[0], a, tx), i1 = res2_cut_x(p.nx, p.lo[0], p.hi[0], a + 1, tx);
    if (i1 - i0 < lim) return 0;
    const int ns = std::max(0, std::min(i1, p.lo[0]) - i0) + std::max(0, i1 - std::max(i0, p.nx - p.hi[0]));
    bx = std::max(bx, i1 - i0);
    nsx = std::max(nsx, ns);
    wx = std::max(wx, 2 * (i1 - i0) + ns);
  }
  for (int a = 0; a < tz; ++a) {
    const int j0 = res2_cut_z(p.nz, a, tz), j1 = res2_cut_z(p.nz, a + 1, tz);
    if (j1 - j0 < lim) return 0;
    const int ns = std::max(0, std::min(j1, p.lo[1]) - j0) + std::max(0, j1 - std::max(j0, p.nz - p.hi[1]));
    bz = std::max(bz, j1 - j0);
    nsz = std::max(nsz, ns);
  }
  // a row counts 32 (48 in an x slab) per 32 columns; a rim packet costs about
  // a third of a cell
  if (bz > 64) return SIZE_MAX;
  *width = bz <= 32 ? 32 : 64;
  *work = 16LL * wx * ((bz + 31) / 32) + (long long)N * (bx + bz) * 2 / 3;
  *words = 2 * N * (bx + bz) * Rim<T>::WORDS;
  return res2_smem(bx, bz, *width, nsx, nsz, N, (int)sizeof(T));
}

}  // namespace

// Tiles of up to SW_RES_FLOOR work all take the same time, that of an exchange
// and one unit's latency, so among those the split with the fewest tiles is
// taken: the SMs that it leaves are free for other solvers' runs.  One solver
// (us per step, tiles in brackets): float order 2 121 x 90 [110] 3.61, [30] 3.45,
// [18] 4.59; 200^2 [136] 3.46, [105] 3.58, [77] 3.75, [63] 4.65; order 4 200^2
// [136] 3.80, [91] 4.06; float64 order 4 121 x 90 [110] 4.74, [44] 4.64, [24] 6.04.
// Four solvers of 121 x 90 on streams of their own, us per step for all: 14.1
// with the least work per tile, 10.4 replayed, 3.7 with this rule.
template <typename T>
bool sw2r_tiles(const P2<T>& p, int N, int blocks, size_t smem, int* tx, int* tz, int* words,
                size_t* bytes, int* got) {
  if (N > SW_RES_ORDER) return false;
  long long best = -1;
  int tiles = 0;
  for (int b = 1; b <= blocks; ++b)
    for (int a = 1; a * b <= blocks; ++a) {
      long long work;
      int w, bw;
      const size_t s = tile_smem(p, N, a, b, &work, &w, &bw);
      if (s == 0) break;  // shorter rows only from here on
      if (work <= SW_RES_FLOOR) work = 0;
      if (s > smem || (best >= 0 && (work > best || (work == best && a * b >= tiles)))) continue;
      best = work;
      tiles = a * b;
      *tx = a;
      *tz = b;
      *words = w;
      *bytes = s;
      *got = bw;
    }
  return best >= 0;
}

template <typename T, int N, int S, int BZ>
static cudaError_t launch2r(const Res2<T>& rs, int it0, int nsteps, int aea, cudaStream_t st) {
  constexpr int NT = sizeof(T) == 4 ? 640 : 512;
  auto kern = k2r_run<T, N, S, BZ, NT>;
  static std::atomic<unsigned long long> done{0};
  static std::mutex mu;
  cudaError_t e = once_per_device(done, mu, [kern] {
    int dev = 0, lim = 0;
    cudaError_t q = cudaGetDevice(&dev);
    if (q == cudaSuccess) q = cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (q == cudaSuccess) q = cudaFuncGetAttributes(&fa, kern);
    if (q == cudaSuccess)
      q = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, lim - (int)fa.sharedSizeBytes);
    return q;
  });
  if (e != cudaSuccess) return e;
  Res2<T> r = rs;
  void* args[] = {&r, &it0, &nsteps, &aea};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(rs.tx * rs.tz), dim3(NT), args, rs.smem, st);
}

template <typename T, int S>
static cudaError_t order2r(const Res2<T>& rs, int order, int it0, int n, int aea, cudaStream_t st) {
#define SW_RES_CASE(n_) \
  case n_: return rs.width == 32 ? launch2r<T, n_, S, 32>(rs, it0, n, aea, st) : launch2r<T, n_, S, 64>(rs, it0, n, aea, st);
  switch (order) {
    SW_RES_CASE(1) SW_RES_CASE(2) SW_RES_CASE(3) SW_RES_CASE(4)
    default: return cudaErrorInvalidValue;
  }
#undef SW_RES_CASE
}

template <typename T>
cudaError_t sw2r_run(const Res2<T>& rs, int scheme, int order, int it0, int nsteps, int aea, cudaStream_t st) {
  const size_t words = res2_inbox_words(rs.tx, rs.tz, rs.stride);
  cudaError_t e = cudaMemsetAsync(rs.inbox, 0, words * sizeof(uint64_t), st);
  if (e != cudaSuccess) return e;
  return scheme == SW2D_SSG_VS ? order2r<T, SW2D_SSG_VS>(rs, order, it0, nsteps, aea, st)
                               : order2r<T, SW2D_SSG_SV>(rs, order, it0, nsteps, aea, st);
}

#define SW_RES_INST(T)                                                                          \
  template bool sw2r_tiles<T>(const P2<T>&, int, int, size_t, int*, int*, int*, size_t*, int*); \
  template cudaError_t sw2r_run<T>(const Res2<T>&, int, int, int, int, int, cudaStream_t);
SW_RES_INST(float)
SW_RES_INST(double)

}  // namespace sw
