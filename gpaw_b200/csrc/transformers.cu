// Restriction / interpolation (replaces _gpaw.Transformer: c/transformers.c,
// c/bmgs/restrict.c, c/bmgs/interpolate.c).
//
// The reference pads each band (c/bc.c), then runs three separable 1-D passes
// with a transpose after each (restrict.c:136-155, interpolate.c:227-257),
// i.e. four trips through memory per band.  Here one kernel does all three
// passes with one read of the input and one write of the output:
//   k >= 4, and k = 2 on unusual grids: blocks of a few output planes, axis 0
//     from global loads, axes 2 and 1 in shared memory
//   k = 2: one thread per coarse column, in-plane values straight from
//     global memory through L1, marching along axis 0
//   k = 2, periodic real rows of whole 16-byte chunks: the same march over
//     planes staged in shared memory
// Real FP64 results agree with the reference to rounding.
//
// Index conventions (single domain, gpaw/transformers.py:31-47):
//   restriction:   coarse local i  <-> fine local centre 2 i + off,
//                  off = 2 beg_out - beg_in (0 periodic, 1 zero boundary)
//   interpolation: fine local f has global index F = f + skip0; even F copies
//                  coarse global F/2, odd F = 2C+1 mixes coarse C-j, C+1+j;
//                  coarse local = global - cbeg (cbeg = beg_in).

#include <algorithm>
#include <cstring>
#include "internal.cuh"

namespace gb {

struct TrArgs {
  const void* in;
  void* out;
  const void* y;      // optional epilogue operand (interpolation)
  int64_t nbatch;
  int ni[3], no[3];   // input / output local sizes
  int pbc[3];
  int off[3];         // restriction centre offsets
  int skip0[3];       // interpolation parity offsets
  int cbeg[3];        // interpolation coarse begin
  int tiles1, tiles2;
  int nsteps;         // marching steps along axis 0 per column
  double alpha, gamma;
  PhaseSets phs;      // Bloch phases per k-point group of bands
  double w[4];        // midpoint weights for pairs at distance 1/2, 3/2, ...
};

__device__ __forceinline__ int tr_mod(int i, int n) {
  int r = i % n;
  return r < 0 ? r + n : r;
}

__device__ __forceinline__ int floor_div(int a, int b) {
  return (a >= 0) ? a / b : -((-a + b - 1) / b);
}

// ---------------------------------------------------------------- any k
// Restriction with k taps per axis, any geometry, boundary and element type.
// A CTA owns T1 x T2 points of IB coarse planes.  The axis-0 pass runs first,
// on values read straight from global memory (2 IB + k - 1 independent,
// coalesced loads per fine column, all boundary rules resolved there); the
// axis-2 and axis-1 passes follow in shared memory.  Nothing marches, so one
// small grid (the density's 112^3 -> 56^3) already fills the GPU: it is
// bound by L2 reads, (2 IB + k - 1) / 2 IB times the halo factor of the tile.
template <typename T_, int K_, int IB_, int T1_, int T2_>
struct RXCfg {
  using T = T_;
  static constexpr int K = K_, IB = IB_, T1 = T1_, T2 = T2_, NT = 256;
  static constexpr int FR = 2 * T1 + 2 * K - 3, FC = 2 * T2 + 2 * K - 3;
  static constexpr size_t SMEM = (size_t)IB * FR * (FC + T2) * sizeof(T);
};

// index i of an axis of n points: the wrapped index (periodic), or -1
__device__ __forceinline__ int tr_index(int i, int n, int pbc, int& side) {
  side = i < 0 ? 1 : i >= n ? 0 : -1;
  if (side < 0) return i;
  return pbc ? tr_mod(i, n) : -1;
}

template <class C>
__global__ void __launch_bounds__(C::NT) restrict_x_kernel(const __grid_constant__ TrArgs a) {
  using T = typename C::T;
  using R = typename Elem<T>::R;
  constexpr int K = C::K, IB = C::IB, T1 = C::T1, T2 = C::T2, FR = C::FR, FC = C::FC, KH = K / 2;
  constexpr int NO = IB + K - 1;                       // odd-offset planes
  constexpr bool CPLX = Elem<T>::cplx;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* X = reinterpret_cast<T*>(smem_raw);               // [IB][FR][FC]
  T* Z = X + IB * FR * FC;                             // [IB][FR][T2]
  const int nf0 = a.ni[0], nf1 = a.ni[1], nf2 = a.ni[2];
  const int nc0 = a.no[0], nc1 = a.no[1], nc2 = a.no[2];
  const int64_t nf12 = (int64_t)nf1 * nf2, nc12 = (int64_t)nc1 * nc2;
  unsigned t = blockIdx.x;
  const int K0 = (int)(t % a.tiles2) * T2;
  t /= a.tiles2;
  const int J0 = (int)(t % a.tiles1) * T1;
  t /= a.tiles1;
  const int I0 = (int)(t % a.nsteps) * IB;
  const int64_t band = t / a.nsteps;
  const T* __restrict__ src = reinterpret_cast<const T*>(a.in) + band * nf12 * nf0;
  T* __restrict__ dst = reinterpret_cast<T*>(a.out) + band * nc12 * nc0;
  const auto& PH = a.phs.ph[phase_set_of(a.phs, band)];
  const bool phased = CPLX && a.phs.any;
  R w[KH];
#pragma unroll
  for (int m = 0; m < KH; ++m) w[m] = (R)a.w[m];
  const R half = (R)0.5;
  const int j0 = 2 * I0 + a.off[0];                    // centre plane of coarse plane I0
  const int r0 = 2 * J0 + a.off[1] - (K - 1), c0 = 2 * K0 + a.off[2] - (K - 1);

  // fine plane j0 + d at an in-plane offset
  auto plane = [&](int d, int64_t off) -> T {
    int side;
    const int j = tr_index(j0 + d, nf0, a.pbc[0], side);
    T v = zero<T>();
    if (j >= 0) v = __ldg(src + j * nf12 + off);
    if (phased && side >= 0) v = phase_mul(v, PH[0][side][0], PH[0][side][1]);
    return v;
  };
  for (int e = threadIdx.x; e < FR * FC; e += C::NT) {
    const int r = e / FC, c = e - r * FC;
    int sy, sz;
    const int y = tr_index(r0 + r, nf1, a.pbc[1], sy), z = tr_index(c0 + c, nf2, a.pbc[2], sz);
    T x[IB];
#pragma unroll
    for (int i = 0; i < IB; ++i) x[i] = zero<T>();
    if (y >= 0 && z >= 0) {
      const int64_t off = (int64_t)y * nf2 + z;
      T ev[IB], od[NO];
#pragma unroll
      for (int i = 0; i < IB; ++i) ev[i] = plane(2 * i, off);
#pragma unroll
      for (int i = 0; i < NO; ++i) od[i] = plane(2 * i - (K - 1), off);
#pragma unroll
      for (int i = 0; i < IB; ++i) {
        T v = ev[i];
        // offsets +-(2m + 1) of plane 2i are odd planes i + KH + m and i + KH - 1 - m
#pragma unroll
        for (int m = 0; m < KH; ++m) v = fmadd(v, w[m], add(od[i + KH + m], od[i + KH - 1 - m]));
        x[i] = scale(half, v);
      }
      if (phased) {
        if (sy >= 0)
#pragma unroll
          for (int i = 0; i < IB; ++i) x[i] = phase_mul(x[i], PH[1][sy][0], PH[1][sy][1]);
        if (sz >= 0)
#pragma unroll
          for (int i = 0; i < IB; ++i) x[i] = phase_mul(x[i], PH[2][sz][0], PH[2][sz][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < IB; ++i) X[i * FR * FC + e] = x[i];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < IB * FR * T2; e += C::NT) {
    const int r = e / T2, k = e - r * T2;              // r counts the rows of all IB planes
    const T* f = X + r * FC + 2 * k + (K - 1);
    T v = f[0];
#pragma unroll
    for (int m = 0; m < KH; ++m) v = fmadd(v, w[m], add(f[2 * m + 1], f[-(2 * m + 1)]));
    Z[e] = scale(half, v);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < IB * T1 * T2; e += C::NT) {
    const int k = e % T2, r = (e / T2) % T1, i = e / (T1 * T2);
    const int I = I0 + i, J = J0 + r, kk = K0 + k;
    if (I >= nc0 || J >= nc1 || kk >= nc2) continue;
    const T* f = Z + (i * FR + 2 * r + (K - 1)) * T2 + k;
    T v = f[0];
#pragma unroll
    for (int m = 0; m < KH; ++m) v = fmadd(v, w[m], add(f[(2 * m + 1) * T2], f[-(2 * m + 1) * T2]));
    dst[I * nc12 + (int64_t)J * nc2 + kk] = scale((R)a.alpha, scale(half, v));
  }
}

// Interpolation, likewise: a CTA owns T1 x T2 fine points of the 2 IB fine
// planes of IB coarse planes; axis 0 from global loads, axes 2 and 1 in
// shared memory.  IB = 4 (8 in FP32) keeps the coarse planes read per cell, (IB
// + k - 1) / IB, near two; with IB = 1 every cell read all k: k = 6, 160 FP32
// grids of 35^3 to 71^3 470 us against 235, one FP64 grid of 56^3 to 112^3 14.7 against 13.3.
template <typename T_, int K_, int IB_, int T1_, int T2_>
struct IXCfg {
  using T = T_;
  static constexpr int K = K_, IB = IB_, T1 = T1_, T2 = T2_, NT = 256;
  static constexpr int CR = T1 / 2 + K, CC = T2 / 2 + K;
  static constexpr size_t SMEM = (size_t)2 * IB * CR * (CC + T2) * sizeof(T);
};

template <class C>
__global__ void __launch_bounds__(C::NT) interpolate_x_kernel(const __grid_constant__ TrArgs a) {
  using T = typename C::T;
  using R = typename Elem<T>::R;
  constexpr int K = C::K, IB = C::IB, T1 = C::T1, T2 = C::T2, CR = C::CR, CC = C::CC, KH = K / 2;
  constexpr int NP = IB + K - 1;                       // coarse planes read
  constexpr bool CPLX = Elem<T>::cplx;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* X = reinterpret_cast<T*>(smem_raw);               // [2 IB][CR][CC]
  T* Z = X + 2 * IB * CR * CC;                         // [2 IB][CR][T2]
  const int nc0 = a.ni[0], nc1 = a.ni[1], nc2 = a.ni[2];
  const int nf0 = a.no[0], nf1 = a.no[1], nf2 = a.no[2];
  const int64_t nc12 = (int64_t)nc1 * nc2, nf12 = (int64_t)nf1 * nf2;
  unsigned t = blockIdx.x;
  const int Z0 = (int)(t % a.tiles2) * T2;
  t /= a.tiles2;
  const int Y0 = (int)(t % a.tiles1) * T1;
  t /= a.tiles1;
  const int cells = (a.nsteps + IB - 1) / IB;
  const int C0 = floor_div(a.skip0[0], 2) + (int)(t % cells) * IB;   // first global coarse plane
  const int64_t band = t / cells;
  const T* __restrict__ src = reinterpret_cast<const T*>(a.in) + band * nc12 * nc0;
  T* __restrict__ dst = reinterpret_cast<T*>(a.out) + band * nf12 * nf0;
  const T* __restrict__ ysrc = a.y ? reinterpret_cast<const T*>(a.y) + band * nf12 * nf0 : nullptr;
  const auto& PH = a.phs.ph[phase_set_of(a.phs, band)];
  const bool phased = CPLX && a.phs.any;
  R w[KH];
#pragma unroll
  for (int m = 0; m < KH; ++m) w[m] = (R)a.w[m];
  // global coarse row / column of staged row / column 0
  const int crow0 = floor_div(Y0 + a.skip0[1], 2) - (KH - 1);
  const int ccol0 = floor_div(Z0 + a.skip0[2], 2) - (KH - 1);

  for (int e = threadIdx.x; e < CR * CC; e += C::NT) {
    const int r = e / CC, c = e - r * CC;
    int sy, sz;
    const int y = tr_index(crow0 + r - a.cbeg[1], nc1, a.pbc[1], sy);
    const int z = tr_index(ccol0 + c - a.cbeg[2], nc2, a.pbc[2], sz);
    T x[2 * IB];
#pragma unroll
    for (int i = 0; i < 2 * IB; ++i) x[i] = zero<T>();
    if (y >= 0 && z >= 0) {
      const int64_t off = (int64_t)y * nc2 + z;
      T p[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        int side;
        const int g = tr_index(C0 - (KH - 1) + i - a.cbeg[0], nc0, a.pbc[0], side);
        p[i] = zero<T>();
        if (g >= 0) p[i] = __ldg(src + g * nc12 + off);
        if (phased && side >= 0) p[i] = phase_mul(p[i], PH[0][side][0], PH[0][side][1]);
      }
#pragma unroll
      for (int i = 0; i < IB; ++i) {
        x[2 * i] = p[KH - 1 + i];
        T v = scale(w[0], add(p[KH - 1 + i], p[KH + i]));
#pragma unroll
        for (int m = 1; m < KH; ++m) v = fmadd(v, w[m], add(p[KH - 1 + i - m], p[KH + i + m]));
        x[2 * i + 1] = v;
      }
      if (phased) {
        if (sy >= 0)
#pragma unroll
          for (int i = 0; i < 2 * IB; ++i) x[i] = phase_mul(x[i], PH[1][sy][0], PH[1][sy][1]);
        if (sz >= 0)
#pragma unroll
          for (int i = 0; i < 2 * IB; ++i) x[i] = phase_mul(x[i], PH[2][sz][0], PH[2][sz][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * IB; ++i) X[i * CR * CC + e] = x[i];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * IB * CR * T2; e += C::NT) {
    const int r = e / T2, fc = e - r * T2;
    const int F = Z0 + fc + a.skip0[2];
    const T* f = X + r * CC + (floor_div(F, 2) - ccol0);
    T v = f[0];
    if (F & 1) {
      v = scale(w[0], add(f[0], f[1]));
#pragma unroll
      for (int m = 1; m < KH; ++m) v = fmadd(v, w[m], add(f[-m], f[1 + m]));
    }
    Z[e] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * IB * T1 * T2; e += C::NT) {
    const int c = e % T2, r = (e / T2) % T1, i = e / (T1 * T2);
    const int f0 = 2 * C0 + i - a.skip0[0], y = Y0 + r, z = Z0 + c;
    if (f0 < 0 || f0 >= nf0 || y >= nf1 || z >= nf2) continue;
    const int F = y + a.skip0[1];
    const T* f = Z + (i * CR + floor_div(F, 2) - crow0) * T2 + c;
    T v = f[0];
    if (F & 1) {
      v = scale(w[0], add(f[0], f[T2]));
#pragma unroll
      for (int m = 1; m < KH; ++m) v = fmadd(v, w[m], add(f[-m * T2], f[(1 + m) * T2]));
    }
    const int64_t o = f0 * nf12 + (int64_t)y * nf2 + z;
    v = scale((R)a.alpha, v);
    if (ysrc) v = fmadd(v, (R)a.gamma, __ldcs(ysrc + o));
    dst[o] = v;
  }
}

// ---------------------------------------------------------------- k = 2
// The preconditioner's transfers on grids whose axes each have the usual
// geometry (periodic: 2 n fine for n coarse points; zero boundary: 2 n + 1),
// whatever the row length, boundary mix, element type and phases.  One thread
// per coarse (axis 1, axis 2) column marches over a few coarse planes; its
// 3 x 3 (restriction) or 2 x 2 (interpolation) in-plane values come straight
// from global memory through L1, so there is no staging and no barrier.
// phase of a cell wrapped over two axes
__device__ __forceinline__ double2 corner_phase(const double (&p)[2], const double (&q)[2]) {
  return make_double2(__fma_rn(p[0], q[0], -__dmul_rn(p[1], q[1])), __fma_rn(p[0], q[1], __dmul_rn(p[1], q[0])));
}

template <typename T, bool PER>
__global__ void __launch_bounds__(256) restrict2_direct_kernel(const __grid_constant__ TrArgs a) {
  using R = typename Elem<T>::R;
  constexpr bool CPLX = Elem<T>::cplx;
  const int nf0 = a.ni[0], nf1 = a.ni[1], nf2 = a.ni[2];
  const int nc0 = a.no[0], nc1 = a.no[1], nc2 = a.no[2];
  const int64_t nf12 = (int64_t)nf1 * nf2, nc12 = (int64_t)nc1 * nc2;
  unsigned t = blockIdx.x;
  const int64_t f = (int64_t)(t % a.tiles1) * 256 + threadIdx.x;
  t /= a.tiles1;
  const int chunk = (int)(t % a.nsteps);
  const int64_t band = t / a.nsteps;
  int K;
  const int J = (int)div_mod(f, nc2, K);
  if (J >= nc1) return;
  const int I_beg = (int)((int64_t)nc0 * chunk / a.nsteps), I_end = (int)((int64_t)nc0 * (chunk + 1) / a.nsteps);
  const auto& PH = a.phs.ph[phase_set_of(a.phs, band)];
  const bool phased = CPLX && PER && a.phs.any;
  const R w0 = (R)a.w[0], half = (R)0.5;
  // fine neighbours of the centre (2J + off, 2K + off): only index -1 of a
  // periodic axis is outside the grid
  const bool wy = PER && a.pbc[1] && J == 0, wz = PER && a.pbc[2] && K == 0;
  const int oz = wz ? nf2 - 1 : -1;
  const int64_t oy = wy ? (int64_t)(nf1 - 1) * nf2 : -nf2;
  const T* __restrict__ p = reinterpret_cast<const T*>(a.in) + band * nf12 * nf0 +
                            (int64_t)(2 * J + a.off[1]) * nf2 + 2 * K + a.off[2];
  auto plane = [&](int j) -> T {
    const bool wx = PER && j < 0;
    const T* c = p + (int64_t)(wx ? j + nf0 : j) * nf12;
    T v[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const T* row = c + (d == 0 ? oy : d == 1 ? 0 : (int64_t)nf2);
      v[d][0] = __ldg(row + oz);
      v[d][1] = __ldg(row);
      v[d][2] = __ldg(row + 1);
    }
    if (phased) {
      // each wrapped cell by its own phase, the corner by the product
      if (wz) {
        v[1][0] = phase_mul(v[1][0], PH[2][1][0], PH[2][1][1]);
        v[2][0] = phase_mul(v[2][0], PH[2][1][0], PH[2][1][1]);
        if (!wy) v[0][0] = phase_mul(v[0][0], PH[2][1][0], PH[2][1][1]);
      }
      if (wy) {
        const double2 c = wz ? corner_phase(PH[1][1], PH[2][1]) : make_double2(PH[1][1][0], PH[1][1][1]);
        v[0][0] = phase_mul(v[0][0], c.x, c.y);
        v[0][1] = phase_mul(v[0][1], PH[1][1][0], PH[1][1][1]);
        v[0][2] = phase_mul(v[0][2], PH[1][1][0], PH[1][1][1]);
      }
    }
    T g[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) g[d] = scale(half, fmadd(v[d][1], w0, add(v[d][2], v[d][0])));
    T u = scale(half, fmadd(g[1], w0, add(g[2], g[0])));
    if (phased && wx) u = phase_mul(u, PH[0][1][0], PH[0][1][1]);
    return u;
  };
  T* __restrict__ o = reinterpret_cast<T*>(a.out) + band * nc12 * nc0 + I_beg * nc12 + (int64_t)J * nc2 + K;
  int j = 2 * I_beg + a.off[0];
  T um = plane(j - 1);
  for (int I = I_beg; I < I_end; ++I, j += 2, o += nc12) {
    const T uc = plane(j), up = plane(j + 1);
    *o = scale((R)a.alpha, scale(half, fmadd(uc, w0, add(up, um))));
    um = up;
  }
}

// One thread per (coarse row cell, fine column): its lanes write consecutive
// fine points (a thread per coarse cell wrote every other one, and took 1.4
// times as long on partial sectors).
template <typename T, bool PER>
__global__ void __launch_bounds__(256) interp2_direct_kernel(const __grid_constant__ TrArgs a) {
  using R = typename Elem<T>::R;
  constexpr bool CPLX = Elem<T>::cplx;
  const int nc0 = a.ni[0], nc1 = a.ni[1], nc2 = a.ni[2];
  const int nf0 = a.no[0], nf1 = a.no[1], nf2 = a.no[2];
  const int64_t nc12 = (int64_t)nc1 * nc2, nf12 = (int64_t)nf1 * nf2;
  // cells C (between coarse points C and C + 1, global numbering): one per
  // coarse point of a periodic axis, one more on a zero-boundary one
  const int m0 = nc0 + a.cbeg[0], m1 = nc1 + a.cbeg[1];
  unsigned t = blockIdx.x;
  const int64_t f = (int64_t)(t % a.tiles1) * 256 + threadIdx.x;
  t /= a.tiles1;
  const int chunk = (int)(t % a.nsteps);
  const int64_t band = t / a.nsteps;
  int zf;
  const int Cy = (int)div_mod(f, nf2, zf);
  if (Cy >= m1) return;
  const int C_beg = (int)((int64_t)m0 * chunk / a.nsteps), C_end = (int)((int64_t)m0 * (chunk + 1) / a.nsteps);
  const auto& PH = a.phs.ph[phase_set_of(a.phs, band)];
  const bool phased = CPLX && PER && a.phs.any;
  const R w0 = (R)a.w[0], alpha = (R)a.alpha, gamma = (R)a.gamma;
  // local coarse row and column of the cell's lower points; an even fine
  // column takes the lower column alone
  const int Fz = zf + a.skip0[2];
  const bool odd = Fz & 1;
  const int y0 = Cy - a.cbeg[1], z0 = (Fz >> 1) - a.cbeg[2];
  const bool wy = PER && a.pbc[1] && y0 + 1 == nc1, wz = PER && a.pbc[2] && z0 + 1 == nc2;
  const bool by0 = y0 >= 0, bz0 = z0 >= 0, by1 = y0 + 1 < nc1 || wy, bz1 = odd && (z0 + 1 < nc2 || wz);
  const int64_t oy = wy ? -(int64_t)(nc1 - 1) * nc2 : nc2;
  const int oz = wz ? -(nc2 - 1) : 1;
  const T* __restrict__ p = reinterpret_cast<const T*>(a.in) + band * nc12 * nc0 + (int64_t)y0 * nc2 + z0;
  // the two fine rows of coarse plane C at this column
  auto plane = [&](int C, T (&u)[2]) {
    int l = C - a.cbeg[0];
    const bool wx = PER && a.pbc[0] && l == nc0;
    if (wx) l = 0;
    const bool in = l >= 0 && l < nc0;
    const T* c = p + (int64_t)l * nc12;
    T A[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool row = in && (h ? by1 : by0);
      T v0 = zero<T>(), v1 = zero<T>();
      if (row && bz0) v0 = __ldg(c + (h ? oy : 0));
      if (row && bz1) v1 = __ldg(c + (h ? oy : 0) + oz);
      if (phased) {
        const bool y = wy && h == 1;
        if (y) v0 = phase_mul(v0, PH[1][0][0], PH[1][0][1]);
        if (y || wz) {
          const double2 c = y && wz ? corner_phase(PH[1][0], PH[2][0])
                                    : y ? make_double2(PH[1][0][0], PH[1][0][1])
                                        : make_double2(PH[2][0][0], PH[2][0][1]);
          v1 = phase_mul(v1, c.x, c.y);
        }
      }
      A[h] = odd ? scale(w0, add(v0, v1)) : v0;
    }
    u[0] = A[0];
    u[1] = scale(w0, add(A[0], A[1]));
    if (phased && wx) {
      u[0] = phase_mul(u[0], PH[0][0][0], PH[0][0][1]);
      u[1] = phase_mul(u[1], PH[0][0][0], PH[0][0][1]);
    }
  };
  // fine local rows and planes are 2 C + parity - skip
  const int fy = 2 * Cy - a.skip0[1];
  const bool sy[2] = {fy >= 0, fy + 1 < nf1};
  const int64_t base = band * nf12 * nf0 + (int64_t)fy * nf2 + zf;
  T* __restrict__ dst = reinterpret_cast<T*>(a.out) + base;
  const T* __restrict__ ysrc = a.y ? reinterpret_cast<const T*>(a.y) + base : nullptr;
  T q[2];
  plane(C_beg, q);
  for (int C = C_beg; C < C_end; ++C) {
    T u[2];
    plane(C + 1, u);
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      const int fp = 2 * C + par - a.skip0[0];
      if (fp < 0 || fp >= nf0) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!sy[h]) continue;
        const int64_t o = fp * nf12 + h * (int64_t)nf2;
        T v = scale(alpha, par ? scale(w0, add(q[h], u[h])) : q[h]);
        if (ysrc) v = fmadd(v, gamma, __ldcs(ysrc + o));
        dst[o] = v;
      }
    }
    q[0] = u[0];
    q[1] = u[1];
  }
}

// ---------------------------------------------------------------- host side
static void midpoint_weights(int k, double* w) {
  // Lagrange weights of the degree-(k-1) interpolant through +-1/2, +-3/2, ...
  // at 0, for the pairs at distance (2j+1)/2 (the k = 2, 4, 6, 8 weights of
  // c/bmgs/restrict.c:36-56 and c/bmgs/interpolate.c:184-197).
  for (int j = 0; j < k / 2; ++j) {
    const double xj = (2 * j + 1) / 2.0;
    double num = 1.0, den = 1.0;
    for (int i = 0; i < k; ++i) {
      const double xi = (2 * i - k + 1) / 2.0;
      if (xi == xj) continue;
      num *= -xi;
      den *= xj - xi;
    }
    w[j] = num / den;
  }
}

static void fill_common(const gb_transformer* t, TrArgs& a, const double* ph, int nk, int64_t nbatch) {
  memset(&a, 0, sizeof(a));
  for (int c = 0; c < 3; ++c) {
    a.ni[c] = (int)t->nin_c[c];
    a.no[c] = (int)t->nout_c[c];
    a.pbc[c] = t->pbc[c];
    a.off[c] = t->off[c];
    a.skip0[c] = t->skip0[c];
    a.cbeg[c] = t->cbeg[c];
  }
  midpoint_weights(t->k, a.w);
  fill_phase_sets(a.phs, ph, nk, nbatch);
}

// every axis periodic with 2 n fine points, or zero-boundary with 2 n + 1
static bool usual_geometry(const gb_transformer* t) {
  for (int c = 0; c < 3; ++c) {
    const int64_t nf = t->interpolate ? t->nout_c[c] : t->nin_c[c], nc = t->interpolate ? t->nin_c[c] : t->nout_c[c];
    const int z = t->pbc[c] ? 0 : 1;
    if (nf != 2 * nc + z) return false;
    if (t->interpolate ? (t->skip0[c] != z || t->cbeg[c] != z) : t->off[c] != z) return false;
  }
  return true;
}

template <class C, typename KernelT>
static int launch_x(KernelT kernel, const TrArgs& a, int64_t blocks, cudaStream_t st) {
  static bool set = false;
  if (!set && C::SMEM > 48 * 1024) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    set = true;
  }
  kernel<<<(unsigned)blocks, C::NT, C::SMEM, st>>>(a);
  return check_launch("transformer kernel");
}

// planes per thread of the k = 2 kernels: chunks of at most 12, more of them
// while the grid would not fill the GPU
static int direct_chunks(int64_t cols, int n0) {
  return (int)std::max<int64_t>(ceil_div(n0, 12), std::min<int64_t>(n0, ceil_div((int64_t)sm_count() * 8, cols)));
}

template <typename T, int K>
static int restrict_x(const gb_transformer* t, const void* in, void* out, int64_t nin, const double* ph,
                      cudaStream_t st, double alpha, int nk) {
  TrArgs a;
  fill_common(t, a, ph, nk, nin);
  a.in = in; a.out = out; a.nbatch = nin; a.alpha = alpha;
  if (K == 2 && usual_geometry(t)) {
    a.tiles1 = ceil_div((int64_t)a.no[1] * a.no[2], 256);
    a.nsteps = direct_chunks(nin * a.tiles1, a.no[0]);
    const unsigned blocks = (unsigned)(nin * a.tiles1 * a.nsteps);
    if (a.pbc[0] || a.pbc[1] || a.pbc[2]) restrict2_direct_kernel<T, true><<<blocks, 256, 0, st>>>(a);
    else restrict2_direct_kernel<T, false><<<blocks, 256, 0, st>>>(a);
    return check_launch("restrict2_direct_kernel");
  }
  using C = RXCfg<T, K, 2, 8, sizeof(T) == 16 ? 16 : 32>;
  a.tiles1 = ceil_div(a.no[1], C::T1);
  a.tiles2 = ceil_div(a.no[2], C::T2);
  a.nsteps = ceil_div(a.no[0], C::IB);
  return launch_x<C>(restrict_x_kernel<C>, a, nin * (int64_t)a.tiles1 * a.tiles2 * a.nsteps, st);
}

// k = 2 restriction of real data on a grid periodic on every axis (the
// preconditioner's and the learned network's first transfer), marching
// along axis 0: a CTA owns TYC coarse rows of one band over a chunk of
// coarse planes; each fine plane it needs (rows 2 J0 - 1 .. 2 J0 + 2 TYC - 1
// plus the wrap-around columns) is staged once with cp.async into a two-slot
// ring, every thread restricts it in-plane for two neighbouring coarse
// points (axis 2, then axis 1: the general kernel's arithmetic, in its
// order) and the axis-0 step takes the last three fine planes from a
// register queue.  Rows must be 16-byte aligned.
// four consecutive values from a 16-byte aligned shared-memory address
__device__ __forceinline__ void load4(const float* f, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(f);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void load4(const double* f, double (&v)[4]) {
  const double2 q0 = reinterpret_cast<const double2*>(f)[0], q1 = reinterpret_cast<const double2*>(f)[1];
  v[0] = q0.x; v[1] = q0.y; v[2] = q1.x; v[3] = q1.y;
}

template <typename T, int TYC>
__global__ void __launch_bounds__(256) restrict2_march_kernel(const TrArgs a, int nch) {
  extern __shared__ __align__(16) unsigned char r2m_smem[];
  T* slot = reinterpret_cast<T*>(r2m_smem);
  constexpr int VEC = 16 / (int)sizeof(T);
  const int nf0 = a.ni[0], nf1 = a.ni[1], nf2 = a.ni[2];
  const int nc0 = a.no[0], nc1 = a.no[1], nc2 = a.no[2];
  const int FR = 2 * TYC + 1, FP = nf2 + 2 * VEC + 8;   // fine column c at VEC + c
  const int tid = threadIdx.x, nt = blockDim.x;
  const int ngx = (nc2 + 1) >> 1;
  const int gx = tid % ngx, ty = tid / ngx;
  const int J0 = blockIdx.y * TYC, J = J0 + ty, K0 = 2 * gx;
  const int64_t b = blockIdx.z;
  const int I_beg = (int)((int64_t)blockIdx.x * nc0 / nch), I_end = (int)((int64_t)(blockIdx.x + 1) * nc0 / nch);
  const T* src = reinterpret_cast<const T*>(a.in) + b * (int64_t)nf0 * nf1 * nf2;
  T* dst = reinterpret_cast<T*>(a.out) + b * (int64_t)nc0 * nc1 * nc2;
  const T w0 = (T)a.w[0], half = (T)0.5, alpha = (T)a.alpha;
  const int r0 = 2 * J0 + a.off[1] - 1;                 // first staged fine row
  auto wrap = [](int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); };
  // the copies of a staged plane: element e = (row r, piece c) is a 16-byte
  // chunk (c < chunks), column -1 or column nf2; a thread's first MAXU
  // elements have their offsets worked out once (no index divisions per plane)
  const int chunks = nf2 / VEC, ne = FR * (chunks + 2);
  constexpr int MAXU = 4;
  int s_off[MAXU], d_off[MAXU];
  unsigned wide = 0u;
#pragma unroll
  for (int u = 0; u < MAXU; ++u) {
    const int e = tid + u * nt;
    s_off[u] = 0;
    d_off[u] = -1;
    if (e < ne) {
      const int r = e / (chunks + 2), c = e % (chunks + 2);
      const int row = wrap(r0 + r, nf1) * nf2;
      if (c < chunks) {
        s_off[u] = row + c * VEC;
        d_off[u] = r * FP + VEC + c * VEC;
        wide |= 1u << u;
      } else if (c == chunks) {
        s_off[u] = row + nf2 - 1;                 // column -1
        d_off[u] = r * FP + VEC - 1;
      } else {
        s_off[u] = row;                           // column nf2
        d_off[u] = r * FP + VEC + nf2;
      }
    }
  }
  auto stage = [&](int p, T* d) {
    const T* pl = src + (int64_t)wrap(p, nf0) * nf1 * nf2;
#pragma unroll
    for (int u = 0; u < MAXU; ++u) {
      if (d_off[u] < 0) continue;
      if (wide & (1u << u)) cp_async16(d + d_off[u], pl + s_off[u]);
      else cp_async_elem(d + d_off[u], pl + s_off[u]);
    }
    for (int e = tid + MAXU * nt; e < ne; e += nt) {
      const int r = e / (chunks + 2), c = e % (chunks + 2);
      const T* row = pl + (int64_t)wrap(r0 + r, nf1) * nf2;
      T* dr = d + r * FP;
      if (c < chunks) cp_async16(dr + VEC + c * VEC, row + c * VEC);
      else if (c == chunks) cp_async_elem(dr + VEC - 1, row + nf2 - 1);   // column -1
      else cp_async_elem(dr + VEC + nf2, row);                          // column nf2
    }
  };
  // the five fine columns 2K - 1 .. 2K + 3 a thread reads per row: one
  // 16-byte load and one scalar when the window start is 16-byte aligned
  const bool vec4 = (a.off[2] % VEC) == 0;
  const int p_beg = 2 * I_beg + a.off[0] - 1, p_end = 2 * (I_end - 1) + a.off[0] + 1;
  stage(p_beg, slot);
  cp_async_commit();
  T q0[2] = {0, 0}, q1[2] = {0, 0}, q2[2] = {0, 0};
  const bool act = ty < TYC && J < nc1;
  for (int p = p_beg; p <= p_end; ++p) {
    const int s = (p - p_beg) & 1;
    if (p + 1 <= p_end) stage(p + 1, slot + (s ^ 1) * FR * FP);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (act) {
      const T* P = slot + s * FR * FP + 2 * ty * FP + VEC + 2 * K0 + a.off[2];
      T g[3][2];
#pragma unroll
      for (int dy = 0; dy < 3; ++dy) {
        const T* f = P + dy * FP;
        T v[4];
        if (vec4) {
          load4(f, v);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = f[i];
        }
        const T fm = f[-1];
        g[dy][0] = half * fmadd(v[0], w0, add(v[1], fm));
        g[dy][1] = half * fmadd(v[2], w0, add(v[3], v[1]));
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        q0[h] = q1[h];
        q1[h] = q2[h];
        q2[h] = half * fmadd(g[1][h], w0, add(g[2][h], g[0][h]));
      }
      const int tI = p - a.off[0] - 1;                  // fine plane 2I + off + 1 just arrived
      if (tI >= 2 * I_beg && (tI & 1) == 0) {
        const int I = tI >> 1;
        T* o = dst + ((int64_t)I * nc1 + J) * nc2 + K0;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (K0 + h < nc2) o[h] = alpha * (half * fmadd(q1[h], w0, add(q2[h], q0[h])));
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
}

template <typename T>
static int restrict2_march_launch(const gb_transformer* t, const void* in, void* out, int64_t nin,
                                  cudaStream_t st, double alpha) {
  constexpr int VEC = 16 / (int)sizeof(T);
  TrArgs a;
  fill_common(t, a, nullptr, 1, nin);
  a.in = in; a.out = out; a.nbatch = nin; a.alpha = alpha;
  const int ngx = (a.no[2] + 1) / 2;
  const int TYC = ngx * 8 <= 256 ? 8 : (ngx * 4 <= 256 ? 4 : 2);
  const int nch = std::max(1, std::min(a.no[0], a.no[0] / 8));
  const size_t smem = (size_t)2 * (2 * TYC + 1) * (a.ni[2] + 2 * VEC + 8) * sizeof(T);
  const dim3 grid((unsigned)nch, (unsigned)((a.no[1] + TYC - 1) / TYC), (unsigned)nin);
  const unsigned threads = (unsigned)(ngx * TYC);
  if (TYC == 8) restrict2_march_kernel<T, 8><<<grid, threads, smem, st>>>(a, nch);
  else if (TYC == 4) restrict2_march_kernel<T, 4><<<grid, threads, smem, st>>>(a, nch);
  else restrict2_march_kernel<T, 2><<<grid, threads, smem, st>>>(a, nch);
  return check_launch("restrict2_march_kernel");
}

template <typename T>
static bool restrict2_march_ok(const gb_transformer* t, int64_t nin, const double* ph) {
  if (!t->pbc[0] || !t->pbc[1] || !t->pbc[2] || nin > 65535 || nin < 1) return false;
  if (ph)
    for (int i = 0; i < 12; ++i)
      if (ph[i] != ((i % 2) ? 0.0 : 1.0)) return false;
  const int64_t nf2 = t->nin_c[2];
  const int64_t ngx = (t->nout_c[2] + 1) / 2;
  const int64_t tyc = ngx * 8 <= 256 ? 8 : (ngx * 4 <= 256 ? 4 : 2);
  // single-wrap periodic indices: at least 2 * TYC fine rows, 2 planes
  return (nf2 * (int64_t)sizeof(T)) % 16 == 0 && ngx * 2 <= 256 && t->nin_c[0] >= 2 &&
         t->nin_c[1] >= 2 * tyc && nf2 >= 2 * (16 / (int)sizeof(T)) && t->nout_c[1] >= 1;
}

// k = 2 interpolation of real data on a grid periodic on every axis (fine
// point 2C on coarse point C), marching along axis 0 over coarse planes: a
// CTA owns TYF fine rows of one band over a chunk of coarse planes; each
// coarse plane (rows F0/2 .. F0/2 + TYF/2 plus the wrap-around column) is
// staged once into a two-slot ring; every thread interpolates it for four
// neighbouring fine columns of its row (axis 2, then axis 1: the general
// kernel's arithmetic, in its order) and, once coarse plane C + 1 is in,
// writes fine planes 2C and 2C + 1 with the alpha / gamma * y epilogue as
// 16-byte vectors.  Rows must be 16-byte aligned.
template <typename T, int TYF>
__global__ void __launch_bounds__(256) interp2_march_kernel(const TrArgs a, int nch) {
  extern __shared__ __align__(16) unsigned char i2m_smem[];
  T* slot = reinterpret_cast<T*>(i2m_smem);
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int CRR = TYF / 2 + 1;
  const int nc0 = a.ni[0], nc1 = a.ni[1], nc2 = a.ni[2];
  const int nf1 = a.no[1], nf2 = a.no[2];
  const int CP = nc2 + 2 * VEC + 8;                    // coarse column c at VEC + c
  const int tid = threadIdx.x, nt = blockDim.x;
  const int ngx = nf2 >> 2;
  const int gx = tid % ngx, ty = tid / ngx;
  const int F0 = blockIdx.y * TYF, F = F0 + ty, k = 4 * gx;
  const int64_t b = blockIdx.z;
  const int C_beg = (int)((int64_t)blockIdx.x * nc0 / nch), C_end = (int)((int64_t)(blockIdx.x + 1) * nc0 / nch);
  const T* src = reinterpret_cast<const T*>(a.in) + b * (int64_t)nc0 * nc1 * nc2;
  const int64_t fplane = (int64_t)nf1 * nf2;
  T* dst = reinterpret_cast<T*>(a.out) + b * 2 * (int64_t)nc0 * fplane;
  const T* ysrc = a.y ? reinterpret_cast<const T*>(a.y) + b * 2 * (int64_t)nc0 * fplane : nullptr;
  const T w0 = (T)a.w[0], alpha = (T)a.alpha, gamma = (T)a.gamma;
  auto wrap = [](int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); };
  // rows of a whole number of 16-byte chunks are copied in chunks, others
  // (a 14-point FP32 row, say) element by element
  const bool rows16 = (nc2 * (int)sizeof(T)) % 16 == 0;
  auto stage = [&](int g, T* d) {
    const T* pl = src + (int64_t)wrap(g, nc0) * nc1 * nc2;
    if (rows16) {
      const int chunks = nc2 / VEC;
      for (int e = tid; e < CRR * (chunks + 1); e += nt) {
        const int r = e / (chunks + 1), c = e % (chunks + 1);
        const T* row = pl + (int64_t)wrap((F0 >> 1) + r, nc1) * nc2;
        T* dr = d + r * CP;
        if (c < chunks) cp_async16(dr + VEC + c * VEC, row + c * VEC);
        else cp_async_elem(dr + VEC + nc2, row);                 // column nc2
      }
    } else {
      for (int e = tid; e < CRR * (nc2 + 1); e += nt) {
        const int r = e / (nc2 + 1), c = e % (nc2 + 1);
        const T* row = pl + (int64_t)wrap((F0 >> 1) + r, nc1) * nc2;
        cp_async_elem(d + r * CP + VEC + c, row + (c < nc2 ? c : 0));   // column nc2 = column 0
      }
    }
  };
  stage(C_beg, slot);
  cp_async_commit();
  T qp[4];                                             // u of the previous coarse plane
  const bool act = ty < TYF && F < nf1;
  for (int g = C_beg; g <= C_end; ++g) {
    const int s = (g - C_beg) & 1;
    if (g + 1 <= C_end) stage(g + 1, slot + (s ^ 1) * CRR * CP);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (act) {
      const T* P = slot + s * CRR * CP + VEC + (k >> 1);
      const int rl = (F >> 1) - (F0 >> 1);
      T A[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const T* row = P + (rl + h) * CP;
        const T c0 = row[0], c1 = row[1], c2 = row[2];
        A[h][0] = c0;
        A[h][1] = w0 * add(c0, c1);
        A[h][2] = c1;
        A[h][3] = w0 * add(c1, c2);
      }
      T u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = (F & 1) ? w0 * add(A[0][q], A[1][q]) : A[0][q];
      if (g > C_beg) {
        const int C = g - 1;
#pragma unroll
        for (int par = 0; par < 2; ++par) {
          const int64_t o = (int64_t)(2 * C + par) * fplane + (int64_t)F * nf2 + k;
          T x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            T v = par == 0 ? qp[q] : w0 * add(qp[q], u[q]);
            v = alpha * v;
            if (ysrc) v = fmadd(v, gamma, ysrc[o + q]);
            x[q] = v;
          }
          if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(dst + o) = make_float4(x[0], x[1], x[2], x[3]);
          } else {
            reinterpret_cast<double2*>(dst + o)[0] = make_double2(x[0], x[1]);
            reinterpret_cast<double2*>(dst + o)[1] = make_double2(x[2], x[3]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) qp[q] = u[q];
    }
    __syncthreads();
  }
  cp_async_wait<0>();
}

template <typename T>
static bool interp2_march_ok(const gb_transformer* t, int64_t nin, const double* ph, const void* y) {
  if (!t->pbc[0] || !t->pbc[1] || !t->pbc[2] || nin > 65535 || nin < 1) return false;
  if (ph)
    for (int i = 0; i < 12; ++i)
      if (ph[i] != ((i % 2) ? 0.0 : 1.0)) return false;
  for (int c = 0; c < 3; ++c)
    if (t->skip0[c] != 0 || t->cbeg[c] != 0 || t->nout_c[c] != 2 * t->nin_c[c]) return false;
  const int64_t nc2 = t->nin_c[2], nf2 = t->nout_c[2];
  const int64_t ngx = nf2 / 4;
  const int64_t tyf = ngx * 8 <= 256 ? 8 : (ngx * 4 <= 256 ? 4 : 2);
  (void)y;
  return nf2 % 4 == 0 && ngx * 2 <= 256 && t->nin_c[0] >= 1 && t->nin_c[1] >= tyf / 2 + 1 &&
         nc2 >= 16 / (int)sizeof(T);
}

template <typename T>
static int interp2_march_launch(const gb_transformer* t, const void* in, void* out, int64_t nin,
                                cudaStream_t st, double alpha, const void* y, double gamma) {
  constexpr int VEC = 16 / (int)sizeof(T);
  TrArgs a;
  fill_common(t, a, nullptr, 1, nin);
  a.in = in; a.out = out; a.nbatch = nin; a.alpha = alpha; a.y = y; a.gamma = gamma;
  const int ngx = a.no[2] / 4;
  const int TYF = ngx * 8 <= 256 ? 8 : (ngx * 4 <= 256 ? 4 : 2);
  const int nch = std::max(1, std::min(a.ni[0], a.ni[0] / 7));
  const size_t smem = (size_t)2 * (TYF / 2 + 1) * (a.ni[2] + 2 * VEC + 8) * sizeof(T);
  const dim3 grid((unsigned)nch, (unsigned)((a.no[1] + TYF - 1) / TYF), (unsigned)nin);
  const unsigned threads = (unsigned)(ngx * TYF);
  if (TYF == 8) interp2_march_kernel<T, 8><<<grid, threads, smem, st>>>(a, nch);
  else if (TYF == 4) interp2_march_kernel<T, 4><<<grid, threads, smem, st>>>(a, nch);
  else interp2_march_kernel<T, 2><<<grid, threads, smem, st>>>(a, nch);
  return check_launch("interp2_march_kernel");
}

template <typename T, int K>
static int restrict_k(const gb_transformer* t, const void* in, void* out, int64_t nin,
                      const double* ph, cudaStream_t st, double alpha, int nk) {
  if constexpr (K == 2 && !Elem<T>::cplx) {
    if (restrict2_march_ok<T>(t, nin, ph)) return restrict2_march_launch<T>(t, in, out, nin, st, alpha);
  }
  return restrict_x<T, K>(t, in, out, nin, ph, st, alpha, nk);
}

template <typename T, int K>
static int interpolate_k(const gb_transformer* t, const void* in, void* out, int64_t nin,
                         const double* ph, cudaStream_t st, double alpha, const void* y, double gamma,
                         int nk) {
  if constexpr (K == 2 && !Elem<T>::cplx) {
    if (interp2_march_ok<T>(t, nin, ph, y)) return interp2_march_launch<T>(t, in, out, nin, st, alpha, y, gamma);
  }
  TrArgs a;
  fill_common(t, a, ph, nk, nin);
  a.in = in; a.out = out; a.nbatch = nin; a.alpha = alpha; a.y = y; a.gamma = gamma;
  if (K == 2 && usual_geometry(t)) {
    a.tiles1 = ceil_div((int64_t)(a.ni[1] + a.cbeg[1]) * a.no[2], 256);
    a.nsteps = direct_chunks(nin * a.tiles1, a.ni[0] + a.cbeg[0]);
    const unsigned blocks = (unsigned)(nin * a.tiles1 * a.nsteps);
    if (a.pbc[0] || a.pbc[1] || a.pbc[2]) interp2_direct_kernel<T, true><<<blocks, 256, 0, st>>>(a);
    else interp2_direct_kernel<T, false><<<blocks, 256, 0, st>>>(a);
    return check_launch("interp2_direct_kernel");
  }
  using C = IXCfg<T, K, sizeof(T) == 4 ? 8 : 4, 16, sizeof(T) == 16 ? 16 : 32>;
  a.tiles1 = ceil_div(a.no[1], C::T1);
  a.tiles2 = ceil_div(a.no[2], C::T2);
  // coarse planes C with 2C - skip0 or 2C + 1 - skip0 in [0, nf0)
  const int cmin = a.skip0[0] >= 0 ? a.skip0[0] / 2 : -((-a.skip0[0] + 1) / 2);
  const int cmax = (a.no[0] - 1 + a.skip0[0]) / 2;
  a.nsteps = cmax - cmin + 1;
  return launch_x<C>(interpolate_x_kernel<C>, a,
                     nin * (int64_t)a.tiles1 * a.tiles2 * ceil_div(a.nsteps, C::IB), st);
}

template <typename T>
static int tr_dispatch(const gb_transformer* t, const void* in, void* out, int64_t nin,
                       const double* ph, cudaStream_t st, double alpha, const void* y, double gamma,
                       int nk) {
  if (t->interpolate) {
    switch (t->k) {
      case 2: return interpolate_k<T, 2>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
      case 4: return interpolate_k<T, 4>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
      case 6: return interpolate_k<T, 6>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
      default: return interpolate_k<T, 8>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
    }
  }
  if (y) return fail(GB_E_UNSUPPORTED, "restriction has no y epilogue");
  switch (t->k) {
    case 2: return restrict_k<T, 2>(t, in, out, nin, ph, st, alpha, nk);
    case 4: return restrict_k<T, 4>(t, in, out, nin, ph, st, alpha, nk);
    case 6: return restrict_k<T, 6>(t, in, out, nin, ph, st, alpha, nk);
    default: return restrict_k<T, 8>(t, in, out, nin, ph, st, alpha, nk);
  }
}

int tr_apply(const gb_transformer* t, const void* in, void* out, int64_t nin, int dtype,
             const double* ph, cudaStream_t st, double alpha, const void* y, double gamma, int nk) {
  if (nk > KMAX) return fail(GB_E_UNSUPPORTED, "more k-point phase sets than one launch takes");
  if (nk > 1 && nin % nk) return fail(GB_E_INVALID, "batch not divisible by the number of phase sets");
  switch (dtype) {
    case GB_DTYPE_F64: return tr_dispatch<double>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
    case GB_DTYPE_F32: return tr_dispatch<float>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
    case GB_DTYPE_C128: return tr_dispatch<double2>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
    default: return tr_dispatch<float2>(t, in, out, nin, ph, st, alpha, y, gamma, nk);
  }
}

}  // namespace gb

using namespace gb;

extern "C" {

int gb_transformer_new(const int64_t size_in[3], const int64_t size_out[3], int k,
                       const int64_t pad_cd[6], const int64_t npad_cd[6], const int64_t skip_cd[6],
                       const int64_t neighbor_cd[6], int real, int interpolate, gb_transformer** out) {
  GB_REQUIRE(out && size_in && size_out && pad_cd && npad_cd && skip_cd && neighbor_cd,
             "gb_transformer_new: null pointer");
  GB_REQUIRE(k == 2 || k == 4 || k == 6 || k == 8, "gb_transformer_new: k must be 2, 4, 6 or 8");
  const int nn = k / 2;
  auto* t = new (std::nothrow) gb_transformer();
  if (!t) return fail(GB_E_NOMEM, "gb_transformer_new: out of host memory");
  t->k = k;
  t->interpolate = interpolate ? 1 : 0;
  t->real = real;
  for (int c = 0; c < 3; ++c) {
    t->nin_c[c] = size_in[c];
    t->nout_c[c] = size_out[c];
    t->pbc[c] = (neighbor_cd[2 * c] >= 0 || neighbor_cd[2 * c + 1] >= 0) ? 1 : 0;
    const int64_t p0 = pad_cd[2 * c], p1 = pad_cd[2 * c + 1];
    if (size_in[c] <= 0 || size_out[c] <= 0 || p0 < 0 || p1 < 0) {
      delete t;
      return fail(GB_E_INVALID, "gb_transformer_new: bad sizes or padding");
    }
    if (!interpolate) {
      // pad0 = 2nn - 1 - (2 beg_out - beg_in)  (gpaw/transformers.py:33)
      t->off[c] = (int)(2 * nn - 1 - p0);
      // output count of the reference: (n_in + pad0 + pad1 - 2k + 3) / 2
      const int64_t nout = (size_in[c] + p0 + p1 - 2 * k + 3) / 2;
      if (nout != size_out[c] || t->off[c] < 0 || t->off[c] > 1) {
        delete t;
        return fail(GB_E_INVALID, "gb_transformer_new: restriction sizes/padding inconsistent");
      }
    } else {
      // pad0 = nn - 1 - beg_out // 2 + beg_in, skip0 = beg_out % 2  (transformers.py:41-46)
      t->skip0[c] = (int)skip_cd[2 * c];
      t->skip1[c] = (int)skip_cd[2 * c + 1];
      t->cbeg[c] = (int)(p0 - nn + 1);
      const int64_t npairs = size_in[c] + p0 + p1 - (k - 1) + t->skip1[c];
      const int64_t nout = 2 * npairs - t->skip0[c] - t->skip1[c];
      if (nout != size_out[c] || t->cbeg[c] < 0 || t->cbeg[c] > 1) {
        delete t;
        return fail(GB_E_INVALID, "gb_transformer_new: interpolation sizes/padding inconsistent");
      }
    }
    (void)npad_cd;
  }
  *out = t;
  return GB_OK;
}

int gb_transformer_apply(const gb_transformer* t, const void* in, void* out, int64_t nin, int dtype,
                         const double* phase_cd, void* stream) {
  GB_REQUIRE(t, "gb_transformer_apply: null transformer");
  GB_REQUIRE(dtype_valid(dtype), "gb_transformer_apply: unknown dtype");
  GB_REQUIRE(nin >= 0, "gb_transformer_apply: negative batch");
  GB_REQUIRE(dtype_complex(dtype) == !t->real,
             "gb_transformer_apply: dtype does not match the transformer's real/complex flag");
  if (nin == 0) return GB_OK;
  GB_REQUIRE(in && out && in != out, "gb_transformer_apply: bad data pointers");
  GB_REQUIRE(!dtype_complex(dtype) || phase_cd, "gb_transformer_apply: complex data needs phase_cd");
  return tr_apply(t, in, out, nin, dtype, dtype_complex(dtype) ? phase_cd : nullptr,
                  (cudaStream_t)stream, 1.0, nullptr, 0.0);
}

int gb_transformer_apply_axpy(const gb_transformer* t, const void* in, void* out, int64_t nin, int dtype,
                              const double* phase_cd, double alpha, const void* y, double gamma, void* stream) {
  GB_REQUIRE(t, "gb_transformer_apply_axpy: null transformer");
  GB_REQUIRE(dtype_valid(dtype), "gb_transformer_apply_axpy: unknown dtype");
  GB_REQUIRE(nin >= 0, "gb_transformer_apply_axpy: negative batch");
  GB_REQUIRE(dtype_complex(dtype) == !t->real,
             "gb_transformer_apply_axpy: dtype does not match the transformer's real/complex flag");
  if (nin == 0) return GB_OK;
  GB_REQUIRE(in && out && in != out, "gb_transformer_apply_axpy: bad data pointers");
  GB_REQUIRE(t->interpolate || !y, "gb_transformer_apply_axpy: restriction has no y term");
  GB_REQUIRE(!dtype_complex(dtype) || phase_cd, "gb_transformer_apply_axpy: complex data needs phase_cd");
  return tr_apply(t, in, out, nin, dtype, dtype_complex(dtype) ? phase_cd : nullptr, (cudaStream_t)stream, alpha,
                  y, gamma);
}

int gb_transformer_free(gb_transformer* t) {
  delete t;
  return GB_OK;
}

int gb_transformer_apply_k(const gb_transformer* t, const void* in, void* out, int64_t nin, int dtype, int nk,
                           const double* phase_kcd, void* stream) {
  GB_REQUIRE(t && dtype_valid(dtype) && nin >= 0, "gb_transformer_apply_k: bad arguments");
  GB_REQUIRE(dtype_complex(dtype) == !t->real, "gb_transformer_apply_k: dtype does not match the transformer");
  GB_REQUIRE(nk >= 1 && nk <= KMAX && nin % nk == 0, "gb_transformer_apply_k: bad number of phase sets");
  if (nin == 0) return GB_OK;
  GB_REQUIRE(in && out && in != out, "gb_transformer_apply_k: bad data pointers");
  GB_REQUIRE(!dtype_complex(dtype) || phase_kcd, "gb_transformer_apply_k: complex data needs phases");
  return tr_apply(t, in, out, nin, dtype, dtype_complex(dtype) ? phase_kcd : nullptr, (cudaStream_t)stream, 1.0,
                  nullptr, 0.0, nk);
}

}  // extern "C"
