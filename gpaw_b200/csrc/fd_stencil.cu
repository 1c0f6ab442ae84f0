// FD stencil operator (replaces _gpaw.Operator: c/operators.c, c/bmgs/fd.c,
// c/bc.c).  Stencils whose points all lie on the three axes (the reference's
// "cfd" case: Laplace on orthorhombic cells, Gradient) take, in this order,
// the TMA kernel of fd_stencil_tma.cu, the row kernel of fd_stencil_rows.cu,
// the tile kernel of fd_stencil_tiles.cu and the kernel here:
//
//  * march_star_kernel -- any layout, boundary mix, phases and radius up to 6.
//    One thread per (axis1, axis2) column marches along axis 0 with a
//    register queue; its in-plane neighbours are read through L1.  There is
//    no staging and no barrier, so it is the fastest form while a call is too
//    small to fill the pipelines of the others (every SM busy for less than
//    ~16 plane tiles of the row kernel), with 7-point FP32 stencils, which
//    read too few neighbours to be bound by L1 (four 31^3 FP64 grids 13 us
//    against 33 us in the row kernel; 160 x 37^3 FP32, radius 1: 33 against
//    37 us), and on rows of fewer than 28 elements.  It also serves the rows
//    that the row kernel's copies do not cover (launch_rows: four rows per warp
//    and plane; radius 3: up to 34 FP64 or complex64 and 68 FP32 elements):
//    160 FP64 bands of 31^3 43 us, 160 FP32 bands of 55^3 216 us, against 69
//    and 279 us in the tile kernel (radius 3, zero boundary).
//
//  * box_kernel   -- any stencil (off-axis points of GUC Laplacians /
//    non-orthogonal gradients, c/bmgs/fd.c generic loop).  3-D tile with a
//    full halo cube in shared memory; correctness path.
//
// Boundary semantics follow c/bc.c:146-258: a halo cell beyond the upper end
// of a periodic axis c holds in[... m ...] * phase_cd[c][0], below the lower
// end in[... n-1-m ...] * phase_cd[c][1]; zero boundaries give zeros.

#include <vector>
#include <cmath>
#include <cstring>
#include <algorithm>
#include <type_traits>
#include "internal.cuh"

namespace gb {


struct StarArgs {
  const void* in;
  void* out;
  int64_t nbatch;
  int n0, n1, n2;
  int pbc0, pbc1, pbc2;
  int tiles, chunks;          // column tiles of a plane, chunks of planes
  double c0;
  double c0diff;              // c0 + sum of the neighbour coefficients (difference form)
  double a[3][2 * HMAX + 1];  // a[axis][m + HMAX]: coefficient of offset m (m != 0)
  PhaseSets phs;              // Bloch phases per k-point group of bands
  // epilogue: out = alpha * S(in) + beta * in + gamma * y   (y may be null)
  double alpha, beta, gamma;
  const void* y;
  const void* vpot;
};

// true modulo: partial tiles of small grids can reach several periods away
// (those cells feed no valid output, but their loads must stay in bounds)
__device__ __forceinline__ int wrap_index(int i, int n) {
  int r = i % n;
  return r < 0 ? r + n : r;
}

// One term of the stencil, in the order and form of star_core.cuh: centre,
// axis 0, axis 2, axis 1, offsets ascending; FP32 as differences, axes 0 and 2
// in pairs of offsets, which symmetric stencils of radius 1 and 3 add before
// they multiply.  A band's result is then the same, bit for bit, in this kernel
// and in the row kernel, so it does not depend on how many bands a call has.
template <typename T>
__device__ __forceinline__ T star_term(T acc, typename Elem<T>::R c, T v, T xc) {
  return fmadd(acc, c, sizeof(typename Elem<T>::R) == 4 ? sub(v, xc) : v);
}

template <bool SYM>
__device__ __forceinline__ float star_pair(float acc, float cp, float cm, float vp, float vm, float xc) {
  if constexpr (SYM) return fmaf(cp, fmaf(-2.f, xc, vp + vm), acc);
  acc = fmaf(cp, vp - xc, acc);
  return fmaf(cm, vm - xc, acc);
}

__device__ __forceinline__ double ld_nc(const double* p) { return __ldg(p); }
__device__ __forceinline__ float ld_nc(const float* p) { return __ldg(p); }
__device__ __forceinline__ double2 ld_nc(const double2* p) { return __ldg(p); }
__device__ __forceinline__ float2 ld_nc(const float2* p) { return __ldg(p); }

template <typename T, int H, bool PER, bool SYM>
__global__ void __launch_bounds__(256, sizeof(T) == 16 ? 2 : 3) march_star_kernel(const __grid_constant__ StarArgs a) {
  using R = typename Elem<T>::R;
  constexpr bool CPLX = Elem<T>::cplx;
  constexpr bool DIFF = sizeof(R) == 4;
  constexpr int NQ = 2 * H + 2;             // 2H + 1 planes in use, one on its way
  // one row per thread (two and three were slower: fewer warps)
  const int n0 = a.n0, n1 = a.n1, n2 = a.n2;
  const int64_t n12 = (int64_t)n1 * n2;
  unsigned u0 = blockIdx.x;
  const unsigned tile = u0 % a.tiles;
  u0 /= a.tiles;
  const int chunk = u0 % a.chunks;
  const int64_t band = u0 / a.chunks;
  const int64_t f = (int64_t)tile * 256 + threadIdx.x;
  int z;
  const int y = (int)div_mod(f, n2, z);
  if (y >= n1) return;
  const int p_begin = (int)((int64_t)n0 * chunk / a.chunks), p_end = (int)((int64_t)n0 * (chunk + 1) / a.chunks);

  const T* __restrict__ src = reinterpret_cast<const T*>(a.in) + band * n12 * n0 + f;
  const auto& PH = a.phs.ph[phase_set_of(a.phs, band)];
  const bool phased = CPLX && PER && a.phs.any;

  // value of the point's plane at row y + d / column z + d: wrapped on a
  // periodic axis, zero outside the others
  auto ld_row = [&](const T* c, int d) -> T {
    int64_t off = (int64_t)d * n2;
    const int side = y + d < 0 ? 1 : y + d >= n1 ? 0 : -1;
    bool ok = side < 0;
    if (PER && a.pbc1 && !ok) {
      off += side ? n12 : -n12;
      ok = true;
    }
    T v = zero<T>();
    if (ok) v = ld_nc(c + off);
    if (phased && side >= 0) v = phase_mul(v, PH[1][side][0], PH[1][side][1]);
    return v;
  };
  auto ld_col = [&](const T* c, int d) -> T {
    const int zz = z + d;
    int off = d;
    int side = zz < 0 ? 1 : zz >= n2 ? 0 : -1;
    bool ok = side < 0;
    if (PER && a.pbc2 && !ok) {
      off += side ? n2 : -n2;
      ok = true;
    }
    T v = zero<T>();
    if (ok) v = ld_nc(c + off);
    if (phased && side >= 0) v = phase_mul(v, PH[2][side][0], PH[2][side][1]);
    return v;
  };
  // the point itself in plane j (any j; zero or wrapped outside the grid)
  auto ld_plane = [&](int j) -> T {
    int side = j < 0 ? 1 : j >= n0 ? 0 : -1;
    bool in = side < 0;
    if (PER && a.pbc0 && !in) {
      j += side ? n0 : -n0;
      in = true;
    }
    T v = zero<T>();
    if (in) v = ld_nc(src + (int64_t)j * n12);
    if (phased && side >= 0) v = phase_mul(v, PH[0][side][0], PH[0][side][1]);
    return v;
  };

  const bool epi = a.alpha != 1.0 || a.beta != 0.0 || a.y != nullptr || a.vpot != nullptr;
  const R c0 = DIFF ? (R)a.c0diff : (R)a.c0;
  T* __restrict__ dst = reinterpret_cast<T*>(a.out) + band * n12 * n0 + f;
  const T* __restrict__ ysrc = a.y ? reinterpret_cast<const T*>(a.y) + band * n12 * n0 + f : nullptr;
  const R* __restrict__ vsrc = a.vpot ? reinterpret_cast<const R*>(a.vpot) + f : nullptr;

  // q[(s + H) % NQ]: plane p_begin + s
  T q[NQ];
#pragma unroll
  for (int s = -H; s <= H; ++s) q[s + H] = ld_plane(p_begin + s);
  for (int pb = p_begin; pb < p_end; pb += NQ) {
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      const int p = pb + u;
      if (p < p_end) {
        if (p + 1 < p_end) q[(u + 2 * H + 1) % NQ] = ld_plane(p + 1 + H);
        const int64_t po = (int64_t)p * n12;
        const T* c = src + po;
        const T xc = q[(u + H) % NQ];
        T yv;
        R vv;
        if (epi) {
          if (ysrc) yv = __ldcs(ysrc + po);
          if (vsrc) vv = __ldg(vsrc + po);
        }
        T x = scale(c0, xc);
#pragma unroll
        for (int m = -H; m <= H; ++m) {
          if constexpr (std::is_same<T, float>::value) {
            if (m > 0)
              x = star_pair<SYM>(x, (R)a.a[0][HMAX + m], (R)a.a[0][HMAX - m], q[(u + H + m + NQ) % NQ],
                                 q[(u + H - m + NQ) % NQ], xc);
          } else {
            if (m) x = star_term(x, (R)a.a[0][m + HMAX], q[(u + H + m + NQ) % NQ], xc);
          }
        }
#pragma unroll
        for (int m = -H; m <= H; ++m) {
          if constexpr (std::is_same<T, float>::value) {
            if (m > 0)
              x = star_pair<SYM>(x, (R)a.a[2][HMAX + m], (R)a.a[2][HMAX - m], ld_col(c, m), ld_col(c, -m), xc);
          } else {
            if (m) x = star_term(x, (R)a.a[2][m + HMAX], ld_col(c, m), xc);
          }
        }
#pragma unroll
        for (int d = -H; d <= H; ++d)
          if (d) x = star_term(x, (R)a.a[1][d + HMAX], ld_row(c, d), xc);
        if (epi) {
          x = fmadd(scale((R)a.alpha, x), (R)a.beta, xc);
          if (ysrc) x = fmadd(x, (R)a.gamma, yv);
          if (vsrc) x = fmadd(x, vv, xc);
        }
        st_cs(dst + po, x);
      }
    }
  }
}

// --------------------------------------------------------------------------
// Generic stencil: arbitrary offsets within a cube of radius M (<= 6).
struct BoxArgs {
  const void* in;
  void* out;
  int64_t nbatch;
  int n0, n1, n2;
  int pbc0, pbc1, pbc2;
  int M;                  // halo radius
  int np;
  int b0, b1, b2;         // tile extents
  int tiles0, tiles1, tiles2;
  double coef[64];
  int off[64][3];
  PhaseSets phs;
  double alpha, beta, gamma;
  const void* y;
  const void* vpot;
  double csum;   // sum of all coefficients (difference form in FP32)
};

template <typename T>
__global__ void __launch_bounds__(256) box_kernel(const BoxArgs args) {
  using R = typename Elem<T>::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);
  const int M = args.M;
  const int E0 = args.b0 + 2 * M, E1 = args.b1 + 2 * M, E2 = args.b2 + 2 * M;
  const int64_t ntile = (int64_t)args.tiles0 * args.tiles1 * args.tiles2;
  const int64_t n12 = (int64_t)args.n1 * args.n2, n012 = n12 * args.n0;
  for (int64_t w = blockIdx.x; w < args.nbatch * ntile; w += gridDim.x) {
    const int64_t band = w / ntile;
    int t = (int)(w % ntile);
    const int x0 = (t / (args.tiles1 * args.tiles2)) * args.b0;
    t %= args.tiles1 * args.tiles2;
    const int y0 = (t / args.tiles2) * args.b1;
    const int z0 = (t % args.tiles2) * args.b2;
    const T* src = reinterpret_cast<const T*>(args.in) + band * n012;
    T* dst = reinterpret_cast<T*>(args.out) + band * n012;
    const auto& PH = args.phs.ph[phase_set_of(args.phs, band)];
    __syncthreads();
    for (int e = threadIdx.x; e < E0 * E1 * E2; e += blockDim.x) {
      const int i2 = e % E2, i1 = (e / E2) % E1, i0 = e / (E1 * E2);
      int g[3] = {x0 - M + i0, y0 - M + i1, z0 - M + i2};
      const int n[3] = {args.n0, args.n1, args.n2};
      const int pbc[3] = {args.pbc0, args.pbc1, args.pbc2};
      double pr = 1.0, pi = 0.0;
      bool zero_cell = false;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (g[c] < 0 || g[c] >= n[c]) {
          if (!pbc[c]) { zero_cell = true; break; }
          const int sd = g[c] < 0;
          const double qr = PH[c][sd][0], qi = PH[c][sd][1];
          const double tr = pr * qr - pi * qi, ti = pr * qi + pi * qr;
          pr = tr; pi = ti;
          g[c] = wrap_index(g[c], n[c]);
        }
      }
      T v = zero<T>();
      if (!zero_cell) {
        v = src[(int64_t)g[0] * n12 + (int64_t)g[1] * args.n2 + g[2]];
        if (args.phs.any) v = phase_mul(v, pr, pi);
      }
      tile[e] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < args.b0 * args.b1 * args.b2; e += blockDim.x) {
      const int i2 = e % args.b2, i1 = (e / args.b2) % args.b1, i0 = e / (args.b1 * args.b2);
      const int gx = x0 + i0, gy = y0 + i1, gz = z0 + i2;
      if (gx >= args.n0 || gy >= args.n1 || gz >= args.n2) continue;
      constexpr bool DIFF = sizeof(R) == 4;
      const T xc0 = tile[((i0 + M) * E1 + (i1 + M)) * E2 + (i2 + M)];
      T x = DIFF ? scale((R)args.csum, xc0) : zero<T>();
      for (int p = 0; p < args.np; ++p) {
        const int j = ((i0 + M + args.off[p][0]) * E1 + (i1 + M + args.off[p][1])) * E2 + (i2 + M + args.off[p][2]);
        x = fmadd(x, (R)args.coef[p], DIFF ? sub(tile[j], xc0) : tile[j]);
      }
      const int64_t gidx = (int64_t)gx * n12 + (int64_t)gy * args.n2 + gz;
      if (args.alpha != 1.0 || args.beta != 0.0 || args.y || args.vpot) {
        const T xc = tile[((i0 + M) * E1 + (i1 + M)) * E2 + (i2 + M)];
        x = fmadd(scale((R)args.alpha, x), (R)args.beta, xc);
        if (args.y) x = fmadd(x, (R)args.gamma, reinterpret_cast<const T*>(args.y)[band * n012 + gidx]);
        if (args.vpot) x = fmadd(x, reinterpret_cast<const R*>(args.vpot)[gidx], xc);
      }
      dst[gidx] = x;
    }
  }
}

// --------------------------------------------------------------------------
// Jacobi relaxation (relax_method 2 of c/bmgs/relax.c:40-66) for real FP64:
//   f <- (1-w) f + w (s - sum_{p != 0} c_p f[. + o_p]) / c_0
// One sweep per launch; the halo is resolved like box_kernel.
__global__ void jacobi_kernel(const BoxArgs args, const double* f_in, double* f_out,
                              const double* s, double w, double c_center) {
  const int64_t n12 = (int64_t)args.n1 * args.n2, N = n12 * args.n0;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < N; g += (int64_t)gridDim.x * blockDim.x) {
    const int i0 = (int)(g / n12), i1 = (int)((g / args.n2) % args.n1), i2 = (int)(g % args.n2);
    double x = 0.0;
    for (int p = 0; p < args.np; ++p) {
      if (args.off[p][0] == 0 && args.off[p][1] == 0 && args.off[p][2] == 0) continue;
      int c3[3] = {i0 + args.off[p][0], i1 + args.off[p][1], i2 + args.off[p][2]};
      const int n[3] = {args.n0, args.n1, args.n2};
      const int pbc[3] = {args.pbc0, args.pbc1, args.pbc2};
      bool z = false;
      for (int c = 0; c < 3; ++c)
        if (c3[c] < 0 || c3[c] >= n[c]) {
          if (!pbc[c]) { z = true; break; }
          c3[c] = wrap_index(c3[c], n[c]);
        }
      if (!z) x += args.coef[p] * f_in[(int64_t)c3[0] * n12 + (int64_t)c3[1] * args.n2 + c3[2]];
    }
    f_out[g] = (1.0 - w) * f_in[g] + w * (s[g] - x) / c_center;
  }
}

}  // namespace gb

namespace gb {


template <typename T, int H>
static int launch_star(const gb_operator* op, const void* in, void* out, int64_t nin,
                       const double* phase_cd, cudaStream_t stream, const Epilogue& ep, int nk) {
  StarArgs a{};
  a.in = in; a.out = out; a.nbatch = nin;
  a.n0 = (int)op->n[0]; a.n1 = (int)op->n[1]; a.n2 = (int)op->n[2];
  a.pbc0 = op->pbc[0]; a.pbc1 = op->pbc[1]; a.pbc2 = op->pbc[2];
  a.c0 = op->center;
  a.c0diff = op->center;
  for (int c = 0; c < 3; ++c)
    for (int m = 0; m < 2 * HMAX + 1; ++m) a.c0diff += op->a[c][m];
  memcpy(a.a, op->a, sizeof(a.a));
  a.alpha = ep.alpha; a.beta = ep.beta; a.gamma = ep.gamma; a.y = ep.y; a.vpot = ep.vpot;
  fill_phase_sets(a.phs, phase_cd, nk, nin);
  // chunks of at most 24 planes (the 2H planes before each are read again,
  // from L2), shorter ones up to eight blocks per SM (with sixteen, more of
  // those planes: 160 FP32 bands of 14^3, radius 3: 16.7 against 12.5 us)
  a.tiles = ceil_div((int64_t)a.n1 * a.n2, 256);
  const int64_t cols = nin * a.tiles;
  a.chunks = (int)std::max<int64_t>(ceil_div(a.n0, 24),
                                    std::min<int64_t>(a.n0, ceil_div((int64_t)sm_count() * 8, cols)));
  const unsigned blocks = (unsigned)(cols * a.chunks);
  const bool per = a.pbc0 || a.pbc1 || a.pbc2;
  // FP32: in pairs of offsets where the row kernel has that form too
  if constexpr (std::is_same<T, float>::value && (H == 1 || H == 3)) {
    if (symmetric_stencil<float>(op)) {
      if (per) march_star_kernel<T, H, true, true><<<blocks, 256, 0, stream>>>(a);
      else march_star_kernel<T, H, false, true><<<blocks, 256, 0, stream>>>(a);
      return check_launch("march_star_kernel");
    }
  }
  if (per) march_star_kernel<T, H, true, false><<<blocks, 256, 0, stream>>>(a);
  else march_star_kernel<T, H, false, false><<<blocks, 256, 0, stream>>>(a);
  return check_launch("march_star_kernel");
}

template <typename T>
static int dispatch_star(const gb_operator* op, const void* in, void* out, int64_t nin,
                         const double* ph, cudaStream_t st, const Epilogue& ep, int nk) {
  switch (op->H) {
    case 1: return launch_star<T, 1>(op, in, out, nin, ph, st, ep, nk);
    case 2: return launch_star<T, 2>(op, in, out, nin, ph, st, ep, nk);
    case 3: return launch_star<T, 3>(op, in, out, nin, ph, st, ep, nk);
    case 4: return launch_star<T, 4>(op, in, out, nin, ph, st, ep, nk);
    case 5: return launch_star<T, 5>(op, in, out, nin, ph, st, ep, nk);
    case 6: return launch_star<T, 6>(op, in, out, nin, ph, st, ep, nk);
    default: return fail(GB_E_UNSUPPORTED, "star stencil radius > 6");
  }
}

static void fill_box_args(const gb_operator* op, BoxArgs& a, const double* phase_cd, int nk = 1,
                          int64_t nbatch = 1) {
  memset(&a, 0, sizeof(a));
  a.alpha = 1.0;
  a.n0 = (int)op->n[0]; a.n1 = (int)op->n[1]; a.n2 = (int)op->n[2];
  a.pbc0 = op->pbc[0]; a.pbc1 = op->pbc[1]; a.pbc2 = op->pbc[2];
  a.M = op->range;
  a.np = op->np;
  a.csum = 0.0;
  for (int p = 0; p < op->np; ++p) {
    a.coef[p] = op->coef[p];
    a.csum += op->coef[p];
    for (int c = 0; c < 3; ++c) a.off[p][c] = op->off[p * 3 + c];
  }
  fill_phase_sets(a.phs, phase_cd, nk, nbatch);
}

template <typename T>
static int launch_box(const gb_operator* op, const void* in, void* out, int64_t nin,
                      const double* phase_cd, cudaStream_t stream, const Epilogue& ep, int nk) {
  BoxArgs a;
  fill_box_args(op, a, phase_cd, nk, nin);
  a.alpha = ep.alpha; a.beta = ep.beta; a.gamma = ep.gamma; a.y = ep.y; a.vpot = ep.vpot;
  a.in = in; a.out = out; a.nbatch = nin;
  a.b0 = 4; a.b1 = 8; a.b2 = 32;
  const int M = a.M;
  size_t smem = (size_t)(a.b0 + 2 * M) * (a.b1 + 2 * M) * (a.b2 + 2 * M) * sizeof(T);
  while (smem > 200 * 1024 && a.b2 > 8) {
    a.b2 /= 2;
    smem = (size_t)(a.b0 + 2 * M) * (a.b1 + 2 * M) * (a.b2 + 2 * M) * sizeof(T);
  }
  a.tiles0 = ceil_div(a.n0, a.b0); a.tiles1 = ceil_div(a.n1, a.b1); a.tiles2 = ceil_div(a.n2, a.b2);
  cudaFuncSetAttribute(box_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int64_t work = nin * (int64_t)a.tiles0 * a.tiles1 * a.tiles2;
  const int64_t blocks = std::min<int64_t>(work, (int64_t)sm_count() * 8);
  box_kernel<T><<<(unsigned)std::max<int64_t>(blocks, 1), 256, smem, stream>>>(a);
  return check_launch("box_kernel");
}

// internal entry used by gb_operator_apply and the preconditioner chain
int op_apply(const gb_operator* op, const void* in, void* out, int64_t nin, int dtype,
             const double* ph, cudaStream_t st, const Epilogue& ep, int nk) {
  if (nk > KMAX) return fail(GB_E_UNSUPPORTED, "more k-point phase sets than one launch takes");
  if (nk > 1 && nin % nk) return fail(GB_E_INVALID, "batch not divisible by the number of phase sets");
  if (op->cfd) {
    const int rc = star_tma_apply(op, in, out, nin, dtype, ph, st, ep, nk);
    if (rc != 1) return rc;
    if (stencil_path() == 2)
      return fail(GB_E_UNSUPPORTED, std::string("TMA stencil path required but not applicable: ") + tma_reason());
    int rr = star_rows_apply(op, in, out, nin, dtype, ph, st, ep, nk);
    if (rr == USE_TILES) rr = star_tiles_apply(op, in, out, nin, dtype, ph, st, ep, nk);
    if (rr != USE_MARCH) return rr;
    switch (dtype) {
      case GB_DTYPE_F64: return dispatch_star<double>(op, in, out, nin, ph, st, ep, nk);
      case GB_DTYPE_F32: return dispatch_star<float>(op, in, out, nin, ph, st, ep, nk);
      case GB_DTYPE_C128: return dispatch_star<double2>(op, in, out, nin, ph, st, ep, nk);
      default: return dispatch_star<float2>(op, in, out, nin, ph, st, ep, nk);
    }
  }
  switch (dtype) {
    case GB_DTYPE_F64: return launch_box<double>(op, in, out, nin, ph, st, ep, nk);
    case GB_DTYPE_F32: return launch_box<float>(op, in, out, nin, ph, st, ep, nk);
    case GB_DTYPE_C128: return launch_box<double2>(op, in, out, nin, ph, st, ep, nk);
    default: return launch_box<float2>(op, in, out, nin, ph, st, ep, nk);
  }
}

}  // namespace gb

using namespace gb;

extern "C" {

int gb_operator_new(const double* coef_p, const int64_t* offset_p, int np,
                    const int64_t size_c[3], int range, const int64_t neighbor_cd[6],
                    int real, int cfd, gb_operator** out) {
  GB_REQUIRE(out && coef_p && offset_p && size_c && neighbor_cd, "gb_operator_new: null pointer");
  GB_REQUIRE(np > 0 && np <= 64, "gb_operator_new: 1 <= np <= 64 stencil points required");
  GB_REQUIRE(range >= 0 && range <= 6, "gb_operator_new: stencil range must be in [0, 6]");
  for (int c = 0; c < 3; ++c) {
    GB_REQUIRE(size_c[c] > 0 && size_c[c] < (1 << 30), "gb_operator_new: bad grid size");
    // the reference asserts the same ("Stencil longer than domain",
    // gpaw/fd_operators.py:53)
    GB_REQUIRE(range <= size_c[c], "gb_operator_new: stencil longer than domain");
  }
  auto* op = new (std::nothrow) gb_operator();
  if (!op) return fail(GB_E_NOMEM, "gb_operator_new: out of host memory");
  op->np = np;
  op->range = range;
  op->real = real;
  for (int c = 0; c < 3; ++c) {
    op->n[c] = size_c[c];
    // single domain: a neighbour >= 0 on an axis means periodic wrap
    op->pbc[c] = (neighbor_cd[2 * c] >= 0 || neighbor_cd[2 * c + 1] >= 0) ? 1 : 0;
  }
  const int64_t M1 = size_c[1] + 2 * range, M2 = size_c[2] + 2 * range;
  op->coef.assign(coef_p, coef_p + np);
  op->off.resize(np * 3);
  bool on_axes = true;
  int H = 0;
  op->diag = 0.0;
  for (int p = 0; p < np; ++p) {
    // decode the linear padded-array offset o0*M1*M2 + o1*M2 + o2, |o_c| <= range
    int64_t o = offset_p[p];
    int64_t o0 = (o >= 0 ? o + (M1 * M2) / 2 : o - (M1 * M2) / 2) / (M1 * M2);
    int64_t r = o - o0 * M1 * M2;
    int64_t o1 = (r >= 0 ? r + M2 / 2 : r - M2 / 2) / M2;
    int64_t o2 = r - o1 * M2;
    if (std::llabs(o0) > range || std::llabs(o1) > range || std::llabs(o2) > range) {
      delete op;
      return fail(GB_E_INVALID, "gb_operator_new: offset outside the padded range");
    }
    op->off[p * 3 + 0] = (int)o0;
    op->off[p * 3 + 1] = (int)o1;
    op->off[p * 3 + 2] = (int)o2;
    const int nz = (o0 != 0) + (o1 != 0) + (o2 != 0);
    if (nz >= 2) on_axes = false;
    H = std::max<int>(H, (int)std::max({std::llabs(o0), std::llabs(o1), std::llabs(o2)}));
    if (o == 0) op->diag = coef_p[p];   // last zero-offset coefficient wins, as in c/operators.c:332-334
  }
  op->cfd = on_axes ? 1 : 0;
  (void)cfd;
  op->H = H;
  op->center = 0.0;
  memset(op->a, 0, sizeof(op->a));
  for (int p = 0; p < np; ++p) {
    const int* o = &op->off[p * 3];
    if (o[0] == 0 && o[1] == 0 && o[2] == 0) { op->center += coef_p[p]; continue; }
    for (int c = 0; c < 3; ++c)
      if (o[c] != 0) op->a[c][o[c] + HMAX] += coef_p[p];
  }
  if (op->H == 0) op->H = 1;
  *out = op;
  return GB_OK;
}

int gb_operator_apply(const gb_operator* op, const void* in, void* out, int64_t nin, int dtype,
                      const double* phase_cd, void* stream) {
  GB_REQUIRE(op, "gb_operator_apply: null operator");
  GB_REQUIRE(dtype_valid(dtype), "gb_operator_apply: unknown dtype");
  GB_REQUIRE(nin >= 0, "gb_operator_apply: negative batch");
  GB_REQUIRE(dtype_complex(dtype) == !op->real,
             "gb_operator_apply: dtype does not match the operator's real/complex flag");
  if (nin == 0) return GB_OK;
  GB_REQUIRE(in && out, "gb_operator_apply: null data pointer");
  GB_REQUIRE(in != out, "gb_operator_apply: in and out must not alias");
  GB_REQUIRE(!dtype_complex(dtype) || phase_cd, "gb_operator_apply: complex data needs phase_cd");
  cudaStream_t st = (cudaStream_t)stream;
  const double* ph = dtype_complex(dtype) ? phase_cd : nullptr;
  return op_apply(op, in, out, nin, dtype, ph, st, Epilogue());
}

int gb_operator_apply_potential(const gb_operator* op, const void* in, void* out, int64_t nin, int dtype,
                                const void* vt, const double* phase_cd, void* stream) {
  GB_REQUIRE(op && vt, "gb_operator_apply_potential: null operator or potential");
  GB_REQUIRE(dtype_valid(dtype) && nin >= 0, "gb_operator_apply_potential: bad dtype or batch");
  GB_REQUIRE(dtype_complex(dtype) == !op->real,
             "gb_operator_apply_potential: dtype does not match the operator's real/complex flag");
  if (nin == 0) return GB_OK;
  GB_REQUIRE(in && out && in != out, "gb_operator_apply_potential: bad data pointers");
  GB_REQUIRE(!dtype_complex(dtype) || phase_cd, "gb_operator_apply_potential: complex data needs phase_cd");
  Epilogue ep;
  ep.vpot = vt;
  return op_apply(op, in, out, nin, dtype, dtype_complex(dtype) ? phase_cd : nullptr, (cudaStream_t)stream, ep);
}

int gb_operator_apply_k(const gb_operator* op, const void* in, void* out, int64_t nin, int dtype, int nk,
                        const double* phase_kcd, const void* vt, void* stream) {
  GB_REQUIRE(op, "gb_operator_apply_k: null operator");
  GB_REQUIRE(dtype_valid(dtype) && nin >= 0, "gb_operator_apply_k: bad dtype or batch");
  GB_REQUIRE(dtype_complex(dtype) == !op->real,
             "gb_operator_apply_k: dtype does not match the operator's real/complex flag");
  GB_REQUIRE(nk >= 1 && nk <= KMAX, "gb_operator_apply_k: nk must be 1 .. 8");
  GB_REQUIRE(nin % nk == 0, "gb_operator_apply_k: the batch must split into nk equal groups");
  if (nin == 0) return GB_OK;
  GB_REQUIRE(in && out && in != out, "gb_operator_apply_k: bad data pointers");
  GB_REQUIRE(!dtype_complex(dtype) || phase_kcd, "gb_operator_apply_k: complex data needs phases");
  Epilogue ep;
  ep.vpot = vt;
  return op_apply(op, in, out, nin, dtype, dtype_complex(dtype) ? phase_kcd : nullptr, (cudaStream_t)stream, ep,
                  nk);
}

int gb_operator_relax(const gb_operator* op, int relax_method, double* f_g, const double* s_g,
                      int nrelax, double w, void* stream) {
  GB_REQUIRE(op && f_g && s_g, "gb_operator_relax: null pointer");
  GB_REQUIRE(op->real, "gb_operator_relax: real operators only");
  if (relax_method != 2)
    return fail(GB_E_UNSUPPORTED, "gb_operator_relax: only weighted Jacobi (method 2) is implemented");
  GB_REQUIRE(op->diag != 0.0, "gb_operator_relax: zero diagonal");
  BoxArgs a;
  fill_box_args(op, a, nullptr);
  const int64_t N = op->n[0] * op->n[1] * op->n[2];
  double* tmp = nullptr;
  if (cudaMallocAsync(&tmp, N * sizeof(double), (cudaStream_t)stream) != cudaSuccess)
    return fail(GB_E_NOMEM, "gb_operator_relax: scratch allocation failed");
  const int blocks = (int)std::min<int64_t>((N + 255) / 256, (int64_t)sm_count() * 8);
  for (int it = 0; it < nrelax; ++it) {
    jacobi_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(a, f_g, tmp, s_g, w, op->diag);
    cudaMemcpyAsync(f_g, tmp, N * sizeof(double), cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
  }
  cudaFreeAsync(tmp, (cudaStream_t)stream);
  return check_launch("jacobi_kernel");
}

int gb_operator_get_diagonal_element(const gb_operator* op, double* d) {
  GB_REQUIRE(op && d, "gb_operator_get_diagonal_element: null pointer");
  *d = op->diag;
  return GB_OK;
}

int gb_operator_free(gb_operator* op) {
  delete op;
  return GB_OK;
}

}  // extern "C"
