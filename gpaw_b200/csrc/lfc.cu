// Localized functions: add / integrate (replaces _gpaw.LFC: c/lfc.c:146-257
// NewLFCObject, 432-505 integrate, 818-885 add, c/lfc.h:79-130 GRID_LOOP).
//
// The reference walks the merged, sorted list of sphere boundaries once per
// band on one core.  Here the same sweep runs once, on the host, when the
// object is built (positions change rarely), and produces two device-side
// indexings of the (grid point, volume, row) incidence:
//
//  * point-major (add):  every grid point covered by at least one sphere owns
//    one thread; it sums  sum_W conj(phase_W) sum_m A_W[row][m] c[x][M_W + m]
//    over the volumes covering it and adds to a[x][G] -- every a[x][G] has a
//    single writer, so there are no atomics and results are deterministic.
//  * function-group-major (integrate): a group is one (atom, radial function)
//    M-range with all its periodic images; one CTA per (group, band block)
//    reduces dv * phase_W * sum_G a[x][G] A_W[row][m] over every image and
//    adds the block's result to c[x][M..M+nm) -- again a single writer.
//
// Derivatives (gb_lfc_derivative, c/lfc.c:1449-1601) are computed on the
// fly from the radial splines: one CTA per (function group, band) walks the
// group's rows, evaluates d/dr_v [f(r) r^l Y_lm] at each point (spline value
// and slope, solid harmonics and their gradients) and reduces
// dv sum_G a[x][G] phase_W d/dr_v Phi to c[x][M][v] -- a single writer.
#include <algorithm>
#include <cstring>
#include <map>
#include <type_traits>
#include <vector>
#include <cooperative_groups.h>
#include "internal.cuh"
#include "spline.cuh"

struct gb_lfc {
  int nW = 0, nM = 0, maxnm = 0;
  int64_t nG = 0;
  double dv = 1.0;
  int nq = 0;
  // device data
  double* A64 = nullptr;      // concatenated rows of every volume
  float* A32 = nullptr;
  int64_t nA = 0;             // doubles in A
  double2* phase = nullptr;   // [nq][nW]
  // add (point-major)
  int64_t P = 0;              // covered points
  int* pt_G = nullptr;        // [P]
  int* pt_off = nullptr;      // [P+1] into contributions
  int64_t C = 0;              // contributions
  int64_t* ct_aoff = nullptr; // [C] offset into A (doubles)
  int* ct_M = nullptr;        // [C]
  int* ct_nm = nullptr;       // [C]
  int* ct_W = nullptr;        // [C]
  // zero-padded FP32 rows of A in contribution order (FP32 real add outside
  // the bricks, at most 16 functions per volume)
  int pad_nm = 0;             // 8 or 16; 0 = not built
  bool pad_full = false;      // every contribution has pad_nm functions at a multiple of 4
  float* A32p = nullptr;      // [C][pad_nm]
  // integrate (group-major)
  int ngroups = 0;
  int* gr_M = nullptr;        // [ngroups]
  int* gr_nm = nullptr;       // [ngroups]
  int* gr_voff = nullptr;     // [ngroups+1] into the volume list
  int* gv_W = nullptr;        // [nW] volumes ordered by group
  int64_t* vol_row0 = nullptr;  // [nW] first global row of W
  int64_t* vol_row1 = nullptr;  // [nW] one past last
  int* row_G = nullptr;       // [rows] grid point of every global row
  int64_t* vol_aoff = nullptr;  // [nW] offset (doubles) of row0 in A
  std::vector<int> h_gr_nm;
  // tensor-core add / integrate for FP64 real data (every volume has <= 16
  // functions): one entry per (volume, 8-point sub-tile of the flattened grid
  // it touches) with its values there as maxnm dense rows [m][p]
  int nf = 0;                 // blocks of 8 functions per entry, 1 or 2; 0 = not built
  int ns = 0;                 // sub-tiles with entries
  int4* st_sub = nullptr;     // [ns][2] sub-tile | mask of its covered points | its entries' range,
                              //   then the first entry's st_M
  int2* st_M = nullptr;       // [ne] first function | function count + covered points << 8 of an entry
  double* st_A = nullptr;     // [ne][maxnm][8]
  int* sg_off = nullptr;      // [ngroups + 1] entries of each function group:
  int4* sg_e = nullptr;       //   entry | sub-tile | covered points, in the order of the sub-tiles
  // brick-tiled FP32 add / integrate for real data (every volume has <= 8
  // functions, nG a multiple of 4): 32-point chunks of four 8-point
  // sub-tiles; one entry per (volume, sub-tile it touches) with the volume's
  // values there as a dense [m][p] 8 x 8 block (zero where the volume does
  // not cover the point or m >= nm); bricks of consecutive chunks
  bool tiled = false;
  int* tch_c = nullptr;       // [nch] chunk index of every chunk with entries
  int* tch_eoff = nullptr;    // [4 nch + 1] entries of (chunk, sub-tile)
  int* te_info = nullptr;     // [ne] slot in its brick | nm << 8
  float* te_A = nullptr;      // [ne][8][8]
  int tbr_n = 0;              // bricks
  int tbr_smax = 1;           // most slots in a brick
  int tbr_emax = 0;           // most entries in a brick
  int tnm = 0;                // functions of every group, 0: they differ
  int* tbr_ch0 = nullptr;     // [tbr_n + 1] chunk range of each brick
  int* tbr_pbase = nullptr;   // [tbr_n + 1] first (brick, slot) pair
  int64_t tpart_n = 0;        // (brick, slot) pairs
  int* tps_M = nullptr;       // [tpart_n] their group's first function
  int* tps_nm = nullptr;      // [tpart_n] and function count
  int* tps_eoff = nullptr;    // [tpart_n + 1] their entries:
  int* tps_info = nullptr;    //   (entry - brick's first) | sub-tile << 16 | nm << 24
  int* tgr_poff = nullptr;    // [ngroups + 1] the (brick, slot) pairs of each
  int* tgr_pidx = nullptr;    //   group, in brick order
  // work space of the tiled path (transposed coefficients, partial sums);
  // grown outside stream capture only
  mutable void* work = nullptr;
  mutable size_t work_bytes = 0;
  std::vector<void*> allocations;
};

namespace gb {

// trivially-copyable device view passed to the kernels
struct LfcView {
  int nW, nM;
  int64_t nG;
  double dv;
  const double2* phase;
  int64_t P;
  const int* pt_G;
  const int* pt_off;
  const int64_t* ct_aoff;
  const int* ct_M;
  const int* ct_nm;
  const int* ct_W;
  const int* gr_M;
  const int* gr_nm;
  const int* gr_voff;
  const int* gv_W;
  const int64_t* vol_row0;
  const int64_t* vol_row1;
  const int* row_G;
  const int64_t* vol_aoff;
};

// grid geometry for on-the-fly positions (h_cv row-major, local sizes, and
// the global index of the local grid's first point)
struct DerivGeom {
  double h[9];
  int64_t n[3], beg[3];
};

static LfcView view(const gb_lfc* l) {
  LfcView v;
  v.nW = l->nW; v.nM = l->nM; v.nG = l->nG; v.dv = l->dv; v.phase = l->phase;
  v.P = l->P; v.pt_G = l->pt_G; v.pt_off = l->pt_off; v.ct_aoff = l->ct_aoff;
  v.ct_M = l->ct_M; v.ct_nm = l->ct_nm; v.ct_W = l->ct_W; v.gr_M = l->gr_M; v.gr_nm = l->gr_nm;
  v.gr_voff = l->gr_voff; v.gv_W = l->gv_W; v.vol_row0 = l->vol_row0;
  v.vol_row1 = l->vol_row1; v.row_G = l->row_G; v.vol_aoff = l->vol_aoff;
  return v;
}

template <typename T>
static T* dalloc(gb_lfc* l, size_t n) {
  void* p = nullptr;
  if (n == 0) n = 1;
  if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) return nullptr;
  l->allocations.push_back(p);
  return reinterpret_cast<T*>(p);
}

template <typename T>
static bool upload(gb_lfc* l, T** dst, const std::vector<T>& src) {
  *dst = dalloc<T>(l, src.size());
  if (!*dst) return false;
  if (!src.empty() && cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
    return false;
  return true;
}

// --------------------------------------------------------------------- add
template <typename T> struct AType { using A = double; };
template <> struct AType<float> { using A = float; };
template <> struct AType<float2> { using A = float; };

// a row of NMAX values of A (or of the coefficients): 16-byte loads when the
// row is full (nm == NMAX == 8) and 16-byte aligned -- a warp then reads its
// 32 rows in two (FP32) or four (FP64) wide requests instead of 8 strided
// ones -- element loads otherwise
template <typename V, int NMAX>
__device__ __forceinline__ void load_row(const V* __restrict__ src, int nm, V (&dst)[NMAX]) {
  if constexpr (NMAX == 8 && (sizeof(V) == 4 || sizeof(V) == 8)) {
    if (nm == 8 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      if constexpr (sizeof(V) == 4) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(src));
        const float4 b = __ldg(reinterpret_cast<const float4*>(src) + 1);
        dst[0] = a.x; dst[1] = a.y; dst[2] = a.z; dst[3] = a.w;
        dst[4] = b.x; dst[5] = b.y; dst[6] = b.z; dst[7] = b.w;
      } else {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const double2 a = __ldg(reinterpret_cast<const double2*>(src) + h);
          dst[2 * h] = a.x;
          dst[2 * h + 1] = a.y;
        }
      }
      return;
    }
  }
#pragma unroll
  for (int m = 0; m < NMAX; ++m) dst[m] = m < nm ? src[m] : (V)0;
}

// one thread per covered point and XB bands; a contribution's NMAX-padded A
// row is loaded once and reused for every band (runtime nm <= NMAX)
template <typename T, int XB, int NMAX>
__global__ void __launch_bounds__(256) lfc_add_kernel(const LfcView l, const typename AType<T>::A* __restrict__ A,
                                                      const T* __restrict__ c_xM, T* __restrict__ a_xG, int64_t nx,
                                                      int q, int64_t per_q) {
  using R = typename Elem<T>::R;
  constexpr bool CPLX = Elem<T>::cplx;
  const int64_t x0 = (int64_t)blockIdx.y * XB;
  const int nb = (int)(nx - x0 < XB ? nx - x0 : XB);
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < l.P; p += (int64_t)gridDim.x * blockDim.x) {
    const int G = l.pt_G[p];
    T acc[XB];
#pragma unroll
    for (int i = 0; i < XB; ++i) acc[i] = zero<T>();
    const int c1 = l.pt_off[p + 1];
    for (int c = l.pt_off[p]; c < c1; ++c) {
      const typename AType<T>::A* Ar = A + l.ct_aoff[c];
      const int M = l.ct_M[c], nm = l.ct_nm[c];
      typename AType<T>::A Aw[NMAX];
      load_row<typename AType<T>::A, NMAX>(Ar, nm, Aw);
      R Av[NMAX];
#pragma unroll
      for (int m = 0; m < NMAX; ++m) Av[m] = (R)Aw[m];
      double pr = 1.0, pi = 0.0;
      if (CPLX && q >= 0 && per_q == 0) {
        const double2 ph = l.phase[(int64_t)q * l.nW + l.ct_W[c]];
        pr = ph.x; pi = -ph.y;   // conj(phase) (c/lfc.c:864)
      }
#pragma unroll
      for (int i = 0; i < XB; ++i) {
        if (i < nb) {
          if (CPLX && q >= 0 && per_q > 0) {
            // k-point of this band: q + band / per_q
            const double2 ph = l.phase[(q + (x0 + i) / per_q) * l.nW + l.ct_W[c]];
            pr = ph.x; pi = -ph.y;
          }
          const T* cx = c_xM + (x0 + i) * l.nM + M;
          T s = zero<T>();
          if constexpr (!CPLX) {
            T cv[NMAX];
            load_row<T, NMAX>(cx, nm, cv);
#pragma unroll
            for (int m = 0; m < NMAX; ++m) s = fmadd(s, Av[m], cv[m]);
          } else {
#pragma unroll
            for (int m = 0; m < NMAX; ++m)
              if (m < nm) s = fmadd(s, Av[m], cx[m]);
          }
          acc[i] = add(acc[i], CPLX ? phase_mul(s, pr, pi) : s);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < XB; ++i) {
      if (i < nb) {
        T* ap = a_xG + (x0 + i) * l.nG + G;
        *ap = add(*ap, acc[i]);
      }
    }
  }
}

// --------------------------------------------------------------- integrate
// one CTA per (function group, XB bands); a group is one atom (all its
// radial functions merged, nm <= NM of them) with all its periodic images
template <typename T, int NM, int XB, int NT>
__global__ void __launch_bounds__(NT) lfc_integrate_kernel(const LfcView l, const typename AType<T>::A* __restrict__ A,
                                                          const T* __restrict__ a_xG, T* __restrict__ c_xM,
                                                          int64_t nx, int q, int group_base, int64_t per_q) {
  using R = typename Elem<T>::R;
  constexpr bool CPLX = Elem<T>::cplx;
  __shared__ T red[NT / 32][XB * NM];
  const int g = group_base + blockIdx.x;
  const int64_t x0 = (int64_t)blockIdx.y * XB;
  const int M = l.gr_M[g];
  const int nm = l.gr_nm[g];
  T acc[XB][NM];
#pragma unroll
  for (int i = 0; i < XB; ++i)
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[i][m] = zero<T>();
  for (int vi = l.gr_voff[g]; vi < l.gr_voff[g + 1]; ++vi) {
    const int W = l.gv_W[vi];
    const int64_t r0 = l.vol_row0[W], r1 = l.vol_row1[W];
    const typename AType<T>::A* AW = A + l.vol_aoff[W];
    double pr = 1.0, pi = 0.0;
    if (CPLX && q >= 0) {
      const double2 ph = l.phase[(int64_t)q * l.nW + W];
      pr = ph.x; pi = ph.y;
    }
    if constexpr (!CPLX) {
      // real data: every image has phase 1, accumulate straight into acc
      // FP32: four rows per pass put 16 gathered loads in flight (1.1x on
      // the Si64 shape); FP64 measured no faster unrolled
      constexpr int RUN = sizeof(R) == 4 ? 4 : 1;
#pragma unroll RUN
      for (int64_t r = r0 + threadIdx.x; r < r1; r += NT) {
        const int G = l.row_G[r];
        typename AType<T>::A Aw[NM];
        load_row<typename AType<T>::A, NM>(AW + (r - r0) * nm, nm, Aw);
        R Ar[NM];
#pragma unroll
        for (int m = 0; m < NM; ++m) Ar[m] = (R)Aw[m];
#pragma unroll
        for (int i = 0; i < XB; ++i) {
          if (x0 + i < nx) {
            const T v = a_xG[(x0 + i) * l.nG + G];
#pragma unroll
            for (int m = 0; m < NM; ++m) acc[i][m] = fmadd(acc[i][m], Ar[m], v);
          }
        }
      }
    } else {
      T part[XB][NM];
#pragma unroll
      for (int i = 0; i < XB; ++i)
#pragma unroll
        for (int m = 0; m < NM; ++m) part[i][m] = zero<T>();
      for (int64_t r = r0 + threadIdx.x; r < r1; r += NT) {
        const int G = l.row_G[r];
        R Ar[NM];
#pragma unroll
        for (int m = 0; m < NM; ++m) Ar[m] = m < nm ? (R)AW[(r - r0) * nm + m] : (R)0;
#pragma unroll
        for (int i = 0; i < XB; ++i) {
          if (x0 + i < nx) {
            const T v = a_xG[(x0 + i) * l.nG + G];
#pragma unroll
            for (int m = 0; m < NM; ++m) part[i][m] = fmadd(part[i][m], Ar[m], v);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < XB; ++i) {
        double qr = pr, qi = pi;
        if (q >= 0 && per_q > 0 && x0 + i < nx) {
          const double2 ph = l.phase[(q + (x0 + i) / per_q) * l.nW + W];
          qr = ph.x; qi = ph.y;
        }
#pragma unroll
        for (int m = 0; m < NM; ++m) acc[i][m] = add(acc[i][m], phase_mul(part[i][m], qr, qi));
      }
    }
  }
  // block reduction: warp shuffles, then across warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < XB; ++i)
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      T v = acc[i][m];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if constexpr (CPLX) {
          v.x += __shfl_down_sync(0xffffffffu, v.x, o);
          v.y += __shfl_down_sync(0xffffffffu, v.y, o);
        } else {
          v += __shfl_down_sync(0xffffffffu, v, o);
        }
      }
      if (lane == 0) red[warp][i * NM + m] = v;
    }
  __syncthreads();
  for (int e = threadIdx.x; e < XB * NM; e += NT) {
    const int i = e / NM, m = e % NM;
    if (x0 + i >= nx || m >= nm) continue;
    T v = zero<T>();
    for (int w = 0; w < NT / 32; ++w) v = add(v, red[w][e]);
    T* cp = c_xM + (x0 + i) * l.nM + M + m;
    *cp = fmadd(*cp, (R)l.dv, v);
  }
}

// -------------------------------------- FP32 real data outside the bricks
// One thread per covered point holds the zero-padded A rows of its first KREG
// contributions in registers (a copy of A in contribution order, so a warp's
// row loads are contiguous) and loops over the bands XU at a time, issuing the
// XU read-modify-write loads of a[x][G] before the coefficient loads and FMAs
// of those bands.  Per band it sums the contributions in point order, m within
// each, as lfc_add_kernel does: the same bits.  (FP32 data widened for the FP64
// matrix instructions below were slower for most calls: 72^3 zero-boundary
// grid, 24 atoms with 5 functions, 160 bands: add 111 against 76 us, integrate
// 163 against 39 us.)
template <int NMAX, bool FULL>
__device__ __forceinline__ void load_coef(const float* __restrict__ cx, int nm, float (&v)[NMAX]) {
  if constexpr (FULL) {
#pragma unroll
    for (int h = 0; h < NMAX / 4; ++h) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(cx) + h);
      v[4 * h] = a.x; v[4 * h + 1] = a.y; v[4 * h + 2] = a.z; v[4 * h + 3] = a.w;
    }
  } else {
#pragma unroll
    for (int m = 0; m < NMAX; ++m) v[m] = m < nm ? __ldg(cx + m) : 0.f;
  }
}

// acc[u] += sum_m A[m] c[x0 + u][M + m], u < NU, cx = &c[x0][M] (the
// contribution's sum is formed first, then added)
template <int NMAX, bool FULL, int NU>
__device__ __forceinline__ void add_contribution(const float (&A)[NMAX], const float* __restrict__ cx, int nM, int nm,
                                                 float (&acc)[NU]) {
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    float cv[NMAX];
    load_coef<NMAX, FULL>(cx, nm, cv);
    float t = 0.f;
#pragma unroll
    for (int m = 0; m < NMAX; ++m) t = fmadd(t, A[m], cv[m]);
    acc[u] += t;
    cx += nM;
  }
}

// bands x0 .. x0 + NU - 1 of one point: a[x][G] += sum_k sum_m A_k[m] c[x][M_k + m]
template <int NMAX, int KREG, bool FULL, int NU>
__device__ __forceinline__ void add_point_bands(const float (&A)[KREG][NMAX], const float* const (&cb)[KREG],
                                                const int (&nmk)[KREG], int K, int k0, const int* __restrict__ ct_M,
                                                const int* __restrict__ ct_nm, const float* __restrict__ Ap,
                                                const float* __restrict__ c_xM, int nM, int64_t x0,
                                                float* __restrict__ ax, int64_t nG) {
  float av[NU], acc[NU];
  float* q = ax;
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    av[u] = *q;
    acc[u] = 0.f;
    q += nG;
  }
  const int64_t xo = x0 * nM;
#pragma unroll
  for (int k = 0; k < KREG; ++k)
    if (k < K) add_contribution<NMAX, FULL, NU>(A[k], cb[k] + xo, nM, nmk[k], acc);
  for (int k = KREG; k < K; ++k) {
    float Ak[NMAX];
    load_coef<NMAX, true>(Ap + (int64_t)(k0 + k) * NMAX, NMAX, Ak);
    add_contribution<NMAX, FULL, NU>(Ak, c_xM + ct_M[k0 + k] + xo, nM, ct_nm[k0 + k], acc);
  }
  q = ax;
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    *q = av[u] + acc[u];
    q += nG;
  }
}

template <int NMAX, int KREG, bool FULL, int XU>
__global__ void __launch_bounds__(256) lfc_add_bands_kernel(const int* __restrict__ pt_G, const int* __restrict__ pt_off,
                                                            const int* __restrict__ ct_M,
                                                            const int* __restrict__ ct_nm,
                                                            const float* __restrict__ Ap, int64_t P,
                                                            const float* __restrict__ c_xM, int nM,
                                                            float* __restrict__ a_xG, int64_t nG, int64_t nx) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= P) return;
  const int k0 = pt_off[p], K = pt_off[p + 1] - k0;
  float A[KREG][NMAX];
  const float* cb[KREG];
  int nmk[KREG];
#pragma unroll
  for (int k = 0; k < KREG; ++k) {
    if (k < K) {
      load_coef<NMAX, true>(Ap + (int64_t)(k0 + k) * NMAX, NMAX, A[k]);
      cb[k] = c_xM + ct_M[k0 + k];
      nmk[k] = ct_nm[k0 + k];
    } else {
#pragma unroll
      for (int m = 0; m < NMAX; ++m) A[k][m] = 0.f;
      cb[k] = c_xM;
      nmk[k] = 0;
    }
  }
  const int64_t nfull = nx / XU * XU;
  float* ax = a_xG + pt_G[p];
  for (int64_t x0 = 0; x0 < nfull; x0 += XU, ax += XU * nG)
    add_point_bands<NMAX, KREG, FULL, XU>(A, cb, nmk, K, k0, ct_M, ct_nm, Ap, c_xM, nM, x0, ax, nG);
  for (int64_t x0 = nfull; x0 < nx; ++x0, ax += nG)
    add_point_bands<NMAX, KREG, FULL, 1>(A, cb, nmk, K, k0, ct_M, ct_nm, Ap, c_xM, nM, x0, ax, nG);
}

static int add_bands(const gb_lfc* l, const float* c, float* a, int64_t nx, cudaStream_t st) {
  const bool full = l->pad_full && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
  const unsigned grid = (unsigned)((l->P + 255) / 256);
  auto kern = l->pad_nm == 8 ? (full ? lfc_add_bands_kernel<8, 4, true, 8> : lfc_add_bands_kernel<8, 4, false, 8>)
                             : (full ? lfc_add_bands_kernel<16, 2, true, 8> : lfc_add_bands_kernel<16, 2, false, 8>);
  kern<<<grid, 256, 0, st>>>(l->pt_G, l->pt_off, l->ct_M, l->ct_nm, l->A32p, l->P, c, l->nM, a, l->nG, nx);
  return check_launch("lfc_add_bands_kernel");
}

// A32p[c][m] = A of contribution c, zero for m >= nm
static __global__ void lfc_pad_rows_kernel(const double* __restrict__ A, const int64_t* __restrict__ ct_aoff,
                                           const int* __restrict__ ct_nm, int64_t C, int F, float* __restrict__ Ap) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < C * F; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = i / F;
    const int m = (int)(i - c * F);
    Ap[i] = m < ct_nm[c] ? (float)A[ct_aoff[c] + m] : 0.f;
  }
}

// ------------------------------------------------ real data, FP64 tensor cores
// For FP64 real data (Gamma point: every periodic image has phase 1) and at
// most 16 functions per volume both products run as m16n8k8 FP64 MMAs on 16
// bands x 8 grid points x 8 functions, the three operands exactly as they lie
// in memory: bands x points (a), points x functions (an entry's dense block)
// and bands x functions (c).
//   integrate: a cluster of four CTAs takes one function group and 16 bands;
//     its 32 warps split the group's entries evenly, and the 32 sums are added
//     in warp order (shared, then distributed shared memory).
//   add: a warp takes one sub-tile and 16 bands, sums its entries and adds
//     the sum to the covered points.
// The split depends on the object alone and every sum has one order, so the
// results depend neither on scheduling nor on how the bands are blocked.  (The
// add of one grid alone takes lfc_add_kernel, whose sums may differ from those
// of a block in the last bits.)
// A sub-tile holds points that a volume does not cover: integrate reads them
// as zeros and add drops what an entry gives there, so that a non-finite
// value reaches the sums it belongs to and no others.
//
// Bound by the latency of gathered operands, so by the warps in flight: one
// 16-band tile per warp.  (Up to five, one read of a block for 80 bands at up
// to 190 registers, took 1.6 times as long for the projections of 160 bands on
// 1 to 64 atoms, in the geometric mean, and 1.3 times for the add; three were
// faster only where they make the last wave, 90 against 108 us for 96 bands of
// 9 functions on 24 atoms.)  The add reads the grid points it updates before
// its sums; in the loop over the stores each load waited for the store before
// it.  Inputs from HBM, 71^3 points, radius 2.1 A, point-major kernels (gathered
// rows, one point per thread) against these:
//   24 atoms x 9 functions, 96 bands:  integrate 127 ->  80 us, add 174 ->  76 us
//   24 atoms x 5 functions, 160 bands: integrate 120 ->  78 us, add 169 ->  96 us
//    4 atoms x 9 functions, 160 bands: integrate  66 ->  40 us, add  77 ->  31 us
__device__ __forceinline__ void mma_f64(double (&d)[4], const double (&a)[4], double b0, double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

constexpr int LM_CLUSTER = 4;              // CTAs per (function group, band block)
constexpr int LM_WARPS = 8;

template <int NF>
__global__ void __cluster_dims__(LM_CLUSTER, 1, 1) __launch_bounds__(32 * LM_WARPS)
    lfc_integrate_mma_kernel(const int* __restrict__ sg_off, const int4* __restrict__ sg_e,
                             const double* __restrict__ st_A, int nr, const int* __restrict__ gr_M,
                             const int* __restrict__ gr_nm, const double* __restrict__ a_xG,
                             double* __restrict__ c_xM, int64_t nx, int64_t nG, int nM, double dv) {
  constexpr int NE = NF * 128;
  __shared__ double red[LM_WARPS * NE];        // [warp][function block][k][lane]
  const int rank = blockIdx.x % LM_CLUSTER, gi = blockIdx.x / LM_CLUSTER;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t x0 = (int64_t)blockIdx.y * 16;
  const int M = gr_M[gi], nm = gr_nm[gi];
  const int e0 = sg_off[gi], ne = sg_off[gi + 1] - e0, w = rank * LM_WARPS + warp;
  const int i0 = e0 + (int)((int64_t)ne * w / (LM_CLUSTER * LM_WARPS));
  const int i1 = e0 + (int)((int64_t)ne * (w + 1) / (LM_CLUSTER * LM_WARPS));
  const double* row[2];
  bool on[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t x = x0 + 8 * h + g;
    on[h] = x < nx;
    row[h] = a_xG + (on[h] ? x : 0) * nG + t;
  }
  double acc[NF][4];
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[f][k] = 0.0;
#pragma unroll 2
  for (int q = i0; q < i1; ++q) {
    const int4 es = __ldg(sg_e + q);
    const int64_t p = (int64_t)es.y * 8;
    const bool in0 = es.z >> t & 1, in1 = es.z >> t & 16;
    const double* blk = st_A + ((int64_t)es.x * nr + g) * 8 + t;
    double av[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      av[h] = on[h] && in0 ? __ldg(row[h] + p) : 0.0;
      av[2 + h] = on[h] && in1 ? __ldg(row[h] + p + 4) : 0.0;
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const bool in = f * 8 + g < nr;
      mma_f64(acc[f], av, in ? __ldg(blk + f * 64) : 0.0, in ? __ldg(blk + f * 64 + 4) : 0.0);
    }
  }
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int k = 0; k < 4; ++k) red[warp * NE + (f * 4 + k) * 32 + lane] = acc[f][k];
  __syncthreads();
  for (int e = threadIdx.x; e < NE; e += 32 * LM_WARPS) {
    double v = red[e];
#pragma unroll
    for (int ww = 1; ww < LM_WARPS; ++ww) v += red[ww * NE + e];
    red[e] = v;
  }
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = rank * 32 * LM_WARPS + threadIdx.x; e < NE; e += LM_CLUSTER * 32 * LM_WARPS) {
    double v = 0.0;
#pragma unroll
    for (int r = 0; r < LM_CLUSTER; ++r) v += cluster.map_shared_rank(red, r)[e];
    const int l = e & 31, k = (e >> 5) & 3, f = e >> 7;
    const int64_t x = x0 + 8 * (k >> 1) + (l >> 2);
    const int m = f * 8 + 2 * (l & 3) + (k & 1);
    if (x < nx && m < nm) {
      double* cp = c_xM + x * nM + M + m;
      *cp = fma(dv, v, *cp);
    }
  }
  cluster.sync();        // the other CTAs may still be reading this one's sums
}

template <int NF>
__global__ void __launch_bounds__(32 * LM_WARPS)
    lfc_add_mma_kernel(int ns, const int4* __restrict__ st_sub, const int2* __restrict__ st_M,
                       const double* __restrict__ st_A, int nr, const double* __restrict__ c_xM,
                       double* __restrict__ a_xG, int64_t nx, int64_t nG, int nM) {
  const int s = blockIdx.x * LM_WARPS + (threadIdx.x >> 5);
  if (s >= ns) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t x0 = (int64_t)blockIdx.y * 16 + g;
  // a sub-tile comes with its first entry, so that the loads of coefficients,
  // block and grid points are one step behind its own
  const int4 sub = __ldg(st_sub + 2 * s), first = __ldg(st_sub + 2 * s + 1);
  const bool on[2] = {x0 < nx, x0 + 8 < nx};
  const double* row[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) row[h] = c_xM + (on[h] ? x0 + 8 * h : 0) * nM + t;
  // points 2 t and 2 t + 1 of bands x0 and x0 + 8: the four loads before the
  // sums, the four stores after them
  double* const ap = a_xG + x0 * nG + (int64_t)sub.x * 8 + 2 * t;
  double old[4], acc[4];
  bool wr[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    wr[k] = on[k >> 1] && (sub.y >> (2 * t + (k & 1)) & 1);
    old[k] = wr[k] ? ap[8 * (k >> 1) * nG + (k & 1)] : 0.0;
    acc[k] = 0.0;
  }
  int2 mn = make_int2(first.x, first.y);
  for (int e = sub.z; e < sub.w; ++e) {
    const int nm = mn.y & 255;
    const bool cov[2] = {(mn.y >> (8 + 2 * t) & 1) != 0, (mn.y >> (9 + 2 * t) & 1) != 0};
    double d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const double* blk = st_A + ((int64_t)e * nr + f * 8 + t) * 8 + g;
      const bool in0 = f * 8 + t < nm, in1 = f * 8 + t + 4 < nm;
      double cv[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double* c = row[h] + mn.x + f * 8;
        cv[h] = on[h] && in0 ? __ldg(c) : 0.0;
        cv[2 + h] = on[h] && in1 ? __ldg(c + 4) : 0.0;
      }
      mma_f64(d, cv, in0 ? __ldg(blk) : 0.0, in1 ? __ldg(blk + 32) : 0.0);
    }
    if (e + 1 < sub.w) mn = __ldg(st_M + e + 1);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (cov[k & 1]) acc[k] += d[k];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (wr[k]) ap[8 * (k >> 1) * nG + (k & 1)] = old[k] + acc[k];
}

// st_A[e][m][p]: the rows of an entry are the points it covers, in order;
// ent_a is the offset of the first one in A
static __global__ void lfc_blocks_kernel(const double* __restrict__ A, const int64_t* __restrict__ ent_a,
                                         const int2* __restrict__ st_M, int64_t ne, int nr, double* __restrict__ st_A) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ne * nr * 8;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = i / (nr * 8);
    const int m = (int)(i / 8 % nr), p = (int)(i & 7);
    const int nm = st_M[e].y & 255, cov = st_M[e].y >> 8;
    st_A[i] = m < nm && (cov >> p & 1) ? A[ent_a[e] + __popc(cov & ((1 << p) - 1)) * nm + m] : 0.0;
  }
}

// the launch grid's second dimension bounds the bands
static bool mma_usable(const gb_lfc* l, int64_t nx) { return l->nf && nx <= 65535 * 16; }

static int integrate_mma(const gb_lfc* l, const double* a, double* c, int64_t nx, cudaStream_t st) {
  if (l->ngroups == 0) return GB_OK;
  const dim3 grid((unsigned)(l->ngroups * LM_CLUSTER), (unsigned)((nx + 15) / 16));
  auto kern = l->nf == 1 ? lfc_integrate_mma_kernel<1> : lfc_integrate_mma_kernel<2>;
  kern<<<grid, 32 * LM_WARPS, 0, st>>>(l->sg_off, l->sg_e, l->st_A, l->maxnm, l->gr_M, l->gr_nm, a, c, nx, l->nG, l->nM,
                                       l->dv);
  return check_launch("lfc_integrate_mma_kernel");
}

static int add_mma(const gb_lfc* l, const double* c, double* a, int64_t nx, cudaStream_t st) {
  if (l->ns == 0) return GB_OK;
  const dim3 grid((unsigned)((l->ns + LM_WARPS - 1) / LM_WARPS), (unsigned)((nx + 15) / 16));
  auto kern = l->nf == 1 ? lfc_add_mma_kernel<1> : lfc_add_mma_kernel<2>;
  kern<<<grid, 32 * LM_WARPS, 0, st>>>(l->ns, l->st_sub, l->st_M, l->st_A, l->maxnm, c, a, nx, l->nG, l->nM);
  return check_launch("lfc_add_mma_kernel");
}

template <typename T, int NM>
static int integrate_nm(const gb_lfc* l, int gbeg, int gcount, const void* a, void* c, int64_t nx, int q,
                        int64_t per_q,
                        cudaStream_t st) {
  // accumulators per thread: XB x NM (twice that for complex images)
  constexpr int XB0 = NM <= 2 ? 16 : (NM <= 4 ? 8 : (NM <= 8 ? 4 : (NM <= 16 ? 2 : 1)));
  constexpr int XB = Elem<T>::cplx ? (XB0 >= 4 ? XB0 / 4 : 1) : XB0;
  constexpr int NT = 128;
  const typename AType<T>::A* A;
  if constexpr (std::is_same<typename AType<T>::A, float>::value) A = l->A32; else A = l->A64;
  dim3 grid((unsigned)gcount, (unsigned)((nx + XB - 1) / XB));
  lfc_integrate_kernel<T, NM, XB, NT><<<grid, NT, 0, st>>>(view(l), A, (const T*)a, (T*)c, nx, q, gbeg, per_q);
  return check_launch("lfc_integrate_kernel");
}

// smallest supported padded function count >= nm
static int nm_class(int nm) {
  for (int c : {1, 2, 4, 8, 16, 32, 64})
    if (nm <= c) return c;
  return 0;
}

static bool tiles_usable(const gb_lfc* l, const void* a);
static int integrate_tiles(const gb_lfc* l, const float* a, float* c, int64_t nx, cudaStream_t st);

template <typename T>
static int integrate_t(const gb_lfc* l, const void* a, void* c, int64_t nx, int q, cudaStream_t st,
                       int64_t per_q = 0) {
  if constexpr (std::is_same<T, float>::value) {
    if (tiles_usable(l, a))
      return integrate_tiles(l, static_cast<const float*>(a), static_cast<float*>(c), nx, st);
  }
  if constexpr (std::is_same<T, double>::value) {
    if (mma_usable(l, nx)) return integrate_mma(l, static_cast<const double*>(a), static_cast<double*>(c), nx, st);
  }
  // groups are sorted by nm on the host; one launch per padded class
  int g = 0;
  while (g < l->ngroups) {
    const int cls = nm_class(l->h_gr_nm[g]);
    int e = g;
    while (e < l->ngroups && nm_class(l->h_gr_nm[e]) == cls) ++e;
    int rc;
    switch (cls) {
      case 1: rc = integrate_nm<T, 1>(l, g, e - g, a, c, nx, q, per_q, st); break;
      case 2: rc = integrate_nm<T, 2>(l, g, e - g, a, c, nx, q, per_q, st); break;
      case 4: rc = integrate_nm<T, 4>(l, g, e - g, a, c, nx, q, per_q, st); break;
      case 8: rc = integrate_nm<T, 8>(l, g, e - g, a, c, nx, q, per_q, st); break;
      case 16: rc = integrate_nm<T, 16>(l, g, e - g, a, c, nx, q, per_q, st); break;
      case 32: rc = integrate_nm<T, 32>(l, g, e - g, a, c, nx, q, per_q, st); break;
      case 64: rc = integrate_nm<T, 64>(l, g, e - g, a, c, nx, q, per_q, st); break;
      default: return fail(GB_E_UNSUPPORTED, "lfc: more than 64 functions in one volume");
    }
    if (rc) return rc;
    g = e;
  }
  return GB_OK;
}

template <typename T, int XB, int NMAX>
static int add_nm(const gb_lfc* l, const void* c, void* a, int64_t nx, int q, cudaStream_t st, int64_t per_q) {
  const typename AType<T>::A* A;
  if constexpr (std::is_same<typename AType<T>::A, float>::value) A = l->A32; else A = l->A64;
  const int NT = 256;
  const int64_t bx = std::min<int64_t>((l->P + NT - 1) / NT, (int64_t)sm_count() * 8);
  dim3 grid((unsigned)bx, (unsigned)((nx + XB - 1) / XB));
  lfc_add_kernel<T, XB, NMAX><<<grid, NT, 0, st>>>(view(l), A, (const T*)c, (T*)a, nx, q, per_q);
  return check_launch("lfc_add_kernel");
}


// ------------------------------------------------ brick-tiled FP32 (real)
// The flattened grid is cut into 32-point chunks of four 8-point sub-tiles;
// an entry is one (volume, sub-tile it touches) with the volume's values
// there as a dense [m][p] 8 x 8 block.  A brick is a run of at most TBRICK
// consecutive chunks with entries that meets at most TSLOTS function groups
// (its slots) and holds at most TBENT entries.  One CTA takes one (brick,
// group of bands: 32 for the add, 64 for the integral) and first copies into
// shared memory, with coalesced 16-byte cp.async copies, the brick's rows of
// a (a band row pitch of 32 TBRICK + 4 floats, free of bank conflicts), its
// entries' blocks and, for the add, the coefficients of its slots as
// [slot][m][band] (rows of cT, c transposed by a first kernel).  A warp works
// on 8 points x 32 bands: lane (q, b) holds points 4 q .. 4 q + 3 of bands b
// and b + 16, so that one 16-byte read of a block's row -- two addresses in
// the warp -- feeds both, and cT holds such pairs side by side.
//  add:        warp w updates sub-tiles w, w + 16, ... in place (one owner
//              per sub-tile): a[x][p] += sum_e sum_m A_e[m][p] c[x][M_e + m];
//              the brick's rows are then written back.
//  integrate:  a warp sums one slot and 32 bands over its entries (lists made
//              on the host) and writes one partial sum per (brick, slot,
//              band); a second kernel adds dv times each group's partials, in
//              brick order, to c.
// No atomics: the results do not depend on scheduling.
// Bound by shared-memory wavefronts and the wait for the copies: (160, 56^3),
// 64 atoms with 5 functions: add 133 -> 109 us, integrate 117 -> 95 us against
// lanes owning one band and all 8 points (three wavefronts per block row and
// 32 bands instead of two in the add, 18 instead of 13 per entry in the
// integral, and twice the instructions).  Adding to a directly in global
// memory, 64 bands per CTA, took 122 us: 16 rows per store instruction.  Half
// as long bricks, 8-warp CTAs: add 118, integrate 102 us.
constexpr int TCH = 32;                    // points per chunk
constexpr int TSLOTS = 16;                 // function groups per brick
constexpr int TBRICK = 8;                  // chunks per brick
constexpr int TBENT = 176;                 // entries per brick (two integrate CTAs per SM)
constexpr int TADD_BAND = 32;              // bands per CTA, add
constexpr int TINT_BAND = 64;              // and integrate
constexpr int TPITCH = TBRICK * TCH + 4;   // floats per band row in shared memory
constexpr int TILE_WARPS = 16;

struct TileView {
  const int* ch_c;      // [nch] chunk index (first point 32 c) of every used chunk
  const int* ch_eoff;   // [4 nch + 1] entries of (chunk, sub-tile)
  const int* e_info;    // [ne] slot | nm << 8
  const float* e_A;     // [ne][8][8]
  const int* br_ch0;    // [nbr + 1] chunk range of each brick
  const int* br_pbase;  // [nbr + 1] first (brick, slot) pair of each brick
  const int* ps_M;      // [npart] group of each (brick, slot): its first function
  const int* ps_nm;     // [npart] and function count
  const int* ps_eoff;   // [npart + 1] entries of each (brick, slot):
  const int* ps_info;   //   (entry - first entry of the brick) | sub-tile << 16 | nm << 24
};

static TileView tile_view(const gb_lfc* l) {
  return TileView{l->tch_c, l->tch_eoff, l->te_info, l->te_A, l->tbr_ch0, l->tbr_pbase,
                  l->tps_M, l->tps_nm, l->tps_eoff, l->tps_info};
}

// the blocks of entries E0 .. E1 - 1
__device__ __forceinline__ void stage_blocks(const TileView& t, int E0, int E1, float* sA) {
  for (int i = threadIdx.x; i < (E1 - E0) * 16; i += blockDim.x) cp_async16(sA + 4 * i, t.e_A + (int64_t)E0 * 64 + 4 * i);
}

__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// f(integral_constant<int, nm>) for 1 <= nm <= 8, uniform in a warp
template <class F>
__device__ __forceinline__ void for_functions(int nm, F&& f) {
  switch (nm) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
  }
}

// cT[M][x0 + 2 b + i] = c[x0 + b + 16 i][M]
__global__ void lfc_coef_transpose_kernel(const float* __restrict__ c, int nM, int R, int ldT, float* __restrict__ cT) {
  __shared__ float tile[32][33];
  const int M0 = blockIdx.x * 32, x0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int x = x0 + i, M = M0 + threadIdx.x;
    tile[i][threadIdx.x] = (x < R && M < nM) ? c[(int64_t)x * nM + M] : 0.f;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int M = M0 + i;
    if (M < nM) cT[(int64_t)M * ldT + x0 + threadIdx.x] = tile[16 * (threadIdx.x & 1) + (threadIdx.x >> 1)][i];
  }
}

// rows x0 .. x0 + nb - 1 of a brick's chunks
__device__ __forceinline__ void stage_rows(const TileView& t, int k0, int nk, const float* __restrict__ a, int64_t nG,
                                           int x0, int nb, float* sa) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int x = warp; x < nb; x += TILE_WARPS) {
    const float* src = a + (int64_t)(x0 + x) * nG;
    for (int i = lane; i < nk * 8; i += 32) {
      const int64_t G = (int64_t)t.ch_c[k0 + (i >> 3)] * TCH + 4 * (i & 7);
      float* d = sa + x * TPITCH + 4 * i;
      if (G < nG) cp_async16(d, src + G);
      else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// acc (points 2 k, 2 k + 1 of band i in acc[i][k]) += nm rows of a block
template <int NM>
__device__ __forceinline__ void add_entry(float2 (&acc)[2][2], const float4* __restrict__ Ab,
                                          const float* __restrict__ cs) {
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    const float4 A = Ab[2 * m];
    const float2 c = *reinterpret_cast<const float2*>(cs + m * TADD_BAND);
    const float2 c0 = make_float2(c.x, c.x), c1 = make_float2(c.y, c.y);
    acc[0][0] = __ffma2_rn(lo2(A), c0, acc[0][0]);
    acc[0][1] = __ffma2_rn(hi2(A), c0, acc[0][1]);
    acc[1][0] = __ffma2_rn(lo2(A), c1, acc[1][0]);
    acc[1][1] = __ffma2_rn(hi2(A), c1, acc[1][1]);
  }
}

// the sub-tiles of a brick; NM: functions of every entry, 0: each entry's own
template <int NM>
__device__ __forceinline__ void add_sub_tiles(const TileView& t, int k0, int nk, const float* sA, const float* sc,
                                              float* sa) {
  const int warp = threadIdx.x >> 5, q = (threadIdx.x >> 4) & 1, b = threadIdx.x & 15;
  const int E0 = t.ch_eoff[4 * k0];
  for (int st = warp; st < 4 * nk; st += TILE_WARPS) {
    const int e0 = t.ch_eoff[4 * k0 + st], e1 = t.ch_eoff[4 * k0 + st + 1];
    if (e0 == e1) continue;
    float4* row = reinterpret_cast<float4*>(sa + b * TPITCH + 8 * st + 4 * q);
    float2 acc[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 u = row[4 * TPITCH * i];
      acc[i][0] = lo2(u);
      acc[i][1] = hi2(u);
    }
    int info = t.e_info[e0];
    for (int e = e0; e < e1; ++e) {
      const float4* Ab = reinterpret_cast<const float4*>(sA + (e - E0) * 64) + q;
      const float* cs = sc + (info & 255) * 8 * TADD_BAND + 2 * b;
      const int nm = info >> 8;
      if (e + 1 < e1) info = t.e_info[e + 1];
      if constexpr (NM > 0) add_entry<NM>(acc, Ab, cs);
      else for_functions(nm, [&](auto n) { add_entry<n.value>(acc, Ab, cs); });
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) row[4 * TPITCH * i] = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
  }
}

__global__ void __launch_bounds__(32 * TILE_WARPS, 2) lfc_add_tiles_kernel(const TileView t,
                                                                         const float* __restrict__ cT, int ldT,
                                                                         float* __restrict__ a, int64_t nG, int R,
                                                                         int sA_floats, int nm_all) {
  extern __shared__ __align__(16) float tsm[];
  float* sa = tsm;
  float* sA = sa + TADD_BAND * TPITCH;
  float* sc = sA + sA_floats;
  const int b = blockIdx.x, x0 = blockIdx.y * TADD_BAND;
  const int nb = min(TADD_BAND, R - x0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k0 = t.br_ch0[b], nk = t.br_ch0[b + 1] - k0;
  stage_rows(t, k0, nk, a, nG, x0, nb, sa);
  stage_blocks(t, t.ch_eoff[4 * k0], t.ch_eoff[4 * (k0 + nk)], sA);
  const int pbase = t.br_pbase[b], S = t.br_pbase[b + 1] - pbase;
  for (int r = 4 * warp + (lane >> 3); r < S * 8; r += 4 * TILE_WARPS) {
    const int s = r >> 3, m = r & 7, x = 4 * (lane & 7);
    if (m < t.ps_nm[pbase + s])
      cp_async16(sc + r * TADD_BAND + x, cT + (int64_t)(t.ps_M[pbase + s] + m) * ldT + x0 + x);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (nm_all) for_functions(nm_all, [&](auto n) { add_sub_tiles<n.value>(t, k0, nk, sA, sc, sa); });
  else add_sub_tiles<0>(t, k0, nk, sA, sc, sa);
  __syncthreads();
  for (int x = warp; x < nb; x += TILE_WARPS) {
    float* dst = a + (int64_t)(x0 + x) * nG;
    for (int i = lane; i < nk * 8; i += 32) {
      const int64_t G = (int64_t)t.ch_c[k0 + (i >> 3)] * TCH + 4 * (i & 7);
      if (G < nG) *reinterpret_cast<float4*>(dst + G) = *reinterpret_cast<const float4*>(sa + x * TPITCH + 4 * i);
    }
  }
}

// acc[i][m] (even / odd point sums of band i) over entries q0 .. q1 - 1 of a
// slot of NM functions
template <int NM>
__device__ __forceinline__ void integrate_entries(float2 (&acc)[2][8], const int* __restrict__ ps_info, int q0, int q1,
                                                  const float* __restrict__ row, const float* __restrict__ sA) {
  constexpr int U = NM <= 6 ? 2 : 1;       // entries in flight, within 64 registers
#pragma unroll U
  for (int e = q0; e < q1; ++e) {
    const int info = __ldg(ps_info + e);
    const float* r = row + 8 * ((info >> 16) & 255);
    const float4 u = *reinterpret_cast<const float4*>(r), v = *reinterpret_cast<const float4*>(r + 16 * TPITCH);
    const float4* Ab = reinterpret_cast<const float4*>(sA + (info & 0xffff) * 64);
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const float4 A = Ab[2 * m];
      acc[0][m] = __ffma2_rn(hi2(A), hi2(u), __ffma2_rn(lo2(A), lo2(u), acc[0][m]));
      acc[1][m] = __ffma2_rn(hi2(A), hi2(v), __ffma2_rn(lo2(A), lo2(v), acc[1][m]));
    }
  }
}

__global__ void __launch_bounds__(32 * TILE_WARPS, 2) lfc_integrate_tiles_kernel(const TileView t,
                                                                               const float* __restrict__ a,
                                                                               int64_t nG, int R,
                                                                               float* __restrict__ part) {
  extern __shared__ __align__(16) float tsm[];
  float* sa = tsm;
  float* sA = sa + TINT_BAND * TPITCH;
  const int br = blockIdx.x, x0 = blockIdx.y * TINT_BAND;
  const int nb = min(TINT_BAND, R - x0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 4, b = lane & 15;
  const int k0 = t.br_ch0[br], nk = t.br_ch0[br + 1] - k0;
  stage_rows(t, k0, nk, a, nG, x0, nb, sa);
  stage_blocks(t, t.ch_eoff[4 * k0], t.ch_eoff[4 * (k0 + nk)], sA);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int pbase = t.br_pbase[br], S = t.br_pbase[br + 1] - pbase, H = nb > 32 ? 2 : 1;
  for (int it = warp; it < S * H; it += TILE_WARPS) {
    const int s = it / H, xb = (it - s * H) * 32 + b;      // bands xb and xb + 16 of the group
    float2 acc[2][8];
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[0][m] = acc[1][m] = make_float2(0.f, 0.f);
    const int q0 = t.ps_eoff[pbase + s], q1 = t.ps_eoff[pbase + s + 1];
    for_functions(t.ps_nm[pbase + s], [&](auto n) {
      integrate_entries<n.value>(acc, t.ps_info, q0, q1, sa + xb * TPITCH + 4 * q, sA + 4 * q);
    });
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float r[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        r[m] = acc[i][m].x + acc[i][m].y;
        r[m] += __shfl_xor_sync(0xffffffffu, r[m], 16);
      }
      // lane half q writes functions 4 q .. 4 q + 3
      if (xb + 16 * i < nb)
        reinterpret_cast<float4*>(part + ((int64_t)(pbase + s) * R + x0 + xb + 16 * i) * 8)[q] =
            q ? make_float4(r[4], r[5], r[6], r[7]) : make_float4(r[0], r[1], r[2], r[3]);
    }
  }
}

// c[x][M_g + m] += dv sum of group g's partials.  A CTA takes 32 outputs
// (x, m) of one group -- four bands -- and eight slices of its partial list:
// thread (slice s, output o) sums partials s, s + 8, ... (32 consecutive
// floats per partial: coalesced), then the eight sums are added in slice
// order.  Fixed order throughout: results do not depend on scheduling.
__global__ void __launch_bounds__(256) lfc_tiles_reduce_kernel(const int* __restrict__ gr_M,
                                                              const int* __restrict__ gr_nm,
                                                              const int* __restrict__ poff,
                                                              const int* __restrict__ pidx,
                                                              const float* __restrict__ part, int R,
                                                              float* __restrict__ c, int nM, float dv) {
  __shared__ float red[8][33];
  const int g = blockIdx.y;
  const int o = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + o;              // output (x, m) = (i / 8, i % 8)
  float s = 0.f;
  if (i < R * 8) {
    const float* pp = part + i;
    const int64_t ps = (int64_t)R * 8;
    const int q1 = poff[g + 1];
    for (int q = poff[g] + sl; q < q1; q += 8) s += pp[pidx[q] * ps];
  }
  red[sl][o] = s;
  __syncthreads();
  if (sl == 0 && i < R * 8) {
    const int x = i >> 3, m = i & 7;
    if (m < gr_nm[g]) {
      float t = red[0][o];
#pragma unroll
      for (int k = 1; k < 8; ++k) t += red[k][o];
      float* cp = c + (int64_t)x * nM + gr_M[g] + m;
      *cp = fmaf(dv, t, *cp);
    }
  }
}

// grow the work space (never inside stream capture)
static int tile_work(const gb_lfc* l, size_t bytes, cudaStream_t st) {
  if (bytes <= l->work_bytes) return GB_OK;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
    return fail(GB_E_INVALID, "lfc: the tiled FP32 path needs a larger work space; make one call of this size "
                              "before capturing it in a graph");
  if (l->work) {
    if (cudaStreamSynchronize(st) != cudaSuccess) return check_launch("lfc work space");
    cudaFree(l->work);
    l->work = nullptr;
    l->work_bytes = 0;
  }
  if (cudaMalloc(&l->work, bytes) != cudaSuccess) {
    l->work = nullptr;
    return fail(GB_E_NOMEM, "lfc: work space allocation failed");
  }
  l->work_bytes = bytes;
  return GB_OK;
}

static int tile_smem_attr() {
  static int done = 0;
  if (!done) {
    const int mxa = (TADD_BAND * TPITCH + TBENT * 64 + TSLOTS * 8 * TADD_BAND) * (int)sizeof(float);
    const int mxi = (TINT_BAND * TPITCH + TBENT * 64) * (int)sizeof(float);
    if (cudaFuncSetAttribute(lfc_add_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mxa) != cudaSuccess ||
        cudaFuncSetAttribute(lfc_integrate_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mxi) !=
            cudaSuccess)
      return check_launch("lfc tiled shared memory");
    done = 1;
  }
  return GB_OK;
}

// usable for this call: FP32 real data, rows 16-byte aligned
static bool tiles_usable(const gb_lfc* l, const void* a) {
  return l->tiled && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
}

// passes of at most 256 bands bound the work space
static int add_tiles(const gb_lfc* l, const float* c, float* a, int64_t nx, cudaStream_t st) {
  if (l->tbr_n == 0) return GB_OK;
  int rc = tile_smem_attr();
  if (rc) return rc;
  const int Rmax = (int)std::min<int64_t>(nx, 256);
  rc = tile_work(l, (size_t)l->nM * ((Rmax + 31) / 32 * 32) * sizeof(float), st);
  if (rc) return rc;
  float* cT = static_cast<float*>(l->work);
  const int sA_floats = l->tbr_emax * 64;
  const int smem = (TADD_BAND * TPITCH + sA_floats + l->tbr_smax * 8 * TADD_BAND) * (int)sizeof(float);
  for (int64_t x0 = 0; x0 < nx; x0 += 256) {
    const int R = (int)std::min<int64_t>(nx - x0, 256);
    const int ldT = (R + 31) / 32 * 32;
    dim3 tg((unsigned)((l->nM + 31) / 32), (unsigned)(ldT / 32));
    lfc_coef_transpose_kernel<<<tg, dim3(32, 8), 0, st>>>(c + x0 * l->nM, l->nM, R, ldT, cT);
    dim3 grid((unsigned)l->tbr_n, (unsigned)(ldT / TADD_BAND));
    lfc_add_tiles_kernel<<<grid, 32 * TILE_WARPS, smem, st>>>(tile_view(l), cT, ldT, a + x0 * l->nG, l->nG, R,
                                                              sA_floats, l->tnm);
    rc = check_launch("lfc_add_tiles_kernel");
    if (rc) return rc;
  }
  return GB_OK;
}

static int integrate_tiles(const gb_lfc* l, const float* a, float* c, int64_t nx, cudaStream_t st) {
  if (l->tbr_n == 0) return GB_OK;
  int rc = tile_smem_attr();
  if (rc) return rc;
  const int Rmax = (int)std::min<int64_t>(nx, 256);
  rc = tile_work(l, (size_t)l->tpart_n * Rmax * 8 * sizeof(float), st);
  if (rc) return rc;
  float* part = static_cast<float*>(l->work);
  const int smem = (TINT_BAND * TPITCH + l->tbr_emax * 64) * (int)sizeof(float);
  for (int64_t x0 = 0; x0 < nx; x0 += 256) {
    const int R = (int)std::min<int64_t>(nx - x0, 256);
    dim3 grid((unsigned)l->tbr_n, (unsigned)((R + TINT_BAND - 1) / TINT_BAND));
    lfc_integrate_tiles_kernel<<<grid, 32 * TILE_WARPS, smem, st>>>(tile_view(l), a + x0 * l->nG, l->nG, R, part);
    rc = check_launch("lfc_integrate_tiles_kernel");
    if (rc) return rc;
    dim3 rg((unsigned)((R * 8 + 31) / 32), (unsigned)l->ngroups);
    lfc_tiles_reduce_kernel<<<rg, 256, 0, st>>>(l->gr_M, l->gr_nm, l->tgr_poff, l->tgr_pidx, part, R,
                                                c + x0 * l->nM, l->nM, (float)l->dv);
    rc = check_launch("lfc_tiles_reduce_kernel");
    if (rc) return rc;
  }
  return GB_OK;
}


template <typename T>
static int add_t(const gb_lfc* l, const void* c, void* a, int64_t nx, int q, cudaStream_t st,
                 int64_t per_q = 0) {
  if (l->P == 0) return GB_OK;
  if constexpr (std::is_same<T, float>::value) {
    if (tiles_usable(l, a)) return add_tiles(l, static_cast<const float*>(c), static_cast<float*>(a), nx, st);
    if (l->A32p) return add_bands(l, static_cast<const float*>(c), static_cast<float*>(a), nx, st);
  }
  if constexpr (std::is_same<T, double>::value) {
    // one grid (a density or potential) would fill one row of sixteen of every
    // tile: 71^3, 24 atoms with 5 functions: 8.9 us, point by point 6.6
    if (nx > 1 && mma_usable(l, nx)) return add_mma(l, static_cast<const double*>(c), static_cast<double*>(a), nx, st);
  }
  constexpr int XB = std::is_same<T, double>::value ? 1 : 8;      // bands per thread
  switch (nm_class(l->maxnm)) {
    case 1: return add_nm<T, XB, 1>(l, c, a, nx, q, st, per_q);
    case 2: return add_nm<T, XB, 2>(l, c, a, nx, q, st, per_q);
    case 4: return add_nm<T, XB, 4>(l, c, a, nx, q, st, per_q);
    case 8: return add_nm<T, XB, 8>(l, c, a, nx, q, st, per_q);
    case 16: return add_nm<T, XB == 1 ? 1 : 4, 16>(l, c, a, nx, q, st, per_q);
    case 32: return add_nm<T, 2, 32>(l, c, a, nx, q, st, per_q);
    case 64: return add_nm<T, 1, 64>(l, c, a, nx, q, st, per_q);
    default: return fail(GB_E_UNSUPPORTED, "lfc: more than 64 functions in one volume");
  }
}

static __global__ void to_float(const double* a, float* b, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

}  // namespace gb

namespace gb {
SplineDev spline_view(const gb_spline* s);

struct SplineM {          // the radial function of one M and its m index
  SplineDev s;
  int m;
};

// one CTA per (function group, band); up to 16 functions per volume
template <typename T>
__global__ void __launch_bounds__(128) lfc_derivative_kernel(const LfcView l, const SplineM* __restrict__ spl,
                                                             const double* __restrict__ pos_W, DerivGeom geo,
                                                             const T* __restrict__ a_xG, T* __restrict__ c_xMv,
                                                             int q) {
  constexpr bool CPLX = Elem<T>::cplx;
  using Acc = typename std::conditional<CPLX, double2, double>::type;
  constexpr int NT = 128, NMV = 48;
  __shared__ Acc red[NT / 32][NMV];
  const int g = blockIdx.x;
  const int64_t x = blockIdx.y;
  const int M0 = l.gr_M[g];
  const int nm = l.gr_nm[g];
  Acc acc[NMV];
#pragma unroll
  for (int i = 0; i < NMV; ++i) acc[i] = zero<Acc>();
  for (int vi = l.gr_voff[g]; vi < l.gr_voff[g + 1]; ++vi) {
    const int W = l.gv_W[vi];
    double pr = 1.0, pi = 0.0;
    if (CPLX && q >= 0) {
      const double2 ph = l.phase[(int64_t)q * l.nW + W];
      pr = ph.x;
      pi = ph.y;
    }
    const double px = pos_W[3 * W], py = pos_W[3 * W + 1], pz = pos_W[3 * W + 2];
    for (int64_t r = l.vol_row0[W] + threadIdx.x; r < l.vol_row1[W]; r += NT) {
      const int64_t G = l.row_G[r];
      const int64_t i2 = G % geo.n[2] + geo.beg[2];
      const int64_t i1 = (G / geo.n[2]) % geo.n[1] + geo.beg[1];
      const int64_t i0 = G / (geo.n[2] * geo.n[1]) + geo.beg[0];
      const double X = geo.h[0] * i0 + geo.h[3] * i1 + geo.h[6] * i2 - px;
      const double Y = geo.h[1] * i0 + geo.h[4] * i1 + geo.h[7] * i2 - py;
      const double Z = geo.h[2] * i0 + geo.h[5] * i1 + geo.h[8] * i2 - pz;
      const double r2 = X * X + Y * Y + Z * Z;
      const double rr = sqrt(r2);
      Acc av;
      if constexpr (CPLX) {
        const T v = a_xG[x * l.nG + G];
        av = make_double2((double)v.x * pr - (double)v.y * pi, (double)v.x * pi + (double)v.y * pr);
      } else {
        av = (double)a_xG[x * l.nG + G];
      }
      // per function: f, df/dr once, then every m
      const double* coef_prev = nullptr;
      double f = 0.0, df = 0.0;
      double Yl[5], dY[15];
      for (int k = 0; k < nm && k < 16; ++k) {
        const SplineM sm = spl[M0 + k];
        if (sm.s.coef != coef_prev || sm.m == 0) {
          spline_eval(sm.s, rr, f, df);
          const double fr = rr > 1e-15 ? df / rr : 0.0;
          solid_harmonics(sm.s.l, fr, X, Y, Z, r2, Yl);        // (df/dr / r) r^l Y_lm
          solid_harmonics_gradient(sm.s.l, f, X, Y, Z, dY);    // f d(r^l Y_lm)/dr_v
          coef_prev = sm.s.coef;
        }
        const double d0 = dY[3 * sm.m] + Yl[sm.m] * X;
        const double d1 = dY[3 * sm.m + 1] + Yl[sm.m] * Y;
        const double d2 = dY[3 * sm.m + 2] + Yl[sm.m] * Z;
#pragma unroll
        for (int kk = 0; kk < 16; ++kk)
          if (kk == k) {
            if constexpr (CPLX) {
              acc[3 * kk] = make_double2(acc[3 * kk].x + av.x * d0, acc[3 * kk].y + av.y * d0);
              acc[3 * kk + 1] = make_double2(acc[3 * kk + 1].x + av.x * d1, acc[3 * kk + 1].y + av.y * d1);
              acc[3 * kk + 2] = make_double2(acc[3 * kk + 2].x + av.x * d2, acc[3 * kk + 2].y + av.y * d2);
            } else {
              acc[3 * kk] += av * d0;
              acc[3 * kk + 1] += av * d1;
              acc[3 * kk + 2] += av * d2;
            }
          }
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NMV; ++i) {
    Acc v = acc[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      if constexpr (CPLX) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
      } else {
        v += __shfl_down_sync(0xffffffffu, v, o);
      }
    }
    if (lane == 0) red[warp][i] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 3 * nm && e < NMV; e += NT) {
    Acc v = zero<Acc>();
    for (int w = 0; w < NT / 32; ++w) v = add(v, red[w][e]);
    T* cp = c_xMv + (x * l.nM + M0) * 3 + e;
    if constexpr (CPLX) {
      cp->x += (typename Elem<T>::R)(v.x * l.dv);
      cp->y += (typename Elem<T>::R)(v.y * l.dv);
    } else {
      *cp += (T)(v * l.dv);
    }
  }
}

template <typename T>
static int derivative_t(const gb_lfc* l, const SplineM* spl, const double* pos, const DerivGeom& geo,
                        const void* a, void* c, int64_t nx, int q, cudaStream_t st) {
  if (l->ngroups == 0) return GB_OK;
  const dim3 grid((unsigned)l->ngroups, (unsigned)nx);
  lfc_derivative_kernel<T><<<grid, 128, 0, st>>>(view(l), spl, pos, geo, static_cast<const T*>(a),
                                                 static_cast<T*>(c), q);
  return check_launch("lfc_derivative_kernel");
}

}  // namespace gb

using namespace gb;

extern "C" {

int gb_lfc_free(gb_lfc* l) {
  if (!l) return GB_OK;
  if (l->work) cudaFree(l->work);
  for (void* p : l->allocations) cudaFree(p);
  delete l;
  return GB_OK;
}

int gb_lfc_new(int nW, const double* A_all, const int64_t* ngm_W, const int* nm_W, const int* M_W, int nB,
               const int* G_B, const int* W_B, double dv, int nq, const double* phase_qW, int64_t nG, int nM,
               gb_lfc** out) {
  GB_REQUIRE(out && nW >= 0 && nB >= 0 && nG > 0 && nM >= 0, "gb_lfc_new: bad arguments");
  GB_REQUIRE(nW == 0 || (A_all && ngm_W && nm_W && M_W && G_B && W_B), "gb_lfc_new: null pointer");
  GB_REQUIRE(nq == 0 || phase_qW, "gb_lfc_new: phases missing");
  GB_REQUIRE(nG < (int64_t)1 << 31, "gb_lfc_new: grid too large for 32-bit point indices");
  auto* l = new (std::nothrow) gb_lfc();
  if (!l) return fail(GB_E_NOMEM, "gb_lfc_new: out of host memory");
  l->nW = nW; l->nG = nG; l->nM = nM; l->dv = dv; l->nq = nq;
  // global row / A offsets per volume
  std::vector<int64_t> row0(nW + 1, 0), aoff(nW + 1, 0);
  for (int W = 0; W < nW; ++W) {
    if (nm_W[W] < 1 || ngm_W[W] < 0 || M_W[W] < 0 || M_W[W] + nm_W[W] > nM) {
      gb_lfc_free(l);
      return fail(GB_E_INVALID, "gb_lfc_new: bad volume description");
    }
    row0[W + 1] = row0[W] + ngm_W[W];
    aoff[W + 1] = aoff[W] + ngm_W[W] * nm_W[W];
    l->maxnm = std::max(l->maxnm, nm_W[W]);
  }
  // GRID_LOOP sweep (c/lfc.h:79-130): the rows of a volume are consumed in
  // increasing G over the runs in which it is current.
  std::vector<int> row_G(row0[nW]);
  std::vector<int64_t> next_row(row0.begin(), row0.end() - 1);
  std::vector<int> cur;                 // current volumes
  std::vector<int> pos_in_cur(nW, -1);
  std::vector<int> pt_G, pt_off(1, 0);
  std::vector<int64_t> ct_aoff;
  std::vector<int> ct_M, ct_nm, ct_W;
  int Ga = 0;
  for (int B = 0; B < nB; ++B) {
    const int Gb = G_B[B];
    if (Gb < Ga || Gb > nG) {
      gb_lfc_free(l);
      return fail(GB_E_INVALID, "gb_lfc_new: boundary list not sorted or out of range");
    }
    if (Gb > Ga && !cur.empty()) {
      for (int G = Ga; G < Gb; ++G) {
        pt_G.push_back(G);
        for (int W : cur) {
          const int64_t r = next_row[W]++;
          if (r >= row0[W + 1]) {
            gb_lfc_free(l);
            return fail(GB_E_INVALID, "gb_lfc_new: boundaries cover more points than a volume has rows");
          }
          row_G[r] = G;
          ct_aoff.push_back(aoff[W] + (r - row0[W]) * nm_W[W]);
          ct_M.push_back(M_W[W]);
          ct_nm.push_back(nm_W[W]);
          ct_W.push_back(W);
        }
        pt_off.push_back((int)ct_W.size());
      }
    }
    const int Wn = W_B[B];
    if (Wn >= 0) {
      if (Wn >= nW || pos_in_cur[Wn] >= 0) {
        gb_lfc_free(l);
        return fail(GB_E_INVALID, "gb_lfc_new: bad volume entry");
      }
      pos_in_cur[Wn] = (int)cur.size();
      cur.push_back(Wn);
    } else {
      const int Wo = -1 - Wn;
      if (Wo >= nW || pos_in_cur[Wo] < 0) {
        gb_lfc_free(l);
        return fail(GB_E_INVALID, "gb_lfc_new: volume leaves before entering");
      }
      const int i = pos_in_cur[Wo];
      cur[i] = cur.back();
      pos_in_cur[cur[i]] = i;
      cur.pop_back();
      pos_in_cur[Wo] = -1;
    }
    Ga = Gb;
  }
  for (int W = 0; W < nW; ++W)
    if (next_row[W] != row0[W + 1]) {
      gb_lfc_free(l);
      return fail(GB_E_INVALID, "gb_lfc_new: volume rows and boundary runs disagree");
    }
  // function groups: volumes sharing (M, nm), ordered by nm for per-class launches
  std::map<std::pair<int, int>, std::vector<int>> groups;   // (nm, M) -> volumes
  for (int W = 0; W < nW; ++W) groups[{nm_W[W], M_W[W]}].push_back(W);
  std::vector<int> gr_M, gr_nm, gr_voff(1, 0), gv_W;
  for (auto& kv : groups) {
    gr_nm.push_back(kv.first.first);
    gr_M.push_back(kv.first.second);
    for (int W : kv.second) gv_W.push_back(W);
    gr_voff.push_back((int)gv_W.size());
  }
  // entries of the tensor-core path, in the order of their sub-tiles: a volume
  // meets its sub-tiles in order, so that placing the volumes one after the
  // other by counted sub-tiles sorts the entries by (sub-tile, volume)
  std::vector<int2> st_M;
  std::vector<int4> st_sub, sg_e;
  std::vector<int> sg_off;
  std::vector<int64_t> ent_a;
  if (l->maxnm <= 16 && nW > 0) {
    l->nf = l->maxnm <= 8 ? 1 : 2;
    const int ngr = (int)gr_M.size();
    std::vector<int> at((size_t)(nG + 7) / 8 + 1, 0), ent_sub, ent_W;
    for (int W = 0; W < nW; ++W)
      for (int64_t r = row0[W]; r < row0[W + 1]; ++r)
        if (r == row0[W] || row_G[r] / 8 != row_G[r - 1] / 8) ++at[row_G[r] / 8 + 1];
    for (size_t i = 1; i < at.size(); ++i) at[i] += at[i - 1];
    const int ne = at.back();
    st_M.resize(ne);
    ent_a.resize(ne);
    ent_sub.resize(ne);
    ent_W.resize(ne);
    for (int W = 0; W < nW; ++W)
      for (int64_t r = row0[W]; r < row0[W + 1];) {
        const int sub = row_G[r] / 8, e = at[sub]++;
        ent_sub[e] = sub;
        ent_W[e] = W;
        ent_a[e] = aoff[W] + (r - row0[W]) * nm_W[W];
        int cov = 0;
        for (; r < row0[W + 1] && row_G[r] / 8 == sub; ++r) cov |= 1 << row_G[r] % 8;
        st_M[e] = make_int2(M_W[W], nm_W[W] | cov << 8);
      }
    std::vector<int> vol_group(nW), gat(ngr + 1, 0);
    for (int gi = 0; gi < ngr; ++gi)
      for (int v = gr_voff[gi]; v < gr_voff[gi + 1]; ++v) vol_group[gv_W[v]] = gi;
    for (int e = 0; e < ne; ++e) ++gat[vol_group[ent_W[e]] + 1];
    for (int gi = 0; gi < ngr; ++gi) gat[gi + 1] += gat[gi];
    sg_off = gat;
    sg_e.resize(ne);
    for (int e = 0; e < ne; ++e) {
      const int cov = st_M[e].y >> 8;
      if (e == 0 || ent_sub[e] != ent_sub[e - 1]) {
        st_sub.push_back(make_int4(ent_sub[e], 0, e, 0));
        st_sub.push_back(make_int4(st_M[e].x, st_M[e].y, 0, 0));
      }
      int4& sub = st_sub[st_sub.size() - 2];
      sub.y |= cov;
      sub.w = e + 1;
      sg_e[gat[vol_group[ent_W[e]]]++] = make_int4(e, ent_sub[e], cov, 0);
    }
    l->ns = (int)st_sub.size() / 2;
  }
  // brick tiling for the FP32 real path
  std::vector<int> tch_c, tch_eoff, te_nm, te_slot, te_lst, te_info, tbr_ch0, tbr_pbase, tps_M, tps_nm, tps_eoff,
      tps_info, tgr_poff, tgr_pidx;
  std::vector<float> te_A;
  int tbr_smax = 1, tbr_emax = 0;
  bool tiled = l->maxnm <= 8 && nG % 4 == 0 && nW > 0;
  if (tiled) {
    const int ngr = (int)gr_M.size();
    std::vector<int> vol_group(nW);
    for (int gi = 0; gi < ngr; ++gi)
      for (int v = gr_voff[gi]; v < gr_voff[gi + 1]; ++v) vol_group[gv_W[v]] = gi;
    // entries: (sub-tile, volume) with their blocks
    struct Ent { int64_t st; int W; int64_t blk; };
    std::vector<Ent> ents;
    std::vector<float> blocks;
    for (int W = 0; W < nW; ++W) {
      int64_t last = -1;
      for (int64_t r = row0[W]; r < row0[W + 1]; ++r) {
        const int64_t G = row_G[r];
        if (G / 8 != last) {
          last = G / 8;
          ents.push_back({last, W, (int64_t)(blocks.size() / 64)});
          blocks.resize(blocks.size() + 64, 0.f);
        }
        float* b = blocks.data() + ents.back().blk * 64;
        for (int m = 0; m < nm_W[W]; ++m)
          b[m * 8 + (int)(G % 8)] = (float)A_all[aoff[W] + (r - row0[W]) * nm_W[W] + m];
      }
    }
    std::sort(ents.begin(), ents.end(),
              [](const Ent& x, const Ent& y) { return x.st != y.st ? x.st < y.st : x.W < y.W; });
    std::vector<int> te_g;   // group of every entry
    tch_eoff.push_back(0);
    for (size_t i = 0; i < ents.size();) {
      const int64_t ch = ents[i].st / 4;
      tch_c.push_back((int)ch);
      for (int j = 0; j < 4; ++j) {
        for (; i < ents.size() && ents[i].st == ch * 4 + j; ++i) {
          te_nm.push_back(nm_W[ents[i].W]);
          te_g.push_back(vol_group[ents[i].W]);
          te_A.insert(te_A.end(), blocks.begin() + ents[i].blk * 64, blocks.begin() + ents[i].blk * 64 + 64);
        }
        tch_eoff.push_back((int)te_nm.size());
      }
    }
    const size_t ne = te_nm.size();
    te_slot.assign(ne, 0);
    te_lst.assign(ne, 0);
    // bricks: <= TBRICK consecutive chunks, <= TSLOTS groups, <= TBENT entries
    std::vector<int> slot_of(ngr, -1), brick_groups, newg;
    std::vector<std::vector<int>> group_parts(ngr);
    tbr_ch0.push_back(0);
    tbr_pbase.push_back(0);
    tps_eoff.push_back(0);
    auto close_brick = [&](int end_chunk) {
      const int b0 = tbr_ch0.back();
      const int E0 = tch_eoff[4 * b0], E1 = tch_eoff[4 * end_chunk];
      for (size_t k = 0; k < brick_groups.size(); ++k) {
        const int g = brick_groups[k];
        group_parts[g].push_back(tbr_pbase.back() + (int)k);
        tps_M.push_back(gr_M[g]);
        tps_nm.push_back(gr_nm[g]);
        for (int e = E0; e < E1; ++e)
          if (te_slot[e] == (int)k) tps_info.push_back((e - E0) | te_lst[e] << 16 | te_nm[e] << 24);
        tps_eoff.push_back((int)tps_info.size());
        slot_of[g] = -1;
      }
      tbr_smax = std::max(tbr_smax, (int)brick_groups.size());
      tbr_emax = std::max(tbr_emax, E1 - E0);
      tbr_pbase.push_back(tbr_pbase.back() + (int)brick_groups.size());
      tbr_ch0.push_back(end_chunk);
      brick_groups.clear();
    };
    auto chunk_groups = [&](size_t ci, bool only_new) {
      newg.clear();
      for (int e = tch_eoff[4 * ci]; e < tch_eoff[4 * ci + 4]; ++e) {
        const int g = te_g[e];
        if ((!only_new || slot_of[g] < 0) && std::find(newg.begin(), newg.end(), g) == newg.end()) newg.push_back(g);
      }
    };
    for (size_t ci = 0; ci < tch_c.size(); ++ci) {
      const int nent = tch_eoff[4 * ci + 4] - tch_eoff[4 * ci];
      chunk_groups(ci, true);
      const int in_brick = (int)ci - tbr_ch0.back();
      if (in_brick > 0 && (in_brick == TBRICK || brick_groups.size() + newg.size() > (size_t)TSLOTS ||
                           tch_eoff[4 * ci + 4] - tch_eoff[4 * tbr_ch0.back()] > TBENT)) {
        close_brick((int)ci);
        chunk_groups(ci, false);
      }
      if (newg.size() > (size_t)TSLOTS || nent > TBENT) {
        tiled = false;   // one chunk is too crowded: keep the point-major kernels
        break;
      }
      for (int g : newg) {
        slot_of[g] = (int)brick_groups.size();
        brick_groups.push_back(g);
      }
      const int kk = (int)ci - tbr_ch0.back();
      for (int j = 0; j < 4; ++j)
        for (int e = tch_eoff[4 * ci + j]; e < tch_eoff[4 * ci + j + 1]; ++e) {
          te_slot[e] = slot_of[te_g[e]];
          te_lst[e] = 4 * kk + j;
        }
    }
    if (tiled) {
      close_brick((int)tch_c.size());
      te_info.resize(ne);
      for (size_t e = 0; e < ne; ++e) te_info[e] = te_slot[e] | te_nm[e] << 8;
      tgr_poff.push_back(0);
      for (int gi = 0; gi < ngr; ++gi) {
        tgr_pidx.insert(tgr_pidx.end(), group_parts[gi].begin(), group_parts[gi].end());
        tgr_poff.push_back((int)tgr_pidx.size());
      }
    }
  }
  l->ngroups = (int)gr_M.size();
  l->h_gr_nm = gr_nm;
  l->P = (int64_t)pt_G.size();
  l->C = (int64_t)ct_W.size();
  l->nA = aoff[nW];
  std::vector<int64_t> vr0(row0.begin(), row0.end() - 1), vr1(row0.begin() + 1, row0.end());
  std::vector<int64_t> va(aoff.begin(), aoff.end() - 1);
  std::vector<double> hA(A_all, A_all + l->nA);
  std::vector<double2> ph;
  for (int64_t i = 0; i < (int64_t)nq * nW; ++i) ph.push_back(make_double2(phase_qW[2 * i], phase_qW[2 * i + 1]));
  bool ok = upload(l, &l->A64, hA) && upload(l, &l->pt_G, pt_G) && upload(l, &l->pt_off, pt_off) &&
            upload(l, &l->ct_aoff, ct_aoff) && upload(l, &l->ct_M, ct_M) && upload(l, &l->ct_nm, ct_nm) &&
            upload(l, &l->ct_W, ct_W) && upload(l, &l->gr_M, gr_M) && upload(l, &l->gr_nm, gr_nm) &&
            upload(l, &l->gr_voff, gr_voff) && upload(l, &l->gv_W, gv_W) && upload(l, &l->vol_row0, vr0) &&
            upload(l, &l->vol_row1, vr1) && upload(l, &l->row_G, row_G) && upload(l, &l->vol_aoff, va) &&
            upload(l, &l->phase, ph);
  if (ok) {
    l->A32 = dalloc<float>(l, l->nA);
    ok = l->A32 != nullptr;
    if (ok && l->nA) {
      to_float<<<std::min<int64_t>((l->nA + 255) / 256, 4096), 256>>>(l->A64, l->A32, l->nA);
      ok = cudaDeviceSynchronize() == cudaSuccess;
    }
  }
  if (ok && !tiled && l->maxnm <= 16 && l->C) {
    l->pad_nm = l->maxnm <= 8 ? 8 : 16;
    l->pad_full = nM % 4 == 0;
    for (size_t i = 0; i < ct_nm.size() && l->pad_full; ++i) l->pad_full = ct_nm[i] == l->pad_nm && ct_M[i] % 4 == 0;
    l->A32p = dalloc<float>(l, l->C * l->pad_nm);
    ok = l->A32p != nullptr;
    if (ok) {
      lfc_pad_rows_kernel<<<(unsigned)std::min<int64_t>((l->C * l->pad_nm + 255) / 256, 4096), 256>>>(
          l->A64, l->ct_aoff, l->ct_nm, l->C, l->pad_nm, l->A32p);
      ok = cudaDeviceSynchronize() == cudaSuccess;
    }
  }
  if (ok && l->nf) {
    const int64_t ne = (int64_t)st_M.size();
    ok = upload(l, &l->st_sub, st_sub) && upload(l, &l->st_M, st_M) && upload(l, &l->sg_off, sg_off) &&
         upload(l, &l->sg_e, sg_e);
    l->st_A = ok ? dalloc<double>(l, ne * l->maxnm * 8) : nullptr;
    int64_t* d_a = nullptr;
    ok = l->st_A && cudaMalloc(&d_a, std::max<size_t>(1, ne) * sizeof(int64_t)) == cudaSuccess;
    if (ok && ne) {
      ok = cudaMemcpy(d_a, ent_a.data(), ne * sizeof(int64_t), cudaMemcpyHostToDevice) == cudaSuccess;
      if (ok) {
        lfc_blocks_kernel<<<(unsigned)std::min<int64_t>((ne * l->maxnm * 8 + 255) / 256, 16384), 256>>>(
            l->A64, d_a, l->st_M, ne, l->maxnm, l->st_A);
        ok = cudaDeviceSynchronize() == cudaSuccess;
      }
    }
    cudaFree(d_a);
  }
  if (ok && tiled) {
    ok = upload(l, &l->tch_c, tch_c) && upload(l, &l->tch_eoff, tch_eoff) && upload(l, &l->te_info, te_info) &&
         upload(l, &l->te_A, te_A) && upload(l, &l->tbr_ch0, tbr_ch0) && upload(l, &l->tbr_pbase, tbr_pbase) &&
         upload(l, &l->tps_M, tps_M) && upload(l, &l->tps_nm, tps_nm) && upload(l, &l->tps_eoff, tps_eoff) &&
         upload(l, &l->tps_info, tps_info) &&
         upload(l, &l->tgr_poff, tgr_poff) && upload(l, &l->tgr_pidx, tgr_pidx);
    l->tiled = ok;
    l->tbr_n = (int)tbr_ch0.size() - 1;
    l->tbr_smax = tbr_smax;
    l->tbr_emax = tbr_emax;
    l->tnm = std::all_of(gr_nm.begin(), gr_nm.end(), [&](int n) { return n == gr_nm[0]; }) ? gr_nm[0] : 0;
    l->tpart_n = tbr_pbase.back();
  }
  if (!ok) {
    gb_lfc_free(l);
    return fail(GB_E_NOMEM, "gb_lfc_new: device allocation / upload failed");
  }
  *out = l;
  return GB_OK;
}

int gb_lfc_tiled(const gb_lfc* l) { return l && l->tiled ? 1 : 0; }

int gb_lfc_add(const gb_lfc* l, const void* c_xM, void* a_xG, int64_t nx, int dtype, int q, void* stream) {
  GB_REQUIRE(l && dtype_valid(dtype) && nx >= 0, "gb_lfc_add: bad arguments");
  if (nx == 0) return GB_OK;
  GB_REQUIRE(c_xM && a_xG, "gb_lfc_add: null array");
  GB_REQUIRE(q < l->nq, "gb_lfc_add: k-point index out of range");
  cudaStream_t st = (cudaStream_t)stream;
  switch (dtype) {
    case GB_DTYPE_F64: return add_t<double>(l, c_xM, a_xG, nx, -1, st);
    case GB_DTYPE_F32: return add_t<float>(l, c_xM, a_xG, nx, -1, st);
    case GB_DTYPE_C128: return add_t<double2>(l, c_xM, a_xG, nx, q, st);
    default: return add_t<float2>(l, c_xM, a_xG, nx, q, st);
  }
}

int gb_lfc_integrate(const gb_lfc* l, const void* a_xG, void* c_xM, int64_t nx, int dtype, int q, void* stream) {
  GB_REQUIRE(l && dtype_valid(dtype) && nx >= 0, "gb_lfc_integrate: bad arguments");
  if (nx == 0) return GB_OK;
  GB_REQUIRE(c_xM && a_xG, "gb_lfc_integrate: null array");
  GB_REQUIRE(q < l->nq, "gb_lfc_integrate: k-point index out of range");
  cudaStream_t st = (cudaStream_t)stream;
  switch (dtype) {
    case GB_DTYPE_F64: return integrate_t<double>(l, a_xG, c_xM, nx, -1, st);
    case GB_DTYPE_F32: return integrate_t<float>(l, a_xG, c_xM, nx, -1, st);
    case GB_DTYPE_C128: return integrate_t<double2>(l, a_xG, c_xM, nx, q, st);
    default: return integrate_t<float2>(l, a_xG, c_xM, nx, q, st);
  }
}

int gb_lfc_add_k(const gb_lfc* l, const void* c_xM, void* a_xG, int64_t nx, int dtype, int nk, void* stream) {
  GB_REQUIRE(l && dtype_valid(dtype) && nx >= 0, "gb_lfc_add_k: bad arguments");
  GB_REQUIRE(dtype_complex(dtype), "gb_lfc_add_k: k-point batches are complex");
  GB_REQUIRE(nk >= 1 && nk <= l->nq && nx % nk == 0, "gb_lfc_add_k: nk must divide the batch and be <= nq");
  if (nx == 0) return GB_OK;
  GB_REQUIRE(c_xM && a_xG, "gb_lfc_add_k: null array");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t per = nx / nk;
  if (dtype == GB_DTYPE_C128) return add_t<double2>(l, c_xM, a_xG, nx, 0, st, per);
  return add_t<float2>(l, c_xM, a_xG, nx, 0, st, per);
}

int gb_lfc_integrate_k(const gb_lfc* l, const void* a_xG, void* c_xM, int64_t nx, int dtype, int nk,
                       void* stream) {
  GB_REQUIRE(l && dtype_valid(dtype) && nx >= 0, "gb_lfc_integrate_k: bad arguments");
  GB_REQUIRE(dtype_complex(dtype), "gb_lfc_integrate_k: k-point batches are complex");
  GB_REQUIRE(nk >= 1 && nk <= l->nq && nx % nk == 0,
             "gb_lfc_integrate_k: nk must divide the batch and be <= nq");
  if (nx == 0) return GB_OK;
  GB_REQUIRE(c_xM && a_xG, "gb_lfc_integrate_k: null array");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t per = nx / nk;
  if (dtype == GB_DTYPE_C128) return integrate_t<double2>(l, a_xG, c_xM, nx, 0, st, per);
  return integrate_t<float2>(l, a_xG, c_xM, nx, 0, st, per);
}

int gb_lfc_derivative(const gb_lfc* l, const void* a_xG, void* c_xMv, int64_t nx, const double h_cv[9],
                      const int64_t n_c[3], const gb_spline* const* spline_M, const int64_t beg_c[3],
                      const double* pos_Wv, int q, int dtype, void* stream) {
  GB_REQUIRE(l && dtype_valid(dtype) && nx >= 0, "gb_lfc_derivative: bad arguments");
  if (nx == 0 || l->nM == 0) return GB_OK;
  GB_REQUIRE(a_xG && c_xMv && h_cv && n_c && beg_c && pos_Wv && spline_M, "gb_lfc_derivative: null argument");
  GB_REQUIRE(q < l->nq, "gb_lfc_derivative: k-point index out of range");
  GB_REQUIRE(nx < 65536, "gb_lfc_derivative: at most 65535 grids per call");
  GB_REQUIRE(n_c[0] * n_c[1] * n_c[2] == l->nG, "gb_lfc_derivative: grid size does not match the object");
  for (int g = 0; g < l->ngroups; ++g)
    if (l->h_gr_nm[g] > 16) return fail(GB_E_UNSUPPORTED, "gb_lfc_derivative: more than 16 functions in a volume");
  // per M: the spline and its m index (m runs 0 .. 2l across consecutive
  // entries of one function, as the reference's spline_M list repeats each
  // function's spline 2l + 1 times)
  std::vector<SplineM> hs(l->nM);
  for (int M = 0; M < l->nM; ++M) {
    const gb_spline* sp = spline_M[M];
    if (!sp) return fail(GB_E_INVALID, "gb_lfc_derivative: null spline in spline_M");
    const int nmf = 2 * sp->l + 1;
    int m = 0;
    if (M > 0 && spline_M[M - 1] == sp && hs[M - 1].m + 1 < nmf) m = hs[M - 1].m + 1;
    hs[M] = SplineM{spline_view(sp), m};
  }
  DerivGeom geo;
  for (int c = 0; c < 3; ++c) {
    geo.n[c] = n_c[c];
    geo.beg[c] = beg_c[c];
  }
  for (int i = 0; i < 9; ++i) geo.h[i] = h_cv[i];
  cudaStream_t st = (cudaStream_t)stream;
  void* work = nullptr;
  const size_t sbytes = hs.size() * sizeof(SplineM), pbytes = (size_t)l->nW * 3 * sizeof(double);
  if (cudaMallocAsync(&work, sbytes + pbytes + 16, st) != cudaSuccess)
    return fail(GB_E_NOMEM, "gb_lfc_derivative: work space allocation failed");
  SplineM* d_spl = static_cast<SplineM*>(work);
  double* d_pos = reinterpret_cast<double*>(static_cast<char*>(work) + (sbytes + 15) / 16 * 16);
  int rc = GB_OK;
  if (cudaMemcpyAsync(d_spl, hs.data(), sbytes, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(d_pos, pos_Wv, pbytes, cudaMemcpyHostToDevice, st) != cudaSuccess)
    rc = fail(GB_E_CUDA, "gb_lfc_derivative: upload failed");
  if (!rc) {
    switch (dtype) {
      case GB_DTYPE_F64: rc = derivative_t<double>(l, d_spl, d_pos, geo, a_xG, c_xMv, nx, -1, st); break;
      case GB_DTYPE_F32: rc = derivative_t<float>(l, d_spl, d_pos, geo, a_xG, c_xMv, nx, -1, st); break;
      case GB_DTYPE_C128: rc = derivative_t<double2>(l, d_spl, d_pos, geo, a_xG, c_xMv, nx, q, st); break;
      default: rc = derivative_t<float2>(l, d_spl, d_pos, geo, a_xG, c_xMv, nx, q, st); break;
    }
  }
  cudaFreeAsync(work, st);
  // the host vectors above were read by the copies: finish them before return
  if (cudaStreamSynchronize(st) != cudaSuccess && !rc) rc = fail(GB_E_CUDA, "gb_lfc_derivative: sync failed");
  return rc;
}

}  // extern "C"
