// FD star stencil in tiles of the (axis1, axis2) plane: radius 4 to 6 on rows so
// long that a CTA of the row kernel holds few of them (fd_stencil_rows.cu has
// the rule and what it measured).
//
// A persistent CTA owns a (T1 x T2) tile of one grid and marches along axis 0.
// Planes (tile + halo) stream through a ring of NS shared-memory slots filled
// by cp.async (no register staging, D planes in flight); every thread keeps a
// register queue of 2H+1 values of its own R1 x R2 points along axis 0, so each
// input element is read from HBM once and from shared memory ~5-7 times.  Zero
// and periodic boundaries (with Bloch phases) are resolved while filling the
// tile: out-of-range cells become zeros or wrapped copies, wrapped copies of
// complex data are multiplied by the phase in a short fix-up pass (only tiles
// that touch a periodic face pay it).  The terms and their order are those of
// star_core.cuh without its symmetric form, so a band has the same bits here
// and in the marching kernel of fd_stencil.cu.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include "internal.cuh"

namespace gb {

struct TileArgs {
  const void* in;
  void* out;
  int64_t nbatch;
  int n0, n1, n2;
  int pbc0, pbc1, pbc2;
  int tiles1, tiles2;
  double c0;
  double c0diff;              // c0 + sum of the neighbour coefficients (difference form)
  double a[3][2 * HMAX + 1];  // a[axis][m + HMAX]: coefficient of offset m (m != 0)
  PhaseSets phs;              // Bloch phases per k-point group of bands
  // epilogue: out = alpha * S(in) + beta * in + gamma * y + vpot * in
  double alpha, beta, gamma;
  const void* y;
  const void* vpot;
};

template <typename T_, int H_, int R1_, int R2_, int TY_, int TZ_, int D_>
struct TileCfg {
  using T = T_;
  static constexpr int H = H_, R1 = R1_, R2 = R2_, TY = TY_, TZ = TZ_, D = D_;
  static constexpr int VEC = 16 / (int)sizeof(T);
  static constexpr int HZ = ((H + VEC - 1) / VEC) * VEC;
  static constexpr int T1 = TY * R1, T2 = TZ * R2;
  static constexpr int W = T2 + 2 * HZ;
  static constexpr int ROWS = T1 + 2 * H;
  static constexpr int PLANE = ROWS * W;
  static constexpr int NS = H + D;
  static constexpr int NT = TY * TZ;
  static constexpr int KH = T2 / VEC;       // chunks in a halo row
  static constexpr int KC = W / VEC;        // chunks in a centre row
  static constexpr int NCHUNK = 2 * H * KH + T1 * KC;
  static constexpr size_t SMEM = (size_t)NS * PLANE * sizeof(T);
  static_assert(R2 % VEC == 0, "R2 must be a multiple of the 16-byte vector");
  static_assert((W * sizeof(T)) % 16 == 0, "row pitch must keep 16-byte alignment");
};

// true modulo: partial tiles of small grids can reach several periods away
// (those cells feed no valid output, but their loads must stay in bounds)
__device__ __forceinline__ int tile_wrap(int i, int n) {
  int r = i % n;
  return r < 0 ? r + n : r;
}

template <class C>
__global__ void __launch_bounds__(C::NT, 2) tile_star_kernel(const TileArgs args) {
  using T = typename C::T;
  using R = typename Elem<T>::R;
  constexpr int H = C::H, R1 = C::R1, R2 = C::R2, TZ = C::TZ, VEC = C::VEC, HZ = C::HZ;
  constexpr int T1 = C::T1, T2 = C::T2, W = C::W, PLANE = C::PLANE, NS = C::NS, D = C::D;
  constexpr bool CPLX = Elem<T>::cplx;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* planes = reinterpret_cast<T*>(smem_raw);

  const int tid = threadIdx.x;
  const int ty = tid / TZ, tz = tid % TZ;
  const int n0 = args.n0, n1 = args.n1, n2 = args.n2;
  const int64_t n12 = (int64_t)n1 * n2;
  const int64_t n012 = n12 * n0;
  const int64_t ntiles = (int64_t)args.tiles1 * args.tiles2;
  const int64_t total = args.nbatch * ntiles * n0;
  int64_t s = total * blockIdx.x / gridDim.x;
  const int64_t s_end = total * (blockIdx.x + 1) / gridDim.x;

  const bool epi = args.alpha != 1.0 || args.beta != 0.0 || args.y != nullptr || args.vpot != nullptr;
  const R* __restrict__ vpot = reinterpret_cast<const R*>(args.vpot);
  const R ealpha = (R)args.alpha, ebeta = (R)args.beta, egamma = (R)args.gamma;
  // FP32: the difference form sum_p c_p (x_p - x_c) + (sum c) x_c keeps the
  // operator exactly constant-annihilating after the coefficients are rounded
  constexpr bool DIFF = sizeof(R) == 4;
  R c0 = DIFF ? (R)args.c0diff : (R)args.c0;
  R a0[2 * H + 1], a1[2 * H + 1], a2[2 * H + 1];
#pragma unroll
  for (int m = 0; m <= 2 * H; ++m) {
    a0[m] = (R)args.a[0][m - H + HMAX];
    a1[m] = (R)args.a[1][m - H + HMAX];
    a2[m] = (R)args.a[2][m - H + HMAX];
  }

  // the k-th offset (+ H) of axes 0 and 2: ascending, in FP32 pairs +1 -1 +2 -2 ..
  auto term = [](int k) {
    if (std::is_same<T, float>::value) return k & 1 ? H - (k / 2 + 1) : H + (k / 2 + 1);
    return k < H ? k : k + 1;
  };

  while (s < s_end) {
    const int64_t col = s / n0;
    const int p_start = (int)(s % n0);
    const int p_end = (int)(s_end - s < (int64_t)(n0 - p_start) ? p_start + (s_end - s) : n0);
    s += p_end - p_start;
    const int64_t band = col / ntiles;
    const int t = (int)(col % ntiles);
    const int y0 = (t / args.tiles2) * T1;
    const int z0 = (t % args.tiles2) * T2;
    const T* __restrict__ src = reinterpret_cast<const T*>(args.in) + band * n012;
    T* __restrict__ dst = reinterpret_cast<T*>(args.out) + band * n012;
    const T* __restrict__ ybase = args.y ? reinterpret_cast<const T*>(args.y) + band * n012 : nullptr;
    const auto& PH = args.phs.ph[phase_set_of(args.phs, band)];
    const bool edge = (y0 - H < 0) || (y0 + T1 + H > n1) || (z0 - HZ < 0) || (z0 + T2 + HZ > n2);

    const int j0 = p_start - H, j1 = p_end + H;   // planes pushed: [j0, j1)

    // plane j -> source plane (or -1 for an all-zero plane) and its phase
    auto plane_src = [&](int j, double& pr, double& pi) -> int {
      pr = 1.0; pi = 0.0;
      if (j >= 0 && j < n0) return j;
      if (!args.pbc0) return -1;
      const int side = j < 0 ? 1 : 0;
      pr = PH[0][side][0]; pi = PH[0][side][1];
      return tile_wrap(j, n0);
    };

    auto issue = [&](int j) {
      double pr, pi;
      const int sp = plane_src(j, pr, pi);
      if (sp < 0) return;
      T* P = planes + ((j - j0) % NS) * PLANE;
      const T* S = src + (int64_t)sp * n12;
      for (int e = tid; e < C::NCHUNK; e += C::NT) {
        int Rw, k;
        if (e < 2 * H * C::KH) {
          const int hr = e / C::KH;
          Rw = hr < H ? hr : hr + T1;
          k = HZ / VEC + e % C::KH;
        } else {
          const int e2 = e - 2 * H * C::KH;
          Rw = H + e2 / C::KC;
          k = e2 % C::KC;
        }
        T* sd = P + Rw * W + k * VEC;
        int y = y0 - H + Rw;
        if (y < 0 || y >= n1) {
          if (!args.pbc1) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) sd[v] = zero<T>();
            continue;
          }
          y = tile_wrap(y, n1);
        }
        const T* row = S + (int64_t)y * n2;
        const int zs = z0 - HZ + k * VEC;
        if (zs >= 0 && zs + VEC <= n2 && ((reinterpret_cast<uintptr_t>(row + zs) & 15) == 0)) {
          cp_async16(sd, row + zs);
        } else {
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            int z = zs + v;
            if (z < 0 || z >= n2) {
              if (!args.pbc2) { sd[v] = zero<T>(); continue; }
              z = tile_wrap(z, n2);
            }
            cp_async_elem(sd + v, row + z);
          }
        }
      }
    };

    // Bloch phase of wrapped in-plane cells (complex data only)
    auto fixup = [&](T* P) {
      for (int e = tid; e < C::NCHUNK * VEC; e += C::NT) {
        const int ec = e / VEC, v = e % VEC;
        int Rw, k;
        if (ec < 2 * H * C::KH) {
          const int hr = ec / C::KH;
          Rw = hr < H ? hr : hr + T1;
          k = HZ / VEC + ec % C::KH;
        } else {
          const int e2 = ec - 2 * H * C::KH;
          Rw = H + e2 / C::KC;
          k = e2 % C::KC;
        }
        const int y = y0 - H + Rw, z = z0 - HZ + k * VEC + v;
        double pr = 1.0, pi = 0.0;
        bool w = false;
        if (args.pbc1 && (y < 0 || y >= n1)) { const int sd = y < 0; pr = PH[1][sd][0]; pi = PH[1][sd][1]; w = true; }
        if (args.pbc2 && (z < 0 || z >= n2)) {
          const int sd = z < 0;
          const double qr = PH[2][sd][0], qi = PH[2][sd][1];
          const double tr = pr * qr - pi * qi, ti = pr * qi + pi * qr;
          pr = tr; pi = ti; w = true;
        }
        if (w) { T* c = P + Rw * W + k * VEC + v; *c = phase_mul(*c, pr, pi); }
      }
    };

    T q[2 * H + 1][R1][R2];
#pragma unroll
    for (int m = 0; m <= 2 * H; ++m)
#pragma unroll
      for (int r = 0; r < R1; ++r)
#pragma unroll
        for (int c = 0; c < R2; ++c) q[m][r][c] = zero<T>();

#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (j0 + d < j1) issue(j0 + d);
      cp_async_commit();
    }

    for (int j = j0; j < j1; ++j) {
      cp_async_wait<D - 1>();
      __syncthreads();
      double pr, pi;
      const int sp = plane_src(j, pr, pi);
      T* P = planes + ((j - j0) % NS) * PLANE;
      if (CPLX && args.phs.any && edge && sp >= 0) {
        fixup(P);
        __syncthreads();
      }
      // push own values of plane j into the axis-0 queue
#pragma unroll
      for (int m = 0; m < 2 * H; ++m)
#pragma unroll
        for (int r = 0; r < R1; ++r)
#pragma unroll
          for (int c = 0; c < R2; ++c) q[m][r][c] = q[m + 1][r][c];
      if (sp >= 0) {
#pragma unroll
        for (int r = 0; r < R1; ++r) {
          T v[R2];
          lds_vec<T, R2>(P + (H + ty * R1 + r) * W + HZ + tz * R2, v);
#pragma unroll
          for (int c = 0; c < R2; ++c) q[2 * H][r][c] = sp != j && args.phs.any ? phase_mul(v[c], pr, pi) : v[c];
        }
      } else {
#pragma unroll
        for (int r = 0; r < R1; ++r)
#pragma unroll
          for (int c = 0; c < R2; ++c) q[2 * H][r][c] = zero<T>();
      }

      const int cpl = j - H;   // centre plane computed this iteration
      if (cpl >= p_start) {
        const T* Pc = planes + ((cpl - j0) % NS) * PLANE;
        T acc[R1][R2];
        // axis 0 (register queue) and axis 2 (row windows)
#pragma unroll
        for (int r = 0; r < R1; ++r) {
          const T* rowp = Pc + (H + ty * R1 + r) * W + tz * R2;
          T wl[HZ], wr[HZ];
          lds_vec<T, HZ>(rowp, wl);
          lds_vec<T, HZ>(rowp + HZ + R2, wr);
#pragma unroll
          for (int c = 0; c < R2; ++c) {
            T x = scale(c0, q[H][r][c]);
#pragma unroll
            for (int k = 0; k < 2 * H; ++k) {
              const int m = term(k);
              x = fmadd(x, a0[m], DIFF ? sub(q[m][r][c], q[H][r][c]) : q[m][r][c]);
            }
#pragma unroll
            for (int k = 0; k < 2 * H; ++k) {
              const int m = term(k);
              const int cc = c + m - H;
              T v;
              if (cc < 0) v = wl[HZ + cc];
              else if (cc >= R2) v = wr[cc - R2];
              else v = q[H][r][cc];
              x = fmadd(x, a2[m], DIFF ? sub(v, q[H][r][c]) : v);
            }
            acc[r][c] = x;
          }
        }
        // axis 1: rows of the own block come from the queue, others from smem
#pragma unroll
        for (int rr = -H; rr < R1 + H; ++rr) {
          T v[R2];
          if (rr >= 0 && rr < R1) {
#pragma unroll
            for (int c = 0; c < R2; ++c) v[c] = q[H][rr][c];
          } else {
            lds_vec<T, R2>(Pc + (H + ty * R1 + rr) * W + HZ + tz * R2, v);
          }
#pragma unroll
          for (int r = 0; r < R1; ++r) {
            const int m = rr - r + H;
            if (m < 0 || m > 2 * H || m == H) continue;
#pragma unroll
            for (int c = 0; c < R2; ++c)
              acc[r][c] = fmadd(acc[r][c], a1[m], DIFF ? sub(v[c], q[H][r][c]) : v[c]);
          }
        }
        // epilogue (fused axpy passes of the multigrid V-cycle)
        if (epi) {
          const T* yp = ybase ? ybase + (int64_t)cpl * n12 : nullptr;
#pragma unroll
          for (int r = 0; r < R1; ++r) {
            const int y = y0 + ty * R1 + r;
#pragma unroll
            for (int c = 0; c < R2; ++c) {
              const int z = z0 + tz * R2 + c;
              T v = fmadd(scale(ealpha, acc[r][c]), ebeta, q[H][r][c]);
              if (yp && y < n1 && z < n2) v = fmadd(v, egamma, yp[(int64_t)y * n2 + z]);
              if (vpot && y < n1 && z < n2) v = fmadd(v, vpot[(int64_t)cpl * n12 + (int64_t)y * n2 + z], q[H][r][c]);
              acc[r][c] = v;
            }
          }
        }
        // store
        T* outp = dst + (int64_t)cpl * n12;
#pragma unroll
        for (int r = 0; r < R1; ++r) {
          const int y = y0 + ty * R1 + r;
          if (y >= n1) continue;
          T* o = outp + (int64_t)y * n2;
          const int z = z0 + tz * R2;
          if (z + R2 <= n2 && ((reinterpret_cast<uintptr_t>(o + z) & 15) == 0)) {
#pragma unroll
            for (int c = 0; c < R2; c += VEC) {
              float4 w4;
              T* e = reinterpret_cast<T*>(&w4);
#pragma unroll
              for (int k = 0; k < VEC; ++k) e[k] = acc[r][c + k];
              __stcs(reinterpret_cast<float4*>(o + z + c), w4);
            }
          } else {
#pragma unroll
            for (int c = 0; c < R2; ++c)
              if (z + c < n2) st_cs(o + z + c, acc[r][c]);
          }
        }
      }
      __syncthreads();
      if (j + D < j1) issue(j + D);
      cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();
  }
}

// ------------------------------------------------------------------ host
template <typename T, int H>
static int launch_tiles(const gb_operator* op, const void* in, void* out, int64_t nin, const double* ph,
                        cudaStream_t st, const Epilogue& ep, int nk) {
  constexpr int F32 = std::is_same<T, float>::value, C128 = std::is_same<T, double2>::value;
  using C = TileCfg<T, H, 2, F32 ? 4 : C128 ? 1 : 2, 8, F32 ? 8 : 16, 2>;
  TileArgs a{};
  a.n0 = (int)op->n[0]; a.n1 = (int)op->n[1]; a.n2 = (int)op->n[2];
  a.tiles1 = ceil_div(a.n1, C::T1);
  a.tiles2 = ceil_div(a.n2, C::T2);
  const int64_t total = nin * (int64_t)a.tiles1 * a.tiles2 * a.n0;
  // too few plane tiles to fill the pipelines
  if (total < 48 * sm_count()) return USE_MARCH;
  static int occ = -1;
  if (occ < 0) {
    cudaFuncSetAttribute(tile_star_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, tile_star_kernel<C>, C::NT, C::SMEM);
    if (occ < 1) occ = 1;
  }
  a.in = in; a.out = out; a.nbatch = nin;
  a.pbc0 = op->pbc[0]; a.pbc1 = op->pbc[1]; a.pbc2 = op->pbc[2];
  a.c0 = op->center;
  a.c0diff = op->center;
  for (int c = 0; c < 3; ++c)
    for (int m = 0; m < 2 * HMAX + 1; ++m) a.c0diff += op->a[c][m];
  memcpy(a.a, op->a, sizeof(a.a));
  a.alpha = ep.alpha; a.beta = ep.beta; a.gamma = ep.gamma; a.y = ep.y; a.vpot = ep.vpot;
  fill_phase_sets(a.phs, ph, nk, nin);
  int64_t blocks = (int64_t)sm_count() * occ;
  // keep at least a few planes per CTA so the prologue (2H planes) stays small
  blocks = std::min<int64_t>(blocks, std::max<int64_t>(1, total / (4 * H + 4)));
  tile_star_kernel<C><<<(unsigned)blocks, C::NT, C::SMEM, st>>>(a);
  return check_launch("tile_star_kernel");
}

template <typename T>
static int dispatch_tiles(const gb_operator* op, const void* in, void* out, int64_t nin, const double* ph,
                          cudaStream_t st, const Epilogue& ep, int nk) {
  switch (op->H) {
    case 4: return launch_tiles<T, 4>(op, in, out, nin, ph, st, ep, nk);
    case 5: return launch_tiles<T, 5>(op, in, out, nin, ph, st, ep, nk);
    default: return launch_tiles<T, 6>(op, in, out, nin, ph, st, ep, nk);
  }
}

int star_tiles_apply(const gb_operator* op, const void* in, void* out, int64_t nin, int dtype, const double* ph,
                     cudaStream_t st, const Epilogue& ep, int nk) {
  switch (dtype) {
    case GB_DTYPE_F64: return dispatch_tiles<double>(op, in, out, nin, ph, st, ep, nk);
    case GB_DTYPE_F32: return dispatch_tiles<float>(op, in, out, nin, ph, st, ep, nk);
    case GB_DTYPE_C128: return dispatch_tiles<double2>(op, in, out, nin, ph, st, ep, nk);
    default: return dispatch_tiles<float2>(op, in, out, nin, ph, st, ep, nk);
  }
}

}  // namespace gb
