// FD star stencil for the layouts the tensor copies of fd_stencil_tma.cu do
// not take: rows that are not whole 16-byte chunks (every zero-boundary grid
// with an even N has N - 1 points per axis) and Bloch phases.
//
// As in the TMA kernel a CTA owns T1 full rows of the (axis1, axis2) plane of
// one band and marches along axis 0 with a register queue of 2H + 1 planes.
// The planes are staged by every warp with one cp.async per element into
// shared-memory rows of the CTA's own pitch, which carry their halo columns
// explicitly (wrapped copies, or zeros): whatever the row length in memory,
// the neighbours are read as aligned 16-byte vectors without boundary tests.
// Each warp copies the same rows of every plane, so their offsets are worked
// out once per segment and a copy costs little more than its instruction.
// Wrapped cells of Bloch states are multiplied by their phase in place when
// their plane lands; they are first read H barriers later, as halo cells of
// the centre plane.  Ring: H + 1 planes in use and two on their way, one
// barrier per plane (deeper rings measured the same).
//
// On 60 FP64 grids of 75^3 the shared-memory data pipe is 62 % busy, issue
// slots 49 % (111 instructions per 32 points), DRAM 33 %: 16 warps per SM wait
// for their shared-memory reads.  (The 32 x 32 tiles before it spent most
// instructions on addresses, boundaries and the unused part of edge tiles:
// (160, 75^3) FP64 zero boundary 1080 -> 433 us, with a potential 1680 -> 506
// us; FP32 768 -> 305 us; (64, 60^3) complex128 with phases 597 -> 225 us, all
// before the compute part alone was unrolled.)
#include <algorithm>
#include <cstring>
#include "star_core.cuh"

namespace gb {

constexpr int ROWS_NT = 256;   // most threads of a CTA (two CTAs per SM at 128 registers)

struct RowsArgs {
  const void* in;
  void* out;
  const void* y;
  const void* vpot;
  int64_t nbatch;
  int n0, n1, n2;
  int pbc0, pbc1, pbc2;
  int TZ, NTC, T1, ROWS, ytiles;
  int pitch;        // elements per shared-memory row: halo, n2 columns, halo
  double c0;
  double c0diff;    // c0 + sum of the neighbour coefficients (difference form)
  double a[3][2 * HMAX + 1];
  double alpha, beta, gamma;
  PhaseSets phs;
};

template <typename T, int H>
struct RowsCfg {
  static constexpr int VEC = 16 / (int)sizeof(T), R2 = VEC;
  static constexpr int HZ = ((H + VEC - 1) / VEC) * VEC;
  static constexpr int D = 2;              // planes in flight
  static constexpr int NS = H + 1 + D;     // ring slots
  static constexpr int RPW = 4;            // most rows a warp copies per plane
};

template <typename T, int H, int R1, int SYM, int EPI>
__global__ void __launch_bounds__(ROWS_NT, 2) rows_star_kernel(const __grid_constant__ RowsArgs a) {
  using R = typename Elem<T>::R;
  using C = RowsCfg<T, H>;
  constexpr bool CPLX = Elem<T>::cplx;
  constexpr int VEC = C::VEC, R2 = C::R2, HZ = C::HZ, D = C::D, NS = C::NS;
  constexpr int NQ = 2 * H + 1;
  constexpr int RPW = RowsCfg<T, H>::RPW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const slots = reinterpret_cast<T*>(smem_raw);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int n0 = a.n0, n1 = a.n1, n2 = a.n2;
  const int pitch = a.pitch, slot_elems = a.ROWS * pitch;
  const int64_t n12 = (int64_t)n1 * n2;
  const int64_t total = a.nbatch * a.ytiles * n0;
  int64_t s = total * blockIdx.x / gridDim.x;
  const int64_t s_end = total * (blockIdx.x + 1) / gridDim.x;

  const bool active = tid < a.NTC;
  const int ctid = active ? tid : 0;
  const int ty = ctid / a.TZ, tz = ctid - ty * a.TZ;
  const int z = tz * R2;
  const int own = (H + ty * R1) * pitch + HZ + z;
  StarCoef<R, H, SYM> coef;
  if (SYM == 1) coef.init(a);
  const bool phased = CPLX && a.phs.any;

  // wrapped columns z = -H .. -1 and n2 .. n2 + H - 1 of a periodic axis 2
  const int hd = lane < H ? lane - H : n2 + lane - H, hs = lane < H ? hd + n2 : hd - n2;
  // the columns of a zero-boundary axis 2 beside the row stay zero
  for (int i = tid; i < NS * slot_elems; i += blockDim.x) slots[i] = zero<T>();

  while (s < s_end) {
    const int64_t col = s / n0;
    const int p_start = (int)(s % n0);
    const int p_end = (int)((s_end - s) < (int64_t)(n0 - p_start) ? p_start + (s_end - s) : n0);
    s += p_end - p_start;
    const int64_t band = col / a.ytiles;
    const int y0 = (int)(col % a.ytiles) * a.T1;
    const T* __restrict__ src = reinterpret_cast<const T*>(a.in) + band * n12 * n0;
    T* __restrict__ dst = reinterpret_cast<T*>(a.out) + band * n12 * n0;
    const T* __restrict__ ybase = a.y ? reinterpret_cast<const T*>(a.y) + band * n12 * n0 : nullptr;
    const auto& PH = a.phs.ph[phase_set_of(a.phs, band)];
    const int yrow = y0 + ty * R1;
    // rows past the last halo row of the grid feed no output
    const int rows = min(a.ROWS, n1 + 2 * H - y0);
    __syncthreads();      // the previous segment has read its last plane
    if (!a.pbc1 && (y0 < H || y0 + a.T1 + H > n1)) {
      // rows outside a zero-boundary axis 1: zero in every slot
      for (int r = warp; r < rows; r += nwarps) {
        const int y = y0 - H + r;
        if (y >= 0 && y < n1) continue;
        for (int i = 0; i < NS; ++i)
          for (int c = HZ + lane; c < HZ + n2; c += 32) slots[i * slot_elems + r * pitch + c] = zero<T>();
      }
    }

    // the rows this warp copies, the same for every plane of the segment
    int soff[RPW], doff[RPW];
    bool con[RPW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
      const int r = warp + i * nwarps;
      int y = y0 - H + r;
      const bool in = y >= 0 && y < n1;
      if (!in) y += y < 0 ? n1 : -n1;
      con[i] = r < rows && (in || a.pbc1);
      soff[i] = y * n2;
      doff[i] = r * pitch + HZ;
    }
    auto issue = [&](int j, int slot) {
      if (a.pbc0) j = j < 0 ? j + n0 : j >= n0 ? j - n0 : j;
      if (j < 0 || j >= n0) return;
      const T* plane = src + (int64_t)j * n12;
      T* P = slots + slot * slot_elems;
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        if (!con[i]) continue;            // uniform in the warp
        const T* g = plane + (soff[i] + lane);
        T* d = P + (doff[i] + lane);
        cp_async_elem_if(d, g, lane < n2);
        cp_async_elem_if(d + 32, g + 32, lane + 32 < n2);
        cp_async_elem_if(d + 64, g + 64, lane + 64 < n2);
        for (int c = lane + 96; c < n2; c += 32) cp_async_elem(P + doff[i] + c, plane + soff[i] + c);
        if (a.pbc2) cp_async_elem_if(P + (doff[i] + hd), plane + (soff[i] + hs), lane < 2 * H);
      }
    };
    const int64_t own_g = (int64_t)p_start * n12 + (int64_t)yrow * n2 + z;
    T* o = dst + own_g;
    const T* yp = EPI == 2 && ybase ? ybase + own_g : nullptr;
    const R* vp = EPI && a.vpot ? reinterpret_cast<const R*>(a.vpot) + own_g : nullptr;
    bool on[R1][R2];
#pragma unroll
    for (int r = 0; r < R1; ++r)
#pragma unroll
      for (int c = 0; c < R2; ++c) on[r][c] = active && yrow + r < n1 && z + c < n2;

    const int j0 = p_start - H, j1 = p_end + H;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (j0 + d < j1) issue(j0 + d, d);
      cp_async_commit();
    }
    T q[NQ][R1][R2];
    int slot = 0;
    int turn = 0;
    for (int j = j0; j < j1; ++j) {
      cp_async_wait<D - 1>();
      __syncthreads();
      // the slot refilled here was last read as the centre plane of step j - 1
      {
        int ns = slot + D;
        if (ns >= NS) ns -= NS;
        if (j + D < j1) issue(j + D, ns);
        cp_async_commit();
      }
      if (phased) {
        // Bloch phases of the wrapped cells of the plane that just landed:
        // they are read when it is the centre plane, H barriers from here
        T* L = slots + slot * slot_elems;
        const int ncol = a.pbc2 ? 2 * H * a.T1 : 0;
        const int top = a.pbc1 ? max(0, H - y0) : 0;                    // wrapped rows above the grid
        const int nrow = a.pbc1 ? top + max(0, rows - (n1 + H - y0)) : 0;
        for (int e = tid; e < ncol + nrow * n2; e += blockDim.x) {
          int off, ax, sd;
          if (e < ncol) {
            const int r = e / (2 * H), k = e - r * (2 * H);
            ax = 2;
            sd = k < H ? 1 : 0;
            off = (H + r) * pitch + HZ + (k < H ? k - H : n2 + k - H);
          } else {
            const int r = (e - ncol) / n2, c = (e - ncol) - r * n2;
            ax = 1;
            sd = r < top ? 1 : 0;
            off = (r < top ? r : n1 + H - y0 + (r - top)) * pitch + HZ + c;
          }
          L[off] = phase_mul(L[off], PH[ax][sd][0], PH[ax][sd][1]);
        }
      }
      const int cpl = j - H;
      T yv[R1][R2];
      R vv[R1][R2];
      if (EPI && cpl >= p_start) {
#pragma unroll
        for (int r = 0; r < R1; ++r)
#pragma unroll
          for (int c = 0; c < R2; ++c) {
            if (EPI == 2) yv[r][c] = ld_if(yp + (r * n2 + c), a.y && on[r][c]);
            vv[r][c] = ld_if(vp + (r * n2 + c), a.vpot && on[r][c]);
          }
      }
      // only this part is unrolled over the turns of the register queue (the
      // whole step seven times over waited for instructions: 68 -> 59 us for 96
      // complex128 bands of 28^3, 580 -> 537 us for 160 FP64 bands of 75^3)
      auto turn_of = [&](auto uc) {
        constexpr int u = uc.value;
        const T* P = slots + slot * slot_elems + own;
        const bool outside = j < 0 || j >= n0;
        if (outside && !a.pbc0) {
#pragma unroll
          for (int r = 0; r < R1; ++r)
#pragma unroll
            for (int c = 0; c < R2; ++c) q[u][r][c] = zero<T>();
        } else {
#pragma unroll
          for (int r = 0; r < R1; ++r) lds_vec<T, R2>(P + r * pitch, q[u][r]);
          if (phased && outside) {
            const int sd = j < 0 ? 1 : 0;
#pragma unroll
            for (int r = 0; r < R1; ++r)
#pragma unroll
              for (int c = 0; c < R2; ++c) q[u][r][c] = phase_mul(q[u][r][c], PH[0][sd][0], PH[0][sd][1]);
          }
        }
        if (cpl >= p_start) {
          const int cu = (u + NQ - H) % NQ;
          int cslot = slot - H;
          if (cslot < 0) cslot += NS;
          const T* Pc = slots + cslot * slot_elems + own;
          T acc[R1][R2];
          star_points<T, H, R1, R2, HZ, SYM>(
              acc, q, u, coef, a,
              [&](int r, T(&w)[HZ]) { lds_vec<T, HZ>(Pc + r * pitch - HZ, w); },
              [&](int r, T(&w)[HZ]) { lds_vec<T, HZ>(Pc + r * pitch + R2, w); },
              [&](int rr, T(&v)[R2]) {
                // a wrapped row among the own ones was queued without its phase
                if (rr < 0 || rr >= R1 || (phased && rr > 0 && yrow + rr >= n1)) lds_vec<T, R2>(Pc + rr * pitch, v);
              },
              // so was the second column of the last pair of an odd row
              [&](int r, int cc, T v) { return phased && cc > 0 && z + cc >= n2 ? Pc[r * pitch + cc] : v; });
#pragma unroll
          for (int r = 0; r < R1; ++r)
#pragma unroll
            for (int c = 0; c < R2; ++c) {
              T v = acc[r][c];
              if (EPI == 2) {
                v = fmadd(scale((R)a.alpha, v), (R)a.beta, q[cu][r][c]);
                if (a.y) v = fmadd(v, (R)a.gamma, yv[r][c]);
              }
              if (EPI && a.vpot) v = fmadd(v, vv[r][c], q[cu][r][c]);
              st_cs_if(o + (r * n2 + c), v, on[r][c]);
            }
          o += n12;
          if (EPI == 2) yp += yp ? n12 : 0;
          if (EPI) vp += vp ? n12 : 0;
        }
      };
      switch (turn) {
        case 0: turn_of(std::integral_constant<int, 0>{}); break;
        case 1: turn_of(std::integral_constant<int, 1 % NQ>{}); break;
        case 2: turn_of(std::integral_constant<int, 2 % NQ>{}); break;
        case 3: if constexpr (NQ > 3) turn_of(std::integral_constant<int, 3 % NQ>{}); break;
        case 4: if constexpr (NQ > 3) turn_of(std::integral_constant<int, 4 % NQ>{}); break;
        case 5: if constexpr (NQ > 5) turn_of(std::integral_constant<int, 5 % NQ>{}); break;
        case 6: if constexpr (NQ > 5) turn_of(std::integral_constant<int, 6 % NQ>{}); break;
        case 7: if constexpr (NQ > 7) turn_of(std::integral_constant<int, 7 % NQ>{}); break;
        case 8: if constexpr (NQ > 7) turn_of(std::integral_constant<int, 8 % NQ>{}); break;
        case 9: if constexpr (NQ > 9) turn_of(std::integral_constant<int, 9 % NQ>{}); break;
        case 10: if constexpr (NQ > 9) turn_of(std::integral_constant<int, 10 % NQ>{}); break;
        case 11: if constexpr (NQ > 11) turn_of(std::integral_constant<int, 11 % NQ>{}); break;
        case 12: if constexpr (NQ > 11) turn_of(std::integral_constant<int, 12 % NQ>{}); break;
      }
      if (++turn == NQ) turn = 0;
      if (++slot == NS) slot = 0;
    }
    cp_async_wait<0>();
  }
}

// ------------------------------------------------------------------ host
template <typename T, int H, int R1, int SYM, int EPI>
static int launch_rows(const gb_operator* op, const void* in, void* out, int64_t nin, const double* ph,
                       cudaStream_t st, const Epilogue& ep, int nk) {
  using C = RowsCfg<T, H>;
  constexpr int R2 = C::R2, HZ = C::HZ;
  auto kern = rows_star_kernel<T, H, R1, SYM, EPI>;
  static int regs = -1;
  if (regs < 0) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return USE_MARCH;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    regs = fa.numRegs;
  }
  RowsArgs a{};
  a.in = in; a.out = out; a.y = ep.y; a.vpot = ep.vpot; a.nbatch = nin;
  a.n0 = (int)op->n[0]; a.n1 = (int)op->n[1]; a.n2 = (int)op->n[2];
  a.pbc0 = op->pbc[0]; a.pbc1 = op->pbc[1]; a.pbc2 = op->pbc[2];
  a.TZ = ceil_div(a.n2, R2);
  a.pitch = a.TZ * R2 + 2 * HZ;
  double best = 0.0;
  int bctas = 0, bty = 0;
  for (int ty = 1; ty * a.TZ <= ROWS_NT; ++ty) {
    const int T1 = ty * R1;
    if (ty > 1 && T1 >= a.n1 + R1) break;
    const int threads = (ty * a.TZ + 31) / 32 * 32;
    const int smem = C::NS * (T1 + 2 * H) * a.pitch * (int)sizeof(T);
    if (smem > 227 * 1024 || T1 + 2 * H > C::RPW * (threads / 32)) continue;
    const int ctas = std::min(65536 / (threads * ((regs + 7) / 8 * 8)), 228 * 1024 / (smem + 1024));
    if (ctas < 1) continue;
    const double cw = std::min(24.0, ctas * (ty * a.TZ / 32.0));
    const double eff = (double)a.n1 / ((double)ceil_div(a.n1, T1) * (T1 + 1.0 * H));
    const double score = cw * eff * (ctas > 1 ? 1.0 : 0.7);
    if (score > best) { best = score; bctas = ctas; bty = ty; }
  }
  // No tile: rows too short for the copies of a warp (four rows per plane).
  if (!bty && a.TZ <= 64) return USE_MARCH;
  // Rows so long that a tile holds few of them, or none: most of what is staged
  // is halo.  The marching kernel takes over at radius 3 and 4 without wrapped
  // halos (radius 3, 40 bands of 24 x 25 x 301 where five warps are left per SM:
  // FP64 119 against 95 us, complex64 148 against 99), in FP32 at radius 5 and 6
  // too (40 bands of 12 x 13 x 701, periodic: 150 us, 290 in the tile kernel)
  // and, at any height, complex128 of radius 5 and 6 (160 bands of 44^3 523
  // against 398 us); the tile kernel the rest (radius 4, 40 periodic complex128 bands of 64 x 64 x
  // 131: 1454 against 521 us; radius 6, 40 FP64 bands of 96^3, five rows per
  // tile, zero boundary: 548 against 449).
  constexpr bool F32 = std::is_same<T, float>::value, C128 = sizeof(T) == 16;
  const bool per = a.pbc0 || a.pbc1 || a.pbc2;
  const int T1 = bty * R1, warps = bctas * ((bty * a.TZ + 31) / 32);
  if (H >= 5) {
    if (C128 && !per) return USE_MARCH;
    if (T1 < 3 || (T1 < 6 && !per && !F32)) return F32 ? USE_MARCH : USE_TILES;
  }
  if (H == 4 && T1 < (F32 && per ? 2 : 3)) return per ? USE_TILES : USE_MARCH;
  if (!bty || (H == 3 && bty == 1 && !per && (C128 || warps < 8))) return USE_MARCH;
  a.NTC = bty * a.TZ; a.T1 = bty * R1; a.ROWS = a.T1 + 2 * H;
  a.ytiles = ceil_div(a.n1, a.T1);
  a.c0 = op->center;
  a.c0diff = op->center;
  for (int c = 0; c < 3; ++c)
    for (int m = 0; m < 2 * HMAX + 1; ++m) a.c0diff += op->a[c][m];
  memcpy(a.a, op->a, sizeof(a.a));
  a.alpha = ep.alpha; a.beta = ep.beta; a.gamma = ep.gamma;
  fill_phase_sets(a.phs, ph, nk, nin);
  const int threads = (a.NTC + 31) / 32 * 32;
  const size_t smem = (size_t)C::NS * a.ROWS * a.pitch * sizeof(T);
  const int64_t total = nin * (int64_t)a.ytiles * a.n0;
  // too few plane tiles to fill the pipelines: the marching kernel
  if (total < 16 * sm_count()) return USE_MARCH;
  int64_t blocks = (int64_t)sm_count() * bctas;
  blocks = std::min<int64_t>(blocks, std::max<int64_t>(1, total / (H + 1)));
  kern<<<(unsigned)blocks, threads, smem, st>>>(a);
  return check_launch("rows_star_kernel");
}

template <typename T>
static int dispatch_rows(const gb_operator* op, const void* in, void* out, int64_t nin, const double* ph,
                         cudaStream_t st, const Epilogue& ep, int nk) {
  const bool sym = symmetric_stencil<typename Elem<T>::R>(op);
  const int epi = ep.y || ep.alpha != 1.0 || ep.beta != 0.0 ? 2 : ep.vpot ? 1 : 0;
  // faster marching (fd_stencil.cu): 7-point FP32 stencils, and rows so short
  // that a plane hardly fills a CTA (FP64, radius 1: 300 bands of 15^3 33 us
  // here, 12 us there; radius 4: 160 bands of 25^3 52 and 35 us)
  if (std::is_same<T, float>::value && op->H == 1) return USE_MARCH;
  if (sizeof(T) < 16 && op->n[2] < 28) return USE_MARCH;
  if (sym && op->H == 1)
    return epi == 2 ? launch_rows<T, 1, 2, 1, 2>(op, in, out, nin, ph, st, ep, nk)
                    : launch_rows<T, 1, 2, 1, 1>(op, in, out, nin, ph, st, ep, nk);
  if (sym && op->H == 3) switch (epi) {
      case 0: return launch_rows<T, 3, 2, 1, 0>(op, in, out, nin, ph, st, ep, nk);
      case 1: return launch_rows<T, 3, 2, 1, 1>(op, in, out, nin, ph, st, ep, nk);
      default: return launch_rows<T, 3, 2, 1, 2>(op, in, out, nin, ph, st, ep, nk);
    }
  switch (op->H) {
    case 1: return launch_rows<T, 1, 2, 0, 2>(op, in, out, nin, ph, st, ep, nk);
    case 2: return launch_rows<T, 2, 2, 0, 2>(op, in, out, nin, ph, st, ep, nk);
    case 3: return launch_rows<T, 3, 2, 0, 2>(op, in, out, nin, ph, st, ep, nk);
    case 4: return launch_rows<T, 4, 1, 0, 2>(op, in, out, nin, ph, st, ep, nk);
    // 160 periodic bands of 56^3, marching against here: FP64 1646 -> 410 us,
    // FP32 1083 -> 293 (radius 6)
    case 5:
      return epi ? launch_rows<T, 5, 1, 0, 2>(op, in, out, nin, ph, st, ep, nk)
                 : launch_rows<T, 5, 1, 0, 0>(op, in, out, nin, ph, st, ep, nk);
    case 6:
      return epi ? launch_rows<T, 6, 1, 0, 2>(op, in, out, nin, ph, st, ep, nk)
                 : launch_rows<T, 6, 1, 0, 0>(op, in, out, nin, ph, st, ep, nk);
    default: return USE_MARCH;
  }
}

int star_rows_apply(const gb_operator* op, const void* in, void* out, int64_t nin, int dtype, const double* ph,
                    cudaStream_t st, const Epilogue& ep, int nk) {
  if (op->n[1] * op->n[2] >= (1LL << 31)) return USE_MARCH;
  switch (dtype) {
    case GB_DTYPE_F64: return dispatch_rows<double>(op, in, out, nin, ph, st, ep, nk);
    case GB_DTYPE_F32: return dispatch_rows<float>(op, in, out, nin, ph, st, ep, nk);
    case GB_DTYPE_C128: return dispatch_rows<double2>(op, in, out, nin, ph, st, ep, nk);
    default: return dispatch_rows<float2>(op, in, out, nin, ph, st, ep, nk);
  }
}

}  // namespace gb
