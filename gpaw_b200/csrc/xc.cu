// Exchange-correlation on the grid (replaces _gpaw.XCFunctional for LDA and
// the PBE family: c/xc/xc.c:73-227, c/xc/pbe.c, c/xc/rpbe.c).
//
// Written from the published forms:
//   * LDA exchange  e_x = -(3/4)(3/pi)^(1/3) n^(1/3) = C1 / r_s
//   * PW92 correlation (Perdew & Wang, PRB 45, 13244 (1992)): the G(r_s)
//     interpolation with the published (A, alpha1, beta1..beta4) for the
//     paramagnetic, ferromagnetic and spin-stiffness channels, and the
//     f(zeta) spin interpolation
//   * PBE (Perdew, Burke & Ernzerhof, PRL 77, 3865 (1996)): exchange
//     enhancement F_x(s) = 1 + kappa - kappa / (1 + mu s^2 / kappa), gradient
//     correction H(r_s, zeta, t); revPBE (kappa = 1.245) and RPBE
//     (F_x = 1 + kappa (1 - exp(-mu s^2 / kappa)))
// Derivatives are taken w.r.t. r_s at fixed |grad n|^2 (a2), as the reference
// does, and combined into
//   e_g = n (e_x + e_c),  v_g += e_x + e_c - r_s (de_x/dr_s + de_c/dr_s) / 3,
//   dedsigma = n (de_x/da2 + de_c/da2)
// with the reference's spin-scaling for two spins (c/xc/xc.c:149-225).
// Densities below NMIN = 1e-10 are clamped (c/xc/xc_gpaw.h).  FP64 only.
// One thread per grid point; HBM-bound for LDA, FP64-pipe-bound for PBE.
#include <algorithm>
#include <cmath>
#include "internal.cuh"

namespace gb {
namespace xc {

constexpr double PI = 3.14159265358979323846;
constexpr double NMIN = 1.0e-10;
// PBE beta and gamma = (1 - ln 2) / pi^2
constexpr double BETA = 0.066725;
constexpr double GAMMA = 0.031091;

struct Par {
  int gga;      // 0: LDA
  int rpbe;     // RPBE exchange form
  double kappa;
  double mu;    // beta pi^2 / 3
  double C0I;   // 3 / (4 pi)
  double C1;    // LDA exchange: e_x = C1 / r_s
  double C2;    // s^2 = a2 (C2 r_s / n)^2
  double C3;    // t^2 = C3 a2 r_s / (n^2 phi^2)
  double CC1;   // 1 / (2^(4/3) - 2)
  double CC2;   // 4 CC1 / 3
  double IF2;   // 1 / f''(0)
};

// PW92 G(r_s) and dG/dr_s:  G = -2 A (1 + a1 r_s) ln(1 + 1 / (2 A Q)),
// Q = b1 r_s^1/2 + b2 r_s + b3 r_s^3/2 + b4 r_s^2
__device__ __forceinline__ double pw92_G(double rtrs, double A, double a1, double b1, double b2,
                                         double b3, double b4, double* dGdrs) {
  const double rs = rtrs * rtrs;
  const double P = -2.0 * A * (1.0 + a1 * rs);
  const double Q = 2.0 * A * rtrs * (b1 + rtrs * (b2 + rtrs * (b3 + rtrs * b4)));
  const double L = log(1.0 + 1.0 / Q);
  const double G = P * L;
  // dQ/drs = A (b1 / rtrs + 2 b2 + 3 b3 rtrs + 4 b4 rs)
  const double dQ = A * (b1 / rtrs + 2.0 * b2 + rtrs * (3.0 * b3 + 4.0 * b4 * rtrs));
  *dGdrs = -2.0 * A * a1 * L - P * dQ / (Q * (Q + 1.0));
  return G;
}

__device__ __forceinline__ double exchange(const Par& p, double n, double rs, double a2,
                                           double* dedrs, double* deda2) {
  double e = p.C1 / rs;
  *dedrs = -e / rs;
  if (p.gga) {
    double c = p.C2 * rs / n;
    c *= c;
    const double s2 = a2 * c;
    double Fx, dFxds2;
    if (p.rpbe) {
      const double x = exp(-p.mu * s2 / p.kappa);
      Fx = 1.0 + p.kappa * (1.0 - x);
      dFxds2 = p.mu * x;
    } else {
      const double x = 1.0 + p.mu * s2 / p.kappa;
      Fx = 1.0 + p.kappa - p.kappa / x;
      dFxds2 = p.mu / (x * x);
    }
    // s^2 ~ r_s^8 at fixed a2
    *dedrs = *dedrs * Fx + e * dFxds2 * 8.0 * s2 / rs;
    *deda2 = e * dFxds2 * c;
    e *= Fx;
  }
  return e;
}

__device__ __forceinline__ double correlation(const Par& p, double n, double rs, double zeta, double a2,
                                              bool spinpol, double* dedrs, double* dedzeta,
                                              double* deda2) {
  const double rtrs = sqrt(rs);
  double de0;
  const double e0 = pw92_G(rtrs, GAMMA, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294, &de0);
  double e;
  double xp = 1.0, xm = 1.0;
  if (spinpol) {
    double de1, dalpha;
    const double e1 = pw92_G(rtrs, 0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517, &de1);
    const double alpha = -pw92_G(rtrs, 0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671, &dalpha);
    dalpha = -dalpha;
    const double zp = 1.0 + zeta, zm = 1.0 - zeta;
    xp = cbrt(zp);
    xm = cbrt(zm);
    const double f = p.CC1 * (zp * xp + zm * xm - 2.0);
    const double f1 = p.CC2 * (xp - xm);
    const double z3 = zeta * zeta * zeta, z4 = z3 * zeta;
    const double x = 1.0 - z4;
    *dedrs = de0 * (1.0 - f * z4) + de1 * f * z4 + dalpha * f * x * p.IF2;
    *dedzeta = 4.0 * z3 * f * (e1 - e0 - alpha * p.IF2) + f1 * (z4 * e1 - z4 * e0 + x * alpha * p.IF2);
    e = e0 + alpha * p.IF2 * f * x + (e1 - e0) * f * z4;
  } else {
    *dedrs = de0;
    e = e0;
  }
  if (p.gga) {
    const double n2 = n * n;
    double phi = 1.0, phi2 = 1.0, phi3 = 1.0;
    if (spinpol) {
      phi = 0.5 * (xp * xp + xm * xm);
      phi2 = phi * phi;
      phi3 = phi * phi2;
    }
    const double t2 = p.C3 * a2 * rs / (n2 * phi2);
    const double y = -e / (GAMMA * phi3);
    const double x = exp(y);
    const double A = (x != 1.0) ? BETA / (GAMMA * (x - 1.0)) : BETA / (GAMMA * y);
    const double At2 = A * t2;
    const double nom = 1.0 + At2;
    const double denom = nom + At2 * At2;
    double H = GAMMA * log(1.0 + BETA * t2 * nom / (denom * GAMMA));
    double tmp = GAMMA * BETA / (denom * (BETA * t2 * nom + GAMMA * denom));
    const double tmp2 = A * A * x / BETA;
    double dAdrs = tmp2 * *dedrs;
    if (spinpol) {
      H *= phi3;
      tmp *= phi3;
      dAdrs /= phi3;
    }
    const double dHdt2 = (1.0 + 2.0 * At2) * tmp;
    const double dHdA = -At2 * t2 * t2 * (2.0 + At2) * tmp;
    // t^2 ~ r_s^7 at fixed a2
    *dedrs += dHdt2 * 7.0 * t2 / rs + dHdA * dAdrs;
    *deda2 = dHdt2 * p.C3 * rs / n2;
    if (spinpol) {
      const double dphidzeta = (1.0 / xp - 1.0 / xm) / 3.0;
      const double dAdzeta = tmp2 * (*dedzeta - 3.0 * e * dphidzeta / phi) / phi3;
      *dedzeta += (3.0 * H / phi - dHdt2 * 2.0 * t2 / phi) * dphidzeta + dHdA * dAdzeta;
      *deda2 /= phi2;
    }
    e += H;
  }
  return e;
}

// One point, spin-paired: e, the increment of v, and dedsigma (GGA).
__device__ __forceinline__ void point_unpolarized(const Par& p, double n, double a2, double& e, double& dv,
                                                  double& ds) {
  if (n < NMIN) n = NMIN;
  const double rs = cbrt(p.C0I / n);
  double dexdrs, dexda2 = 0.0, decdrs, decda2 = 0.0, dz;
  const double ex = exchange(p, n, rs, a2, &dexdrs, &dexda2);
  const double ec = correlation(p, n, rs, 0.0, a2, false, &decdrs, &dz, &decda2);
  ds = n * (dexda2 + decda2);
  e = n * (ex + ec);
  dv = ex + ec - rs * (dexdrs + decdrs) / 3.0;
}

// One point, spin-polarised: sigma and dedsigma are (up up, up down, down down).
__device__ __forceinline__ void point_polarized(const Par& p, double nu, double nd, const double (&sg)[3], double& e,
                                                double (&dv)[2], double (&ds)[3]) {
  double na = 2.0 * nu;
  if (na < NMIN) na = NMIN;
  const double rsa = cbrt(p.C0I / na);
  double nb = 2.0 * nd;
  if (nb < NMIN) nb = NMIN;
  const double rsb = cbrt(p.C0I / nb);
  const double n = 0.5 * (na + nb);
  const double rs = cbrt(p.C0I / n);
  const double zeta = 0.5 * (na - nb) / n;
  double dexadrs, dexada2 = 0.0, dexbdrs, dexbda2 = 0.0, decdrs, decdzeta, decda2 = 0.0;
  double exa, exb, ec;
  if (p.gga) {
    exa = exchange(p, na, rsa, 4.0 * sg[0], &dexadrs, &dexada2);
    exb = exchange(p, nb, rsb, 4.0 * sg[2], &dexbdrs, &dexbda2);
    const double a2 = sg[0] + 2.0 * sg[1] + sg[2];
    ec = correlation(p, n, rs, zeta, a2, true, &decdrs, &decdzeta, &decda2);
    ds[0] = 2.0 * na * dexada2 + n * decda2;
    ds[1] = 2.0 * n * decda2;
    ds[2] = 2.0 * nb * dexbda2 + n * decda2;
  } else {
    exa = exchange(p, na, rsa, 0.0, &dexadrs, &dexada2);
    exb = exchange(p, nb, rsb, 0.0, &dexbdrs, &dexbda2);
    ec = correlation(p, n, rs, zeta, 0.0, true, &decdrs, &decdzeta, &decda2);
  }
  e = 0.5 * (na * exa + nb * exb) + n * ec;
  dv[0] = exa + ec - (rsa * dexadrs + rs * decdrs) / 3.0 - (zeta - 1.0) * decdzeta;
  dv[1] = exb + ec - (rsb * dexbdrs + rs * decdrs) / 3.0 - (zeta + 1.0) * decdzeta;
}

__global__ void xc_unpolarized(const Par p, int64_t ng, double* __restrict__ e_g,
                               const double* __restrict__ n_g, double* __restrict__ v_g,
                               const double* __restrict__ sigma_g, double* __restrict__ dedsigma_g) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < ng;
       g += (int64_t)gridDim.x * blockDim.x) {
    double e, dv, ds;
    point_unpolarized(p, n_g[g], p.gga ? sigma_g[g] : 0.0, e, dv, ds);
    if (p.gga) dedsigma_g[g] = ds;
    e_g[g] = e;
    v_g[g] += dv;
  }
}

__global__ void xc_polarized(const Par p, int64_t ng, double* __restrict__ e_g,
                             const double* __restrict__ n_sg, double* __restrict__ v_sg,
                             const double* __restrict__ sigma_xg, double* __restrict__ dedsigma_xg) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < ng;
       g += (int64_t)gridDim.x * blockDim.x) {
    double e, dv[2], ds[3], sg[3] = {0.0, 0.0, 0.0};
    if (p.gga)
#pragma unroll
      for (int x = 0; x < 3; ++x) sg[x] = sigma_xg[x * ng + g];
    point_polarized(p, n_sg[g], n_sg[ng + g], sg, e, dv, ds);
    if (p.gga)
#pragma unroll
      for (int x = 0; x < 3; ++x) dedsigma_xg[x * ng + g] = ds[x];
    e_g[g] = e;
    v_sg[g] += dv[0];
    v_sg[ng + g] += dv[1];
  }
}

// GGA on the grid in two launches.  The first evaluates, per point, grad n
// (central differences along the axes, neighbours through L1), sigma, the
// functional, and stores the flux 2 (de/dsigma_ss) grad n_s + (de/dsigma_ud)
// grad n_s'; the second subtracts its divergence from v.  Separate gradients,
// sums, products and divergences took 27 launches, each through memory: 594
// us for PBE on 151^3 points against 201 us for the two.  The first (146 us)
// is bound by the functional's FP64 arithmetic, the second (54 us) by the
// flux, whose three arrays no longer fit L2 beside the others at that size
// (marching along axis 0 to read one of them once measured the same).
constexpr int GH = 4;                      // largest stencil radius
struct GradArgs {
  int n[3], pbc[3], H;
  double c0[3], a[3][2 * GH + 1];          // centre and offset coefficients of d/dx_v along axis v
};

// sum_m a_v[m] f[. + m along axis v] (f: this point; i: its index on the axis);
// the loads are issued together
template <int H>
__device__ __forceinline__ double axis_derivative(const GradArgs& ga, const double* __restrict__ f, int v, int i,
                                                  int64_t stride) {
  double w[2 * H + 1];
#pragma unroll
  for (int m = -H; m <= H; ++m) {
    int j = i + m;
    bool ok = true;
    if (j < 0 || j >= ga.n[v]) {
      ok = ga.pbc[v];
      j += j < 0 ? ga.n[v] : -ga.n[v];
    }
    w[m + H] = ok ? __ldg(f + (j - i) * stride) : 0.0;
  }
  double x = ga.c0[v] * w[H];
#pragma unroll
  for (int m = -H; m <= H; ++m)
    if (m) x = fma(ga.a[v][m + GH], w[m + H], x);
  return x;
}

template <int NS, int H>
__global__ void __launch_bounds__(256) gga_flux_kernel(const Par p, const __grid_constant__ GradArgs ga, int64_t ng,
                                                       double* __restrict__ e_g, const double* __restrict__ n_sg,
                                                       double* __restrict__ v_sg, double* __restrict__ flux) {
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (g >= ng) return;
  const int64_t st[3] = {(int64_t)ga.n[1] * ga.n[2], ga.n[2], 1};
  int i[3];
  i[0] = (int)div_mod(div_mod(g, ga.n[2], i[2]), ga.n[1], i[1]);
  double d[3][NS];
#pragma unroll
  for (int v = 0; v < 3; ++v)
#pragma unroll
    for (int s = 0; s < NS; ++s) d[v][s] = axis_derivative<H>(ga, n_sg + s * ng + g, v, i[v], st[v]);
  double e;
  if constexpr (NS == 1) {
    const double sg = d[0][0] * d[0][0] + d[1][0] * d[1][0] + d[2][0] * d[2][0];
    double dv, ds;
    point_unpolarized(p, n_sg[g], sg, e, dv, ds);
    v_sg[g] += dv;
#pragma unroll
    for (int v = 0; v < 3; ++v) flux[v * ng + g] = 2.0 * ds * d[v][0];
  } else {
    double dv[2], ds[3];
    const double sg[3] = {d[0][0] * d[0][0] + d[1][0] * d[1][0] + d[2][0] * d[2][0],
                          d[0][0] * d[0][1] + d[1][0] * d[1][1] + d[2][0] * d[2][1],
                          d[0][1] * d[0][1] + d[1][1] * d[1][1] + d[2][1] * d[2][1]};
    point_polarized(p, n_sg[g], n_sg[ng + g], sg, e, dv, ds);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      v_sg[s * ng + g] += dv[s];
#pragma unroll
      for (int v = 0; v < 3; ++v)
        flux[(v * 2 + s) * ng + g] = 2.0 * ds[2 * s] * d[v][s] + ds[1] * d[v][1 - s];
    }
  }
  e_g[g] = e;
}

template <int H>
__global__ void __launch_bounds__(256) gga_divergence_kernel(const __grid_constant__ GradArgs ga, int64_t ng, int ns,
                                                             double* __restrict__ v_sg,
                                                             const double* __restrict__ flux) {
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (g >= ng) return;
  const int s = blockIdx.y;
  const int64_t st[3] = {(int64_t)ga.n[1] * ga.n[2], ga.n[2], 1};
  int i[3];
  i[0] = (int)div_mod(div_mod(g, ga.n[2], i[2]), ga.n[1], i[1]);
  double v = v_sg[s * ng + g];
#pragma unroll
  for (int c = 0; c < 3; ++c) v -= axis_derivative<H>(ga, flux + (c * ns + s) * ng + g, c, i[c], st[c]);
  v_sg[s * ng + g] = v;
}

static Par make_par(int code) {
  Par p{};
  p.gga = code != -1;
  p.rpbe = code == 2;
  p.kappa = code == 1 ? 1.245 : 0.804;
  p.mu = BETA * PI * PI / 3.0;
  p.C0I = 3.0 / (4.0 * PI);
  p.C1 = -9.0 / (8.0 * PI) * cbrt(2.0 * PI / 3.0);
  p.C2 = 1.0 / cbrt(18.0 * PI);
  p.C3 = PI * cbrt(4.0 / (9.0 * PI)) / 16.0;
  p.CC1 = 1.0 / (pow(2.0, 4.0 / 3.0) - 2.0);
  p.CC2 = 4.0 * p.CC1 / 3.0;
  // f''(0) = CC1 * (4/9) * 2 = 8 CC1 / 9
  p.IF2 = 9.0 / (8.0 * p.CC1);
  return p;
}

}  // namespace xc
}  // namespace gb

using namespace gb;

extern "C" int gb_xc_calculate(int code, int nspins, int64_t ng, double* e_g, const double* n_sg,
                               double* v_sg, const double* sigma_xg, double* dedsigma_xg,
                               void* stream) {
  GB_REQUIRE(code == -1 || code == 0 || code == 1 || code == 2,
             "gb_xc_calculate: code must be -1 (LDA), 0 (PBE), 1 (revPBE) or 2 (RPBE)");
  GB_REQUIRE(nspins == 1 || nspins == 2, "gb_xc_calculate: nspins must be 1 or 2");
  GB_REQUIRE(ng >= 0, "gb_xc_calculate: negative size");
  if (ng == 0) return GB_OK;
  GB_REQUIRE(e_g && n_sg && v_sg, "gb_xc_calculate: null array");
  GB_REQUIRE(code == -1 || (sigma_xg && dedsigma_xg), "gb_xc_calculate: GGA needs sigma and dedsigma");
  const xc::Par p = xc::make_par(code);
  const int threads = 256;
  const int64_t blocks = std::min<int64_t>((ng + threads - 1) / threads, (int64_t)sm_count() * 16);
  if (nspins == 1)
    xc::xc_unpolarized<<<(unsigned)blocks, threads, 0, (cudaStream_t)stream>>>(p, ng, e_g, n_sg, v_sg, sigma_xg,
                                                                              dedsigma_xg);
  else
    xc::xc_polarized<<<(unsigned)blocks, threads, 0, (cudaStream_t)stream>>>(p, ng, e_g, n_sg, v_sg, sigma_xg,
                                                                            dedsigma_xg);
  return check_launch("xc kernel");
}

extern "C" int gb_gga_calculate(int code, int nspins, const gb_operator* grad0, const gb_operator* grad1,
                                const gb_operator* grad2, double* e_g, const double* n_sg, double* v_sg,
                                double* flux, void* stream) {
  GB_REQUIRE(code == 0 || code == 1 || code == 2, "gb_gga_calculate: code must be 0 (PBE), 1 (revPBE) or 2 (RPBE)");
  GB_REQUIRE(nspins == 1 || nspins == 2, "gb_gga_calculate: nspins must be 1 or 2");
  GB_REQUIRE(grad0 && grad1 && grad2 && e_g && n_sg && v_sg && flux, "gb_gga_calculate: null pointer");
  const gb_operator* op[3] = {grad0, grad1, grad2};
  xc::GradArgs ga{};
  for (int c = 0; c < 3; ++c) {
    GB_REQUIRE(op[c]->real && op[c]->cfd && op[c]->H <= xc::GH, "gb_gga_calculate: gradients must be real, on the "
                                                               "axes and of radius at most 4");
    ga.H = std::max(ga.H, op[c]->H);
    ga.c0[c] = op[c]->center;
    for (int d = 0; d < 3; ++d) {
      GB_REQUIRE(op[c]->n[d] == op[0]->n[d] && op[c]->pbc[d] == op[0]->pbc[d],
                 "gb_gga_calculate: the gradients are on different grids");
      for (int m = 0; m < 2 * HMAX + 1; ++m)
        GB_REQUIRE(d == c || op[c]->a[d][m] == 0.0, "gb_gga_calculate: gradient c must lie along axis c");
    }
    ga.n[c] = (int)op[0]->n[c];
    ga.pbc[c] = op[0]->pbc[c];
    for (int m = -xc::GH; m <= xc::GH; ++m) ga.a[c][m + xc::GH] = op[c]->a[c][m + HMAX];
  }
  for (int c = 0; c < 3; ++c) GB_REQUIRE(ga.H <= ga.n[c], "gb_gga_calculate: stencil longer than domain");
  const int64_t ng = op[0]->n[0] * op[0]->n[1] * op[0]->n[2];
  const xc::Par p = xc::make_par(code);
  const unsigned blocks = (unsigned)((ng + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
#define GB_GGA(HH)                                                                                              \
  case HH:                                                                                                      \
    if (nspins == 1) xc::gga_flux_kernel<1, HH><<<blocks, 256, 0, st>>>(p, ga, ng, e_g, n_sg, v_sg, flux);     \
    else xc::gga_flux_kernel<2, HH><<<blocks, 256, 0, st>>>(p, ga, ng, e_g, n_sg, v_sg, flux);                 \
    xc::gga_divergence_kernel<HH><<<dim3(blocks, (unsigned)nspins), 256, 0, st>>>(ga, ng, nspins, v_sg, flux); \
    break
  switch (ga.H) {
    GB_GGA(1);
    GB_GGA(2);
    GB_GGA(3);
    GB_GGA(4);
  }
#undef GB_GGA
  return check_launch("gga_flux_kernel / gga_divergence_kernel");
}
