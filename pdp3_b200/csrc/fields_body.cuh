// Per-node Yee updates of the axisymmetric (r, phi, z) grid, shared by the
// per-run kernels (fields.cu) and the ensemble's persistent kernel.
//
// Every operation is the upstream one, correctly rounded and in its order; a
// division by a value that many nodes share is a quotient by that value's
// reciprocal (the library division is ten times its instructions) wherever
// that is the same.
#pragma once

#include "pdp3g_internal.cuh"

namespace pdp3g {

#define FIDX(i, k) ((size_t)(i) * (size_t)nz + (size_t)(k))

// The divisions of a node: quotient, and whether a dividend was one it does not
// serve (neither +0, which a fresh grid is full of, nor within 2^-960 to
// 2^960: the tail of a pulse, an unstable run's infinities).
struct Quotients {
  bool odd = false;
  __device__ __forceinline__ double operator()(double a, double b, double y) {
    const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
    odd |= ((hi & 0x7fffffffu) - 0x03f00000u > 0x78000000u) & ((hi | lo) != 0u);
    return quotient(a, b, y);
  }
};
// the division itself
struct Divisions {
  static constexpr bool odd = false;
  __device__ __forceinline__ double operator()(double a, double b, double) {
    return quotient_edge(a, b);
  }
};

// HField::calc_field, src/hField.cpp:93-157, node (i, k) with
// i in [0, nr-1], k in [0, nz-2]: H_r for every i, H_phi and H_z for
// i <= nr-2.  H_half = H_old + dH/2 (H_z: H_old - dH/2, upstream convention).
// False, and nothing written, if div met a dividend that it does not serve.
// The old values are read before that test, which no load would pass (65 x 257
// nodes, FP32 contexts: E update 4.8 -> 3.9 us).
template <class DIV>
__device__ __forceinline__ bool h_node(const GridDev &g, DIV div, int i, int k) {
  const int nr = g.nr, nz = g.nz;
  const double dr = g.dr, dz = g.dz, dt = g.dt;
  constexpr double inv_mu = 1.0 / MAGN_CONST;
  const double ephi_ik = g.ephi[FIDX(i, k)];
  const double ephi_ik1 = g.ephi[FIDX(i, k + 1)];
  const bool inside = i < nr - 1;
  const double a = div(dt * (ephi_ik1 - ephi_ik), dz * MAGN_CONST, g.inv_dzmu);
  const double hr = g.hr[FIDX(i, k)];
  double b = 0.0, c = 0.0, hphi = 0.0, hz = 0.0;
  if (inside) {
    hphi = g.hphi[FIDX(i, k)];
    hz = g.hz[FIDX(i, k)];
    b = div(dt * (div(g.ez[FIDX(i + 1, k)] - g.ez[FIDX(i, k)], dr, g.inv_dr) -
                  div(g.er[FIDX(i, k + 1)] - g.er[FIDX(i, k)], dz, g.inv_dz)),
            MAGN_CONST, inv_mu);
    const double ephi_i1k = g.ephi[FIDX(i + 1, k)];
    const double d2 = 2.0 * dr * (i + 0.5);
    c = div(dt * (div(ephi_i1k + ephi_ik, d2, rcp_ulp(d2)) +
                  div(ephi_i1k - ephi_ik, dr, g.inv_dr)),
            MAGN_CONST, inv_mu);
  }
  if (div.odd) return false;
  const size_t ng = (size_t)nr * nz;
  const double hrh = hr + a / 2;
  g.hrh[FIDX(i, k)] = hrh;
  if (g.hh32) g.hh32[FIDX(i, k)] = (float)hrh;
  g.hr[FIDX(i, k)] = hr + a;
  if (inside) {
    const double hphih = hphi + b / 2;
    g.hphih[FIDX(i, k)] = hphih;
    if (g.hh32) g.hh32[ng + FIDX(i, k)] = (float)hphih;
    g.hphi[FIDX(i, k)] = hphi + b;
    const double hzh = hz - c / 2;
    g.hzh[FIDX(i, k)] = hzh;
    if (g.hh32) g.hh32[2 * ng + FIDX(i, k)] = (float)hzh;
    g.hz[FIDX(i, k)] = hz - c;
  }
  return true;
}

// EField::calc_field, src/eField.cpp:85-170 (epsilon == 1), node (i, k)
// with i in [0, nr-2], k in [0, nz-2] and the currents there:
//   E_r   i in [0, nr-2], k in [1, nz-2]
//   E_phi i in [1, nr-2], k in [1, nz-2]
//   E_z   i = 0 (on-axis form, 4/dr * H_phi), k in [0, nz-2];
//         i in [1, nr-2], k in [0, nz-2] (interior form, also the k = 0 row)
// False as h_node.
template <class DIV>
__device__ __forceinline__ bool e_node(const GridDev &g, DIV div, int i, int k, double jr,
                                       double jphi, double jz) {
  const int nz = g.nz;
  const double dr = g.dr, dz = g.dz, dt = g.dt;
  const double epsx2 = 2 * 1.0 * EPSILON0;
  const double sigma_t = g.sigma[FIDX(i, k)] * dt;
  const double den = epsx2 + sigma_t, inv_den = rcp_ulp(den);
  const double koef_e = quotient(epsx2 - sigma_t, den, inv_den);
  const double koef_h = quotient(2 * dt, den, inv_den);
  const double hphi_ik = g.hphi[FIDX(i, k)], ez = g.ez[FIDX(i, k)];
  double r = 0.0, z, phi = 0.0, er = 0.0, ephi = 0.0;
  if (k >= 1) {
    er = g.er[FIDX(i, k)];
    r = jr + div(hphi_ik - g.hphi[FIDX(i, k - 1)], dz, g.inv_dz);
  }
  if (i == 0) {
    z = jz - quotient(4.0, dr, g.inv_dr) * hphi_ik;
  } else {
    const double hphi_m = g.hphi[FIDX(i - 1, k)];
    const double d2 = 2.0 * dr * i;
    z = jz - div(hphi_ik - hphi_m, dr, g.inv_dr) - div(hphi_ik + hphi_m, d2, rcp_ulp(d2));
    if (k >= 1) {
      ephi = g.ephi[FIDX(i, k)];
      phi = jphi - div(g.hr[FIDX(i, k)] - g.hr[FIDX(i, k - 1)], dz, g.inv_dz) +
            div(g.hz[FIDX(i, k)] - g.hz[FIDX(i - 1, k)], dr, g.inv_dr);
    }
  }
  if (div.odd) return false;
  const size_t ng = (size_t)g.nr * nz;
  if (k >= 1) {
    const double v = er * koef_e - r * koef_h;
    g.er[FIDX(i, k)] = v;
    if (g.e32) g.e32[FIDX(i, k)] = (float)v;
  }
  const double v = ez * koef_e - z * koef_h;
  g.ez[FIDX(i, k)] = v;
  if (g.e32) g.e32[2 * ng + FIDX(i, k)] = (float)v;
  if (i >= 1 && k >= 1) {
    const double w = ephi * koef_e - phi * koef_h;
    g.ephi[FIDX(i, k)] = w;
    if (g.e32) g.e32[ng + FIDX(i, k)] = (float)w;
  }
  return true;
}

// The rare nodes go out of line as a whole: a branch at every division would
// stand in the chain that the update waits for (4096-particle step, 17 x 33
// nodes: 15.4 us with div_rn at each, 14.4 so).
static __device__ __noinline__ void h_node_exact(const GridDev &g, int i, int k) {
  h_node(g, Divisions{}, i, k);
}
static __device__ __noinline__ void e_node_exact(const GridDev &g, int i, int k, double jr,
                                                 double jphi, double jz) {
  e_node(g, Divisions{}, i, k, jr, jphi, jz);
}
__device__ __forceinline__ void yee_h_node(const GridDev &g, int i, int k) {
  if (!h_node(g, Quotients{}, i, k)) h_node_exact(g, i, k);
}
__device__ __forceinline__ void yee_e_node(const GridDev &g, int i, int k, double jr, double jphi,
                                           double jz) {
  if (!e_node(g, Quotients{}, i, k, jr, jphi, jz)) e_node_exact(g, i, k, jr, jphi, jz);
}

#undef FIDX

}  // namespace pdp3g
