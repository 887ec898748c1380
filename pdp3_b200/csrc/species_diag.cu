// The per-species diagnostics of LoadInitParam::dump_data on the device.
//
// TemperatureClassic (src/temperatureClassic.cpp:57-159): per cell
// (CELL_NUMBER of r and z) the sums of |v|, v_r, v_phi, v_z and the particle
// count, then T = m v_sc^2 / 2 with v_sc^2 = ((sum |v|)^2 - |sum v|^2) /
// count^2 (relativistic m c^2 (gamma - 1) at v_sc > 5e7 m/s), in
// electronvolts; empty cells give NaN (0/0), as upstream.
//
// ParticlesDensity (src/particlesDensity.cpp:45-257) and charge_weighting
// (src/particles.cpp:101-226): each particle's mass_array / EL_MASS or charge
// spread over the four nodes around it by ring-piece volumes.
//
// Compiled with --fmad=false: cell numbers, velocities and the temperature's
// per-cell arithmetic are rounded as upstream; the ring pieces are formed in
// cell units; sums run over a lane's particles, a warp's lanes and FP64 atomics.
#include "pdp3g_internal.cuh"

namespace pdp3g {

constexpr double REL_LIMIT = 5e7;  // src/temperatureClassic.cpp:4-6

// threads per CTA; CTAs per SM (the temperature's kernels, of 76 registers: 3)
constexpr int DIAG_THREADS = 256, DIAG_BLOCKS = 4;
constexpr int PER_LANE = 4;                         // consecutive particles of a lane

// The per-particle passes below read 16 to 40 bytes of a particle and add a
// few FP64 sums per cell; with one particle per lane and the library's
// divisions they were bound by the FP64 pipe and by the warp sums.  Here a
// lane takes four consecutive particles (16-byte loads of each array), adds
// up those that share a cell, and only then joins the warp's sum over runs
// of lanes and the atomics: a quarter of the shuffles, and the factors that
// depend on the cell alone are applied once per run.  33.5M sorted particles
// on 257 x 2049 nodes, FP32 form: charge and density 186 and 179 us (604 and
// 630 before; 83 us at the copy rate), temperature 314 us (570 before); 118
// instructions a particle keep the issue slots 68% busy.

// the species getter's r = (cell + f) d and its CELL_NUMBER, ceil(r / d) - 1.
// Away from the cell's ends that is the cell itself: the two roundings move
// r / d by less than 3 x 2^-53 x 2^20 < 4e-10 cells, and a float below 1 is
// at most 1 - 6e-8.
__device__ __forceinline__ int getter_cell(int cell, float f, double d) {
  if (f > 1e-9f && f < 1.0f && cell < (1 << 20)) return cell;
  const double x = (cell + (double)f) * d;
  return (int)ceil(x / d) - 1;
}

// x / d, inv = 1 / d: correctly rounded for a position that may lie in a cell;
// another one, infinite or not a number included, only has to stay so
__device__ __forceinline__ double in_cells(double x, double d, double inv) {
  return near_f64(x) ? quotient(x, d, inv) : x * inv;
}

// Sums of N values over a lane's consecutive particles of one cell; a change
// of cell gives the finished run to flush(key, v).
template <int N>
struct LaneRun {
  int key = -1;
  double v[N];
  template <class F>
  __device__ __forceinline__ void start(int k, F &&flush) {
    if (k == key) return;
    if (key >= 0) flush(key, v);
    key = k;
#pragma unroll
    for (int j = 0; j < N; j++) v[j] = 0.0;
  }
  // every lane of the warp calls it
  template <class F>
  __device__ __forceinline__ void finish(F &&flush) {
    if (key < 0) {
#pragma unroll
      for (int j = 0; j < N; j++) v[j] = 0.0;
    }
    if (warp_run_sum_f64<N>(key, v) && key >= 0) flush(key, v);
  }
};

// four consecutive values from p on, those below n (the rest 0)
template <class T4, class T>
__device__ __forceinline__ void load4(const T *a, long long p, long long n, T (&out)[PER_LANE]) {
  if (p + PER_LANE <= n) {
    const T4 q = *reinterpret_cast<const T4 *>(a + p);
    out[0] = q.x;
    out[1] = q.y;
    out[2] = q.z;
    out[3] = q.w;
  } else {
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) out[j] = p + j < n ? a[p + j] : T(0);
  }
}

__device__ __forceinline__ void load4(const double *a, long long p, long long n,
                                      double (&out)[PER_LANE]) {
  if (p + PER_LANE <= n) {
    const double2 q0 = *reinterpret_cast<const double2 *>(a + p);
    const double2 q1 = *reinterpret_cast<const double2 *>(a + p + 2);
    out[0] = q0.x;
    out[1] = q0.y;
    out[2] = q1.x;
    out[3] = q1.y;
  } else {
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) out[j] = p + j < n ? a[p + j] : 0.0;
  }
}

// the loops run whole warps (every lane takes part in the warp sums): p is
// the first of this lane's particles
#define PDP3G_LANE_LOOP(p, n)                                                                 \
  for (long long p = (blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31)) * PER_LANE,   \
                 p##_end = (n), p##_stride = (long long)gridDim.x * blockDim.x * PER_LANE;    \
       p < p##_end; p += p##_stride)

// ---- temperature -----------------------------------------------------------
// acc: 5 grids [nr][nz]: sum |v|, sum v_r, sum v_phi, sum v_z, count.  A cell
// outside the grid adds nothing.  Cell numbers, velocities and |v| are
// rounded as the upstream expressions round them.

struct TempFlush {
  double *acc;
  size_t ng;
  __device__ __forceinline__ void operator()(int key, const double *v) const {
#pragma unroll
    for (int j = 0; j < 5; j++) atomicAdd(acc + j * ng + key, v[j]);
  }
};

__device__ __forceinline__ void temp_add(const GridDev &g, LaneRun<5> &run, const TempFlush &flush,
                                         int ri, int zk, double vr, double vphi, double vz) {
  if ((unsigned)ri >= (unsigned)g.nr || (unsigned)zk >= (unsigned)g.nz) return;
  run.start(ri * g.nz + zk, flush);
  const double v2 = vr * vr + vphi * vphi + vz * vz;
  run.v[0] += v2 > 1e-290 && v2 < 1e290 ? sqrt_rn(v2, rsqrt_ulp(v2)) : sqrt(v2);
  run.v[1] += vr;
  run.v[2] += vphi;
  run.v[3] += vz;
  run.v[4] += 1.0;
}

__global__ void __launch_bounds__(DIAG_THREADS, 3)
    k_temp_accum_f64(GridDev g, SpeciesDev s, double *acc) {
  const TempFlush flush{acc, (size_t)g.nr * g.nz};
  PDP3G_LANE_LOOP(w0, s.n) {
    const long long p = w0 + (threadIdx.x & 31) * PER_LANE;
    double r[PER_LANE], z[PER_LANE], vr[PER_LANE], vphi[PER_LANE], vz[PER_LANE];
    load4(s.r, p, s.n, r);
    load4(s.z, p, s.n, z);
    load4(s.vr, p, s.n, vr);
    load4(s.vphi, p, s.n, vphi);
    load4(s.vz, p, s.n, vz);
    LaneRun<5> run;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++)
      if (p + j < s.n)
        temp_add(g, run, flush, (int)ceil(in_cells(r[j], g.dr, g.inv_dr)) - 1,
                 (int)ceil(in_cells(z[j], g.dz, g.inv_dz)) - 1, vr[j], vphi[j], vz[j]);
    run.finish(flush);
  }
}

// the cell-local form, read as FP64 r, z, v exactly as the species getter
// does (r = (i + f_r) dr, v = u c / sqrt(1 + u^2)), then CELL_NUMBER as above
__global__ void __launch_bounds__(DIAG_THREADS, 3)
    k_temp_accum_f32(GridDev g, SpeciesF32 s, double *acc) {
  const TempFlush flush{acc, (size_t)g.nr * g.nz};
  PDP3G_LANE_LOOP(w0, s.n) {
    const long long p = w0 + (threadIdx.x & 31) * PER_LANE;
    int c[PER_LANE];
    float fr[PER_LANE], fz[PER_LANE], u[3][PER_LANE];
    load4<int4>(s.cell, p, s.n, c);
    load4<float4>(s.fr, p, s.n, fr);
    load4<float4>(s.fz, p, s.n, fz);
    load4<float4>(s.ur, p, s.n, u[0]);
    load4<float4>(s.uphi, p, s.n, u[1]);
    load4<float4>(s.uz, p, s.n, u[2]);
    LaneRun<5> run;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) {
      if (p + j >= s.n) continue;
      const int i = row_of(g, c[j]), k = c[j] - i * (g.nz - 1);
      const double ur = u[0][j], up = u[1][j], uz = u[2][j];
      const double x = 1.0 + (ur * ur + up * up + uz * uz);
      const double root = sqrt_rn(x, rsqrt_ulp(x));
      const double gc = quotient(LIGHT_SPEED, root, rcp_ulp(root));
      temp_add(g, run, flush, getter_cell(i, fr[j], g.dr), getter_cell(k, fz[j], g.dz), ur * gc,
               up * gc, uz * gc);
    }
    run.finish(flush);
  }
}

// TemperatureClassic::normalize over r < nr-1, z < nz-1 (others left 0)
__global__ void k_temp_normalize(GridDev g, const double *acc, double mass, double charge,
                                 double *t_out) {
  const int nr = g.nr, nz = g.nz;
  const size_t ng = (size_t)nr * nz;
  const long long total = (long long)(nr - 1) * (nz - 1);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(q / (nz - 1)), z = (int)(q - (long long)r * (nz - 1));
    const size_t t = (size_t)r * nz + z;
    const double sum = acc[t], vr = acc[ng + t], vp = acc[2 * ng + t], vz = acc[3 * ng + t];
    const double cnt = acc[4 * ng + t];
    const double v_vec_sum_2 = vr * vr + vp * vp + vz * vz;
    const double v_sc_sum_2 = (sum * sum - v_vec_sum_2) / (cnt * cnt);
    double tv;
    if (v_sc_sum_2 < REL_LIMIT * REL_LIMIT) {
      tv = mass * v_sc_sum_2 / 2;
    } else {
      // lib::get_gamma (src/lib.cpp:45-70): beta == 1 gives 1e100; beta > 1
      // is an upstream exit, gamma 1 here
      const double beta = v_sc_sum_2 / LIGHT_SPEED_POW_2;
      double gamma = beta > 1 ? 1.0 : 1 / sqrt(1.0 - beta);
      if (isinf(gamma)) gamma = 1e100;
      tv = mass * LIGHT_SPEED_POW_2 * (gamma - 1);
    }
    t_out[t] = tv / fabs(charge);
  }
}

// ---- ring-piece weighting --------------------------------------------------
// Particles::charge_weighting (src/particles.cpp:101-226) and
// ParticlesDensity::calc_density (src/particlesDensity.cpp:45-257) spread a
// particle over the four nodes around it by the volumes of ring pieces.  With
// x = r / dr = i + f and z / dz = k + h the upstream expressions are, per
// unit of the particle's value,
//   node (i,   .): (1 - f)(2 i + f) / (2 x) / V_i
//   node (i+1, .): f (2 i + 1 + f) / (2 x)  / V_(i+1)
// times 1 - h (node k) or h (node k + 1), V_i = 2 PI dz dr^2 i, and a quarter
// of PI dz dr^2 on the axis; for x <= 1/2 (then i = 0) the first numerator is
// f^2 - f + 1/2 and both denominators 2 f^2 + 1/2.  The three branches agree
// where they meet, and no difference of squared radii is formed.  V_i is
// applied once per run of particles in a cell.

// values of CHARGE outside the grid raise ERR_OUT_OF_GRID; the density skips
// them, as upstream's bounds test does
template <bool CHARGE>
__device__ __forceinline__ void ring_nodes(const GridDev &g, double *out, double scale, int i,
                                           int k, const double *v) {
  const double a = i == 0 ? 8.0 * scale : scale * rcp_ulp((double)i);
  const double b = scale * rcp_ulp(i + 1.0);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int ii = i + (j & 1), kk = k + (j >> 1);
    if ((unsigned)ii < (unsigned)g.nr && (unsigned)kk < (unsigned)g.nz)
      atomicAdd(out + (size_t)ii * g.nz + kk, v[j] * ((j & 1) ? b : a));
    else if (CHARGE)
      atomicOr(g.err, ERR_OUT_OF_GRID);
  }
}

template <bool CHARGE>
struct RingFlush {
  const GridDev &g;
  double *out, scale;
  __device__ __forceinline__ void operator()(int key, const double *v) const {
    const int i = row_of(g, key);
    ring_nodes<CHARGE>(g, out, scale, i, key - i * (g.nz - 1), v);
  }
};

// one particle of weight w at x = i + f, z / dz = k + h
template <bool CHARGE>
__device__ __forceinline__ void ring_add(const GridDev &g, LaneRun<4> &run,
                                         const RingFlush<CHARGE> &flush, int i, int k, double f,
                                         double h, double w) {
  const double x = i + f;
  double num0 = (1.0 - f) * (x + i), den = x + x;
  const double num1 = f * (x + i + 1.0);
  if (x <= 0.5) {
    num0 = fma(f, f, 0.5 - f);
    den = fma(2.0 * f, f, 0.5);
  }
  const double q = w * rcp_ulp(den), g0 = q * num0, g1 = q * num1, h1 = 1.0 - h;
  if ((unsigned)i < (unsigned)(g.nr - 1) && (unsigned)k < (unsigned)(g.nz - 1)) {
    run.start(i * (g.nz - 1) + k, flush);
    run.v[0] = fma(g0, h1, run.v[0]);
    run.v[1] = fma(g1, h1, run.v[1]);
    run.v[2] = fma(g0, h, run.v[2]);
    run.v[3] = fma(g1, h, run.v[3]);
  } else {
    const double v[4] = {g0 * h1, g1 * h1, g0 * h, g1 * h};
    ring_nodes<CHARGE>(g, flush.out, flush.scale, i, k, v);
  }
}

// scale: the species' factor (charge, or mass / EL_MASS) over 2 PI dz dr^2
template <bool CHARGE>
__global__ void __launch_bounds__(DIAG_THREADS, DIAG_BLOCKS)
    k_ring_f64(GridDev g, SpeciesDev s, double scale, double *out) {
  const RingFlush<CHARGE> flush{g, out, scale};
  PDP3G_LANE_LOOP(w0, s.n) {
    const long long p = w0 + (threadIdx.x & 31) * PER_LANE;
    double r[PER_LANE], z[PER_LANE], w[PER_LANE];
    load4(s.r, p, s.n, r);
    load4(s.z, p, s.n, z);
    load4(s.w, p, s.n, w);
    LaneRun<4> run;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) {
      if (p + j >= s.n || (CHARGE && s.alive != nullptr && !s.alive[p + j])) continue;
      if (CHARGE && !(isfinite(r[j]) && isfinite(z[j]))) {
        atomicOr(g.err, ERR_NAN);
        continue;
      }
      const double x = in_cells(r[j], g.dr, g.inv_dr), y = in_cells(z[j], g.dz, g.inv_dz);
      int i = (int)ceil(x) - 1, k = (int)ceil(y) - 1;
      if (x <= 0.5) i = 0;
      if (CHARGE) {
        i = max(i, 0);
        k = max(k, 0);
      }
      ring_add(g, run, flush, i, k, x - i, y - k, w[j]);
    }
    run.finish(flush);
  }
}

// the cell-local form: the cell and the offsets are x and z / dz already (a
// particle on the face of its cell weighs the same from either side)
template <bool CHARGE>
__global__ void __launch_bounds__(DIAG_THREADS, DIAG_BLOCKS)
    k_ring_f32(GridDev g, SpeciesF32 s, double scale, double *out) {
  const RingFlush<CHARGE> flush{g, out, scale};
  PDP3G_LANE_LOOP(w0, s.n) {
    const long long p = w0 + (threadIdx.x & 31) * PER_LANE;
    int c[PER_LANE];
    float fr[PER_LANE], fz[PER_LANE], w[PER_LANE];
    load4<int4>(s.cell, p, s.n, c);
    load4<float4>(s.fr, p, s.n, fr);
    load4<float4>(s.fz, p, s.n, fz);
    load4<float4>(s.w, p, s.n, w);
    LaneRun<4> run;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) {
      if (p + j >= s.n || (CHARGE && s.alive != nullptr && !s.alive[p + j])) continue;
      const int i = row_of(g, c[j]);
      ring_add(g, run, flush, i, c[j] - i * (g.nz - 1), fr[j], fz[j], w[j]);
    }
    run.finish(flush);
  }
}

static int blocks_of(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 8) b = 148 * 8;
  return (int)(b < 1 ? 1 : b);
}

// CTAs of a pass over n particles: at most four per SM, which for the ring
// kernels is one resident set; of the temperature's kernels three are resident,
// and the rest follows in a second, partial round
static int lane_blocks(long long n) {
  const long long per = (long long)DIAG_THREADS * PER_LANE, b = (n + per - 1) / per;
  return (int)(b > 148 * DIAG_BLOCKS ? 148 * DIAG_BLOCKS : b);
}

void launch_temperature_f64(const GridDev &g, const SpeciesDev &s, double *acc, cudaStream_t st) {
  if (s.n > 0) k_temp_accum_f64<<<lane_blocks(s.n), DIAG_THREADS, 0, st>>>(g, s, acc);
}

void launch_temperature_f32(const GridDev &g, const SpeciesF32 &s, double *acc, cudaStream_t st) {
  if (s.n > 0) k_temp_accum_f32<<<lane_blocks(s.n), DIAG_THREADS, 0, st>>>(g, s, acc);
}

void launch_temperature_normalize(const GridDev &g, const double *acc, double mass, double charge,
                                  double *t_out, cudaStream_t st) {
  k_temp_normalize<<<blocks_of((long long)(g.nr - 1) * (g.nz - 1)), 256, 0, st>>>(g, acc, mass,
                                                                                 charge, t_out);
}

static double ring_scale(const GridDev &g, double value) {
  return value / (2. * PI * g.dz * g.dr * g.dr);
}

void launch_charge_density_f64(const GridDev &g, const SpeciesDev &s, double *rho,
                               cudaStream_t st) {
  if (s.n > 0)
    k_ring_f64<true><<<lane_blocks(s.n), DIAG_THREADS, 0, st>>>(g, s, ring_scale(g, s.charge),
                                                                rho);
}

void launch_charge_density_f32(const GridDev &g, const SpeciesF32 &s, double charge, double *rho,
                               cudaStream_t st) {
  if (s.n > 0)
    k_ring_f32<true><<<lane_blocks(s.n), DIAG_THREADS, 0, st>>>(g, s, ring_scale(g, charge), rho);
}

void launch_density_f64(const GridDev &g, const SpeciesDev &s, double *out, cudaStream_t st) {
  if (s.n > 0)
    k_ring_f64<false><<<lane_blocks(s.n), DIAG_THREADS, 0, st>>>(
        g, s, ring_scale(g, s.mass / EL_MASS), out);
}

void launch_density_f32(const GridDev &g, const SpeciesF32 &s, double mass, double *out,
                        cudaStream_t st) {
  if (s.n > 0)
    k_ring_f32<false><<<lane_blocks(s.n), DIAG_THREADS, 0, st>>>(
        g, s, ring_scale(g, mass / EL_MASS), out);
}

}  // namespace pdp3g
