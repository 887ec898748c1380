// Initial electrostatic field: PoissonDirichlet::poisson_solve
// (src/poissonDirichlet.cpp:23-98) on the device.
//
//   1. every radial row of rho gets a sine transform along z
//      (Fourier::fast_sine_transform, src/math/fourier.cpp:17-51: the odd
//      extension of length 2 n_grid_z + 2 through the radix-2 FFT of
//      Fourier::fast_fourier_alg, :93-142), one CTA per row in shared memory;
//   2. per axial mode k, the radial three-point equation is swept (the
//      upstream's alpha/beta recurrence and back substitution, one thread
//      per k; the mode constant b is evaluated on the host with its libm);
//   3. the inverse sine transform of every row of phi;
//   4. E_r = (phi_i - phi_i+1) / dr, E_z = (phi_k - phi_k+1) / dz.
//
// Compiled with --fmad=false: every step keeps the upstream's operation
// order; the FFT's twiddle factors come from CUDA's sin/cos instead of the
// host libm, so phi and E agree with the upstream's to rounding (about
// 1e-13 relative), not bit for bit.
#include "pdp3g_internal.cuh"

namespace pdp3g {

constexpr int DST_THREADS = 512;
constexpr int DST_MAX_LEN = 8192;  // 2 n_grid_z + 2: 182 KB of shared memory

// W = exp(i (-PI 2 k) / (2 n_step)) of every butterfly, as (cos, sin): entry
// k (len / 2 / n_step).  The angle of an entry is the same double whichever
// n_step asks for it (they differ by powers of two), so one table of the last
// stage serves all.
__global__ void k_twiddles(double2 *w, int half) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= half) return;
  double ws, wc;
  sincos(-PI * (double)2.0 * k / (half * 2), &ws, &wc);
  w[k] = make_double2(wc, ws);
}

// one unused slot in eight (data) or sixteen (row) keeps the strided accesses
// off one bank
__device__ __forceinline__ int pad8(int m) { return m + (m >> 3); }
__device__ __forceinline__ int pad16(int m) { return m + (m >> 4); }

// R butterfly stages (n_step, 2 n_step, ..) of the 2^R elements x, whose
// first has the in-block index k
template <int R>
__device__ __forceinline__ void butterflies(double2 (&x)[1 << R], const double2 *w, int half,
                                            int log2_step, int k) {
#pragma unroll
  for (int s = 0; s < R; s++) {
    double2 t[1 << (R - 1)];  // twiddles of this stage
#pragma unroll
    for (int j = 0; j < (1 << s); j++)
      t[j] = __ldg(w + (size_t)(k + (j << log2_step)) * (half >> (log2_step + s)));
#pragma unroll
    for (int j = 0; j < (1 << R); j++) {
      if (j & (1 << s)) continue;
      const double2 c = t[j & ((1 << s) - 1)], a = x[j], v = x[j | (1 << s)];
      // W * v as the complex product (a + bi)(c + di) = (ac - bd) + (ad + bc)i
      const double tr = c.x * v.x - c.y * v.y, ti = c.x * v.y + c.y * v.x;
      x[j] = make_double2(a.x + tr, a.y + ti);
      x[j | (1 << s)] = make_double2(a.x - tr, a.y - ti);
    }
  }
}

template <int R>
__device__ __forceinline__ void butterfly_pass(double2 *sh, const double2 *w, int len,
                                               int log2_step) {
  for (int q = threadIdx.x; q < (len >> R); q += blockDim.x) {
    const int k = q & ((1 << log2_step) - 1);
    const int base = ((q >> log2_step) << (log2_step + R)) + k;
    double2 x[1 << R];
#pragma unroll
    for (int j = 0; j < (1 << R); j++) x[j] = sh[pad8(base + (j << log2_step))];
    butterflies<R>(x, w, len / 2, log2_step, k);
#pragma unroll
    for (int j = 0; j < (1 << R); j++) sh[pad8(base + (j << log2_step))] = x[j];
  }
  __syncthreads();
}

// the transform of a row of in ([nr][nz]) into the same row of out.  Bound by
// shared memory: three radix-2 stages are made in registers per trip (four
// trips of a 4096-point row instead of twelve), the bit reversal and the odd
// extension happen on the first load, the twiddles come from a table: 257
// rows of 2047 nodes in 23 us (67 with a trip and a sincos per stage).
__global__ void __launch_bounds__(DST_THREADS) k_sine_transform(const double *in, double *out,
                                                                const double2 *w, int nz, int len,
                                                                int log2_len, bool inverse) {
  extern __shared__ double2 sh[];
  double *line = reinterpret_cast<double *>(sh + pad8(len));
  const size_t row = (size_t)blockIdx.x * nz;
  for (int k = threadIdx.x; k < nz; k += blockDim.x) line[pad16(k)] = in[row + k];
  __syncthreads();
  // a_sinc: 0 at 0 and nz + 1, a[k] at k + 1, -a[k] at 2 nz - k + 1, taken in
  // bit-reversed order; then the stages n_step = 1, 2, 4
  for (int q = threadIdx.x; q < (len >> 3); q += blockDim.x) {
    double2 x[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int m = (int)(__brev((unsigned)(8 * q + j)) >> (32 - log2_len));
      double v = 0.0;
      if (m >= 1 && m <= nz) v = line[pad16(m - 1)];
      if (m >= nz + 2) v = -line[pad16(2 * nz + 1 - m)];
      x[j] = make_double2(v, 0.0);
    }
    butterflies<3>(x, w, len / 2, 0, 0);
#pragma unroll
    for (int j = 0; j < 8; j++) sh[pad8(8 * q + j)] = x[j];
  }
  __syncthreads();
  int done = 3;
  for (; done + 3 <= log2_len; done += 3) butterfly_pass<3>(sh, w, len, done);
  if (log2_len - done == 2) butterfly_pass<2>(sh, w, len, done);
  if (log2_len - done == 1) butterfly_pass<1>(sh, w, len, done);
  // a[k] = real(-1 / (2i) * a_sinc[k + 1]) = real((0 + 0.5i) * a_sinc[k + 1])
  for (int k = threadIdx.x; k < nz; k += blockDim.x) {
    const double2 x = sh[pad8(k + 1)];
    double v = 0.0 * x.x - 0.5 * x.y;
    if (inverse) v = v * 2.0 / (nz + 1);
    out[row + k] = v;
  }
}

// the radial sweep of mode k (one thread per k); alpha, beta: [nr][nz]
// scratch; fi[nr-1][k] is the boundary value (set_fi_on_z: 0).  A serial
// chain of nr steps per mode: what counts is a step's latency.  Rows are read
// SWEEP_AHEAD at a time, and the chain carries one reciprocal and its exact
// quotient (rcp_ulp, quotient) instead of two divisions: 257 rows of 2047 modes
// in 37 us (249 before; 47 with batches of 8 rows).  beta's dividend may leave
// quotient's range in rows far from any charge (2 ulps of a value below 1e-280
// there; testing it in the chain costs 26 us) or for charges above 1e280.
constexpr int SWEEP_AHEAD = 16, SWEEP_THREADS = 32;

__global__ void __launch_bounds__(SWEEP_THREADS)
    k_poisson_sweep(const double *__restrict__ t, const double *__restrict__ b_mode,
                    double *__restrict__ fi, double *__restrict__ alpha,
                    double *__restrict__ beta, int nr, int nz, double dr) {
  const int k = blockIdx.x * SWEEP_THREADS + threadIdx.x;
  if (k >= nz) return;
  const double b = b_mode[k], dr2 = dr * dr;
  double al = 4. / (2. + b), be = dr2 * t[k] / EPSILON0 / (2. + b);
  alpha[(size_t)nz + k] = al;
  beta[(size_t)nz + k] = be;
  // rows past the last are read as the last and their results dropped, so
  // that a whole batch is one straight run of code
  const int last = nr - 2;
  double next[SWEEP_AHEAD];
#pragma unroll
  for (int j = 0; j < SWEEP_AHEAD; j++) next[j] = t[(size_t)min(1 + j, last) * nz + k];
  for (int i0 = 1; i0 <= last; i0 += SWEEP_AHEAD) {
    double a[SWEEP_AHEAD], c[SWEEP_AHEAD], d[SWEEP_AHEAD];
#pragma unroll
    for (int j = 0; j < SWEEP_AHEAD; j++) {
      const double two_i = 2. * (i0 + j), h = quotient(1., two_i, rcp_ulp(two_i));
      a[j] = 1. - h;
      c[j] = 1. + h;
      d[j] = quotient(dr2 * next[j], EPSILON0, 1. / EPSILON0);
      next[j] = t[(size_t)min(i0 + SWEEP_AHEAD + j, last) * nz + k];
    }
#pragma unroll
    for (int j = 0; j < SWEEP_AHEAD; j++) {
      const double den = b - al * a[j], y = rcp_ulp(den);
      be = quotient(d[j] + be * a[j], den, y);
      al = quotient(c[j], den, y);
      if (i0 + j <= last) {
        alpha[(size_t)(i0 + j + 1) * nz + k] = al;
        beta[(size_t)(i0 + j + 1) * nz + k] = be;
      }
    }
  }
  // back from the last row, by the same batches
  double f = fi[(size_t)(nr - 1) * nz + k], av[SWEEP_AHEAD], bv[SWEEP_AHEAD];
#pragma unroll
  for (int j = 0; j < SWEEP_AHEAD; j++) {
    const size_t q = (size_t)max(nr - 1 - j, 1) * nz + k;
    av[j] = alpha[q];
    bv[j] = beta[q];
  }
  for (int i0 = nr - 2; i0 >= 0; i0 -= SWEEP_AHEAD) {
    double ac[SWEEP_AHEAD], bc[SWEEP_AHEAD];
#pragma unroll
    for (int j = 0; j < SWEEP_AHEAD; j++) {
      ac[j] = av[j];
      bc[j] = bv[j];
      const size_t q = (size_t)max(i0 - SWEEP_AHEAD + 1 - j, 1) * nz + k;
      av[j] = alpha[q];
      bv[j] = beta[q];
    }
#pragma unroll
    for (int j = 0; j < SWEEP_AHEAD; j++) {
      f = bc[j] + ac[j] * f;
      if (i0 - j >= 0) fi[(size_t)(i0 - j) * nz + k] = f;
    }
  }
}

// e1[i][k] = (fi[i][k] - fi[i+1][k]) / dr (i < nr-1); e3[i][k] = (fi[i][k] -
// fi[i][k+1]) / dz (k < nz-1); the last row of E_r and column of E_z keep
// their values
__global__ void k_poisson_field(const double *fi, double *er, double *ez, int nr, int nz,
                                double dr, double dz) {
  const long long total = (long long)nr * nz;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(q / nz), k = (int)(q - (long long)i * nz);
    if (i < nr - 1) er[q] = (fi[q] - fi[q + nz]) / dr;
    if (k < nz - 1) ez[q] = (fi[q] - fi[q + 1]) / dz;
  }
}

// 0 if 2 nz + 2 is a power of two the shared-memory FFT holds, else -1
int poisson_check(int nz) {
  const int len = 2 * nz + 2;
  if (len > DST_MAX_LEN || (len & (len - 1)) != 0) return -1;
  return 0;
}

cudaError_t launch_poisson_twiddles(int nz, double2 *w, cudaStream_t st) {
  const int half = nz + 1;
  k_twiddles<<<(half + 255) / 256, 256, 0, st>>>(w, half);
  return cudaGetLastError();
}

cudaError_t launch_poisson(const GridDev &g, const double *rho, double *t, double *fi,
                           double *alpha, double *beta, const double2 *w, const double *b_mode,
                           double *er, double *ez, cudaStream_t st) {
  const int nr = g.nr, nz = g.nz, len = 2 * nz + 2;
  int log2_len = 0;
  while ((1 << log2_len) < len) log2_len++;
  const size_t smem =
      sizeof(double2) * (size_t)(len + len / 8) + sizeof(double) * (size_t)(nz + nz / 16 + 1);
  cudaError_t e = cudaFuncSetAttribute(k_sine_transform,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int threads = len / 8 < DST_THREADS ? (len / 8 < 32 ? 32 : len / 8) : DST_THREADS;
  k_sine_transform<<<nr, threads, smem, st>>>(rho, t, w, nz, len, log2_len, false);
  k_poisson_sweep<<<(nz + SWEEP_THREADS - 1) / SWEEP_THREADS, SWEEP_THREADS, 0, st>>>(
      t, b_mode, fi, alpha, beta, nr, nz, g.dr);
  k_sine_transform<<<nr, threads, smem, st>>>(fi, fi, w, nz, len, log2_len, true);
  long long blocks = ((long long)nr * nz + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  k_poisson_field<<<(int)blocks, 256, 0, st>>>(fi, er, ez, nr, nz, g.dr, g.dz);
  return cudaGetLastError();
}

}  // namespace pdp3g
