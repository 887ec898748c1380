// Yee FDTD updates of the axisymmetric (r, phi, z) grid.
//
// Compiled with --fmad=false: the arithmetic keeps the upstream operation
// order so the FP64 result matches the CPU step bit for bit.
//
// The kernels are streaming stencils (one thread per node, the z index fastest
// so warps read contiguous rows; the r-neighbour rows come from L2).
// Algorithmic bytes per node: H update reads E (3) and H (3), writes H (3) and
// H_half (3): 96 B; E update reads E (3), H (3), J (3), sigma, writes E (3):
// 104 B.
#include "fields_body.cuh"

namespace pdp3g {

// 32 x 8 nodes per CTA; rows beyond gridDim.y * 8 in further rounds.  Six CTAs of
// the H update per SM (40 registers), five of the E update (48): the call for
// the rare node would else take 48 and 64, and a grid of many rounds wants the
// warps (513 x 4097 nodes: H update 48.5 -> 46.2 us; 257 x 2049 nodes in a wake
// step: E update 17.0 -> 14.4 us).
constexpr int FZ = 32, FR = 8, H_BLOCKS = 6, E_BLOCKS = 5;

static dim3 field_grid(const GridDev &g) {
  const int rows = (g.nr + FR - 1) / FR;
  return dim3((g.nz + FZ - 1) / FZ, rows < 65535 ? rows : 65535);
}

// H update over i in [0, nr-1], k in [0, nz-2]; RESET: J = 0 at every node
template <bool RESET>
__global__ void __launch_bounds__(FZ * FR, H_BLOCKS)
    k_yee_h(const __grid_constant__ GridDev g) {
  const int k = blockIdx.x * FZ + threadIdx.x;
  if (k >= g.nz) return;
  for (int i = blockIdx.y * FR + threadIdx.y; i < g.nr; i += gridDim.y * FR) {
    if (RESET) {
      const size_t n = (size_t)i * g.nz + k;
      g.jr[n] = 0.0;
      g.jphi[n] = 0.0;
      g.jz[n] = 0.0;
    }
    if (k < g.nz - 1) yee_h_node(g, i, k);
  }
}

// the deposits at node (i, k) of the up to four cells around it (GridDev::j8)
__device__ __forceinline__ void cell_deposits(const GridDev &g, int i, int k, double &jr,
                                              double &jphi, double &jz) {
  const int ncz = g.nz - 1;
  const double2 *j8 = reinterpret_cast<const double2 *>(g.j8);
  const long long cell = (long long)i * ncz + k;
  const bool i0 = i < g.nr - 1, i1 = i > 0, k0 = k < ncz, k1 = k > 0;
  if (i0 && k0) {
    const double2 v = j8[4 * cell];
    jphi += v.x;
    jz += v.y;
    jr += j8[4 * cell + 3].x;
  }
  if (i1 && k0) {
    const double2 v = j8[4 * (cell - ncz) + 1];
    jphi += v.x;
    jz += v.y;
  }
  if (i0 && k1) {
    const double2 v = j8[4 * (cell - 1) + 2];
    jphi += v.x;
    jr += v.y;
  }
  if (i1 && k1) jphi += j8[4 * (cell - ncz - 1) + 3].y;
}

// J += the cells' deposits
__global__ void __launch_bounds__(FZ * FR) k_unpack_j(const __grid_constant__ GridDev g) {
  const int k = blockIdx.x * FZ + threadIdx.x;
  if (k >= g.nz) return;
  for (int i = blockIdx.y * FR + threadIdx.y; i < g.nr; i += gridDim.y * FR) {
    double jr = 0, jphi = 0, jz = 0;
    cell_deposits(g, i, k, jr, jphi, jz);
    const size_t n = (size_t)i * g.nz + k;
    g.jr[n] += jr;
    g.jphi[n] += jphi;
    g.jz[n] += jz;
  }
}

// E update over i in [0, nr-2], k in [0, nz-2]; UNPACK: J += the cells' deposits
// at every node first; d_time: *d_time += dt (src/loadInitParam.cpp:586)
template <bool UNPACK>
__global__ void __launch_bounds__(FZ * FR, E_BLOCKS)
    k_yee_e(const __grid_constant__ GridDev g, double *d_time) {
  const int k = blockIdx.x * FZ + threadIdx.x;
  if (d_time && blockIdx.y == 0 && threadIdx.y == 0 && k == 0) *d_time = *d_time + g.dt;
  if (k >= g.nz) return;
  for (int i = blockIdx.y * FR + threadIdx.y; i < g.nr; i += gridDim.y * FR) {
    const size_t n = (size_t)i * g.nz + k;
    double jr = g.jr[n], jphi = g.jphi[n], jz = g.jz[n];
    if (UNPACK) {
      double r = 0, phi = 0, z = 0;
      cell_deposits(g, i, k, r, phi, z);
      g.jr[n] = jr += r;
      g.jphi[n] = jphi += phi;
      g.jz[n] = jz += z;
    }
    if (i < g.nr - 1 && k < g.nz - 1) yee_e_node(g, i, k, jr, jphi, jz);
  }
}

__global__ void k_to_f32(const double *src, float *dst, size_t n) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n;
       t += (size_t)gridDim.x * blockDim.x)
    dst[t] = (float)src[t];
}

// thread t = 6 cell + c: the 2x2 nodes of the cell of component c
// (0-2 E_r, E_phi, E_z from e32; 3-5 the half-step H_r, H_phi, H_z from hh32)
__global__ void k_pack_quads(GridDev g, float4 *q) {
  const int nz = g.nz, ncz = nz - 1;
  const long long ng = (long long)g.nr * nz, ncells = (long long)(g.nr - 1) * ncz;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 6 * ncells;
       t += (long long)gridDim.x * blockDim.x) {
    const long long cell = t / 6;
    const int c = (int)(t - cell * 6);
    const int i = (int)(cell / ncz), k = (int)(cell - (long long)i * ncz);
    const float *f = (c < 3 ? g.e32 : g.hh32) + (c % 3) * ng + (long long)i * nz + k;
    q[t] = make_float4(__ldg(f), __ldg(f + nz), __ldg(f + 1), __ldg(f + nz + 1));
    if (c < 4 && g.j8) reinterpret_cast<double2 *>(g.j8)[4 * cell + c] = make_double2(0.0, 0.0);
  }
}

static int grid_blocks(long long total) {
  long long b = (total + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

void launch_yee_h(const GridDev &g, cudaStream_t st) {
  k_yee_h<false><<<field_grid(g), dim3(FZ, FR), 0, st>>>(g);
}

void launch_yee_e(const GridDev &g, cudaStream_t st) {
  k_yee_e<false><<<field_grid(g), dim3(FZ, FR), 0, st>>>(g, nullptr);
}

void launch_unpack_j(const GridDev &g, cudaStream_t st) {
  k_unpack_j<<<field_grid(g), dim3(FZ, FR), 0, st>>>(g);
}

void launch_field_begin(const GridDev &g, cudaStream_t st) {
  k_yee_h<true><<<field_grid(g), dim3(FZ, FR), 0, st>>>(g);
}

void launch_field_end(const GridDev &g, double *d_time, cudaStream_t st) {
  if (g.j8)
    k_yee_e<true><<<field_grid(g), dim3(FZ, FR), 0, st>>>(g, d_time);
  else
    k_yee_e<false><<<field_grid(g), dim3(FZ, FR), 0, st>>>(g, d_time);
}

void launch_pack_quads(const GridDev &g, float4 *q, cudaStream_t st) {
  k_pack_quads<<<grid_blocks(6LL * (g.nr - 1) * (g.nz - 1)), 256, 0, st>>>(g, q);
}

void launch_to_f32(const double *src, float *dst, size_t n, cudaStream_t st) {
  long long b = ((long long)n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  k_to_f32<<<(int)b, 256, 0, st>>>(src, dst, n);
}
}  // namespace pdp3g
