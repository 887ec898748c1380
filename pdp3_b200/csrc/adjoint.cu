// Adjoint (vector-Jacobian product) of the FP32 cell-local PDP3 step.
//
// Reverse of one step s, given the adjoints of the state after it
// (lE, lH: FP64 grids; la, lb, lu: FP32 per particle):
//   1  E update   E' = ke E - kh (J + curl H')   (src/eField.cpp:85-170)
//        lJ = -kh lE',  lH' += curl^T(-kh lE'),  lE = ke lE'
//   2  particles  (adjoint_particle.cuh reverse on each particle's tape,
//        recomputed from the stored post-injection state of step s)
//        la/lb/lu updated in place, lw += ..., lE += gather^T, lHh += gather^T
//   3  injection  slots injected at step s: their z and u_z were set from the
//        beam velocity, so lb/luz go to d/dv_beam and are then cleared
//   4  H update   H' = H + a(E), Hh = H + a(E)/2    (src/hField.cpp:93-157)
//        lE += a^T(lH' + lHh/2),  lH = lH' + lHh
// Stencil transposes scatter with FP64 atomics.
#include <algorithm>
#include <climits>

#include "adjoint_particle.cuh"
#include "pdp3g_internal.cuh"

namespace pdp3g {

#define AIDX(i, k) ((size_t)(i) * (size_t)nz + (size_t)(k))

// step 1: E update transposed, node (i, k) of the E update's range:
// lJ = -kh lE', lH += curl^T(-kh lE'), lE = ke lE' (the scatter goes to lH
// only, so each thread can scale its own lE in place).  One or two rounds of
// CTAs at the window's grids, so a thread's chain counts: the divisions here
// and in k_adj_h take shared reciprocals and one exact residual each (rcp_ulp,
// div_rn; the values are those of a division), and k_adj_active issues all its
// loads at once (64 x 512 cells: the three together 25 -> 19 us per step).
__global__ void k_adj_e(GridDev g, AdjGrids A) {
  const int nr = g.nr, nz = g.nz;
  const double dr = g.dr, dz = g.dz, dt = g.dt, inv_dr = g.inv_dr, inv_dz = g.inv_dz;
  const long long total = (long long)(nr - 1) * (nz - 1);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = row_of(g, (int)t), k = (int)t - i * (nz - 1);
    const double epsx2 = 2 * 1.0 * EPSILON0;
    const double sigma_t = g.sigma[AIDX(i, k)] * dt;
    const double den = epsx2 + sigma_t, inv = rcp_ulp(den);
    const double kh = quotient(2 * dt, den, inv);
    const double ke = quotient(epsx2 - sigma_t, den, inv);
    if (k >= 1) {  // E_r
      const double gr = -kh * A.lEr[AIDX(i, k)];
      A.lJr[AIDX(i, k)] = (float)gr;
      const double q = div_rn(gr, dz, inv_dz);
      atomicAdd(&A.lHphi[AIDX(i, k)], q);
      atomicAdd(&A.lHphi[AIDX(i, k - 1)], -q);
      A.lEr[AIDX(i, k)] *= ke;
    }
    const double gz = -kh * A.lEz[AIDX(i, k)];
    A.lJz[AIDX(i, k)] = (float)gz;
    A.lEz[AIDX(i, k)] *= ke;
    if (i == 0) {  // on-axis E_z: 4/dr H_phi
      atomicAdd(&A.lHphi[AIDX(i, k)], div_rn(-4.0 * gz, dr, inv_dr));
    } else {
      const double two = 2.0 * dr * i, half = quotient(1.0, two, rcp_ulp(two));
      atomicAdd(&A.lHphi[AIDX(i, k)], gz * (-inv_dr - half));
      atomicAdd(&A.lHphi[AIDX(i - 1, k)], gz * (inv_dr - half));
      if (k >= 1) {  // E_phi
        const double gp = -kh * A.lEphi[AIDX(i, k)];
        A.lJphi[AIDX(i, k)] = (float)gp;
        const double qz = div_rn(gp, dz, inv_dz), qr = div_rn(gp, dr, inv_dr);
        atomicAdd(&A.lHr[AIDX(i, k)], -qz);
        atomicAdd(&A.lHr[AIDX(i, k - 1)], qz);
        atomicAdd(&A.lHz[AIDX(i, k)], qr);
        atomicAdd(&A.lHz[AIDX(i - 1, k)], -qr);
        A.lEphi[AIDX(i, k)] *= ke;
      }
    }
  }
}

// Between steps 1 and 2: cell (i, k) is active when any adjoint of J that
// the particles starting in it read is nonzero.  A particle's step moves it
// at most half a cell (Courant 0.5), so its mid-step and path cells lie
// within one cell of its start cell and the nodes it reads adjoints of J at
// within i-1..i+2, k-1..k+2.  The adjoints of the fields spread from the
// probe by one node per step (the Yee stencil), so early in the reverse most
// cells are inactive; a particle whose own adjoints are zero in an inactive
// cell has a reverse whose every output is zero (the reverse is linear in
// them) and is skipped.
__global__ void k_adj_active(GridDev g, AdjGrids A, uint8_t *active) {
  const int nr = g.nr, nz = g.nz, ncz = nz - 1;
  const long long total = (long long)(nr - 1) * ncz;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = row_of(g, (int)t), k = (int)t - i * ncz;
    // 48 loads in flight at once; -0.0f counts as zero
    unsigned any = 0;
#pragma unroll
    for (int di = -1; di <= 2; di++)
#pragma unroll
      for (int dk = -1; dk <= 2; dk++) {
        const size_t n = AIDX(min(max(i + di, 0), nr - 1), min(max(k + dk, 0), nz - 1));
        any |= __float_as_uint(A.lJr[n]) | __float_as_uint(A.lJphi[n]) | __float_as_uint(A.lJz[n]);
      }
    active[t] = (any << 1) ? 1 : 0;
  }
}

// step 4: H update transposed, every node: where the H update ran,
// lE += a^T(lH + lHh/2) and lH += lHh; everywhere lHh = 0 (the half-step
// values the update did not write never change, so their adjoints are
// dropped).  The scatter goes to lE only.
__global__ void k_adj_h(GridDev g, AdjGrids A) {
  const int nr = g.nr, nz = g.nz;
  const double dt = g.dt, drm = g.dr * MAGN_CONST, dzm = g.dz * MAGN_CONST;
  const double inv_drm = rcp_ulp(drm), inv_mu = 1.0 / MAGN_CONST, inv_dr = g.inv_dr;
  const double ca = quotient(dt, dzm, g.inv_dzmu);
  const long long total = (long long)nr * nz;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / nz), k = (int)(t - (long long)i * nz);
    if (k <= nz - 2) {
      const double la = A.lHr[t] + 0.5 * A.lHhr[t];
      atomicAdd(&A.lEphi[AIDX(i, k + 1)], la * ca);
      atomicAdd(&A.lEphi[AIDX(i, k)], -la * ca);
      A.lHr[t] += A.lHhr[t];
      if (i < nr - 1) {
        const double lb = A.lHphi[t] + 0.5 * A.lHhphi[t];
        const double qr = div_rn(lb * dt, drm, inv_drm), qz = div_rn(lb * dt, dzm, g.inv_dzmu);
        atomicAdd(&A.lEz[AIDX(i + 1, k)], qr);
        atomicAdd(&A.lEz[AIDX(i, k)], -qr);
        atomicAdd(&A.lEr[AIDX(i, k + 1)], -qz);
        atomicAdd(&A.lEr[AIDX(i, k)], qz);
        // H_z -= c, Hh_z = H_z - c/2
        const double lc = -(A.lHz[t] + 0.5 * A.lHhz[t]);
        const double rr = 2.0 * g.dr * (i + 0.5), p = quotient(1.0, rr, rcp_ulp(rr));
        atomicAdd(&A.lEphi[AIDX(i + 1, k)], div_rn(lc * dt * (p + inv_dr), MAGN_CONST, inv_mu));
        atomicAdd(&A.lEphi[AIDX(i, k)], div_rn(lc * dt * (p - inv_dr), MAGN_CONST, inv_mu));
        A.lHphi[t] += A.lHhphi[t];
        A.lHz[t] += A.lHhz[t];
      }
    }
    A.lHhr[t] = 0.0;
    A.lHhphi[t] = 0.0;
    A.lHhz[t] = 0.0;
  }
}

// adjoint of J at (i, k), 0 outside the grid
__device__ __forceinline__ float lget(const GridDev &g, const float *f, int i, int k) {
  if ((unsigned)i >= (unsigned)g.nr || (unsigned)k >= (unsigned)g.nz) return 0.0f;
  return __ldg(f + (size_t)i * g.nz + k);
}

__device__ __forceinline__ void ladd(const GridDev &g, double *f, int i, int k, double v) {
  if (v == 0.0 || (unsigned)i >= (unsigned)g.nr || (unsigned)k >= (unsigned)g.nz) return;
  atomicAdd(f + (size_t)i * g.nz + k, v);
}

#ifndef ADJ_THREADS_PER_CTA
#define ADJ_THREADS_PER_CTA 128
#endif
#ifndef ADJ_MIN_BLOCKS
#define ADJ_MIN_BLOCKS 4  // CTAs per SM the register budget is sized for (128 registers)
#endif
// the particle reverse keeps its tape in registers: with the warp-level
// reduction of the field-node adjoints (no shared tile, no barrier), 512
// resident threads of 128 registers beat 1024 of 64 with the tape spilled;
// 128-thread CTAs (4 per SM) end the grid-stride loop with a shorter tail
// than 256-thread ones (2 per SM)
constexpr int ADJ_THREADS = ADJ_THREADS_PER_CTA;
static_assert(ADJ_THREADS % 16 == 0, "prefetch sizes are multiples of 16 bytes");
#ifndef ADJ_PREFETCH_AHEAD
#define ADJ_PREFETCH_AHEAD 1  // CTA iterations between a chunk's prefetch and its use
#endif
// One lane asks L2 for the particle chunk that this CTA steps after the
// current one (the reverse is latency-bound: 16 warps per SM), when that
// chunk is a full one: every prefetched byte lies inside the arrays.
__device__ __forceinline__ void prefetch_chunk(const AdjSpeciesDev &S, long long next) {
  if ((next + 1) * ADJ_THREADS > S.st.n) return;
  const long long q = next * ADJ_THREADS;
  constexpr unsigned B4 = 4u * ADJ_THREADS;
  prefetch_l2(S.st.cell + q, B4);
  prefetch_l2(S.st.fr + q, B4);
  prefetch_l2(S.st.fz + q, B4);
  prefetch_l2(S.st.ur + q, B4);
  prefetch_l2(S.st.uphi + q, B4);
  prefetch_l2(S.st.uz + q, B4);
  prefetch_l2(S.st.w + q, B4);
  if (S.st.alive) prefetch_l2(S.st.alive + q, ADJ_THREADS);
  prefetch_l2(S.la + q, B4);
  prefetch_l2(S.lb + q, B4);
  prefetch_l2(S.lur + q, B4);
  prefetch_l2(S.luphi + q, B4);
  prefetch_l2(S.luz + q, B4);
  prefetch_l2(S.lw + q, 2 * B4);
}

// Warp-level segmented sum over runs of consecutive lanes with the same key
// (particles of a cell with the same half-cell quadrant share their 24 gather
// nodes); the last lane of each run holds the run's totals.  Stops at the
// longest run: the quadrants of a cell alternate, so runs are mostly short.
template <int N>
__device__ __forceinline__ bool warp_seg_sum(int key, float (&v)[N]) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(FULL, key, 1);
  const int next = __shfl_down_sync(FULL, key, 1);
  const bool head = lane == 0 || prev != key;
  const bool tail = lane == 31 || next != key;
  const unsigned heads = __ballot_sync(FULL, head);
  const unsigned le = lane == 31 ? FULL : ((2u << lane) - 1u);
  const int seg_start = 31 - __clz(heads & le);
  const int longest = __reduce_max_sync(FULL, key >= 0 ? lane - seg_start : 0);
#pragma unroll 1
  for (int off = 1; off <= longest; off <<= 1) {
#pragma unroll
    for (int j = 0; j < N; j++) {
      const float y = __shfl_up_sync(FULL, v[j], off);
      if (lane >= seg_start + off) v[j] += y;
    }
  }
  return tail && key >= 0;
}

// ---- sums of the field-node adjoints over a warp ---------------------------
// The particles of a cell gather from 37 nodes: per component 2 or, in a
// dimension whose weighting is half a cell off, 3 of which a particle uses
// the lower or the upper 2.  The totals of a warp's runs (warp_seg_sum) in
// one cell are added in FP64 over all 37 nodes together by halving: in each
// of five steps a lane keeps half of its values and hands the other half to
// its partner (37, 19, 10, 5, 3, 2 values: 39 exchanges), so the sums end up
// spread over the lanes, which add them to the grids side by side.  Without
// it every run's last lane made 24 additions, and as the quadrants alternate
// within a cell those were three quarters of the lanes: additions at L2 bound
// the kernel (1M electrons, drifted for 200 steps: 99 us, ions 96 us; now 85 and 53).
constexpr int FOOT = 37;  // nodes of the six components

// node s of the footprint: component (E_r, E_phi, E_z, H_r, H_phi, H_z) and
// the offset from the cell's node
struct FootNode {
  int comp, di, dk;
};
__device__ __forceinline__ FootNode foot_node(int s) {
  for (int comp = 0; comp < 6; comp++) {
    const bool rh = adj::comp_rhalf(comp / 3, comp % 3), zh = adj::comp_zhalf(comp / 3, comp % 3);
    const int nr = rh ? 3 : 2, n = nr * (zh ? 3 : 2);
    if (s < n) return FootNode{comp, s % nr - (rh ? 1 : 0), s / nr - (zh ? 1 : 0)};
    s -= n;
  }
  return FootNode{0, 0, 0};
}

// lf: the 4 nodes (ir, kz), (ir+1, kz), (ir, kz+1), (ir+1, kz+1) of each
// component; r_lo, z_lo: the half weighting starts one node below the cell's
__device__ __forceinline__ void foot_values(const float (&lf)[24], bool r_lo, bool z_lo,
                                            float (&w)[FOOT]) {
  int s = 0;
#pragma unroll
  for (int comp = 0; comp < 6; comp++) {
    const bool rh = adj::comp_rhalf(comp / 3, comp % 3), zh = adj::comp_zhalf(comp / 3, comp % 3);
    const int nr = rh ? 3 : 2;
    float row[2][3];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const float x0 = lf[comp * 4 + 2 * q], x1 = lf[comp * 4 + 2 * q + 1];
      row[q][0] = rh && !r_lo ? 0.0f : x0;
      row[q][1] = rh && !r_lo ? x0 : x1;
      row[q][2] = r_lo ? 0.0f : x1;
    }
#pragma unroll
    for (int j = 0; j < nr; j++) {
      if (zh) {
        w[s + j] = z_lo ? row[0][j] : 0.0f;
        w[s + nr + j] = z_lo ? row[1][j] : row[0][j];
        w[s + 2 * nr + j] = z_lo ? 0.0f : row[1][j];
      } else {
        w[s + j] = row[0][j];
        w[s + nr + j] = row[1][j];
      }
    }
    s += nr * (zh ? 3 : 2);
  }
}

template <int N, int BIT>
struct Halve {
  static constexpr int H = (N + 1) / 2;
  // FP64 totals of v over the warp, those this lane keeps in out (the first
  // exchange still hands over floats)
  template <class T>
  static __device__ __forceinline__ void sum(const T (&v)[N], double (&out)[2]) {
    const bool hi = threadIdx.x & BIT;
    double keep[H];
#pragma unroll
    for (int j = 0; j < H; j++) {
      const T a = v[j], b = j + H < N ? v[j + H < N ? j + H : 0] : T(0);
      keep[j] = (double)(hi ? b : a) + (double)__shfl_xor_sync(0xffffffffu, hi ? a : b, BIT);
    }
    Halve<H, BIT / 2>::sum(keep, out);
  }
  // which those are (-1: none)
  static __device__ __forceinline__ int kept(int lane, int j) {
    const int k = Halve<H, BIT / 2>::kept(lane, j);
    if (k < 0 || !(lane & BIT)) return k;
    return k + H < N ? k + H : -1;
  }
};
template <int N>
struct Halve<N, 0> {
  static_assert(N == 2, "two totals a lane");
  static __device__ __forceinline__ void sum(const double (&v)[N], double (&out)[2]) {
    out[0] = v[0];
    out[1] = v[1];
  }
  static __device__ __forceinline__ int kept(int, int j) { return j; }
};

// the totals of one cell onto the grids: tab = this lane's two nodes
__device__ __forceinline__ void foot_add(const GridDev &g, const AdjGrids &A,
                                         const FootNode *tab, int cell, const float (&w)[FOOT]) {
  double tot[2];
  Halve<FOOT, 16>::sum(w, tot);
  const int i = row_of(g, cell), k = cell - i * (g.nz - 1);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const FootNode f = tab[j];
    if (f.comp < 0) continue;
    double *grid = f.comp < 3 ? (f.comp == 0 ? A.lEr : (f.comp == 1 ? A.lEphi : A.lEz))
                              : (f.comp == 3 ? A.lHhr : (f.comp == 4 ? A.lHhphi : A.lHhz));
    ladd(g, grid, i + f.di, k + f.dk, tot[j]);
  }
}

// Cells of a warp added up one by one; with more, each run adds its own.  A
// round of halving costs about 290 instructions, a warp's run additions about
// as much time as three (250 steps, 32 particles per cell: 49.2 ms with 2,
// 49.9 with 4, 50.1 with 8; after 500 more steps of drift 50.6, 50.9, 55.3;
// 57.5 with none).
constexpr int ADJ_MAX_CELLS = 2;

// step 2: particles.  Q = E and the half-step H of step s as per-cell quads
// (the 2x2 nodes of a cell, GridDev::q32's layout, as the forward step
// gathered them).  Each thread takes one particle; the 24
// field-node adjoints of a warp's particles are summed over runs of lanes
// that share their gather nodes (particles sorted by cell) and each run adds
// its totals to the FP64 grids.  Warps are independent.  WALLS: whether the
// wall-reflection jump terms (face bit 1) are compiled in.
template <bool WALLS>
__global__ void __launch_bounds__(ADJ_THREADS, ADJ_MIN_BLOCKS) k_adj_particles(
    GridDev g, const float4 *Q, AdjSpeciesDev S, AdjGrids A, const uint8_t *active, int face,
    float face_h) {
  const int ncz = g.nz - 1;
  __shared__ FootNode foot[32][2];
  if (threadIdx.x < 32)
    for (int j = 0; j < 2; j++) {
      const int s = Halve<FOOT, 16>::kept(threadIdx.x, j);
      foot[threadIdx.x][j] = s < 0 ? FootNode{-1, 0, 0} : foot_node(s);
    }
  __syncthreads();
  adj::Consts<float> C;
  C.ke = S.st.ke;
  C.kb = S.st.kb;
  C.cr = S.st.cr;
  C.cz = S.st.cz;
  C.kphi = S.st.kphi;
  C.kz = S.st.kz;
  C.kr = S.st.kr;
  C.nr = g.nr;
  C.nz = g.nz;
  C.bunch = S.st.kind == KIND_BUNCH;
  C.face = face;
  C.face_h = face_h;
  const long long nchunks = (S.st.n + ADJ_THREADS - 1) / ADJ_THREADS;
  for (long long chunk = blockIdx.x; chunk < nchunks; chunk += gridDim.x) {
    if (threadIdx.x == 0) prefetch_chunk(S, chunk + ADJ_PREFETCH_AHEAD * (long long)gridDim.x);
    const long long p = chunk * ADJ_THREADS + threadIdx.x;
    // every load of the particle at once: one trip to memory, also for a
    // particle that turns out to have nothing to do (its lines are in L2 by
    // the prefetch)
    const long long q = min(p, S.st.n - 1);
    const float sa = S.st.fr[q], sb = S.st.fz[q], su0 = S.st.ur[q], su1 = S.st.uphi[q],
                su2 = S.st.uz[q], sw = S.st.w[q];
    const float pa = S.la[q], pb = S.lb[q], pu0 = S.lur[q], pu1 = S.luphi[q], pu2 = S.luz[q];
    const double pw = S.lw[q];
    const int c = S.st.cell[q];
    bool live = p < S.st.n && (S.st.alive == nullptr || S.st.alive[q]);
    if (c < 0 || c >= (g.nr - 1) * ncz) live = false;  // flagged by the forward step
    // zero adjoints of the particle and none of J within its reach (k_adj_active):
    // every output of its reverse is zero, nothing to do.  Tested bitwise (a
    // sign-only -0.0f counts as nonzero, which only costs a reverse that adds
    // zeros).
    const unsigned bits = __float_as_uint(pa) | __float_as_uint(pb) | __float_as_uint(pu0) |
                          __float_as_uint(pu1) | __float_as_uint(pu2);
    if (live && bits == 0u && !active[c]) live = false;
    if (__all_sync(0xffffffffu, !live)) continue;  // the whole warp: no sums to add either
    const int ci = row_of(g, c), ck = c - ci * ncz;
    float lf[24];  // this lane's field-node adjoints
    int key = -1, q_ir_h = ci, q_kz_h = ck;
    if (!live) {
#pragma unroll
      for (int j = 0; j < 24; j++) lf[j] = 0.0f;
    } else {
      adj::Tape<float> tp;
      tp.i = ci;
      tp.k = ck;
      tp.a = sa;
      tp.b = sb;
      tp.u[0] = su0;
      tp.u[1] = su1;
      tp.u[2] = su2;
      tp.w = sw;
      adj::gather_weights(tp);
      // node rows/columns of the two weightings (clamped as the forward gather)
      const int ir_h = min(tp.ir_h, g.nr - 2), ir_n = min(tp.i, g.nr - 2);
      const int kz_h = min(tp.kz_h, g.nz - 2), kz_n = min(tp.k, g.nz - 2);
#pragma unroll
      for (int cc = 0; cc < 3; cc++) {
        {
          const int ir = adj::comp_rhalf(0, cc) ? ir_h : ir_n;
          const int kz = adj::comp_zhalf(0, cc) ? kz_h : kz_n;
          const float4 v = __ldg(Q + 6 * ((size_t)ir * ncz + kz) + cc);
          tp.fe[cc][0] = v.x;
          tp.fe[cc][1] = v.y;
          tp.fe[cc][2] = v.z;
          tp.fe[cc][3] = v.w;
        }
        {
          const int ir = adj::comp_rhalf(1, cc) ? ir_h : ir_n;
          const int kz = adj::comp_zhalf(1, cc) ? kz_h : kz_n;
          const float4 v = __ldg(Q + 6 * ((size_t)ir * ncz + kz) + 3 + cc);
          tp.fh[cc][0] = v.x;
          tp.fh[cc][1] = v.y;
          tp.fh[cc][2] = v.z;
          tp.fh[cc][3] = v.w;
        }
      }
      adj::forward(C, tp);
      float l_jphi[4] = {lget(g, A.lJphi, tp.i1, tp.k1), lget(g, A.lJphi, tp.i1 + 1, tp.k1),
                         lget(g, A.lJphi, tp.i1, tp.k1 + 1),
                         lget(g, A.lJphi, tp.i1 + 1, tp.k1 + 1)};
      float l_piece[3][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}};
      if (tp.path_ok) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
          if (q > tp.np) continue;
          const int qi = tp.pci(q), qk = tp.pck(q);
          l_piece[q][0] = lget(g, A.lJz, qi, qk);
          l_piece[q][1] = lget(g, A.lJz, qi + 1, qk);
          l_piece[q][2] = lget(g, A.lJr, qi, qk);
          l_piece[q][3] = lget(g, A.lJr, qi, qk + 1);
        }
      }
      const float l_uout[3] = {pu0, pu1, pu2};
      float l_a, l_b, l_u[3], l_w, l_fe[3][4], l_fh[3][4];
      adj::reverse<float, WALLS>(C, tp, pa, pb, l_uout, l_jphi, l_piece, l_a, l_b,
                                 l_u, l_w, l_fe, l_fh);
      S.la[p] = l_a;
      S.lb[p] = l_b;
      S.lur[p] = l_u[0];
      S.luphi[p] = l_u[1];
      S.luz[p] = l_u[2];
      S.lw[p] = pw + (double)l_w;
#pragma unroll
      for (int cc = 0; cc < 3; cc++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
          lf[cc * 4 + q] = l_fe[cc][q];
          lf[12 + cc * 4 + q] = l_fh[cc][q];
        }
      // lanes with the same cell and half-cell quadrant share the 24 nodes
      key = (c * 2 + (tp.ir_h == ci ? 1 : 0)) * 2 + (tp.kz_h == ck ? 1 : 0);
      q_ir_h = ir_h;
      q_kz_h = kz_h;
    }
    const bool tail = warp_seg_sum<24>(key, lf);
    // the cells of the runs, one lane of each
    const unsigned peers = __match_any_sync(0xffffffffu, tail ? c : -1);
    unsigned cells = __ballot_sync(0xffffffffu, tail && (peers & ((1u << (threadIdx.x & 31)) - 1)) == 0);
    if (__popc(cells) <= ADJ_MAX_CELLS) {
      if (!tail) {
#pragma unroll
        for (int j = 0; j < 24; j++) lf[j] = 0.0f;
      }
      float w[FOOT];
      foot_values(lf, q_ir_h < ci, q_kz_h < ck, w);
      const FootNode *tab = foot[threadIdx.x & 31];
      if ((cells & (cells - 1)) == 0) {  // one cell: the other lanes hold zeros
        foot_add(g, A, tab, __shfl_sync(0xffffffffu, c, __ffs(cells) - 1), w);
      } else {
        for (; cells; cells &= cells - 1) {
          const int cell = __shfl_sync(0xffffffffu, c, __ffs(cells) - 1);
          float m[FOOT];
#pragma unroll
          for (int j = 0; j < FOOT; j++) m[j] = c == cell ? w[j] : 0.0f;
          foot_add(g, A, tab, cell, m);
        }
      }
    } else if (tail) {
#pragma unroll
      for (int cc = 0; cc < 6; cc++) {
        const int ir = adj::comp_rhalf(cc / 3, cc % 3) ? q_ir_h : ci;
        const int kz = adj::comp_zhalf(cc / 3, cc % 3) ? q_kz_h : ck;
        double *grid = cc < 3 ? (cc == 0 ? A.lEr : (cc == 1 ? A.lEphi : A.lEz))
                              : (cc == 3 ? A.lHhr : (cc == 4 ? A.lHhphi : A.lHhz));
        ladd(g, grid, ir, kz, lf[cc * 4 + 0]);
        ladd(g, grid, ir + 1, kz, lf[cc * 4 + 1]);
        ladd(g, grid, ir, kz + 1, lf[cc * 4 + 2]);
        ladd(g, grid, ir + 1, kz + 1, lf[cc * 4 + 3]);
      }
    }
  }
}

// step 3: injected slots [start, start+count): z = dl rr + dz/2 with
// dl = v dt and u_z = gamma(v) v / c.  Adds their d/dv into *lv and clears
// lb, luz (the values they replaced had no influence).
__global__ void k_adj_inject(AdjSpeciesDev S, long long start, long long count, double dt,
                             double dz, double velocity, const double *inv_pow11, double *lv) {
  double acc = 0;
  const double beta2 = velocity * velocity / LIGHT_SPEED_POW_2;
  const double duz_dv = 1.0 / (LIGHT_SPEED * pow(1.0 - beta2, 1.5));
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < count;
       j += (long long)gridDim.x * blockDim.x) {
    const long long idx = start + j;
    if (idx >= S.st.n) continue;
    int int_vel = (int)floor((double)(unsigned)idx);
    double ost = 0, rr = 0;
    int order = 1;
    while (int_vel >= 1 && order < 40) {
      ost = int_vel % 11;
      rr = rr + ost * inv_pow11[order];
      int_vel = (int)((int_vel - ost) / 11);
      order = order + 1;
    }
    acc += (double)S.lb[idx] * (dt * rr / dz) + (double)S.luz[idx] * duz_dv;
    S.lb[idx] = 0.0f;
    S.luz[idx] = 0.0f;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc != 0.0) atomicAdd(lv, acc);
}

// loss = sum over the probe nodes of E_z^2 V (node volume); seeds lE_z = 2 E_z V
__global__ void k_adj_seed(GridDev g, AdjGrids A, int r0, int r1, int z0, int z1,
                           double *loss) {
  const int nz = g.nz;
  const double dr = g.dr, dz = g.dz;
  const long long w = (long long)(z1 - z0), total = (long long)(r1 - r0) * w;
  double acc = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = r0 + (int)(t / w), k = z0 + (int)(t - (t / w) * w);
    const double vol = i == 0 ? PI * dz * dr * dr / 4. : 2.0 * PI * dz * dr * dr * i;
    const double ez = g.ez[AIDX(i, k)];
    acc += ez * ez * vol;
    A.lEz[AIDX(i, k)] = 2.0 * ez * vol;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, acc);
}

static int blocks_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b > 148 * 16) b = 148 * 16;
  return (int)(b < 1 ? 1 : b);
}

void adj_launch_e(const GridDev &g, const AdjGrids &A, cudaStream_t st) {
  k_adj_e<<<blocks_for((long long)(g.nr - 1) * (g.nz - 1), 256), 256, 0, st>>>(g, A);
}

void adj_launch_h(const GridDev &g, const AdjGrids &A, cudaStream_t st) {
  k_adj_h<<<blocks_for((long long)g.nr * g.nz, 256), 256, 0, st>>>(g, A);
}

void adj_launch_active(const GridDev &g, const AdjGrids &A, uint8_t *active, cudaStream_t st) {
  k_adj_active<<<blocks_for((long long)(g.nr - 1) * (g.nz - 1), 256), 256, 0, st>>>(g, A, active);
}

void adj_launch_particles(const GridDev &g, const float4 *Q, const AdjSpeciesDev &S,
                          const AdjGrids &A, const uint8_t *active, int face, float face_h,
                          cudaStream_t st) {
  if (S.st.n <= 0) return;
  const long long nchunks = (S.st.n + ADJ_THREADS - 1) / ADJ_THREADS;
  auto kernel = (face & 2) ? k_adj_particles<true> : k_adj_particles<false>;
  int bpsm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, kernel, ADJ_THREADS, 0) !=
          cudaSuccess || bpsm < 1)
    bpsm = 1;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const long long blocks = std::min<long long>(nchunks, (long long)bpsm * nsm);
  kernel<<<(int)std::max<long long>(blocks, 1), ADJ_THREADS, 0, st>>>(g, Q, S, A, active,
                                                                         face, face_h);
}

void adj_launch_inject(const AdjSpeciesDev &S, long long start, long long count, double dt,
                       double dz, double velocity, const double *inv_pow11, double *lv,
                       cudaStream_t st) {
  if (count <= 0) return;
  k_adj_inject<<<blocks_for(count, 256), 256, 0, st>>>(S, start, count, dt, dz, velocity,
                                                        inv_pow11, lv);
}

void adj_launch_seed(const GridDev &g, const AdjGrids &A, int r0, int r1, int z0, int z1,
                     double *loss, cudaStream_t st) {
  const long long n = (long long)(r1 - r0) * (z1 - z0);
  k_adj_seed<<<blocks_for(n, 256), 256, 0, st>>>(g, A, r0, r1, z0, z1, loss);
}

}  // namespace pdp3g
