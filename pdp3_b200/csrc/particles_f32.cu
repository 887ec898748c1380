// FP32 cell-local form of the particle phase of one PDP3 step.
//
// Particle state (structure of arrays, 28 B read / 24 B written per step):
//   cell   int32   i * (n_grid_z - 1) + k, the upstream cell
//                  (CELL_NUMBER, include/geometry.h:44: r in (i dr, (i+1) dr])
//   fr, fz float   in-cell offsets r/dr - i and z/dz - k, in (0, 1]
//   ur, uphi, uz float   momentum per mass over c, u = gamma v / c
//   w      float   macroparticle weight (physical particles carried)
//   alive  uint8   bunch species only
//
// The step is the upstream one (gather, relativistic Boris or the upstream
// Vay, two half moves with the rz rotation, azimuthal deposition at the
// mid-step position, reflection or loss at the walls, r-z deposition along
// the step, velocity rotation), written in cell-local units so that every
// quantity that the upstream code forms as a difference of two large
// numbers is formed from offsets instead:
//
// * gather weights: (r2^2 - r1^2) = (r2 - r1)(r2 + r1) with r2 - r1 an exact
//   small offset (EField::get_field src/eField.cpp:204-316, including its
//   CELL_VOLUME(i+3) and CELL_VOLUME(i+2) normalisation);
// * rz rotation: r' - x = y^2 / (x + r') instead of sqrt(x^2+y^2) - x;
// * r-z deposition (Particles::simple_current_distribution,
//   src/particles.cpp:333-474): with rho_m the segment's mid radius in
//   cells, f_m its offset and s = (d_rho/2)/rho_m, the closed forms reduce to
//     j_z(i)   ~ d_zeta [(1 - f_m)(2i + f_m) + i(i+1) eps] / (i rho_m)
//     j_z(i+1) ~ d_zeta [f_m (2i + 1 + f_m) - i(i+1) eps] / ((i+1) rho_m)
//     j_r(i,k) ~ d_rho beta/2 - d_zeta d_rho/4 + i(i+1)/2 [d_rho beta/(rho_o rho_n)
//                - d_zeta d_rho/(2 rho_n rho_m) - d_zeta eps/rho_m]    / (i + 1/2)
//   (j_r(i,k+1) the same with beta -> 1 - beta, d_zeta -> -d_zeta), where
//   eps = atanh(s)/s - 1 carries the upstream log((r_o+dr)/r_o) term.  These
//   are the upstream integrals rearranged; they are smooth in d_rho -> 0 and
//   d_zeta -> 0, where the upstream switches to strict_motion_weighting
//   (src/particles.cpp:786-988), whose z-only and i = 0 forms they equal.
//
// A lane steps two particles at a time with packed FP32 instructions and keeps
// running sums of their deposits while the cell stays the same; a segmented
// warp sum per chunk and FP64 atomics then add the runs to the cells' eight
// sums (GridDev::j8; particles sorted by cell make the runs long).
#include <algorithm>

#include "particles_f32.cuh"

namespace pdp3g {

// ---- two particles at once: x holds one, y the next.  Each operation below is
// one packed instruction (fma.rn.f32x2 and its forms), lane-wise the same as
// the scalar operation, so a particle's result does not depend on its partner.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float rcp(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(rcp(a.x), rcp(a.y)); }
__device__ __forceinline__ float2 rsqrt2(float2 a) {
  return make_float2(rsqrtf(a.x), rsqrtf(a.y));
}
__device__ __forceinline__ float2 dot2(const float2 a[3], const float2 b[3], float2 c) {
  return fma2(a[0], b[0], fma2(a[1], b[1], fma2(a[2], b[2], c)));
}

// Constants of the pair step as packed operands (both halves equal): read as
// one 64-bit uniform load each.
struct PairConst {
  float2 ke, kb, cr, cz, kphi, kz2, kr, vay_e, vay_b, inv_c2, c, inv_c;
  float2 m1, half, one, one5, two, four, third, fifth, seventh, ninth;
};

static PairConst pair_const(const SpeciesF32 &s) {
  const auto d = [](float x) { return make_float2(x, x); };
  return PairConst{d(s.ke), d(s.kb), d(s.cr), d(s.cz), d(s.kphi), d(2.0f * s.kz), d(s.kr),
                   d(s.vay_e), d(s.vay_b), d(s.inv_c2), d((float)LIGHT_SPEED),
                   d((float)(1.0 / LIGHT_SPEED)), d(-1.0f), d(0.5f), d(1.0f), d(1.5f), d(2.0f),
                   d(4.0f), d(1.0f / 3.0f), d(0.2f), d(1.0f / 7.0f), d(1.0f / 9.0f)};
}

// a . b and a . a
__device__ __forceinline__ float2 in2(const float2 a[3], const float2 b[3]) {
  return fma2(a[0], b[0], fma2(a[1], b[1], mul(a[2], b[2])));
}
__device__ __forceinline__ float2 sq2(const float2 a[3]) { return in2(a, a); }

// the quads' sum at one particle
__device__ __forceinline__ float quad_sum(float4 v, float c00, float c10, float c01, float c11) {
  return fmaf(v.x, c00, fmaf(v.y, c10, fmaf(v.z, c01, v.w * c11)));
}

// E and the half-step H of a pair at offsets a, b of the cells c (rows i,
// columns k, row table entries Ra, Rb), from the cells' packed quads.  Weights
// as weights_rhalf, weights_rnode and weights_zhalf, the node volumes'
// reciprocals from the table.
__device__ __forceinline__ void gather_pair(const GridDev &g, const PairConst &K, int2 c, int2 i,
                                            int2 k, float2 fi, float2 a, float2 b, float4 Ra,
                                            float4 Rb, float2 e[3], float2 h[3]) {
  const int ncz = g.nz - 1;
  // the half-node components' block lies one row (column) lower in the cell's
  // lower half
  const bool lra = !(a.x > 0.5f || i.x == 0), lrb = !(a.y > 0.5f || i.y == 0);
  const bool lza = !(b.x > 0.5f || k.x == 0), lzb = !(b.y > 0.5f || k.y == 0);
  const float2 hr = make_float2(lra ? 0.5f : -0.5f, lrb ? 0.5f : -0.5f);
  const float2 hz = make_float2(lza ? 0.5f : -0.5f, lzb ? 0.5f : -0.5f);
  const float2 rx = make_float2(Ra.x, Rb.x), rz = make_float2(Ra.z, Rb.z);
  const float2 h0i = make_float2(lra ? Ra.x : Ra.y, lrb ? Rb.x : Rb.y);
  const float2 h1i = make_float2(lra ? Ra.z : Ra.w, lrb ? Rb.z : Rb.w);
  const float2 sn = fma2(fi, K.two, a);  // 2 i + a
  // half rows: t = a + hr, (1 - t)(2 ir + 1 + t), t (2 ir + 2 + t)
  const float2 t = add(a, hr), sh = fma2(hr, K.m1, sn);
  const float2 wh0 = mul(mul(fma2(t, K.m1, K.one), sh), h0i);
  const float2 wh1 = mul(mul(t, add(sh, K.one)), h1i);
  const float2 wn0 = mul(mul(fma2(a, K.m1, K.one), sn), rx);
  const float2 wn1 = mul(mul(a, add(sn, K.one)), rz);
  const float2 zh1 = add(b, hz), zh0 = fma2(zh1, K.m1, K.one), zn0 = fma2(b, K.m1, K.one);
  // the particle's cell, one row lower, one column lower, both
  const float4 *nna = g.q32 + 6 * (size_t)(unsigned)c.x, *nnb = g.q32 + 6 * (size_t)(unsigned)c.y;
  const float4 *hna = g.q32 + 6 * (size_t)(unsigned)(c.x - (lra ? ncz : 0));
  const float4 *hnb = g.q32 + 6 * (size_t)(unsigned)(c.y - (lrb ? ncz : 0));
  const float4 *nha = nna - (lza ? 6 : 0), *nhb = nnb - (lzb ? 6 : 0);
  const float4 *hha = hna - (lza ? 6 : 0), *hhb = hnb - (lzb ? 6 : 0);
  const float2 hn00 = mul(wh0, zn0), hn10 = mul(wh1, zn0), hn01 = mul(wh0, b), hn11 = mul(wh1, b);
  e[0].x = quad_sum(__ldg(hna + 0), hn00.x, hn10.x, hn01.x, hn11.x);
  e[0].y = quad_sum(__ldg(hnb + 0), hn00.y, hn10.y, hn01.y, hn11.y);
  h[2].x = quad_sum(__ldg(hna + 5), hn00.x, hn10.x, hn01.x, hn11.x);
  h[2].y = quad_sum(__ldg(hnb + 5), hn00.y, hn10.y, hn01.y, hn11.y);
  const float2 nn00 = mul(wn0, zn0), nn10 = mul(wn1, zn0), nn01 = mul(wn0, b), nn11 = mul(wn1, b);
  e[1].x = quad_sum(__ldg(nna + 1), nn00.x, nn10.x, nn01.x, nn11.x);
  e[1].y = quad_sum(__ldg(nnb + 1), nn00.y, nn10.y, nn01.y, nn11.y);
  const float2 nh00 = mul(wn0, zh0), nh10 = mul(wn1, zh0), nh01 = mul(wn0, zh1),
               nh11 = mul(wn1, zh1);
  e[2].x = quad_sum(__ldg(nha + 2), nh00.x, nh10.x, nh01.x, nh11.x);
  e[2].y = quad_sum(__ldg(nhb + 2), nh00.y, nh10.y, nh01.y, nh11.y);
  h[0].x = quad_sum(__ldg(nha + 3), nh00.x, nh10.x, nh01.x, nh11.x);
  h[0].y = quad_sum(__ldg(nhb + 3), nh00.y, nh10.y, nh01.y, nh11.y);
  const float2 hh00 = mul(wh0, zh0), hh10 = mul(wh1, zh0), hh01 = mul(wh0, zh1),
               hh11 = mul(wh1, zh1);
  h[1].x = quad_sum(__ldg(hha + 4), hh00.x, hh10.x, hh01.x, hh11.x);
  h[1].y = quad_sum(__ldg(hhb + 4), hh00.y, hh10.y, hh01.y, hh11.y);
}

// push_f32 of two particles
template <int PUSHER>
__device__ __forceinline__ float2 push_pair(const PairConst &K, const float2 e[3],
                                            const float2 h[3], float2 u[3]) {
  const float2 one = K.one;
  if constexpr (PUSHER == 1) {
    float2 vel[3], bb[3], nb[3], vt[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      vt[j] = mul(u[j], K.c);
      bb[j] = mul(h[j], K.vay_b);
      nb[j] = neg(bb[j]);
      vel[j] = fma2(e[j], K.vay_e, vt[j]);
    }
    float2 gm = rsqrt2(fma2(sq2(vt), K.inv_c2, one));
    vel[0] = fma2(gm, fma2(vt[1], bb[2], mul(vt[2], nb[1])), vel[0]);
    vel[1] = fma2(gm, fma2(vt[2], bb[0], mul(vt[0], nb[2])), vel[1]);
    vel[2] = fma2(gm, fma2(vt[0], bb[1], mul(vt[1], nb[0])), vel[2]);
    // alpha = 1 / gamma^2 of the new velocity
    float2 alpha = fma2(sq2(vel), K.inv_c2, one);
    const float2 B2 = sq2(bb);
    float2 sg = fma2(B2, K.m1, alpha);
    const float2 vb = in2(vel, bb);
    const float2 d = fma2(sg, sg, mul(K.four, fma2(vb, vb, B2)));
    alpha = rsqrt2(mul(K.half, add(sg, make_float2(sqrtf(d.x), sqrtf(d.y)))));
#pragma unroll
    for (int j = 0; j < 3; j++) {
      bb[j] = mul(bb[j], alpha);
      nb[j] = neg(bb[j]);
    }
    sg = mul(rcp2(dot2(bb, bb, one)), K.inv_c);
    alpha = in2(vel, bb);
    u[0] = mul(sg, fma2(alpha, bb[0], fma2(bb[2], vel[1], fma2(nb[1], vel[2], vel[0]))));
    u[1] = mul(sg, fma2(alpha, bb[1], fma2(bb[0], vel[2], fma2(nb[2], vel[0], vel[1]))));
    u[2] = mul(sg, fma2(alpha, bb[2], fma2(bb[1], vel[0], fma2(nb[0], vel[1], vel[2]))));
    return rsqrt2(dot2(u, u, one));
  } else {
  float2 um[3], tb[3], nt[3];
#pragma unroll
  for (int j = 0; j < 3; j++) um[j] = fma2(K.ke, e[j], u[j]);
  float2 kg = K.kb;
  if (PUSHER == 0) kg = mul(kg, rsqrt2(dot2(um, um, one)));
#pragma unroll
  for (int j = 0; j < 3; j++) {
    tb[j] = mul(h[j], kg);
    nt[j] = neg(tb[j]);
  }
  const float2 c2 = mul(K.two, rcp2(dot2(tb, tb, one)));
  const float2 w0 = fma2(um[1], tb[2], fma2(um[2], nt[1], um[0]));
  const float2 w1 = fma2(um[2], tb[0], fma2(um[0], nt[2], um[1]));
  const float2 w2 = fma2(um[0], tb[1], fma2(um[1], nt[0], um[2]));
  u[0] = fma2(K.ke, e[0], fma2(c2, fma2(w1, tb[2], mul(w2, nt[1])), um[0]));
  u[1] = fma2(K.ke, e[1], fma2(c2, fma2(w2, tb[0], mul(w0, nt[2])), um[1]));
  u[2] = fma2(K.ke, e[2], fma2(c2, fma2(w0, tb[1], mul(w1, nt[0])), um[2]));
  return PUSHER == 0 ? rsqrt2(dot2(u, u, one)) : one;
  }
}


// One-warp CTAs (loop control and addresses are then warp-uniform: 1.30 against
// 1.44 ms with two warps), 16 per SM at 128 registers: 18 or 20 per SM take 96
// registers, and the spills cost more than the warps hide (1.31, 1.16 against
// 1.12 ms per 64-ppc wake step).
constexpr int PAIR_THREADS = 32, PAIR_BLOCKS = 16;
constexpr int PAIR_MAX = 2;  // pairs per lane of a chunk

// Particles whose step leaves its cell (at the mid-step or the end), meets a
// wall or moves by more than a fifth of its radius: left as they were and kept
// here until there are 32 of them, so that the scalar form of the whole step
// runs with full warps however few they are.
struct SlowQueue {
  static constexpr int CAP = 31 + 64 * PAIR_MAX;  // a chunk adds at most all of its particles
  int p[CAP];
  int count;
};

// the scalar step of the last min(32, count) entries, one per lane, deposits
// straight into J
template <int PUSHER>
static __device__ __noinline__ void queue_drain(const GridDev &g, const SpeciesF32 &s,
                                                SlowQueue &Q) {
  const int lane = threadIdx.x & 31, n = Q.count, e = n - 1 - lane, ncz = g.nz - 1;
  if (e >= 0) {
    const int p = Q.p[e];
    const int c = s.cell[p], i = row_of(g, c), k = c - i * ncz;
    const float a = s.fr[p], b = s.fz[p];
    float u[3] = {s.ur[p], s.uphi[p], s.uz[p]};
    int ir, kz;
    float wrh0, wrh1, wrn0, wrn1, wzh0, wzh1;
    weights_rhalf(i, a, ir, wrh0, wrh1);
    weights_rnode(i, a, wrn0, wrn1);
    weights_zhalf(k, b, kz, wzh0, wzh1);
    const float wzn0 = 1.0f - b, wzn1 = b;
    const auto quad = [&](int row, int col, int comp, float w0, float w1, float z0, float z1) {
      const float4 v = __ldg(g.q32 + 6 * (size_t)(row * ncz + col) + comp);
      return z0 * (v.x * w0 + v.y * w1) + z1 * (v.z * w0 + v.w * w1);
    };
    const float ef[3] = {quad(ir, k, 0, wrh0, wrh1, wzn0, wzn1),
                         quad(i, k, 1, wrn0, wrn1, wzn0, wzn1),
                         quad(i, kz, 2, wrn0, wrn1, wzh0, wzh1)};
    const float hf[3] = {quad(i, kz, 3, wrn0, wrn1, wzh0, wzh1),
                         quad(ir, kz, 4, wrh0, wrh1, wzh0, wzh1),
                         quad(ir, k, 5, wrh0, wrh1, wzn0, wzn1)};
    const float inv_g = push_f32(s, PUSHER, ef, hf, u);
    float an, bn;
    int in, kn;
    bool alive_now;
    DepDirect dep;
    move_deposit_f32(g, s, dep, i, k, a, b, s.w[p], inv_g, u, in, kn, an, bn, alive_now);
    if (s.alive) s.alive[p] = alive_now ? 1 : 0;
    s.cell[p] = in * ncz + kn;
    s.fr[p] = an;
    s.fz[p] = bn;
    s.ur[p] = u[0];
    s.uphi[p] = u[1];
    s.uz[p] = u[2];
  }
  __syncwarp();
  if (lane == 0) Q.count = n > 32 ? n - 32 : 0;
  __syncwarp();
}

// Deposits on their way to J: a cell's eight values per lane, in GridDev::j8's
// order.
struct DepList {
  float v[32][8];
  int cell[32];
};

// Adds each lane's values v of a cell (if `some`) into the cells' FP64 sums:
// every lane of the warp calls it; eight lanes take one cell's values, so that
// an atomic instruction touches 8 sectors, not 32.
__device__ __forceinline__ void list_add(const GridDev &g, DepList &L, int lane, bool some,
                                         int cell, const float v[8]) {
  const unsigned mask = __ballot_sync(0xffffffffu, some);
  if (mask == 0) return;
  if (some) {
    const int e = __popc(mask & ((1u << lane) - 1u));
    L.cell[e] = cell;
    *reinterpret_cast<float4 *>(&L.v[e][0]) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4 *>(&L.v[e][4]) = make_float4(v[4], v[5], v[6], v[7]);
  }
  __syncwarp();
  const int n8 = 8 * __popc(mask);
#pragma unroll 2
  for (int q = lane; q < n8; q += 32)
    atomicAdd(g.j8 + 8 * (size_t)(unsigned)L.cell[q >> 3] + (q & 7), (double)L.v[q >> 3][q & 7]);
  __syncwarp();
}

// A chunk's state in shared memory, each lane's 2 `pairs` particles in the
// lane's own 8 or 16 bytes per array: cell, fr, fz, ur, uphi, uz, w.  Only the
// lane itself reads and writes them, so no barrier stands between a copy and
// its use.  With two pairs, every second group of eight lanes steps its second
// pair first: a half warp's 8-byte accesses then fall on 32 different banks.
struct PairStage {
  float v[7][32 * 2 * PAIR_MAX];
};

__device__ __forceinline__ void copy_async(float *dst, const void *src, bool wide) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (wide)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

// Starts the copy of this lane's particles [p0, p0 + m) (all 2 `pairs` of them
// with asynchronous copies of 8 or 16 bytes: p0 is a multiple of that and every
// array starts a device allocation; fewer one by one) and commits it.
__device__ __forceinline__ void stage_start(PairStage &S, const SpeciesF32 &s, int p0,
                                            int m, int pairs, int lane) {
  const void *src[7] = {s.cell + p0, s.fr + p0, s.fz + p0, s.ur + p0,
                        s.uphi + p0, s.uz + p0, s.w + p0};
  if (m == 2 * pairs) {
#pragma unroll
    for (int j = 0; j < 7; j++) copy_async(&S.v[j][2 * pairs * lane], src[j], pairs == 2);
  } else {
    for (int e = 0; e < m; e++)
#pragma unroll
      for (int j = 0; j < 7; j++) S.v[j][2 * pairs * lane + e] = ((const float *)src[j])[e];
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// The staged results of this lane's particles back to s
__device__ __forceinline__ void stage_store(const PairStage &S, const SpeciesF32 &s, int p0,
                                            int m, int pairs, int lane) {
  float *const dst[6] = {nullptr, s.fr, s.fz, s.ur, s.uphi, s.uz};
  if (m == 4) {
#pragma unroll
    for (int j = 1; j < 6; j++)
      *reinterpret_cast<float4 *>(dst[j] + p0) =
          *reinterpret_cast<const float4 *>(&S.v[j][2 * pairs * lane]);
  } else if (m == 2) {
#pragma unroll
    for (int j = 1; j < 6; j++)
      *reinterpret_cast<float2 *>(dst[j] + p0) =
          *reinterpret_cast<const float2 *>(&S.v[j][2 * pairs * lane]);
  } else {
    for (int e = 0; e < m; e++)
#pragma unroll
      for (int j = 1; j < 6; j++) dst[j][p0 + e] = S.v[j][2 * pairs * lane + e];
  }
}

// The particle phase of one species.  A lane steps `pairs` pairs of
// consecutive particles of a chunk while the warp's next chunk is copied into
// shared memory; one segmented warp sum per chunk then adds the lanes' runs
// into the cells' FP64 deposits.  ALIVE: the species has alive flags.
// Bound by issue and by the latency of the quads' loads: 295 warp instructions
// per 32 particles (about 600 one particle at a time), issue 54% busy, the L1
// data path 58%, DRAM 45% of the measured copy.  67M particles at 64 per cell:
// 1.66 -> 1.15 ms per step while they are sorted by cell (HBM floor 0.54 ms),
// 2.15-2.33 -> 1.31-1.43 ms after 400-1600 steps; 268M particles with Vay and a
// re-sort in 20 steps: 7.29 -> 5.32 ms; 1M particles: 47.6 -> 42 us, 59-70 ->
// 50-52 us unsorted.
// What the parts measured on the sorted 67M: packed pairs alone 1.55; the queue
// instead of a call per slow particle 1.30 (one-warp CTAs); the staged copies
// 1.20; running sums in registers and the staging without bank conflicts 1.17;
// a cell's quads side by side 1.12; the cells' deposits instead of atomics into
// the three J grids 1.15, but 1.31-1.43 instead of 1.48-1.69 unsorted.
template <bool ALIVE, int PUSHER>
__global__ void __launch_bounds__(PAIR_THREADS, PAIR_BLOCKS)
    k_push_deposit_f32(const __grid_constant__ GridDev g, const __grid_constant__ SpeciesF32 s,
                       const __grid_constant__ PairConst K, int pairs) {
  __shared__ SlowQueue queue;
  __shared__ __align__(16) PairStage stage[2];
  __shared__ __align__(16) DepList list;
  const int lane = threadIdx.x, ncz = g.nz - 1;
  if (lane == 0) queue.count = 0;
  __syncwarp();
  const int chunk = 64 * pairs, n = (int)s.n, nchunks = (n + chunk - 1) / chunk;
  const unsigned cells = (unsigned)(g.nr - 1) * (unsigned)ncz;
  // this lane's particles of chunk ch: [p0, p0 + m)
  int p0 = (int)blockIdx.x * chunk + 2 * pairs * lane;
  int m = max(0, min(2 * pairs, n - p0));
  stage_start(stage[0], s, p0, m, pairs, lane);
  const int swap = pairs == 2 && (lane & 8) ? 2 : 0;
  int buf = 0;
  for (int ch = blockIdx.x; ch < nchunks; ch += gridDim.x, buf ^= 1) {
    const int p1 = p0 + (int)gridDim.x * chunk;
    const int m1 = max(0, min(2 * pairs, n - p1));
    stage_start(stage[buf ^ 1], s, p1, m1, pairs, lane);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    PairStage &S = stage[buf];
    // the lane's running sums of its first particle's cell, in j8's order
    int run = -1;
    float sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (int j0 = 0; j0 < 2 * pairs; j0 += 2) {
      const int jp = j0 ^ swap;
      const int p = p0 + jp;
      const int e0 = 2 * pairs * lane + jp;
      bool live_a = jp < m, live_b = jp + 1 < m;
      if (ALIVE) {
        live_a = live_a && s.alive[p] != 0;
        live_b = live_b && s.alive[p + 1] != 0;
        if (!__any_sync(0xffffffffu, live_a || live_b)) continue;
      }
      const auto load = [&](int j) { return *reinterpret_cast<const float2 *>(&S.v[j][e0]); };
      const float2 cf = load(0);
      int2 c = make_int2(__float_as_int(cf.x), __float_as_int(cf.y));
      // what a skipped particle computes beside the others is not used: it only
      // needs a cell whose fields it can read
      if (!live_a) c.x = 0;
      if (!live_b) c.y = 0;
      if (max((unsigned)c.x, (unsigned)c.y) >= cells) {
        flag32(g, ERR_OUT_OF_GRID);
        live_a = live_a && (unsigned)c.x < cells;
        live_b = live_b && (unsigned)c.y < cells;
        if (!live_a) c.x = 0;
        if (!live_b) c.y = 0;
      }
      float2 a = load(1), b = load(2);
      float2 u[3] = {load(3), load(4), load(5)};
      const int2 i = make_int2(row_of(g, c.x), row_of(g, c.y));
      const int2 k = make_int2(c.x - i.x * ncz, c.y - i.y * ncz);
      const float2 fi = make_float2((float)i.x, (float)i.y);
      const float4 Ra = __ldg(g.row32 + i.x), Rb = __ldg(g.row32 + i.y);
      float2 e[3], h[3];
      gather_pair(g, K, c, i, k, fi, a, b, Ra, Rb, e, h);
      const float2 rx = make_float2(Ra.x, Rb.x), ry = make_float2(Ra.y, Rb.y);
      const float2 ig = push_pair<PUSHER>(K, e, h, u);
      if ((live_a && !(ig.x == ig.x)) || (live_b && !(ig.y == ig.y))) flag32(g, ERR_NAN);
      // read again rather than kept in registers over the push
      asm volatile("" ::: "memory");
      a = load(1);
      b = load(2);
      // ---- half moves and rz rotations in cells (move_deposit_f32's, for a
      // particle that stays in its cell)
      const float2 vg = mul(ig, K.cr);
      const float2 dr_h = mul(u[0], vg), dy = mul(u[1], vg);
      const float2 dz_h = mul(u[2], mul(ig, K.cz));
      const float2 dy2 = mul(dy, dy);
      const float2 xa = add(a, dr_h), x = add(fi, xa);
      const float2 t1 = fma2(x, x, dy2), inv1 = rsqrt2(t1);
      const float2 a1 = fma2(dy2, rcp2(fma2(t1, inv1, x)), xa);
      const float2 b1 = add(b, dz_h);
      const float2 xa2 = add(a1, dr_h), bn = add(b1, dz_h);
      const float2 x2 = add(fi, xa2);
      const float2 t2 = fma2(x2, x2, dy2), inv2 = rsqrt2(t2);
      const float2 an = fma2(dy2, rcp2(fma2(t2, inv2, x2)), xa2);
      const float2 dro = fma2(a, K.m1, an), dze = fma2(b, K.m1, bn);
      const float2 fm = mul(K.half, add(a, an));
      const float2 irm = rcp2(add(fi, fm));
      const float2 hd = mul(K.half, dro), sh = mul(hd, irm), s2 = mul(sh, sh);
      // the end and the mid-step point in (0, 1] in both directions, the wall
      // cells' limits, and a short enough radial move
      const auto in_cell = [&](float xf, float a1f, float b1f, float xa2f, float bnf, float anf,
                               float s2f) {
        return fminf(fminf(fminf(a1f, b1f), fminf(xa2f, bnf)), xf) > 0.0f &&
               fmaxf(fmaxf(a1f, b1f), fmaxf(anf, bnf)) <= 1.0f && s2f < 0.01f;
      };
      bool ok_a = in_cell(x.x, a1.x, b1.x, xa2.x, bn.x, an.x, s2.x);
      bool ok_b = in_cell(x.y, a1.y, b1.y, xa2.y, bn.y, an.y, s2.y);
      if (max((unsigned)(i.x - 1), (unsigned)(i.y - 1)) >= (unsigned)(g.nr - 3) ||
          max((unsigned)(k.x - 1), (unsigned)(k.y - 1)) >= (unsigned)(g.nz - 3)) {
        const auto off_wall = [&](int ic, int kc, float xa2f, float bnf) {
          return (ic > 0 || xa2f >= 0.5f) && (ic < g.nr - 2 || xa2f <= 0.5f) &&
                 (kc > 0 || bnf >= 0.5f) && (kc < g.nz - 2 || bnf <= 0.5f);
        };
        ok_a = ok_a && off_wall(i.x, k.x, xa2.x, bn.x);
        ok_b = ok_b && off_wall(i.y, k.y, xa2.y, bn.y);
      }
      const bool do_a = live_a && ok_a, do_b = live_b && ok_b;
      if (live_a && !ok_a) queue.p[atomicAdd(&queue.count, 1)] = p;
      if (live_b && !ok_b) queue.p[atomicAdd(&queue.count, 1)] = p + 1;
      // ---- deposits, in j8's order
      const float2 w = load(6);
      const float2 fi2 = add(fi, fi);
      float2 v[8];
      {
        // azimuthal current at the mid-step point (src/particles.cpp:688-784)
        const float2 pre = mul(mul(mul(K.kphi, w), mul(u[1], ig)), inv1);
        const float2 q = add(fi2, a1);
        const float2 wa = mul(mul(fma2(a1, K.m1, K.one), q), mul(rx, pre));
        const float2 wb = mul(mul(a1, add(q, K.one)), mul(ry, pre));
        const float2 g0 = fma2(b1, K.m1, K.one);
        v[0] = mul(g0, wa);
        v[2] = mul(g0, wb);
        v[4] = mul(b1, wa);
        v[7] = mul(b1, wb);
      }
      {
        // r-z current of the one piece (piece_values; row 0 needs no case of
        // its own: 2 R.x = 8 there and fi (fi + 1) = 0)
        const float2 eps = mul(s2, fma2(s2, fma2(s2, fma2(s2, K.ninth, K.seventh), K.fifth),
                                        K.third));
        const float2 ii = fma2(fi, fi, fi), iie = mul(ii, eps);
        const float2 dzi = mul(dze, irm), kzw = mul(mul(K.kz2, w), dzi);
        const float2 q = add(fi2, fm);
        v[1] = mul(mul(kzw, rx), fma2(fma2(fm, K.m1, K.one), q, iie));
        v[3] = mul(mul(kzw, ry), fma2(iie, K.m1, mul(fm, add(q, K.one))));
        const float2 hh = mul(K.half, ii);
        const float2 q1 = mul(dro, mul(rcp2(add(fi, a)), inv2));
        const float2 beta = fma2(b, K.m1, K.one);
        const float2 q23 = mul(dzi, fma2(hd, inv2, eps));
        const float2 kr = mul(mul(K.kr, w), rcp2(add(fi, K.half)));
        const float2 in_r = fma2(hh, q1, hd);
        const float2 sub = fma2(mul(K.half, hd), dze, mul(hh, q23));
        const float2 lo = fma2(sub, K.m1, mul(beta, in_r));
        v[6] = mul(kr, lo);
        v[5] = mul(kr, fma2(lo, K.m1, in_r));
      }
      // A particle of the run's cell joins it; another one (a cell boundary, or
      // an unsorted particle among sorted ones) goes to J by itself.
      if (run < 0) run = do_a ? c.x : (do_b ? c.y : -1);
      const bool in_a = do_a && c.x == run, in_b = do_b && c.y == run;
      if (in_a && in_b) {
#pragma unroll
        for (int j = 0; j < 8; j++) sum[j] += v[j].x + v[j].y;
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++) sum[j] += (in_a ? v[j].x : 0.0f) + (in_b ? v[j].y : 0.0f);
      }
      // back_velocity_to_rz (src/particles.cpp:1005-1015): cos = x/r, sin = y/r
      const float2 st = mul(dy, inv2), ct = mul(x2, inv2);
      const float2 n0 = fma2(ct, u[0], neg(mul(st, u[1]))), n1 = fma2(st, u[0], mul(ct, u[1]));
      const float2 r[5] = {an, bn, n0, n1, u[2]};
      if (do_a && do_b) {
#pragma unroll
        for (int j = 0; j < 5; j++) *reinterpret_cast<float2 *>(&S.v[1 + j][e0]) = r[j];
      } else if (do_a) {
#pragma unroll
        for (int j = 0; j < 5; j++) S.v[1 + j][e0] = r[j].x;
      } else if (do_b) {
#pragma unroll
        for (int j = 0; j < 5; j++) S.v[1 + j][e0 + 1] = r[j].y;
      }
      float w8[8];
#pragma unroll
      for (int j = 0; j < 8; j++) w8[j] = v[j].x;
      list_add(g, list, lane, do_a && !in_a, c.x, w8);
#pragma unroll
      for (int j = 0; j < 8; j++) w8[j] = v[j].y;
      list_add(g, list, lane, do_b && !in_b, c.y, w8);
    }
    stage_store(S, s, p0, m, pairs, lane);
    p0 = p1;
    m = m1;
    __syncwarp();
    // ---- the warp's runs of lanes in one cell, summed into their last lane
    const unsigned FULL = 0xffffffffu;
    const int prev = __shfl_up_sync(FULL, run, 1), next = __shfl_down_sync(FULL, run, 1);
    const unsigned heads = __ballot_sync(FULL, lane == 0 || prev != run);
    const int start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    const int longest = __reduce_max_sync(FULL, lane - start);
#pragma unroll 1
    for (int off = 1; off <= longest; off <<= 1) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float y = __shfl_up_sync(FULL, sum[j], off);
        if (lane >= start + off) sum[j] += y;
      }
    }
    list_add(g, list, lane, (lane == 31 || next != run) && run >= 0, run, sum);
    while (queue.count >= 32) queue_drain<PUSHER>(g, s, queue);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (queue.count > 0) queue_drain<PUSHER>(g, s, queue);
}

// pairs per lane and CTAs of a launch over n particles; blocks_per_sm: a cap of
// that many 256-thread CTAs' worth per SM (0: as many as are resident)
static void launch_shape(long long n, int n_sm, int blocks_per_sm, int &pairs, int &blocks) {
  const long long slots = (long long)n_sm * PAIR_BLOCKS * PAIR_THREADS;
  // two pairs halve the warp sums once every warp still gets two chunks of them
  pairs = n >= 8 * slots ? 2 : 1;
  const long long b = (n + 2LL * PAIR_THREADS * pairs - 1) / (2LL * PAIR_THREADS * pairs);
  long long cap = (long long)n_sm * PAIR_BLOCKS;
  if (blocks_per_sm > 0) cap = std::min(cap, (long long)n_sm * blocks_per_sm * 256 / PAIR_THREADS);
  blocks = (int)std::min(b, cap);
}

// one kernel per pusher (0 relativistic Boris, 1 upstream Vay, 2 classic
// Boris), and one for species with alive flags
template <bool ALIVE>
static void launch_f32_kernel(const GridDev &g, const SpeciesF32 &s, int pusher, int n_sm,
                              int blocks_per_sm, cudaStream_t st) {
  int pairs, blocks;
  const PairConst K = pair_const(s);
  launch_shape(s.n, n_sm, blocks_per_sm, pairs, blocks);
  if (pusher == 1)
    k_push_deposit_f32<ALIVE, 1><<<blocks, PAIR_THREADS, 0, st>>>(g, s, K, pairs);
  else if (pusher == 2)
    k_push_deposit_f32<ALIVE, 2><<<blocks, PAIR_THREADS, 0, st>>>(g, s, K, pairs);
  else
    k_push_deposit_f32<ALIVE, 0><<<blocks, PAIR_THREADS, 0, st>>>(g, s, K, pairs);
}

// ---- the adjoint window's step: the scalar form, one particle at a time in
// the order and with the roundings that the window's gradients are compared
// on (the mean-field jump terms amplify the last bit of a trajectory).

// One thread of the CTA asks L2 for the input state of the CTA's next chunk
// (full chunks only: every prefetched byte lies inside the arrays).
__device__ __forceinline__ void prefetch_f32_chunk(const SpeciesF32 &s, long long next) {
  if ((next + 1) * F32_CHUNK > s.n) return;
  const long long q = next * F32_CHUNK;
  constexpr unsigned B4 = 4u * F32_CHUNK;
  prefetch_l2(s.cell + q, B4);
  prefetch_l2(s.fr + q, B4);
  prefetch_l2(s.fz + q, B4);
  prefetch_l2(s.ur + q, B4);
  prefetch_l2(s.uphi + q, B4);
  prefetch_l2(s.uz + q, B4);
  prefetch_l2(s.w + q, B4);
  if (s.alive) prefetch_l2(s.alive + q, F32_CHUNK);
}

template <bool OUT>
__global__ void __launch_bounds__(F32_THREADS, F32_MIN_BLOCKS)
    k_window_step_f32(GridDev g, SpeciesF32 s, SpeciesOut o) {
  const long long nchunks = (s.n + F32_CHUNK - 1) / F32_CHUNK;
  for (long long chunk = blockIdx.x; chunk < nchunks; chunk += gridDim.x) {
    if (threadIdx.x == 0) prefetch_f32_chunk(s, chunk + (long long)gridDim.x);
    f32_chunk<OUT, 0, true>(g, s, o, 0, chunk);
  }
}

// Bunch::bunch_inject in the cell-local form: z = dl * random_reverse(idx, 11)
// + dz/2 (computed in FP64 as upstream), v_z = v_beam (u_z = gamma v / c).
__device__ __forceinline__ void inject_slot_f32(const SpeciesF32 &s, long long idx, double dl,
                                                double half_dz, double dz, int ncz, float uz,
                                                const double *inv_pow11) {
  int int_vel = (int)floor((double)(unsigned)idx);
  double ost = 0, rr = 0;
  int order = 1;
  while (int_vel >= 1 && order < 40) {
    ost = int_vel % 11;
    rr = rr + ost * inv_pow11[order];
    int_vel = (int)((int_vel - ost) / 11);
    order = order + 1;
  }
  if (idx < s.n) {
    const double z = dl * rr + half_dz;
    int k = (int)ceil(z / dz) - 1;
    if (k < 0) k = 0;
    if (k > ncz - 1) k = ncz - 1;
    const int c = s.cell[idx];
    const int i = c / ncz;
    s.cell[idx] = i * ncz + k;
    s.fz[idx] = (float)(z / dz - k);
    s.uz[idx] = uz;
    s.alive[idx] = 1;
  }
}

__global__ void k_bunch_inject_f32(SpeciesF32 s, long long start, long long count, double dl,
                                   double half_dz, double dz, int ncz, float uz,
                                   const double *inv_pow11) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < count;
       j += (long long)gridDim.x * blockDim.x)
    inject_slot_f32(s, start + j, dl, half_dz, dz, ncz, uz, inv_pow11);
}

// the same with the schedule evaluated from the device time (a captured step)
__global__ void k_bunch_inject_f32_dev(SpeciesF32 s, const double *d_t, double begin, double end,
                                       double dt, unsigned pis, double dl, double half_dz,
                                       double dz, int ncz, float uz, const double *inv_pow11) {
  long long start, count;
  if (!inject_window(*d_t, begin, end, dt, pis, (unsigned)s.n, start, count)) return;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < count;
       j += (long long)gridDim.x * blockDim.x)
    inject_slot_f32(s, start + j, dl, half_dz, dz, ncz, uz, inv_pow11);
}

// cell-local FP32 state -> FP64 r, z, v (and w when w_out is given)
__global__ void k_cell_to_f64(SpeciesF32 s, double dr, double dz, int ncz, double *r, double *z,
                              double *vr, double *vphi, double *vz, double *w_out) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < s.n;
       p += (long long)gridDim.x * blockDim.x) {
    const int c = s.cell[p];
    const int i = c / ncz, k = c - (c / ncz) * ncz;
    r[p] = (i + (double)s.fr[p]) * dr;
    z[p] = (k + (double)s.fz[p]) * dz;
    const double ur = s.ur[p], up = s.uphi[p], uz = s.uz[p];
    const double c_over_g = LIGHT_SPEED / sqrt(1.0 + (ur * ur + up * up + uz * uz));
    vr[p] = ur * c_over_g;
    vphi[p] = up * c_over_g;
    vz[p] = uz * c_over_g;
    if (w_out) w_out[p] = s.w[p];
  }
}

// FP64 r, z, v (and w when given) -> cell-local FP32 state; a NaN position,
// a cell outside the grid or v >= c raises the matching error flag.
__global__ void k_f64_to_cell(SpeciesF32 s, const double *r, const double *z, const double *vr,
                              const double *vphi, const double *vz, const double *w_in,
                              double dr, double dz, int nr, int nz, unsigned *err) {
  const int ncz = nz - 1;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < s.n;
       p += (long long)gridDim.x * blockDim.x) {
    const double rp = r[p], zp = z[p];
    if (!isfinite(rp) || !isfinite(zp)) {
      atomicOr(err, ERR_NAN);
      continue;
    }
    int i = (int)ceil(rp / dr) - 1, k = (int)ceil(zp / dz) - 1;
    if (i < 0) i = 0;
    if (k < 0) k = 0;
    if (i > nr - 2 || k > nz - 2) {
      atomicOr(err, ERR_OUT_OF_GRID);
      i = min(i, nr - 2);
      k = min(k, nz - 2);
    }
    s.cell[p] = i * ncz + k;
    s.fr[p] = (float)(rp / dr - i);
    s.fz[p] = (float)(zp / dz - k);
    const double v2 = __dadd_rn(__dadd_rn(__dmul_rn(vr[p], vr[p]), __dmul_rn(vphi[p], vphi[p])),
                                __dmul_rn(vz[p], vz[p]));
    if (!(v2 < LIGHT_SPEED_POW_2)) {
      atomicOr(err, ERR_V_GE_C);
      continue;
    }
    const double gc = 1.0 / (LIGHT_SPEED * sqrt(1.0 - v2 / LIGHT_SPEED_POW_2));
    s.ur[p] = (float)(vr[p] * gc);
    s.uphi[p] = (float)(vphi[p] * gc);
    s.uz[p] = (float)(vz[p] * gc);
    if (w_in) ((float *)s.w)[p] = (float)w_in[p];
  }
}

void launch_cell_to_f64(const SpeciesF32 &s, double dr, double dz, int ncz, double *r, double *z,
                        double *vr, double *vphi, double *vz, double *w_out, cudaStream_t st) {
  if (s.n <= 0) return;
  long long blocks = (s.n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  k_cell_to_f64<<<(int)blocks, 256, 0, st>>>(s, dr, dz, ncz, r, z, vr, vphi, vz, w_out);
}

void launch_f64_to_cell(const SpeciesF32 &s, const double *r, const double *z, const double *vr,
                        const double *vphi, const double *vz, const double *w_in, double dr,
                        double dz, int nr, int nz, unsigned *err, cudaStream_t st) {
  if (s.n <= 0) return;
  long long blocks = (s.n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  k_f64_to_cell<<<(int)blocks, 256, 0, st>>>(s, r, z, vr, vphi, vz, w_in, dr, dz, nr, nz, err);
}

void launch_push_deposit_f32(const GridDev &g, const SpeciesF32 &s, int pusher, int n_sm,
                             int blocks_per_sm, cudaStream_t st) {
  // the kernel counts particles in 32 bits: a larger species in parts
  constexpr long long PART = 1LL << 30;
  for (long long q = 0; q < s.n; q += PART) {
    SpeciesF32 v = s;
    v.n = std::min(PART, s.n - q);
    v.cell += q;
    v.fr += q;
    v.fz += q;
    v.ur += q;
    v.uphi += q;
    v.uz += q;
    v.w += q;
    if (v.alive) {
      v.alive += q;
      launch_f32_kernel<true>(g, v, pusher, n_sm, blocks_per_sm, st);
    } else {
      launch_f32_kernel<false>(g, v, pusher, n_sm, blocks_per_sm, st);
    }
  }
}

void launch_window_step_f32(const GridDev &g, const SpeciesF32 &s, const SpeciesOut &o, int n_sm,
                            cudaStream_t st) {
  if (s.n <= 0) return;
  const long long chunks = (s.n + F32_CHUNK - 1) / F32_CHUNK;
  const int blocks = (int)std::min(chunks, (long long)n_sm * F32_MIN_BLOCKS);
  if (o.cell == s.cell)
    k_window_step_f32<false><<<blocks, F32_THREADS, 0, st>>>(g, s, o);
  else
    k_window_step_f32<true><<<blocks, F32_THREADS, 0, st>>>(g, s, o);
}

void launch_bunch_inject_f32(const SpeciesF32 &s, long long start, long long count, double dl,
                             double half_dz, double dz, int ncz, float uz,
                             const double *inv_pow11, cudaStream_t st) {
  if (count <= 0) return;
  long long blocks = (count + 255) / 256;
  if (blocks > 1024) blocks = 1024;
  k_bunch_inject_f32<<<(int)blocks, 256, 0, st>>>(s, start, count, dl, half_dz, dz, ncz, uz,
                                                  inv_pow11);
}

void launch_bunch_inject_f32_dev(const SpeciesF32 &s, const double *d_t, double begin,
                                 double end, double dt, unsigned pis, double dl, double half_dz,
                                 double dz, int ncz, float uz, const double *inv_pow11,
                                 cudaStream_t st) {
  if (pis == 0) return;
  long long blocks = ((long long)pis + 255) / 256;
  if (blocks > 1024) blocks = 1024;
  k_bunch_inject_f32_dev<<<(int)blocks, 256, 0, st>>>(s, d_t, begin, end, dt, pis, dl, half_dz,
                                                      dz, ncz, uz, inv_pow11);
}

}  // namespace pdp3g
