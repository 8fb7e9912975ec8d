// The fused BSSN right-hand side / RK stage kernel for sm_100a, behind the C
// ABI of include/bssn_b200.h. This header holds the kernel template and its
// host launch template; the instantiations are spread over the stream_*.cu
// translation units (declared in stream_launch.h) so that the library compiles
// in parallel.
//
// One persistent CTA of 512 threads per SM walks 256-point tiles. Two threads
// share each point, one of each role, so that the point's accumulators fit two
// 128-register threads and the SM holds 16 warps instead of 8:
//
//   geometry role (threads 0..255):    gt0..5 -> metric -> Gt0..2 -> chi -> alpha
//   transport role (threads 256..511): K, At0..5, B0..2, beta0..2, then the
//                                      closing algebra and the stores
//
// Each role stages its fields' haloed tiles into shared memory with cp.async
// (the transport role two fields ahead: its axial steps are shorter than a
// copy takes), differentiates them at its points and folds the derivatives
// into its accumulators at once; no derivative is written to memory. The
// geometry role hands its part of a point (24 values) to the transport role
// through shared memory and goes on with the next tile while the transport
// role closes this one.
//
// What bounds it: latency at 16 warps, then the shared-memory pipe (59 % of
// its wavefronts on a 102^3 array; 24 % of the FP64 pipe, 1.34 instructions a
// cycle). A 134^3 array, RK4 stage 1 with KO6: 2.30 ms for the one-thread-per-
// point form with 8 warps (255 registers), 1.69 ms now; RHS 2.00 -> 1.34 ms;
// constraints 1.69 -> 0.88 ms; KO order 8 3.42 -> 1.92 ms. Measured and not
// kept: two points a thread (256 threads, 255 registers; a quarter fewer
// instructions, but the 240 KB of code then waits for instruction fetches half
// of the time: 3.15 ms unrolled, 2.17 ms with one field loop for both roles);
// bulk row copies for the staging (2,540 cycles a box against 1,790 with
// cp.async and 1,650 with a tensor copy, which block pools cannot use).
//
// Stencils follow 3D/src/bssn3d/derivative_bundle.py:31-48 and
// common/src/mcs_common/derivatives.py:35-106: the centred sixth-order
// coefficients (integer sums of paired taps, scaled once), index clamped at
// the array ends, mixed second derivatives as a first derivative along the
// lower axis, then along the higher axis of that result.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "../../include/bssn_b200.h"
#include "host_util.h"
#include "stream.cuh"

namespace bssn {

constexpr int NTHREADS = 256;  // points per tile = threads per role

// A tile shape X x Y x Z (Z along the contiguous axis, X*Y*Z = 256).
template <int X_, int Y_, int Z_>
struct Shape {
  static constexpr int X = X_, Y = Y_, Z = Z_;
  static_assert(X_ * Y_ * Z_ == NTHREADS, "one point per thread of a role");
  static_assert(Z_ == 8 || Z_ == 16, "half-warps hold whole z rows");
};
using DefaultShape = Shape<4, 4, 16>;

enum Mode : int { MODE_RHS = 1, MODE_STAGE = 2, MODE_CON = 3, MODE_NORM = 4, MODE_MSRK = 5 };

struct Args {
  const double* F;  // stage input (24, n)
  const double* U;  // u_n (stage mode)
  double* ACC;      // accumulator (stage mode)
  double* OUT;      // RHS | next stage / new state | derivatives | constraints
  const double* S;  // 16 scalars (device)
  long long Sx, Sy, Sz, n;
  int ntx, nty, ntz;
  int stage;
  int use_ko;
  double ko_sigma;
  double chi_floor, alpha_floor;
  int ng;             // norm mode: ghost width of the interior
  double* partials;   // norm mode: [gridDim.x][2] per-CTA sums (scratch)
  const bssn_b200_block* blocks;  // batched mode: block table (device), else NULL
  int nblocks;
  int ntiles;         // batched mode: total tiles over all blocks
  double* OUT2;       // MSRK stage 0: partial Y3
  double* OUT3;       // MSRK stage 0: partial y_{n+1}
  double coef[9];     // MSRK: a20, a21, a30, a31, a32, b0, b1, b2, b3
  double ctime;       // MSRK: this stage's node (stage time t + ctime * dt)
};

// Stencil sums. The symmetric taps are paired first (v[+k] - v[-k] for the
// first derivative, v[+k] + v[-k] for the even stencils; the KO sum shares
// the second derivative's pairs), then combined with the integer coefficients
// of common/src/mcs_common/derivatives.py:35-49 from the outermost pair
// inwards, each step one fused multiply-add; the caller applies the scale
// factor. The reference forms sum_k (c_k / den * factor) * v_k
// (derivatives.py:78-88); the two orders differ by rounding only. The CPU
// oracle evaluates the same operations in the same order, so the derivatives
// match it bit for bit. v points at the centre tap, st is the tap stride.
__device__ __forceinline__ double c1_sum(double m3, double m2, double m1, double p1, double p2, double p3) {
  const double a1 = __dsub_rn(p1, m1), a2 = __dsub_rn(p2, m2), a3 = __dsub_rn(p3, m3);
  return __fma_rn(45.0, a1, __fma_rn(-9.0, a2, a3));
}
__device__ __forceinline__ double c2_sum(double v0, double s1, double s2, double s3) {
  return __fma_rn(-490.0, v0, __fma_rn(270.0, s1, __fma_rn(-27.0, s2, __dadd_rn(s3, s3))));
}
__device__ __forceinline__ double ko6_sum(double v0, double s1, double s2, double s3) {
  return __fma_rn(-20.0, v0, __fma_rn(15.0, s1, __fma_rn(-6.0, s2, s3)));
}
__device__ __forceinline__ double ko8_sum(double v0, double s1, double s2, double s3, double s4) {
  return __fma_rn(-70.0, v0, __fma_rn(56.0, s1, __fma_rn(-28.0, s2, __fma_rn(8.0, s3, -s4))));
}
// first-derivative sum of the 7 taps around p (stride st)
__device__ __forceinline__ double c1_at(const double* p, int st) {
  return c1_sum(p[-3 * st], p[-2 * st], p[-st], p[st], p[2 * st], p[3 * st]);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(double* smem, const double* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(smem)), "l"(gmem) : "memory");
}
// predicated without a branch
__device__ __forceinline__ void cp_async16_if(unsigned on, double* smem, const double* gmem) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}\n" ::"r"(
                   smem_addr(smem)),
               "l"(gmem), "r"(on)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
template <int ID, int N>
__device__ __forceinline__ void bar_sync() { asm volatile("bar.sync %0, %1;\n" ::"n"(ID), "n"(N) : "memory"); }
template <int ID, int N>
__device__ __forceinline__ void bar_arrive() { asm volatile("bar.arrive %0, %1;\n" ::"n"(ID), "n"(N) : "memory"); }

// named barriers: one per role for its field steps, three between the roles
enum : int { BAR_GEO = 1, BAR_TRA = 2, BAR_FULL = 3, BAR_FREE_GT = 4, BAR_FREE = 5, BAR_READY = 6 };

// Compile-time loop: body(std::integral_constant<int, I>) for I = B .. E-1, so
// that every per-field branch and register-array index is resolved statically.
template <int B, int E>
struct Unroll {
  template <class Body>
  __device__ __forceinline__ static void run(Body&& body) {
    body(std::integral_constant<int, B>{});
    Unroll<B + 1, E>::run(body);
  }
};
template <int E>
struct Unroll<E, E> {
  template <class Body>
  __device__ __forceinline__ static void run(Body&&) {}
};

// z pitch of staged rows: >= the row length and 8 mod 16 doubles, so the
// 16 threads of a half-warp (one or two z rows) hit 16 distinct bank pairs.
__host__ __device__ constexpr int zpitch(int len) { return len <= 8 ? 8 : ((len - 8 + 15) / 16) * 16 + 8; }

// Exchanged values of a point, geometry role -> transport role.
enum : int {
  X_GT = 0,      // 6: advection + KO of gt
  X_X = 6,       // 6: alpha R - D_iD_j alpha, the terms of the geometry role
  X_LAPA = 12,   // gt^ij D_iD_j alpha
  X_RG = 13,     // 3: its terms of Gt's rate, KO included
  X_RB = 16,     // 3: its terms of B's rate
  X_CAL = 19,    // 3: metric-computed contracted Christoffel symbol
  X_ALPHA = 22,  // advection + KO of alpha
  X_CHI = 23,    // advection + KO of chi, and the Ricci part of its damping
  X_N = 24,
  XC_TRR = 0, XC_MOM = 1, XC_N = 4  // constraints
};

template <int R, class T>
struct TileGeom {
  static constexpr int TX = T::X, TY = T::Y, TZ = T::Z;
  // Staged box: 3 halo points in x and y; in z a window of TZ + 8 that starts
  // 4 (or, at an odd z0, 3) points before the tile, so that its 16-byte pairs
  // are aligned. KO order 8 reads one more point along each axis: the z
  // window holds it, the x and y faces at distance 4 are extra rows.
  static constexpr int HX = TX + 6, HY = TY + 6, ZW = TZ + 8, NCH = ZW / 2;
  static constexpr int PZ = zpitch(ZW), SX = HY * PZ, SY = PZ;
  static constexpr int BOX = HX * HY, XF = R == 4 ? 2 * TY : 0, YF = R == 4 ? 2 * TX : 0;
  static constexpr int NROW = BOX + XF + YF;
  static constexpr int VOL = NROW * PZ;
  // mixed-derivative passes: d/dx sums over the y halo (and the z halo of the
  // central rows), d/dy sums over the z halo
  static constexpr int TP = TZ == 16 ? 24 : 14;
  static constexpr int T1Y = TY + 6, T1VOL = TX * T1Y * TP, T2VOL = TX * TY * TP, TVOL = T1VOL + T2VOL;
  // Their halo comes in columns, a thread a column: TX sums along x at every
  // cell of the y halo and of the z halo of the central rows, TY sums along y
  // at every cell of the z halo.
  static constexpr int NCA = 6 * TZ, NCB = 6 * TY, NCC = 6 * TX;
  static_assert(NCA + NCB + NCC <= NTHREADS, "a column a thread");
  static constexpr int RPP = NTHREADS / NCH, NPASS = (NROW + RPP - 1) / RPP;  // rows staged per pass, passes
  static constexpr size_t TABLES = (size_t)4 * NROW * sizeof(int);
  static constexpr size_t slots(int k) { return (size_t)k * NTHREADS * sizeof(double); }
  static constexpr size_t need(int nbuf, int nslot) {
    return (size_t)(nbuf * VOL + 2 * TVOL) * sizeof(double) + slots(X_N + nslot) + TABLES;
  }
  static constexpr size_t CAP = 232448 - 832;  // shared memory per CTA less the static part
  // The richest layout that fits: NB buffers of the transport role, and the
  // geometry role's own copy of the point values (PIPE, it runs up to a tile
  // ahead) or one copy for both roles. LEAN leaves At out of the point values
  // (read from global memory where it is used): of the geometry role's (LEAN_A)
  // or of both. In the order of the ladder, doubles per point in brackets:
  //   0  three buffers, LEAN_A (18 + 11)     KO <= 6: 4x4x16
  //   1  two buffers (18 + 17)               KO <= 6: 2x8x16
  //   2  two buffers, LEAN_A (18 + 11)       KO 8: 4x4x16, 2x8x16
  //   3  two buffers, LEAN (12 + 11)         KO <= 6: 4x8x8, 8x4x8
  //   4  two buffers, LEAN, one copy (12)    KO 8: 4x8x8, 8x4x8
  static constexpr int FIT = need(5, 18 + 11) <= CAP ? 0 : need(4, 18 + 17) <= CAP ? 1 : need(4, 18 + 11) <= CAP ? 2
                           : need(4, 12 + 11) <= CAP ? 3 : 4;
  static constexpr int NB = FIT == 0 ? 3 : 2;
  static constexpr bool PIPE = FIT <= 3, LEAN = FIT >= 3, LEAN_A = FIT != 1;
  static constexpr int NPB = LEAN ? 12 : 18, NPA = PIPE ? (LEAN_A ? 11 : 17) : 0;
  static constexpr size_t SMEM = need(2 + NB, NPB + NPA);
  static_assert(SMEM <= CAP, "tile does not fit shared memory");
};

struct TileDesc {
  long long base, n;      // first double of the block, points per field
  int sx, sy, sz, core;
  int x0, y0, z0, zs;     // first point of the tile, first staged z
  int al;                 // 16-byte row copies allowed
  double f1[3], f2[3], fk[3], fm[3];  // stencil scale factors (scales())
  double cahd;            // C dx^2 / (dt (10 dx^2 + 1))
  int tile0, tile_end;    // tiles of its block
};

// Scalars of the launch, in shared memory.
struct RunParams {
  double eta, lam0, lam1, lam2, lam3, lamf0, lamf1, dt, ssl;
};

// Scale factors of a grid or block; executed by one warp, a division a lane.
//   f1 = 1 / (60 h)           first derivative
//   f2 = 1 / (180 h h)        diagonal second derivative
//   fk = sigma / (64 h)       Kreiss-Oliger, order 6 (sigma / (256 h) for order 8)
//   fm = f1_i * f1_j          mixed second derivative, pairs xy, xz, yz
template <int R>
__device__ __forceinline__ void scales(TileDesc* d, double hx, double hy, double hz, double dx, double ko_sigma,
                                       double cahd_c, double dt, int lane) {
  const int a = lane % 3, kind = lane / 3;
  const double h = a == 0 ? hx : (a == 1 ? hy : hz), dx2 = dx * dx;
  const double num = kind == 2 ? ko_sigma : (kind == 3 ? cahd_c * dx2 : 1.0);
  const double den = kind == 0 ? 60.0 * h : (kind == 1 ? (180.0 * h) * h : (kind == 2 ? (R == 4 ? 256.0 : 64.0) * h : dt * (10.0 * dx2 + 1.0)));
  const double q = num / den;
  const double fi = __shfl_sync(0xffffffffu, q, a == 2 ? 1 : 0), fj = __shfl_sync(0xffffffffu, q, a == 0 ? 1 : 2);
  if (kind == 0) { d->f1[a] = q; d->fm[a] = fi * fj; }
  if (kind == 1) d->f2[a] = q;
  if (kind == 2) d->fk[a] = q;
  if (lane == 9) d->cahd = q;
}

// Fill the descriptor of one tile; executed by one warp. `from`: a filled
// descriptor of the same launch (its block and scale factors are reused while
// the block stays the same), or NULL.
template <int R, class T>
__device__ __forceinline__ void fill_desc(const Args& args, int tile, TileDesc* d, const TileDesc* from) {
  const int lane = threadIdx.x & 31;
  if (from && (!args.blocks || tile < from->tile_end)) {
    const double* a = from->f1;
    double* b = d->f1;
    if (lane < 13) b[lane] = a[lane];
    if (lane == 0) {
      d->base = from->base; d->n = from->n;
      d->sx = from->sx; d->sy = from->sy; d->sz = from->sz; d->core = from->core;
      d->tile0 = from->tile0; d->tile_end = from->tile_end;
    }
  } else {
    long long base = 0;
    int sx = (int)args.Sx, sy = (int)args.Sy, sz = (int)args.Sz, core = 0, tile0 = 0;
    double hx = args.S[13], hy = args.S[14], hz = args.S[15], dx = args.S[3];
    if (args.blocks) {
      int lo = 0, nb = args.nblocks;  // last block with tile0 <= tile, 32 ways a step
      while (nb > 1) {
        const int step = (nb + 31) >> 5, idx = lo + lane * step;
        const unsigned ok = __ballot_sync(0xffffffffu, idx < lo + nb && args.blocks[idx].tile0 <= tile);
        const int last = 31 - __clz(ok);
        lo += last * step;
        nb = min(step, nb - last * step);
      }
      const bssn_b200_block& bk = args.blocks[lo];
      base = bk.offset;
      sx = bk.sx; sy = bk.sy; sz = bk.sz;
      core = bk.core;
      tile0 = bk.tile0;
      hx = bk.h[0]; hy = bk.h[1]; hz = bk.h[2];
      dx = hx;
    }
    scales<R>(d, hx, hy, hz, dx, args.ko_sigma, args.S[1], args.S[2], lane);
    if (lane == 0) {
      d->base = base;
      d->n = (long long)sx * sy * sz;
      d->sx = sx; d->sy = sy; d->sz = sz; d->core = core;
      d->tile0 = tile0;
      d->tile_end = tile0 + ((sx - 2 * core + T::X - 1) / T::X) * ((sy - 2 * core + T::Y - 1) / T::Y) *
                                ((sz - 2 * core + T::Z - 1) / T::Z);
    }
  }
  if (lane == 0) {
    const int core = d->core, lt = tile - d->tile0;
    const int nty = (d->sy - 2 * core + T::Y - 1) / T::Y, ntz = (d->sz - 2 * core + T::Z - 1) / T::Z;
    const int t = lt / ntz, tz = lt - t * ntz, tx = t / nty, ty = t - tx * nty;
    d->x0 = core + tx * T::X;
    d->y0 = core + ty * T::Y;
    const int z0 = core + tz * T::Z;
    d->z0 = z0;
    const int zs = z0 - (R == 3 && (z0 & 1) ? 3 : 4);
    d->zs = zs;
    d->al = (d->sz & 1) == 0 && (d->base & 1) == 0 && (zs & 1) == 0 && (reinterpret_cast<uintptr_t>(args.F) & 15) == 0;
  }
}

// Place of staged row r relative to the tile: the box in C order, then (KO
// order 8) the x and y faces at distance 4.
template <int R, class T>
__device__ __forceinline__ void row_place(int r, int& dx, int& dy) {
  using G = TileGeom<R, T>;
  if (r < G::BOX) {
    dx = r / G::HY - 3;
    dy = r % G::HY - 3;
  } else if ((r -= G::BOX) < G::XF) {
    dx = r / T::Y ? T::X + 3 : -4;
    dy = r % T::Y;
  } else {
    r -= G::XF;
    dy = r / T::X ? T::Y + 3 : -4;
    dx = r % T::X;
  }
}

// Offset of every staged row's z = 0 in a field, the index clamped at the
// array ends (derivatives.py:83-84).
template <int R, class T>
__device__ __forceinline__ void fill_rows(const TileDesc& d, int* rows, int rt) {
  for (int r = rt; r < TileGeom<R, T>::NROW; r += NTHREADS) {
    int dx, dy;
    row_place<R, T>(r, dx, dy);
    rows[r] = (min(max(d.x0 + dx, 0), d.sx - 1) * d.sy + min(max(d.y0 + dy, 0), d.sy - 1)) * d.sz;
  }
}

// Thread rt stages the 16-byte pair rt % NCH of rows rt / NCH + RPP * pass.
struct StagePlace {
  int row0, ch;
  unsigned cross;  // bit p: the row of pass p lies in the axial cross
};
template <int R, class T>
__device__ __forceinline__ StagePlace stage_place(int rt) {
  using G = TileGeom<R, T>;
  StagePlace s;
  s.row0 = rt / G::NCH;
  s.ch = 2 * (rt % G::NCH);
  s.cross = 0;
  if (s.row0 >= G::RPP) s.row0 = G::NROW;  // idle
  for (int p = 0; p < G::NPASS; ++p) {
    const int r = s.row0 + p * G::RPP;
    if (r < G::NROW) {
      int dx, dy;
      row_place<R, T>(r, dx, dy);
      if (r >= G::BOX || (dx >= 0 && dx < T::X) || (dy >= 0 && dy < T::Y)) s.cross |= 1u << p;
    }
  }
  return s;
}

// Copies that stage one field's tile (ALL: every row; else the rows an axial
// stencil reads): pairs that are aligned and inside the array's z range
// (`whole`) as 16 bytes, others as two clamped 8-byte copies. src: the field
// at this thread's first staged z.
template <int R, class T, bool ALL>
__device__ __forceinline__ void stage_rows(double* buf, const double* __restrict__ src, const int* rows, const StagePlace& sp,
                                           bool whole, const TileDesc& d) {
  using G = TileGeom<R, T>;
  double* const to = buf + sp.row0 * G::PZ + sp.ch;
  rows += sp.row0;
  if (whole) {
#pragma unroll
    for (int p = 0; p < G::NPASS; ++p) {
      if (ALL && (p + 1) * G::RPP <= G::NROW) cp_async16(to + p * G::RPP * G::PZ, src + rows[p * G::RPP]);
      else cp_async16_if(ALL ? sp.row0 + p * G::RPP < G::NROW : sp.cross >> p & 1, to + p * G::RPP * G::PZ,
                         src + rows[min(p * G::RPP, G::NROW - 1 - sp.row0)]);
    }
  } else {
    const int z = d.zs + sp.ch;
    const int za = min(max(z, 0), d.sz - 1) - z, zb = min(max(z + 1, 0), d.sz - 1) - z;
#pragma unroll 1
    for (int p = 0; p < G::NPASS; ++p) {
      if (ALL ? sp.row0 + p * G::RPP < G::NROW : (sp.cross >> p & 1)) {
        const int o = rows[p * G::RPP];
        cp_async8(to + p * G::RPP * G::PZ, src + (o + za));
        cp_async8(to + p * G::RPP * G::PZ + 1, src + (o + zb));
      }
    }
  }
}

// Copies of the tile's point values, fields [0, NF) less SKIP, into slots
// [slot][point]: 16-byte pairs of points where they are aligned and inside the
// covered range, else every point's (clamped) value on its own. Every thread
// copies values that others read.
template <int NF, int SKIP, class T>
__device__ __forceinline__ void stage_points(double* slots, const double* __restrict__ F, const TileDesc& d, int rt) {
  constexpr int HP = NTHREADS / 2, TZ2 = T::Z / 2;
  const int pr = rt & (HP - 1), half = rt / HP;  // pair of points, parity of the field
  const int z = 2 * (pr % TZ2), y = pr / TZ2 % T::Y, x = pr / (TZ2 * T::Y);
  const int mx = d.sx - 1 - d.core, my = d.sy - 1 - d.core, mz = d.sz - 1 - d.core;
  const int gx = min(d.x0 + x, mx), gy = min(d.y0 + y, my), gz = d.z0 + z;
  const double* src = F + d.base + (long long)(gx * d.sy + gy) * d.sz;
  const long long n = d.n;
  double* to = slots + 2 * pr;
  constexpr int NS = SKIP < NF ? NF - 1 : NF;
  if (d.al && !(gz & 1) && gz + 1 <= mz) {
#pragma unroll
    for (int s = 0; s < NS; s += 2) {
      const int slot = s + half;
      if (s + 1 < NS || slot < NS) cp_async16(to + slot * NTHREADS, src + (slot < SKIP ? slot : slot + 1) * n + gz);
    }
  } else {
    const int za = min(gz, mz), zb = min(gz + 1, mz);
#pragma unroll 1
    for (int slot = half; slot < NS; slot += 2) {
      const double* f = src + (slot < SKIP ? slot : slot + 1) * n;
      cp_async8(to + slot * NTHREADS, f + za);
      cp_async8(to + slot * NTHREADS + 1, f + zb);
    }
  }
  cp_async_commit();
}

// Derivatives of one field at this thread's point.
struct Derivs {
  double s1[3], d2[6], ko;
};

// Per-thread constants of the derivative code.
struct PointPlace {
  int c;               // centre tap in a staged buffer, less the z shift
  int xm4, xp4, ym4, yp4;  // taps at distance 4 (KO order 8)
  int t1c, t2c;        // centre in T1 and T2
  int col, to;         // halo column: first source cell (z is 4 up) and first target
};

template <int R, class T>
__device__ __forceinline__ PointPlace point_place(int rt) {
  using G = TileGeom<R, T>;
  constexpr int TX = T::X, TY = T::Y, TZ = T::Z;
  const int lz = rt % TZ, ly = (rt / TZ) % TY, lx = rt / (TZ * TY);
  PointPlace p;
  p.c = (lx + 3) * G::SX + (ly + 3) * G::SY + lz;
  p.xm4 = lx >= 1 ? p.c - 4 * G::SX : (G::BOX + ly) * G::PZ + lz;
  p.xp4 = lx <= TX - 2 ? p.c + 4 * G::SX : (G::BOX + TY + ly) * G::PZ + lz;
  p.ym4 = ly >= 1 ? p.c - 4 * G::SY : (G::BOX + G::XF + lx) * G::PZ + lz;
  p.yp4 = ly <= TY - 2 ? p.c + 4 * G::SY : (G::BOX + G::XF + TX + lx) * G::PZ + lz;
  p.t1c = (lx * G::T1Y + ly + 3) * G::TP + lz + 3;
  p.t2c = (lx * TY + ly) * G::TP + lz + 3;
  // columns: the y halo on the first NCA threads, the z halos on the last
  int q = rt, k = q / TZ, z = q % TZ, y = k < 3 ? k - 3 : TY + k - 3;
  p.col = (y + 3) * G::SY + z + 4;
  p.to = (y + 3) * G::TP + z + 3;
  q = rt - (NTHREADS - G::NCB - G::NCC);
  if (q >= 0) {
    const bool along_y = q >= G::NCB;
    if (along_y) q -= G::NCB;
    k = q % 6;
    z = k < 3 ? k - 3 : TZ + k - 3;
    q /= 6;  // the column's y (along x) or x (along y)
    p.col = along_y ? (q + 3) * G::SX + z + 4 : (q + 3) * G::SY + z + 4;
    p.to = along_y ? G::T1VOL + q * TY * G::TP + z + 3 : (q + 3) * G::TP + z + 3;
  }
  return p;
}

// N first-derivative sums along a column of N + 6 cells.
template <int N>
__device__ __forceinline__ void column_sums(const double* __restrict__ p, int st, double* __restrict__ to, int tst) {
  double v[N + 6];
#pragma unroll
  for (int k = 0; k < N + 6; ++k) v[k] = p[k * st];
#pragma unroll
  for (int k = 0; k < N; ++k) to[k * tst] = c1_sum(v[k], v[k + 1], v[k + 2], v[k + 4], v[k + 5], v[k + 6]);
}

// One field's first-derivative sums s1 (unscaled), scaled second derivatives
// and KO term at this thread's point. WAIT: also wait for the point values.
// ROUND: the KO axes are added with a rounding each (the derivative bundle's
// stated arithmetic) instead of fused.
template <int R, class T, bool D2, bool KO, int BAR, bool WAIT, bool ROUND = false>
__device__ __forceinline__ void field_derivs(const double* __restrict__ cur, double* __restrict__ T1,
                                             const PointPlace& pp, const TileDesc& w,
                                             int rt, Derivs& d) {
  using G = TileGeom<R, T>;
  constexpr int st[3] = {G::SX, G::SY, 1};
  double* const T2 = T1 + G::T1VOL;
  const double* const v0p = cur + pp.c;
  const double v0 = v0p[0];
  d.ko = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double m1 = v0p[-st[a]], m2 = v0p[-2 * st[a]], m3 = v0p[-3 * st[a]];
    const double p1 = v0p[st[a]], p2 = v0p[2 * st[a]], p3 = v0p[3 * st[a]];
    const double s = c1_sum(m3, m2, m1, p1, p2, p3);
    d.s1[a] = s;
    if (D2 && a == 0) T1[pp.t1c] = s;  // this point's own sums; the halo's follow
    if (D2 && a == 1) T2[pp.t2c] = s;
    if (D2 || KO) {
      const double s1 = __dadd_rn(p1, m1), s2 = __dadd_rn(p2, m2), s3 = __dadd_rn(p3, m3);
      if (D2) d.d2[sym(a, a)] = __dmul_rn(c2_sum(v0, s1, s2, s3), w.f2[a]);
      if (KO) {
        double sk;
        if (R == 4) {
          const double m4 = a == 0 ? cur[pp.xm4] : (a == 1 ? cur[pp.ym4] : v0p[-4]);
          const double p4 = a == 0 ? cur[pp.xp4] : (a == 1 ? cur[pp.yp4] : v0p[4]);
          sk = ko8_sum(v0, s1, s2, s3, __dadd_rn(p4, m4));
        } else {
          sk = ko6_sum(v0, s1, s2, s3);
        }
        if (ROUND) d.ko = __dadd_rn(d.ko, __dmul_rn(sk, w.fk[a]));
        else d.ko = a == 0 ? __dmul_rn(sk, w.fk[a]) : __fma_rn(sk, w.fk[a], d.ko);
      }
    }
  }
  if (D2) {
    // T1 = unscaled d/dx sums over the y halo of the tile and over the z halo
    // of its own rows, T2 = unscaled d/dy sums over the z halo
    if (rt < G::NCA || (rt >= NTHREADS - G::NCB - G::NCC && rt < NTHREADS - G::NCC))
      column_sums<T::X>(cur + (pp.col - 4), G::SX, T1 + pp.to, G::T1Y * G::TP);
    else if (rt >= NTHREADS - G::NCC)
      column_sums<T::Y>(cur + (pp.col - 4), G::SY, T1 + pp.to, G::TP);
  }
  if (WAIT) cp_async_wait<1>();
  if (D2 || WAIT) bar_sync<BAR, NTHREADS>();
  if (D2) {
    d.d2[sym(0, 1)] = __dmul_rn(c1_at(T1 + pp.t1c, G::TP), w.fm[0]);
    d.d2[sym(0, 2)] = __dmul_rn(c1_at(T1 + pp.t1c, 1), w.fm[1]);
    d.d2[sym(1, 2)] = __dmul_rn(c1_at(T2 + pp.t2c, 1), w.fm[2]);
  }
}

__device__ __forceinline__ void inverse_metric(const double (&g)[6], double (&gu)[6]) {
  const double a00 = g[3] * g[5] - g[4] * g[4], a01 = g[2] * g[4] - g[1] * g[5], a02 = g[1] * g[4] - g[2] * g[3];
  const double a11 = g[0] * g[5] - g[2] * g[2], a12 = g[1] * g[2] - g[0] * g[4], a22 = g[0] * g[3] - g[1] * g[1];
  const double idet = 1.0 / (g[0] * a00 + g[1] * a01 + g[2] * a02);
  gu[0] = a00 * idet; gu[1] = a01 * idet; gu[2] = a02 * idet;
  gu[3] = a11 * idet; gu[4] = a12 * idet; gu[5] = a22 * idet;
}

// det^(-1/3) of the conformal metric, with pow(det, -1/3)'s values at zeros,
// infinities (inf, 0) and negative determinants (NaN). rcbrt and not pow: 0.50
// against 1.33 ulp of error over [1/8, 8] (and 36 over 2^+-300, as -1/3 is not a
// double), and a stage kernel with pow is slower (128^3 step 0.5 %, 49x56x64 with
// KO order 8 1.0 %, 96^3 RK4-2(2) step 1.5 %).
__device__ __forceinline__ double unit_det_scale(double det) {
  const double r = rcbrt(fabs(det));
  return det < 0.0 && r > 0.0 ? __longlong_as_double(0x7ff8000000000000LL) : r;
}

// Algebraic enforcement of one point (evolve.py:93-119): unit conformal
// determinant and traceless A~ with the unit-det inverse. v: gt, At. The one
// form of it: the stage kernels and the enforce entry give the same bytes.
__device__ __forceinline__ void enforce_metric(double (&v)[12]) {
  double* const g = v;
  double* const a = v + 6;
  const double det = g[0] * (g[3] * g[5] - g[4] * g[4]) - g[1] * (g[1] * g[5] - g[4] * g[2]) +
                     g[2] * (g[1] * g[4] - g[3] * g[2]);
  const double scale = unit_det_scale(det);
#pragma unroll
  for (int q = 0; q < 6; ++q) g[q] = g[q] * scale;
  const double iuxx = g[3] * g[5] - g[4] * g[4];
  const double iuxy = g[2] * g[4] - g[1] * g[5];
  const double iuxz = g[1] * g[4] - g[2] * g[3];
  const double iuyy = g[0] * g[5] - g[2] * g[2];
  const double iuyz = g[1] * g[2] - g[0] * g[4];
  const double iuzz = g[0] * g[3] - g[1] * g[1];
  const double trA = iuxx * a[0] + iuyy * a[3] + iuzz * a[5] + 2.0 * (iuxy * a[1] + iuxz * a[2] + iuyz * a[4]);
  const double third = trA / 3.0;
#pragma unroll
  for (int q = 0; q < 6; ++q) a[q] = a[q] - g[q] * third;
}

// fields of the two roles, in their order
template <bool CONS>
__host__ __device__ constexpr int geo_field(int i) {
  return i < 6 ? F_GT + i
       : CONS ? F_CHI
       : i < 9 ? F_GTI + i - 6
       : i == 9 ? F_CHI
       : F_ALPHA;
}
template <bool CONS>
__host__ __device__ constexpr int tra_field(int i) {
  return i == 0 ? F_K
       : i < 7 ? F_AT + i - 1
       : CONS ? F_GTI + i - 7
       : i < 10 ? F_B + i - 7
       : F_BETA + i - 10;
}

// KO: the Kreiss-Oliger terms are part of the rate (stage modes).
template <int R, int MODE, bool KO, class T = DefaultShape>
__global__ void __launch_bounds__(2 * NTHREADS, 1) stream_kernel(const __grid_constant__ Args args) {
  using G = TileGeom<R, T>;
  constexpr int TX = T::X, TY = T::Y, TZ = T::Z;
  constexpr bool CONS = MODE == MODE_CON || MODE == MODE_NORM;
  constexpr bool PIPE = G::PIPE, LEAN = G::LEAN, LEAN_A = G::LEAN_A;
  constexpr int NGEO = CONS ? 7 : 11, NTRA = CONS ? 10 : 13;
  constexpr int NB = G::NB, NBUF = 2 + NB;
  extern __shared__ __align__(128) double smem[];
  __shared__ TileDesc s_desc[2][2];
  __shared__ RunParams s_par;

  const int tid = threadIdx.x;
  const int role = tid >= NTHREADS;
  const int rt = tid & (NTHREADS - 1);
  double* const X = smem + NBUF * G::VOL + 2 * G::TVOL + rt;   // [X_N][256] exchanged values of this point
  double* const pB = X + X_N * NTHREADS;                    // [NPB][256] point values (state order)
  double* const pA = PIPE ? pB + G::NPB * NTHREADS : pB;    // [NPA][256] the geometry role's copy (without K)
  double* const tab = smem + NBUF * G::VOL + 2 * G::TVOL + (X_N + G::NPB + G::NPA) * NTHREADS;
  int* const rows = reinterpret_cast<int*>(tab) + role * 2 * G::NROW;
  double* const T1 = smem + NBUF * G::VOL + role * G::TVOL;
  double* cur = smem + role * 2 * G::VOL;  // staged field, and the ones in flight
  double* nxt = cur + G::VOL;
  double* far = cur + (NB - 1) * G::VOL;   // transport role: the buffer freed last step
  TileDesc* const desc = s_desc[role];

  const int ntiles = args.blocks ? args.ntiles : args.ntx * args.nty * args.ntz;
  int par = 0;
  // ---- prologue: first tile's descriptor, rows and first field -------------
  if ((tid & (NTHREADS - 1)) < 32) fill_desc<R, T>(args, blockIdx.x, &desc[0], nullptr);
  if (tid == 0) {
    const double* S = args.S;
    s_par.eta = S[0]; s_par.dt = S[2];
    s_par.lam0 = S[7]; s_par.lam1 = S[8]; s_par.lam2 = S[9]; s_par.lam3 = S[10];
    s_par.lamf0 = S[11]; s_par.lamf1 = S[12];
    // stage times t, t + dt/2, t + dt/2, t + dt (evolve.py:125-131) or the MSRK nodes (:139-153)
    double t = S[6];
    if (MODE == MODE_STAGE) t += (args.stage == 0 ? 0.0 : (args.stage == 3 ? 1.0 : 0.5)) * S[2];
    if (MODE == MODE_MSRK) t += args.ctime * S[2];
    s_par.ssl = S[4] * exp(-0.5 * t * t / (S[5] * S[5]));
  }
  __syncthreads();
  fill_rows<R, T>(desc[0], rows, rt);
  __syncthreads();
  const PointPlace place = point_place<R, T>(rt);
  const int lz = rt % TZ, ly = (rt / TZ) % TY, lx = rt / (TZ * TY);
  double norm_h = 0.0, norm_m = 0.0;

  const StagePlace splace = stage_place<R, T>(rt);
  // this thread's first staged z of the tile's field 0, and whether its pairs go as 16 bytes
  const double* Fz;
  unsigned nfield;
  bool whole, copies;
  auto aim = [&](const TileDesc& d) {
    const int z = d.zs + splace.ch;
    Fz = args.F + (d.base + z);
    nfield = (unsigned)d.n;
    whole = d.al && z >= 0 && z + 1 < d.sz;
    // The last covered point, sz - 1 - core, reads R further: pairs past that
    // stay as they are (inside the array they are copied all the same, so that
    // a margin of R or more needs no cells past its end).
    copies = splace.row0 < G::NROW && z < d.sz + max(R - d.core, 0);
  };
  using AllRows = std::true_type;
  using CrossRows = std::false_type;
  // issue the copies of `field` of the tile aimed at into buf
  auto issue = [&](auto all, const TileDesc& d, const int* rw, int field, double* buf) {
    if (copies)
      stage_rows<R, T, decltype(all)::value>(buf, Fz + (long long)field * nfield, rw, splace, whole, d);
    cp_async_commit();
  };
  aim(desc[0]);

  if (role == 0) {
    // ======================= geometry role =================================
    issue(AllRows{}, desc[0], rows, geo_field<CONS>(0), cur);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const TileDesc& d = desc[par];
      const bool has_next = tile + (int)gridDim.x < ntiles;
      auto fld = [&](int k) -> double {
        if (LEAN_A && k >= F_AT) {  // this point (one past the covered range: the nearest covered one)
          const int gx = min(d.x0 + lx, d.sx - 1 - d.core), gy = min(d.y0 + ly, d.sy - 1 - d.core),
                    gz = min(d.z0 + lz, d.sz - 1 - d.core);
          return __ldg(args.F + d.base + k * d.n + ((long long)(gx * d.sy + gy) * d.sz + gz));
        }
        return PIPE ? pA[(k < F_K ? k : k - 1) * NTHREADS] : pA[k * NTHREADS];
      };
      const int dz = d.z0 - d.zs;
      double gu[6], R_[6], C1[3][6], dchi[3], bf[3];  // C1 holds d_a gt_p until the metric is complete
      Unroll<0, NGEO>::run([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        constexpr int f = geo_field<CONS>(i);
        cp_async_wait<0>();
        bar_sync<BAR_GEO, NTHREADS>();
        if (i == 0 && PIPE) stage_points<LEAN_A ? 12 : 18, F_K, T>(pA - rt, args.F, d, rt);
        constexpr bool D2 = has_d2(f), N2 = i + 1 == NGEO || has_d2(geo_field<CONS>(i + 1 < NGEO ? i + 1 : i));
        if (i + 1 < NGEO) issue(std::integral_constant<bool, N2>{}, d, rows + par * G::NROW, geo_field<CONS>(i + 1), nxt);
        else if (has_next) {
          aim(desc[par ^ 1]);
          issue(AllRows{}, desc[par ^ 1], rows + (par ^ 1) * G::NROW, geo_field<CONS>(0), nxt);
        }
        if (has_next) {
          if (i == 0 && rt < 32) fill_desc<R, T>(args, tile + gridDim.x, &desc[par ^ 1], &d);
          if (i == 1) fill_rows<R, T>(desc[par ^ 1], rows + (par ^ 1) * G::NROW, rt);
        }
        Derivs v;
        field_derivs<R, T, D2, KO, BAR_GEO, i == 0 && PIPE>(cur + dz, T1, place, d, rt, v);
        {
          double* t = cur; cur = nxt; nxt = t;
        }
        if (i == 0) {
          if (!PIPE) bar_sync<BAR_READY, 2 * NTHREADS>();
          double g[6];
#pragma unroll
          for (int p = 0; p < 6; ++p) g[p] = fld(F_GT + p);
          inverse_metric(g, gu);
#pragma unroll
          for (int a = 0; a < 3; ++a) bf[a] = CONS ? 0.0 : fld(F_BETA + a) * d.f1[a];
          if (PIPE && tile != (int)blockIdx.x) bar_sync<BAR_FREE_GT, 2 * NTHREADS>();
        }
        double d1[3];  // scaled first derivatives; advection takes the sums and beta / (60 h)
#pragma unroll
        for (int a = 0; a < 3; ++a) d1[a] = __dmul_rn(v.s1[a], d.f1[a]);
        const double adv = bf[0] * v.s1[0] + bf[1] * v.s1[1] + bf[2] * v.s1[2];
        if (i < 6) {  // gt_p: first derivatives kept, second derivatives into R_p
          constexpr int p = i < 6 ? i : 0;
          if (!CONS) X[(X_GT + p) * NTHREADS] = adv + v.ko;
#pragma unroll
          for (int a = 0; a < 3; ++a) C1[a][p] = d1[a];
          double s = 0.0;
#pragma unroll
          for (int q = 0; q < 6; ++q) s += symw(q) * gu[q] * v.d2[q];
          R_[p] = -0.5 * s;
        }
        if (i == 5) {  // Christoffel symbols of the first kind and the quadratic Ricci terms
          double G1[3][6];
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int p = 0; p < 6; ++p) {
              const int a = sym_i(p), b = sym_j(p);
              G1[k][p] = 0.5 * (C1[a][sym(k, b)] + C1[b][sym(k, a)] - C1[k][p]);
            }
          double cl[3], cal[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            cl[k] = 0.0;
#pragma unroll
            for (int p = 0; p < 6; ++p) {
              C1[k][p] = G1[k][p];
              cl[k] += symw(p) * gu[p] * C1[k][p];
            }
          }
          if (PIPE && tile != (int)blockIdx.x) bar_sync<BAR_FREE, 2 * NTHREADS>();
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            cal[k] = gu[sym(k, 0)] * cl[0] + gu[sym(k, 1)] * cl[1] + gu[sym(k, 2)] * cl[2];
            if (!CONS) X[(X_CAL + k) * NTHREADS] = cal[k];
          }
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const int a = sym_i(p), b = sym_j(p);
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) s += cal[k] * (C1[a][sym(b, k)] + C1[b][sym(a, k)]);
            R_[p] += 0.5 * s;
          }
          // R_ij += G^k_li G_jk^l + G^k_lj G_ik^l + G^k_il G_kj^l, one k at a
          // time: with E = G^k gt^-1 the first two are E_i^q G_jqk and its
          // transpose, the third E_i^q G_kqj
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            double C2[6], E[3][3];
#pragma unroll
            for (int p = 0; p < 6; ++p)
              C2[p] = gu[sym(k, 0)] * C1[0][p] + gu[sym(k, 1)] * C1[1][p] + gu[sym(k, 2)] * C1[2][p];
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
              for (int q = 0; q < 3; ++q)
                E[m][q] = C2[sym(m, 0)] * gu[sym(0, q)] + C2[sym(m, 1)] * gu[sym(1, q)] + C2[sym(m, 2)] * gu[sym(2, q)];
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
              for (int j = 0; j < 3; ++j) {
                const double s = E[m][0] * C1[j][sym(0, k)] + E[m][1] * C1[j][sym(1, k)] + E[m][2] * C1[j][sym(2, k)];
                R_[sym(m, j)] += m == j ? 2.0 * s : s;
                if (m <= j)
                  R_[sym(m, j)] += E[m][0] * C1[k][sym(0, j)] + E[m][1] * C1[k][sym(1, j)] + E[m][2] * C1[k][sym(2, j)];
              }
          }
        }
        if (f >= F_GTI && f < F_B) {  // Gt^k: derivative terms of R and advection
          constexpr int k = f >= F_GTI && f < F_B ? f - F_GTI : 0;
          X[(X_RG + k) * NTHREADS] = adv + v.ko;
          X[(X_RB + k) * NTHREADS] = (1.0 - s_par.lam3) * adv;
          double g[3];
#pragma unroll
          for (int m = 0; m < 3; ++m) g[m] = fld(F_GT + sym(k, m));
#pragma unroll
          for (int p = 0; p < 6; ++p) R_[p] += 0.5 * (g[sym_i(p)] * d1[sym_j(p)] + g[sym_j(p)] * d1[sym_i(p)]);
        }
        if (f == F_CHI) {
          const double ichi = 1.0 / fld(F_CHI);
          const double rchi = adv + v.ko;
          double up[3], sq = 0.0, lap = 0.0;  // raised gradient
#pragma unroll
          for (int a = 0; a < 3; ++a) dchi[a] = d1[a];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            up[k] = gu[sym(k, 0)] * dchi[0] + gu[sym(k, 1)] * dchi[1] + gu[sym(k, 2)] * dchi[2];
            sq += up[k] * dchi[k];
          }
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            v.d2[p] = v.d2[p] - (C1[0][p] * up[0] + C1[1][p] * up[1] + C1[2][p] * up[2]);
            lap += symw(p) * gu[p] * v.d2[p];
          }
          const double hichi = 0.5 * ichi, qichi2 = 0.25 * ichi * ichi;
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const double g = fld(F_GT + p);
            R_[p] += hichi * (v.d2[p] + g * lap) - qichi2 * (dchi[sym_i(p)] * dchi[sym_j(p)] + 3.0 * g * sq);
          }
          double trR = 0.0;
#pragma unroll
          for (int p = 0; p < 6; ++p) trR += symw(p) * gu[p] * R_[p];
          if (!CONS) {
            const double chi = fld(F_CHI);
            X[X_CHI * NTHREADS] = rchi + d.cahd * chi * (chi * trR);
          } else {
            double A[6];
#pragma unroll
            for (int p = 0; p < 6; ++p) A[p] = fld(F_AT + p);
            X[XC_TRR * NTHREADS] = trR;
            // M_a = -gt^jk (G^m_ja A_km + 3/2 A_ka d_j chi / chi), with B = gt^-1 A gt^-1
            double M[3][3];  // M[j][m] = gt^jk A_km
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
              for (int m = 0; m < 3; ++m)
                M[j][m] = gu[sym(j, 0)] * A[sym(0, m)] + gu[sym(j, 1)] * A[sym(1, m)] + gu[sym(j, 2)] * A[sym(2, m)];
            double B[3][3];
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
              for (int m = 0; m < 3; ++m)
                B[j][m] = M[j][0] * gu[sym(0, m)] + M[j][1] * gu[sym(1, m)] + M[j][2] * gu[sym(2, m)];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
              double m = 0.0, c = 0.0;
#pragma unroll
              for (int j = 0; j < 3; ++j) {
                c += M[j][a] * dchi[j];
#pragma unroll
                for (int k = 0; k < 3; ++k) m += B[j][k] * C1[k][sym(j, a)];
              }
              X[(XC_MOM + a) * NTHREADS] = -m - 1.5 * c * ichi;
            }
          }
        }
        if (f == F_ALPHA) {  // D_iD_j alpha, the traces, and Gt's terms in A^ij
          const double al = fld(F_ALPHA), ichi = 1.0 / fld(F_CHI), hichi = 0.5 * ichi;
          X[X_ALPHA * NTHREADS] = s_par.lam0 * adv + v.ko;
          double up[3], gca = 0.0;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            up[k] = gu[sym(k, 0)] * d1[0] + gu[sym(k, 1)] * d1[1] + gu[sym(k, 2)] * d1[2];
            gca += up[k] * dchi[k];
          }
          double lapa = 0.0;
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const int a = sym_i(p), b = sym_j(p);
            const double dda = v.d2[p] - (C1[0][p] * up[0] + C1[1][p] * up[1] + C1[2][p] * up[2]) +
                               hichi * (d1[a] * dchi[b] + d1[b] * dchi[a] - fld(F_GT + p) * gca);
            lapa += symw(p) * gu[p] * dda;
            X[(X_X + p) * NTHREADS] = al * R_[p] - dda;
          }
          X[X_LAPA * NTHREADS] = lapa;
          double A[6], M[3][3], AU[6], w[3], t[3];
#pragma unroll
          for (int p = 0; p < 6; ++p) A[p] = fld(F_AT + p);
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j)
              M[k][j] = A[sym(k, 0)] * gu[sym(0, j)] + A[sym(k, 1)] * gu[sym(1, j)] + A[sym(k, 2)] * gu[sym(2, j)];
#pragma unroll
          for (int p = 0; p < 6; ++p)
            AU[p] = gu[sym(sym_i(p), 0)] * M[0][sym_j(p)] + gu[sym(sym_i(p), 1)] * M[1][sym_j(p)] +
                    gu[sym(sym_i(p), 2)] * M[2][sym_j(p)];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            w[k] = 2.0 * d1[k] + 3.0 * al * ichi * dchi[k];
            double s = 0.0;  // G_kij A^ij
#pragma unroll
            for (int p = 0; p < 6; ++p) s += symw(p) * C1[k][p] * AU[p];
            t[k] = 2.0 * al * s;
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const double r = gu[sym(k, 0)] * t[0] + gu[sym(k, 1)] * t[1] + gu[sym(k, 2)] * t[2] -
                             (AU[sym(k, 0)] * w[0] + AU[sym(k, 1)] * w[1] + AU[sym(k, 2)] * w[2]);
            X[(X_RG + k) * NTHREADS] += r;
            X[(X_RB + k) * NTHREADS] += r;
          }
        }
      });
      bar_arrive<BAR_FULL, 2 * NTHREADS>();
      par ^= 1;
    }
  } else {
    // ======================= transport role ================================
    issue(CrossRows{}, desc[0], rows, tra_field<CONS>(0), cur);
    if (NB == 3) issue(CrossRows{}, desc[0], rows, tra_field<CONS>(1), nxt);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const TileDesc& d = desc[par];
      const bool has_next = tile + (int)gridDim.x < ntiles;
      const long long n = d.n;
      long long gidx;
      bool inside;
      {
        const int gx = d.x0 + lx, gy = d.y0 + ly, gz = d.z0 + lz;
        const int mx = d.sx - 1 - d.core, my = d.sy - 1 - d.core, mz = d.sz - 1 - d.core;
        inside = gx <= mx && gy <= my && gz <= mz;
        gidx = d.base + ((long long)min(gx, mx) * d.sy + min(gy, my)) * d.sz + min(gz, mz);
      }
      auto fld = [&](int k) -> double { return k < G::NPB ? pB[k * NTHREADS] : __ldg(args.F + (gidx + k * n)); };
      const int dz = d.z0 - d.zs;
      double gu[6], bf[3], r_K, r_At[6], r_B[3], r_Gt[3], Rg[6], db[3][3], r_beta[3], mom[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) mom[a] = 0.0;
#pragma unroll
      for (int p = 0; p < 6; ++p) Rg[p] = 0.0;
      Unroll<0, NTRA>::run([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        constexpr int f = tra_field<CONS>(i);
        constexpr int LA = NB - 1, J = (i + LA) % NTRA;  // field issued now, LA steps ahead
        constexpr bool D2 = has_d2(f);
        using Rows = std::integral_constant<bool, has_d2(tra_field<CONS>(J))>;
        cp_async_wait<NB - 2>();
        bar_sync<BAR_TRA, NTHREADS>();
        if (i == 0) stage_points<G::NPB, 99, T>(pB - rt, args.F, d, rt);
        if (i + LA < NTRA) {
          issue(Rows{}, d, rows + par * G::NROW, tra_field<CONS>(J), far);
        } else if (has_next) {
          if (i + LA == NTRA) aim(desc[par ^ 1]);
          issue(Rows{}, desc[par ^ 1], rows + (par ^ 1) * G::NROW, tra_field<CONS>(J), far);
        } else {
          cp_async_commit();  // keeps the group count
        }
        if (has_next) {
          if (i == 0 && rt < 32) fill_desc<R, T>(args, tile + gridDim.x, &desc[par ^ 1], &d);
          if (i == 1) fill_rows<R, T>(desc[par ^ 1], rows + (par ^ 1) * G::NROW, rt);
        }
        Derivs v;
        field_derivs<R, T, D2, KO, BAR_TRA, i == 0>(cur + dz, T1, place, d, rt, v);
        if (NB == 3) {
          double* t = cur; cur = nxt; nxt = far; far = t;
        } else {
          double* t = cur; cur = nxt; nxt = t; far = t;
        }
        if (i == 0) {
          if (!PIPE) bar_sync<BAR_READY, 2 * NTHREADS>();
          double g[6];
#pragma unroll
          for (int p = 0; p < 6; ++p) g[p] = fld(F_GT + p);
          inverse_metric(g, gu);
#pragma unroll
          for (int a = 0; a < 3; ++a) bf[a] = CONS ? 0.0 : fld(F_BETA + a) * d.f1[a];
        }
        double d1[3];  // scaled first derivatives; advection takes the sums and beta / (60 h)
#pragma unroll
        for (int a = 0; a < 3; ++a) d1[a] = __dmul_rn(v.s1[a], d.f1[a]);
        const double adv = bf[0] * v.s1[0] + bf[1] * v.s1[1] + bf[2] * v.s1[2];
        if (f == F_K) {
          if (CONS) {
#pragma unroll
            for (int a = 0; a < 3; ++a) mom[a] -= (2.0 / 3.0) * d1[a];
          } else {
            r_K = adv + v.ko;
#pragma unroll
            for (int a = 0; a < 3; ++a)
              r_Gt[a] = -(4.0 / 3.0) * fld(F_ALPHA) *
                        (gu[sym(a, 0)] * d1[0] + gu[sym(a, 1)] * d1[1] + gu[sym(a, 2)] * d1[2]);
          }
        } else if (f >= F_AT && f < F_AT + 6) {
          constexpr int p = f >= F_AT && f < F_AT + 6 ? f - F_AT : 0;
          if (CONS) {
            // g~^jk d_j A~_ki, A~_ki = A~_p for {k, i} = pair p
            const int a = sym_i(p), k = sym_j(p);
            mom[a] += gu[sym(0, k)] * d1[0] + gu[sym(1, k)] * d1[1] + gu[sym(2, k)] * d1[2];
            if (a != k) mom[k] += gu[sym(0, a)] * d1[0] + gu[sym(1, a)] * d1[1] + gu[sym(2, a)] * d1[2];
          } else {
            r_At[p] = adv + v.ko;
          }
        } else if (f >= F_B) {
          constexpr int k = f >= F_B ? f - F_B : 0;
          r_B[k] = s_par.lam2 * adv + v.ko;
        } else if (f >= F_GTI) {  // (constraints) derivative terms of R
          constexpr int k = f >= F_GTI && f < F_B ? f - F_GTI : 0;
#pragma unroll
          for (int p = 0; p < 6; ++p)
            Rg[p] += 0.5 * (fld(F_GT + sym(k, sym_i(p))) * d1[sym_j(p)] + fld(F_GT + sym(k, sym_j(p))) * d1[sym_i(p)]);
        } else {
          constexpr int k = f >= F_BETA && f < F_AT ? f - F_BETA : 0;
          r_beta[k] = s_par.lam1 * adv + v.ko;
          double lapb = 0.0;
#pragma unroll
          for (int q = 0; q < 6; ++q) lapb += symw(q) * gu[q] * v.d2[q];
          r_Gt[k] += lapb;
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            db[k][j] = d1[j];
            r_Gt[j] += (1.0 / 3.0) * (gu[sym(j, 0)] * v.d2[sym(0, k)] + gu[sym(j, 1)] * v.d2[sym(1, k)] +
                                      gu[sym(j, 2)] * v.d2[sym(2, k)]);
          }
        }
      });
      // ---- closing algebra: the geometry role's values have arrived ---------
      bar_sync<BAR_FULL, 2 * NTHREADS>();
      const double t23 = 2.0 / 3.0;
      if (CONS) {
        double trR = X[XC_TRR * NTHREADS];
        const double x0 = X[XC_MOM * NTHREADS], x1 = X[(XC_MOM + 1) * NTHREADS], x2 = X[(XC_MOM + 2) * NTHREADS];
        if (PIPE && has_next) {
          bar_arrive<BAR_FREE_GT, 2 * NTHREADS>();
          bar_arrive<BAR_FREE, 2 * NTHREADS>();
        }
        double A[6], M[3][3], AA = 0.0;
#pragma unroll
        for (int p = 0; p < 6; ++p) { A[p] = fld(F_AT + p); trR += symw(p) * gu[p] * Rg[p]; }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            M[k][j] = A[sym(k, 0)] * gu[sym(0, j)] + A[sym(k, 1)] * gu[sym(1, j)] + A[sym(k, 2)] * gu[sym(2, j)];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int j = 0; j < 3; ++j) AA += M[k][j] * M[j][k];
        const double K = fld(F_K), H = fld(F_CHI) * trR + t23 * K * K - AA;
        double m[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double gA = fld(F_GTI) * A[sym(a, 0)] + fld(F_GTI + 1) * A[sym(a, 1)] + fld(F_GTI + 2) * A[sym(a, 2)];
          m[a] = mom[a] + (a == 0 ? x0 : (a == 1 ? x1 : x2)) - gA;
        }
        if (MODE == MODE_CON) {
          double* O = args.OUT + gidx;
          if (inside) { O[0] = H; O[n] = m[0]; O[2 * n] = m[1]; O[3 * n] = m[2]; }
        } else {
          const int g = args.ng, gx = d.x0 + lx, gy = d.y0 + ly, gz = d.z0 + lz;
          if (inside && gx >= g && gx < d.sx - g && gy >= g && gy < d.sy - g && gz >= g && gz < d.sz - g) {
            norm_h += H * H;
            norm_m += m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
          }
        }
      } else {
        // Rates into shared memory, each over a value that no later rate reads:
        // At (LEAN: kept in registers), chi, K, alpha and beta over their point
        // values, gt over X_X, Gt and B over gt's point values.
        const double divb = db[0][0] + db[1][1] + db[2][2];
        const double al = fld(F_ALPHA), chi = fld(F_CHI), K = fld(F_K);
        double A[6], AA = 0.0;
#pragma unroll
        for (int p = 0; p < 6; ++p) A[p] = fld(F_AT + p);
        double rAt[6];
        {
          double Xp[6], M[3][3], trX = 0.0;
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            Xp[p] = X[(X_X + p) * NTHREADS];
            trX += symw(p) * gu[p] * Xp[p];
          }
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j)
              M[k][j] = A[sym(k, 0)] * gu[sym(0, j)] + A[sym(k, 1)] * gu[sym(1, j)] + A[sym(k, 2)] * gu[sym(2, j)];
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) AA += M[k][j] * M[j][k];
          const double third_trX = (1.0 / 3.0) * trX;
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const int a = sym_i(p), b = sym_j(p);
            const double aga = M[a][0] * A[sym(0, b)] + M[a][1] * A[sym(1, b)] + M[a][2] * A[sym(2, b)];
            double r = r_At[p] - t23 * A[p] * divb + chi * (Xp[p] - fld(F_GT + p) * third_trX) + al * (K * A[p] - 2.0 * aga);
#pragma unroll
            for (int k = 0; k < 3; ++k) r += A[sym(a, k)] * db[k][b] + A[sym(b, k)] * db[k][a];
            if (LEAN) rAt[p] = r; else pB[(F_AT + p) * NTHREADS] = r;
          }
        }
        {
          double g[6];
#pragma unroll
          for (int p = 0; p < 6; ++p) g[p] = fld(F_GT + p);
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const int a = sym_i(p), b = sym_j(p);
            double r = X[(X_GT + p) * NTHREADS] - t23 * g[p] * divb - 2.0 * al * A[p];
#pragma unroll
            for (int k = 0; k < 3; ++k) r += g[sym(a, k)] * db[k][b] + g[sym(b, k)] * db[k][a];
            X[(X_X + p) * NTHREADS] = r;
          }
        }
        if (PIPE && has_next) bar_arrive<BAR_FREE_GT, 2 * NTHREADS>();
        {
          pB[F_CHI * NTHREADS] = X[X_CHI * NTHREADS] + t23 * chi * (al * K - divb) + d.cahd * chi * (t23 * K * K - AA);
          pB[F_K * NTHREADS] = r_K - chi * X[X_LAPA * NTHREADS] + al * (K * K * (1.0 / 3.0) + AA);
          const double sq = sqrt(chi);
          pB[F_ALPHA * NTHREADS] = X[X_ALPHA * NTHREADS] - 2.0 * al * K - s_par.ssl * sq * (al - sq);
        }
        {
          const double lf = 0.75 * (s_par.lamf0 + s_par.lamf1 * al);
          double cal[3];
#pragma unroll
          for (int a = 0; a < 3; ++a) cal[a] = X[(X_CAL + a) * NTHREADS];
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const double Ba = fld(F_B + a);
            const double r = r_Gt[a] + t23 * cal[a] * divb -
                             (cal[0] * db[a][0] + cal[1] * db[a][1] + cal[2] * db[a][2]);
            pB[(F_BETA + a) * NTHREADS] = r_beta[a] + lf * Ba;
            pB[(F_GT + a) * NTHREADS] = r + X[(X_RG + a) * NTHREADS];
            pB[(F_GT + 3 + a) * NTHREADS] = r + X[(X_RB + a) * NTHREADS] - s_par.eta * Ba + r_B[a];
          }
        }
        // ---- update and stores: 12 fields at a time, their u_n and running
        // sums all loaded before the first is stored
        const int stage = args.stage;
        const double dt = s_par.dt;
        const bool last = MODE == MODE_STAGE ? stage == 3 : (MODE == MODE_MSRK && stage == 2);
        const bool need_acc = MODE == MODE_STAGE ? stage != 0 : (MODE == MODE_MSRK && stage < 2);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          // part 0: gt, At; part 1: alpha, chi, K, beta, Gt, B
          auto field = [&](int q) {
            return part == 0 ? (q < 6 ? F_GT + q : F_AT + q - 6)
                             : (q < 3 ? q : (q < 6 ? F_BETA + q - 3 : F_GTI + q - 6));
          };
          double r[12];
          if (MODE == MODE_RHS) {
#pragma unroll
            for (int q = 0; q < 12; ++q) {
              r[q] = part == 0 ? (q < 6 ? X[(X_X + q) * NTHREADS] : (LEAN ? rAt[q < 6 ? 0 : q - 6] : pB[(F_AT + q - 6) * NTHREADS]))
                               : (q < 3 ? pB[q * NTHREADS] : (q < 6 ? pB[(F_BETA + q - 3) * NTHREADS] : pB[(F_GT + q - 6) * NTHREADS]));
              if (inside) args.OUT[gidx + (long long)field(q) * n] = r[q];
            }
          } else {
            double u[12], acc[12];
#pragma unroll
            for (int q = 0; q < 12; ++q) {
              u[q] = args.U[gidx + (long long)field(q) * n];
              acc[q] = need_acc ? args.ACC[gidx + (long long)field(q) * n] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 12; ++q) {
              const long long o = gidx + (long long)field(q) * n;
              const double rate =
                  part == 0 ? (q < 6 ? X[(X_X + q) * NTHREADS] : (LEAN ? rAt[q < 6 ? 0 : q - 6] : pB[(F_AT + q - 6) * NTHREADS]))
                            : (q < 3 ? pB[q * NTHREADS] : (q < 6 ? pB[(F_BETA + q - 3) * NTHREADS] : pB[(F_GT + q - 6) * NTHREADS]));
              if (MODE == MODE_STAGE) {
                if (stage == 3) {
                  r[q] = u[q] + (dt / 6.0) * (acc[q] + rate);
                } else {
                  r[q] = u[q] + (stage == 2 ? dt : 0.5 * dt) * rate;
                  if (inside) args.ACC[o] = stage == 0 ? rate : acc[q] + 2.0 * rate;
                }
              } else {
                const double* c = args.coef;
                if (stage == 0) {
                  r[q] = u[q] + dt * (c[0] * acc[q] + c[1] * rate);
                  if (inside) {
                    args.ACC[o] = rate;
                    args.OUT2[o] = u[q] + dt * (c[2] * acc[q] + c[3] * rate);
                    args.OUT3[o] = u[q] + dt * (c[5] * acc[q] + c[6] * rate);
                  }
                } else if (stage == 1) {
                  r[q] = u[q] + dt * (c[4] * rate);
                  if (inside) args.ACC[o] = acc[q] + dt * (c[7] * rate);
                } else {
                  r[q] = u[q] + dt * (c[8] * rate);
                }
              }
            }
            if (part == 0 && last) enforce_metric(r);
            if (part == 1 && last) {
              r[0] = fmax(r[0], args.alpha_floor);
              r[1] = fmax(r[1], args.chi_floor);
            }
#pragma unroll
            for (int q = 0; q < 12; ++q)
              if (inside) args.OUT[gidx + (long long)field(q) * n] = r[q];
          }
          if (part == 0 && PIPE && has_next) bar_arrive<BAR_FREE, 2 * NTHREADS>();
        }
      }
      par ^= 1;
    }
  }
  if (MODE == MODE_NORM) {
    // fixed-order block reduction of the transport role's sums (reuses the staging buffers)
    __syncthreads();
    double* red = smem;
    if (role) {
      red[2 * rt] = norm_h;
      red[2 * rt + 1] = norm_m;
    }
    __syncthreads();
    for (int w = NTHREADS / 2; w > 0; w >>= 1) {
      if (tid < w) {
        red[2 * tid] += red[2 * (tid + w)];
        red[2 * tid + 1] += red[2 * (tid + w) + 1];
      }
      __syncthreads();
    }
    if (tid == 0) {
      args.partials[2 * blockIdx.x] = red[0];
      args.partials[2 * blockIdx.x + 1] = red[1];
    }
  }
}

}  // namespace bssn

namespace bssn_host {
// Internal linkage for everything below: each translation unit keeps its own
// per-device flags, and two loaded copies of the library never share them.
namespace {

// Opt a kernel into its dynamic shared memory once per device.
template <class K>
int set_smem(K kern, size_t smem, int* flags) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return bssn_host::cuda_fail("cudaGetDevice", e);
  if (dev < 0 || dev >= kMaxDev) return bssn_host::fail(BSSN_B200_EINVAL, "device ordinal out of range");
  if (!flags[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return bssn_host::cuda_fail("cudaFuncSetAttribute", e);
    flags[dev] = 1;
  }
  return 0;
}

template <int R, int MODE, bool KO, class T = bssn::DefaultShape>
int launch_stream(const bssn::Args& a, cudaStream_t stream, int grid) {
  constexpr size_t smem = bssn::TileGeom<R, T>::SMEM;
  auto kern = bssn::stream_kernel<R, MODE, KO, T>;
  static int flags[kMaxDev] = {0};
  int rc = set_smem(kern, smem, flags);
  if (rc) return rc;
  kern<<<grid, 2 * bssn::NTHREADS, smem, stream>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return bssn_host::cuda_fail("stream kernel launch", e);
  return 0;
}

}  // namespace
}  // namespace bssn_host
