// bssn_b200 — the C ABI of include/bssn_b200.h and the kernels around the
// fused stream kernel (stream_kernel.cuh, instantiated by the stream_*.cu
// translation units): the derivative bundle, the algebra on derivatives from
// memory, norms, enforcement and the periodic sync.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <string>
#include <type_traits>

#include "../../include/bssn_b200.h"
#include "host_util.h"
#include "stream.cuh"
#include "stream_kernel.cuh"
#include "stream_launch.h"

namespace bssn {
__device__ __forceinline__ Params load_params(const double* __restrict__ S) {
  Params P;
  P.eta = S[0]; P.cahd_c = S[1]; P.dt = S[2]; P.dx = S[3];
  P.ssl_h = S[4]; P.ssl_sigma = S[5]; P.t = S[6];
  P.lam0 = S[7]; P.lam1 = S[8]; P.lam2 = S[9]; P.lam3 = S[10];
  P.lamf0 = S[11]; P.lamf1 = S[12];
  P.hx = S[13]; P.hy = S[14]; P.hz = S[15];
  return P;
}

// Final-stage values of the fields that algebraic enforcement rewrites are
// held back (gt0..5, At0..5, chi, alpha); the rest are stored directly.
__device__ __forceinline__ bool hold_for_enforce(double* en, int k, double un) {
  if (k >= F_GT && k < F_GT + 6) en[k - F_GT] = un;
  else if (k >= F_AT && k < F_AT + 6) en[6 + k - F_AT] = un;
  else if (k == F_CHI) en[12] = un;
  else if (k == F_ALPHA) en[13] = un;
  else return false;
  return true;
}

// Enforces the held values of one point and stores them.
__device__ __forceinline__ void store_enforced(double (&en)[14], double* O, long long n, double chi_floor,
                                               double alpha_floor) {
  double v[12];
#pragma unroll
  for (int q = 0; q < 12; ++q) v[q] = en[q];
  enforce_metric(v);
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    O[(long long)(F_GT + q) * n] = v[q];
    O[(long long)(F_AT + q) * n] = v[6 + q];
  }
  O[(long long)F_CHI * n] = fmax(en[12], chi_floor);
  O[(long long)F_ALPHA * n] = fmax(en[13], alpha_floor);
}

// ---------------------------------------------------------------------------
// Derivative bundle to global memory (the bssn_b200_derivatives entry): the
// staging and the stencils of the stream kernel, one field at a time,
// double-buffered, every result stored at once. 1.3 KB are written and 0.2 KB
// read per point (KO on), so the stores should be all that counts: three CTAs
// per SM (77-78 registers, 49 KB each) keep them going while others
// differentiate. An 86^3 array with KO6: 0.64 ms with single buffering, one
// 8-byte copy a cell and 36 taps per mixed derivative, 0.43 ms now (2.2 TB/s,
// 1.9 of it stores; copy latency and the shared-memory pipe bound it).
// ---------------------------------------------------------------------------
template <int R>
struct DerivLayout {
  using G = TileGeom<R, DefaultShape>;
  static constexpr size_t SMEM = (size_t)(2 * G::VOL + G::TVOL) * sizeof(double) + (size_t)2 * G::NROW * sizeof(int);
};

template <int R, bool KO>
__global__ void __launch_bounds__(NTHREADS, 3) deriv_kernel(const __grid_constant__ Args args) {
  using T = DefaultShape;
  using G = TileGeom<R, T>;
  extern __shared__ __align__(128) double smem[];
  __shared__ TileDesc s_desc[2];
  double* const T1 = smem + 2 * G::VOL;
  int* const rows = reinterpret_cast<int*>(T1 + G::TVOL);
  double* cur = smem;
  double* nxt = smem + G::VOL;
  const int tid = threadIdx.x;
  const int lz = tid % T::Z, ly = (tid / T::Z) % T::Y, lx = tid / (T::Z * T::Y);
  const PointPlace place = point_place<R, T>(tid);
  const StagePlace splace = stage_place<R, T>(tid);
  const long long n = args.n;
  const int ntiles = args.ntx * args.nty * args.ntz;
  auto issue = [&](int f, const TileDesc& d, const int* rw, double* buf) {
    const int z = d.zs + splace.ch;
    if (splace.row0 < G::NROW && z < d.sz + R) {
      const bool whole = d.al && z >= 0 && z + 1 < d.sz;
      if (has_d2(f)) stage_rows<R, T, true>(buf, args.F + (f * n + z), rw, splace, whole, d);
      else stage_rows<R, T, false>(buf, args.F + (f * n + z), rw, splace, whole, d);
    }
    cp_async_commit();
  };
  if (tid < 32) fill_desc<R, T>(args, blockIdx.x, &s_desc[0], nullptr);
  __syncthreads();
  fill_rows<R, T>(s_desc[0], rows, tid);
  __syncthreads();
  issue(0, s_desc[0], rows, cur);
  int par = 0;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const TileDesc& d = s_desc[par];
    const bool has_next = tile + (int)gridDim.x < ntiles;
    const int gx = d.x0 + lx, gy = d.y0 + ly, gz = d.z0 + lz, dz = d.z0 - d.zs;
    const bool inside = gx < d.sx && gy < d.sy && gz < d.sz;
    double* const out = args.OUT + ((long long)gx * d.sy + gy) * d.sz + gz;
#pragma unroll 1
    for (int f = 0; f < NFIELD; ++f) {
      cp_async_wait<0>();
      __syncthreads();
      if (f + 1 < NFIELD) issue(f + 1, d, rows + par * G::NROW, nxt);
      else if (has_next) issue(0, s_desc[par ^ 1], rows + (par ^ 1) * G::NROW, nxt);
      if (has_next) {
        if (f == 0 && tid < 32) fill_desc<R, T>(args, tile + gridDim.x, &s_desc[par ^ 1], &d);
        if (f == 1) fill_rows<R, T>(s_desc[par ^ 1], rows + (par ^ 1) * G::NROW, tid);
      }
      Derivs v;
      if (has_d2(f)) {
        field_derivs<R, T, true, KO, 1, false, true>(cur + dz, T1, place, d, tid, v);
        if (inside) {
          double* const o = out + (long long)d2slot(f, 0) * n;
#pragma unroll
          for (int p = 0; p < 6; ++p) o[p * n] = v.d2[p];
        }
      } else {
        field_derivs<R, T, false, KO, 1, false, true>(cur + dz, T1, place, d, tid, v);
      }
      if (inside) {
        double* const o = out + (long long)d1slot(f, 0) * n;
#pragma unroll
        for (int a = 0; a < 3; ++a) o[a * n] = __dmul_rn(v.s1[a], d.f1[a]);
        if (KO) out[(long long)(NDERIV + f) * n] = v.ko;
      }
      double* t = cur; cur = nxt; nxt = t;
    }
    par ^= 1;
  }
}

// Second pass of the constraint norms: the per-CTA partial sums in index
// order (deterministic for a given grid), then RMS over the interior
// (3D/src/bssn3d/constraints.py:53-62).
__global__ void norm_finalize_kernel(const double* __restrict__ partials, int nparts, double count,
                                     double* __restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double h = 0.0, m = 0.0;
    for (int i = 0; i < nparts; ++i) {
      h += partials[2 * i];
      m += partials[2 * i + 1];
    }
    out[0] = sqrt(h / count);
    out[1] = sqrt(m / count);
  }
}

// Partial-sum slots for bssn_b200_constraint_norms_static, the entry point for
// callers that cannot allocate device memory. It is a file-scope device array:
// every GPU that loads this library holds it (4 KB) until the process exits,
// and every call of that entry point reuses it.
// CTAs whose partial sums fit (2 doubles each). The norm launch runs at most
// one CTA per SM, so 256 covers every GPU with up to 256 SMs (B200: 148); a
// GPU with more is refused by the entry point's size check.
constexpr int kStaticNormCtas = 256;
static __device__ __align__(256) double g_static_norm_partials[2 * kStaticNormCtas];

// t <- t + dt in the device scalar pack, between captured RK4 steps
// (the fori_loop carry update of 3D/src/bssn3d/evolve.py:186-193).
__global__ void advance_time_kernel(double* S) {
  if (threadIdx.x == 0 && blockIdx.x == 0) S[6] = S[6] + S[2];
}

struct Scalars {
  double v[16];
};
__global__ void set_scalars_kernel(double* __restrict__ S, const __grid_constant__ Scalars s) {
  if (threadIdx.x < 16) S[threadIdx.x] = s.v[threadIdx.x];
}

// Algebra only: derivatives supplied by the caller (the reference's
// algebra-only microbenchmark interface, 3D/src/bssn3d/cuda/gen_algebra_cuda.py:55-96),
// consumed in the stream order of the fused kernel.
__global__ void __launch_bounds__(128) algebra_kernel(const double* __restrict__ F, const double* __restrict__ D,
                                                      const double* __restrict__ S, double* __restrict__ OUT,
                                                      long long n) {
  const Params P = load_params(S);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    auto fld = [&](int k) -> double { return __ldg(F + (long long)k * n + q); };
    auto drv = [&](int s) -> double { return __ldg(D + (long long)s * n + q); };
    Stream acc;
    acc.init(fld);
    Unroll<0, NFIELD>::run([&](auto ic) {
      constexpr int f = stream_field(decltype(ic)::value);
      double d1[3], d2[6];
#pragma unroll
      for (int a = 0; a < 3; ++a) d1[a] = drv(d1slot(f, a));
#pragma unroll
      for (int p = 0; p < 6; ++p) d2[p] = has_d2(f) ? drv(d2slot(f, p)) : 0.0;
      acc.consume(f, d1, d2, 0.0, P, fld);
    });
    auto emit = [&](int k, double v) { OUT[(long long)k * n + q] = v; };
    acc.finalize(fld, P, emit);
  }
}

// One RK4 stage from precomputed derivatives over the covered points
// [core, s - core)^3 of every block of a block list: the algebra of
// algebra_kernel on the stage input Y with the block's spacing and the stage
// time, the KO sums taken from slots 138..161 of D when ko_slots is set, and
// the stage epilogue of the stream kernel (evolve.py:125-131, the final stage
// with algebraic enforcement). Derivative slot s of block b is at
// D + (offset_b / 24) * nslot + s * n_b. Points are enumerated block by block
// (pts0 = prefix of covered points), one thread per point.
__global__ void __launch_bounds__(128) stage_derivs_kernel(
    const double* __restrict__ U, const double* __restrict__ Y, double* __restrict__ ACC, double* __restrict__ OUT,
    const double* __restrict__ D, int nslot, const double* __restrict__ S, int stage, int ko_slots,
    double chi_floor, double alpha_floor, const bssn_b200_block* __restrict__ blocks, int nblocks,
    const long long* __restrict__ pts0, long long npoints) {
  const Params P0 = load_params(S);
  const double cs = stage == 0 ? 0.0 : (stage == 3 ? 1.0 : 0.5);
  const double dt = P0.dt;
  const double hstep = (stage == 2) ? dt : 0.5 * dt;
  const double w6 = dt / 6.0;
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * blockDim.x;
  // warps walk the points together (q0 is the warp's first point), so the
  // block lookup is one 32-way search per warp instead of one per point
  for (long long q0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); q0 < npoints; q0 += stride) {
    const long long q = q0 + lane;
    int lo = 0, nb = nblocks;  // last block whose first point is <= q0 (pts0[0] = 0)
    while (nb > 1) {
      const int step = (nb + 31) >> 5;
      const int idx = lo + lane * step;
      const unsigned ok = __ballot_sync(0xffffffffu, idx < lo + nb && pts0[idx] <= q0);
      const int last = 31 - __clz(ok);
      lo += last * step;
      nb = min(step, nb - last * step);
    }
    while (lo + 1 < nblocks && pts0[lo + 1] <= q) ++lo;  // a warp that straddles blocks
    if (q >= npoints) continue;
    const bssn_b200_block bk = blocks[lo];
    const int c = bk.core;
    const int ey = bk.sy - 2 * c, ez = bk.sz - 2 * c;
    const int lq = (int)(q - pts0[lo]);
    const int z = lq % ez + c, y = (lq / ez) % ey + c, x = lq / (ez * ey) + c;
    const long long n = (long long)bk.sx * bk.sy * bk.sz;
    const long long p = ((long long)x * bk.sy + y) * bk.sz + z;
    const long long gidx = bk.offset + p;
    const double* Dq = D + (bk.offset / 24) * nslot + p;
    Params P = P0;
    P.dx = bk.h[0]; P.hx = bk.h[0]; P.hy = bk.h[1]; P.hz = bk.h[2];
    P.t = P0.t + cs * P0.dt;  // stage time t, t+dt/2, t+dt/2, t+dt (evolve.py:125-131)
    auto fld = [&](int k) -> double { return __ldg(Y + gidx + (long long)k * n); };
    auto drv = [&](int s) -> double { return __ldg(Dq + (long long)s * n); };
    Stream acc;
    acc.init(fld);
    Unroll<0, NFIELD>::run([&](auto ic) {
      constexpr int f = stream_field(decltype(ic)::value);
      double d1[3], d2[6];
#pragma unroll
      for (int a = 0; a < 3; ++a) d1[a] = drv(d1slot(f, a));
#pragma unroll
      for (int pp = 0; pp < 6; ++pp) d2[pp] = has_d2(f) ? drv(d2slot(f, pp)) : 0.0;
      acc.consume(f, d1, d2, ko_slots ? drv(138 + f) : 0.0, P, fld);
    });
    double* A = ACC + gidx;
    double* O = OUT + gidx;
    double en[14];
#pragma unroll
    for (int k = 0; k < 14; ++k) en[k] = 0.0;
    auto emit = [&](int k, double rate) {
      const long long o = (long long)k * n;
      const double u = U[gidx + o];
      if (stage == 0) {
        A[o] = rate;
        O[o] = u + hstep * rate;
      } else if (stage < 3) {
        A[o] = A[o] + 2.0 * rate;
        O[o] = u + hstep * rate;
      } else {
        const double un = u + w6 * (A[o] + rate);
        if (!hold_for_enforce(en, k, un)) O[o] = un;
      }
    };
    acc.finalize(fld, P, emit);
    if (stage == 3) store_enforced(en, O, n, chi_floor, alpha_floor);
  }
}

__global__ void enforce_kernel(double* __restrict__ U, long long n, double chi_floor, double alpha_floor) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    double v[12];
#pragma unroll
    for (int k = 0; k < 6; ++k) { v[k] = U[(F_GT + k) * n + q]; v[6 + k] = U[(F_AT + k) * n + q]; }
    enforce_metric(v);
#pragma unroll
    for (int k = 0; k < 6; ++k) { U[(F_GT + k) * n + q] = v[k]; U[(F_AT + k) * n + q] = v[6 + k]; }
    U[F_CHI * n + q] = fmax(U[F_CHI * n + q], chi_floor);
    U[F_ALPHA * n + q] = fmax(U[F_ALPHA * n + q], alpha_floor);
  }
}

// Periodic ghost sync in one pass. The axis-by-axis sync (ghosts [0, ng) <-
// [S - 2 ng, S - ng), [S - ng, S) <- [ng, 2 ng), x then y then z) leaves every
// ghost point with the interior value at its index wrapped on all three axes,
// so each point takes it directly: one launch that reads interiors and writes
// ghosts, instead of three that each wait for the last. A thread takes one
// point and moves its 24 fields. With the stage buffers synced in place, a
// 49x56x64 RK4 step: 872 -> 733 us.
__global__ void periodic_kernel(double* __restrict__ U, int Sx, int Sy, int Sz, int ng) {
  const long long n = (long long)Sx * Sy * Sz;
  auto wrap = [&](int c, int S) { return c < ng ? c + S - 2 * ng : (c >= S - ng ? c - (S - 2 * ng) : c); };
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int p = (int)q, z = p % Sz, t = p / Sz, y = t % Sy, x = t / Sy;  // fewer than 2^31 points (check_grid)
    const int wx = wrap(x, Sx), wy = wrap(y, Sy), wz = wrap(z, Sz);
    if (wx == x && wy == y && wz == z) continue;
    const long long src = ((long long)wx * Sy + wy) * Sz + wz;
    double v[NFIELD];
#pragma unroll
    for (int f = 0; f < NFIELD; ++f) v[f] = U[f * n + src];
#pragma unroll
    for (int f = 0; f < NFIELD; ++f) U[f * n + q] = v[f];
  }
}

}  // namespace bssn

// ======================================================================
// host side
// ======================================================================
namespace {

thread_local std::string g_err;

int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}

int cuda_fail(const char* what, cudaError_t e) {
  return fail(BSSN_B200_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

using bssn_host::kMaxDev;
using bssn_host::set_smem;

int device_sms(int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail("cudaGetDevice", e);
  static int cache[kMaxDev] = {0};
  if (dev >= 0 && dev < kMaxDev && cache[dev] > 0) {
    *sms = cache[dev];
    return 0;
  }
  int v = 0;
  e = cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail("cudaDeviceGetAttribute", e);
  if (dev >= 0 && dev < kMaxDev) cache[dev] = v;
  *sms = v;
  return 0;
}

template <int R, bool KO>
int launch_deriv(const bssn::Args& a, cudaStream_t stream, int grid) {
  constexpr size_t smem = bssn::DerivLayout<R>::SMEM;
  auto kern = bssn::deriv_kernel<R, KO>;
  static int flags[kMaxDev] = {0};
  int rc = set_smem(kern, smem, flags);
  if (rc) return rc;
  kern<<<grid, bssn::NTHREADS, smem, stream>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("derivative kernel launch", e);
  return 0;
}

int check_grid(long long Sx, long long Sy, long long Sz) {
  if (Sx < 1 || Sy < 1 || Sz < 1) return fail(BSSN_B200_EINVAL, "grid extents must be >= 1");
  if (Sx > (1LL << 31) / Sy / Sz) return fail(BSSN_B200_EINVAL, "grid has more than 2^31 points");
  return 0;
}

// Fill the shape fields of `a` and the persistent grid size (one CTA per SM).
int prepare(bssn::Args* a, long long Sx, long long Sy, long long Sz, int ctas_per_sm, int* grid) {
  int rc = check_grid(Sx, Sy, Sz);
  if (rc) return rc;
  int sms = 0;
  rc = device_sms(&sms);
  if (rc) return rc;
  a->Sx = Sx; a->Sy = Sy; a->Sz = Sz;
  a->n = Sx * Sy * Sz;
  using D = bssn::DefaultShape;
  a->ntx = (int)((Sx + D::X - 1) / D::X);
  a->nty = (int)((Sy + D::Y - 1) / D::Y);
  a->ntz = (int)((Sz + D::Z - 1) / D::Z);
  const long long ntiles = (long long)a->ntx * a->nty * a->ntz;
  const long long cap = (long long)sms * ctas_per_sm;
  *grid = (int)(ntiles < cap ? ntiles : cap);
  return 0;
}

void variant_shape(int variant, int* tx, int* ty, int* tz) {
  static const int shapes[BSSN_B200_NVARIANTS][3] = {{4, 4, 16}, {2, 8, 16}, {4, 8, 8}, {8, 4, 8}};
  *tx = shapes[variant][0];
  *ty = shapes[variant][1];
  *tz = shapes[variant][2];
}

// One stream-kernel launch on the default tile (variant 0) or a batched tile
// variant; the instantiations live in the stream_*.cu translation units.
int launch_single(int R, int mode, const bssn::Args& a, cudaStream_t st, int grid) {
  switch (mode) {
    case bssn::MODE_STAGE: return bssn_host::launch_stage_modes(R, mode, a, st, grid);
    case bssn::MODE_MSRK: return bssn_host::launch_msrk_modes(R, mode, a, st, grid);
    default: return bssn_host::launch_rhs_modes(R, mode, a, st, grid);
  }
}

int launch_variant(int R, int mode, const bssn::Args& a, cudaStream_t st, int grid, int variant) {
  if (variant == 0) return launch_single(R, mode, a, st, grid);
  if (variant < 0 || variant >= BSSN_B200_NVARIANTS) return fail(BSSN_B200_EINVAL, "variant out of range");
  return R == 4 ? bssn_host::launch_batch_r4(mode, variant, a, st, grid)
                : bssn_host::launch_batch_r3(mode, variant, a, st, grid);
}

int prepare_batch(bssn::Args* a, const bssn_b200_block* blocks, int nblocks, int ntiles, int variant, int* grid) {
  if (!blocks) return fail(BSSN_B200_EINVAL, "batch: NULL block table");
  if (nblocks < 1) return fail(BSSN_B200_EINVAL, "batch: nblocks must be >= 1");
  if (ntiles < 1) return fail(BSSN_B200_EINVAL, "batch: ntiles must be >= 1 (run bssn_b200_batch_plan)");
  if (variant < 0 || variant >= BSSN_B200_NVARIANTS) return fail(BSSN_B200_EINVAL, "batch: variant out of range");
  int sms = 0;
  int rc = device_sms(&sms);
  if (rc) return rc;
  a->blocks = blocks;
  a->nblocks = nblocks;
  a->ntiles = ntiles;
  *grid = ntiles < sms ? ntiles : sms;
  return 0;
}

}  // namespace

namespace bssn_host {
int fail(int code, const std::string& msg) { return ::fail(code, msg); }
int cuda_fail(const char* what, cudaError_t e) { return ::cuda_fail(what, e); }
int device_sms(int* sms) { return ::device_sms(sms); }
}  // namespace bssn_host

extern "C" {

int bssn_b200_batch_plan(bssn_b200_block* host_blocks, int nblocks, int variant) {
  if (!host_blocks || nblocks < 1) {
    fail(BSSN_B200_EINVAL, "batch_plan: empty block table");
    return -1;
  }
  if (variant < 0 || variant >= BSSN_B200_NVARIANTS) {
    fail(BSSN_B200_EINVAL, "batch_plan: variant out of range");
    return -1;
  }
  int tx, ty, tz;
  variant_shape(variant, &tx, &ty, &tz);
  long long t0 = 0;
  for (int b = 0; b < nblocks; ++b) {
    bssn_b200_block& bk = host_blocks[b];
    if (bk.sx < 1 || bk.sy < 1 || bk.sz < 1 || bk.offset < 0 || !(bk.h[0] > 0) || !(bk.h[1] > 0) || !(bk.h[2] > 0)) {
      fail(BSSN_B200_EINVAL, "batch_plan: block " + std::to_string(b) + " has a bad extent, offset or spacing");
      return -1;
    }
    if ((long long)bk.sx * bk.sy * bk.sz >= (1LL << 31)) {
      fail(BSSN_B200_EINVAL, "batch_plan: block " + std::to_string(b) + " has 2^31 points or more");
      return -1;
    }
    if (bk.core < 0 || 2 * bk.core >= bk.sx || 2 * bk.core >= bk.sy || 2 * bk.core >= bk.sz) {
      fail(BSSN_B200_EINVAL, "batch_plan: block " + std::to_string(b) + " has a core margin that leaves no points");
      return -1;
    }
    bk.tile0 = (int)t0;
    const int c2 = 2 * bk.core;
    t0 += (long long)((bk.sx - c2 + tx - 1) / tx) * ((bk.sy - c2 + ty - 1) / ty) * ((bk.sz - c2 + tz - 1) / tz);
    if (t0 > (1LL << 30)) {
      fail(BSSN_B200_EINVAL, "batch_plan: too many tiles");
      return -1;
    }
  }
  return (int)t0;
}

int bssn_b200_batch_rhs(void* stream, const double* F, const double* S, double* OUT,
                        const bssn_b200_block* blocks, int nblocks, int ntiles, int variant) {
  if (!F || !S || !OUT) return fail(BSSN_B200_EINVAL, "batch_rhs: NULL operand");
  if (OUT == F) return fail(BSSN_B200_EINVAL, "batch_rhs: OUT must not alias F");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare_batch(&a, blocks, nblocks, ntiles, variant, &grid);
  if (rc) return rc;
  a.F = F; a.S = S; a.OUT = OUT;
  return launch_variant(3, bssn::MODE_RHS, a, static_cast<cudaStream_t>(stream), grid, variant);
}

int bssn_b200_batch_rk4_stage(void* stream, int stage, const double* U, const double* Y, double* ACC,
                              double* YNEXT, const double* S, double ko_sigma, int ko_order,
                              double chi_floor, double alpha_floor, const bssn_b200_block* blocks,
                              int nblocks, int ntiles, int variant) {
  if (stage < 0 || stage > 3) return fail(BSSN_B200_EINVAL, "batch_rk4_stage: stage must be 0..3");
  if (!U || !Y || !ACC || !YNEXT || !S) return fail(BSSN_B200_EINVAL, "batch_rk4_stage: NULL operand");
  if (YNEXT == Y) return fail(BSSN_B200_EINVAL, "batch_rk4_stage: YNEXT must not alias Y");
  if (stage < 3 && YNEXT == U) return fail(BSSN_B200_EINVAL, "batch_rk4_stage: YNEXT may alias U only at stage 3");
  if (ACC == Y || ACC == U || ACC == YNEXT) return fail(BSSN_B200_EINVAL, "batch_rk4_stage: ACC must not alias another operand");
  const bool use_ko = ko_sigma > 0.0;
  if (use_ko && ko_order != 6 && ko_order != 8) return fail(BSSN_B200_EINVAL, "batch_rk4_stage: ko_order must be 6 or 8");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare_batch(&a, blocks, nblocks, ntiles, variant, &grid);
  if (rc) return rc;
  a.F = Y; a.U = U; a.ACC = ACC; a.OUT = YNEXT; a.S = S;
  a.stage = stage;
  a.use_ko = use_ko ? 1 : 0;
  a.ko_sigma = use_ko ? ko_sigma : 0.0;
  a.chi_floor = chi_floor; a.alpha_floor = alpha_floor;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (use_ko && ko_order == 8) return launch_variant(4, bssn::MODE_STAGE, a, st, grid, variant);
  return launch_variant(3, bssn::MODE_STAGE, a, st, grid, variant);
}

const char* bssn_b200_last_error(void) { return g_err.c_str(); }

const char* bssn_b200_version(void) { return "bssn_b200 0.3 sm_100a"; }

int bssn_b200_async_copy_errors(int* count) {
  if (!count) return fail(BSSN_B200_EINVAL, "async_copy_errors: NULL operand");
  *count = 0;
  return 0;
}

int bssn_b200_set_scalars(void* stream, double* S, const double* host_scalars) {
  if (!S || !host_scalars) return fail(BSSN_B200_EINVAL, "set_scalars: NULL operand");
  bssn::Scalars s;
  std::memcpy(s.v, host_scalars, sizeof(s.v));
  bssn::set_scalars_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(S, s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("set_scalars launch", e);
  return 0;
}

int bssn_b200_rhs(void* stream, const double* F, const double* S, double* OUT, long long Sx,
                  long long Sy, long long Sz) {
  if (!F || !S || !OUT) return fail(BSSN_B200_EINVAL, "rhs: NULL operand");
  if (OUT == F) return fail(BSSN_B200_EINVAL, "rhs: OUT must not alias F");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 1, &grid);
  if (rc) return rc;
  a.F = F; a.S = S; a.OUT = OUT;
  return launch_single(3, bssn::MODE_RHS, a, static_cast<cudaStream_t>(stream), grid);
}

int bssn_b200_constraints(void* stream, const double* F, const double* S, double* OUT,
                          long long Sx, long long Sy, long long Sz) {
  if (!F || !S || !OUT) return fail(BSSN_B200_EINVAL, "constraints: NULL operand");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 1, &grid);
  if (rc) return rc;
  a.F = F; a.S = S; a.OUT = OUT;
  return launch_single(3, bssn::MODE_CON, a, static_cast<cudaStream_t>(stream), grid);
}

size_t bssn_b200_norms_scratch_bytes(void) {
  int sms = 0;
  if (device_sms(&sms)) return 0;
  return (size_t)sms * 2 * sizeof(double);
}

int bssn_b200_constraint_norms(void* stream, const double* F, const double* S, long long Sx,
                               long long Sy, long long Sz, int ng, double* scratch,
                               size_t scratch_bytes, double* OUT2) {
  if (!F || !S || !OUT2) return fail(BSSN_B200_EINVAL, "constraint_norms: NULL operand");
  if (ng < 0 || 2LL * ng >= Sx || 2LL * ng >= Sy || 2LL * ng >= Sz)
    return fail(BSSN_B200_EINVAL, "constraint_norms: the interior [ng, S-ng) is empty");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 1, &grid);
  if (rc) return rc;
  if (!scratch) return fail(BSSN_B200_EINVAL, "constraint_norms: scratch is NULL");
  if (scratch_bytes < (size_t)grid * 2 * sizeof(double))
    return fail(BSSN_B200_EINVAL, "constraint_norms: scratch smaller than bssn_b200_norms_scratch_bytes()");
  a.F = F; a.S = S; a.ng = ng; a.partials = scratch;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = launch_single(3, bssn::MODE_NORM, a, st, grid);
  if (rc) return rc;
  const double count = (double)(Sx - 2 * ng) * (double)(Sy - 2 * ng) * (double)(Sz - 2 * ng);
  bssn::norm_finalize_kernel<<<1, 32, 0, st>>>(scratch, grid, count, OUT2);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("norm_finalize launch", e);
  return 0;
}

int bssn_b200_constraint_norms_static(void* stream, const double* F, const double* S, long long Sx,
                                      long long Sy, long long Sz, int ng, double* OUT2) {
  if (!F || !S || !OUT2) return fail(BSSN_B200_EINVAL, "constraint_norms_static: NULL operand");
  if (ng < 0 || 2LL * ng >= Sx || 2LL * ng >= Sy || 2LL * ng >= Sz)
    return fail(BSSN_B200_EINVAL, "constraint_norms_static: the interior [ng, S-ng) is empty");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail("cudaGetDevice", e);
  if (dev < 0 || dev >= kMaxDev) return fail(BSSN_B200_EINVAL, "constraint_norms_static: device ordinal out of range");
  // In host code g_static_norm_partials names a host-side stand-in, not device
  // memory: resolve its address on this device once, with the device current.
  // Two host threads that race here resolve the same address; the atomic slot
  // makes the publication well defined.
  static std::atomic<double*> addr[kMaxDev];
  double* partials = addr[dev].load(std::memory_order_acquire);
  if (!partials) {
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&partials), bssn::g_static_norm_partials);
    if (e != cudaSuccess) return cuda_fail("cudaGetSymbolAddress(static norm partials)", e);
    addr[dev].store(partials, std::memory_order_release);
  }
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 1, &grid);
  if (rc) return rc;
  if (grid > bssn::kStaticNormCtas)
    return fail(BSSN_B200_EINVAL, "constraint_norms_static: this launch needs " + std::to_string(grid) +
                                      " CTA partial sums but the static array holds " +
                                      std::to_string(bssn::kStaticNormCtas) +
                                      "; use bssn_b200_constraint_norms with a caller buffer");
  return bssn_b200_constraint_norms(stream, F, S, Sx, Sy, Sz, ng, partials,
                                    sizeof(double) * 2 * bssn::kStaticNormCtas, OUT2);
}

int bssn_b200_rk4_stage(void* stream, int stage, const double* U, const double* Y, double* ACC,
                        double* YNEXT, const double* S, double ko_sigma, int ko_order,
                        double chi_floor, double alpha_floor, long long Sx, long long Sy, long long Sz) {
  if (stage < 0 || stage > 3) return fail(BSSN_B200_EINVAL, "rk4_stage: stage must be 0..3");
  if (!U || !Y || !ACC || !YNEXT || !S) return fail(BSSN_B200_EINVAL, "rk4_stage: NULL operand");
  if (YNEXT == Y) return fail(BSSN_B200_EINVAL, "rk4_stage: YNEXT must not alias Y");
  if (stage < 3 && YNEXT == U) return fail(BSSN_B200_EINVAL, "rk4_stage: YNEXT may alias U only at stage 3");
  if (ACC == Y || ACC == U || ACC == YNEXT) return fail(BSSN_B200_EINVAL, "rk4_stage: ACC must not alias another operand");
  const bool use_ko = ko_sigma > 0.0;
  if (use_ko && ko_order != 6 && ko_order != 8) return fail(BSSN_B200_EINVAL, "rk4_stage: ko_order must be 6 or 8");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 1, &grid);
  if (rc) return rc;
  a.F = Y; a.U = U; a.ACC = ACC; a.OUT = YNEXT; a.S = S;
  a.stage = stage;
  a.use_ko = use_ko ? 1 : 0;
  a.ko_sigma = use_ko ? ko_sigma : 0.0;
  a.chi_floor = chi_floor; a.alpha_floor = alpha_floor;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (use_ko && ko_order == 8) return launch_single(4, bssn::MODE_STAGE, a, st, grid);
  return launch_single(3, bssn::MODE_STAGE, a, st, grid);
}

int bssn_b200_msrk_stage(void* stream, int stage, const double* U, const double* Y, double* ACC,
                         double* OUT, double* OUT2, double* OUT3, const double* S, const double* coef,
                         double ko_sigma, int ko_order, double chi_floor, double alpha_floor,
                         long long Sx, long long Sy, long long Sz) {
  if (stage < 0 || stage > 2) return fail(BSSN_B200_EINVAL, "msrk_stage: stage must be 0..2");
  if (!U || !Y || !OUT || !S || !coef) return fail(BSSN_B200_EINVAL, "msrk_stage: NULL operand");
  if (stage < 2 && !ACC) return fail(BSSN_B200_EINVAL, "msrk_stage: ACC is required at stages 0 and 1");
  if (stage == 0 && (!OUT2 || !OUT3)) return fail(BSSN_B200_EINVAL, "msrk_stage: OUT2 and OUT3 are required at stage 0");
  for (int i = 0; i < 9; ++i)
    if (!std::isfinite(coef[i])) return fail(BSSN_B200_EINVAL, "msrk_stage: coefficients must be finite");
  // Y is read with its stencil halo: no output may overwrite it
  if (OUT == Y || (stage < 2 && ACC == Y) || (stage == 0 && (OUT2 == Y || OUT3 == Y)))
    return fail(BSSN_B200_EINVAL, "msrk_stage: an output aliases the stage input Y");
  if (stage == 0) {
    const void* outs[4] = {ACC, OUT, OUT2, OUT3};
    for (int i = 0; i < 4; ++i) {
      if (outs[i] == U) return fail(BSSN_B200_EINVAL, "msrk_stage: stage-0 outputs must not alias U");
      for (int j = i + 1; j < 4; ++j)
        if (outs[i] == outs[j]) return fail(BSSN_B200_EINVAL, "msrk_stage: stage-0 outputs must be distinct");
    }
  } else if (stage == 1 && (ACC == U || ACC == OUT)) {
    return fail(BSSN_B200_EINVAL, "msrk_stage: ACC must not alias U or OUT at stage 1");
  }
  const bool use_ko = ko_sigma > 0.0;
  if (use_ko && ko_order != 6 && ko_order != 8) return fail(BSSN_B200_EINVAL, "msrk_stage: ko_order must be 6 or 8");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 1, &grid);
  if (rc) return rc;
  a.F = Y; a.U = U; a.ACC = ACC; a.OUT = OUT; a.OUT2 = OUT2; a.OUT3 = OUT3; a.S = S;
  for (int i = 0; i < 9; ++i) a.coef[i] = coef[i];
  a.ctime = stage == 0 ? 0.0 : (stage == 1 ? coef[0] + coef[1] : coef[2] + coef[3] + coef[4]);
  a.stage = stage;
  a.use_ko = use_ko ? 1 : 0;
  a.ko_sigma = use_ko ? ko_sigma : 0.0;
  a.chi_floor = chi_floor; a.alpha_floor = alpha_floor;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (use_ko && ko_order == 8) return launch_single(4, bssn::MODE_MSRK, a, st, grid);
  return launch_single(3, bssn::MODE_MSRK, a, st, grid);
}

int bssn_b200_derivatives(void* stream, const double* F, const double* S, double* DOUT,
                          double ko_sigma, int ko_order, long long Sx, long long Sy, long long Sz) {
  if (!F || !S || !DOUT) return fail(BSSN_B200_EINVAL, "derivatives: NULL operand");
  const bool use_ko = ko_sigma > 0.0;
  if (use_ko && ko_order != 6 && ko_order != 8) return fail(BSSN_B200_EINVAL, "derivatives: ko_order must be 6 or 8");
  bssn::Args a{};
  int grid = 0;
  int rc = prepare(&a, Sx, Sy, Sz, 3, &grid);
  if (rc) return rc;
  a.F = F; a.S = S; a.OUT = DOUT;
  a.use_ko = use_ko ? 1 : 0;
  a.ko_sigma = use_ko ? ko_sigma : 0.0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (use_ko && ko_order == 8) return launch_deriv<4, true>(a, st, grid);
  return use_ko ? launch_deriv<3, true>(a, st, grid) : launch_deriv<3, false>(a, st, grid);
}

int bssn_b200_rhs_algebra(void* stream, const double* F, const double* D, const double* S, double* OUT,
                          long long npts) {
  if (!F || !D || !S || !OUT) return fail(BSSN_B200_EINVAL, "rhs_algebra: NULL operand");
  if (npts < 1 || npts > (1LL << 31) - 1) return fail(BSSN_B200_EINVAL, "rhs_algebra: npts out of range");
  int sms = 0;
  int rc = device_sms(&sms);
  if (rc) return rc;
  long long blocks = (npts + 127) / 128;
  const long long cap = (long long)sms * 16;
  if (blocks > cap) blocks = cap;
  bssn::algebra_kernel<<<(int)blocks, 128, 0, static_cast<cudaStream_t>(stream)>>>(F, D, S, OUT, npts);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("rhs_algebra launch", e);
  return 0;
}

int bssn_b200_batch_rk4_stage_derivs(void* stream, int stage, const double* U, const double* Y, double* ACC,
                                     double* YNEXT, const double* D, const double* S, int ko_slots,
                                     double chi_floor, double alpha_floor, const bssn_b200_block* blocks,
                                     int nblocks, const long long* pts0, long long npoints) {
  if (stage < 0 || stage > 3) return fail(BSSN_B200_EINVAL, "batch_rk4_stage_derivs: stage must be 0..3");
  if (!U || !Y || !ACC || !YNEXT || !D || !S || !blocks || !pts0)
    return fail(BSSN_B200_EINVAL, "batch_rk4_stage_derivs: NULL operand");
  if (YNEXT == Y) return fail(BSSN_B200_EINVAL, "batch_rk4_stage_derivs: YNEXT must not alias Y");
  if (stage < 3 && YNEXT == U) return fail(BSSN_B200_EINVAL, "batch_rk4_stage_derivs: YNEXT may alias U only at stage 3");
  if (ACC == Y || ACC == U || ACC == YNEXT)
    return fail(BSSN_B200_EINVAL, "batch_rk4_stage_derivs: ACC must not alias another operand");
  if (nblocks < 1 || npoints < 1) return fail(BSSN_B200_EINVAL, "batch_rk4_stage_derivs: empty block list");
  int sms = 0;
  int rc = device_sms(&sms);
  if (rc) return rc;
  long long grid = (npoints + 127) / 128;
  const long long cap = (long long)sms * 16;
  if (grid > cap) grid = cap;
  bssn::stage_derivs_kernel<<<(int)grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      U, Y, ACC, YNEXT, D, ko_slots ? 162 : 138, S, stage, ko_slots ? 1 : 0, chi_floor, alpha_floor, blocks, nblocks,
      pts0, npoints);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("batch_rk4_stage_derivs launch", e);
  return 0;
}

int bssn_b200_advance_time(void* stream, double* S) {
  if (!S) return fail(BSSN_B200_EINVAL, "advance_time: NULL operand");
  bssn::advance_time_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(S);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("advance_time launch", e);
  return 0;
}

int bssn_b200_enforce(void* stream, double* U, long long npts, double chi_floor, double alpha_floor) {
  if (!U) return fail(BSSN_B200_EINVAL, "enforce: NULL operand");
  if (npts < 1) return fail(BSSN_B200_EINVAL, "enforce: npts must be >= 1");
  int sms = 0;
  int rc = device_sms(&sms);
  if (rc) return rc;
  long long blocks = (npts + 255) / 256;
  const long long cap = (long long)sms * 8;
  if (blocks > cap) blocks = cap;
  bssn::enforce_kernel<<<(int)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(U, npts, chi_floor, alpha_floor);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("enforce launch", e);
  return 0;
}

int bssn_b200_periodic_sync(void* stream, double* U, long long Sx, long long Sy, long long Sz, int ng) {
  if (!U) return fail(BSSN_B200_EINVAL, "periodic_sync: NULL operand");
  int rc = check_grid(Sx, Sy, Sz);
  if (rc) return rc;
  if (ng < 1 || 3LL * ng > Sx || 3LL * ng > Sy || 3LL * ng > Sz)
    return fail(BSSN_B200_EINVAL, "periodic_sync: need 1 <= ng and 3*ng <= every extent");
  int sms = 0;
  rc = device_sms(&sms);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long blocks = (Sx * Sy * Sz + 255) / 256, cap = 8LL * sms;
  bssn::periodic_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, st>>>(U, (int)Sx, (int)Sy, (int)Sz, ng);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("periodic_sync launch", e);
  return 0;
}

}  // extern "C"
