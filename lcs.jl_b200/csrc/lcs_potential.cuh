// lcs_potential.cuh -- the time-blocked HSMAC couple in potential form.
//
// A sweep of hsmac.jl:1-35 changes the velocity only by dp of the cells:
// U(i) += dxi (dp(i) - dp(i+1)), and P by dti dp.  With Phi(c) the sum of a
// cell's dp since the couple began, D its divergence then and c_a = 1/da^2,
//   div(c) = D(c) + sum_a c_a (2 Phi(c) - Phi(c - e_a) - Phi(c + e_a)),
//   Phi(c) += -omega dl div(c),
// so the couple needs one unknown and one right-hand side instead of U, V, W
// and P, and U, V, W, P are updated once at its end.  A cell is visited in the
// reference's order and sees the same div up to rounding (the sums are taken
// in another order); the fields agree with the element-wise sweeps to about
// 1e-15 in FP64.
//
// Periodic images.  The reference refills the halo once per group of three
// sweeps (time blocking, hsmac.jl:131-201) and sweeps the boxes [-1, n+3],
// [0, n+2] and [1, n+1]: the cells beyond the interior are swept redundantly
// and not quite as their images are, because the boxes shrink.  The flux
// through the face n uses Phi of cell n + 1, not of its image 1.  So with
// J = sum over the groups of Phi(1) - Phi(n+1), the velocity of that face is
// U0 + dxi (Phi(n) - Phi(1) + J), and a purely periodic Phi is right when
// D(n) gets + c J and D(1) gets - c J.  k_pot_jump adds each group's J to D
// (and keeps J for the last update of the velocity); the x jumps, one value
// per row, are added where D is read.
//
// One group = three red-black sweeps = six half sweeps, done in one pass over
// the grid (k_pot_sweep): 3 values of T a cell through HBM per group, against
// 24 for three element-wise sweeps.  With overlap, the first sweep visits the
// core [2, n] and then the z, y and x slabs of the rest one after the other
// (halo.jl:349-366): k_pot_slab computes Phi of the slabs after that sweep
// beforehand, in place, from the core cells next to them, which it computes too.
#pragma once

#include "../../include/lcs_b200.h"
#include "lcs_kernels.cuh"
#include "lcs_hsmac_rw.cuh"
#include "lcs_potential.h"

namespace lcs {
namespace {

template <typename T> __device__ __forceinline__ T pfma(T a, T b, T c);
template <> __device__ __forceinline__ double pfma<double>(double a, double b, double c) { return __fma_rn(a, b, c); }
template <> __device__ __forceinline__ float pfma<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// div of a cell from Phi = x, the sums of its neighbours along each axis and D.
// Each axis's second difference first, so that the roundings are those of the
// neighbours' sums, and exactly twice x is taken from them.  With k0 x, k0 the
// rounded 2 (cx + cy + cz), three multiply-adds fewer (a sweep 1 to 3 % faster:
// FP64 512^3 1.80 and 1.86 ms, 256^3 351 and 361 us), the error is larger than
// the element-wise sweeps' and not only by the sum's own roundings: k0's makes
// the operator one of Helmholtz.  300 sweeps, P against extended precision:
// FP64 64^3 8e-15, element by element 8e-16, and this 1.4e-16; FP32 512^3
// 1.3e-5, 6.4e-6 and 4e-7 (against FP64).
template <typename T>
__device__ __forceinline__ T pot_div(T x, T sx, T sy, T sz, T d, T cx, T cy, T cz) {
  return pfma<T>(cx, pfma<T>(T(2), x, -sx), pfma<T>(cy, pfma<T>(T(2), x, -sy), pfma<T>(cz, pfma<T>(T(2), x, -sz), d)));
}

__device__ __forceinline__ int pot_wrap(int i, int n) {  // 1-based image of i in -n < i
  i = i < 1 ? i + n : i;
  while (i > n) i -= n;
  return i;
}
// the two potentials: the group's input is spare buffer pot_cur, its output the other
template <typename T> __device__ __forceinline__ T* pot_buf(const Ctx* ctx, int which) {
  return (T*)ctx->vel[kSetSpare][which];
}
template <typename T> __device__ __forceinline__ T* pot_rhs(const Ctx* ctx) { return (T*)ctx->vel[kSetSpare][2]; }

// index of a coordinate among the layers kept compact of Phi / of D, -1 if it is none
__device__ __forceinline__ int pot_layer(int i, int nx) { return i <= 4 ? 2 + i : i >= nx - 2 ? i - (nx - 2) : -1; }
__device__ __forceinline__ int pot_dlayer(int i, int nx) { return i <= 3 ? 1 + i : i >= nx - 1 ? i - (nx - 1) : -1; }

// Start of a couple: D = div U (periodic, in FP64, rounded once), Phi = 0, J = 0.
// Bound by HBM: 3 fields read, 2 written (512^3: FP64 1.2 ms, FP32 0.75).
template <typename T>
__global__ void __launch_bounds__(256) k_pot_setup(const __grid_constant__ PotGroup<T> ga, Grid g, int set, PotGeom pg) {
  const int m = blockIdx.y;
  Ctx* ctx = ga.ctx[m];
  const T* U = (const T*)ctx->vel[set][0];
  const T* V = (const T*)ctx->vel[set][1];
  const T* W = (const T*)ctx->vel[set][2];
  T* phi = pot_buf<T>(ctx, 0);
  T* D = pot_rhs<T>(ctx);
  T* s = ga.scratch[m];
  const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const int hx = nx / 2;
  const int total = hx * ny * nz;  // < 2^31 (host)
  for (int t = blockIdx.x * 256 + threadIdx.x; t < total; t += gridDim.x * 256) {
    const int i = 1 + 2 * (t % hx);
    const int u = t / hx;
    const int j = 1 + u % ny, k = 1 + u / ny;
    const int64_t c = g.at(i, j, k);
    const int64_t cw = i > 1 ? c - 1 : g.at(nx, j, k);
    const int64_t cs = j > 1 ? c - g.px : g.at(i, ny, k);
    const int64_t cb = k > 1 ? c - g.pz : g.at(i, j, nz);
    const double ua = U[cw], ub = U[c], uc = U[c + 1];
    const double a = pg.dxi * (ub - ua) + pg.dyi * ((double)V[c] - (double)V[cs]) + pg.dzi * ((double)W[c] - (double)W[cb]);
    const double b = pg.dxi * (uc - ub) + pg.dyi * ((double)V[c + 1] - (double)V[cs + 1]) +
                     pg.dzi * ((double)W[c + 1] - (double)W[cb + 1]);
    const int o = pg.s.at(i, j, k);
    st2<T>(D + o, (T)a, (T)b);
    st2<T>(phi + o, T(0), T(0));
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int l = pot_dlayer(i + q, nx);
      if (l >= 0) s[pg.s.dx + ((int64_t)l * nz + (k - 1)) * ny + (j - 1)] = (T)(q ? b : a);
    }
  }
  // Phi next to the faces, and the jumps
  const int64_t zero = pg.s.dx - pg.s.l[0];
  for (int64_t t = blockIdx.x * 256 + threadIdx.x; t < zero; t += gridDim.x * 256) s[pg.s.l[0] + t] = T(0);
  for (int64_t t = pg.s.j[0] + blockIdx.x * 256 + threadIdx.x; t < pg.s.total; t += gridDim.x * 256) s[t] = T(0);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctx->pot_cur = 0;
    ctx->pot_pending = 0;
    ctx->pot_redo = 0;
    ctx->pot_round = 0.0;
    ctx->pot_since = 0;
    ctx->pot_check = 0;
  }
}

// The exit tests of a group's three sweeps, from their sums of div^2 (FP32:
// each with `round`, that of the stored velocity).  The state of the loop and
// of the potential after them.
__device__ __forceinline__ void pot_exit(Ctx* ctx, const HsmacCoef& cf, const double sum[3], double round) {
  int again = 0;  // the exit lies inside the group: run it again up to that sweep
  for (int q = 0; q < 3; q++) {
    hsmac_check(ctx, cf, sum[q] + round, 1);
    if (ctx->cs.done) {
      if (q < 2 && isfinite(ctx->cs.div)) again = q + 1;
      break;
    }
  }
  if (again) {
    ctx->cs.done = 0;
    ctx->cs.cont = 1;
  }
  ctx->pot_redo = again;
  ctx->pot_pending = again ? 0 : 1;
  if (!again) ctx->pot_cur = 1 - ctx->pot_cur;
}

// FP32: this block's share of the sum over the cells of e^2, where e is the
// divergence of the velocity as it would be stored for the potential `phi` (a
// group's output, its jumps pending) less the divergence that the sweeps see
// there.  It holds every rounding between the two: of the velocity's faces, of
// D and of the sweeps' own sums.  Bound by the latency of its loads.
template <typename T>
__device__ __forceinline__ double pot_round_sum(const Ctx* ctx, const Grid& g, int set, const T* __restrict__ phi,
                                                const T* __restrict__ s, const PotGeom& pg) {
  const T* __restrict__ U = (const T*)ctx->vel[set][0];
  const T* __restrict__ V = (const T*)ctx->vel[set][1];
  const T* __restrict__ W = (const T*)ctx->vel[set][2];
  const T* __restrict__ D = pot_rhs<T>(ctx);
  const int nx = pg.s.nx, ny = pg.s.ny, nz = pg.s.nz, px = pg.s.px, pz = pg.s.pz;
  const T cx = (T)pg.cx, cy = (T)pg.cy, cz = (T)pg.cz;
  double acc = 0.0;
  const int hx = nx / 2, total = hx * ny * nz;  // < 2^31 (host)
  // of a cell and an axis: the divergence of its two faces as stored, and the
  // sum of its two neighbours as the sweeps see them.  lo, hi: the neighbours'
  // images; a, b: the low and the high face's velocity; first, last: the cell
  // lies there, f: its place on that face.
  auto axis = [&](int ax, T p, T lo, T hi, T a, T b, bool first, bool last, int f, double di, T* nsum) {
    T vlo = p, vhi = hi;  // the high neighbour of the low face's cell, and of this one, as k_pot_apply has them
    T slo = lo, shi = hi;
    if (first || last) {
      const T e = s[pg.s.e[ax] + f], head = first ? p : hi;  // Phi(1)
      const T jmp = s[pg.s.j[ax] + f] + (head - e);
      if (first) {
        vlo = head - jmp;
        slo = lo + (head - e);
      }
      if (last) {
        vhi = head - jmp;
        shi = e;
      }
    }
    *nsum = slo + shi;
    const T d = (T)di;
    return di * ((double)pfma<T>(d, p - vhi, b) - (double)pfma<T>(d, lo - vlo, a));
  };
  for (int t = blockIdx.x * 256 + threadIdx.x; t < total; t += gridDim.x * 256) {
    const int i = 1 + 2 * (t % hx), r = t / hx, j = 1 + r % ny, k = 1 + r / ny;
    const int o = pg.s.at(i, j, k);
    const int64_t c = g.at(i, j, k);
    const bool x1 = i == 1, xn = i + 1 == nx, y1 = j == 1, yn = j == ny, z1 = k == 1, zn = k == nz;
    const pair_t<T> p = lds2(phi + o), u = lds2(U + c), v = lds2(V + c), w = lds2(W + c);
    const T pw = phi[x1 ? o + (nx - 1) : o - 1], pe = phi[xn ? o - (nx - 2) : o + 2], uw = U[x1 ? c + (nx - 1) : c - 1];
    const pair_t<T> ps = lds2(phi + (y1 ? o + (ny - 1) * px : o - px)), pn = lds2(phi + (yn ? o - (ny - 1) * px : o + px));
    const pair_t<T> pb = lds2(phi + (z1 ? o + (nz - 1) * pz : o - pz)), pt = lds2(phi + (zn ? o - (nz - 1) * pz : o + pz));
    const pair_t<T> vs = lds2(V + (y1 ? g.at(i, ny, k) : c - g.px)), wb = lds2(W + (z1 ? g.at(i, j, nz) : c - g.pz));
    pair_t<T> d = lds2(D + o);  // (without the x jumps so far)
    const int fx = (k - 1) * ny + (j - 1), fy = (k - 1) * nx + (i - 1), fz = (j - 1) * nx + (i - 1);
    if (x1) d.x -= cx * s[pg.s.j[0] + fx];
    if (xn) d.y += cx * s[pg.s.j[0] + fx];
    T sx, sy, sz;
    double div = axis(0, p.x, pw, p.y, uw, u.x, x1, false, fx, pg.dxi, &sx);
    div += axis(1, p.x, ps.x, pn.x, vs.x, v.x, y1, yn, fy, pg.dyi, &sy);
    div += axis(2, p.x, pb.x, pt.x, wb.x, w.x, z1, zn, fz, pg.dzi, &sz);
    const double ea = div - (double)pot_div<T>(p.x, sx, sy, sz, d.x, cx, cy, cz);
    div = axis(0, p.y, p.x, pe, u.x, u.y, false, xn, fx, pg.dxi, &sx);
    div += axis(1, p.y, ps.y, pn.y, vs.y, v.y, y1, yn, fy + 1, pg.dyi, &sy);
    div += axis(2, p.y, pb.y, pt.y, wb.y, w.y, z1, zn, fz + 1, pg.dzi, &sz);
    const double eb = div - (double)pot_div<T>(p.y, sx, sy, sz, d.y, cx, cy, cz);
    acc += ea * ea + eb * eb;
  }
  return acc;
}

// FP32, after a couple that ran to its last sweep: the rounding of the stored
// velocity into the residual that the log shows (a couple that left by the exit
// test has it: k_pot_jump).  12 us at 32^3, 71 at 192^3, 0.92 ms at 512^3
// (a cell a thread 1.8).
template <typename T>
__global__ void __launch_bounds__(256) k_pot_round(const __grid_constant__ PotGroup<T> ga, Grid g, int set, PotGeom pg,
                                                   HsmacCoef cf) {
  __shared__ double red[8];
  __shared__ int last;
  const int m = blockIdx.y;
  Ctx* ctx = ga.ctx[m];
  if (ctx->cs.done || !ctx->pot_pending) return;
  const double acc = pot_round_sum<T>(ctx, g, set, pot_buf<T>(ctx, ctx->pot_cur), ga.scratch[m], pg);
  const double b = block_sum<256>(acc, red);
  if (threadIdx.x == 0) ga.partials[m][blockIdx.x] = b;
  if (!last_block(&ctx->ticket, gridDim.x, &last)) return;
  const double sum = sum_partials<256>(ga.partials[m], (int)gridDim.x, red);
  if (threadIdx.x != 0) return;
  ctx->ticket = 0;
  ctx->pot_round = sum * (cf.count / ((double)pg.s.nx * pg.s.ny * pg.s.nz));
  ctx->cs.sum = ctx->pot_sum[2] + ctx->pot_round;
  ctx->cs.div = sqrt(ctx->cs.sum / cf.count);
}

// The last group's jumps into J and D (nothing when it has none pending: the
// first group, and a group that is run again).  One thread per face cell; the
// cells of two faces belong to the z face, so each D is written once.  Bound by
// its launch (3 us up to 256^3, 10 at 512^3).
//
// FP32: the exit test is on the divergence of the velocity, which is stored in
// FP32, and that rounding has a divergence of its own that the potential does
// not show (u_rms 1: 3.3e-7, 6.4e-7 and 1.28e-6 rms at 32^3, 64^3 and 128^3).
// So when a sweep's own residual would let the couple end, its group's tests
// wait (pot_check = 1): this kernel, the first of the next group, measures the
// rounding at the group's output (pot_round_sum) and its last block runs the
// tests; that group's other kernels do nothing (cs.cont = 2 until the next one).
// A measurement holds for the sweeps after it while it keeps the residual above
// the exit by a factor of two in the square, for at most kPotRoundAge of them
// (a couple at 32^3 passes an exit of 1e-8 after about 180 sweeps and goes on to
// 300: one measurement, 25 us; every 24 sweeps they took 8 % of a step).
// Its registers are bounded for the jumps' sake (512^3: FP32 23 us with 64, 34
// with 96; FP64 22 us with 32, 26 with 62).
constexpr int kPotRoundAge = 256;
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 7)
    k_pot_jump(const __grid_constant__ PotGroup<T> ga, Grid g, int set, PotGeom pg, HsmacCoef cf, PotLoop loop) {
  const int m = blockIdx.y;
  Ctx* ctx = ga.ctx[m];
  const int done = ctx->cs.done, cont = ctx->cs.cont, pending = ctx->pot_pending, check = ctx->pot_check;  // one latency
  if (done || !cont) return;
  if constexpr (sizeof(T) == 4) {
    if (check) {
      __shared__ double red[8];
      __shared__ int last;
      const double acc = pot_round_sum<T>(ctx, g, set, pot_buf<T>(ctx, 1 - ctx->pot_cur), ga.scratch[m], pg);
      const double b = block_sum<256>(acc, red);
      if (threadIdx.x == 0) ga.partials[m][blockIdx.x] = b;
      if (!last_block(&ctx->ticket, gridDim.x, &last)) return;
      const double sum = sum_partials<256>(ga.partials[m], (int)gridDim.x, red);
      if (threadIdx.x != 0) return;
      ctx->ticket = 0;
      ctx->pot_round = sum * (cf.count / ((double)pg.s.nx * pg.s.ny * pg.s.nz));
      ctx->pot_since = ctx->cs.itr;
      ctx->pot_check = 0;
      pot_exit(ctx, cf, ctx->pot_sum, ctx->pot_round);
      if (ctx->cs.cont) ctx->cs.cont = 2;
      if (loop.on) cudaGraphSetConditional(loop.handle, couple_goes_on(ctx, loop.max_groups) ? 1u : 0u);
      return;
    }
    if (cont == 2 && blockIdx.x == 0 && threadIdx.x == 0) ctx->cs.cont = 1;  // (2 or 1: the other blocks go on alike)
  }
  if (!pending) return;
  const int nx = pg.s.nx, ny = pg.s.ny, nz = pg.s.nz;
  T* D = pot_rhs<T>(ctx);
  T* s = ga.scratch[m];
  const int fx = ny * nz, fy = nx * nz, fz = nx * ny;
  T* dxl = s + pg.s.dx;
  const T cx = (T)pg.cx, cy = (T)pg.cy, cz = (T)pg.cz;
  auto at = [&](int i, int j, int k) { return pg.s.at(i, j, k); };
  // Phi(1) is layer 3 of the seven
  auto jx = [&](int j, int k) {
    const int f = (k - 1) * ny + (j - 1);
    return s[pg.s.l[0] + (int64_t)3 * fx + f] - s[pg.s.e[0] + f];
  };
  auto jy = [&](int i, int k) {
    const int f = (k - 1) * nx + (i - 1);
    return s[pg.s.l[1] + (int64_t)3 * fy + f] - s[pg.s.e[1] + f];
  };
  auto jz = [&](int i, int j) {
    const int f = (j - 1) * nx + (i - 1);
    return s[pg.s.l[2] + (int64_t)3 * fz + f] - s[pg.s.e[2] + f];
  };
  for (int t = blockIdx.x * 256 + threadIdx.x; t < fx + fy + fz; t += gridDim.x * 256) {
    if (t < fz) {  // z faces: k = 1 and k = n, with the y jumps of their rows j = 1, n
      const int i = 1 + t % nx, j = 1 + t / nx;
      const T d = jz(i, j);
      s[pg.s.j[2] + t] += d;
      T lo = -(cz * d), hi = cz * d;
      if (j == 1 || j == ny) {
        const T sg = j == 1 ? -cy : cy;
        lo += sg * jy(i, 1);
        hi += sg * jy(i, nz);
      }
      D[at(i, j, 1)] += lo;
      D[at(i, j, nz)] += hi;
    } else if (t < fz + fy) {
      const int u = t - fz, i = 1 + u % nx, k = 1 + u / nx;
      const T d = jy(i, k);
      s[pg.s.j[1] + u] += d;
      if (k > 1 && k < nz) {
        D[at(i, 1, k)] -= cy * d;
        D[at(i, ny, k)] += cy * d;
      }
    } else {  // the x jumps, and the compact x layers of D (which hold every jump)
      const int u = t - fz - fy, j = 1 + u % ny, k = 1 + u / ny;
      const T d = jx(j, k);
      s[pg.s.j[0] + u] += d;
      const bool ye = j == 1 || j == ny, ze = k == 1 || k == nz;
#pragma unroll
      for (int l = 0; l < kPotDLayers; l++) {
        const int i = l < 2 ? nx - 1 + l : l - 1;
        T add = l == 1 ? cx * d : l == 2 ? -(cx * d) : T(0);
        if (ye) add += (j == 1 ? -cy : cy) * jy(i, k);
        if (ze) add += (k == 1 ? -cz : cz) * jz(i, j);
        if (l == 1 || l == 2 || ye || ze) dxl[(int64_t)l * fx + u] += add;
      }
    }
  }
}

// The first sweep of an overlap group next to the faces, into the halo and the
// outer layers of Phi: the slabs (positions -1 .. 1 and n+1 .. n+3 along an
// axis; z slabs first, then y, then x), and of the core, which comes before
// them, the layers 2 and n (both colours) and colour 0 of the layers 3 and
// n-1.  With these in place k_pot_sweep leaves them alone in its first sweep
// and never needs the values from before it: colour 0 of layer 4 reads colour
// 1 of layer 3, which is not touched here, and colour 1 of layer 3 reads
// colour 0, which is final.
//
// A block takes 32 x 32 columns along one axis AX through both slabs: the low
// one needs Phi at -2 .. 4 and the high one at n-2 .. n+4, the same 7 images
// (n-2, n-1, n, 1, 2, 3, 4; kept compact by k_pot_sweep, since along x they
// would be two sectors of every row), and D at 5 of them.  Phases, in-plane
// neighbours through shared memory and a barrier between them: colours 0 and 1
// of the core, then of the z slabs, the y slabs and the x slabs, as far as the
// block's columns and its axis need them.  Blocks at the rim of a y or x slab
// so sweep the few cells of the earlier slabs beside it themselves, and no
// block waits for another: one launch for the three axes.  A cell that two
// blocks sweep is stored by one of them; the other's may differ from it in the
// last bits, since a block sums the axes in its own order and an x block's D has
// its jumps added one by one.  Bound by the latency of its loads and its four to
// eight phases (17 to 19 us up to 128^3, 98 and 112 at 512^3 in FP32 and FP64).
// A value reaches at most 5 columns (both colours of the x, the y and the z slab,
// where the y slab crosses to the z slab in place), so 22 x 22 of the columns are
// the block's own.
template <typename T, int AX>
__device__ __forceinline__ void pot_slab_body(const PotGroup<T>& ga, const PotGeom& pg, int m, int tile, T* sh,
                                              double* red) {
  constexpr int PL = 1024;
  Ctx* ctx = ga.ctx[m];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = threadIdx.x;
  const int nx = pg.s.nx, ny = pg.s.ny, nz = pg.s.nz;
  const int n[3] = {nx, ny, nz};
  constexpr int UA = AX == 0 ? 1 : 0, VA = AX == 2 ? 1 : 2;
  const int nu = n[UA], nv = n[VA], nn = n[AX];
  const int ulo = AX == 0 ? 2 : -1, uhi = AX == 0 ? nu : nu + 3;
  const int vlo = AX == 2 ? -1 : 2, vhi = AX == 2 ? nv + 3 : nv;
  const int gu = (uhi - ulo + kPotSlab) / kPotSlab;
  const int u0 = ulo + (tile % gu) * kPotSlab - 5, v0 = vlo + (tile / gu) * kPotSlab - 5;
  const int u = u0 + tx, v = v0 + ty;
  T* phi = pot_buf<T>(ctx, ctx->pot_cur);
  const T* D = pot_rhs<T>(ctx);
  const T* s = ga.scratch[m];
  const int uw = pot_wrap(u, nu), vw = pot_wrap(v, nv);
  const int64_t face = (int64_t)nu * nv, f = (int64_t)(vw - 1) * nu + (uw - 1);
  const bool mine = tx >= 5 && tx < 5 + kPotSlab && ty >= 5 && ty < 5 + kPotSlab && u <= uhi && v <= vhi;
  // what the column's cells are: its place in the core and in the slabs of the two other axes
  const bool uc = u >= 2 && u <= nu, vc = v >= 2 && v <= nv;
  const bool ur = u >= -1 && u <= nu + 3, vr = v >= -1 && v <= nv + 3;
  const bool isC = uc && vc;
  const bool isZ = AX == 2 ? ur && vr : ur && vr && !vc;
  const bool isY = AX == 1 ? ur && vc : AX == 0 && ur && !uc && vc;
  T lo[7], hi[7], d[5];
  // images n-2, n-1, n, 1, 2, 3, 4 of the column
#pragma unroll
  for (int q = 0; q < 7; q++) {
    const int w = q < 3 ? nn - 2 + q : q - 2;
    lo[q] = hi[q] = s[pg.s.l[AX] + q * face + f];
    if (q >= 1 && q <= 5) {
      if constexpr (AX == 2) d[q - 1] = D[pg.s.at(uw, vw, w)];
      if constexpr (AX == 1) d[q - 1] = D[pg.s.at(uw, w, vw)];
      if constexpr (AX == 0) d[q - 1] = s[pg.s.dx + (q - 1) * face + f];
      if constexpr (AX != 0) {  // the x jump of D
        if (uw == 1 || uw == nx) {
          const T jv = s[pg.s.j[0] + (AX == 2 ? (int64_t)(w - 1) * ny + (vw - 1) : (int64_t)(vw - 1) * ny + (w - 1))];
          d[q - 1] += (uw == 1 ? -(T)pg.cx : (T)pg.cx) * jv;
        }
      }
    }
  }
  const T cu = (T)(UA == 0 ? pg.cx : pg.cy), cv = (T)(VA == 1 ? pg.cy : pg.cz),
          cn = (T)(AX == 0 ? pg.cx : AX == 1 ? pg.cy : pg.cz), wd = (T)pg.wd;
  // planes in shared memory: lo 1 .. 5, then hi 1 .. 5
#pragma unroll
  for (int q = 0; q < 5; q++) {
    sh[q * PL + c] = lo[1 + q];
    sh[(5 + q) * PL + c] = hi[1 + q];
  }
  const int cl = tx > 0 ? c - 1 : c, cr = tx < 31 ? c + 1 : c, cd = ty > 0 ? c - 32 : c, cup = ty < 31 ? c + 32 : c;
  const int par = (u + v) & 1;
  double acc = 0.0;
  // one cell: layer q of `a`, in shared memory in the planes from `base`
  // (cells of one colour never read each other: in place)
  auto relax = [&](T* a, int q, int base, bool count) {
    T* p = sh + (base + q - 1) * PL;
    const T su = p[cl] + p[cr], sv = p[cd] + p[cup], sn = a[q - 1] + a[q + 1];
    const T div = pot_div<T>(a[q], su, sv, sn, d[q - 1], cu, cv, cn);
    a[q] = pfma<T>(wd, div, a[q]);
    p[c] = a[q];
    if (count) acc += (double)div * (double)div;
  };
  // positions: lo q -> q - 2, hi q -> n - 2 + q (n even): both have the parity of q
  auto has = [&](int q, int color) { return ((par + q) & 1) == color; };
  // core cells of these layers that belong to an axis before this one: it
  // stores them and counts them in the residual (each cell once, whatever the
  // order of the blocks)
  auto outer = [&](int p, int pn, int c0) { return p == 2 || p == pn || (c0 == 0 && (p == 3 || p == pn - 1)); };
  auto own_core = [&](int c0) { return mine && isC && !(AX != 2 && outer(v, nv, c0)) && !(AX == 0 && outer(u, nu, c0)); };
  // a colour of the slab cells: lo 1-3, hi 3-5 (this axis's own slabs), or of
  // the columns in another slab: all layers
  auto slab = [&](bool is, int color, bool own) {
    __syncthreads();
    if (!is) return;
    const bool count = own && mine && u >= 1 && u <= nu + 1 && v >= 1 && v <= nv + 1;  // cells 1 and n+1 count
#pragma unroll
    for (int q = 1; q <= 5; q++)
      if (has(q, color) && (q <= 3 || !own)) relax(lo, q, 0, count && q == 3);
#pragma unroll
    for (int q = 1; q <= 5; q++)
      if (has(q, color) && (q >= 3 || !own)) relax(hi, q, 5, count && q == 3);
  };
  __syncthreads();
  if (isC) {  // colour 0 of the core layers 2, 3 and n-1, n
    const bool count = own_core(0);
    if (has(4, 0)) {
      relax(lo, 4, 0, count);
      relax(hi, 2, 5, count);
    } else {
      relax(lo, 5, 0, count);
      relax(hi, 1, 5, count);
    }
  }
  __syncthreads();
  if (isC && has(4, 1)) {  // colour 1 of the layers 2 and n
    const bool count = own_core(1);
    relax(lo, 4, 0, count);
    relax(hi, 2, 5, count);
  }
  if (AX == 2 || v0 <= 1 || v0 + 31 > nv) {  // (the same for the whole block)
    slab(isZ, 0, AX == 2);
    slab(isZ, 1, AX == 2);
  }
  if constexpr (AX != 2) {
    if (AX == 1 || u0 <= 1 || u0 + 31 > nu) {
      slab(isY, 0, AX == 1);
      slab(isY, 1, AX == 1);
    }
  }
  if constexpr (AX == 0) {
    slab(isC, 0, true);
    slab(isC, 1, true);
  }
  if (mine) {
    auto put = [&](int p, T val) {
      phi[AX == 2 ? pg.s.at(u, v, p) : AX == 1 ? pg.s.at(u, p, v) : pg.s.at(p, u, v)] = val;
    };
#pragma unroll
    for (int q = 0; q < 3; q++) {
      put(q - 1, lo[1 + q]);
      put(nn + 1 + q, hi[3 + q]);
    }
    if (own_core(has(4, 0) ? 0 : 1)) {
      put(2, lo[4]);
      put(nn, hi[2]);
    }
    if (has(5, 0) && own_core(0)) {
      put(3, lo[5]);
      put(nn - 1, hi[1]);
    }
  }
  const double sum = block_sum<kPotSlabThreads>(acc, red);
  if (threadIdx.x == 0) ga.partials[m][pg.slab_part + blockIdx.x] = sum;
}
// blocks: the tiles of the z slabs, then of the y and x slabs (slab0: first tile of each axis)
template <typename T>
__global__ void __launch_bounds__(kPotSlabThreads) k_pot_slab(const __grid_constant__ PotGroup<T> ga, PotGeom pg) {
  extern __shared__ __align__(16) unsigned char pot_smem[];
  __shared__ double red[32];
  const int m = blockIdx.y, b = blockIdx.x;
  const Ctx* ctx = ga.ctx[m];
  // (a group that runs again finds these in place)
  const int done = ctx->cs.done, cont = ctx->cs.cont, redo = ctx->pot_redo;
  if (done || cont != 1 || redo) return;
  T* sh = (T*)pot_smem;  // [10][32][32]
  if (b < pg.slab0[1]) pot_slab_body<T, 2>(ga, pg, m, b, sh, red);
  else if (b < pg.slab0[0]) pot_slab_body<T, 1>(ga, pg, m, b - pg.slab0[1], sh, red);
  else pot_slab_body<T, 0>(ga, pg, m, b - pg.slab0[0], sh, red);
}

// Zero where a mask word is zero (a select without a branch, also for NaN).
__device__ __forceinline__ float pot_keep(float v, int mask) { return __int_as_float(__float_as_int(v) & mask); }
__device__ __forceinline__ double pot_keep(double v, int mask) {
  return __hiloint2double(__double2hiint(v) & mask, __double2loint(v) & mask);
}

// Three red-black sweeps (six half sweeps) in one pass.
//
// A CTA owns TX x TY columns and streams along z: at plane t it loads plane t,
// then half sweep h = 1 .. 6 runs at plane t - h, and plane t - 6 is stored.
// Half sweep h of a cell reads its z neighbours as half sweep h - 1 left them
// (planes t - h - 1 and t - h + 1, registers of this thread), its x neighbours
// (the pair's other cell and the adjacent lane's) and its y neighbours (rows
// of this thread, or of the warps above and below through shared memory, which
// they wrote one plane ago): one barrier a plane.  Every half sweep makes one
// more cell at the tile's edge invalid, hence the 6 cells around the outputs;
// nothing there is masked.  Colours: with x-pairs (odd, even) the cell that
// half sweep h updates at plane t - h is the pair's left one in every second
// row and plane, whatever h; planes go by twos (template U), so the side and
// the registers are known at compile time.
// Planes whose half sweeps all lie where every box reaches run without masks
// (FULL); elsewhere one bit test per cell and half sweep.
//
// With overlap, k_pot_slab has put the first sweep's values into the halo and
// the outer layers; without, the halo is the periodic image, read in place
// (pairs never straddle the period: n is even).
//
// A launch at 512^3: FP32 1.10 ms (12 x 4 rows), FP64 1.86 ms (8 x 4), where the
// three element-wise sweeps with their slabs and fill take 3.7 and 6.2; at the
// HBM peak its 3 values a cell take 0.25 and 0.49.  It is bound by instruction
// issue and latency (FP32 at 384^3, FP64 at 256^3): issue 47 and 27 % of the
// cycles (63 and 44 % of those of an SM that has a CTA), DRAM 19 and 16 %, the
// shared-memory pipe 44 and 54 %.  The tile is as tall as the
// registers allow (168 and 254 a thread): a row's two colours at 7 planes live
// in them, and D, read once in three half sweeps each, in shared memory.
template <typename T, int NW, int RW>
__global__ void __launch_bounds__(PotTile<T, NW, RW>::NT, 1)
    k_pot_sweep(const __grid_constant__ PotGroup<T> ga, PotGeom pg, HsmacCoef cf, PotLoop loop) {
  using L = PotTile<T, NW, RW>;
  using T2 = pair_t<T>;
  constexpr int UF = 2;  // planes between two moves of the registers
  constexpr int NP = UF + 7;  // registers of a colour: planes t .. t - 7 and UF - 1 more
  extern __shared__ __align__(16) unsigned char pot_smem[];
  __shared__ double red[32];
  __shared__ int last_flag;
  T* sD = (T*)pot_smem;                // [6][2][ROWS][32]
  T* sX = (T*)pot_smem + L::d_elems;   // [2][6][NW][2][32]
  int* sZ = (int*)((T*)pot_smem + L::d_elems + L::x_elems);  // box bits of the planes kb - 13 ..
  const int m = blockIdx.y;
  Ctx* ctx = ga.ctx[m];
  const int done = ctx->cs.done, cont = ctx->cs.cont, cur = ctx->pot_cur, redo = ctx->pot_redo;
  if (done || cont != 1) return;
  const int nsw = redo ? redo : 3;  // sweeps of this pass
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nx = pg.s.nx, ny = pg.s.ny, nz = pg.s.nz;
  const T* __restrict__ phi = pot_buf<T>(ctx, cur);
  const T* __restrict__ D = pot_rhs<T>(ctx);
  T* __restrict__ out = pot_buf<T>(ctx, 1 - cur);
  T* __restrict__ s = ga.scratch[m];
  const T cx = (T)pg.cx, cy = (T)pg.cy, cz = (T)pg.cz, wd = (T)pg.wd;

  double racc[3] = {0.0, 0.0, 0.0};

  // a z chunk of a tile column, in units of two planes
  const int nu = (nz + 2) / 2, col = blockIdx.x / pg.nc, ch = blockIdx.x % pg.nc;
  const int ua = (int)((int64_t)ch * nu / pg.nc), ub = (int)((int64_t)(ch + 1) * nu / pg.nc);
  const int x0 = 1 + (col % pg.gx) * L::TX, y0 = 1 + (col / pg.gx) * L::TY;  // both odd
  const int kb = 1 + 2 * ua, ke = min(nz + 1, 2 * ub);                       // kb odd
  const int xL = x0 - 6 + 2 * lane;
  const int j0 = y0 - 6 + w * RW;
  const int xw = pot_wrap(xL, nx);  // xw odd: the pair (xw, xw + 1)
  // where a position's Phi is: itself (clamped: positions past -1 .. n+3 are never used), or its image
  auto where = [&](int i, int n) { return pg.overlap ? max(-1, min(i, n + 3)) : pot_wrap(i, n); };
  uint32_t roff[RW], doff[RW];  // byte offsets within a plane
#pragma unroll
  for (int r = 0; r < RW; r++) {
    roff[r] = (uint32_t)(pg.s.at(where(xL, nx), where(j0 + r, ny), -1) * sizeof(T));
    doff[r] = (uint32_t)(pg.s.at(xw, pot_wrap(j0 + r, ny), -1) * sizeof(T));
  }
  auto cell = [](const T* base, uint32_t off) { return reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off); };

  // boxes a coordinate lies in: bits 0, 1 the first sweep's two colours, 2 and
  // 3 the second and third sweeps; bits 4 .. 7 the same and the tile's own; 8 its own
  const int o0 = pg.overlap ? 4 : -1, o1 = pg.overlap ? -2 : 3, o2 = pg.overlap ? 3 : -1, o3 = pg.overlap ? -1 : 3;
  auto bits = [&](int i, int n, int olo, int ohi) {
    const int in = (int)(i >= o0 && i <= n + o1) | (int)(i >= o2 && i <= n + o3) << 1 |
                   (int)(i >= 0 && i <= n + 2 && nsw > 1) << 2 | (int)(i >= 1 && i <= n + 1 && nsw > 2) << 3;
    const bool own = i >= olo && i <= ohi && i <= n + 1;
    return in | (own ? in << 4 | 256 : 0);
  };
  int mL[RW], mR[RW];  // of the pair's cells
  {
    const int bL = bits(xL, nx, x0, x0 + L::TX - 1), bR = bits(xL + 1, nx, x0, x0 + L::TX - 1);
#pragma unroll
    for (int r = 0; r < RW; r++) {
      const int by = bits(j0 + r, ny, y0, y0 + L::TY - 1);
      mL[r] = bL & by;
      mR[r] = bR & by;
    }
  }
  int keep[RW];  // all ones where the pair is the tile's own
#pragma unroll
  for (int r = 0; r < RW; r++) {
    keep[r] = (mL[r] & 256) ? -1 : 0;
    asm volatile("" : "+r"(keep[r]));  // (else turned back into a test and a select for each use)
  }
  // the tile holds cells of the layers next to the faces, or past them
  const bool edge_y = j0 <= 4 || j0 + RW - 1 >= ny - 2, edge_x = xL <= 3 || xL >= nx - 3;
  const bool xyf = nsw == 3 && x0 - 5 >= 4 && x0 + L::TX + 4 <= nx - 2 && y0 - 5 >= 4 && y0 + L::TY + 4 <= ny - 2;
  // planes whose half sweeps all run, and are owned, without masks
  const int zf_lo = xyf ? max(kb, 4) + 6 : INT_MAX, zf_hi = min(ke, nz - 2) + 1;
  // the x jump: D of image 1 (the pair's left cell) and of image n (its right one)
  const bool jump1 = xw == 1, jumpn = xw + 1 == nx;
  int jrow[RW];
#pragma unroll
  for (int r = 0; r < RW; r++) jrow[r] = pot_wrap(j0 + r, ny) - 1;
  const int wlo = w > 0 ? w - 1 : 0, whi = w < NW - 1 ? w + 1 : NW - 1;

  T A[RW][NP], B[RW][NP];  // colours 0 and 1 of the pair
  T2 pf[RW], pd[RW];       // the next plane, in flight
  T jx[RW];                // its x jump
#pragma unroll
  for (int r = 0; r < RW; r++) {
#pragma unroll
    for (int q = 0; q < NP; q++) A[r][q] = B[r][q] = T(0);
    jx[r] = T(0);
  }
  for (int q = tid; q < (int)(L::d_elems + L::x_elems); q += L::NT) sD[q] = T(0);
  for (int q = tid; q <= ke - kb + 21; q += L::NT) sZ[q] = bits(kb - 13 + q, nz, kb, ke);

  auto load_plane = [&](int k) {
    const int kw = pot_wrap(k, nz);
    const T* p = phi + (int64_t)(where(k, nz) + 1) * pg.s.pz;
    const T* d = D + (int64_t)(kw + 1) * pg.s.pz;
#pragma unroll
    for (int r = 0; r < RW; r++) {
      pf[r] = lds2(cell(p, roff[r]));
      pd[r] = lds2(cell(d, doff[r]));
    }
    if (jump1 || jumpn) {
#pragma unroll
      for (int r = 0; r < RW; r++) jx[r] = s[pg.s.j[0] + (int64_t)(kw - 1) * ny + jrow[r]];
    }
  };

  const int ks = kb - 6, kend = ke + 6;
  constexpr int DS = L::ROWS * 32;  // one colour of one plane of D
  T* const dbase = sD + (w * RW) * 32 + lane;
  int slot[6];  // offsets of the planes t - 1 .. t - 6 of D (the last one's is plane t's next)
#pragma unroll
  for (int q = 0; q < 6; q++) slot[q] = q * 2 * DS;

  auto step = [&](int t, auto u_tag, auto full_tag) {
    constexpr int U = decltype(u_tag)::value;
    constexpr bool FULL = decltype(full_tag)::value;
    constexpr int I0 = UF - 1 - U;  // register of plane t; plane t - h is I0 + h
    const T* xin = sX + ((U & 1) ^ 1) * (6 * NW * 64) + lane;
    T* xout = sX + (U & 1) * (6 * NW * 64) + w * 64 + lane;
    const int s6 = slot[5];
    T d6[RW];  // D of the sixth half sweep: plane t takes its slot
#pragma unroll
    for (int r = 0; r < RW; r++) {
      d6[r] = dbase[s6 + DS + r * 32];
      const bool Lft = ((r + U) & 1) != 0;  // colour 0 of plane t is the left cell when row + plane is odd
      T dl = pd[r].x, dr = pd[r].y;
      if constexpr (!FULL) {
        if (jump1) dl -= cx * jx[r];
        if (jumpn) dr += cx * jx[r];
      }
      A[r][I0] = Lft ? pf[r].x : pf[r].y;
      B[r][I0] = Lft ? pf[r].y : pf[r].x;
      dbase[s6 + r * 32] = Lft ? dl : dr;
      dbase[s6 + DS + r * 32] = Lft ? dr : dl;
    }
    load_plane(min(t + 1, kend));
    auto half = [&](auto h_tag) {
      constexpr int H = decltype(h_tag)::value;
      constexpr int I = I0 + H, SW = (H - 1) / 2, BIT = H <= 2 ? H - 1 : SW + 1;
      int zb = 0;
      if constexpr (!FULL) zb = sZ[t - H - (kb - 13)];
#pragma unroll
      for (int r = 0; r < RW; r++) {
        T(*X)[NP] = (H & 1) ? A : B;
        T(*Y)[NP] = (H & 1) ? B : A;
        const bool Lft = ((r + U) & 1) == 0;  // the updated cell is the pair's left one
        const T y = Y[r][I];
        const T xn = Lft ? shfl_up1(y) : shfl_down1(y);
        const T yd = r > 0 ? Y[r > 0 ? r - 1 : 0][I] : xin[((H - 1) * NW + wlo) * 64 + 32];
        const T yu = r < RW - 1 ? Y[r < RW - 1 ? r + 1 : 0][I] : xin[((H - 1) * NW + whi) * 64];
        const T dv = H == 6 ? d6[r] : dbase[slot[H - 1] + ((H & 1) ? 0 : DS) + r * 32];
        const T x = X[r][I];
        const T div = pot_div<T>(x, y + xn, yd + yu, Y[r][I - 1] + Y[r][I + 1], dv, cx, cy, cz);
        const T xnew = pfma<T>(wd, div, x);
        double dv2;
        if constexpr (FULL) {
          X[r][I] = xnew;
          dv2 = (double)pot_keep(div, keep[r]);
        } else {
          const int mm = (Lft ? mL[r] : mR[r]) & zb;
          X[r][I] = (mm & (1 << BIT)) ? xnew : x;
          dv2 = (double)((mm & (16 << BIT)) ? div : T(0));
        }
        racc[SW] = __fma_rn(dv2, dv2, racc[SW]);
      }
    };
    half(std::integral_constant<int, 1>{});
    half(std::integral_constant<int, 2>{});
    half(std::integral_constant<int, 3>{});
    half(std::integral_constant<int, 4>{});
    half(std::integral_constant<int, 5>{});
    half(std::integral_constant<int, 6>{});
    // rows at the warp's edges for the next plane's half sweeps
#pragma unroll
    for (int h = 0; h < 6; h++) {
      T(*Y)[NP] = (h & 1) ? A : B;
      xout[h * NW * 64] = Y[0][I0 + h];
      xout[h * NW * 64 + 32] = Y[RW - 1][I0 + h];
    }
    // plane t - 6
    const int q = t - 6;
    if (FULL || (q >= kb && q <= ke)) {
      T* o = out + (int64_t)(q + 1) * pg.s.pz;
#pragma unroll
      for (int r = 0; r < RW; r++) {
        const bool Lft = ((r + U) & 1) != 0;  // of plane t - 6, like plane t
        const T vl = Lft ? A[r][I0 + 6] : B[r][I0 + 6], vr = Lft ? B[r][I0 + 6] : A[r][I0 + 6];
        if (FULL ? (mL[r] & 256) != 0 : (mL[r] & 256) && xL <= nx && j0 + r <= ny && q <= nz)
          st2<T>(const_cast<T*>(cell(o, roff[r])), vl, vr);
      }
      if (!FULL && (edge_x || edge_y || q <= 4 || q >= nz - 2)) {
        // the layers next to the faces, and the cells n+1 (E)
#pragma unroll
        for (int r = 0; r < RW; r++) {
          if (!(mL[r] & 256)) continue;
          const bool Lft = ((r + U) & 1) != 0;
          const T vl = Lft ? A[r][I0 + 6] : B[r][I0 + 6], vr = Lft ? B[r][I0 + 6] : A[r][I0 + 6];
          const int j = j0 + r;
          const bool ix = xL <= nx, iy = j <= ny, iz = q <= nz;
          T* X = s + (int64_t)(q - 1) * ny + (j - 1);          // x faces: [..][nz][ny]
          T* Y = s + (int64_t)(q - 1) * nx + (xL - 1);         // y faces: [..][nz][nx]
          T* Z = s + (int64_t)(j - 1) * nx + (xL - 1);         // z faces: [..][ny][nx]
          if (ix && iy && iz) {
            const int ly = pot_layer(j, ny), lz = pot_layer(q, nz), l0 = pot_layer(xL, nx), l1 = pot_layer(xL + 1, nx);
            if (l0 >= 0) X[pg.s.l[0] + (int64_t)l0 * ny * nz] = vl;
            if (l1 >= 0) X[pg.s.l[0] + (int64_t)l1 * ny * nz] = vr;
            if (ly >= 0) Y[pg.s.l[1] + (int64_t)ly * nx * nz] = vl, Y[pg.s.l[1] + (int64_t)ly * nx * nz + 1] = vr;
            if (lz >= 0) Z[pg.s.l[2] + (int64_t)lz * nx * ny] = vl, Z[pg.s.l[2] + (int64_t)lz * nx * ny + 1] = vr;
          } else if (iy && iz) {
            if (xL == nx + 1) X[pg.s.e[0]] = vl;
          } else if (ix && iz) {
            Y[pg.s.e[1]] = vl, Y[pg.s.e[1] + 1] = vr;
          } else if (ix && iy) {
            Z[pg.s.e[2]] = vl, Z[pg.s.e[2] + 1] = vr;
          }
        }
      }
    }
#pragma unroll
    for (int h = 5; h > 0; h--) slot[h] = slot[h - 1];
    slot[0] = s6;
    __syncthreads();
  };

  using T_ = std::true_type;
  using F_ = std::false_type;
  load_plane(ks);
  __syncthreads();
  for (int t = ks; t <= kend; t += UF) {  // (planes past kend: of no use, and never stored)
    if (t >= zf_lo && t + UF - 1 <= zf_hi) {
      step(t, std::integral_constant<int, 0>{}, T_{});
      step(t + 1, std::integral_constant<int, 1>{}, T_{});
    } else {
      step(t, std::integral_constant<int, 0>{}, F_{});
      step(t + 1, std::integral_constant<int, 1>{}, F_{});
    }
#pragma unroll
    for (int r = 0; r < RW; r++)
#pragma unroll
      for (int q = 6; q >= 0; q--) {
        A[r][UF + q] = A[r][q];
        B[r][UF + q] = B[r][q];
      }
  }

  // residuals of the pass's sweeps; the last CTA runs the exit tests
  const unsigned int nb = gridDim.x;
  double* part = ga.partials[m];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const double bs = block_sum<L::NT>(racc[q], red);
    if (tid == 0) part[3 * blockIdx.x + q] = bs;
  }
  if (!last_block(&ctx->ticket, nb, &last_flag)) return;
  const double round = sizeof(T) == 4 ? ctx->pot_round : 0.0;
  const int itr = ctx->cs.itr, since = ctx->pot_since;
  double sum[3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    double v = 0.0;
    for (int b = tid; b < (int)nb; b += L::NT) v += __ldcg(&part[3 * b + q]);
    if (q == 0)
      for (int b = tid; b < pg.nslab; b += L::NT) v += __ldcg(&part[pg.slab_part + b]);
    sum[q] = block_sum<L::NT>(v, red);
  }
  if (tid != 0) return;
  ctx->ticket = 0;
  if (redo) {
    ctx->cs.done = 1;
    ctx->cs.cont = 0;
    ctx->pot_redo = 0;
    ctx->pot_pending = 1;
    ctx->pot_cur = 1 - cur;
  } else {
    bool wait = false;
    if constexpr (sizeof(T) == 4) {
      const double least = fmin(sum[0], fmin(sum[1], sum[2]));
      wait = least <= pg.exit_sum && itr + 2 >= cf.itrmin && isfinite(sum[0] + sum[1] + sum[2]) &&
             (least + 0.5 * round <= pg.exit_sum || itr >= since + kPotRoundAge);
      if (wait || itr + 3 >= cf.itrmax)  // (k_pot_jump or k_pot_round adds the rounding to them)
        for (int q = 0; q < 3; q++) ctx->pot_sum[q] = sum[q];
    }
    if (wait) ctx->pot_check = 1;
    else pot_exit(ctx, cf, sum, round);
  }
  if (loop.on) cudaGraphSetConditional(loop.handle, couple_goes_on(ctx, loop.max_groups) ? 1u : 0u);
}

// End of a couple: the velocity and P from Phi, and their halos, which the
// element-wise sweeps leave near the images too.  Bound by HBM: 5 fields read,
// 4 written (512^3: FP64 2.1 ms, FP32 1.3).
template <typename T>
__global__ void __launch_bounds__(256) k_pot_apply(const __grid_constant__ PotGroup<T> ga, Grid g, int set, PotGeom pg) {
  const int m = blockIdx.y;
  Ctx* ctx = ga.ctx[m];
  T* U = (T*)ctx->vel[set][0];
  T* V = (T*)ctx->vel[set][1];
  T* W = (T*)ctx->vel[set][2];
  T* P = ga.P[m];
  const T* phi = pot_buf<T>(ctx, ctx->pot_cur);
  const T* s = ga.scratch[m];
  const bool pend = ctx->pot_pending != 0;
  const T dxi = (T)pg.dxi, dyi = (T)pg.dyi, dzi = (T)pg.dzi, dti = (T)(1.0 / ctx->scal[0]);
  const int nx = g.n[0], ny = g.n[1], nz = g.n[2], hx = nx / 2, px = pg.s.px, pz = pg.s.pz;
  const int total = hx * ny * nz;
  for (int t = blockIdx.x * 256 + threadIdx.x; t < total; t += gridDim.x * 256) {
    const int i = 1 + 2 * (t % hx);
    const int u = t / hx;
    const int j = 1 + u % ny, k = 1 + u / ny;
    const int o = pg.s.at(i, j, k);
    const pair_t<T> p = lds2(phi + o);
    // Phi of the cells past the last one: n+1 as the groups swept it
    auto past = [&](T first, int axis, int f) { return first - (s[pg.s.j[axis] + f] + (pend ? first - s[pg.s.e[axis] + f] : T(0))); };
    T east;
    if (i + 1 < nx) east = phi[o + 2];
    else east = past(phi[o - (nx - 2)], 0, (k - 1) * ny + (j - 1));
    pair_t<T> north, top;
    if (j < ny) {
      north = lds2(phi + o + px);
    } else {
      const pair_t<T> q = lds2(phi + o - (ny - 1) * px);
      const int f = (k - 1) * nx + (i - 1);
      north = mk2<T>(past(q.x, 1, f), past(q.y, 1, f + 1));
    }
    if (k < nz) {
      top = lds2(phi + o + pz);
    } else {
      const pair_t<T> q = lds2(phi + o - (nz - 1) * pz);
      const int f = (j - 1) * nx + (i - 1);
      top = mk2<T>(past(q.x, 2, f), past(q.y, 2, f + 1));
    }
    const int64_t c = g.at(i, j, k);
    const pair_t<T> u2 = lds2(U + c), v2 = lds2(V + c), w2 = lds2(W + c), q2 = lds2(P + c);
    T* const f[4] = {U, V, W, P};
    const T a[4] = {pfma<T>(dxi, p.x - p.y, u2.x), pfma<T>(dyi, p.x - north.x, v2.x), pfma<T>(dzi, p.x - top.x, w2.x),
                    pfma<T>(dti, p.x, q2.x)};
    const T b[4] = {pfma<T>(dxi, p.y - east, u2.y), pfma<T>(dyi, p.y - north.y, v2.y), pfma<T>(dzi, p.y - top.y, w2.y),
                    pfma<T>(dti, p.y, q2.y)};
#pragma unroll
    for (int q = 0; q < 4; q++) st2<T>(f[q] + c, a[q], b[q]);
    // the pair's images in the halo
    auto span = [&](int w, int n, int* lo, int* hi) {  // shifts by -n, 0, n that stay within 1 - h .. n + h
      *lo = w > n - g.h ? -1 : 0;
      *hi = w <= g.h ? 1 : 0;
    };
    int xl, xh, yl, yh, zl, zh, xl2, xh2;
    span(i, nx, &xl, &xh);
    span(i + 1, nx, &xl2, &xh2);
    span(j, ny, &yl, &yh);
    span(k, nz, &zl, &zh);
    if (xl2 | xh | yl | yh | zl | zh)
      for (int dz = zl; dz <= zh; dz++)
        for (int dy = yl; dy <= yh; dy++)
          for (int dx = -1; dx <= 1; dx++) {
            if (!(dx | dy | dz)) continue;
            const int64_t h = g.at(i + dx * nx, j + dy * ny, k + dz * nz);
#pragma unroll
            for (int q = 0; q < 4; q++) {
              if (dx >= xl && dx <= xh) f[q][h] = a[q];
              if (dx >= xl2 && dx <= xh2) f[q][h + 1] = b[q];
            }
          }
  }
}

template <typename T>
PotKernels<T> make_pot_kernels() {
  using L = PotTiles<T>;
  PotKernels<T> k;
  k.setup = k_pot_setup<T>;
  k.jump = k_pot_jump<T>;
  k.slab = k_pot_slab<T>;
  k.sweep[0] = k_pot_sweep<T, L::Tall::NW, L::Tall::RW>;
  k.sweep[1] = k_pot_sweep<T, L::Mid::NW, L::Mid::RW>;
  k.sweep[2] = k_pot_sweep<T, L::Flat::NW, L::Flat::RW>;
  k.round = nullptr;
  if constexpr (sizeof(T) == 4) k.round = k_pot_round<T>;
  k.apply = k_pot_apply<T>;
  return k;
}

}  // namespace
}  // namespace lcs
