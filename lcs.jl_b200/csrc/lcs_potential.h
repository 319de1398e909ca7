// lcs_potential.h -- what the engine and the kernels of the couple in potential
// form (lcs_potential.cuh) share: layouts, launch arguments, tiles, and the
// kernels' addresses.
//
// The kernels are compiled by themselves (lcs_pot_f64.cu, lcs_pot_f32.cu): in
// one translation unit with the element-wise sweep k_hsmac_rw they change its
// register allocation (122 and 124 registers in FP64, a spill in the group
// form), and it takes 17.7 us alone and 18.3 beside them at 32^3.
#pragma once

#include "lcs_common.cuh"

namespace lcs {

constexpr int kPotLayers = 7;  // layers next to a face kept compact: n-2, n-1, n, 1, 2, 3, 4
constexpr int kPotDLayers = 5; // of D along x: n-1, n, 1, 2, 3
constexpr int kPotSlab = 22;   // a slab tile's own columns (32 less 5 on each side)
constexpr int kPotSlabThreads = 1024;

// Layout of Phi and D (each in one of the spare velocity buffers): positions
// -1 .. n+3 along each axis, x fastest, rows on 32-byte boundaries; an odd x
// starts an aligned pair.  Offsets (elements of T) of the couple's small
// arrays in its scratch.
struct PotScratch {
  int nx, ny, nz, px;   // px: row pitch
  int pz;               // plane pitch (a field holds < 2^31 elements)
  int64_t l[3], dx, e[3], j[3], total;
  __host__ __device__ __forceinline__ int at(int i, int j, int k) const { return (k + 1) * pz + (j + 1) * px + (i + 1); }
};
__host__ __device__ inline PotScratch pot_scratch(const int n[3], int elem) {
  PotScratch p;
  p.nx = n[0];
  p.ny = n[1];
  p.nz = n[2];
  const int a = 32 / elem;
  p.px = (n[0] + 6 + a - 1) / a * a;
  p.pz = p.px * (n[1] + 5);
  const int64_t x = n[0], y = n[1], z = n[2];
  const int64_t face[3] = {y * z, x * z, x * y};
  int64_t o = 0;
  for (int a3 = 0; a3 < 3; a3++) {  // Phi next to the faces: [7][nz][ny], [7][nz][nx], [7][ny][nx]
    p.l[a3] = o;
    o += kPotLayers * face[a3];
  }
  p.dx = o;  // [5][nz][ny]
  o += kPotDLayers * face[0];
  for (int a3 = 0; a3 < 3; a3++) {  // Phi of the cells n+1 after a group: [nz][ny], [nz][nx], [ny][nx]
    p.e[a3] = o;
    o += face[a3];
  }
  for (int a3 = 0; a3 < 3; a3++) {  // the jumps, same shapes
    p.j[a3] = o;
    o += face[a3];
  }
  p.total = o;
  return p;
}

// Handles that run the same launches side by side (one for a run alone).
constexpr int kPotMax = 64;
template <typename T>
struct PotGroup {
  Ctx* ctx[kPotMax];
  T* P[kPotMax];
  T* scratch[kPotMax];
  double* partials[kPotMax];
};

struct PotGeom {
  PotScratch s;
  int overlap;
  int kind, gx, gy;        // tile of k_pot_sweep (host's choice), tile columns along x and y
  int nseg, nc;            // CTAs; z chunks of a column
  int slab_part, nslab;    // residual partials of the slab tiles: first, count
  int slab0[3];            // first tile of an axis's slabs (z, y, x in turn)
  double cx, cy, cz, wd;   // 1/dx^2 .., -omega dl
  double dxi, dyi, dzi;
  double exit_sum;         // the exit test's bound on a sweep's sum of div^2 (a hair above it)
};

constexpr int kPotMaxChunk = 1024, kPotMaxPlanes = kPotMaxChunk + 24;

// Tile of k_pot_sweep: NW warps of RW rows (RW even); a lane owns an x-pair.
template <typename T, int NWARPS, int ROWS_A_WARP>
struct PotTile {
  static constexpr int NW = NWARPS, RW = ROWS_A_WARP;
  static constexpr int NT = 32 * NW, ROWS = NW * RW;
  static constexpr int TX = 52, TY = ROWS - 12;  // outputs: 6 cells less on every side
  static constexpr size_t d_elems = (size_t)6 * 2 * ROWS * 32;   // D of 6 planes, split by colour
  static constexpr size_t x_elems = (size_t)2 * 6 * NW * 2 * 32; // rows at the warps' edges, double buffered
  static constexpr size_t bytes = (d_elems + x_elems) * sizeof(T) + kPotMaxPlanes * sizeof(int);
  static_assert(RW % 2 == 0, "a warp's first row has the same parity in every warp");
};

// The loop of a couple inside a step graph: the last CTA of a group's sweep
// sets its condition (a run alone; a batch group has a kernel for it, which
// looks at all its members).
struct PotLoop {
  int on, max_groups;
  cudaGraphConditionalHandle handle;
};

// The tiles that the sweep is compiled for.
template <typename T>
struct PotTiles {
  static constexpr bool F64 = sizeof(T) == 8;
  using Tall = PotTile<T, F64 ? 8 : 12, 4>;               // FP64 20 output rows, FP32 36
  using Mid = PotTile<T, F64 ? 8 : 16, F64 ? 4 : 2>;      // FP32 20 output rows (FP64: the same as Tall)
  using Flat = PotTile<T, 8, 2>;                          // 4 output rows
};

constexpr size_t kPotSlabPlanes = 10;  // of 32 x 32 values in a slab block's shared memory

template <typename T>
struct PotKernels {
  void (*setup)(PotGroup<T>, Grid, int, PotGeom);
  void (*jump)(PotGroup<T>, Grid, int, PotGeom, HsmacCoef, PotLoop);
  void (*slab)(PotGroup<T>, PotGeom);
  void (*sweep[3])(PotGroup<T>, PotGeom, HsmacCoef, PotLoop);  // Tall, Mid, Flat
  void (*round)(PotGroup<T>, Grid, int, PotGeom, HsmacCoef);   // FP32 only
  void (*apply)(PotGroup<T>, Grid, int, PotGeom);
};
const PotKernels<double>& pot_kernels_f64();
const PotKernels<float>& pot_kernels_f32();
inline const PotKernels<double>& pot_kernels(double) { return pot_kernels_f64(); }
inline const PotKernels<float>& pot_kernels(float) { return pot_kernels_f32(); }

}  // namespace lcs
