// step_f64.cu -- one upwind time step in FP64 (the reference's advect() body,
// upwind/cxx/upwind.cxx:64-84), ping-pong between two device fields instead
// of the reference's copy pass (:59-62).
//
// Two arithmetics share one memory pattern:
//   EXACT  f' = ((f - c_z (f_zu - f)) - c_y (f_yu - f)) - c_x (f_xu - f), every
//          operation separately rounded, in the reference's axis order
//          j = 0..ndims-1: bit-identical to the reference compiled without
//          FMA.  9 FP64 operations per cell.
//   FMA    f' = w f + a_z f_zu + a_y f_yu + a_x f_xu (a_j = -c_j,
//          w = ((1 - a_z) - a_y) - a_x): 4 per cell.
// On GB300 both are bound by the FP64 pipe, not by HBM (the block-fixed-point
// kernel in step_fixed.cu is the bandwidth-class path), so what counts is the
// cost of an FP64 operation (f64_regs.cuh) and an even share of the cells for
// every SM.  Per step, against rows dealt to CTAs and DADD / DMUL / DFMA with
// constants: EXACT 192^3 133 -> 106 us (67 of the pipe's 67 cycles per
// operation and warp), FMA 2048^2 38 -> 30.3 us, FMA 128^3 20.5 -> 16.5 us, FMA 512^3
// 1490 -> 897 us (150 GCUPS).  Small grids are bound by the launches: see plan_f64.
//
// Layout: row-major, x (last reference axis) contiguous; consecutive threads
// take consecutive cells, and the upstream neighbours come through L1 and L2.
#include <algorithm>
#include <cmath>

#include "f64_regs.cuh"
#include "fdb_internal.h"

namespace fdb {
namespace {

constexpr int kThreads = 256;

// One cell from its value and its upstream values, by FP64 operations with
// three register operands (f64_regs.cuh).
template <int ARITH>
__device__ __forceinline__ double cell(double o, double uz, double uy, double ux,
                                       const Coeffs3& c, const F64Regs& k) {
  if (ARITH == FDB_ARITH_EXACT) {
    double t = o;
    t = k.sub(t, k.mul(c.cz, k.sub(uz, o)));
    t = k.sub(t, k.mul(c.cy, k.sub(uy, o)));
    t = k.sub(t, k.mul(c.cx, k.sub(ux, o)));
    return t;
  }
  return fma(c.ax, ux, fma(c.ay, uy, fma(c.az, uz, k.mul(c.w, o))));
}

// The coefficients that `cell` uses, in registers.
template <int ARITH>
__device__ __forceinline__ Coeffs3 reg_coeffs(const Coeffs3& c, const RegLoader& reg) {
  Coeffs3 r = c;
  if (ARITH == FDB_ARITH_EXACT) {
    r.cz = reg(c.cz);
    r.cy = reg(c.cy);
    r.cx = reg(c.cx);
  } else {
    r.az = reg(c.az);
    r.ay = reg(c.ay);
    r.ax = reg(c.ax);
    r.w = reg(c.w);
  }
  return r;
}

// One axis of k_step3's walk over the cells: the upstream neighbour is at
// offset d, or at offset w for the cells at index `edge`.  I: uint32_t, or
// uint64_t for extents above 2^31.
template <typename I>
struct Walk {
  int64_t d, w;
  I n, edge, step;  // extent; edge index; the axis' digit of the grid stride
};

// One step.  Thread t of T takes the cells t, t + T, ...: the FP64 pipe is the
// bound, and every SM gets the same number of cells however the rows fall.  The
// cell's (z, y, x) advance by the digits of T, so that no division is left in
// the loop.
template <int ARITH, typename I>
__global__ void __launch_bounds__(kThreads)
k_step3(const double* in, double* __restrict__ out, int64_t ntot, Walk<I> az,
        Walk<I> ay, Walk<I> ax, const Coeffs3 coeffs) {
  __shared__ double s_slots[kThreads];
  const RegLoader reg(s_slots);
  const F64Regs k(reg);
  const Coeffs3 c = reg_coeffs<ARITH>(coeffs, reg);
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= ntot) return;
  const uint64_t row = (uint64_t)i / ax.n;
  I x = (I)((uint64_t)i % ax.n), y = (I)(row % ay.n), z = (I)(row / ay.n);
  cudaGridDependencySynchronize();  // the launch before has written `in` and read `out`
  for (; i < ntot; i += stride) {
    const double o = in[i];
    const double uz = in[i + (z == az.edge ? az.w : az.d)];
    const double uy = in[i + (y == ay.edge ? ay.w : ay.d)];
    const double ux = in[i + (x == ax.edge ? ax.w : ax.d)];
    out[i] = cell<ARITH>(o, uz, uy, ux, c, k);
    x += ax.step;
    I carry = x >= ax.n;
    if (carry) x -= ax.n;
    y += ay.step + carry;
    carry = y >= ay.n;
    if (carry) y -= ay.n;
    z += az.step + carry;
  }
}

// K steps of a small grid in one launch.  A CTA computes a tile of t[] output
// cells from a region with K more cells upstream on every axis it does not
// span (h = 1; an axis it spans wraps inside the region, h = 0).  The region
// passes through two shared-memory buffers, one barrier per step; the halo is
// computed redundantly, one cell less of it per step.  The cell's arithmetic
// is k_step3's, so the result has the same bits.  A step's latency (index
// arithmetic, shared-memory loads, a chain of FP64 operations, a barrier) is
// what counts at these sizes: as many threads as a step has cells, up to 1024.
struct TileArgs {
  int n[3], t[3], h[3], flip[3];  // z, y, x; flip: the axis reversed (upstream at +1)
  int tiles[3];
  int K;
};

constexpr int kTileThreads = 1024;

// i / d for i d < 2^32 (d >= 1): the product with the reciprocal rounded up
struct SmallDiv {
  uint32_t m;
  int d;
  __device__ __forceinline__ explicit SmallDiv(int d_)
      : m(d_ > 1 ? 0xFFFFFFFFu / (uint32_t)d_ + 1u : 0u), d(d_) {}
  __device__ __forceinline__ int div(int i) const {
    return d > 1 ? (int)__umulhi((uint32_t)i, m) : i;
  }
};

template <int ARITH>
__global__ void __launch_bounds__(kTileThreads)
k_steps_tile(const double* in, double* __restrict__ out, const TileArgs a,
             const Coeffs3 coeffs) {
  extern __shared__ double s_buf[];
  __shared__ double s_slots[kTileThreads];
  const RegLoader reg(s_slots);
  const F64Regs regs(reg);
  const Coeffs3 c = reg_coeffs<ARITH>(coeffs, reg);
  int b = blockIdx.x;
  const int x0 = b % a.tiles[2] * a.t[2];
  b /= a.tiles[2];
  const int y0 = b % a.tiles[1] * a.t[1];
  const int z0 = b / a.tiles[1] * a.t[0];
  // region extents and first cell (logical)
  const int ez = min(a.t[0], a.n[0] - z0) + a.h[0] * a.K, bz = z0 - a.h[0] * a.K;
  const int ey = min(a.t[1], a.n[1] - y0) + a.h[1] * a.K, by = y0 - a.h[1] * a.K;
  const int ex = min(a.t[2], a.n[2] - x0) + a.h[2] * a.K, bx = x0 - a.h[2] * a.K;
  const int plane = ey * ex, cells = ez * plane;
  // region cell -> offset in the field
  auto axis = [&](int k, int p) {
    while (p < 0) p += a.n[k];
    return a.flip[k] ? a.n[k] - 1 - p : p;
  };
  auto field = [&](int z, int y, int x) -> int64_t {
    return ((int64_t)axis(0, bz + z) * a.n[1] + axis(1, by + y)) * a.n[2] + axis(2, bx + x);
  };
  const SmallDiv dx(ex), dy(ey);
  cudaGridDependencySynchronize();  // the launch before has written `in` and read `out`
  for (int i = threadIdx.x; i < cells; i += blockDim.x) {
    const int r = dx.div(i), z = dy.div(r);
    s_buf[i] = in[field(z, r - z * ey, i - r * ex)];
  }
  __syncthreads();
  for (int t = 1; t <= a.K; ++t) {
    const double* src = s_buf + ((t - 1) & 1) * cells;
    double* dst = s_buf + (t & 1) * cells;
    // cells valid after t steps: t more from the upstream end of a halo
    const int oz = a.h[0] * t, oy = a.h[1] * t, ox = a.h[2] * t;
    const int wy = ey - oy, wx = ex - ox;
    const int count = (ez - oz) * wy * wx;
    const SmallDiv ddx(wx), ddy(wy);
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      const int r = ddx.div(i), rz = ddy.div(r);
      const int x = i - r * wx + ox, y = r - rz * wy + oy, z = rz + oz;
      const int j = (z * ey + y) * ex + x;
      const double o = src[j];
      const double uz = src[z > 0 ? j - plane : j + (ez - 1) * plane];
      const double uy = src[y > 0 ? j - ex : j + (ey - 1) * ex];
      const double ux = src[x > 0 ? j - 1 : j + ex - 1];
      const double v = cell<ARITH>(o, uz, uy, ux, c, regs);
      if (t == a.K)
        out[field(z, y, x)] = v;
      else
        dst[j] = v;
    }
    __syncthreads();
  }
}

struct GenericArgs {
  int ndims;
  uint64_t n[FDB_MAX_DIMS];
  uint64_t dimProd[FDB_MAX_DIMS];
  int up[FDB_MAX_DIMS];
  double coeff[FDB_MAX_DIMS];
};

// Any number of axes (up to FDB_MAX_DIMS), the reference's own per-cell index
// reconstruction (getIndexSet/getFlatIndex, upwind.cxx:122-134) and EXACT
// arithmetic.  Used for ndims > 3 only.
__global__ void k_step_generic(const double* __restrict__ in, double* __restrict__ out,
                               uint64_t ntot, GenericArgs a) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < ntot;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const double o = in[i];
    double t = o;
    for (int j = 0; j < a.ndims; ++j) {
      const uint64_t ij = (i / a.dimProd[j]) % a.n[j];
      uint64_t iu = ij;
      if (a.up[j] < 0) iu = (ij == 0) ? a.n[j] - 1 : ij - 1;
      else iu = (ij + 1 == a.n[j]) ? 0 : ij + 1;
      const uint64_t upI = i - ij * a.dimProd[j] + iu * a.dimProd[j];
      t = __dsub_rn(t, __dmul_rn(a.coeff[j], __dsub_rn(in[upI], o)));
    }
    out[i] = t;
  }
}

template <typename I>
Walk<I> make_walk(int64_t n, int64_t stride, int up, int64_t digit) {
  Walk<I> w;
  w.n = (I)n;
  w.step = (I)digit;
  w.edge = up < 0 ? (I)0 : (I)(n - 1);
  w.d = up < 0 ? -stride : stride;
  w.w = up < 0 ? (n - 1) * stride : -(n - 1) * stride;
  return w;
}

constexpr int kSms = 152;
// Time of a chained launch of k_steps_tile beyond its FP64 work, and of each of
// its steps; of k_step3; and of a cell update at one SM (4 FP64 operations),
// in the tiles and streamed, in us.  Fitted to 100 .. 280,000 cells.
constexpr double kTileUs = 1.55, kTileStepUs = 0.41, kStreamUs = 1.75;
constexpr double kTileCellUs = 2.1e-3, kStreamCellUs = 1.1e-3;
constexpr size_t kTileSmem = 96 * 1024;

// Steps per launch and the tile of the FP64 path by those times: the fewest us
// per step (K = 1: k_step3).  Only grids whose FP64 work is short against a
// launch gain from K > 1: the halo is FP64 work, so a tile has to win by a
// tenth.  Measured, us per step of a chain (one step per launch before
// dependent launches 4.1): 16^3 1.73 with k_step3, 1.13 in tiles; 2000 cells in
// one dimension 1.89, 0.66; 32^3 1.89, 1.85; 48^3 2.31, 3.20.
struct F64Plan {
  int K = 1;
  TileArgs a{};
};

F64Plan plan_f64(const Geom& g, int arith, int steps) {
  F64Plan best;
  const double ops = arith == FDB_ARITH_EXACT ? 9.0 / 4.0 : 1.0;
  double best_cost = kStreamUs + (double)g.ntot / kSms * kStreamCellUs * ops;
  if (steps < 2 || best_cost > 2.0 * kStreamUs) return best;
  best_cost *= 0.9;
  const int n[3] = {(int)g.nz, (int)g.ny, (int)g.nx};
  const int cz[] = {1, 2, 4, 8}, cy[] = {2, 4, 8, 16}, cx[] = {8, 16, 32, 64};
  for (int K : {2, 3, 4, 6, 8}) {
    if (K > steps) break;
    for (int tz : cz)
      for (int ty : cy)
        for (int tx : cx) {
          const int t[3] = {std::min(tz, n[0]), std::min(ty, n[1]), std::min(tx, n[2])};
          int h[3];
          double tiles = 1.0, region = 1.0, work = 0.0;
          for (int k = 0; k < 3; ++k) {
            h[k] = t[k] < n[k];
            tiles *= (n[k] + t[k] - 1) / t[k];
            region *= t[k] + h[k] * K;
          }
          if (region * 16 > kTileSmem) continue;
          for (int s = 0; s < K; ++s)  // s = steps still to go
            work += (double)(t[0] + h[0] * s) * (t[1] + h[1] * s) * (t[2] + h[2] * s);
          const double us = kTileUs + K * kTileStepUs +
                            std::ceil(tiles / kSms) * work * kTileCellUs * ops;
          const double cost = us / K;
          if (cost < best_cost) {
            best_cost = cost;
            best.K = K;
            for (int k = 0; k < 3; ++k) {
              best.a.n[k] = n[k];
              best.a.t[k] = t[k];
              best.a.h[k] = h[k];
              best.a.tiles[k] = (n[k] + t[k] - 1) / t[k];
            }
          }
        }
  }
  best.a.flip[0] = g.upz > 0;
  best.a.flip[1] = g.upy > 0;
  best.a.flip[2] = g.upx > 0;
  return best;
}

template <int ARITH>
int launch_steps_tile(const TileArgs& a, const Coeffs3& c, const double* in, double* out,
                      cudaStream_t s) {
  size_t cells = 1;
  for (int k = 0; k < 3; ++k) cells *= a.t[k] + a.h[k] * a.K;
  if (cells * 16 > 40 * 1024)  // with the static slots, above what needs no opt-in
    FDB_CUDA_TRY(cudaFuncSetAttribute(
        k_steps_tile<ARITH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem));
  size_t first = 1;  // cells of the first step
  for (int k = 0; k < 3; ++k) first *= a.t[k] + a.h[k] * (a.K - 1);
  FDB_CUDA_TRY(launch_dependent(
      k_steps_tile<ARITH>, a.tiles[0] * a.tiles[1] * a.tiles[2],
      (unsigned)std::min<size_t>(kTileThreads, (first + 31) / 32 * 32), cells * 16, s, in, out, a,
      c));
  note_launch();
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

template <typename I>
cudaError_t step3(const Geom& g, const Coeffs3& c, int arith, const double* in, double* out,
           cudaStream_t s) {
  // The same number of cells for every CTA.  6 are resident per SM (38 to 40
  // registers): of 8, the last two run nearly alone, and in a dependent launch they
  // fall unevenly on the SMs.  Whole waves, where a thread still has a few cells.  FMA, us per step with 8 / 12 / 18 per SM: 512^3
  // 1036 / 919 / 897, 4000 x 3000 94.6 / 84.1 / 83.5, 208^3 69.9 / 63.5 / 62.9, 192^3
  // 55.7 / 49.9 / 50.7, 2048^2 30.3 / 30.0 / 30.4, 144^3 22.1 / 22.2 / 22.3, 128^3 16.6
  // / 17.1 / 16.9 (normal launches of 8: 512^3 947, 2048^2 32.9).  EXACT 512^3 1978 /
  // 1963 / 1955.
  const int per_sm = g.ntot >= 8000000 ? 18 : g.ntot >= 3000000 ? 12 : 8;
  int64_t grid = ((int64_t)g.ntot + kThreads - 1) / kThreads;  // a cell per thread at least
  if (grid > kSms * per_sm) grid = kSms * per_sm;
  const int64_t stride = grid * kThreads;
  const int64_t dy = stride / g.nx;
  const Walk<I> ax = make_walk<I>(g.nx, 1, g.upx, stride % g.nx);
  const Walk<I> ay = make_walk<I>(g.ny, g.nx, g.upy, dy % g.ny);
  const Walk<I> az = make_walk<I>(g.nz, g.ny * g.nx, g.upz, dy / g.ny);
  return launch_dependent(arith == FDB_ARITH_EXACT ? k_step3<FDB_ARITH_EXACT, I>
                                                   : k_step3<FDB_ARITH_FMA, I>,
                          (unsigned)grid, kThreads, 0, s, in, out, g.ntot, az, ay, ax, c);
}

}  // namespace

int launch_step_f64(const Geom& g, const Coeffs3& c, int arith, const double* in, double* out,
                    cudaStream_t s) {
  if (fault_injected("launch")) return fail(FDB_ERR_INJECTED, "injected launch failure");
  if (std::max(g.nz, std::max(g.ny, g.nx)) <= ((int64_t)1 << 31))
    FDB_CUDA_TRY(step3<uint32_t>(g, c, arith, in, out, s));
  else
    FDB_CUDA_TRY(step3<uint64_t>(g, c, arith, in, out, s));
  note_launch();
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

int launch_advect_f64(const Geom& g, const Coeffs3& c, int arith, int steps, double** buf, int* cur,
                      cudaStream_t s) {
  const F64Plan p = plan_f64(g, arith, steps);
  for (int done = 0; done < steps;) {
    const int k = std::min(p.K, steps - done);
    if (k == 1) {
      FDB_TRY(launch_step_f64(g, c, arith, buf[*cur], buf[*cur ^ 1], s));
    } else {
      if (fault_injected("launch")) return fail(FDB_ERR_INJECTED, "injected launch failure");
      TileArgs a = p.a;
      a.K = k;
      FDB_TRY(arith == FDB_ARITH_EXACT
                  ? launch_steps_tile<FDB_ARITH_EXACT>(a, c, buf[*cur], buf[*cur ^ 1], s)
                  : launch_steps_tile<FDB_ARITH_FMA>(a, c, buf[*cur], buf[*cur ^ 1], s));
    }
    *cur ^= 1;
    done += k;
  }
  return FDB_OK;
}

int launch_step_generic(const Geom& g, double dt, const double* in, double* out,
                        cudaStream_t s) {
  if (fault_injected("launch")) return fail(FDB_ERR_INJECTED, "injected launch failure");
  GenericArgs a{};
  a.ndims = g.ndims;
  for (int j = 0; j < g.ndims; ++j) {
    a.n[j] = g.n[j];
    a.dimProd[j] = g.dimProd[j];
    a.up[j] = g.up[j];
    a.coeff[j] = ref_coeff(g, j, dt);
  }
  uint64_t blocks = (g.ntot + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  k_step_generic<<<(unsigned)blocks, 256, 0, s>>>(in, out, g.ntot, a);
  note_launch();
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

}  // namespace fdb
