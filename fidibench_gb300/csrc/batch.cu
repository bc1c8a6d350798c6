// batch.cu -- many independent upwind problems of uneven sizes and
// velocities advanced in one persistent launch (no reference counterpart;
// each instance is the reference's advect(), upwind/cxx/upwind.cxx:51-86).
//
// Work.  advect(steps) is cut into time blocks of K steps.  A work item is
// one packed tile of one instance in one time block: rectangles of output
// cells laid side by side in the lanes and stacked in the warps of a CTA
// (pack_instance), so that the remainder strips of uneven axes share CTAs
// instead of padding one each.  Items are numbered block-major, instance,
// tile.  One persistent grid (the resident CTAs of the device) takes items
// from an atomic counter in that order.
//
// Dependencies.  A tile of block b reads its upstream halo from the
// neighbouring tiles' block b-1 output, so before starting it waits until
// all block b-1 tiles of *its own instance* are done (a per-instance
// completion counter); other instances keep the GPU busy meanwhile, and no
// grid-wide barrier separates the blocks.  Items are taken in block order,
// so every item a CTA waits for was taken earlier by a running CTA that only
// waits for still earlier items: the waits cannot deadlock.  Every wait is
// bounded (clock64 budget): on expiry the CTA sets an error bit and leaves,
// the others follow, and the host reports FDB_ERR_TIMEOUT.
//
// Storage order.  An instance's three axes may be stored permuted: the order
// whose packed tiles march the fewest tile-planes (choose_order).  The update
// sums exact integer products, so the result does not depend on the order of
// the axes; set_field, get_field and init_sphere translate between the
// caller's order and the stored one.
// Instances that the single-field path advances in FP64 keep their order, so
// the looped comparator stays bit-identical to fdb_upwind_advect for all.
//
// Memory.  All instances' fields live in two arenas (ping-pong by block).
// Halo data written by other CTAs during the launch is read with L1-bypassing
// loads (ld.global.cg); a tile's stores are fenced before its completion is
// published.  Each instance has its own three-slot scale ring (see
// step_fixed.cu), advanced per block by the instance's tile 0.
//
// An advect is three launches (counter and scale-ring reset, per-instance max|f|
// pre-pass, persistent kernel), each dependent on the one before.  The device
// tables of the plan stay until the tuning, a time step or a velocity changes;
// the forward and the transposed problem have their own.  A caller may capture an
// advect whose tables are there: the batch then keeps those tables to its end and
// its fields in the same arena.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <fstream>
#include <sstream>
#include <string>
#include <type_traits>
#include <vector>

#include "batch_max.h"
#include "step_fixed.cuh"

using fdb::fx::FixedArgs;
using fdb::fx::ScaleSlot;

namespace fdb {
namespace bt {

struct InstDev {
  FixedArgs a;        // geometry, tiling, coefficients, guard (slot pointers unused)
  int64_t offset;     // first cell of the instance in the arenas
  int items;          // tiles per time block
  int item_base;      // first item of the instance within a block
};

// One packed tile: rectangles of gw lanes x gh warps of one instance, laid
// out (32 / gw) across the lanes and (W / gh) down the warps, row-major from
// groups[group_base]; each marches nout + K planes.
struct ItemDev {
  int inst;
  int gw, gh;
  int group_base;
  int nout;
};

constexpr long long kWaitCycles = 4000000000ll;  // ~2 s at 2 GHz

// depth of the persistent launch when none is set (the kernel is issue-bound,
// so the smaller halo of depth 2 outweighs its extra field traffic), and the
// depth the storage order is chosen for
constexpr int kDefaultDepth = 2;

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// 4-row shapes: at least 32 warps per SM (64 registers per thread, no
// spills); 6-row shapes: 20 warps, 8-row shapes: 16 warps (their rows need the
// registers).  kLeft: the x - 1 neighbour from the plane history (LEFT_SMEM of
// advance_tile), which the 4-warp shapes take and the 64-register ones do not
// (slower there).  kOff32: 32-bit byte offsets (planes below 4 GB), faster at
// K = 2 (256 uneven instances 447 -> 458 GCUPS) and slower at K = 3.
template <int K, int R, int W, bool kLeft, bool kOff32>
__global__ void __launch_bounds__(32 * W, (R > 6 ? 512 : R > 4 ? 640 : 1024) / (32 * W))
k_batch_fixed(const InstDev* __restrict__ insts, const ItemDev* __restrict__ items,
              const fx::TileGroup* __restrict__ groups, int items_per_block, int nblocks,
              int steps, int64_t* arena0, int64_t* arena1, ScaleSlot* slots, unsigned* done,
              unsigned* queue, int* err, unsigned wait_bias, long long wait_cycles) {
  extern __shared__ __align__(16) int64_t s_dyn[];  // plane history [K][R][threads]
  cudaGridDependencySynchronize();
  __shared__ int64_t s_row[2][W][32];
  __shared__ unsigned long long s_or[W];
  __shared__ int s_w;
  __shared__ int s_stop;
  __shared__ __align__(16) FixedArgs s_a;
  __shared__ __align__(16) fx::LevelCoeffs s_lev;

  const long long total = (long long)nblocks * items_per_block;
  for (;;) {
    if (threadIdx.x == 0) {
      s_w = (int)atomicAdd(queue, 1u);
      s_stop = (*(volatile int*)err != 0);
    }
    __syncthreads();
    const int w = s_w;
    if (w >= total || s_stop) break;
    const int b = w / items_per_block;
    const int item = w - b * items_per_block;
    const ItemDev it = items[item];
    const int i = it.inst;
    const InstDev& I = insts[i];
    const int local = item - I.item_base;
    // the item's FixedArgs into shared memory: under the register cap the
    // tile loop re-reads the coefficients at every level, and a shared-memory
    // read is cheaper than a global one (the previous item's readers passed
    // the barrier at the end of its iteration)
    {
      static_assert(sizeof(FixedArgs) % 4 == 0, "FixedArgs is copied as 32-bit words");
      const int* src = reinterpret_cast<const int*>(&I.a);
      int* dst = reinterpret_cast<int*>(&s_a);
      for (int k = threadIdx.x; k < (int)(sizeof(FixedArgs) / 4); k += blockDim.x) dst[k] = src[k];
      // the coefficients of this block's levels: steps b K + 1 .. (b + 1) K
      if (threadIdx.x < 3 * K) {
        const int t = threadIdx.x / 3, j = threadIdx.x - 3 * t;
        const QCoeff q = j == 0 ? I.a.qz : (j == 1 ? I.a.qy : I.a.qx);
        const int n = b * K + t + 1;
        s_lev.q[t][j] = step_qcoeff(q, n, n == steps);
      }
    }

    // wait until every block b-1 tile of this instance is done
    if (threadIdx.x == 0 && b > 0) {
      const unsigned need = (unsigned)b * (unsigned)I.items + wait_bias;
      const long long t0 = clock64();
      while (ld_acquire(done + i) < need) {
        if (clock64() - t0 > wait_cycles) {
          atomicOr(err, 2);
          s_stop = 1;
          break;
        }
        __nanosleep(200);
      }
    }
    __syncthreads();
    if (s_stop) break;

    ScaleSlot* sl = slots + 3 * i;
    int s, d;
    if (!scale_from_slot(sl + (b % 3), s_a.guard, &s, &d) && threadIdx.x == 0) atomicOr(err, 1);
    if (local == 0 && threadIdx.x == 0) {
      ScaleSlot* rs = sl + ((b + 2) % 3);
      rs->m = 0ull;
      rs->kind = 1;
      sl[(b + 1) % 3].s = s;
      sl[(b + 1) % 3].kind = 1;
    }
    auto scale = [s, d](int* s_to, int* d_to) {
      *s_to = s;
      *d_to = d;
    };
    // this thread's rectangle of the packed tile (lanes and warps past the
    // last full rectangle join the last one, beyond its outputs)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ncol = 32 / it.gw, nrow = W / it.gh;
    const int col = min(lane / it.gw, ncol - 1);
    const int rg = min(warp / it.gh, nrow - 1);
    const fx::TileGroup grp = groups[it.group_base + rg * ncol + col];
    const int64_t* in = ((b & 1) ? arena1 : arena0) + I.offset;
    int64_t* out = ((b & 1) ? arena0 : arena1) + I.offset;
    unsigned long long my_or = 0ull;
    // the last block holds the advect's last step, whose coefficients have all
    // 62 bits; the same code for every block would cost the others the three
    // products and the registers of a0
    auto tile = [&](auto full, int levels, bool out_f64) {
      fx::advance_tile<K, R, W, true, fx::kLoadL2Regs, decltype(full)::value, false, kLeft, true,
                       kOff32>(
          s_a, s_lev, 0, 0, 0, it.nout, levels, b == 0, out_f64, scale, in, out, s_dyn, s_row,
          my_or, grp, lane - col * it.gw, (warp - rg * it.gh) * R);
    };
    if (b == nblocks - 1)
      tile(std::integral_constant<int, fx::kAllFull>{}, steps - b * K, true);
    else
      tile(std::integral_constant<int, fx::kNoneFull>{}, K, false);
    fx::cta_or<W>(my_or, s_or, &sl[(b + 1) % 3].m);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(done + i, 1u);
  }
}

// max|f| of every instance (FP64 bit patterns) into slot 0 of its ring (kind 0,
// cleared by k_batch_reset), one chunk of cells per block (max_chunks) and four
// loads in flight per thread.  Bound by HBM: 256 instances (223 M cells) 257 us,
// 6.9 TB/s; 512^3 beside 2000 of 8^3 166 us, 6.5 TB/s.
__global__ void __launch_bounds__(256)
k_batch_absmax(const double* arena, const int64_t* __restrict__ offs,
               const uint64_t* __restrict__ sizes, const uint64_t* __restrict__ first, int count,
               uint64_t cells, ScaleSlot* slots) {
  __shared__ unsigned long long sh[8];
  const uint64_t chunks = first[count];
  cudaGridDependencySynchronize();
  for (uint64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    int i = 0, hi = count;  // the instance whose chunks contain this one
    while (hi - i > 1) {
      const int mid = (i + hi) >> 1;
      if (first[mid] <= c) i = mid;
      else hi = mid;
    }
    const double* f = arena + offs[i];
    const uint64_t begin = (c - first[i]) * cells;
    const uint64_t end = min(sizes[i], begin + cells);
    unsigned long long m = 0ull;
    auto take = [&](double x) {
      const unsigned long long bits =
          (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
      m = bits > m ? bits : m;
    };
    uint64_t k = begin + threadIdx.x;
    for (; k + 3 * 256 < end; k += 4 * 256) {
      const double x0 = f[k], x1 = f[k + 256], x2 = f[k + 512], x3 = f[k + 768];
      take(x0);
      take(x1);
      take(x2);
      take(x3);
    }
    for (; k < end; k += 256) take(f[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
      m = v > m ? v : m;
    }
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) m = sh[w] > m ? sh[w] : m;
      atomicMax(&slots[3 * (int64_t)i].m, m);
    }
    __syncthreads();
  }
}

// Work queue, completion counters and scale rings at the start of an advect.
__global__ void k_batch_reset(ScaleSlot* slots, unsigned* done, unsigned* queue, int count) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 3 * count; k += gridDim.x * blockDim.x) {
    slots[k].m = 0ull;
    slots[k].s = 0;
    slots[k].kind = (k % 3 == 0) ? 0 : 1;
    if (k < count) done[k] = 0u;
    if (k == 0) *queue = 0u;
  }
}

// per-instance sums: block b sums part (b % per_inst) of instance b / per_inst
__global__ void __launch_bounds__(256)
k_batch_sum_partial(const double* __restrict__ arena, const int64_t* __restrict__ offs,
                    const uint64_t* __restrict__ sizes, int count, int per_inst,
                    double* __restrict__ part) {
  __shared__ double sh[256];
  const int i = blockIdx.x / per_inst;
  const int pi = blockIdx.x - i * per_inst;
  const uint64_t n = sizes[i];
  const uint64_t chunk = (n + per_inst - 1) / per_inst;
  const uint64_t lo = (uint64_t)pi * chunk;
  const uint64_t hi = lo + chunk < n ? lo + chunk : n;
  double acc = 0.0;
  for (uint64_t k = lo + threadIdx.x; k < hi; k += 256) acc = acc + arena[offs[i] + k];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void k_batch_sum_final(const double* __restrict__ part, int count, int per_inst,
                                  double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  double acc = 0.0;
  for (int p = 0; p < per_inst; ++p) acc = acc + part[i * per_inst + p];
  out[i] = acc;
}

// One instance between the caller's axis order (the 3-D view (z, y, x) of
// its description, extents n) and the stored order (stored axis k = view
// axis p[k]): to_view = false writes dst in stored order from src in view
// order, true the other way.
__global__ void __launch_bounds__(256)
k_permute3(const double* __restrict__ src, double* __restrict__ dst, uint64_t n0, uint64_t n1,
           uint64_t n2, int p0, int p1, int p2, int to_view) {
  const uint64_t n[3] = {n0, n1, n2};
  const uint64_t e1 = n[p1], e2 = n[p2];
  const uint64_t total = n0 * n1 * n2;
  for (uint64_t i = blockIdx.x * 256ull + threadIdx.x; i < total; i += (uint64_t)gridDim.x * 256ull) {
    const uint64_t c2 = i % e2;
    const uint64_t t = i / e2;
    const uint64_t c1 = t % e1;
    const uint64_t c0 = t / e1;
    uint64_t r[3];
    r[p0] = c0;
    r[p1] = c1;
    r[p2] = c2;
    const uint64_t v = (r[0] * n1 + r[1]) * n2 + r[2];
    if (to_view)
      dst[v] = src[i];
    else
      dst[i] = src[v];
  }
}

// One instance's place in the caller's concatenated fields and in the arenas,
// and its share of the work items of k_batch_io.
struct IoDev {
  int64_t user, arena;  // first cell
  uint32_t n[3];        // extents of the 3-D view
  int p[3];             // stored axis k = view axis p[k]
  uint32_t item0;       // first work item
};

constexpr uint32_t kIoChunk = 4096;  // cells of a work item of an instance stored row by row

// Work items of an instance: chunks of cells when its rows stay rows (the x
// axis last in both orders), else 32 x 32 tiles of (stored row axis, x) for
// every index of the remaining axis.
uint64_t io_items(const uint32_t n[3], const int p[3]) {
  if (p[2] == 2) {
    const uint64_t cells = (uint64_t)n[0] * n[1] * n[2];
    return (cells + kIoChunk - 1) / kIoChunk;
  }
  const int a = p[2], o = 1 - a;
  return (uint64_t)n[o] * ((n[a] + 31) / 32) * ((n[2] + 31) / 32);
}

// All instances between the caller's concatenated fields (view order) and an
// arena (stored order) in one launch: to_view = false writes the arena `dst`
// from the caller's `src`, true the other way.  16 B per cell at 3.7 TB/s, bound by
// the index arithmetic and the one tile in flight per CTA; tiles pass through
// shared memory so that both sides are read and written in rows.  Against one copy
// or strided permutation and one synchronisation per instance: fields in,
// advect(50) and fields out of 256 instances (223 M cells) 43.1 -> 27.1 ms.
__global__ void __launch_bounds__(256)
k_batch_io(const double* __restrict__ src, double* __restrict__ dst,
           const IoDev* __restrict__ table, int count, uint32_t items, int to_view) {
  __shared__ double tile[32][33];
  for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
    int lo = 0, hi = count;  // the instance whose items contain this one
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (table[mid].item0 <= item) lo = mid;
      else hi = mid;
    }
    const IoDev& I = table[lo];
    uint32_t w = item - I.item0;
    const uint32_t n1 = I.n[1], n2 = I.n[2];
    if (I.p[2] == 2) {
      const uint64_t cells = (uint64_t)I.n[0] * n1 * n2;
      const bool same = I.p[0] == 0;
      const uint32_t e1 = same ? n1 : I.n[0];  // rows per stored plane
      const uint64_t end = min(cells, (uint64_t)(w + 1) * kIoChunk);
      for (uint64_t i = (uint64_t)w * kIoChunk + threadIdx.x; i < end; i += 256) {
        uint64_t v = i;  // the cell's place in the view
        if (!same) {
          const uint64_t row = i / n2;
          const uint64_t c0 = row / e1, c1 = row - c0 * e1;
          v = (c1 * n1 + c0) * n2 + (i - row * n2);
        }
        if (to_view) dst[I.user + v] = src[I.arena + i];
        else dst[I.arena + i] = src[I.user + v];
      }
      continue;
    }
    const int a = I.p[2], o = 1 - a;
    const uint32_t na = I.n[a];
    const uint32_t t2 = (n2 + 31) / 32, ta = (na + 31) / 32;
    const uint32_t x0 = w % t2 * 32;
    w /= t2;
    const uint32_t a0 = w % ta * 32, io = w / ta;
    // strides of the view axes a, o and x in the caller's and the stored layout
    const uint64_t ua = a == 0 ? (uint64_t)n1 * n2 : n2, uo = a == 0 ? n2 : (uint64_t)n1 * n2;
    const uint64_t sx = I.p[1] == 2 ? na : (uint64_t)I.n[o] * na;
    const uint64_t so = I.p[1] == 2 ? (uint64_t)n2 * na : na;
    const int64_t user = I.user + (int64_t)(io * uo), arena = I.arena + (int64_t)(io * so);
    const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (to_view) {
      for (uint32_t j = ty; j < 32; j += 8)
        if (x0 + j < n2 && a0 + tx < na) tile[j][tx] = src[arena + (x0 + j) * sx + a0 + tx];
      __syncthreads();
      for (uint32_t j = ty; j < 32; j += 8)
        if (a0 + j < na && x0 + tx < n2) dst[user + (a0 + j) * ua + x0 + tx] = tile[tx][j];
    } else {
      for (uint32_t j = ty; j < 32; j += 8)
        if (a0 + j < na && x0 + tx < n2) tile[tx][j] = src[user + (a0 + j) * ua + x0 + tx];
      __syncthreads();
      for (uint32_t j = ty; j < 32; j += 8)
        if (x0 + j < n2 && a0 + tx < na) dst[arena + (x0 + j) * sx + a0 + tx] = tile[j][tx];
    }
    __syncthreads();
  }
}

// Extents, velocities and lengths of the 3-D view (z, y, x) of a described
// instance (missing leading axes: extent 1, velocity 0).
void view3(const Geom& g, uint64_t n[3], double v[3], double L[3]) {
  const int jj[3] = {g.jz, g.jy, g.jx};
  for (int a = 0; a < 3; ++a) {
    const int j = jj[a];
    n[a] = j < 0 ? 1 : g.n[j];
    v[a] = j < 0 ? 0.0 : g.v[j];
    L[a] = j < 0 ? 1.0 : g.L[j];
  }
}

// Packed tiles of one instance of nx x ny x nz cells (stored axes).  The x axis is cut
// into segments of 32 - K outputs (a warp's width) and a remainder of rx
// outputs (rx + K lanes); the y axis into ranges of R W - K outputs (all W
// warps) and a remainder of ry outputs (ceil((ry + K) / R) warps).  The
// rectangles of one size (lanes x warps) are packed side by side and stacked,
// (32 / lanes) x (W / warps) to a tile.  To fill the tiles, the z axis of
// those rectangles may be cut into s ranges of zl planes, each marched from
// its own K warm-up planes; s minimises tiles x planes (with tz > 0, a range
// holds at most tz planes).  The last range ends at the last plane and may
// overlap the one before: the cells of the overlap are computed from the same
// inputs by the same integer arithmetic in both and stored twice with the
// same value, which no tile reads before the next time block.  Every other
// output cell lies in exactly one rectangle.
int pack_instance(int nx, int ny, int nz, int inst, int K, int R, int W, int tz,
                  std::vector<ItemDev>* items, std::vector<fx::TileGroup>* groups) {
  struct Seg {
    int o, n, units;  // first output, outputs, lanes (x) or warps (y)
  };
  // [0]: full segments, [1]: the remainder (at most one)
  std::vector<Seg> xs[2], ys[2];
  const int Tx = 32 - K, Ty = R * W - K;
  for (int j = 0; j < nx / Tx; ++j) xs[0].push_back({j * Tx, Tx, 32});
  if (nx % Tx) xs[1].push_back({nx / Tx * Tx, nx % Tx, nx % Tx + K});
  for (int j = 0; j < ny / Ty; ++j) ys[0].push_back({j * Ty, Ty, W});
  if (ny % Ty) ys[1].push_back({ny / Ty * Ty, ny % Ty, (ny % Ty + K + R - 1) / R});
  for (int xc = 0; xc < 2; ++xc) {
    for (int yc = 0; yc < 2; ++yc) {
      if (xs[xc].empty() || ys[yc].empty()) continue;
      const int gw = xs[xc][0].units, gh = ys[yc][0].units;
      const int ncol = 32 / gw, nrow = W / gh, P = ncol * nrow;
      const int64_t c = (int64_t)xs[xc].size() * (int64_t)ys[yc].size();
      // z ranges: the count sp of ranges that minimises tiles x planes
      const int s_min = tz > 0 ? (nz + tz - 1) / tz : 1;
      const int s_max = std::min(nz, std::max(s_min, P));
      int zl_best = nz;
      int64_t best_cost = INT64_MAX;
      for (int sp = s_min; sp <= s_max; ++sp) {
        const int64_t zl = (nz + sp - 1) / sp;
        const int64_t zr = (nz + zl - 1) / zl;
        const int64_t cost = ((c * zr + P - 1) / P) * (zl + K);
        if (cost < best_cost) {
          best_cost = cost;
          zl_best = (int)zl;
        }
      }
      const int zl = zl_best;
      const int zr = (nz + zl - 1) / zl;
      int in_item = 0;
      for (const Seg& x : xs[xc]) {
        for (const Seg& y : ys[yc]) {
          for (int k = 0; k < zr; ++k) {
            if (in_item == 0) items->push_back({inst, gw, gh, (int)groups->size(), zl});
            fx::TileGroup g;
            g.x0 = x.o;
            g.xout = x.n;
            g.y0 = y.o;
            g.yout = y.n;
            g.z0 = (int)std::min<int64_t>((int64_t)k * zl, nz - zl);
            groups->push_back(g);
            if (++in_item == P) in_item = 0;
          }
        }
      }
      // the last tile's unused rectangles store nothing
      for (; in_item != 0 && in_item < P; ++in_item) groups->push_back(fx::TileGroup{});
    }
  }
  return FDB_OK;
}

// Tiles x planes marched per time block by pack_instance's tiles.
int64_t packed_cost(int nx, int ny, int nz, int K, int R, int W) {
  std::vector<ItemDev> items;
  std::vector<fx::TileGroup> groups;
  pack_instance(nx, ny, nz, 0, K, R, W, 0, &items, &groups);
  int64_t c = 0;
  for (const ItemDev& it : items) c += it.nout + K;
  return c;
}

// Stored order of an instance with view extents n: the permutation whose
// packed tiles (pack_instance at the default depth with 4 rows x 8 warps)
// march the fewest tile-planes per time block; ties keep the view order.
// Orders whose stored plane has 2^31 cells or more are skipped (the fixed
// kernel's limit).
std::array<int, 3> choose_order(const uint64_t n[3]) {
  static const int ps[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
  std::array<int, 3> best = {0, 1, 2};
  int64_t best_cost = INT64_MAX;
  for (const auto& p : ps) {
    if (n[p[1]] * n[p[2]] >= (1ull << 31) || n[p[0]] >= (1ull << 31)) continue;
    const int64_t cost =
        packed_cost((int)n[p[2]], (int)n[p[1]], (int)n[p[0]], kDefaultDepth, 4, 8);
    if (cost < best_cost) {
      best_cost = cost;
      best = {p[0], p[1], p[2]};
    }
  }
  return best;
}

template <int K, int R, int W, bool kLeft = false, bool kOff32 = K == 2>
int launch_batch_kernel(int grid, const InstDev* insts, const ItemDev* items,
                        const fx::TileGroup* groups, int ipb, int nblocks, int steps, int64_t* a0,
                        int64_t* a1, ScaleSlot* slots, unsigned* done, unsigned* queue, int* err,
                        unsigned wait_bias, long long wait_cycles, cudaStream_t st) {
  constexpr int smem = K * R * 32 * W * (int)sizeof(int64_t);
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(k_batch_fixed<K, R, W, kLeft, kOff32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         smem);
    configured = true;
  }
  FDB_CUDA_TRY(launch_dependent(k_batch_fixed<K, R, W, kLeft, kOff32>, (unsigned)grid, 32 * W, smem,
                                st, insts, items, groups, ipb, nblocks, steps, a0, a1, slots,
                                done, queue, err, wait_bias, wait_cycles));
  return FDB_OK;
}

template <int K, int R, int W, bool kLeft = false, bool kOff32 = K == 2>
int resident_ctas_of() {
  constexpr int smem = K * R * 32 * W * (int)sizeof(int64_t);
  cudaFuncSetAttribute(k_batch_fixed<K, R, W, kLeft, kOff32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_fixed<K, R, W, kLeft, kOff32>, 32 * W, smem);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::max(1, per_sm) * std::max(1, sms);
}

using LaunchFn = int (*)(int, const InstDev*, const ItemDev*, const fx::TileGroup*, int, int,
                         int, int64_t*, int64_t*,
                         ScaleSlot*, unsigned*, unsigned*, int*, unsigned, long long,
                         cudaStream_t);
using ResidentFn = int (*)();

struct Variant {
  int K, shape;
  LaunchFn launch;
  ResidentFn resident;
  bool wide = false;  // serves planes of 4 GB and more where another entry does not
};

// compiled (K, shape) combinations of the batched kernel
const Variant kVariants[] = {
    {2, fx::kR4W16S, launch_batch_kernel<2, 4, 16>, resident_ctas_of<2, 4, 16>},
    {3, fx::kR4W16S, launch_batch_kernel<3, 4, 16>, resident_ctas_of<3, 4, 16>},
    {4, fx::kR4W16S, launch_batch_kernel<4, 4, 16>, resident_ctas_of<4, 4, 16>},
    {2, fx::kR4W8S, launch_batch_kernel<2, 4, 8>, resident_ctas_of<2, 4, 8>},
    {3, fx::kR4W8S, launch_batch_kernel<3, 4, 8>, resident_ctas_of<3, 4, 8>},
    {4, fx::kR4W8S, launch_batch_kernel<4, 4, 8>, resident_ctas_of<4, 4, 8>},
    {2, fx::kR8W8S, launch_batch_kernel<2, 8, 8>, resident_ctas_of<2, 8, 8>},
    {3, fx::kR8W8S, launch_batch_kernel<3, 8, 8>, resident_ctas_of<3, 8, 8>},
    {4, fx::kR8W8S, launch_batch_kernel<4, 8, 8>, resident_ctas_of<4, 8, 8>},
    // by the automatic choice only
    {2, fx::kR6W4L, launch_batch_kernel<2, 6, 4, true>, resident_ctas_of<2, 6, 4, true>},
    {3, fx::kR6W4L, launch_batch_kernel<3, 6, 4, true>, resident_ctas_of<3, 6, 4, true>},
    // planes of 4 GB and more at K = 2
    {2, fx::kR4W16S, launch_batch_kernel<2, 4, 16, false, false>,
     resident_ctas_of<2, 4, 16, false, false>, true},
    {2, fx::kR4W8S, launch_batch_kernel<2, 4, 8, false, false>,
     resident_ctas_of<2, 4, 8, false, false>, true},
    {2, fx::kR8W8S, launch_batch_kernel<2, 8, 8, false, false>,
     resident_ctas_of<2, 8, 8, false, false>, true},
    {2, fx::kR6W4L, launch_batch_kernel<2, 6, 4, true, false>,
     resident_ctas_of<2, 6, 4, true, false>, true},
};

const Variant* find_variant(int K, int shape, bool wide) {
  for (const Variant& v : kVariants)
    if (v.K == K && v.shape == shape && v.wide == (wide && K == 2)) return &v;
  return nullptr;
}

}  // namespace bt
}  // namespace fdb

using namespace fdb;
using namespace fdb::bt;

// A plan and its device tables.  captured: a graph of the caller holds their
// addresses, so that they are neither rewritten nor freed before the batch is.
struct PlanTables {
  bool captured = false;
  const Variant* v = nullptr;  // null: no plan
  int shape = -1, tz = 0;
  std::vector<double> dt;
  int ipb = 0, resident = 0;
  InstDev* d_insts = nullptr;
  ItemDev* d_items = nullptr;
  size_t item_cap = 0;
  fx::TileGroup* d_groups = nullptr;
  size_t group_cap = 0;
};

struct fdb_batch {
  int count = 0;
  std::vector<Geom> geoms;      // as stored (the kernels' geometry)
  std::vector<Geom> geoms_ref;  // as described by the caller
  std::vector<std::array<int, 3>> order;  // stored axis k = view axis order[k]
  std::vector<char> permuted;
  double* d_stage = nullptr;  // one instance in the caller's order
  uint64_t stage_cells = 0;
  // batched adjoint storage (grown on demand): checkpoints, segment buffers
  // (two int64 chains, then int32 states two per buffer), adjoint ping-pong,
  // lambda_T / dL/df0 in the stored layout, the caller-order copy, scratch
  std::vector<double*> adj_ckpt, adj_seg;
  double* adj_lam[2] = {nullptr, nullptr};
  double* adj_io[2] = {nullptr, nullptr};
  double* adj_user = nullptr;
  double* adj_dda = nullptr;
  void* adj_scratch = nullptr;
  size_t adj_scratch_bytes = 0;
  // adjoint form (FDB_TUNE_ADJOINT): 0 = dL/dv in closed form, 1 = step by step
  int adj_mode = 0;
  DeviceScratch contract;  // the closed form's contraction tables and partials
  std::vector<int64_t> offsets;  // cells
  std::vector<uint64_t> sizes;
  int64_t total = 0;
  double* arena[2] = {nullptr, nullptr};
  int cur = 0;
  PlanTables tables[2];  // the forward problem's, the transposed one's
  std::vector<void*> retired;  // tables of captured advects whose plan was replaced
  // an advect was captured: from then on every advect leaves the fields in the
  // arena it found them in, which is the one the caller's graph reads and writes
  bool captured = false;
  ScaleSlot* d_slots = nullptr;
  unsigned* d_done = nullptr;
  unsigned* d_queue = nullptr;
  int* d_err = nullptr;
  int64_t* d_offs = nullptr;
  uint64_t* d_sizes = nullptr;
  MaxChunks max;  // work items of the max|f| pass
  uint64_t* d_max_first = nullptr;
  double* d_part = nullptr;
  double* d_sums = nullptr;
  double* h_sums = nullptr;
  double* d_plain_scratch = nullptr;  // per-instance scratch of the looped comparator
  IoDev* d_io = nullptr;              // k_batch_io's table (null: too many work items)
  uint32_t io_items = 0;
  cudaStream_t own = nullptr, stream = nullptr;
  // tuning as set (0 / -1 = automatic), and what the launches take
  int K = 0, shape = -1, tz = 0;
  int eff_K = 0, eff_shape = -1, eff_tz = 0;
};

namespace {

constexpr int kSumPerInst = 16;

int bcheck(fdb_batch* b) {
  if (!b) return fail(FDB_ERR_INVALID, "null batch");
  return FDB_OK;
}

int bsync(fdb_batch* b) {
  int* h_err = reinterpret_cast<int*>(b->h_sums + b->count);
  FDB_CUDA_TRY(cudaMemcpyAsync(h_err, b->d_err, sizeof(int), cudaMemcpyDeviceToHost, b->stream));
  FDB_CUDA_TRY(cudaStreamSynchronize(b->stream));
  const int herr = *h_err;
  if (herr) {
    FDB_CUDA_TRY(cudaMemset(b->d_err, 0, sizeof(int)));
    if (herr & 2)
      return fail(FDB_ERR_TIMEOUT, "batched kernel: a bounded wait for a neighbour tile expired");
    return fail(FDB_ERR_NONFINITE, "batched kernel: an instance field holds NaN or Inf");
  }
  return FDB_OK;
}

template <typename T>
int balloc(T** p, size_t count) {
  if (fault_injected("alloc")) return fail(FDB_ERR_INJECTED, "injected allocation failure");
  cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T));
  if (e != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return fail(FDB_ERR_ALLOC, std::string("cudaMalloc failed: ") + cudaGetErrorString(e));
  }
  return FDB_OK;
}

// The tuning or a velocity changed: the plans are built again.
void drop_plans(fdb_batch* b) {
  for (PlanTables& t : b->tables) t.v = nullptr;
}

int check_dts(fdb_batch* b, const double* dt) {
  if (!dt) return fail(FDB_ERR_INVALID, "null dt array");
  for (int i = 0; i < b->count; ++i)
    if (!isfinite(dt[i])) return fail(FDB_ERR_INVALID, "dt must be finite");
  return FDB_OK;
}

// An instance whose plane takes 4 GB or more (beyond 32-bit byte offsets).
bool wide_planes(const fdb_batch* b) {
  for (const Geom& g : b->geoms)
    if ((uint64_t)g.ny * g.nx >= (1ull << 29)) return true;
  return false;
}

int is_capturing(fdb_batch* b, bool* yes) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  FDB_CUDA_TRY(cudaStreamIsCapturing(b->stream, &st));
  *yes = st != cudaStreamCaptureStatusNone;
  return FDB_OK;
}

// The plan of an advect with these settings into `t` (kept from the last call if
// nothing changed): tiles, instance arguments, their device copies.  transposed:
// every upwind direction reversed, the coefficients unchanged.
int make_plan(fdb_batch* b, const double* dt, int K, int shape, int tz, bool transposed,
              PlanTables* t) {
  if (t->v && t->v->K == K && t->shape == shape && t->tz == tz &&
      memcmp(t->dt.data(), dt, b->count * sizeof(double)) == 0)
    return FDB_OK;
  t->v = nullptr;
  const Variant* v = find_variant(K, shape, wide_planes(b));
  if (!v) return fail(FDB_ERR_UNSUPPORTED, "no batched kernel compiled for this depth/shape");
  std::vector<InstDev> insts(b->count);
  std::vector<ItemDev> items;
  std::vector<fx::TileGroup> groups;
  const int resident = v->resident();
  const int R = fx::shape_rows(shape), W = fx::shape_warps(shape);
  int base = 0;
  for (int i = 0; i < b->count; ++i) {
    const Geom& g = b->geoms[i];
    const Coeffs3 c = coeffs3(g, dt[i]);
    if (fixed_supported(g, c, K) != FDB_OK) return FDB_ERR_UNSUPPORTED;
    InstDev& I = insts[i];
    I.a = make_fixed_args(transposed ? transposed_geom(g) : g, c, shape, K,
                          tz > 0 ? tz : (int)g.nz, resident);
    I.a.scale_log = nullptr;
    I.offset = b->offsets[i];
    const size_t first = items.size();
    FDB_TRY(pack_instance(I.a.nx, I.a.ny, I.a.nz, i, K, R, W, tz, &items, &groups));
    const size_t n = items.size() - first;
    if (n > (1u << 24)) return fail(FDB_ERR_UNSUPPORTED, "instance has too many tiles");
    I.items = (int)n;
    I.item_base = base;
    base += I.items;
  }
  if (groups.size() >= (1ull << 31))
    return fail(FDB_ERR_UNSUPPORTED, "batched plan exceeds 2^31 tile rectangles");
  bool capturing = false;
  FDB_TRY(is_capturing(b, &capturing));
  if (capturing)
    return fail(FDB_ERR_CUDA, "a batched advect with new settings cannot be captured (its tables "
                              "are copied from the host): run it once before the capture");
  if (t->captured) {
    for (void* p : {(void*)t->d_insts, (void*)t->d_items, (void*)t->d_groups})
      b->retired.push_back(p);
    *t = PlanTables();
  }
  if (!t->d_insts) FDB_TRY(balloc(&t->d_insts, (size_t)b->count));
  if (items.size() > t->item_cap) {
    if (t->d_items) cudaFree(t->d_items);
    t->d_items = nullptr;
    t->item_cap = 0;
    FDB_TRY(balloc(&t->d_items, items.size()));
    t->item_cap = items.size();
  }
  if (groups.size() > t->group_cap) {
    if (t->d_groups) cudaFree(t->d_groups);
    t->d_groups = nullptr;
    t->group_cap = 0;
    FDB_TRY(balloc(&t->d_groups, groups.size()));
    t->group_cap = groups.size();
  }
  FDB_CUDA_TRY(cudaMemcpyAsync(t->d_insts, insts.data(), insts.size() * sizeof(InstDev),
                               cudaMemcpyHostToDevice, b->stream));
  FDB_CUDA_TRY(cudaMemcpyAsync(t->d_items, items.data(), items.size() * sizeof(ItemDev),
                               cudaMemcpyHostToDevice, b->stream));
  FDB_CUDA_TRY(cudaMemcpyAsync(t->d_groups, groups.data(), groups.size() * sizeof(fx::TileGroup),
                               cudaMemcpyHostToDevice, b->stream));
  FDB_CUDA_TRY(cudaStreamSynchronize(b->stream));  // the sources end with this call
  t->shape = shape;
  t->tz = tz;
  t->dt.assign(dt, dt + b->count);
  t->ipb = base;
  t->resident = resident;
  t->v = v;
  return FDB_OK;
}

int run_batched(fdb_batch* b, int steps, const double* dt, int K, int shape, int tz,
                bool transposed = false) {
  PlanTables& t = b->tables[transposed ? 1 : 0];
  FDB_TRY(make_plan(b, dt, K, shape, tz, transposed, &t));
  const int nblocks = (steps + K - 1) / K;
  if ((int64_t)nblocks * t.ipb >= (1ll << 31))
    return fail(FDB_ERR_UNSUPPORTED, "batched work queue exceeds 2^31 items");
  bool capturing = false;
  FDB_TRY(is_capturing(b, &capturing));
  const int grid = (int)std::min<int64_t>((int64_t)nblocks * t.ipb, t.resident);
  cudaStream_t st = b->stream;
  k_batch_reset<<<(3 * b->count + 255) / 256, 256, 0, st>>>(b->d_slots, b->d_done, b->d_queue,
                                                            b->count);
  const unsigned max_blocks = (unsigned)std::min<uint64_t>(b->max.first.back(), 0x7FFFFFFF);
  FDB_CUDA_TRY(launch_dependent(k_batch_absmax, max_blocks, 256, 0, st, b->arena[b->cur],
                                b->d_offs, b->d_sizes, b->d_max_first, b->count, b->max.cells,
                                b->d_slots));
  int64_t* a0 = (int64_t*)b->arena[b->cur];
  int64_t* a1 = (int64_t*)b->arena[b->cur ^ 1];
  // FDB_FAULT=timeout makes every dependency unsatisfiable and the wait
  // budget ~1 ms, so the bounded-wait error path runs without a GPU fault
  const bool inject = fault_injected("timeout");
  FDB_TRY(t.v->launch(grid, t.d_insts, t.d_items, t.d_groups, t.ipb, nblocks, steps, a0, a1,
                      b->d_slots, b->d_done, b->d_queue, b->d_err, inject ? (1u << 30) : 0u,
                      inject ? 2000000ll : kWaitCycles, st));
  note_launch(3);
  FDB_CUDA_TRY(cudaGetLastError());
  if (capturing) t.captured = b->captured = true;
  // an odd number of blocks ends in the other arena; the transposed steps run on
  // the adjoint buffers, which no graph holds (their calls wait for the stream)
  if (!b->captured || transposed)
    b->cur ^= (nblocks & 1);
  else if (nblocks & 1)
    FDB_CUDA_TRY(cudaMemcpyAsync(a0, a1, (size_t)b->total * 8, cudaMemcpyDeviceToDevice, st));
  return FDB_OK;
}

// The comparator: the plain per-field kernels looped over the instances,
// K steps per fixed-point launch; K <= 0: what fdb_upwind_advect runs for
// each instance (the fixed kernel at its default depth where it is
// supported and preferred, the FP64 kernel otherwise).  Every instance ends
// in the same arena: the one most instances end in (once captured: the one they
// began in); the others are copied across.
int run_looped(fdb_batch* b, int steps, const double* dt, int K) {
  const size_t per = (fixed_scratch_bytes() + 7) / 8;
  std::vector<int> fin(b->count);
  for (int i = 0; i < b->count; ++i) {
    const Geom& g = b->geoms[i];
    const Coeffs3 c = coeffs3(g, dt[i]);
    double* bufs[2] = {b->arena[0] + b->offsets[i], b->arena[1] + b->offsets[i]};
    int cur = b->cur;
    // depth and arithmetic as fdb_upwind_advect picks them for the described
    // instance (the stored order does not change the fixed-point result)
    const Geom& gr = b->geoms_ref[i];
    FixedTuning t;
    t.depth = K > 0 ? K : default_depth(gr);
    if (fixed_supported(g, c, t.depth) == FDB_OK && (K > 0 || fixed_preferred(gr))) {
      FDB_TRY(launch_advect_fixed_ex(g, c, steps, t, bufs, &cur, b->d_plain_scratch + i * per,
                                     per * 8, nullptr, b->stream));
    } else {
      FDB_TRY(launch_advect_f64(g, c, FDB_ARITH_FMA, steps, bufs, &cur, b->stream));
    }
    fin[i] = cur;
  }
  int ones = 0;
  for (int i = 0; i < b->count; ++i) ones += fin[i];
  bool capturing = false;
  FDB_TRY(is_capturing(b, &capturing));
  b->captured |= capturing;
  const int new_cur = b->captured ? b->cur : 2 * ones > b->count ? 1 : 0;
  for (int i = 0; i < b->count; ++i) {
    if (fin[i] == new_cur) continue;
    FDB_CUDA_TRY(cudaMemcpyAsync(b->arena[new_cur] + b->offsets[i], b->arena[fin[i]] + b->offsets[i],
                                 b->sizes[i] * 8, cudaMemcpyDeviceToDevice, b->stream));
  }
  b->cur = new_cur;
  return FDB_OK;
}

// Fills in the tuning that is not set (b->eff_*).
//
// Depth 2 or 3 and CTAs of 4 rows x 8 warps or 6 rows x 4 warps: the fewest
// computed rows, sum over the packed tiles of (planes + K) R W (K + 0.86) / K
// (0.86 levels: a plane's load, scale and store), as in the single-field
// choice.  Ranges of z: few long tiles per time block leave CTAs idle until
// the block's last tile is done, short ones repeat K warm-up planes each.
// With q the tile-planes of a block per resident CTA, 3 sqrt(q) + q / 30 planes
// (at least 8) is within 7 % of the best of a sweep (12 .. 200 instances, q from 3
// to 340); from q = 400 on whole columns are best.  Measured, advect GCUPS,
// depth 2, 4 rows and whole columns -> this: 8 x 96^3 99 -> 271; 40 x 64^3
// 200 -> 375; 33 instances of [61, 98]^3 211 -> 349; 64 x 128^3 465 -> 496.
//
// Batches whose tiles of 8 planes at depth 4 fill at most half of the resident
// CTAs wait for one tile after the other, block by block: the fewest blocks win.
// 40 steps, us, rule above -> depth 4: 8 of [24, 40]^3 271 -> 237; 8 of [40, 64]^3
// 345 -> 325; 4 x 48^3 339 -> 255; 4 x 64^3 360 -> 304.  Beyond half it loses: 4 x
// 96^3 (576 tiles) 502 -> 512, 12 of [64, 90]^3 738 -> 794.
void choose_tuning(fdb_batch* b) {
  struct Cand {
    int K, shape;
  };
  static const Cand cands[] = {
      {2, fx::kR4W8S}, {3, fx::kR4W8S}, {2, fx::kR6W4L}, {3, fx::kR6W4L}};
  std::vector<Cand> list;
  for (const Cand& c : cands)
    if ((b->K <= 0 || b->K == c.K) && (b->shape < 0 || b->shape == c.shape)) list.push_back(c);
  // a setting outside the candidates: itself, the rest at their first choice
  if (list.empty())
    list.push_back({b->K > 0 ? b->K : kDefaultDepth, b->shape >= 0 ? b->shape : (int)fx::kR4W8S});
  auto pack = [&](const Cand& c, int tz, std::vector<ItemDev>* items) {
    std::vector<fx::TileGroup> groups;
    items->clear();
    for (int i = 0; i < b->count; ++i) {
      const Geom& g = b->geoms[i];
      pack_instance((int)g.nx, (int)g.ny, (int)g.nz, i, c.K, fx::shape_rows(c.shape),
                    fx::shape_warps(c.shape), tz, items, &groups);
    }
  };
  double best = 0.0;
  std::vector<ItemDev> items;
  const Variant* deep = find_variant(4, fx::kR4W8S, wide_planes(b));
  if (deep && (b->K <= 0 || b->K == 4) && (b->shape < 0 || b->shape == fx::kR4W8S) && b->tz <= 0) {
    pack({4, fx::kR4W8S}, 8, &items);
    if (2 * (int)items.size() <= deep->resident()) {
      b->eff_K = 4;
      b->eff_shape = fx::kR4W8S;
      b->eff_tz = 8;
      return;
    }
  }
  for (const Cand& c : list) {
    int tz = b->tz;
    if (tz <= 0) {
      const Variant* v = find_variant(c.K, c.shape, wide_planes(b));
      pack(c, 0, &items);
      double planes = 0.0;
      for (const ItemDev& it : items) planes += it.nout;
      const double q = planes / (v ? v->resident() : 1);
      tz = q >= 400.0 ? 0 : std::max(8, (int)ceil(3.0 * sqrt(q) + q / 30.0));
    }
    pack(c, tz, &items);
    double cost = 0.0;
    for (const ItemDev& it : items) cost += it.nout + c.K;
    cost *= fx::shape_rows(c.shape) * fx::shape_warps(c.shape) * (1.0 + 0.86 / c.K);
    if (best == 0.0 || cost < best) {
      best = cost;
      b->eff_K = c.K;
      b->eff_shape = c.shape;
      b->eff_tz = tz;
    }
  }
}

int effective_K(fdb_batch* b) { return b->eff_K; }

void free_batch_adjoint(fdb_batch* b) {
  for (double* p : b->adj_ckpt) cudaFree(p);
  for (double* p : b->adj_seg) cudaFree(p);
  b->adj_ckpt.clear();
  b->adj_seg.clear();
  for (double*& p : b->adj_lam) {
    if (p) cudaFree(p);
    p = nullptr;
  }
  for (double*& p : b->adj_io) {
    if (p) cudaFree(p);
    p = nullptr;
  }
  if (b->adj_user) cudaFree(b->adj_user);
  if (b->adj_dda) cudaFree(b->adj_dda);
  if (b->adj_scratch) cudaFree(b->adj_scratch);
  b->adj_user = nullptr;
  b->adj_dda = nullptr;
  b->adj_scratch = nullptr;
  b->adj_scratch_bytes = 0;
}

// Whether a kernel on the current device may read and write p (a copy may also
// reach another GPU's memory).  FDB_FAULT=foreign denies it for every pointer but
// the batch's own.
bool on_current_device(const void* p) {
  if (fault_injected("foreign")) return false;
  int dev = 0;
  cudaPointerAttributes at{};
  if (cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (at.type == cudaMemoryTypeDevice && at.device == dev) || at.type == cudaMemoryTypeManaged;
}

// Whether p lies in one of the batch's own field buffers.
bool own_memory(const fdb_batch* b, const void* p) {
  const struct {
    const double* at;
    uint64_t cells;
  } bufs[] = {{b->arena[0], (uint64_t)b->total},   {b->arena[1], (uint64_t)b->total},
              {b->adj_lam[0], (uint64_t)b->total}, {b->adj_lam[1], (uint64_t)b->total},
              {b->adj_io[0], (uint64_t)b->total},  {b->adj_io[1], (uint64_t)b->total},
              {b->adj_user, (uint64_t)b->total},   {b->d_stage, b->stage_cells}};
  const uintptr_t x = (uintptr_t)p;
  for (const auto& m : bufs)
    if (m.at && x >= (uintptr_t)m.at && x < (uintptr_t)(m.at + m.cells)) return true;
  return false;
}

// instance i between the caller's order and the stored order (see k_permute3);
// src and dst are memory that a kernel may use
int launch_permute(fdb_batch* b, int i, const double* src, double* dst, bool to_view) {
  for (const void* p : {(const void*)src, (const void*)dst})
    if (!own_memory(b, p) && !on_current_device(p))
      return fail(FDB_ERR_INVALID, "permutation of memory that the current device cannot reach");
  uint64_t n3[3];
  double v3[3], L3[3];
  view3(b->geoms_ref[i], n3, v3, L3);
  const std::array<int, 3>& o = b->order[i];
  const uint64_t blocks = std::min<uint64_t>((b->sizes[i] + 255) / 256, 152 * 16);
  k_permute3<<<(unsigned)blocks, 256, 0, b->stream>>>(src, dst, n3[0], n3[1], n3[2], o[0], o[1],
                                                       o[2], to_view ? 1 : 0);
  note_launch();
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

// k_batch_io's table: the caller's layout holds the instances one after another.
int make_io_table(fdb_batch* b) {
  std::vector<IoDev> t(b->count);
  uint64_t items = 0;
  int64_t user = 0;
  for (int i = 0; i < b->count; ++i) {
    uint64_t n3[3];
    double v3[3], L3[3];
    view3(b->geoms_ref[i], n3, v3, L3);
    IoDev& I = t[i];
    I.user = user;
    I.arena = b->offsets[i];
    for (int k = 0; k < 3; ++k) {
      if (n3[k] >= (1ull << 32)) return FDB_OK;  // copied instance by instance
      I.n[k] = (uint32_t)n3[k];
      I.p[k] = b->order[i][k];
    }
    I.item0 = (uint32_t)items;
    items += io_items(I.n, I.p);
    if (items >= (1ull << 31)) return FDB_OK;
    user += (int64_t)b->sizes[i];
  }
  FDB_TRY(balloc(&b->d_io, t.size()));
  FDB_CUDA_TRY(cudaMemcpyAsync(b->d_io, t.data(), t.size() * sizeof(IoDev),
                               cudaMemcpyHostToDevice, b->stream));
  FDB_CUDA_TRY(cudaStreamSynchronize(b->stream));  // the source ends with this call
  b->io_items = (uint32_t)items;
  return FDB_OK;
}

// Cells of the caller's concatenated fields.
uint64_t user_cells(const fdb_batch* b) {
  uint64_t c = 0;
  for (uint64_t z : b->sizes) c += z;
  return c;
}

// Every instance between the caller's concatenated fields (device memory) and
// an arena, on the batch's stream: one launch, or instance by instance where
// the table does not serve or the caller's memory is another GPU's, which only
// copies reach: a permuted instance then passes through d_stage.
int io_all(fdb_batch* b, const double* src, double* dst, bool to_view) {
  if (b->d_io && on_current_device(to_view ? dst : src)) {
    const uint32_t blocks = std::min<uint32_t>(b->io_items, 152 * 8);
    k_batch_io<<<blocks, 256, 0, b->stream>>>(src, dst, b->d_io, b->count, b->io_items,
                                              to_view ? 1 : 0);
    note_launch();
    FDB_CUDA_TRY(cudaGetLastError());
    return FDB_OK;
  }
  uint64_t user = 0;
  for (int i = 0; i < b->count; ++i) {
    const double* s = src + (to_view ? b->offsets[i] : (int64_t)user);
    double* d = dst + (to_view ? (int64_t)user : b->offsets[i]);
    const bool perm = b->permuted[i];
    if (perm && to_view) {
      FDB_TRY(launch_permute(b, i, s, b->d_stage, true));
      s = b->d_stage;
    }
    FDB_CUDA_TRY(cudaMemcpyAsync(perm && !to_view ? b->d_stage : d, s, b->sizes[i] * 8,
                                 cudaMemcpyDeviceToDevice, b->stream));
    if (perm && !to_view) FDB_TRY(launch_permute(b, i, b->d_stage, d, false));
    user += b->sizes[i];
  }
  return FDB_OK;
}

int effective_shape(fdb_batch* b) { return b->eff_shape; }

int effective_tz(fdb_batch* b) { return b->eff_tz; }

}  // namespace

extern "C" {

int fdb_batch_create(int count, const fdb_instance_desc* descs, fdb_batch** out) {
  if (!out) return fail(FDB_ERR_INVALID, "null output batch pointer");
  *out = nullptr;
  if (count <= 0 || !descs) return fail(FDB_ERR_INVALID, "count must be > 0 with descriptors");
  fdb_batch* b = new fdb_batch();
  b->count = count;
  for (int i = 0; i < count; ++i) {
    Geom g;
    const fdb_instance_desc& d = descs[i];
    if (d.ndims < 1 || d.ndims > 3) {
      delete b;
      return fail(FDB_ERR_INVALID, "batched instances have 1 to 3 axes");
    }
    int rc = make_geom(d.ndims, d.velocity, d.lengths, d.num_cells, &g);
    if (rc) {
      delete b;
      return rc;
    }
    // stored order: permuted only where the single-field path would run the
    // (order-independent) fixed kernel
    uint64_t n3[3];
    double v3[3], L3[3];
    view3(g, n3, v3, L3);
    const std::array<int, 3> ord =
        fixed_preferred(g) ? choose_order(n3) : std::array<int, 3>{0, 1, 2};
    const bool perm = !(ord[0] == 0 && ord[1] == 1 && ord[2] == 2);
    Geom gs = g;
    if (perm) {
      uint64_t np[3];
      double vp[3], Lp[3];
      for (int k = 0; k < 3; ++k) {
        np[k] = n3[ord[k]];
        vp[k] = v3[ord[k]];
        Lp[k] = L3[ord[k]];
      }
      rc = make_geom(3, vp, Lp, np, &gs);
      if (rc) {
        delete b;
        return rc;
      }
      b->stage_cells = std::max<uint64_t>(b->stage_cells, g.ntot);
    }
    b->geoms.push_back(gs);
    b->geoms_ref.push_back(g);
    b->order.push_back(ord);
    b->permuted.push_back(perm ? 1 : 0);
    b->offsets.push_back(b->total);
    b->sizes.push_back(g.ntot);
    // keep every instance 256-byte aligned in the arenas
    b->total += (int64_t)((g.ntot + 31) / 32 * 32);
  }
  cudaError_t e = cudaStreamCreateWithFlags(&b->own, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete b;
    return cuda_fail(e, "cudaStreamCreate");
  }
  b->stream = b->own;
  b->max = max_chunks(b->sizes);
  const size_t per = (fixed_scratch_bytes() + 7) / 8;
  int rc = FDB_OK;
  if ((rc = balloc(&b->arena[0], b->total)) || (rc = balloc(&b->arena[1], b->total)) ||
      (rc = balloc(&b->d_slots, 3 * count)) ||
      (rc = balloc(&b->d_done, count)) || (rc = balloc(&b->d_queue, 1)) ||
      (rc = balloc(&b->d_err, 1)) || (rc = balloc(&b->d_offs, count)) ||
      (rc = balloc(&b->d_sizes, count)) ||
      (rc = balloc(&b->d_max_first, (size_t)count + 1)) ||
      (rc = balloc(&b->d_part, count * kSumPerInst)) ||
      (rc = balloc(&b->d_sums, count)) || (rc = balloc(&b->d_plain_scratch, per * count)) ||
      (b->stage_cells && (rc = balloc(&b->d_stage, b->stage_cells)))) {
    fdb_batch_destroy(b);
    return rc;
  }
  e = cudaMallocHost((void**)&b->h_sums, (count + 1) * sizeof(double));  // and the error word
  if (e == cudaSuccess) e = cudaMemsetAsync(b->d_err, 0, sizeof(int), b->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(b->d_plain_scratch, 0, per * count * 8, b->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(b->arena[0], 0, b->total * 8, b->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(b->d_offs, b->offsets.data(), count * 8, cudaMemcpyHostToDevice, b->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(b->d_sizes, b->sizes.data(), count * 8, cudaMemcpyHostToDevice, b->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(b->d_max_first, b->max.first.data(), (count + 1) * 8,
                        cudaMemcpyHostToDevice, b->stream);
  if (e != cudaSuccess) {
    fdb_batch_destroy(b);
    return cuda_fail(e, "batch set-up");
  }
  choose_tuning(b);
  rc = make_io_table(b);
  // each instance starts like the reference constructor: f = 0, f[0] = 1
  for (int i = 0; i < count && !rc; ++i)
    rc = launch_fill_corner(b->arena[0] + b->offsets[i], b->sizes[i], b->stream);
  if (!rc) rc = bsync(b);
  if (rc) {
    fdb_batch_destroy(b);
    return rc;
  }
  *out = b;
  return FDB_OK;
}

int fdb_batch_destroy(fdb_batch* b) {
  if (!b) return FDB_OK;
  if (b->stream) cudaStreamSynchronize(b->stream);
  drop_plans(b);
  void* ps[] = {b->arena[0], b->arena[1], b->d_slots,  b->d_done,  b->d_queue, b->d_err,    b->d_offs,
                b->d_sizes,  b->d_part,  b->d_sums,  b->d_plain_scratch, b->d_stage,
                b->d_io, b->d_max_first};
  for (void* p : ps)
    if (p) cudaFree(p);
  for (PlanTables& t : b->tables) {
    cudaFree(t.d_insts);
    cudaFree(t.d_items);
    cudaFree(t.d_groups);
  }
  for (void* p : b->retired) cudaFree(p);
  free_batch_adjoint(b);
  b->contract.release();
  if (b->h_sums) cudaFreeHost(b->h_sums);
  if (b->own) cudaStreamDestroy(b->own);
  delete b;
  return FDB_OK;
}

int fdb_batch_set_velocity(fdb_batch* b, int index, const double* velocity) {
  FDB_TRY(bcheck(b));
  if (index < 0 || index >= b->count || !velocity)
    return fail(FDB_ERR_INVALID, "bad index or velocity");
  const Geom& old = b->geoms_ref[index];
  Geom g;
  FDB_TRY(make_geom(old.ndims, velocity, old.L, old.n, &g));
  Geom gs = g;
  if (b->permuted[index]) {
    uint64_t n3[3];
    double v3[3], L3[3];
    view3(g, n3, v3, L3);
    uint64_t np[3];
    double vp[3], Lp[3];
    const std::array<int, 3>& o = b->order[index];
    for (int k = 0; k < 3; ++k) {
      np[k] = n3[o[k]];
      vp[k] = v3[o[k]];
      Lp[k] = L3[o[k]];
    }
    FDB_TRY(make_geom(3, vp, Lp, np, &gs));
  }
  FDB_TRY(bsync(b));
  b->geoms_ref[index] = g;
  b->geoms[index] = gs;
  drop_plans(b);
  return FDB_OK;
}

int fdb_batch_storage_order(fdb_batch* b, int index, int* order3) {
  FDB_TRY(bcheck(b));
  if (index < 0 || index >= b->count || !order3) return fail(FDB_ERR_INVALID, "bad index or output");
  for (int k = 0; k < 3; ++k) order3[k] = b->order[index][k];
  return FDB_OK;
}

int fdb_batch_count(fdb_batch* b, int* count, uint64_t* total_cells) {
  FDB_TRY(bcheck(b));
  if (count) *count = b->count;
  if (total_cells) {
    uint64_t t = 0;
    for (uint64_t s : b->sizes) t += s;
    *total_cells = t;
  }
  return FDB_OK;
}

int fdb_batch_set_field(fdb_batch* b, int index, const double* src, int is_device) {
  FDB_TRY(bcheck(b));
  if (index < 0 || index >= b->count || !src) return fail(FDB_ERR_INVALID, "bad index or source");
  double* dst = b->arena[b->cur] + b->offsets[index];
  const bool perm = b->permuted[index];
  FDB_CUDA_TRY(cudaMemcpyAsync(perm ? b->d_stage : dst, src, b->sizes[index] * 8,
                               is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                               b->stream));
  if (perm) FDB_TRY(launch_permute(b, index, b->d_stage, dst, false));
  return bsync(b);
}

int fdb_batch_get_field(fdb_batch* b, int index, double* dst, int is_device) {
  FDB_TRY(bcheck(b));
  if (index < 0 || index >= b->count || !dst) return fail(FDB_ERR_INVALID, "bad index or destination");
  const double* src = b->arena[b->cur] + b->offsets[index];
  const bool perm = b->permuted[index];
  if (perm) FDB_TRY(launch_permute(b, index, src, b->d_stage, true));
  FDB_CUDA_TRY(cudaMemcpyAsync(dst, perm ? b->d_stage : src, b->sizes[index] * 8,
                               is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                               b->stream));
  return bsync(b);
}

int fdb_batch_set_fields(fdb_batch* b, const double* src, int is_device) {
  FDB_TRY(bcheck(b));
  if (!src) return fail(FDB_ERR_INVALID, "null source");
  if (is_device) {
    FDB_TRY(io_all(b, src, b->arena[b->cur], false));
    return bsync(b);
  }
  for (int i = 0; i < b->count; src += b->sizes[i], ++i)
    FDB_TRY(fdb_batch_set_field(b, i, src, 0));
  return FDB_OK;
}

int fdb_batch_get_fields(fdb_batch* b, double* dst, int is_device) {
  FDB_TRY(bcheck(b));
  if (!dst) return fail(FDB_ERR_INVALID, "null destination");
  if (is_device) {
    FDB_TRY(io_all(b, b->arena[b->cur], dst, true));
    return bsync(b);
  }
  for (int i = 0; i < b->count; dst += b->sizes[i], ++i)
    FDB_TRY(fdb_batch_get_field(b, i, dst, 0));
  return FDB_OK;
}

int fdb_batch_init_sphere(fdb_batch* b, int index, const double* center, double radius,
                          double noise_amp, uint64_t seed) {
  FDB_TRY(bcheck(b));
  if (index < 0 || index >= b->count || !center) return fail(FDB_ERR_INVALID, "bad index or centre");
  double* dst = b->arena[b->cur] + b->offsets[index];
  const bool perm = b->permuted[index];
  // generated in the caller's order (the generator is a function of the
  // reference's cell index), then stored
  FDB_TRY(launch_sphere_noise(b->geoms_ref[index], center, radius, noise_amp, seed,
                              perm ? b->d_stage : dst, b->stream));
  if (perm) FDB_TRY(launch_permute(b, index, b->d_stage, dst, false));
  return bsync(b);
}

int fdb_batch_set_stream(fdb_batch* b, void* cuda_stream) {
  FDB_TRY(bcheck(b));
  FDB_TRY(bsync(b));
  b->stream = cuda_stream ? (cudaStream_t)cuda_stream : b->own;
  drop_plans(b);
  return FDB_OK;
}

int fdb_batch_set_tuning(fdb_batch* b, int key, int value) {
  FDB_TRY(bcheck(b));
  if (key == FDB_TUNE_DEPTH) {
    if (value < 0 || value == 1 || value > 4) return fail(FDB_ERR_INVALID, "batched depth is 0, 2, 3 or 4");
    b->K = value;
  } else if (key == FDB_TUNE_SHAPE) {
    if (!(value == -1 || value == fx::kR4W16S || value == fx::kR4W8S || value == fx::kR8W8S))
      return fail(FDB_ERR_INVALID, "batched shape is -1, 2 (8x8), 3 (4x16) or 4 (4x8)");
    b->shape = value;
  } else if (key == FDB_TUNE_TILE_Z) {
    if (value < 0) return fail(FDB_ERR_INVALID, "tile_z must be >= 0");
    b->tz = value;
  } else if (key == FDB_TUNE_ADJOINT) {
    if (value < 0 || value > 2) return fail(FDB_ERR_INVALID, "adjoint form must be 0, 1 or 2");
    b->adj_mode = value;
    return FDB_OK;
  } else {
    return fail(FDB_ERR_INVALID, "unknown tuning key");
  }
  choose_tuning(b);
  drop_plans(b);
  return FDB_OK;
}

int fdb_batch_advect(fdb_batch* b, int num_steps, const double* dt) {
  NvtxScope nvtx_("fdb.batch.advect");
  FDB_TRY(bcheck(b));
  if (num_steps < 0) return fail(FDB_ERR_INVALID, "num_steps must be >= 0");
  FDB_TRY(check_dts(b, dt));
  if (num_steps == 0) return FDB_OK;
  const int rc = run_batched(b, num_steps, dt, effective_K(b), effective_shape(b), effective_tz(b));
  if (rc == FDB_ERR_UNSUPPORTED) {
    // some instance is outside the fixed kernel's domain: loop the plain path
    return run_looped(b, num_steps, dt, effective_K(b));
  }
  return rc;
}

int fdb_batch_advect_looped(fdb_batch* b, int num_steps, const double* dt) {
  NvtxScope nvtx_("fdb.batch.advect_looped");
  FDB_TRY(bcheck(b));
  if (num_steps < 0) return fail(FDB_ERR_INVALID, "num_steps must be >= 0");
  FDB_TRY(check_dts(b, dt));
  if (num_steps == 0) return FDB_OK;
  return run_looped(b, num_steps, dt, b->K);
}

// The transposed problems run on the adjoint buffers adj_lam[0..1] (the
// fields are untouched): each instance's upwind directions reversed, its
// coefficients unchanged, in its storage order.
//
// adj_lam[0] = the caller's concatenated fields `in`, permuted into the
// storage order.
static int batch_lam_load(fdb_batch* b, const double* in, int is_device) {
  const size_t T = (size_t)b->total;
  int rc = FDB_OK;
  for (auto& p : b->adj_lam)
    if (!rc && !p) rc = balloc(&p, T);
  if (!rc && !b->adj_user) rc = balloc(&b->adj_user, T);
  if (rc) {
    free_batch_adjoint(b);
    return rc;
  }
  const double* lt = in;
  if (!is_device) {
    FDB_CUDA_TRY(cudaMemcpyAsync(b->adj_user, in, user_cells(b) * 8, cudaMemcpyHostToDevice,
                                 b->stream));
    lt = b->adj_user;
  }
  return io_all(b, lt, b->adj_lam[0], false);
}

// S transposed steps of every instance: the persistent launch on the adjoint
// buffers; *lc (in/out) names the buffer that holds the state.
static int batch_lam_steps(fdb_batch* b, int S, const double* dt, int* lc) {
  if (S <= 0) return FDB_OK;
  const int cur = b->cur;
  std::swap(b->arena[0], b->adj_lam[0]);
  std::swap(b->arena[1], b->adj_lam[1]);
  b->cur = *lc;
  const int rc = run_batched(b, S, dt, effective_K(b), effective_shape(b), effective_tz(b), true);
  *lc = b->cur;
  std::swap(b->arena[0], b->adj_lam[0]);
  std::swap(b->arena[1], b->adj_lam[1]);
  b->cur = cur;
  return rc;
}

// adj_lam[lc] back to the caller's order into `out`.
static int batch_lam_store(fdb_batch* b, int lc, double* out, int is_device) {
  FDB_TRY(io_all(b, b->adj_lam[lc], is_device ? out : b->adj_user, true));
  if (!is_device)
    FDB_CUDA_TRY(cudaMemcpyAsync(out, b->adj_user, user_cells(b) * 8, cudaMemcpyDeviceToHost,
                                 b->stream));
  return FDB_OK;
}

// out = (A^T)^S in for all instances at once; the fields are untouched.
static int batch_transposed(fdb_batch* b, int S, const double* dt, const double* lambda_T,
                            double* grad_f0, int is_device) {
  FDB_TRY(batch_lam_load(b, lambda_T, is_device));
  int lc = 0;
  FDB_TRY(batch_lam_steps(b, S, dt, &lc));
  FDB_TRY(batch_lam_store(b, lc, grad_f0, is_device));
  return bsync(b);
}

// dL/dv of every instance from dL/da of its stored axes: stored axis k is
// view axis order[k], i.e. reference axis jj[order[k]];
// a_j = -dt v_j up_j / dx_j  =>  dL/dv_j = dL/da_j (-dt up_j / dx_j).
static void batch_velocity_grad(fdb_batch* b, const double* dt, const double* dda,
                                double* grad_v) {
  for (int i = 0; i < b->count; ++i) {
    const Geom& gr = b->geoms_ref[i];
    const int jj[3] = {gr.jz, gr.jy, gr.jx};
    for (int k = 0; k < 3; ++k) grad_v[3 * i + k] = 0.0;
    for (int k = 0; k < 3; ++k) {
      const int j = jj[b->order[i][k]];
      if (j >= 0) grad_v[3 * i + j] = dda[3 * i + k] * (-dt[i] * (double)gr.up[j] / gr.dx[j]);
    }
  }
}

// The full gradient in closed form for every instance (the single-field
// derivation: A, A^T and every D_j commute on the periodic grid, so
// dL/da_j = S <lam^1, D_j f0> with lam^1 = (A^T)^(S-1) lam_T): S - 1
// transposed steps, one contraction per instance with its field (still f0),
// the last transposed step, then the forward advect to f_T.
static int batch_adjoint_closed_form(fdb_batch* b, int S, const double* dt,
                                     const double* lambda_T, double* grad_f0, double* grad_v,
                                     int is_device, bool advance_fields) {
  const int n = b->count;
  if (!b->adj_dda) FDB_TRY(balloc(&b->adj_dda, 3 * (size_t)n));
  FDB_TRY(batch_lam_load(b, lambda_T, is_device));
  int lc = 0;
  FDB_TRY(batch_lam_steps(b, S - 1, dt, &lc));
  FDB_TRY(launch_vel_contract(n, b->geoms.data(), b->offsets.data(), b->arena[b->cur],
                              b->adj_lam[lc], b->adj_dda, b->contract, b->stream));
  FDB_TRY(batch_lam_steps(b, 1, dt, &lc));
  FDB_TRY(batch_lam_store(b, lc, grad_f0, is_device));
  if (advance_fields)
    FDB_TRY(run_batched(b, S, dt, effective_K(b), effective_shape(b), effective_tz(b)));
  std::vector<double> dda(3 * (size_t)n);
  FDB_CUDA_TRY(cudaMemcpyAsync(dda.data(), b->adj_dda, dda.size() * 8, cudaMemcpyDeviceToHost,
                               b->stream));
  FDB_TRY(bsync(b));
  b->contract.host.clear();
  for (double& x : dda) x *= (double)S;
  batch_velocity_grad(b, dt, dda.data(), grad_v);
  return FDB_OK;
}

// dL/df0 only (fdb_batch_adjoint with grad_v = NULL): the batch advances to
// f_T, then the transposed launch gives (A^T)^S lambda_T.
static int batch_adjoint_f0_only(fdb_batch* b, int S, const double* dt, const double* lambda_T,
                                 double* grad_f0, int is_device) {
  if (S > 0 && b->adj_mode != 2)  // form 2 keeps the fields at f0
    FDB_TRY(run_batched(b, S, dt, effective_K(b), effective_shape(b), effective_tz(b)));
  return batch_transposed(b, S, dt, lambda_T, grad_f0, is_device);
}

int fdb_batch_advect_transposed(fdb_batch* b, int num_steps, const double* dt, const double* in,
                                double* out, int is_device) {
  NvtxScope nvtx_("fdb.batch.advect_transposed");
  FDB_TRY(bcheck(b));
  if (num_steps < 0) return fail(FDB_ERR_INVALID, "num_steps must be >= 0");
  FDB_TRY(check_dts(b, dt));
  if (!in || !out) return fail(FDB_ERR_INVALID, "null input or output");
  return batch_transposed(b, num_steps, dt, in, out, is_device);
}

int fdb_batch_adjoint(fdb_batch* b, int num_steps, const double* dt, const double* lambda_T,
                      double* grad_f0, double* grad_v, int checkpoint_every, int is_device) {
  NvtxScope nvtx_("fdb.batch.adjoint");
  FDB_TRY(bcheck(b));
  if (num_steps < 0) return fail(FDB_ERR_INVALID, "num_steps must be >= 0");
  FDB_TRY(check_dts(b, dt));
  if (!lambda_T || !grad_f0) return fail(FDB_ERR_INVALID, "null lambda_T or grad_f0");
  if (checkpoint_every < 0) return fail(FDB_ERR_INVALID, "checkpoint_every must be >= 0");
  const int S = num_steps;
  int K = checkpoint_every;
  if (K == 0) K = std::max(1, (int)ceil(sqrt((double)std::max(S, 1))));
  if (K > std::max(S, 1)) K = std::max(S, 1);
  const int nseg = (S + K - 1) / K;
  const int n = b->count;
  if (!grad_v) return batch_adjoint_f0_only(b, S, dt, lambda_T, grad_f0, is_device);
  // every instance in the fixed kernel's domain (forward and transposed steps)
  std::vector<Coeffs3> cs(n);
  for (int i = 0; i < n; ++i) {
    cs[i] = coeffs3(b->geoms[i], dt[i]);
    if (fixed_supported(b->geoms[i], cs[i], 1) != FDB_OK ||
        fixed_supported(b->geoms[i], cs[i], effective_K(b)) != FDB_OK)
      return fail(FDB_ERR_UNSUPPORTED, "batched adjoint: instance " + std::to_string(i) +
                                           " is outside the fixed-point kernel's domain");
  }
  if (b->adj_mode != 1) {
    if (S == 0) {  // dL/df0 = lambda_T, dL/dv = 0
      uint64_t cells = 0;
      for (uint64_t z : b->sizes) cells += z;
      FDB_TRY(bsync(b));
      FDB_CUDA_TRY(cudaMemcpy(grad_f0, lambda_T, cells * 8,
                              is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToHost));
      for (int i = 0; i < 3 * n; ++i) grad_v[i] = 0.0;
      return FDB_OK;
    }
    NvtxScope nvtx_c("fdb.batch.adjoint.closed_form");
    return batch_adjoint_closed_form(b, S, dt, lambda_T, grad_f0, grad_v, is_device,
                                     b->adj_mode == 0);
  }
  // storage
  const size_t T = (size_t)b->total;
  const int nsegbuf = adjoint_fixed_segment_buffers(K);
  const int grid = batch_adjoint_grid(n, b->geoms.data());
  const size_t sb = batch_adjoint_scratch_bytes(n, K, grid);
  if ((int)b->adj_ckpt.size() < nseg || (int)b->adj_seg.size() < nsegbuf || !b->adj_lam[0] ||
      b->adj_scratch_bytes < sb) {
    free_batch_adjoint(b);
    b->adj_ckpt.assign(nseg, nullptr);
    b->adj_seg.assign(nsegbuf, nullptr);
    int rc = FDB_OK;
    for (auto& p : b->adj_ckpt)
      if (!rc) rc = balloc(&p, T);
    for (auto& p : b->adj_seg)
      if (!rc) rc = balloc(&p, T);
    for (auto& p : b->adj_lam)
      if (!rc) rc = balloc(&p, T);
    for (auto& p : b->adj_io)
      if (!rc) rc = balloc(&p, T);
    if (!rc) rc = balloc(&b->adj_user, T);
    if (!rc) rc = balloc(&b->adj_dda, 3 * (size_t)n);
    if (!rc) rc = balloc((char**)&b->adj_scratch, sb);
    if (rc) {
      free_batch_adjoint(b);
      return rc;
    }
    b->adj_scratch_bytes = sb;
  }
  const uint64_t cells = user_cells(b);
  // forward with checkpoints (the persistent launch): ckpt[s] = f^{sK}
  for (int sg = 0; sg < nseg; ++sg) {
    FDB_CUDA_TRY(cudaMemcpyAsync(b->adj_ckpt[sg], b->arena[b->cur], T * 8,
                                 cudaMemcpyDeviceToDevice, b->stream));
    const int len = std::min(K, S - sg * K);
    FDB_TRY(run_batched(b, len, dt, effective_K(b), effective_shape(b), effective_tz(b)));
  }
  // lambda_T into the stored layout
  const double* lt = lambda_T;
  if (!is_device) {
    FDB_CUDA_TRY(cudaMemcpyAsync(b->adj_user, lambda_T, cells * 8, cudaMemcpyHostToDevice,
                                 b->stream));
    lt = b->adj_user;
  }
  FDB_TRY(io_all(b, lt, b->adj_io[0], false));
  BatchAdjointIO io;
  std::vector<int32_t*> hi(K);
  for (int k = 0; k < K; ++k) hi[k] = (int32_t*)b->adj_seg[2 + k / 2] + (k & 1) * T;
  io.count = n;
  io.geoms = b->geoms.data();
  io.coeffs = cs.data();
  io.offsets = b->offsets.data();
  io.d_offs = b->d_offs;
  io.d_sizes = b->d_sizes;
  io.S = S;
  io.K = K;
  io.nseg = nseg;
  io.ckpt = b->adj_ckpt.data();
  io.chain[0] = (int64_t*)b->adj_seg[0];
  io.chain[1] = (int64_t*)b->adj_seg[1];
  io.state_hi = hi.data();
  io.lam[0] = (int64_t*)b->adj_lam[0];
  io.lam[1] = (int64_t*)b->adj_lam[1];
  io.lam_T = b->adj_io[0];
  io.grad_f0 = b->adj_io[1];
  io.dda3 = b->adj_dda;
  io.err = b->d_err;
  io.scratch = b->adj_scratch;
  FDB_TRY(batch_adjoint_run(io, b->stream));
  // dL/df0 back to the caller's order
  FDB_TRY(io_all(b, b->adj_io[1], is_device ? grad_f0 : b->adj_user, true));
  if (!is_device)
    FDB_CUDA_TRY(cudaMemcpyAsync(grad_f0, b->adj_user, cells * 8, cudaMemcpyDeviceToHost,
                                 b->stream));
  std::vector<double> dda(3 * (size_t)n);
  FDB_CUDA_TRY(cudaMemcpyAsync(dda.data(), b->adj_dda, dda.size() * 8, cudaMemcpyDeviceToHost,
                               b->stream));
  FDB_TRY(bsync(b));
  if (grad_v) batch_velocity_grad(b, dt, dda.data(), grad_v);
  return FDB_OK;
}

int fdb_batch_checksums(fdb_batch* b, double* out) {
  FDB_TRY(bcheck(b));
  if (!out) return fail(FDB_ERR_INVALID, "null output");
  k_batch_sum_partial<<<b->count * kSumPerInst, 256, 0, b->stream>>>(
      b->arena[b->cur], b->d_offs, b->d_sizes, b->count, kSumPerInst, b->d_part);
  k_batch_sum_final<<<(b->count + 127) / 128, 128, 0, b->stream>>>(b->d_part, b->count,
                                                                   kSumPerInst, b->d_sums);
  note_launch(2);
  FDB_CUDA_TRY(cudaGetLastError());
  FDB_CUDA_TRY(cudaMemcpyAsync(b->h_sums, b->d_sums, b->count * sizeof(double),
                               cudaMemcpyDeviceToHost, b->stream));
  FDB_TRY(bsync(b));
  memcpy(out, b->h_sums, b->count * sizeof(double));
  return FDB_OK;
}

// Small autotuner: times each compiled (depth, shape) of the batched kernel,
// and whole-z versus 32-plane tiles, on a copy of the current fields for
// `num_steps` steps; keeps the fastest.  With a cache path, results are
// stored per problem class (instance count, cell-count bucket, largest axis,
// GPU name) and reused without timing.
int fdb_batch_autotune(fdb_batch* b, int num_steps, const double* dt, const char* cache_path,
                       int* chosen) {
  FDB_TRY(bcheck(b));
  FDB_TRY(check_dts(b, dt));
  if (num_steps <= 0) return fail(FDB_ERR_INVALID, "num_steps must be > 0");
  uint64_t cells = 0;
  uint64_t maxn = 0;
  for (const Geom& g : b->geoms) {
    cells += g.ntot;
    maxn = std::max<uint64_t>(maxn, std::max<uint64_t>(g.nx, std::max<uint64_t>(g.ny, g.nz)));
  }
  int dev = 0;
  cudaDeviceProp prop;
  FDB_CUDA_TRY(cudaGetDevice(&dev));
  FDB_CUDA_TRY(cudaGetDeviceProperties(&prop, dev));
  std::ostringstream cls;
  cls << "count=" << b->count << ";cells_log2=" << (int)floor(log2((double)std::max<uint64_t>(cells, 1)))
      << ";maxn=" << maxn << ";steps=" << num_steps << ";gpu=" << prop.name;
  std::string key = cls.str();
  for (char& ch : key)
    if (ch == ' ') ch = '_';
  if (cache_path && *cache_path) {
    std::ifstream in(cache_path);
    std::string line;
    while (std::getline(in, line)) {
      std::istringstream ls(line);
      std::string k;
      int K, sh, tz;
      if (ls >> k >> K >> sh >> tz && k == key &&
          (sh == -1 ? (K >= 2 && K <= 4) : find_variant(K, sh, false) != nullptr)) {
        b->K = K;
        b->shape = sh;
        b->tz = tz;
        choose_tuning(b);
        drop_plans(b);
        if (chosen) {
          chosen[0] = K;
          chosen[1] = sh;
          chosen[2] = tz;
        }
        return FDB_OK;
      }
    }
  }
  // time candidates on a copy: the fields are restored afterwards
  double* save = nullptr;
  FDB_TRY(balloc(&save, b->total));
  FDB_CUDA_TRY(cudaMemcpyAsync(save, b->arena[b->cur], b->total * 8, cudaMemcpyDeviceToDevice,
                               b->stream));
  const int cur0 = b->cur;
  EventPool events;
  cudaEvent_t e0 = events.make(), e1 = events.make();
  if (!e0 || !e1) {
    cudaFree(save);
    return fail(FDB_ERR_CUDA, "autotune: cudaEventCreate failed");
  }
  // {depth, shape, tile_z} as run, and as kept: the automatic choice (its depth,
  // the rest automatic), then every compiled form that can be asked for, in
  // whole columns and in ranges of 32 planes
  struct Try {
    int K, shape, tz, keep_shape, keep_tz;
  };
  const int set[3] = {b->K, b->shape, b->tz};
  b->K = 0;
  b->shape = -1;
  b->tz = 0;
  choose_tuning(b);
  std::vector<Try> tries = {{b->eff_K, b->eff_shape, b->eff_tz, -1, 0}};
  b->K = set[0];
  b->shape = set[1];
  b->tz = set[2];
  choose_tuning(b);
  const int whole = (int)std::min<uint64_t>(maxn, 1u << 30);
  for (const Variant& v : kVariants)
    if (v.shape < fx::kNumShapes && !v.wide)
      for (int tz : {whole, 32}) tries.push_back({v.K, v.shape, tz, v.shape, tz});
  float best = 1e30f;
  Try kept = tries[0];
  int rc = FDB_OK;
  for (const Try& t : tries) {
    for (int rep = 0; rep < 2 && !rc; ++rep) {  // rep 0 warms up and makes the plan
      b->cur = cur0;
      cudaMemcpyAsync(b->arena[cur0], save, b->total * 8, cudaMemcpyDeviceToDevice, b->stream);
      cudaEventRecord(e0, b->stream);
      rc = run_batched(b, num_steps, dt, t.K, t.shape, t.tz);
      cudaEventRecord(e1, b->stream);
      if (rc == FDB_ERR_UNSUPPORTED) {
        rc = FDB_OK;
        break;
      }
      if (!rc) rc = bsync(b);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (!rc && rep == 1 && ms < best) {
        best = ms;
        kept = t;
      }
    }
  }
  b->cur = cur0;
  cudaMemcpyAsync(b->arena[cur0], save, b->total * 8, cudaMemcpyDeviceToDevice, b->stream);
  cudaStreamSynchronize(b->stream);
  cudaFree(save);
  if (rc) return rc;
  b->K = kept.K;
  b->shape = kept.keep_shape;
  b->tz = kept.keep_tz;
  choose_tuning(b);
  drop_plans(b);
  if (chosen) {
    chosen[0] = b->K;
    chosen[1] = b->shape;
    chosen[2] = b->tz;
  }
  if (cache_path && *cache_path) {
    std::ofstream o(cache_path, std::ios::app);
    o << key << ' ' << b->K << ' ' << b->shape << ' ' << b->tz << '\n';
  }
  return FDB_OK;
}

}  // extern "C"
