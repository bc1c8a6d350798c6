// step_fixed.cu -- temporally blocked upwind kernel in 64-bit block-fixed-point.
//
// One launch advances the field by K steps (K = 1..4).  Within one advect()
// call the field stays in fixed point in HBM between launches: the first
// launch reads FP64 and converts f -> F = round(f * 2^s), the inner launches
// read and write int64 F (8 B, like FP64), and the last launch converts back
// and writes FP64.  Each launch streams every cell once: 16 B of HBM traffic
// per cell per K steps.  The arithmetic runs on the integer pipes
// (IMAD/IADD3/LOP3/SHFL); GB300 retires only ~2 FP64 operations per clock
// per SM, which would cap a native FP64 step near 150 GCUPS.
//
// Precision.  The scale keeps |F| < 2^(59-g) at a launch's input (g guard
// bits cover the step's max-norm growth G^K), so one unit of F is at most
// 2^-(58-g) of max|f|.  One step adds at most 2 units of rounding per cell (8
// units in all on the last one) and 2.25 of the coefficients' remainder
// (fixed_point.cuh), so after 100 steps the field is within ~1e-15 of the
// reference's FP64 arithmetic relative to max|f| (the bar is 1e-13).  Cells below
// one unit are held as 0, an absolute error below the same bound.
//
// Update.  F' = F + sum_j a_j (F_up_j - F) with a_j in [0, 1] held in Q1.62
// (A = a1 2^32 + a0, a0 balanced to [-2^31, 2^31)).  For D = d1 2^32 + d0:
//   A D / 2^64 = a1 d1 + (a1 d0 + a0 d1) 2^-32 + a0 d0 2^-64
// the a1 d1 products are summed exactly; the six a1 d0 and a0 d1 partial
// products of the three axes are summed exactly in one offset unsigned
// 64-bit word whose high word is taken (one rounding to nearest);
// F' = F + 4 * sum (fixed_point.cuh fixed_update).  The rounding is unbiased
// and a zero difference contributes exactly zero.  All steps of an advect but
// the last take a_j as a1 alone, the coefficient error of one step carried to
// the next and settled by the last one (fixed_point.cuh), so that six products
// remain (fixed_update6).  The products bound the kernel: a 32 x 32 -> 64-bit
// multiply holds the FMA-heavy integer pipe for four cycles per warp.
// Measured against nine products on every step: set_field, advect(100) and
// get_field at 512^3 30.75 -> 25.31 ms; 64 fields of 128^3, forward and
// transposed, 77.0 -> 63.8 ms.
//
// Geometry.  Axes are relabelled so that every upstream neighbour is at -1
// (axis j reversed when v_j < 0, upwind.cxx:34-35).  A CTA of W warps owns an
// output tile of (32-K) x (R*W-K) cells in (x, y) and marches along z over tz
// output planes after K warm-up planes.  Lanes are consecutive x (coalesced
// 256 B row accesses), each thread holds R consecutive y rows of one column
// in registers (R x W = 8x4 for all but small or thin grids, see
// auto_config).  Per level: x-1 from lane-1 (its history slot, or SHFL), y-1
// from the thread's previous row (row 0 from the warp above through shared
// memory, one __syncthreads per level), z-1 from the thread's K-deep history
// of the previous plane.  The next plane is loaded into registers (or, in the
// older shapes, with cp.async into shared memory) while the current one is
// computed.  The upstream halo (K columns, K rows, K planes) is the only
// redundant work; periodic wrap is applied to the coordinates of the loaded
// rows and planes.
//
// Scale protocol (no host synchronisation).  Three device slots hold
// {m, s, kind}: kind 0 = m is the FP64 bit pattern of max|f| (from the
// pre-pass), kind 1 = m is an OR of |F| over the field held at scale s.
// Launch i reads slot i%3, ORs its output into slot (i+1)%3 (block 0 also
// writes s and kind there) and clears slot (i+2)%3 for launch i+1.
#include <math.h>

#include "step_fixed.cuh"

namespace fdb {

using fx::FixedArgs;
using fx::ScaleSlot;

double growth_bound(const Coeffs3& c) { return fabs(c.w) + c.az + c.ay + c.ax; }

int guard_bits(const Coeffs3& c, int K) {
  const double G = growth_bound(c);
  if (G <= 1.0) return 0;
  return (int)ceil(K * log2(G)) + 1;
}

namespace {

using fx::kMaxDepth;

// max|f| as the bit pattern of |f| (monotone for non-negative doubles; NaN
// and Inf patterns exceed every finite one) -> slot {m, kind 0}.
__global__ void __launch_bounds__(256)
k_absmax_bits(const double* f, uint64_t n, ScaleSlot* slot) {
  __shared__ unsigned long long sh[8];
  unsigned long long m = 0ull;
  cudaGridDependencySynchronize();
  auto take = [&](double x) {
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
    m = b > m ? b : m;
  };
  const uint64_t step = (uint64_t)gridDim.x * 256ull;
  uint64_t i = blockIdx.x * 256ull + threadIdx.x;
  for (; i + 3 * step < n; i += 4 * step) {  // four loads in flight
    const double x0 = f[i], x1 = f[i + step], x2 = f[i + 2 * step], x3 = f[i + 3 * step];
    take(x0);
    take(x1);
    take(x2);
    take(x3);
  }
  for (; i < n; i += step) take(f[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
    m = v > m ? v : m;
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = sh[w] > m ? sh[w] : m;
    atomicMax(&slot->m, m);
  }
}

__global__ void k_slots_init(ScaleSlot* slots) {
  if (threadIdx.x < 3) {
    slots[threadIdx.x].m = 0ull;
    slots[threadIdx.x].s = 0;
    slots[threadIdx.x].kind = threadIdx.x == 0 ? 0 : 1;
  }
}


}  // namespace

// Tiling and coefficients of one field for the fixed kernel (slot pointers
// are left null).  tz_override > 0 fixes the output planes per CTA.
fx::FixedArgs make_fixed_args(const Geom& g, const Coeffs3& c, int shape, int K, int tz_override,
                              int64_t resident_ctas) {
  const int R = fx::shape_rows(shape), W = fx::shape_warps(shape);
  FixedArgs a{};
  a.nz = (int)g.nz;
  a.ny = (int)g.ny;
  a.nx = (int)g.nx;
  a.fz = g.upz > 0;
  a.fy = g.upy > 0;
  a.fx = g.upx > 0;
  a.tx = 32 - K;
  a.ty = R * W - K;
  a.tiles_x = (a.nx + a.tx - 1) / a.tx;
  a.tiles_y = (a.ny + a.ty - 1) / a.ty;
  const int64_t txy = (int64_t)a.tiles_x * a.tiles_y;
  int tz = tz_override;
  if (tz <= 0) {
    // about four waves of the resident CTAs
    const int64_t want = 4 * resident_ctas;
    int64_t cz = (want + txy - 1) / txy;
    if (cz < 1) cz = 1;
    tz = (int)((a.nz + cz - 1) / cz);
    if (tz < 4 * K) tz = 4 * K;
  }
  if (tz > a.nz) tz = a.nz;
  a.tz = tz;
  a.tiles_z = (a.nz + tz - 1) / tz;
  a.qz = make_qcoeff(c.az);
  a.qy = make_qcoeff(c.ay);
  a.qx = make_qcoeff(c.ax);
  a.guard = guard_bits(c, K);
  // the planes whose outputs set the next scale: the geometry's own planes
  // of the internal z axis (all of them unless a slab names its own)
  a.or_z0 = 0;
  a.or_z1 = a.nz;
  if (g.own_n > 0 && g.jz == 0) {
    const int p0 = (int)g.own0, p1 = (int)(g.own0 + g.own_n);  // physical
    a.or_z0 = a.fz ? a.nz - p1 : p0;
    a.or_z1 = a.fz ? a.nz - p0 : p1;
  }
  return a;
}

namespace fx {

long long plan_slabs(FixedArgs& a, int sms, int per_sm, int cap) {
  const long long txy = (long long)a.tiles_x * a.tiles_y;
  const int nz = a.nz;
  if (txy <= 0 || nz <= 0) {
    a.nslab = 0;
    return 0;
  }
  const long long n_sm = sms > 0 ? sms : 1;
  const long long res = n_sm * (per_sm > 0 ? per_sm : 1);
  const long long fill = (txy * nz + 2 * n_sm - 1) / (2 * n_sm);  // planes of two CTAs per SM
  const int min_planes = fill < 3 ? 3 : (fill > 8 ? 8 : (int)fill);
  int z = 0, i = 0;
  const long long per_tile = res / txy;  // slabs the GPU holds at once
  if (cap <= 0 && per_tile >= 9 && nz >= 8 * per_tile && per_tile <= kMaxSlabs) {
    for (; i < per_tile; ++i) a.slab_z[i] = (int)((long long)nz * i / per_tile);
    z = nz;
  }
  while (z < nz) {
    const int rem = nz - z;
    const int left = kMaxSlabs - i;
    long long h = (txy * rem + res - 1) / res;  // remaining planes per resident CTA
    if (cap > 0 && h > cap) h = cap;
    if (h < min_planes && (cap <= 0 || cap >= min_planes)) h = min_planes;
    if (h * left < rem) h = (rem + left - 1) / left;
    if (h > rem) h = rem;
    a.slab_z[i++] = z;
    z += (int)h;
  }
  a.slab_z[i] = nz;
  a.nslab = i;
  return txy * i;
}

}  // namespace fx

int launch_fixed_one(const Geom& g, const Coeffs3& c, int shape, int K, const void* in, void* out,
                     bool in_f64, bool out_f64, ScaleSlot* slots, int i, int* err,
                     int tz_override, int guard_K, int* scale_log, CoeffCarry* carry,
                     cudaStream_t st, int32_t* const* gout) {
  if (gout && (shape != fx::kR4W8S || in_f64 || out_f64 || K < 1 || K > 4))
    return fail(FDB_ERR_UNSUPPORTED, "level output needs the default shape and int64 in/out");
  // 8 x 152 resident 256-thread CTAs, scaled to this shape's CTA size
  FixedArgs a = make_fixed_args(g, c, shape, K, tz_override,
                                (int64_t)2 * 152 * 256 / (32 * fx::shape_warps(shape)));
  // guard bits sized for the call's full depth, also on a shorter final
  // launch, so that every launch of a call uses the same headroom rule as the
  // batched kernel (which sizes them once per instance)
  a.guard = guard_bits(c, guard_K);
  a.slot_in = slots + (i % 3);
  a.slot_out = slots + ((i + 1) % 3);
  a.slot_reset = slots + ((i + 2) % 3);
  a.err = err;
  a.scale_log = scale_log;
  const QCoeff q[3] = {a.qz, a.qy, a.qx};
  for (int t = 0; t < K; ++t)
    for (int j = 0; j < 3; ++j)
      a.lev.q[t][j] =
          gout ? q[j] : step_qcoeff_carry(q[j], &carry->r[j], out_f64 && t == K - 1);
  // the grid is at most tiles_x * tiles_y CTAs for each of min(nz, kMaxSlabs) slabs
  if ((int64_t)a.tiles_x * a.tiles_y * (a.nz < fx::kMaxSlabs ? a.nz : fx::kMaxSlabs) > 0x7FFFFFFF)
    return fail(FDB_ERR_UNSUPPORTED, "grid too large for the fixed kernel");
  const int64_t* pin = (const int64_t*)in;
  int64_t* pout = (int64_t*)out;
  const int cap = tz_override > 0 ? tz_override : 0;
  if (gout) {
    for (int t = 0; t < K; ++t) a.gout[t] = gout[t];
    fx::launch_r4w8s_store_g(K, cap, pin, pout, a, st);
    note_launch();
    FDB_CUDA_TRY(cudaGetLastError());
    return FDB_OK;
  }
  switch (shape) {
    case fx::kR4W16: fx::launch_r4w16(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR8W8S: fx::launch_r8w8s(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR4W16S: fx::launch_r4w16s(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR4W8S: fx::launch_r4w8s(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR4W8L: fx::launch_r4w8l(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR6W8L: fx::launch_r6w8l(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR8W4L: fx::launch_r8w4l(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR6W4L: fx::launch_r6w4l(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    case fx::kR4W4L: fx::launch_r4w4l(K, in_f64, out_f64, cap, pin, pout, a, st); break;
    default: fx::launch_r8w8(K, in_f64, out_f64, cap, pin, pout, a, st); break;
  }
  note_launch();
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

namespace {

// The launch the automatic choice takes for g (depth K given, or 0: any).
//
// Shapes: 4 warps (one per SM sub-partition) of 8, 6 or 4 rows, the plane
// history in shared memory.  Few warps with many rows win: a level's barrier
// waits for 4 warps instead of 8, and 8 independent rows per thread hide the
// latency of the products better than more warps do.  Measured (inner launch,
// K = 3, GCUPS, 8x4 / 6x8 / 4x8 / 8x8): 512^3 610 / 572 / 547 / 571; 256^3
// 502 / 482 / 464 / 440.
//
// A launch of K steps costs the computed tiles (32 columns x R W rows, of which
// 32 - K and R W - K are output) times K levels plus the per-plane work (load,
// scale, store), 0.86 levels, per step: minimal
//   ceil(nx / (32 - K)) ceil(ny / (R W - K)) R W (1 + 0.86 / K) f(R)
// with f the measured cost of a computed row against 8 rows per thread.  It
// picks the winners of a sweep over 64^3 .. 512^3 and uneven grids, or within
// 7 % of them (winner's K: 4 at 128, 192, 384, 448; 3 at 256, 288, 512).
// Grids whose 8-row tiles give less than half a wave of CTAs (8 planes each)
// are bound by the latency of a CTA's march: 4 rows (more CTAs) and K = 4
// (64^3: 94 against 85 GCUPS for 8 rows).
struct Config {
  int K, shape;
};
Config auto_config(const Geom& g, int K_asked) {
  struct Cand {
    int shape;
    double f;
  };
  static const Cand cands[] = {{fx::kR8W4L, 1.0}, {fx::kR6W4L, 1.02}, {fx::kR4W4L, 1.1}};
  const int K_hi = K_asked > 0 ? K_asked : kMaxDepth;
  const int K_lo = K_asked > 0 ? K_asked : 2;
  const auto tiles = [&](int K, int rows) {
    return std::ceil((double)g.nx / (32 - K)) * std::ceil((double)g.ny / (rows - K));
  };
  constexpr double kHalfWave = 152 * 4 / 2;  // CTAs
  // planes of 4 GB and more: beyond the 4-warp shapes' 32-bit offsets
  if ((uint64_t)g.ny * g.nx >= (1ull << 29))
    return {K_asked > 0 ? K_asked : 3, fx::kR6W8L};
  if (tiles(K_hi, 32) * std::ceil(g.nz / 8.0) < kHalfWave) return {K_hi, fx::kR4W4L};
  Config best{K_hi, fx::kR8W4L};
  double best_cost = 0.0;
  for (int K = K_hi; K >= K_lo; --K) {
    for (const Cand& c : cands) {
      const int rows = fx::shape_rows(c.shape) * fx::shape_warps(c.shape);
      const double cost = tiles(K, rows) * rows * (1.0 + 0.86 / K) * c.f;
      if (best_cost == 0.0 || cost < best_cost) {
        best_cost = cost;
        best = {K, c.shape};
      }
    }
  }
  return best;
}

// The shape of a launch of k <= K steps in an advect of depth K.  One step per
// launch is conversion work for the most part, with few chains to overlap:
// 4 rows at 6 CTAs per SM (advect(1) at 256^3, FP64 in and out: 194 GCUPS
// against 175 for 8 rows).
int default_shape(const Geom& g, int K, int k) {
  const int shape = auto_config(g, K).shape;
  return k == 1 && shape != fx::kR6W8L ? (int)fx::kR4W4L : shape;
}

}  // namespace

int default_depth(const Geom& g) { return auto_config(g, 0).K; }

int fixed_supported(const Geom& g, const Coeffs3& c, int depth) {
  if (g.ndims > 3) return fail(FDB_ERR_UNSUPPORTED, "fixed kernel serves ndims <= 3");
  const int K = depth > 0 ? depth : default_depth(g);
  if (K > kMaxDepth) return fail(FDB_ERR_UNSUPPORTED, "fixed kernel temporal depth must be <= 4");
  const double as[3] = {c.az, c.ay, c.ax};
  for (double x : as)
    if (!(x >= 0.0 && x <= 1.0))
      return fail(FDB_ERR_UNSUPPORTED, "fixed kernel needs Courant numbers a_j in [0, 1]");
  if (guard_bits(c, K) > 16)
    return fail(FDB_ERR_UNSUPPORTED, "step growth too large for the fixed kernel's headroom");
  if (g.nx >= (1 << 30) || g.ny >= (1 << 30) || g.nz >= (1 << 30) ||
      g.nx * g.ny >= ((int64_t)1 << 31))
    return fail(FDB_ERR_UNSUPPORTED, "fixed kernel needs ny*nx < 2^31");
  return FDB_OK;
}

bool fixed_preferred(const Geom& g) {
  // tiles are (32-K) x (R*W-K) cells in (x, y); small grids are cheaper in FP64
  return g.ndims <= 3 && g.nx >= 16 && g.ny >= 16 && g.nz >= 8 && g.ntot >= (1u << 18);
}

int fx_num_shapes() { return fx::kNumShapes; }

size_t fixed_scratch_bytes() { return 3 * sizeof(ScaleSlot) + 4 * sizeof(int); }

int* fixed_error_word(double* d_scratch) { return (int*)((ScaleSlot*)d_scratch + 3); }

int launch_scale_prepass(const Geom& g, const double* f, double* d_scratch, cudaStream_t s) {
  ScaleSlot* slots = (ScaleSlot*)d_scratch;
  // max|f| over the geometry's own planes of axis 0 (all planes unless a
  // slab names its own: its halo planes hold other ranks' values)
  uint64_t first = 0, count = g.ntot;
  if (g.own_n > 0) {
    const uint64_t plane = g.ntot / g.n[0];
    first = g.own0 * plane;
    count = g.own_n * plane;
  }
  k_slots_init<<<1, 32, 0, s>>>(slots);
  uint64_t blocks = (count + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  if (blocks < 1) blocks = 1;
  FDB_CUDA_TRY(launch_dependent(k_absmax_bits, (unsigned)blocks, 256, 0, s, f + first, count, slots));
  note_launch(2);
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

int launch_fixed_block(const Geom& g, const Coeffs3& c, int k, const FixedTuning& tune,
                       int guard_K, double** buf, int* cur, bool in_f64, bool out_f64,
                       double* d_scratch, int i, CoeffCarry* carry, cudaStream_t s) {
  if (fault_injected("launch")) return fail(FDB_ERR_INJECTED, "injected launch failure");
  const int shape = (tune.shape >= 0 && tune.shape < fx::kNumShapes)
                        ? tune.shape
                        : default_shape(g, guard_K, k);
  FDB_TRY(launch_fixed_one(g, c, shape, k, buf[*cur], buf[*cur ^ 1], in_f64, out_f64,
                           (ScaleSlot*)d_scratch, i, fixed_error_word(d_scratch), tune.tz, guard_K,
                           nullptr, carry, s));
  *cur ^= 1;
  return FDB_OK;
}

uint64_t* scale_word(double* d_scratch, int i) {
  return reinterpret_cast<uint64_t*>(&((ScaleSlot*)d_scratch + (i % 3))->m);
}

int launch_advect_fixed_ex(const Geom& g, const Coeffs3& c, int steps, const FixedTuning& tune,
                           double** buf, int* cur, double* d_scratch, size_t scratch_bytes,
                           int* scale_slot, cudaStream_t s) {
  if (fault_injected("launch")) return fail(FDB_ERR_INJECTED, "injected launch failure");
  if (scratch_bytes < fixed_scratch_bytes() || !d_scratch)
    return fail(FDB_ERR_INVALID, "fixed kernel scratch missing");
  if (steps <= 0) return FDB_OK;
  ScaleSlot* slots = (ScaleSlot*)d_scratch;
  int* err = fixed_error_word(d_scratch);
  const int K = tune.depth > 0 ? tune.depth : default_depth(g);
  const bool shape_set = tune.shape >= 0 && tune.shape < fx::kNumShapes;
  int i0 = (scale_slot && *scale_slot >= 0) ? *scale_slot : -1;
  if (i0 < 0) {
    FDB_TRY(launch_scale_prepass(g, buf[*cur], d_scratch, s));
    i0 = 0;
  }
  const int nlaunch = (steps + K - 1) / K;
  int i = i0;
  CoeffCarry carry;
  for (int l = 0, done = 0; l < nlaunch; ++l, ++i) {
    const int k = (steps - done) < K ? (steps - done) : K;
    const int shape = shape_set ? tune.shape : default_shape(g, K, k);
    FDB_TRY(launch_fixed_one(g, c, shape, k, buf[*cur], buf[*cur ^ 1], l == 0, l == nlaunch - 1,
                             slots, i, err, tune.tz, K, nullptr, &carry, s));
    *cur ^= 1;
    done += k;
  }
  if (scale_slot) *scale_slot = i % 3;
  return FDB_OK;
}

}  // namespace fdb
