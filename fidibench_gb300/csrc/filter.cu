// filter.cu -- the constant-coefficient stencil Filter (include/fdb_filter.h),
// the GPU form of the reference's cxx/Filter.cpp on one process.
//
// out[i] = sum over the terms (std::map order of the offsets) of
// w_t * in[neighbour_t(i)], each product and each sum separately rounded and
// accumulated from +0 as in Filter.cpp:192-260, so the output is
// bit-identical to the reference.  The first term replaces `0 + p` by p with
// -0 turned into +0 (the only case in which the sum differs from p).
//
// GB300's FP64 pipe bounds the kernel, so it spends as few of its cycles as the
// bits allow: additions and products are three-register DFMAs (f64_regs.cuh),
// and a weight of +-2^k (k >= 0, among them 1, -1 and the 2-D Laplacian's -4)
// goes with its addition into one DFMA: w x is exact unless it overflows, which
// the operand's exponent tells, so that one rounding is the sum's.  Threads
// take every T-th cell, an equal share for every SM.  Per apply, against DADD
// and DMUL one cell per thread: 2-D Laplacian 8000^2 (4 operations instead of
// 5) 0.87 -> 0.44 ms; 3-D Laplacian of 12.5 M cells (7) 0.24 -> 0.16 ms; the
// pipe's own time is 0.43 and 0.15 ms.
//
// Layout: column-major like the reference (axis 0 fastest).  Up to 3 axes use
// k_filter3; cells whose every neighbour is inside the grid use precomputed
// linear offsets, the others wrap each axis (FDB_WRAP_REFERENCE reproduces the
// reference's `%= size_t` of a negative int, see fdb_filter.h).  More axes
// use a generic kernel that decodes every index.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "f64_regs.cuh"
#include "fdb_filter.h"
#include "fdb_internal.h"

namespace {

constexpr int kMaxFastTerms = 32;
constexpr int kMaxTerms = 256;

struct FTerm {
  long long lin;
  double w;
  int o[3];
  // w = +-2^k, k >= 0: the high word from which |x| on w x overflows
  // (0x7FF00000 - k 2^20); any other weight: 0
  unsigned fuse;
};

struct FArgs3 {
  int n[3], step[3];  // extents; the grid stride's digit on each axis
  long long r[3];     // 2^64 mod n (reference wrap) or 0 (periodic)
  int lo[3], hi[3];   // neighbours stay inside for i in [lo, n - hi)
  long long ntot;
  int nterms;
  FTerm t[kMaxFastTerms];
};

// (2^64 + v) mod n for v < 0 (reference) or the periodic wrap (r = 0), and v
// mod n for v >= 0
__device__ __forceinline__ long long wrap_axis(long long v, long long n, long long r) {
  long long u = v >= 0 ? v : v + r;
  if (u < 0) u += n;
  else if (u >= n) u -= n;
  if (u >= 0 && u < n) return u;  // offsets up to an extent
  u %= n;
  return u < 0 ? u + n : u;
}

// first term: 0 + p, i.e. p with -0 -> +0
__device__ __forceinline__ double first_sum(double p) {
  const int hi = __double2hiint(p), lo = __double2loint(p);
  return __hiloint2double(hi == (int)0x80000000u && lo == 0 ? 0 : hi, lo);
}

__device__ __forceinline__ double negate(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
}

// acc + round(w v), as a call: inlined, the two operations would be predicated,
// and a predicated FP64 instruction holds the pipe whether it writes or not.
__device__ __noinline__ double add_product(double acc, double w, double v, double one,
                                           double minus_zero) {
  return __fma_rn(__fma_rn(w, v, minus_zero), one, acc);
}

constexpr int kFThreads = 256;

// NT > 0: a stencil of exactly NT terms, unrolled: the loads of all terms in
// flight at once, weights in registers, offsets from the kernel's arguments.
// NT = 0: any number, one term after the other.  CENTRE: the middle term's
// weight needs its product (a Laplacian's -6; star stencils have their centre
// there in the map order), the others do not.
template <int NT, bool CENTRE>
__global__ void __launch_bounds__(kFThreads, 4)
k_filter3(const double* in, double* __restrict__ out, const FArgs3 a) {
  __shared__ double s_slots[kFThreads];
  const fdb::RegLoader reg(s_slots);
  const fdb::F64Regs f64(reg);
  double wr[NT > 0 ? NT : 1];
#pragma unroll
  for (int k = 0; k < NT; ++k) wr[k] = reg(a.t[k].w);
  cudaGridDependencySynchronize();  // the launch before has written `in` and read `out`
  const int nterms = NT > 0 ? NT : a.nterms;
  const long long stride = (long long)gridDim.x * kFThreads;
  long long i = (long long)blockIdx.x * kFThreads + threadIdx.x;
  const unsigned n0 = a.n[0], n1 = a.n[1];
  const unsigned long long row = (unsigned long long)i / n0;
  unsigned x = (unsigned)((unsigned long long)i % n0);
  unsigned y = (unsigned)(row % n1), z = (unsigned)(row / n1);

  auto first = [&](double w, unsigned fuse, double v) {
    if (fuse == 0x7FF00000u)  // w = +-1: v with w's sign, on the integer side
      return first_sum(__hiloint2double(
          __double2hiint(v) ^ (__double2hiint(w) & (int)0x80000000u), __double2loint(v)));
    return first_sum(add_product(f64.minus_zero, w, v, f64.one, f64.minus_zero));
  };
  auto add = [&](double acc, double w, unsigned fuse, double v) {
    const unsigned mag = (unsigned)__double2hiint(v) & 0x7FFFFFFFu;
    // fused: w v is exact (or infinite or NaN with v)
    if (fuse != 0u && (mag < fuse || mag >= 0x7FF00000u)) return __fma_rn(w, v, acc);
    return add_product(acc, w, v, f64.one, f64.minus_zero);
  };
  for (; i < a.ntot; i += stride) {
    const bool inside = (int)x >= a.lo[0] && (int)x < a.n[0] - a.hi[0] && (int)y >= a.lo[1] &&
                        (int)y < a.n[1] - a.hi[1] && (int)z >= a.lo[2] && (int)z < a.n[2] - a.hi[2];
    auto wrapped = [&](const FTerm& t) -> long long {
      const long long jx = wrap_axis((long long)x + t.o[0], a.n[0], a.r[0]);
      const long long jy = wrap_axis((long long)y + t.o[1], a.n[1], a.r[1]);
      const long long jz = wrap_axis((long long)z + t.o[2], a.n[2], a.r[2]);
      return jx + a.n[0] * (jy + a.n[1] * jz);
    };
    double acc;
    if (NT > 0) {
      double v[NT > 0 ? NT : 1];
      if (inside) {
#pragma unroll
        for (int k = 0; k < NT; ++k) v[k] = in[i + a.t[k].lin];
      } else {
#pragma unroll
        for (int k = 0; k < NT; ++k) v[k] = in[wrapped(a.t[k])];
      }
      acc = first(wr[0], a.t[0].fuse, v[0]);
#pragma unroll
      for (int k = 1; k < NT; ++k) {
        if (CENTRE && k == NT / 2)
          acc = f64.add(acc, f64.mul(wr[k], v[k]));
        else
          acc = add(acc, wr[k], a.t[k].fuse, v[k]);
      }
    } else {
      auto load = [&](int k) { return in[inside ? i + a.t[k].lin : wrapped(a.t[k])]; };
      acc = first(a.t[0].w, a.t[0].fuse, load(0));
      for (int k = 1; k < nterms; ++k) acc = add(acc, a.t[k].w, a.t[k].fuse, load(k));
    }
    out[i] = acc;
    x += a.step[0];
    unsigned carry = x >= n0;
    if (carry) x -= n0;
    y += a.step[1] + carry;
    carry = y >= n1;
    if (carry) y -= n1;
    z += a.step[2] + carry;
  }
}

struct FArgsN {
  int ndims;
  int nterms;
  unsigned long long n[FDB_MAX_DIMS];
  unsigned long long prod[FDB_MAX_DIMS];
  long long r[FDB_MAX_DIMS];
  unsigned long long ntot;
};

// generic: any number of axes, terms in global memory (offsets [t][ndims])
__global__ void __launch_bounds__(256)
k_filter_nd(const double* __restrict__ in, double* __restrict__ out, const FArgsN a,
            const int* __restrict__ offs, const double* __restrict__ w) {
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < a.ntot;
       i += (unsigned long long)gridDim.x * 256ull) {
    double acc = 0.0;
    for (int k = 0; k < a.nterms; ++k) {
      unsigned long long j = 0;
      for (int d = 0; d < a.ndims; ++d) {
        const long long ind = (long long)(i / a.prod[d] % a.n[d]);
        j += a.prod[d] *
             (unsigned long long)wrap_axis(ind + offs[k * a.ndims + d], (long long)a.n[d], a.r[d]);
      }
      // w = +-1 skips the product (x * +-1 exactly)
      const double v = __ldg(in + j);
      const double p = w[k] == 1.0 ? v : w[k] == -1.0 ? negate(v) : __dmul_rn(w[k], v);
      acc = (k == 0) ? first_sum(p) : __dadd_rn(acc, p);
    }
    out[i] = acc;
  }
}

}  // namespace

struct fdb_filter {
  int ndims = 0;
  uint64_t n[FDB_MAX_DIMS] = {0};
  double xmins[FDB_MAX_DIMS] = {0};
  double xmaxs[FDB_MAX_DIMS] = {0};
  uint64_t ntot = 0;
  std::vector<int> offs;  // [nterms][ndims], map order
  std::vector<double> w;
  int wrap = FDB_WRAP_REFERENCE;
  double* buf[2] = {nullptr, nullptr};  // in = buf[cur], out = buf[cur ^ 1]
  int cur = 0;
  double* part = nullptr;
  double* dsum = nullptr;
  double* hsum = nullptr;
  int* d_offs = nullptr;
  double* d_w = nullptr;
  cudaStream_t own = nullptr;
  cudaStream_t stream = nullptr;
};

namespace {

using fdb::fail;

int falloc(void** p, size_t bytes) {
  if (fdb::fault_injected("alloc")) return fail(FDB_ERR_INJECTED, "injected allocation failure");
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return fail(FDB_ERR_ALLOC, std::string("cudaMalloc of ") + std::to_string(bytes) +
                                   " bytes failed: " + cudaGetErrorString(e));
  }
  return FDB_OK;
}

int check(fdb_filter* f) { return f ? FDB_OK : fail(FDB_ERR_INVALID, "null filter handle"); }

bool lex_less(const int* a, const int* b, int nd) {
  return std::lexicographical_compare(a, a + nd, b, b + nd);
}

// 2^64 mod n
long long pow2_64_mod(uint64_t n) { return (long long)((~0ull % n + 1) % n); }

int launch_apply(fdb_filter* f) {
  if (fdb::fault_injected("launch")) return fail(FDB_ERR_INJECTED, "injected launch failure");
  const double* in = f->buf[f->cur];
  double* out = f->buf[f->cur ^ 1];
  const int nt = (int)f->w.size();
  if (f->ndims <= 3 && nt <= kMaxFastTerms) {
    FArgs3 a{};
    // 8 CTAs per SM, the same number of cells for each: two even waves of 4 (60 to 64
    // registers with 3 to 7 terms).  Fewer for grids with less than a cell per thread.
    long long blocks = std::min<long long>(((long long)f->ntot + kFThreads - 1) / kFThreads,
                                           152 * (2048 / kFThreads));
    long long rest = blocks * kFThreads;  // the grid stride, in digits of the extents
    a.ntot = (long long)f->ntot;
    for (int d = 0; d < 3; ++d) {
      a.n[d] = d < f->ndims ? (int)f->n[d] : 1;
      a.step[d] = d < 2 ? (int)(rest % a.n[d]) : (int)std::min<long long>(rest, a.n[d]);
      rest /= a.n[d];
      a.r[d] = f->wrap == FDB_WRAP_REFERENCE ? pow2_64_mod((uint64_t)a.n[d]) : 0;
      a.lo[d] = 0;
      a.hi[d] = 0;
    }
    a.nterms = nt;
    for (int k = 0; k < nt; ++k) {
      FTerm& t = a.t[k];
      long long lin = 0, stride = 1;
      for (int d = 0; d < 3; ++d) {
        t.o[d] = d < f->ndims ? f->offs[(size_t)k * f->ndims + d] : 0;
        lin += stride * t.o[d];
        stride *= a.n[d];
        a.lo[d] = std::max(a.lo[d], -t.o[d]);
        a.hi[d] = std::max(a.hi[d], t.o[d]);
      }
      t.lin = lin;
      t.w = f->w[k];
      int e = 0;
      const double m = std::frexp(std::fabs(t.w), &e);  // |w| = m 2^e, m in [1/2, 1)
      t.fuse = m == 0.5 && e >= 1 && e <= 1000 ? 0x7FF00000u - ((unsigned)(e - 1) << 20) : 0u;
    }
    using Kernel = void (*)(const double*, double*, const FArgs3);
    static const Kernel kernels[] = {
        k_filter3<0, false>, k_filter3<1, false>, k_filter3<2, false>, k_filter3<3, false>,
        k_filter3<4, false>, k_filter3<5, false>, k_filter3<6, false>, k_filter3<7, false>};
    Kernel kernel = kernels[nt <= 7 ? nt : 0];
    if ((nt == 3 || nt == 5 || nt == 7) && a.t[nt / 2].fuse == 0u)
      kernel = nt == 3 ? k_filter3<3, true> : nt == 5 ? k_filter3<5, true> : k_filter3<7, true>;
    FDB_CUDA_TRY(fdb::launch_dependent(kernel, (unsigned)blocks, kFThreads, 0, f->stream, in, out,
                                       a));
  } else {
    FArgsN a{};
    a.ndims = f->ndims;
    a.nterms = nt;
    unsigned long long p = 1;
    for (int d = 0; d < f->ndims; ++d) {
      a.n[d] = f->n[d];
      a.prod[d] = p;
      p *= f->n[d];
      a.r[d] = f->wrap == FDB_WRAP_REFERENCE ? pow2_64_mod(f->n[d]) : 0;
    }
    a.ntot = f->ntot;
    uint64_t blocks = (f->ntot + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    k_filter_nd<<<(unsigned)blocks, 256, 0, f->stream>>>(in, out, a, f->d_offs, f->d_w);
  }
  fdb::note_launch();
  FDB_CUDA_TRY(cudaGetLastError());
  return FDB_OK;
}

}  // namespace

extern "C" {

int fdb_filter_create(int ndims, const uint64_t* dims, const double* xmins, const double* xmaxs,
                      int nterms, const int* offsets, const double* weights, fdb_filter** out) {
  if (!out) return fail(FDB_ERR_INVALID, "null output pointer");
  *out = nullptr;
  if (ndims < 1 || ndims > FDB_MAX_DIMS) return fail(FDB_ERR_INVALID, "ndims must be in [1, 8]");
  if (nterms < 1 || nterms > kMaxTerms) return fail(FDB_ERR_INVALID, "nterms must be in [1, 256]");
  if (!dims || !xmins || !xmaxs || !offsets || !weights)
    return fail(FDB_ERR_INVALID, "null argument");
  fdb_filter* f = new fdb_filter();
  f->ndims = ndims;
  f->ntot = 1;
  for (int d = 0; d < ndims; ++d) {
    if (dims[d] == 0 || dims[d] >= (1ull << 31)) {
      delete f;
      return fail(FDB_ERR_INVALID, "each dimension must be in [1, 2^31)");
    }
    f->n[d] = dims[d];
    f->xmins[d] = xmins[d];
    f->xmaxs[d] = xmaxs[d];
    f->ntot *= dims[d];
  }
  // std::map order: sorted offsets, the first weight of a repeated offset
  std::vector<int> order;
  for (int t = 0; t < nterms; ++t) {
    const int* o = offsets + (size_t)t * ndims;
    bool dup = false;
    for (int k : order)
      if (std::memcmp(offsets + (size_t)k * ndims, o, sizeof(int) * ndims) == 0) dup = true;
    if (dup) continue;
    for (int d = 0; d < ndims; ++d)
      if (o[d] <= -(1 << 30) || o[d] >= (1 << 30)) {
        delete f;
        return fail(FDB_ERR_INVALID, "stencil offsets must be below 2^30 in magnitude");
      }
    order.insert(std::upper_bound(order.begin(), order.end(), t,
                                  [&](int a, int b) {
                                    return lex_less(offsets + (size_t)a * ndims,
                                                    offsets + (size_t)b * ndims, ndims);
                                  }),
                 t);
  }
  for (int t : order) {
    for (int d = 0; d < ndims; ++d) f->offs.push_back(offsets[(size_t)t * ndims + d]);
    const double w = weights[t];
    f->w.push_back(w);
  }
  cudaError_t e = cudaStreamCreateWithFlags(&f->own, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete f;
    return fdb::cuda_fail(e, "cudaStreamCreate");
  }
  f->stream = f->own;
  int rc = falloc((void**)&f->buf[0], f->ntot * sizeof(double));
  if (rc == FDB_OK) rc = falloc((void**)&f->buf[1], f->ntot * sizeof(double));
  if (rc == FDB_OK) rc = falloc((void**)&f->part, fdb::reduce_partials(f->ntot) * sizeof(double));
  if (rc == FDB_OK) rc = falloc((void**)&f->dsum, sizeof(double));
  if (rc == FDB_OK) rc = falloc((void**)&f->d_offs, f->offs.size() * sizeof(int));
  if (rc == FDB_OK) rc = falloc((void**)&f->d_w, f->w.size() * sizeof(double));
  if (rc == FDB_OK && cudaMallocHost((void**)&f->hsum, sizeof(double)) != cudaSuccess)
    rc = fail(FDB_ERR_ALLOC, "cudaMallocHost failed");
  if (rc == FDB_OK) {
    e = cudaMemcpyAsync(f->d_offs, f->offs.data(), f->offs.size() * sizeof(int),
                        cudaMemcpyHostToDevice, f->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(f->d_w, f->w.data(), f->w.size() * sizeof(double),
                          cudaMemcpyHostToDevice, f->stream);
    // inData and outData start at zero (std::vector::resize, Filter.cpp:54-55)
    if (e == cudaSuccess) e = cudaMemsetAsync(f->buf[0], 0, f->ntot * sizeof(double), f->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(f->buf[1], 0, f->ntot * sizeof(double), f->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
    if (e != cudaSuccess) rc = fdb::cuda_fail(e, "filter set-up copies");
  }
  if (rc != FDB_OK) {
    fdb_filter_destroy(f);
    return rc;
  }
  *out = f;
  return FDB_OK;
}

int fdb_filter_destroy(fdb_filter* f) {
  if (!f) return FDB_OK;
  if (f->own) cudaStreamSynchronize(f->own);
  if (f->stream && f->stream != f->own) cudaStreamSynchronize(f->stream);
  cudaFree(f->buf[0]);
  cudaFree(f->buf[1]);
  cudaFree(f->part);
  cudaFree(f->dsum);
  cudaFree(f->d_offs);
  cudaFree(f->d_w);
  if (f->hsum) cudaFreeHost(f->hsum);
  if (f->own) cudaStreamDestroy(f->own);
  delete f;
  return FDB_OK;
}

int fdb_filter_set_in_data(fdb_filter* f, const double* src, int is_device) {
  FDB_TRY(check(f));
  if (!src) return fail(FDB_ERR_INVALID, "null source");
  FDB_CUDA_TRY(cudaMemcpyAsync(f->buf[f->cur], src, f->ntot * sizeof(double),
                               is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                               f->stream));
  if (!is_device) FDB_CUDA_TRY(cudaStreamSynchronize(f->stream));
  return FDB_OK;
}

int fdb_filter_get_data(fdb_filter* f, int which, double* dst, int is_device) {
  FDB_TRY(check(f));
  if (!dst || (which != 0 && which != 1)) return fail(FDB_ERR_INVALID, "bad destination");
  const double* src = f->buf[which == 0 ? f->cur : (f->cur ^ 1)];
  FDB_CUDA_TRY(cudaMemcpyAsync(dst, src, f->ntot * sizeof(double),
                               is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                               f->stream));
  FDB_CUDA_TRY(cudaStreamSynchronize(f->stream));
  return FDB_OK;
}

int fdb_filter_apply(fdb_filter* f) {
  fdb::NvtxScope nvtx_("fdb.filter.apply");
  FDB_TRY(check(f));
  return launch_apply(f);
}

int fdb_filter_copy_out_to_in(fdb_filter* f) {
  FDB_TRY(check(f));
  FDB_CUDA_TRY(cudaMemcpyAsync(f->buf[f->cur], f->buf[f->cur ^ 1], f->ntot * sizeof(double),
                               cudaMemcpyDeviceToDevice, f->stream));
  return FDB_OK;
}

int fdb_filter_iterate(fdb_filter* f, int iterations) {
  fdb::NvtxScope nvtx_("fdb.filter.iterate");
  FDB_TRY(check(f));
  if (iterations < 0) return fail(FDB_ERR_INVALID, "iterations must be >= 0");
  for (int k = 0; k < iterations; ++k) {
    FDB_TRY(launch_apply(f));
    f->cur ^= 1;  // the output becomes the input ...
  }
  if (iterations > 0) {
    // ... and, as after copyOutToIn, the output holds the same field
    FDB_CUDA_TRY(cudaMemcpyAsync(f->buf[f->cur ^ 1], f->buf[f->cur], f->ntot * sizeof(double),
                                 cudaMemcpyDeviceToDevice, f->stream));
  }
  return FDB_OK;
}

int fdb_filter_checksum(fdb_filter* f, int which, double* out) {
  FDB_TRY(check(f));
  if (!out || (which != 0 && which != 1)) return fail(FDB_ERR_INVALID, "bad checksum request");
  FDB_TRY(fdb::launch_sum(f->buf[which == 0 ? f->cur : (f->cur ^ 1)], f->ntot, f->part, f->dsum,
                          f->stream));
  FDB_CUDA_TRY(cudaMemcpyAsync(f->hsum, f->dsum, sizeof(double), cudaMemcpyDeviceToHost,
                               f->stream));
  FDB_CUDA_TRY(cudaStreamSynchronize(f->stream));
  *out = *f->hsum;
  return FDB_OK;
}

int fdb_filter_set_wrap(fdb_filter* f, int mode) {
  FDB_TRY(check(f));
  if (mode != FDB_WRAP_REFERENCE && mode != FDB_WRAP_PERIODIC)
    return fail(FDB_ERR_INVALID, "unknown wrap mode");
  f->wrap = mode;
  return FDB_OK;
}

int fdb_filter_set_stream(fdb_filter* f, void* cuda_stream) {
  FDB_TRY(check(f));
  FDB_CUDA_TRY(cudaStreamSynchronize(f->stream));
  f->stream = cuda_stream ? (cudaStream_t)cuda_stream : f->own;
  return FDB_OK;
}

int fdb_filter_info(fdb_filter* f, uint64_t* ntot, int* nterms) {
  FDB_TRY(check(f));
  if (ntot) *ntot = f->ntot;
  if (nterms) *nterms = (int)f->w.size();
  return FDB_OK;
}

int fdb_filter_synchronize(fdb_filter* f) {
  FDB_TRY(check(f));
  FDB_CUDA_TRY(cudaStreamSynchronize(f->stream));
  return FDB_OK;
}

}  // extern "C"
