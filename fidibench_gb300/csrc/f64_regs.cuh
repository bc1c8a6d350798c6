// f64_regs.cuh -- FP64 additions and multiplications as three-register DFMAs.
//
// GB300's FP64 pipe holds a warp (per SM sub-partition) 67 cycles for a DFMA
// whose three operands are per-thread registers, but 80 cycles for a DADD, a
// DMUL or a DFMA with a constant or uniform-register operand (measured in
// register-only loops).  Kernels bound by that pipe therefore add as
// a * 1 + b and multiply as a * b + (-0), with 1, -1, -0 and their coefficients
// in registers: the same values, rounded once, signed zeros included.
#pragma once

namespace fdb {

// Values in per-thread registers: each passes through the thread's own word of
// shared memory, so that the compiler neither knows the value nor that it is
// the same in all threads (either would make it a constant or uniform operand).
struct RegLoader {
  volatile double* slot;
  __device__ __forceinline__ explicit RegLoader(double* s_slots) : slot(s_slots + threadIdx.x) {}
  __device__ __forceinline__ double operator()(double x) const {
    *slot = x;
    return *slot;
  }
};

struct F64Regs {
  double one, minus_one, minus_zero;
  __device__ __forceinline__ explicit F64Regs(const RegLoader& reg)
      : one(reg(1.0)), minus_one(reg(-1.0)), minus_zero(reg(-0.0)) {}
  __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
  __device__ __forceinline__ double sub(double a, double b) const {
    return __fma_rn(b, minus_one, a);
  }
  __device__ __forceinline__ double mul(double a, double b) const {
    return __fma_rn(a, b, minus_zero);
  }
};

}  // namespace fdb
