// BLAS-1 over MRHS fields (no counterpart in the reference, which has no
// linear algebra; cg_inverter is an empty stub at src/qcu.cu:173 of the
// reference).
//
// A field is `n` complex elements in RHS-innermost order, so element e
// belongs to RHS e % nrhs.  Coefficients are per-RHS device arrays of
// double2 (complex).  FP32 fields are updated in FP32 arithmetic and FP64
// fields in FP64.  Reductions accumulate in FP64 and return per-RHS results
// into device arrays, in a fixed order (deterministic).
#pragma once

#include "qcu_common.cuh"

namespace qcu {

struct FieldRef {
  void* data = nullptr;
  int prec = PREC_DOUBLE;  // PREC_DOUBLE or PREC_SINGLE for BLAS operands
  int64_t n = 0;           // complex elements = vh * ncomp * nrhs
  int nrhs = 1;
};

// Second stage of the reductions: one warp per RHS r adds the block partials
// l, l + 32, ... in its lanes l, then the lanes in a fixed shuffle tree
// (deterministic); every lane returns the sum.
#ifdef __CUDACC__
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double shfl_xor(double v, int off) { return __shfl_xor_sync(0xffffffffu, v, off); }
__device__ __forceinline__ double2 shfl_xor(double2 v, int off) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, off), __shfl_xor_sync(0xffffffffu, v.y, off));
}
template <typename A>
__device__ __forceinline__ A sum_partials(const A* __restrict__ partials, int nblocks, int nrhs, int r, int lane) {
  A s = A{};
  constexpr int U = 8;  // partials loaded together: their latency, not their sum, is the kernel's time
  for (int b = lane; b < nblocks; b += 32 * U) {
    A v[U];
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = b + 32 * u < nblocks ? partials[(int64_t)(b + 32 * u) * nrhs + r] : A{};
#pragma unroll
    for (int u = 0; u < U; u++) s = s + v[u];
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s = s + shfl_xor(s, off);
  return s;
}
#endif

// block partials of a reduction, [block][nrhs], summed by the kernel that uses them
struct Partials {
  const double* norm = nullptr;    // |.|^2 (or the first of two)
  const double* norm2 = nullptr;   // the second
  const double2* dot = nullptr;
  int blocks = 0;
};

class Blas {
 public:
  // scratch for the two-stage reductions is owned by the caller (Workspace):
  // max_blocks x QCU_MAX_RHS x 4 doubles
  Blas(double* partials, int max_blocks) : partials_(partials), max_blocks_(max_blocks) {}

  // y = a_r x + b_r y
  void axpby(const double2* a, const FieldRef& x, const double2* b, const FieldRef& y, cudaStream_t st);
  // z = a_r x + b_r y + c_r z
  void axpbypcz(const double2* a, const FieldRef& x, const double2* b, const FieldRef& y, const double2* c,
                const FieldRef& z, cudaStream_t st);
  // y = a_r x + b_r y, then out[r] = |y_r|^2 (double)
  void axpby_norm(const double2* a, const FieldRef& x, const double2* b, const FieldRef& y, double* out,
                  cudaStream_t st);
  // out[r] = |x_r|^2; exact: every product formed in FP64 (exact for FP32
  // inputs), else FP32 fields form their products in FP32 (summed in FP64)
  void norm2(const FieldRef& x, double* out, cudaStream_t st, bool exact = true);
  // out[r] = <x_r, y_r> = sum conj(x) y  (double2); FP32 fields form the
  // products in FP32, summed in FP64
  void cdot(const FieldRef& x, const FieldRef& y, double2* out, cudaStream_t st);
  // hi += lo (any BLAS precisions), elementwise
  void add_to(const FieldRef& lo, const FieldRef& hi, cudaStream_t st);
  // y = x, with precision conversion
  void copy(const FieldRef& x, const FieldRef& y, cudaStream_t st);
  void zero(const FieldRef& x, cudaStream_t st);

  // Fused operations of the Krylov solvers on fields of one precision; the
  // block partials are left for the next scalar kernel (sum_partials) and
  // live until the next reduction.
  // |x|^2 (products as norm2 with exact = false)
  Partials norm2_partials(const FieldRef& x, cudaStream_t st);
  // <x, y> and |x|^2
  Partials dot_norm(const FieldRef& x, const FieldRef& y, cudaStream_t st);
  // <x, y>
  Partials dot_partials(const FieldRef& x, const FieldRef& y, cudaStream_t st);
  // s -= a_r q, r -= a_r w; |s|^2 (norm), |r|^2 (norm2)
  Partials cg_update(const double2* a, const FieldRef& q, const FieldRef& s, const FieldRef& w, const FieldRef& r,
                     cudaStream_t st);
  // x += a_r p, then p = r + b_r p; real a and b
  void cg_direction(const double2* a, const double2* b, const FieldRef& r, const FieldRef& p, const FieldRef& x,
                    cudaStream_t st);
  // x += a_r p + o_r s, then s -= o_r t; |s|^2, <r0, s>
  Partials bicg_update(const double2* a, const double2* o, const FieldRef& p, const FieldRef& s, const FieldRef& t,
                       const FieldRef& r0, const FieldRef& x, cudaStream_t st);

  // Masked moves: only the RHS with sel[r] != 0 are read and written.
  // xh += xl, xl = 0, and d = be - xh unless d is empty (FP64 xh, be, d)
  void fold(const int* sel, const FieldRef& xl, const FieldRef& xh, const FieldRef& be, const FieldRef& d,
            cudaStream_t st);
  // y = x, and z = x unless z is empty (same precision as y); x empty: y = 0
  void select_copy(const int* sel, const FieldRef& x, const FieldRef& y, const FieldRef& z, cudaStream_t st);
  // out[r] = |x_r|^2 for the selected RHS (0 for the others) of the FP64 field x, and y = x in y's precision
  void residual(const int* sel, const FieldRef& x, const FieldRef& y, double* out, cudaStream_t st);

  static int blocks_for(int64_t n);

 private:
  // scratch: a double2 array, then two double arrays, each max_blocks_ x QCU_MAX_RHS
  double2* dots() const { return reinterpret_cast<double2*>(partials_); }
  double* norms(int k) const;
  double* partials_;
  int max_blocks_;
};

}  // namespace qcu
