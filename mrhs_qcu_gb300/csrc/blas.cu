// BLAS-1 kernels over MRHS fields (see blas.h).
//
// Thread mapping: thread k handles R consecutive complex elements (one
// 128-bit vector for FP64 R=1 / FP32 R=2) and strides over the field with a
// stride that is a multiple of nrhs, so every thread stays on the same R RHS
// and keeps private FP64 partial sums.  Block reduction: per RHS, one warp
// sums the block's partials with shuffles; a second kernel adds the
// per-block results in block order.  No atomics, so results are bitwise
// reproducible for a given launch shape.
#include <algorithm>

#include "blas.h"
#include "layout.h"  // QCU_MAX_RHS

namespace qcu {
namespace {

constexpr int kMaxBlocks = 1024;
constexpr int kMaxThreads = 1024;  // block_size: a multiple of 32 and of the RHS groups (31 groups: 992)

template <typename T> struct V2;
template <> struct V2<double> { using t = double2; };
template <> struct V2<float> { using t = float2; };

template <int P> struct BT;
template <> struct BT<PREC_DOUBLE> { using real = double; };
template <> struct BT<PREC_SINGLE> { using real = float; };

struct Shape {
  int64_t nchunks;  // n / R
  int R;
  int G;            // nrhs / R
  int nrhs;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 tof(double2 a) { return make_float2((float)a.x, (float)a.y); }

// FP64 values of a complex element, and back (integer-pipe conversions, qcu_common.cuh)
__device__ __forceinline__ double2 ld(const double2* p) { return *p; }
__device__ __forceinline__ double2 ld(const float2* p) { return Store<PREC_SINGLE>::to_z(*p); }
__device__ __forceinline__ void st(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void st(float2* p, double2 v) { *p = Store<PREC_SINGLE>::from_z(v); }

// FP64 sum of FP32 products in groups of four.  One conversion and FP64
// addition per product is bound by the FP64 pipe (2 lanes a cycle and SM, and
// the conversion issues there too): the norm of 24^3x48 SU(3) nrhs 12 FP32
// took 195 us against 56 us of HBM time (75 now).  So the products of a group are added in
// FP32 with their rounding errors kept (Knuth's TwoSum): the sum goes to FP64, the
// errors, added in FP32 with theirs kept in turn, with every fourth group (1.25 additions a
// group instead of 2: <x, y> with |x|^2 at 16^3x32 SU(4) nrhs 16 89 -> 59 us, <x, y> 62 -> 48),
// and theirs at the end.  Against an exact sum of the same products the error is the plain FP64
// sum's, also where the products span many binades (64 products over 8 decades: 0.7e-17 of the
// sum of magnitudes, plain 1.5e-17; without the third level 49e-17).  A group that
// leaves FP32's range, or is not finite, is added product by product (a call: as
// predicated instructions it would hold the FP64 pipe).
constexpr int kGroup = 4;
static __device__ __noinline__ double add_plainly(double acc, float a, float b, float c, float d) {
  acc += (double)a;
  acc += (double)b;
  acc += (double)c;
  return acc + (double)d;
}
struct GroupSum {
  float p[kGroup];
  float rest = 0.f;   // rounding errors of the groups since the last FP64 addition of them (every fourth)
  float rest2 = 0.f;  // rounding errors of these
  int groups = 0;
  __device__ __forceinline__ void set(int u, float v) { p[u] = v; }  // u: a constant once the loops are unrolled
  // a + b, and its rounding error
  static __device__ __forceinline__ float two_sum(float a, float b, float& err) {
    const float s = __fadd_rn(a, b), c = __fsub_rn(s, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, c)), __fsub_rn(b, c));
    return s;
  }
  __device__ __forceinline__ void flush(double& acc) {
    float lo, e, lo2 = 0.f, hi = two_sum(p[0], p[1], lo);
#pragma unroll
    for (int u = 2; u < kGroup; u++) {
      hi = two_sum(hi, p[u], e);
      lo = two_sum(lo, e, e);
      lo2 = __fadd_rn(lo2, e);
    }
    if (fabsf(hi) <= 3.402823466e38f) {
      acc += to_f64(hi);
      rest = two_sum(rest, lo, e);
      rest2 = __fadd_rn(rest2, __fadd_rn(lo2, e));
    } else {
      acc = add_plainly(acc, p[0], p[1], p[2], p[3]);
    }
    if ((++groups & 3) == 0) {
      acc += to_f64(rest);
      rest = 0.f;
    }
  }
  __device__ __forceinline__ void finish(double& acc) { acc += to_f64(rest) + to_f64(rest2); }
};
// FP64 products accumulate as they are formed
__device__ __forceinline__ void add_square(double& acc, double2 v) {
  acc = fma(v.x, v.x, acc);
  acc = fma(v.y, v.y, acc);
}
__device__ __forceinline__ void add_conj(double2& acc, double2 u, double2 v) {  // conj(u) v
  acc.x = fma(u.x, v.x, acc.x);
  acc.x = fma(u.y, v.y, acc.x);
  acc.y = fma(u.x, v.y, acc.y);
  acc.y = fma(-u.y, v.x, acc.y);
}
// per-RHS sums of one thread: FP32 fields in groups, FP64 fields directly
template <int P>
struct NormSum {
  double acc = 0.0;
  GroupSum g;
  __device__ __forceinline__ void add(int u, float2 v) { g.set(u, fmaf(v.x, v.x, v.y * v.y)); }
  __device__ __forceinline__ void add(int, double2 v) { add_square(acc, v); }
  __device__ __forceinline__ void flush() {
    if constexpr (P == PREC_SINGLE) g.flush(acc);
  }
  __device__ __forceinline__ double total() {
    if constexpr (P == PREC_SINGLE) g.finish(acc);
    return acc;
  }
};
template <int P>
struct DotSum {  // conj(u) v
  double2 acc = make_double2(0.0, 0.0);
  GroupSum re, im;
  __device__ __forceinline__ void add(int k, float2 u, float2 v) {
    re.set(k, fmaf(u.x, v.x, u.y * v.y));
    im.set(k, fmaf(u.x, v.y, -u.y * v.x));
  }
  __device__ __forceinline__ void add(int, double2 u, double2 v) { add_conj(acc, u, v); }
  __device__ __forceinline__ void flush() {
    if constexpr (P == PREC_SINGLE) {
      re.flush(acc.x);
      im.flush(acc.y);
    }
  }
  __device__ __forceinline__ double2 total() {
    if constexpr (P == PREC_SINGLE) {
      re.finish(acc.x);
      im.finish(acc.y);
    }
    return acc;
  }
};
template <typename A, typename S, int R>
__device__ __forceinline__ void totals(A (&out)[R], S (&sums)[R]) {
#pragma unroll
  for (int i = 0; i < R; i++) out[i] = sums[i].total();
}

// chunk c of a field: R complex elements, one 16-byte vector for FP32 R = 2 and FP64 R = 1
template <int R>
__device__ __forceinline__ void load_chunk(const float2* f, int64_t c, float2 (&v)[R]) {
  if constexpr (R == 2) {
    const float4 q = reinterpret_cast<const float4*>(f)[c];
    v[0] = make_float2(q.x, q.y);
    v[1] = make_float2(q.z, q.w);
  } else {
#pragma unroll
    for (int i = 0; i < R; i++) v[i] = f[c * R + i];
  }
}
template <int R>
__device__ __forceinline__ void store_chunk(float2* f, int64_t c, const float2 (&v)[R]) {
  if constexpr (R == 2) {
    reinterpret_cast<float4*>(f)[c] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
  } else {
#pragma unroll
    for (int i = 0; i < R; i++) f[c * R + i] = v[i];
  }
}
template <int R>
__device__ __forceinline__ void load_chunk(const double2* f, int64_t c, double2 (&v)[R]) {
#pragma unroll
  for (int i = 0; i < R; i++) v[i] = f[c * R + i];
}
template <int R>
__device__ __forceinline__ void store_chunk(double2* f, int64_t c, const double2 (&v)[R]) {
#pragma unroll
  for (int i = 0; i < R; i++) f[c * R + i] = v[i];
}
// y + a x in the fields' own arithmetic
__device__ __forceinline__ float2 add_mul(float2 a, float2 x, float2 y) {
  return make_float2(fmaf(a.x, x.x, fmaf(-a.y, x.y, y.x)), fmaf(a.x, x.y, fmaf(a.y, x.x, y.y)));
}
__device__ __forceinline__ double2 add_mul(double2 a, double2 x, double2 y) {
  return make_double2(fma(a.x, x.x, fma(-a.y, x.y, y.x)), fma(a.x, x.y, fma(a.y, x.x, y.y)));
}
__device__ __forceinline__ void coeff(double2 a, float2& c) { c = tof(a); }
__device__ __forceinline__ void coeff(double2 a, double2& c) { c = a; }

// dynamic shared memory of the reducing kernels: R values of each thread (reduce_bytes)
template <typename A>
__device__ __forceinline__ A* reduce_smem() {
  extern __shared__ double2 blas_smem[];
  return reinterpret_cast<A*>(blas_smem);
}

// block-level per-RHS reduction of `vals` (R values per thread) into
// out[blockIdx.x * nrhs + r]
template <typename A>
__device__ void block_reduce(A* sm, const A* vals, int R, int G, int nrhs, A* out) {
  const int t = threadIdx.x, B = blockDim.x;
  for (int i = 0; i < R; i++) sm[t * R + i] = vals[i];
  __syncthreads();
  const int lane = t & 31, warp = t >> 5, nw = B >> 5;
  const int per = B / G;
  for (int r = warp; r < nrhs; r += nw) {
    const int g = r / R, i = r % R;
    A s;
    s = A{};
    for (int m = lane; m < per; m += 32) {
      const A v = sm[(g + m * G) * R + i];
      s = s + v;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s = s + shfl_xor(s, off);
    if (lane == 0) out[(int64_t)blockIdx.x * nrhs + r] = s;
  }
}


// ---------------------------------------------------------------------------
template <int PX, int PY, int R, bool NORM>
__global__ void __launch_bounds__(kMaxThreads, 1) axpby_kernel(const double2* __restrict__ a, const void* __restrict__ xv, const double2* __restrict__ b,
                             void* __restrict__ yv, Shape s, double* partials) {
  using EX = typename V2<typename BT<PX>::real>::t;
  using EY = typename V2<typename BT<PY>::real>::t;
  const EX* x = static_cast<const EX*>(xv);
  EY* y = static_cast<EY*>(yv);
  const int g = threadIdx.x % s.G;
  double2 ca[R], cb[R];
  double acc[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    ca[i] = a ? a[g * R + i] : make_double2(1.0, 0.0);
    cb[i] = b ? b[g * R + i] : make_double2(1.0, 0.0);
    acc[i] = 0.0;
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if constexpr (PX == PREC_SINGLE && PY == PREC_SINGLE) {
    // FP32 fields: FP32 arithmetic (the FP64 pipe of this GPU is a small
    // fraction of the FP32 one); the norm's per-thread sum stays FP64
    float2 fa[R], fb[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      fa[i] = tof(ca[i]);
      fb[i] = tof(cb[i]);
    }
    // U chunks loaded ahead of the stores (which the loads may not pass)
    constexpr int U = NORM ? kGroup : 1;
    NormSum<PREC_SINGLE> sum[R];
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c0 < s.nchunks; c0 += U * stride) {
      float2 xs[U][R], ys[U][R];
#pragma unroll
      for (int u = 0; u < U; u++) {
#pragma unroll
        for (int i = 0; i < R; i++) xs[u][i] = ys[u][i] = make_float2(0.f, 0.f);
        if (c0 + u * stride >= s.nchunks) continue;
        load_chunk<R>(x, c0 + u * stride, xs[u]);
        load_chunk<R>(y, c0 + u * stride, ys[u]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
#pragma unroll
        for (int i = 0; i < R; i++) {
          const float2 v = cmulf(fa[i], xs[u][i]), w = cmulf(fb[i], ys[u][i]);
          ys[u][i] = make_float2(v.x + w.x, v.y + w.y);
          if (NORM) sum[i].add(u, ys[u][i]);
        }
        if (c0 + u * stride < s.nchunks) store_chunk<R>(y, c0 + u * stride, ys[u]);
      }
      if (NORM) {
#pragma unroll
        for (int i = 0; i < R; i++) sum[i].flush();
      }
    }
    totals(acc, sum);
  } else if (b == nullptr) {
    // b = 1: no multiply of y (FP64 arithmetic is bound by the FP64 pipe here)
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < s.nchunks; c += stride) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int64_t e = c * R + i;
        const double2 v = cmul(ca[i], ld(x + e)) + ld(y + e);
        st(y + e, v);
        if (NORM) add_square(acc[i], v);
      }
    }
  } else {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < s.nchunks; c += stride) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int64_t e = c * R + i;
        const double2 v = cmul(ca[i], ld(x + e)) + cmul(cb[i], ld(y + e));
        st(y + e, v);
        if (NORM) add_square(acc[i], v);
      }
    }
  }
  if (NORM) {
    block_reduce<double>(reduce_smem<double>(), acc, R, s.G, s.nrhs, partials);
  }
}

template <int P, int R>
__global__ void __launch_bounds__(kMaxThreads, 1) axpbypcz_kernel(const double2* __restrict__ a, const void* __restrict__ xv,
                                const double2* __restrict__ b, const void* __restrict__ yv,
                                const double2* __restrict__ c, void* __restrict__ zv, Shape s) {
  using E = typename V2<typename BT<P>::real>::t;
  const E* x = static_cast<const E*>(xv);
  const E* y = static_cast<const E*>(yv);
  E* z = static_cast<E*>(zv);
  const int g = threadIdx.x % s.G;
  double2 ca[R], cb[R], cc[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    ca[i] = a[g * R + i];
    cb[i] = b[g * R + i];
    cc[i] = c ? c[g * R + i] : make_double2(1.0, 0.0);
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if constexpr (P == PREC_SINGLE) {  // FP32 fields: FP32 arithmetic
    float2 fa[R], fb[R], fc[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      fa[i] = tof(ca[i]);
      fb[i] = tof(cb[i]);
      fc[i] = tof(cc[i]);
    }
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < s.nchunks; k += stride) {
      float2 xs[R], ys[R], zs[R];
      if constexpr (R == 2) {
        const float4 xq = reinterpret_cast<const float4*>(x)[k], yq = reinterpret_cast<const float4*>(y)[k],
                     zq = reinterpret_cast<const float4*>(z)[k];
        xs[0] = make_float2(xq.x, xq.y);
        xs[1] = make_float2(xq.z, xq.w);
        ys[0] = make_float2(yq.x, yq.y);
        ys[1] = make_float2(yq.z, yq.w);
        zs[0] = make_float2(zq.x, zq.y);
        zs[1] = make_float2(zq.z, zq.w);
      } else {
#pragma unroll
        for (int i = 0; i < R; i++) {
          xs[i] = x[k * R + i];
          ys[i] = y[k * R + i];
          zs[i] = z[k * R + i];
        }
      }
      float2 o[R];
#pragma unroll
      for (int i = 0; i < R; i++) {
        const float2 u = cmulf(fa[i], xs[i]), v = cmulf(fb[i], ys[i]), w = cmulf(fc[i], zs[i]);
        o[i] = make_float2(u.x + v.x + w.x, u.y + v.y + w.y);
      }
      if constexpr (R == 2) {
        reinterpret_cast<float4*>(z)[k] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
      } else {
#pragma unroll
        for (int i = 0; i < R; i++) z[k * R + i] = o[i];
      }
    }
  } else {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < s.nchunks; k += stride) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int64_t e = k * R + i;
        st(z + e, cmul(ca[i], ld(x + e)) + cmul(cb[i], ld(y + e)) + cmul(cc[i], ld(z + e)));
      }
    }
  }
}

// MODE 0: |x|^2, 1: <x, y>.  FAST (FP32 fields): the products in FP32, summed
// in FP64; otherwise every product is formed in FP64 (exact for FP32 inputs).
template <int PX, int PY, int R, int MODE, bool FAST = false>
__global__ void __launch_bounds__(kMaxThreads, 1) reduce_kernel(const void* __restrict__ xv, const void* __restrict__ yv, Shape s, void* partials) {
  using EX = typename V2<typename BT<PX>::real>::t;
  using EY = typename V2<typename BT<PY>::real>::t;
  const EX* x = static_cast<const EX*>(xv);
  const EY* y = static_cast<const EY*>(yv);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // FAST: FP32 products in groups; else the elements in FP64
  constexpr int PS = FAST ? PREC_SINGLE : PREC_DOUBLE;
  auto val = [](const EX& e) {
    if constexpr (FAST)
      return e;
    else
      return ld(&e);
  };
  if constexpr (MODE == 0) {
    NormSum<PS> sum[R];
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c0 < s.nchunks; c0 += kGroup * stride) {
      EX v[kGroup][R];
#pragma unroll
      for (int u = 0; u < kGroup; u++) {
#pragma unroll
        for (int i = 0; i < R; i++) v[u][i] = EX{};
        if (c0 + u * stride < s.nchunks) load_chunk<R>(x, c0 + u * stride, v[u]);
      }
#pragma unroll
      for (int i = 0; i < R; i++) {
#pragma unroll
        for (int u = 0; u < kGroup; u++) sum[i].add(u, val(v[u][i]));
        sum[i].flush();
      }
    }
    double acc[R];
    totals(acc, sum);
    block_reduce<double>(reduce_smem<double>(), acc, R, s.G, s.nrhs, static_cast<double*>(partials));
  } else {
    static_assert(PX == PY, "one precision");
    DotSum<PS> sum[R];
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c0 < s.nchunks; c0 += kGroup * stride) {
      EX a[kGroup][R], b[kGroup][R];
#pragma unroll
      for (int u = 0; u < kGroup; u++) {
#pragma unroll
        for (int i = 0; i < R; i++) a[u][i] = EX{}, b[u][i] = EX{};
        if (c0 + u * stride >= s.nchunks) continue;
        load_chunk<R>(x, c0 + u * stride, a[u]);
        load_chunk<R>(y, c0 + u * stride, b[u]);
      }
#pragma unroll
      for (int i = 0; i < R; i++) {
#pragma unroll
        for (int u = 0; u < kGroup; u++) sum[i].add(u, val(a[u][i]), val(b[u][i]));
        sum[i].flush();
      }
    }
    double2 acc[R];
    totals(acc, sum);
    block_reduce<double2>(reduce_smem<double2>(), acc, R, s.G, s.nrhs, static_cast<double2*>(partials));
  }
}

// ---- fused kernels of the Krylov iterations (solver.cu) ----------------------
// s -= a q, r -= a w; partial |s|^2 (part) and |r|^2 (part2)
template <int P, int R>
__global__ void __launch_bounds__(kMaxThreads, 1) cg_update_kernel(const double2* __restrict__ a, const void* __restrict__ qv, void* __restrict__ sv,
                                 const void* __restrict__ wv, void* __restrict__ rv, Shape sh, double* part,
                                 double* part2) {
  using E = typename V2<typename BT<P>::real>::t;
  const E *q = static_cast<const E*>(qv), *w = static_cast<const E*>(wv);
  E *s = static_cast<E*>(sv), *r = static_cast<E*>(rv);
  const int g = threadIdx.x % sh.G;
  E na[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    const double2 c = a[g * R + i];
    coeff(make_double2(-c.x, -c.y), na[i]);
  }
  NormSum<P> sums[R], sumr[R];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = 2;  // chunks loaded ahead of the stores
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < sh.nchunks;) {
#pragma unroll
    for (int k = 0; k < kGroup; k += U, c += U * stride) {
      E qs[U][R], ss[U][R], ws[U][R], rs[U][R];
#pragma unroll
      for (int u = 0; u < U; u++) {
#pragma unroll
        for (int i = 0; i < R; i++) qs[u][i] = ss[u][i] = ws[u][i] = rs[u][i] = E{};
        if (c + u * stride >= sh.nchunks) continue;
        load_chunk<R>(q, c + u * stride, qs[u]);
        load_chunk<R>(s, c + u * stride, ss[u]);
        load_chunk<R>(w, c + u * stride, ws[u]);
        load_chunk<R>(r, c + u * stride, rs[u]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
#pragma unroll
        for (int i = 0; i < R; i++) {
          ss[u][i] = add_mul(na[i], qs[u][i], ss[u][i]);
          rs[u][i] = add_mul(na[i], ws[u][i], rs[u][i]);
          sums[i].add(k + u, ss[u][i]);
          sumr[i].add(k + u, rs[u][i]);
        }
        if (c + u * stride >= sh.nchunks) continue;
        store_chunk<R>(s, c + u * stride, ss[u]);
        store_chunk<R>(r, c + u * stride, rs[u]);
      }
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
      sums[i].flush();
      sumr[i].flush();
    }
  }
  double accs[R], accr[R];
  totals(accs, sums);
  totals(accr, sumr);
  block_reduce<double>(reduce_smem<double>(), accs, R, sh.G, sh.nrhs, part);
  __syncthreads();
  block_reduce<double>(reduce_smem<double>(), accr, R, sh.G, sh.nrhs, part2);
}

// x += a p, p = r + b p (a and b real)
template <int P, int R>
__global__ void __launch_bounds__(kMaxThreads, 1) cg_direction_kernel(const double2* __restrict__ a, const double2* __restrict__ b,
                                    const void* __restrict__ rv, void* __restrict__ pv, void* __restrict__ xv,
                                    Shape sh) {
  using E = typename V2<typename BT<P>::real>::t;
  const E* r = static_cast<const E*>(rv);
  E *p = static_cast<E*>(pv), *x = static_cast<E*>(xv);
  const int g = threadIdx.x % sh.G;
  E ca[R], cb[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    coeff(a[g * R + i], ca[i]);
    coeff(b[g * R + i], cb[i]);
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < sh.nchunks; c += stride) {
    E rs[R], ps[R], xs[R];
    load_chunk<R>(r, c, rs);
    load_chunk<R>(p, c, ps);
    load_chunk<R>(x, c, xs);
#pragma unroll
    for (int i = 0; i < R; i++) {
      xs[i].x = fma(ca[i].x, ps[i].x, xs[i].x);
      xs[i].y = fma(ca[i].x, ps[i].y, xs[i].y);
      ps[i].x = fma(cb[i].x, ps[i].x, rs[i].x);
      ps[i].y = fma(cb[i].x, ps[i].y, rs[i].y);
    }
    store_chunk<R>(x, c, xs);
    store_chunk<R>(p, c, ps);
  }
}

// partial <x, y> (part2) and |x|^2 (part)
template <int P, int R>
__global__ void __launch_bounds__(kMaxThreads, 1) dot_norm_kernel(const void* __restrict__ xv, const void* __restrict__ yv, Shape sh, double* part,
                                double2* part2) {
  using E = typename V2<typename BT<P>::real>::t;
  const E *x = static_cast<const E*>(xv), *y = static_cast<const E*>(yv);
  NormSum<P> nrm[R];
  DotSum<P> dot[R];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = kGroup;
  for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c0 < sh.nchunks; c0 += U * stride) {
    E a[U][R], b[U][R];
#pragma unroll
    for (int u = 0; u < U; u++) {
#pragma unroll
      for (int i = 0; i < R; i++) a[u][i] = E{}, b[u][i] = E{};
      if (c0 + u * stride >= sh.nchunks) continue;
      load_chunk<R>(x, c0 + u * stride, a[u]);
      load_chunk<R>(y, c0 + u * stride, b[u]);
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
#pragma unroll
      for (int u = 0; u < U; u++) {
        dot[i].add(u, a[u][i], b[u][i]);
        nrm[i].add(u, a[u][i]);
      }
      dot[i].flush();
      nrm[i].flush();
    }
  }
  double2 accd[R];
  double accn[R];
  totals(accd, dot);
  totals(accn, nrm);
  block_reduce<double2>(reduce_smem<double2>(), accd, R, sh.G, sh.nrhs, part2);
  __syncthreads();
  block_reduce<double>(reduce_smem<double>(), accn, R, sh.G, sh.nrhs, part);
}

// x += a p + o s, s -= o t; partial |s|^2 (part) and <r0, s> (part2)
template <int P, int R>
__global__ void __launch_bounds__(kMaxThreads, 1) bicg_update_kernel(const double2* __restrict__ a, const double2* __restrict__ o,
                                   const void* __restrict__ pv, void* __restrict__ sv, const void* __restrict__ tv,
                                   const void* __restrict__ r0v, void* __restrict__ xv, Shape sh, double* part,
                                   double2* part2) {
  using E = typename V2<typename BT<P>::real>::t;
  const E *p = static_cast<const E*>(pv), *t = static_cast<const E*>(tv), *r0 = static_cast<const E*>(r0v);
  E *s = static_cast<E*>(sv), *x = static_cast<E*>(xv);
  const int g = threadIdx.x % sh.G;
  E ca[R], co[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    coeff(a[g * R + i], ca[i]);
    coeff(o[g * R + i], co[i]);
  }
  NormSum<P> nrm[R];
  DotSum<P> dot[R];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < sh.nchunks;) {
#pragma unroll
    for (int u = 0; u < kGroup; u++, c += stride) {
      E ps[R] = {}, ss[R] = {}, ts[R] = {}, rs[R] = {}, xs[R] = {};
      const bool in = c < sh.nchunks;
      if (in) {
        load_chunk<R>(p, c, ps);
        load_chunk<R>(s, c, ss);
        load_chunk<R>(t, c, ts);
        load_chunk<R>(r0, c, rs);
        load_chunk<R>(x, c, xs);
      }
#pragma unroll
      for (int i = 0; i < R; i++) {
        E no;
        no.x = -co[i].x;
        no.y = -co[i].y;
        xs[i] = add_mul(co[i], ss[i], add_mul(ca[i], ps[i], xs[i]));
        ss[i] = add_mul(no, ts[i], ss[i]);
        nrm[i].add(u, ss[i]);
        dot[i].add(u, rs[i], ss[i]);
      }
      if (in) {
        store_chunk<R>(x, c, xs);
        store_chunk<R>(s, c, ss);
      }
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
      nrm[i].flush();
      dot[i].flush();
    }
  }
  double2 accd[R];
  double accn[R];
  totals(accd, dot);
  totals(accn, nrm);
  block_reduce<double2>(reduce_smem<double2>(), accd, R, sh.G, sh.nrhs, part2);
  __syncthreads();
  block_reduce<double>(reduce_smem<double>(), accn, R, sh.G, sh.nrhs, part);
}

// ---- masked moves between fields of selected RHS (no arithmetic on the others) ----
// xh += xl, xl = 0; d = be - xh where d is given (FP64 xh, be, d; xl in P)
template <int P>
__global__ void fold_kernel(const int* __restrict__ sel, void* __restrict__ xlv, double2* __restrict__ xh,
                            const double2* __restrict__ be, double2* __restrict__ d, Shape sh) {
  using E = typename V2<typename BT<P>::real>::t;
  if (!sel[threadIdx.x % sh.G]) return;
  E* xl = static_cast<E*>(xlv);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < sh.nchunks; c += stride) {
    const double2 v = ld(xl + c) + xh[c];
    xh[c] = v;
    xl[c] = E{};
    if (d) {
      const double2 b = be[c];
      d[c] = make_double2(b.x - v.x, b.y - v.y);
    }
  }
}

// y = x (converted), z = x where z is given; x = nullptr: y = 0
template <int PX, int PY>
__global__ void select_copy_kernel(const int* __restrict__ sel, const void* __restrict__ xv, void* __restrict__ yv,
                                   void* __restrict__ zv, Shape sh) {
  using EX = typename V2<typename BT<PX>::real>::t;
  using EY = typename V2<typename BT<PY>::real>::t;
  if (!sel[threadIdx.x % sh.G]) return;
  const EX* x = static_cast<const EX*>(xv);
  EY *y = static_cast<EY*>(yv), *z = static_cast<EY*>(zv);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < sh.nchunks; c += stride) {
    EY e{};
    if (x) {
      if constexpr (PX == PY)
        e = x[c];
      else
        st(&e, ld(x + c));
    }
    y[c] = e;
    if (z) z[c] = e;
  }
}

// partial |x|^2 of the FP64 field x over every RHS; selected RHS: y = x converted to P
template <int P>
__global__ void residual_kernel(const int* __restrict__ sel, const double2* __restrict__ x, void* __restrict__ yv,
                                Shape sh, double* part) {
  using E = typename V2<typename BT<P>::real>::t;
  E* y = static_cast<E*>(yv);
  const bool mine = sel[threadIdx.x % sh.G] != 0;
  double acc[1] = {0.0};
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = 4;  // elements loaded ahead of the stores
  if (mine)
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < sh.nchunks; c += U * stride) {
      double2 v[U];
#pragma unroll
      for (int u = 0; u < U; u++) v[u] = c + u * stride < sh.nchunks ? x[c + u * stride] : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < U; u++) {
        add_square(acc[0], v[u]);
        if (c + u * stride < sh.nchunks) st(y + c + u * stride, v[u]);
      }
    }
  block_reduce<double>(reduce_smem<double>(), acc, 1, sh.G, sh.nrhs, part);
}

// one warp per RHS: lane l sums the block partials l, l + 32, ... in order,
// then a fixed shuffle tree adds the lanes (deterministic)
template <typename A>
__global__ void finalize_kernel(const A* __restrict__ partials, int nblocks, int nrhs, A* out) {
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= nrhs) return;  // whole warps leave together
  const A s = sum_partials(partials, nblocks, nrhs, r, lane);
  if (lane == 0) out[r] = s;
}

// launch of finalize_kernel: 4 RHS (warps) per block
template <typename A>
void finalize(const A* partials, int nblocks, int nrhs, A* out, cudaStream_t st) {
  finalize_kernel<A><<<(nrhs + 3) / 4, 128, 0, st>>>(partials, nblocks, nrhs, out);
}

template <int PX, int PY>
__global__ void add_copy_kernel(const void* __restrict__ xv, void* __restrict__ yv, int64_t n, int add) {
  using EX = typename V2<typename BT<PX>::real>::t;
  using EY = typename V2<typename BT<PY>::real>::t;
  const EX* x = static_cast<const EX*>(xv);
  EY* y = static_cast<EY*>(yv);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    double2 v = ld(x + e);
    if (add) v = v + ld(y + e);
    st(y + e, v);
  }
}

Shape make_shape(const FieldRef& f, int R) {
  Shape s;
  s.R = R;
  s.nrhs = f.nrhs;
  s.G = f.nrhs / R;
  s.nchunks = f.n / R;
  return s;
}

// two complex FP32 elements (one 16-byte vector) per thread when nrhs is even
// and every operand is 16-byte aligned
int pick_r(const FieldRef& f, const void* other = nullptr, const void* third = nullptr) {
  const uintptr_t al = (uintptr_t)f.data | (uintptr_t)other | (uintptr_t)third;
  return (f.prec == PREC_SINGLE && f.nrhs % 2 == 0 && al % 16 == 0) ? 2 : 1;
}

// block size: a multiple of both G (so the RHS of a thread is fixed) and 32
int block_size(int G) {
  int b = G;
  while (b % 32) b += G;
  while (b < 192 && b * 2 <= 1024) b *= 2;
  return b;
}

int grid_for(int64_t nchunks, int block) {
  int64_t g = (nchunks + block - 1) / block;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, kMaxBlocks));
}

int device_sms() {
  static const int sms = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      n = 0;
    return n > 0 ? n : 152;
  }();
  return sms;
}

// Grid of a reducing kernel: one even wave.  1024 threads an SM always fit (at most 64 registers a thread,
// 32 KB of shared memory), so every SM takes the same number of blocks at once.  1024 blocks of 128 threads
// with 32 KB each made 1.12 waves of 6 blocks, and left the second half of the time to a tenth of the
// blocks: at 16^3x32 SU(4) nrhs 16, us, before / now: BiCGStab update 274 / 167, <x, y> with |x|^2 119 / 89,
// <x, y> 84 / 62.
int reduce_grid(int64_t nchunks, int block) {
  const int64_t g = (nchunks + block - 1) / block;
  const int64_t wave = (int64_t)device_sms() * std::max(1, 1024 / block);
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, std::min<int64_t>(wave, kMaxBlocks)));
}
template <typename A>
size_t reduce_bytes(int block, int R) {
  return (size_t)block * R * sizeof(A);
}

void check_field(const FieldRef& f) {
  QCU_REQUIRE(f.prec == PREC_DOUBLE || f.prec == PREC_SINGLE, QCU_ERR_UNSUPPORTED,
              "BLAS operands must be FP64 or FP32 fields");
  QCU_REQUIRE(f.nrhs >= 1 && f.n % f.nrhs == 0, QCU_ERR_INVALID_ARGUMENT, "bad field shape");
}

}  // namespace

int Blas::blocks_for(int64_t n) { return kMaxBlocks; }

void Blas::axpby(const double2* a, const FieldRef& x, const double2* b, const FieldRef& y, cudaStream_t st) {
  check_field(x);
  check_field(y);
  QCU_REQUIRE(x.n == y.n && x.nrhs == y.nrhs, QCU_ERR_INVALID_ARGUMENT, "axpby: shape mismatch");
  const int R = (x.prec == y.prec) ? pick_r(x, y.data) : 1;
  Shape s = make_shape(x, R);
  const int B = block_size(s.G);
  QCU_REQUIRE(B <= 1024, QCU_ERR_UNSUPPORTED, "nrhs too large for BLAS block");
  const int grid = grid_for(s.nchunks, B);
  if (x.prec == PREC_DOUBLE && y.prec == PREC_DOUBLE)
    axpby_kernel<PREC_DOUBLE, PREC_DOUBLE, 1, false><<<grid, B, 0, st>>>(a, x.data, b, y.data, s, nullptr);
  else if (x.prec == PREC_SINGLE && y.prec == PREC_SINGLE && R == 2)
    axpby_kernel<PREC_SINGLE, PREC_SINGLE, 2, false><<<grid, B, 0, st>>>(a, x.data, b, y.data, s, nullptr);
  else if (x.prec == PREC_SINGLE && y.prec == PREC_SINGLE)
    axpby_kernel<PREC_SINGLE, PREC_SINGLE, 1, false><<<grid, B, 0, st>>>(a, x.data, b, y.data, s, nullptr);
  else if (x.prec == PREC_SINGLE && y.prec == PREC_DOUBLE)
    axpby_kernel<PREC_SINGLE, PREC_DOUBLE, 1, false><<<grid, B, 0, st>>>(a, x.data, b, y.data, s, nullptr);
  else
    axpby_kernel<PREC_DOUBLE, PREC_SINGLE, 1, false><<<grid, B, 0, st>>>(a, x.data, b, y.data, s, nullptr);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::axpby_norm(const double2* a, const FieldRef& x, const double2* b, const FieldRef& y, double* out,
                      cudaStream_t st) {
  check_field(x);
  check_field(y);
  QCU_REQUIRE(x.n == y.n && x.nrhs == y.nrhs && x.prec == y.prec, QCU_ERR_INVALID_ARGUMENT,
              "axpby_norm: shape/precision mismatch");
  const int R = pick_r(x, y.data);
  Shape s = make_shape(x, R);
  const int B = block_size(s.G);
  QCU_REQUIRE(B <= 1024, QCU_ERR_UNSUPPORTED, "nrhs too large for BLAS block");
  const int grid = reduce_grid(s.nchunks, B);
  const size_t sm = reduce_bytes<double>(B, R);
  QCU_REQUIRE(grid <= max_blocks_, QCU_ERR_INVALID_ARGUMENT, "partials too small");
  if (x.prec == PREC_DOUBLE)
    axpby_kernel<PREC_DOUBLE, PREC_DOUBLE, 1, true><<<grid, B, sm, st>>>(a, x.data, b, y.data, s, partials_);
  else if (R == 2)
    axpby_kernel<PREC_SINGLE, PREC_SINGLE, 2, true><<<grid, B, sm, st>>>(a, x.data, b, y.data, s, partials_);
  else
    axpby_kernel<PREC_SINGLE, PREC_SINGLE, 1, true><<<grid, B, sm, st>>>(a, x.data, b, y.data, s, partials_);
  QCU_CHECK_CUDA(cudaGetLastError());
  finalize<double>(partials_, grid, x.nrhs, out, st);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::axpbypcz(const double2* a, const FieldRef& x, const double2* b, const FieldRef& y, const double2* c,
                    const FieldRef& z, cudaStream_t st) {
  check_field(x);
  QCU_REQUIRE(x.prec == y.prec && y.prec == z.prec && x.n == y.n && y.n == z.n, QCU_ERR_INVALID_ARGUMENT,
              "axpbypcz: shape/precision mismatch");
  const int R = pick_r(x, y.data, z.data);
  Shape s = make_shape(x, R);
  const int B = block_size(s.G);
  QCU_REQUIRE(B <= 1024, QCU_ERR_UNSUPPORTED, "nrhs too large for BLAS block");
  const int grid = grid_for(s.nchunks, B);
  if (x.prec == PREC_DOUBLE)
    axpbypcz_kernel<PREC_DOUBLE, 1><<<grid, B, 0, st>>>(a, x.data, b, y.data, c, z.data, s);
  else if (R == 2)
    axpbypcz_kernel<PREC_SINGLE, 2><<<grid, B, 0, st>>>(a, x.data, b, y.data, c, z.data, s);
  else
    axpbypcz_kernel<PREC_SINGLE, 1><<<grid, B, 0, st>>>(a, x.data, b, y.data, c, z.data, s);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::norm2(const FieldRef& x, double* out, cudaStream_t st, bool exact) {
  check_field(x);
  const int R = pick_r(x);
  Shape s = make_shape(x, R);
  const int B = block_size(s.G);
  QCU_REQUIRE(B <= 1024, QCU_ERR_UNSUPPORTED, "nrhs too large for BLAS block");
  const int grid = reduce_grid(s.nchunks, B);
  const size_t sm = reduce_bytes<double>(B, R);
  if (x.prec == PREC_DOUBLE)
    reduce_kernel<PREC_DOUBLE, PREC_DOUBLE, 1, 0><<<grid, B, sm, st>>>(x.data, x.data, s, partials_);
  else if (R == 2 && exact)
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 2, 0><<<grid, B, sm, st>>>(x.data, x.data, s, partials_);
  else if (R == 2)
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 2, 0, true><<<grid, B, sm, st>>>(x.data, x.data, s, partials_);
  else if (exact)
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 1, 0><<<grid, B, sm, st>>>(x.data, x.data, s, partials_);
  else
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 1, 0, true><<<grid, B, sm, st>>>(x.data, x.data, s, partials_);
  QCU_CHECK_CUDA(cudaGetLastError());
  finalize<double>(partials_, grid, x.nrhs, out, st);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::cdot(const FieldRef& x, const FieldRef& y, double2* out, cudaStream_t st) {
  check_field(x);
  check_field(y);
  QCU_REQUIRE(x.n == y.n && x.nrhs == y.nrhs && x.prec == y.prec, QCU_ERR_INVALID_ARGUMENT,
              "cdot: shape/precision mismatch");
  const int R = pick_r(x, y.data);
  Shape s = make_shape(x, R);
  const int B = block_size(s.G);
  QCU_REQUIRE(B <= 1024, QCU_ERR_UNSUPPORTED, "nrhs too large for BLAS block");
  const int grid = reduce_grid(s.nchunks, B);
  const size_t sm = reduce_bytes<double2>(B, R);
  double2* p2 = reinterpret_cast<double2*>(partials_);
  if (x.prec == PREC_DOUBLE)
    reduce_kernel<PREC_DOUBLE, PREC_DOUBLE, 1, 1><<<grid, B, sm, st>>>(x.data, y.data, s, p2);
  else if (R == 2)
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 2, 1, true><<<grid, B, sm, st>>>(x.data, y.data, s, p2);
  else
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 1, 1, true><<<grid, B, sm, st>>>(x.data, y.data, s, p2);
  QCU_CHECK_CUDA(cudaGetLastError());
  finalize<double2>(p2, grid, x.nrhs, out, st);
  QCU_CHECK_CUDA(cudaGetLastError());
}

double* Blas::norms(int k) const { return partials_ + (size_t)(2 + k) * max_blocks_ * QCU_MAX_RHS; }

namespace {
struct Launch {
  Shape s;
  int R, block, grid;   // grid of a kernel without reductions
  int rgrid;            // of a reducing kernel
  size_t norm_sm, dot_sm;  // its shared memory
};
Launch plan(const FieldRef& f, int R) {
  Launch l;
  l.R = R;
  l.s = make_shape(f, R);
  l.block = block_size(l.s.G);
  QCU_REQUIRE(l.block <= 1024, QCU_ERR_UNSUPPORTED, "nrhs too large for BLAS block");
  l.grid = grid_for(l.s.nchunks, l.block);
  l.rgrid = reduce_grid(l.s.nchunks, l.block);
  l.norm_sm = reduce_bytes<double>(l.block, R);
  l.dot_sm = reduce_bytes<double2>(l.block, R);
  return l;
}
void check_same(const FieldRef& a, const FieldRef& b, const char* what) {
  check_field(a);
  check_field(b);
  QCU_REQUIRE(a.n == b.n && a.nrhs == b.nrhs && a.prec == b.prec, QCU_ERR_INVALID_ARGUMENT,
              std::string(what) + ": shape/precision mismatch");
}
}  // namespace

Partials Blas::norm2_partials(const FieldRef& x, cudaStream_t st) {
  check_field(x);
  const Launch l = plan(x, pick_r(x));
  double* p = norms(0);
  if (x.prec == PREC_DOUBLE)
    reduce_kernel<PREC_DOUBLE, PREC_DOUBLE, 1, 0><<<l.rgrid, l.block, l.norm_sm, st>>>(x.data, x.data, l.s, p);
  else if (l.R == 2)
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 2, 0, true><<<l.rgrid, l.block, l.norm_sm, st>>>(x.data, x.data, l.s, p);
  else
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 1, 0, true><<<l.rgrid, l.block, l.norm_sm, st>>>(x.data, x.data, l.s, p);
  QCU_CHECK_CUDA(cudaGetLastError());
  return Partials{p, nullptr, nullptr, l.rgrid};
}

Partials Blas::dot_partials(const FieldRef& x, const FieldRef& y, cudaStream_t st) {
  check_same(x, y, "dot");
  const Launch l = plan(x, pick_r(x, y.data));
  if (x.prec == PREC_DOUBLE)
    reduce_kernel<PREC_DOUBLE, PREC_DOUBLE, 1, 1><<<l.rgrid, l.block, l.dot_sm, st>>>(x.data, y.data, l.s, dots());
  else if (l.R == 2)
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 2, 1, true><<<l.rgrid, l.block, l.dot_sm, st>>>(x.data, y.data, l.s, dots());
  else
    reduce_kernel<PREC_SINGLE, PREC_SINGLE, 1, 1, true><<<l.rgrid, l.block, l.dot_sm, st>>>(x.data, y.data, l.s, dots());
  QCU_CHECK_CUDA(cudaGetLastError());
  return Partials{nullptr, nullptr, dots(), l.rgrid};
}

Partials Blas::dot_norm(const FieldRef& x, const FieldRef& y, cudaStream_t st) {
  check_same(x, y, "dot_norm");
  const Launch l = plan(x, pick_r(x, y.data));
  if (x.prec == PREC_DOUBLE)
    dot_norm_kernel<PREC_DOUBLE, 1><<<l.rgrid, l.block, l.dot_sm, st>>>(x.data, y.data, l.s, norms(0), dots());
  else if (l.R == 2)
    dot_norm_kernel<PREC_SINGLE, 2><<<l.rgrid, l.block, l.dot_sm, st>>>(x.data, y.data, l.s, norms(0), dots());
  else
    dot_norm_kernel<PREC_SINGLE, 1><<<l.rgrid, l.block, l.dot_sm, st>>>(x.data, y.data, l.s, norms(0), dots());
  QCU_CHECK_CUDA(cudaGetLastError());
  return Partials{norms(0), nullptr, dots(), l.rgrid};
}

Partials Blas::cg_update(const double2* a, const FieldRef& q, const FieldRef& s, const FieldRef& w, const FieldRef& r,
                         cudaStream_t st) {
  check_same(q, s, "cg_update");
  check_same(w, r, "cg_update");
  check_same(q, r, "cg_update");
  const int R = std::min(pick_r(q, s.data), pick_r(w, r.data));
  const Launch l = plan(q, R);
  if (q.prec == PREC_DOUBLE)
    cg_update_kernel<PREC_DOUBLE, 1><<<l.rgrid, l.block, l.norm_sm, st>>>(a, q.data, s.data, w.data, r.data, l.s, norms(0), norms(1));
  else if (R == 2)
    cg_update_kernel<PREC_SINGLE, 2><<<l.rgrid, l.block, l.norm_sm, st>>>(a, q.data, s.data, w.data, r.data, l.s, norms(0), norms(1));
  else
    cg_update_kernel<PREC_SINGLE, 1><<<l.rgrid, l.block, l.norm_sm, st>>>(a, q.data, s.data, w.data, r.data, l.s, norms(0), norms(1));
  QCU_CHECK_CUDA(cudaGetLastError());
  return Partials{norms(0), norms(1), nullptr, l.rgrid};
}

void Blas::cg_direction(const double2* a, const double2* b, const FieldRef& r, const FieldRef& p, const FieldRef& x,
                        cudaStream_t st) {
  check_same(r, p, "cg_direction");
  check_same(p, x, "cg_direction");
  const Launch l = plan(r, pick_r(r, p.data, x.data));
  if (r.prec == PREC_DOUBLE)
    cg_direction_kernel<PREC_DOUBLE, 1><<<l.grid, l.block, 0, st>>>(a, b, r.data, p.data, x.data, l.s);
  else if (l.R == 2)
    cg_direction_kernel<PREC_SINGLE, 2><<<l.grid, l.block, 0, st>>>(a, b, r.data, p.data, x.data, l.s);
  else
    cg_direction_kernel<PREC_SINGLE, 1><<<l.grid, l.block, 0, st>>>(a, b, r.data, p.data, x.data, l.s);
  QCU_CHECK_CUDA(cudaGetLastError());
}

Partials Blas::bicg_update(const double2* a, const double2* o, const FieldRef& p, const FieldRef& s,
                           const FieldRef& t, const FieldRef& r0, const FieldRef& x, cudaStream_t st) {
  check_same(p, s, "bicg_update");
  check_same(t, r0, "bicg_update");
  check_same(p, x, "bicg_update");
  check_same(p, t, "bicg_update");
  const int R = std::min(pick_r(p, s.data, t.data), pick_r(r0, x.data));
  const Launch l = plan(p, R);
  if (p.prec == PREC_DOUBLE)
    bicg_update_kernel<PREC_DOUBLE, 1><<<l.rgrid, l.block, l.dot_sm, st>>>(a, o, p.data, s.data, t.data, r0.data, x.data, l.s, norms(0), dots());
  else if (R == 2)
    bicg_update_kernel<PREC_SINGLE, 2><<<l.rgrid, l.block, l.dot_sm, st>>>(a, o, p.data, s.data, t.data, r0.data, x.data, l.s, norms(0), dots());
  else
    bicg_update_kernel<PREC_SINGLE, 1><<<l.rgrid, l.block, l.dot_sm, st>>>(a, o, p.data, s.data, t.data, r0.data, x.data, l.s, norms(0), dots());
  QCU_CHECK_CUDA(cudaGetLastError());
  return Partials{norms(0), nullptr, dots(), l.rgrid};
}

// the masked moves keep one RHS per thread (R = 1), so a thread is selected or leaves at once
void Blas::fold(const int* sel, const FieldRef& xl, const FieldRef& xh, const FieldRef& be, const FieldRef& d,
                cudaStream_t st) {
  check_field(xl);
  check_field(xh);
  QCU_REQUIRE(xl.n == xh.n && xh.prec == PREC_DOUBLE, QCU_ERR_INVALID_ARGUMENT, "fold: shape/precision mismatch");
  const Launch l = plan(xl, 1);
  double2 *h = static_cast<double2*>(xh.data), *dd = static_cast<double2*>(d.data);
  const double2* b = static_cast<const double2*>(be.data);
  if (xl.prec == PREC_DOUBLE)
    fold_kernel<PREC_DOUBLE><<<l.grid, l.block, 0, st>>>(sel, xl.data, h, b, dd, l.s);
  else
    fold_kernel<PREC_SINGLE><<<l.grid, l.block, 0, st>>>(sel, xl.data, h, b, dd, l.s);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::select_copy(const int* sel, const FieldRef& x, const FieldRef& y, const FieldRef& z, cudaStream_t st) {
  check_field(y);
  QCU_REQUIRE(!x.data || x.n == y.n, QCU_ERR_INVALID_ARGUMENT, "select_copy: shape mismatch");
  const Launch l = plan(y, 1);
  const int px = x.data ? x.prec : y.prec;
  if (px == PREC_DOUBLE && y.prec == PREC_DOUBLE)
    select_copy_kernel<PREC_DOUBLE, PREC_DOUBLE><<<l.grid, l.block, 0, st>>>(sel, x.data, y.data, z.data, l.s);
  else if (px == PREC_DOUBLE)
    select_copy_kernel<PREC_DOUBLE, PREC_SINGLE><<<l.grid, l.block, 0, st>>>(sel, x.data, y.data, z.data, l.s);
  else if (y.prec == PREC_DOUBLE)
    select_copy_kernel<PREC_SINGLE, PREC_DOUBLE><<<l.grid, l.block, 0, st>>>(sel, x.data, y.data, z.data, l.s);
  else
    select_copy_kernel<PREC_SINGLE, PREC_SINGLE><<<l.grid, l.block, 0, st>>>(sel, x.data, y.data, z.data, l.s);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::residual(const int* sel, const FieldRef& x, const FieldRef& y, double* out, cudaStream_t st) {
  check_field(x);
  check_field(y);
  QCU_REQUIRE(x.n == y.n && x.prec == PREC_DOUBLE, QCU_ERR_INVALID_ARGUMENT, "residual: shape/precision mismatch");
  const Launch l = plan(x, 1);
  const double2* xp = static_cast<const double2*>(x.data);
  if (y.prec == PREC_DOUBLE)
    residual_kernel<PREC_DOUBLE><<<l.rgrid, l.block, l.norm_sm, st>>>(sel, xp, y.data, l.s, norms(0));
  else
    residual_kernel<PREC_SINGLE><<<l.rgrid, l.block, l.norm_sm, st>>>(sel, xp, y.data, l.s, norms(0));
  QCU_CHECK_CUDA(cudaGetLastError());
  finalize<double>(norms(0), l.rgrid, x.nrhs, out, st);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::add_to(const FieldRef& lo, const FieldRef& hi, cudaStream_t st) {
  check_field(lo);
  check_field(hi);
  QCU_REQUIRE(lo.n == hi.n, QCU_ERR_INVALID_ARGUMENT, "add_to: shape mismatch");
  const int grid = grid_for(lo.n, 256);
  if (lo.prec == PREC_SINGLE && hi.prec == PREC_DOUBLE)
    add_copy_kernel<PREC_SINGLE, PREC_DOUBLE><<<grid, 256, 0, st>>>(lo.data, hi.data, lo.n, 1);
  else if (lo.prec == PREC_DOUBLE && hi.prec == PREC_DOUBLE)
    add_copy_kernel<PREC_DOUBLE, PREC_DOUBLE><<<grid, 256, 0, st>>>(lo.data, hi.data, lo.n, 1);
  else if (lo.prec == PREC_SINGLE && hi.prec == PREC_SINGLE)
    add_copy_kernel<PREC_SINGLE, PREC_SINGLE><<<grid, 256, 0, st>>>(lo.data, hi.data, lo.n, 1);
  else
    add_copy_kernel<PREC_DOUBLE, PREC_SINGLE><<<grid, 256, 0, st>>>(lo.data, hi.data, lo.n, 1);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::copy(const FieldRef& x, const FieldRef& y, cudaStream_t st) {
  check_field(x);
  check_field(y);
  QCU_REQUIRE(x.n == y.n, QCU_ERR_INVALID_ARGUMENT, "copy: shape mismatch");
  const int grid = grid_for(x.n, 256);
  if (x.prec == PREC_SINGLE && y.prec == PREC_DOUBLE)
    add_copy_kernel<PREC_SINGLE, PREC_DOUBLE><<<grid, 256, 0, st>>>(x.data, y.data, x.n, 0);
  else if (x.prec == PREC_DOUBLE && y.prec == PREC_DOUBLE)
    add_copy_kernel<PREC_DOUBLE, PREC_DOUBLE><<<grid, 256, 0, st>>>(x.data, y.data, x.n, 0);
  else if (x.prec == PREC_SINGLE && y.prec == PREC_SINGLE)
    add_copy_kernel<PREC_SINGLE, PREC_SINGLE><<<grid, 256, 0, st>>>(x.data, y.data, x.n, 0);
  else
    add_copy_kernel<PREC_DOUBLE, PREC_SINGLE><<<grid, 256, 0, st>>>(x.data, y.data, x.n, 0);
  QCU_CHECK_CUDA(cudaGetLastError());
}

void Blas::zero(const FieldRef& x, cudaStream_t st) {
  QCU_CHECK_CUDA(cudaMemsetAsync(x.data, 0, (size_t)x.n * prec_complex_bytes(x.prec), st));
}

}  // namespace qcu
