// FP64 Wilson hop with the colour multiply in block fixed point.
//
// The FP64 pipe of sm_103a takes 2 multiply-adds per clock and SM, and 840 of them a site and RHS kept
// it 97% busy at SU(3).  32 x 32 -> 64-bit integer multiply-adds run at about 16 times that rate.  So
// only the projection (12 operations a hop at SU(3)) is left on the FP64 pipe, and the colour multiply
// and the sum over hops are done in integers:
//
//   projected spinor   the 4N real parts of a neighbour's two rows, 59 bits over their common exponent
//   link               its 2N^2 real parts, 59 bits over theirs (SU(8): both 58)
//   product            limbs of 28 and 31 bits, the low ones balanced (SU(8): 28 and 30), the three larger limb
//                      products summed exactly in two 64-bit accumulators a component; only low x low (2^-58 of
//                      the operands' largest parts, at most) is left out
//   sum over hops      64-bit integers over the largest hop's exponent
//   result             rounded once to double (nearest even); the xpay epilogue stays FP64
//
// No sum can overflow (the bounds stand beside the constants), and none rounds before the last step
// but by the right shifts to the accumulator's unit.  Relative L2 error against quad precision on random
// fields: SU(3), SU(4) 0.71e-16, SU(5) to SU(8) 0.74e-16, where the FP64 multiply-adds have 1.46e-16, 1.54e-16
// and 1.61e-16 to 1.80e-16.
//
// One hop, us, FP64 multiply-adds / this: SU(3) 24^3x48 nrhs 12 5763 / 1747, SU(4) 16^3x32 nrhs 16
// 2460 / 779, SU(3) 14x10x6x18 nrhs 5 62 / 27; in the split form SU(3) 12^3x24 nrhs 1 46 / 21, SU(6)
// 16^3x32 nrhs 16 4978 / 2486, SU(8) 8378 / 4187, SU(6) 8^3x16 nrhs 1 99 / 19.  It is bound by
// instruction issue and latency (SU(3): 9500 instructions a warp, 216 wide multiply-adds a hop; issue 54%, the
// integer pipe 51%, FP64 35% busy, 15 warps an SM); the small sizes by the latency of one warp a scheduler.
//
// A common exponent keeps the digits of a part only down to its unit.  So a site takes the FP64 multiply-adds
// (fp64_site) when a part of its result is made up of small products only (fix_parts_hold), when its hops lie more
// than kFixSpan binades apart, when anything it reads is infinite or NaN, and when the result could leave the
// normal range.  Where a field's structure sends every site there, a hop takes the time of both: one-colour
// spinors on near-unit links, us, against FP64 multiply-adds alone: SU(3) 24^3x48 nrhs 12 6850 / 5763, SU(4)
// 16^3x32 nrhs 16 2970 / 2460, SU(6) 16^3x32 nrhs 16 8340 / 4978.
#pragma once

namespace qcu {
namespace detail {

// the FP64 SU(N) hops that run in fixed point; from SU(5) on only in the split form (a thread cannot hold
// the sums of 8N parts)
__host__ __device__ constexpr bool fix_hop(int prec, int N) { return prec == PREC_DOUBLE && N >= 3 && N <= 8; }
__host__ __device__ constexpr bool fix_split_only(int N) { return N > 4; }

// The hops of a site may lie this many binades apart (the shift that asr takes).
constexpr int kFixSpan = 31;

// A part is |F| < 2^B over its common exponent, B = 64 - kFixShift, as limbs F = hi 2^s + lo, s = kFixSplit,
// |hi| <= 2^(B - s), |lo| <= 2^(s - 1).  Over a component's 2N products:
//   high  |sum uh hh|            <= 2N 2^(2B - 2s)
//   mid   |sum uh hl + ul hh|    <= 2N 2^B          (N = 7: 2^62.8, and the rounding bits fit)
// A hop's product in the accumulator's unit 2^(2s - x), x = kFixExtra, is (high << x) + (mid >> (s - x)).  Its
// exact value is at most 2N F^2 / 2^(2s - x) <= 2^60 - 2^8 for every N, and what is left out and rounded is at
// most 5 units, so eight of them stay below 2^63.
template <int N>
constexpr uint32_t kFixShift = N <= 7 ? 5 : 6;  // right shift of a mantissa whose top bit is bit 63
template <int N>
constexpr uint32_t kFixSplit = N <= 7 ? 31 : 30;
template <int N>
constexpr uint32_t kFixExtra = N <= 4 ? 1 : 0;

// A part of the result holds when its eight products add up to this many times 2^48 units (2^57, 2^56 for N > 4,
// is a largest product): fix_parts_hold.
template <int N>
constexpr uint32_t kFixMag = N <= 4 ? 24 : 32;

struct Limbs {
  int32_t hi, lo;
};

__device__ __forceinline__ uint32_t biased_exp(double x) { return ((uint32_t)__double2hiint(x) >> 20) & 0x7ffu; }

// x over the biased exponent es - kFixShift of the largest part; flip 0x80000000 negates.  A zero's shift is es,
// so es must be above 63.
template <int N>
__device__ __forceinline__ Limbs to_limbs(double x, uint32_t es, uint32_t flip) {
  constexpr uint32_t kSplit = kFixSplit<N>;
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mh = __funnelshift_l(lo, hi, 11) | 0x80000000u, ml = lo << 11;
  const uint32_t s = es - ((hi >> 20) & 0x7ffu);
  unsigned long long f;
  asm("shr.u64 %0, %1, %2;" : "=l"(f) : "l"(((unsigned long long)mh << 32) | ml), "r"(s));  // shifts above 63 give 0
  const int32_t sign = ((int32_t)(hi ^ flip) >> 31) | 1;
  const uint32_t top = (uint32_t)((f + (1u << (kSplit - 1))) >> kSplit);
  return Limbs{(int32_t)top * sign, (int32_t)((uint32_t)f - (top << kSplit)) * sign};
}

// v >> s for s up to 31, which a site's shifts are while its hops lie within kFixSpan (or v is 0); with larger
// ones, whose sites take FP64, it is any value (a 64-bit shift instruction pair costs 1.5% of the hop)
__device__ __forceinline__ long long asr(long long v, uint32_t s) {
  const int32_t h = (int32_t)(v >> 32);
  const uint32_t lo = __funnelshift_r((uint32_t)v, (uint32_t)h, s);
  return (long long)(((unsigned long long)(uint32_t)(h >> (s & 31u)) << 32) | lo);
}

// a sum T over hops of largest exponent E is T 2^(E - 2172 + 2 kFixShift + 2 kFixSplit - kFixExtra):
// from_fix(T, E + kFixBias)
template <int N>
constexpr int kFixBias = 2 * (int)kFixShift<N> + 2 * (int)kFixSplit<N> - (int)kFixExtra<N> - 1087;
// T as a double, rounded to nearest even: the result's biased exponent is e + 1 - clz(|T|); T = 0 gives +0
__device__ __forceinline__ double from_fix(long long T, int e) {
  const uint32_t sg = (uint32_t)((unsigned long long)T >> 63);
  const unsigned long long m0 = (unsigned long long)(T < 0 ? -T : T);
  const int z = __clzll((long long)m0);
  const unsigned long long m = m0 << (z & 63);
  unsigned long long q = m >> 11;
  const uint32_t rem = (uint32_t)m & 0x7ffu;
  q += (rem + ((uint32_t)q & 1u)) > 0x400u ? 1ull : 0ull;
  const uint32_t qh = (uint32_t)(q >> 32) + ((uint32_t)(e - z) << 20) + (sg << 31);
  return m0 ? __hiloint2double((int)qh, (int)(uint32_t)q) : 0.0;
}

// One link as limbs, in the order in which the hop multiplies (backward: conjugate transposed; the
// boundary sign included), and the exponent of its largest part.
template <int N>
struct FixLink {
  int4 u[N * N];  // re.hi, re.lo, im.hi, im.lo
  uint32_t e;
};

// where hop h's link lies, and the signs of its parts
template <int N>
struct FixLinkAt {
  const double2* lb;
  uint32_t sa, sb;  // strides of a and b
  uint32_t rf, jf;  // sign flips of the real and imaginary parts
  __device__ __forceinline__ FixLinkAt(const DslashArgs& A, const SiteXyzt& X, int h, uint32_t nb) {
    const int mu = h >> 1;
    const bool bwd = h & 1;
    const uint32_t vh = (uint32_t)A.geo.vh, p = (uint32_t)A.parity;
    lb = static_cast<const double2*>(A.gauge) +
         ((mu * 2u + (bwd ? 1u - p : p)) * (uint32_t)(N * N) * vh + (bwd ? nb : X.site));
    sa = (bwd ? 1u : (uint32_t)N) * vh;
    sb = (bwd ? (uint32_t)N : 1u) * vh;
    const bool wrap = mu == 3 && A.antiperiodic_t && (bwd ? X.t == 0 : X.t == (uint32_t)A.geo.L[3] - 1);
    rf = wrap ? 0x80000000u : 0u;
    jf = rf ^ (bwd ? 0x80000000u : 0u);
  }
  __device__ __forceinline__ double2 load(int a, int b) const { return __ldg(lb + (a * sa + b * sb)); }
  __device__ __forceinline__ int4 limbs(double2 v, uint32_t e) const {
    const Limbs r = to_limbs<N>(v.x, e + kFixShift<N>, rf), i = to_limbs<N>(v.y, e + kFixShift<N>, jf);
    return make_int4(r.hi, r.lo, i.hi, i.lo);
  }
};

template <int N>
__device__ __forceinline__ FixLink<N> load_fix_link(const DslashArgs& A, const SiteXyzt& X, int h, uint32_t nb) {
  const FixLinkAt<N> at(A, X, h, nb);
  double2 u[N][N];
  FixLink<N> L;
  L.e = 0;
#pragma unroll
  for (int a = 0; a < N; a++)
#pragma unroll
    for (int b = 0; b < N; b++) u[a][b] = at.load(a, b);
#pragma unroll
  for (int a = 0; a < N; a++)
#pragma unroll
    for (int b = 0; b < N; b++) L.e = max(L.e, max(biased_exp(u[a][b].x), biased_exp(u[a][b].y)));
#pragma unroll
  for (int a = 0; a < N; a++)
#pragma unroll
    for (int b = 0; b < N; b++) L.u[a * N + b] = at.limbs(u[a][b], L.e);
  return L;
}

// Links of a block's sites in shared memory, converted once for all the RHS of a site (in each thread the
// conversion was a third of the instructions: SU(3) 24^3x48 nrhs 12 3140 us, with 24 parts a hop converted
// instead of the 12 projected ones, against 1685 as the rest of the kernel was then): [site][hop] records of the N^2 elements (int4), their
// negated imaginary parts (int2), and the exponent
template <int N>
constexpr uint32_t kFixRec = N * N + N * N / 2 + 1;
template <int N>
constexpr uint32_t kFixSite = (8 * kFixRec<N>) | 1;  // int4; odd, so that two sites' records lie in other banks

// the FP64 multiply-adds, out of line: predicated FP64 operations would hold the pipe in every warp
template <int N>
__device__ __noinline__ void fp64_site(const DslashArgs& A, const SiteXyzt& X, uint32_t rhs) {
  site_rhs<PREC_DOUBLE, N, 1, false, false>(A, X, rhs, 0, 1);
}

// the sums of one site and RHS
template <int N>
struct FixAcc {
  long long up[2][N][2];  // rows 0 and 1
  long long lo[2][N][2];  // the rows that take the products of rows 0 and 1 (3 and 2 for x and y, 2 and 3 for z and t)
  uint32_t mag[N] = {};     // sums of fix_mag of the products of row 0 (low half) and row 1: of x and y, then of z and t
  uint32_t mag_xy[N];       // those of x and y, over the exponent E_xy
  int E = 0, E_xy = 0;      // largest exponent of a hop; of one of x and y
  uint32_t rows = 0;        // bit i: projected row i is not zero in some hop of x or y; bit 2 + i: of z or t
  bool bad = false;
};

// |re| and |im| of a product, whichever is smaller, in 2^32 units
__device__ __forceinline__ uint32_t fix_least(long long re, long long im) {
  return (uint32_t)min(abs((int32_t)(re >> 32)), abs((int32_t)(im >> 32)));
}
// both halves of m shifted right by s
__device__ __forceinline__ uint32_t fix_mag_shift(uint32_t m, uint32_t s) {
  return s > 15u ? 0u : (m >> s) & ((0xffffu >> s) * 0x10001u);
}

// s = +1 / -1 of hop h as a sign bit, and the sign s g(u_perm) with which the product of row i enters the lower row
__device__ __forceinline__ uint32_t fix_sign(const DslashArgs& A, int h) {
  return ((h & 1) != (A.dagger != 0)) ? 0u : 0x80000000u;
}
__device__ __forceinline__ long long fix_lower_sign(const DslashArgs& A, int h, int i) {  // 0 or -1
  const int mu = h >> 1;
  const uint32_t g = fix_sign(A, h) ^ ((i ? mu == 0 : mu != 3) ? 0x80000000u : 0u);
  return (long long)(int32_t)g >> 31;
}

// the neighbour's spinor; rows 2 and 3 (y) in the order in which rows 0 and 1 (x) meet them
template <int N>
__device__ __forceinline__ void fix_load(double2 (&x)[2][N], double2 (&y)[2][N], const DslashArgs& A, uint32_t nb,
                                         uint32_t rhs, int mu) {
  const uint32_t nrhs = (uint32_t)A.nrhs, cs_bytes = (uint32_t)A.geo.vh * nrhs * 16u;
  const char* base = reinterpret_cast<const char*>(static_cast<const double2*>(A.in) + (nb * nrhs + rhs));
  const char* low = base + (uint64_t)(2 * N) * cs_bytes;
  const uint64_t up = (uint64_t)N * cs_bytes, r0 = mu < 2 ? up : 0u, r1 = up - r0;
#pragma unroll
  for (int a = 0; a < N; a++) {
    x[0][a] = __ldg(reinterpret_cast<const double2*>(base + (uint64_t)a * cs_bytes));
    x[1][a] = __ldg(reinterpret_cast<const double2*>(base + (uint64_t)(N + a) * cs_bytes));
    y[0][a] = __ldg(reinterpret_cast<const double2*>(low + r0 + (uint64_t)a * cs_bytes));
    y[1][a] = __ldg(reinterpret_cast<const double2*>(low + r1 + (uint64_t)a * cs_bytes));
  }
}
// h_u = x_u + s g(u) y_u, into x
template <int N>
__device__ __forceinline__ void fix_project(double2 (&x)[2][N], const double2 (&y)[2][N], const DslashArgs& A, int h) {
  const int mu = h >> 1;
  const bool imag = !(mu & 1);
  const uint32_t sgn = fix_sign(A, h);
  const double k0 = __hiloint2double((int)(0x3ff00000u | (sgn ^ (mu == 1 ? 0x80000000u : 0u))), 0);
  const double k1 = __hiloint2double((int)(0x3ff00000u | (sgn ^ (mu == 2 ? 0x80000000u : 0u))), 0);
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int a = 0; a < N; a++) {
      const double k = i ? k1 : k0;
      x[i][a].x = fma(imag ? -k : k, imag ? y[i][a].y : y[i][a].x, x[i][a].x);
      x[i][a].y = fma(k, imag ? y[i][a].x : y[i][a].y, x[i][a].y);
    }
}

// Hop h: out.begin(exponent, bits of the rows that are not zero, not for fixed point), then
// out.put(a, t) for the products of colour a, t[projected row][re, im], in the hop's own unit.
template <int N, bool SHARED, typename Out>
__device__ __forceinline__ void fix_hop_products(Out& out, const DslashArgs& A, const SiteXyzt& X, uint32_t rhs,
                                                 const int4* links, int h) {
  const int mu = h >> 1;
  const uint32_t nb = X.neighbour(A, h);
  double2 x[2][N], y[2][N];
  fix_load<N>(x, y, A, nb, rhs, mu);
  // SHARED: records in shared memory; else in registers, or from SU(5) on, where they would not fit, read
  // twice, for the exponent and (from L1) for each product
  constexpr bool kTwice = !SHARED && fix_split_only(N);
  FixLink<SHARED || kTwice ? 1 : N> own;
  const FixLinkAt<N> at(A, X, h, nb);
  const int4* rec = links + h * kFixRec<N>;
  uint32_t eu;
  if constexpr (SHARED) {
    eu = (uint32_t)reinterpret_cast<const int2*>(rec + N * N)[N * N].x;
  } else if constexpr (kTwice) {
    eu = 0;
#pragma unroll 4
    for (int k = 0; k < N * N; k++) {
      const double2 v = at.load(k / N, k % N);
      eu = max(eu, max(biased_exp(v.x), biased_exp(v.y)));
    }
  } else {
    own = load_fix_link<N>(A, X, h, nb);
    eu = own.e;
  }

  fix_project<N>(x, y, A, h);
  uint32_t er[2] = {0, 0};  // the rows' largest exponents
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int a = 0; a < N; a++) er[i] = max(er[i], max(biased_exp(x[i][a].x), biased_exp(x[i][a].y)));
  const uint32_t ep = max(er[0], er[1]);
  bool bad = ep == 0x7ffu || eu == 0x7ffu || eu < 200u;
  int eh = (int)(ep + eu);
  uint32_t es = ep + kFixShift<N>;
  if (er[0] == 0 || er[1] == 0) {  // rows of zeros add nothing; of subnormal parts: FP64
#pragma unroll
    for (int i = 0; i < 2; i++) {
      long long any = 0;
#pragma unroll
      for (int a = 0; a < N; a++) any |= __double_as_longlong(x[i][a].x) | __double_as_longlong(x[i][a].y);
      bad |= er[i] == 0 && (any << 1) != 0;
    }
  }
  if (es < 64) {  // no shift takes a zero's implicit leading bit away (to_limbs): zeros only, or FP64
    bad |= ep != 0;
    eh = 0;
    es = 64;
  }
  Limbs hr[2][N], hi[2][N];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int a = 0; a < N; a++) {
      hr[i][a] = to_limbs<N>(x[i][a].x, es, 0u);
      hi[i][a] = to_limbs<N>(x[i][a].y, es, 0u);
    }

  out.begin(eh, (er[0] ? 1u : 0u) | (er[1] ? 2u : 0u), bad);

#pragma unroll fix_split_only(N) ? 1 : N
  for (int a = 0; a < N; a++) {
    long long H[2][2], M[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int c = 0; c < 2; c++) H[i][c] = 0, M[i][c] = 1ll << (kFixSplit<N> - kFixExtra<N> - 1);
#pragma unroll
    for (int b = 0; b < N; b++) {
      int4 u;
      int2 n;  // the negated imaginary part
      if constexpr (SHARED) {
        u = rec[a * N + b];
        n = reinterpret_cast<const int2*>(rec + N * N)[a * N + b];
      } else {
        u = kTwice ? at.limbs(at.load(a, b), eu) : own.u[kTwice ? 0 : a * N + b];
        n = make_int2(-u.z, -u.w);
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const Limbs re = hr[i][b], im = hi[i][b];
        H[i][0] += (long long)u.x * re.hi;
        M[i][0] += (long long)u.x * re.lo;
        M[i][0] += (long long)u.y * re.hi;
        H[i][0] += (long long)n.x * im.hi;
        M[i][0] += (long long)n.x * im.lo;
        M[i][0] += (long long)n.y * im.hi;
        H[i][1] += (long long)u.x * im.hi;
        M[i][1] += (long long)u.x * im.lo;
        M[i][1] += (long long)u.y * im.hi;
        H[i][1] += (long long)u.z * re.hi;
        M[i][1] += (long long)u.z * re.lo;
        M[i][1] += (long long)u.w * re.hi;
      }
    }
    long long t[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int c = 0; c < 2; c++) t[i][c] = (H[i][c] << kFixExtra<N>) + (M[i][c] >> (kFixSplit<N> - kFixExtra<N>));
    out.put(a, t);
  }
}

// hop h added to a site's sums
template <int N>
struct FixAdd {
  FixAcc<N>& S;
  const DslashArgs& A;
  int h;
  uint32_t d = 0;  // the hop's shift to the sums' exponent
  // brings the sums so far and this hop to the larger exponent
  __device__ __forceinline__ void begin(int eh, uint32_t rows, bool bad) {
    S.bad |= bad;
    S.rows |= rows << (h < 4 ? 0 : 2);
    d = (uint32_t)(S.E - eh);
    if (eh > S.E) {
      const uint32_t up = (uint32_t)(eh - S.E);
      S.bad |= S.E != 0 && up > kFixSpan;
#pragma unroll
      for (int a = 0; a < N; a++) {
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int c = 0; c < 2; c++) {
            S.up[i][a][c] = asr(S.up[i][a][c], up);
            S.lo[i][a][c] = asr(S.lo[i][a][c], up);
          }
        S.mag[a] = fix_mag_shift(S.mag[a], up);
      }
      S.E = eh;
      d = 0;
    }
    S.bad |= eh != 0 && d > kFixSpan;
  }
  // lower rows: lo(u) += s g(u_perm) (im ? i : 1) t_u
  __device__ __forceinline__ void put(int a, const long long (&t)[2][2]) {
    uint32_t least[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const long long t0 = asr(t[i][0], d), t1 = asr(t[i][1], d), m = fix_lower_sign(A, h, i);
      S.up[i][a][0] += t0;
      S.up[i][a][1] += t1;
      const bool imag = !((h >> 1) & 1);
      const long long mr = m ^ (imag ? -1ll : 0ll);
      S.lo[i][a][0] += ((imag ? t1 : t0) ^ mr) - mr;
      S.lo[i][a][1] += ((imag ? t0 : t1) ^ m) - m;
      least[i] = fix_least(t0, t1);
    }
    S.mag[a] += __byte_perm(least[0], least[1], 0x7632);
  }
};

template <int N, bool SHARED>
__device__ __forceinline__ void fix_hop_into(FixAcc<N>& S, const DslashArgs& A, const SiteXyzt& X, uint32_t rhs,
                                             const int4* links, int h) {
  FixAdd<N> add{S, A, h};
  fix_hop_products<N, SHARED>(add, A, X, rhs, links, h);
}

// whether a site's exponents are within the format (E: the largest of a hop; 0: all zeros)
__device__ __forceinline__ bool fix_exponent_holds(int E) { return E == 0 || (E >= 1100 && E <= 3000); }

// A site's sums carry an absolute error of about a unit (1.3 to 1.6 rms: the left-out low x low products and the
// roundings to the unit).  FP64 multiply-adds have none where all the products of a part are small, and a link
// part or a spinor part 2^-k of its largest has only B - k bits here.  So a part holds if the magnitudes of its
// eight hops' products add up to kFixMag 2^48 units, or if they are exact zeros (its projected rows are zero in
// every hop), and a site with a part that does not hold takes FP64.  Over random, near-unit, unit and widely scaled
// links and full, one-colour, one-spin, real, point-like and widely scaled spinors the error of the parts that hold,
// relative to the sum of their products' magnitudes, is below that of FP64 multiply-adds: for SU(3) rms 0.07 to
// 0.63 2^-53 against 0.19 to 0.71, largest 0.6 to 4.6 2^-53 against 1.5 to 4.7.  Of random sites (Haar links,
// Gaussian spinors) about 1e-8 do not hold.  For SU(3) and SU(4) the smaller of a complex product's two parts
// stands for both, and one register holds both rows of a colour: with a sum for every part the registers spill,
// SU(3) 24^3x48 nrhs 12 2330 us against 1747.
template <int N>
__device__ __forceinline__ bool fix_parts_hold(const FixAcc<N>& S) {
  bool ok = true;
#pragma unroll
  for (int a = 0; a < N; a++) {
    const uint32_t m = fix_mag_shift(S.mag_xy[a], (uint32_t)(S.E - S.E_xy));
    const uint32_t xy[2] = {m & 0xffffu, m >> 16}, zt[2] = {S.mag[a] & 0xffffu, S.mag[a] >> 16};
#pragma unroll
    for (int i = 0; i < 2; i++) {  // the upper row i, and the lower row 2 + i, which takes the other row of x and y
      ok &= (S.rows & (5u << i)) == 0 || xy[i] + zt[i] >= kFixMag<N>;
      ok &= (S.rows & ((2u >> i) | (4u << i))) == 0 || xy[1 - i] + zt[i] >= kFixMag<N>;
    }
  }
  return ok;
}

// links: the site's records in shared memory (SHARED)
template <int N, bool SHARED>
__device__ __forceinline__ void fix_site(const DslashArgs& A, const SiteXyzt& X, uint32_t rhs, const int4* links) {
  prefetch_x<PREC_DOUBLE, N, 1>(A, X.site, rhs);
  FixAcc<N> S;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int a = 0; a < N; a++) S.up[i][a][0] = S.up[i][a][1] = S.lo[i][a][0] = S.lo[i][a][1] = 0;
  // one hop body for all eight (its gamma chosen by selects): with a body each for the imaginary and the
  // real gammas the instruction cache cost more than the selects, by 2% at SU(3) 24^3x48 nrhs 12 and by 18%
  // at SU(4) 16^3x32 nrhs 16, 128 registers
#pragma unroll 1
  for (int h = 0; h < 8; h++) {
    fix_hop_into<N, SHARED>(S, A, X, rhs, links, h);
    if (h == 3) {
      S.E_xy = S.E;
#pragma unroll
      for (int a = 0; a < N; a++) {
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const long long v = S.lo[0][a][c];
          S.lo[0][a][c] = S.lo[1][a][c];
          S.lo[1][a][c] = v;
        }
        S.mag_xy[a] = S.mag[a];
        S.mag[a] = 0;
      }
    }
  }

  if (S.bad || !fix_exponent_holds(S.E) || !fix_parts_hold(S)) {
    fp64_site<N>(A, X, rhs);
    return;
  }
  C2<double> out[4][N][1];
  const int e = S.E + kFixBias<N>;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int a = 0; a < N; a++) {
      out[i][a][0].x = from_fix(S.up[i][a][0], e);
      out[i][a][0].y = from_fix(S.up[i][a][1], e);
      out[2 + i][a][0].x = from_fix(S.lo[i][a][0], e);
      out[2 + i][a][0].y = from_fix(S.lo[i][a][1], e);
    }
  store_out<PREC_DOUBLE, N, 1>(out, A, X.site, rhs);
}

// Sites whose links a block of `block` threads holds in shared memory (0: each thread converts its own).
// Below four RHS groups a site's conversion is shared by too few threads to pay for its round trip.
template <int N>
__host__ __device__ constexpr uint32_t fix_shared_sites(uint32_t groups, uint32_t block) {
  const uint32_t n = (block - 1) / groups + 2;
  return groups >= 4 && n * kFixSite<N> * 16u <= 48u * 1024u ? n : 0;
}

// The block's threads gid0 .. gid0 + blockDim.x - 1 of a launch, R right-hand sides each.
template <int N, int R>
__device__ __forceinline__ void fix_block(const DslashArgs& A, uint32_t gid0) {
  extern __shared__ int4 fix_smem[];
  const uint32_t groups = A.div_groups.d, vh = (uint32_t)A.geo.vh;
  const uint32_t ns = fix_shared_sites<N>(groups, blockDim.x);
  uint32_t first, grp, site;
  A.div_groups.divmod(gid0, first, grp);
  if (ns) {
    for (uint32_t i = threadIdx.x; i < 8u * ns; i += blockDim.x) {
      const uint32_t h = i / ns, k = i - h * ns;
      if (first + k >= vh) continue;
      const SiteXyzt X = decode_site(A, first + k);
      const FixLink<N> L = load_fix_link<N>(A, X, (int)h, X.neighbour(A, (int)h));
      int4* d = fix_smem + (k * kFixSite<N> + h * kFixRec<N>);
#pragma unroll
      for (int c = 0; c < N * N; c++) {
        d[c] = L.u[c];
        reinterpret_cast<int2*>(d + N * N)[c] = make_int2(-L.u[c].z, -L.u[c].w);
      }
      reinterpret_cast<int2*>(d + N * N)[N * N] = make_int2((int)L.e, 0);
    }
    __syncthreads();
  }
  A.div_groups.divmod(gid0 + threadIdx.x, site, grp);
  if (site >= vh) return;
  const SiteXyzt X = decode_site(A, site);
#pragma unroll 1
  for (int r = 0; r < R; r++) {
    const uint32_t rhs = grp * R + r;
    if (A.mask && !A.mask[rhs]) continue;
    if (ns)
      fix_site<N, true>(A, X, rhs, fix_smem + (site - first) * kFixSite<N>);
    else
      fix_site<N, false>(A, X, rhs, nullptr);
  }
}

// The same site and RHS on eight threads, one a hop: thread h * U + u of a block of 8 U does hop h of the
// block's u-th site and RHS, leaves its products in shared memory, and sums and stores the components h and
// h + 8 (complex parts).  The sums take the hops in the same order and by the same shifts, so the result is
// the same to the bit.  For launches with about a warp a scheduler, whose time is one thread's chain of
// hops; where the GPU is full, the exchange and the links converted by every thread cost more.  One
// thread a site and RHS / eight, us: SU(3) 8^4 nrhs 1 23 / 8.6, nrhs 4 23 / 12.7, 12^3x24 nrhs 1 29 / 21,
// 14x10x6x18 nrhs 5 27 / 33, 24^3x48 nrhs 12 1747 / 2808; SU(4) 8^4 nrhs 2 36 / 10.9.  The autotuner
// times both.  A site that takes FP64 does so on its eight threads too.
template <int N>
constexpr uint32_t kFixSplitUnit = 8 * (4 * N * 8 + 8) + 8;  // bytes of a site and RHS
// the largest block up to `block` whose products stay within 48 KB
template <int N>
int fix_split_block_size(int block) {
  while (block > 32 && (uint32_t)block / 8 * kFixSplitUnit<N> > 48u * 1024u) block -= 32;
  return block;
}

template <int N>
struct FixShare {
  long long* v;  // [4 N][U] of this hop: part (2 i N + 2 a + c)
  int2* e;       // exponent; rows that are not zero, and bit 2: not for fixed point
  uint32_t U;
  __device__ __forceinline__ void begin(int eh, uint32_t rows, bool bad) {
    *e = make_int2(eh, (int)(rows | (bad ? 4u : 0u)));
  }
  __device__ __forceinline__ void put(int a, const long long (&t)[2][2]) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int c = 0; c < 2; c++) v[(2 * (i * N + a) + c) * U] = t[i][c];
  }
};

// hop h's products in FP64 multiply-adds, by fp64_site's operations, to where FixShare has them
template <int N>
__device__ __noinline__ void fp64_hop_products(double* v, uint32_t U, const DslashArgs& A, const SiteXyzt& X, uint32_t rhs,
                                               int h) {
  const uint32_t nb = X.neighbour(A, h);
  double2 x[2][N], y[2][N];
  fix_load<N>(x, y, A, nb, rhs, h >> 1);
  fix_project<N>(x, y, A, h);
  const FixLinkAt<N> at(A, X, h, nb);
#pragma unroll 1
  for (int a = 0; a < N; a++) {
    double2 t[2];
#pragma unroll
    for (int b = 0; b < N; b++) {
      const double2 u = at.load(a, b);
      const double ur = flip_sign(u.x, at.rf != 0), ui = flip_sign(u.y, at.jf != 0);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        t[i].x = b ? fma(ur, x[i][b].x, t[i].x) : ur * x[i][b].x;
        t[i].y = b ? fma(ur, x[i][b].y, t[i].y) : ur * x[i][b].y;
        t[i].x = fma(-ui, x[i][b].y, t[i].x);
        t[i].y = fma(ui, x[i][b].x, t[i].y);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
      v[(2 * (i * N + a)) * U] = t[i].x;
      v[(2 * (i * N + a) + 1) * U] = t[i].y;
    }
  }
}

// the component comp (complex part of row comp / N) of a site and RHS: the eight hops' products summed in FP64
template <int N>
__device__ __noinline__ double2 fp64_sum(const double* vals, uint32_t U, uint32_t u, const DslashArgs& A, uint32_t comp) {
  const int row = (int)comp / N, a = (int)comp - row * N;
  double2 s;
#pragma unroll 1
  for (int g = 0; g < 8; g++) {
    const int mu = g >> 1, i = row < 2 ? row : mu < 2 ? 3 - row : row - 2;
    const double* v = vals + ((g * 4 * N + 2 * (i * N + a)) * U + u);
    double re = v[0], im = v[U];
    if (row >= 2) {
      const bool neg = fix_lower_sign(A, g, i) != 0, imag = !(mu & 1);
      const double t = re;
      re = flip_sign(imag ? im : re, neg != imag);
      im = flip_sign(imag ? t : im, neg);
    }
    s.x = g ? s.x + re : re;
    s.y = g ? s.y + im : im;
  }
  return s;
}

template <int N>
__device__ __forceinline__ void fix_split_block(const DslashArgs& A, uint32_t blk) {
  extern __shared__ int4 fix_smem[];
  const uint32_t U = blockDim.x / 8, h = threadIdx.x / U, u = threadIdx.x - h * U;
  long long* vals = reinterpret_cast<long long*>(fix_smem);
  int2* exps = reinterpret_cast<int2*>(vals + 8 * 4 * N * U);
  int* fails = reinterpret_cast<int*>(exps + 8 * U);  // [U] the site does not hold
  const uint32_t vh = (uint32_t)A.geo.vh, nrhs = (uint32_t)A.nrhs, cs = vh * nrhs;
  uint32_t site, rhs;
  A.div_groups.divmod(blk * U + u, site, rhs);
  const bool live = site < vh && (!A.mask || A.mask[rhs]);
  const SiteXyzt X = decode_site(A, live ? site : 0);
  const uint32_t o = X.site * nrhs + rhs;
  constexpr int K = (4 * N + 7) / 8;
  double2 xv[K];
  if (h == 0) fails[u] = 0;
  if (live) {
    if (A.x) {
#pragma unroll
      for (int k = 0; k < K; k++)
        if (h + 8 * k < 4 * N) xv[k] = __ldg(static_cast<const double2*>(A.x) + (o + (h + 8 * k) * cs));
    }
    FixShare<N> share{vals + (h * 4 * N * U + u), exps + (h * U + u), U};
    fix_hop_products<N, false>(share, A, X, rhs, nullptr, (int)h);
  }
  __syncthreads();

  double2 r[K];
  bool bad = false;
  if (live) {
    uint32_t rows = 0;
    int E = 0;
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const int2 e = exps[g * U + u];
      rows |= (uint32_t)(e.y & 3) << (g < 4 ? 0 : 2);
      bad |= (e.y & 4) != 0 || (E != 0 && e.x - E > kFixSpan) || (e.x != 0 && E - e.x > kFixSpan);
      E = max(E, e.x);
    }
    bad |= !fix_exponent_holds(E);
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t comp = h + 8 * k;
      if (comp >= 4 * N) break;
      const int row = (int)comp / N, a = (int)comp - row * N;
      // the projected rows that feed this one, of x and y and of z and t
      const int i0 = row < 2 ? row : 3 - row, i1 = row < 2 ? row : row - 2;
      long long s0 = 0, s1 = 0;
      uint32_t m0 = 0, m1 = 0;  // SU(3), SU(4): as FixAcc::mag and mag_xy; else |real part| and |imaginary part|
      int Es = 0;
#pragma unroll
      for (int g = 0; g < 8; g++) {
        const int mu = g >> 1, eg = exps[g * U + u].x, i = mu < 2 ? i0 : i1;
        if (eg > Es) {
          const uint32_t up = (uint32_t)(eg - Es);
          s0 = asr(s0, up);
          s1 = asr(s1, up);
          m0 = fix_mag_shift(m0, up);
          m1 = fix_mag_shift(m1, up);
          Es = eg;
        }
        const uint32_t d = (uint32_t)(Es - eg);
        const long long* v = vals + ((g * 4 * N + 2 * (i * N + a)) * U + u);
        const long long t0 = asr(v[0], d), t1 = asr(v[U], d);
        if constexpr (fix_split_only(N)) {
          const bool imag = row >= 2 && !(mu & 1);
          m0 += (uint32_t)abs((int32_t)((imag ? t1 : t0) >> 32)) >> 16;
          m1 += (uint32_t)abs((int32_t)((imag ? t0 : t1) >> 32)) >> 16;
        } else {
          m0 += fix_least(t0, t1) >> 16;
          if (g == 3) m1 = m0, m0 = 0;
        }
        if (row < 2) {
          s0 += t0;
          s1 += t1;
        } else {
          const long long m = fix_lower_sign(A, g, i);
          if (!(mu & 1)) {
            s0 -= (t1 ^ m) - m;
            s1 += (t0 ^ m) - m;
          } else {
            s0 += (t0 ^ m) - m;
            s1 += (t1 ^ m) - m;
          }
        }
      }
      bad |= (rows & ((1u << i0) | (4u << i1))) != 0 && (fix_split_only(N) ? min(m0, m1) : m0 + m1) < kFixMag<N>;
      r[k] = make_double2(from_fix(s0, Es + kFixBias<N>), from_fix(s1, Es + kFixBias<N>));
    }
    if (bad) fails[u] = 1;
  }
  if (__syncthreads_or(bad)) {  // FP64 multiply-adds for the sites that do not hold, one hop a thread
    const bool again = live && fails[u];
    double* d = reinterpret_cast<double*>(vals);
    if (again) fp64_hop_products<N>(d + (h * 4 * N * U + u), U, A, X, rhs, (int)h);
    __syncthreads();
    if (again) {
#pragma unroll
      for (int k = 0; k < K; k++)
        if (h + 8 * k < 4 * N) r[k] = fp64_sum<N>(d, U, u, A, h + 8 * k);
    }
  }
  if (!live) return;
  const double ca = A.a_rhs_d ? A.a_rhs_d[rhs] : A.a;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const uint32_t comp = h + 8 * k;
    if (comp >= 4 * N) break;
    // store_out's operations
    if (A.x) {
      if (A.b == 1.0)
        r[k] = make_double2(fma(ca, r[k].x, xv[k].x), fma(ca, r[k].y, xv[k].y));
      else
        r[k] = make_double2(fma(A.b, xv[k].x, ca * r[k].x), fma(A.b, xv[k].y, ca * r[k].y));
    } else if (A.a_rhs_d || A.a != 1.0) {
      r[k] = make_double2(r[k].x * ca, r[k].y * ca);
    }
    static_cast<double2*>(A.out)[o + comp * cs] = r[k];
  }
}

}  // namespace detail
}  // namespace qcu
