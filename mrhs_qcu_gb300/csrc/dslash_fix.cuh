// FP64 Wilson hop with the colour multiply in block fixed point.
//
// The FP64 pipe of sm_103a takes 2 multiply-adds per clock and SM, and 840 of them a site and RHS kept
// it 97% busy at SU(3).  32 x 32 -> 64-bit integer multiply-adds run at about 16 times that rate.  So
// only the projection (12 operations a hop at SU(3)) is left on the FP64 pipe, and the colour multiply
// and the sum over hops are done in integers:
//
//   projected spinor   the 4N real parts of a neighbour's two rows, 59 bits over their common exponent
//   link               its 2N^2 real parts, 59 bits over theirs
//   product            limbs of 28 and 31 bits, the three larger limb products summed exactly in two
//                      64-bit accumulators a component; only low x low (2^-56 of the operands' largest
//                      parts, at most) is left out
//   sum over hops      64-bit integers over the largest hop's exponent
//   result             rounded once to double (nearest even); the xpay epilogue stays FP64
//
// No sum can overflow (the bounds stand beside the constants), and none rounds before the last step
// but by the right shifts to the accumulator's unit.  Relative L2 error against quad precision on random
// fields: SU(3), SU(4) 0.84e-16, SU(5) to SU(8) 1.20e-16 to 1.24e-16, where the FP64 multiply-adds have
// 1.45e-16, 1.54e-16 and 1.62e-16 to 1.8e-16.
//
// One hop, us, FP64 multiply-adds / this: SU(3) 24^3x48 nrhs 12 5826 / 1660, SU(4) 16^3x32 nrhs 16
// 2480 / 743, SU(3) 14x10x6x18 nrhs 5 59 / 27; in the split form SU(3) 12^3x24 nrhs 1 44 / 19, SU(6)
// 16^3x32 nrhs 16 4983 / 2286, SU(8) 8383 / 4037, SU(6) 8^3x16 nrhs 1 100 / 19.  It is bound by
// instruction issue and latency (SU(3): 8300 instructions a warp, 216 wide multiply-adds a hop; the
// multiplier 53% busy, the integer pipe 43%, FP64 33%, 12 or 16 warps an SM); the small sizes by the
// latency of one warp a scheduler.
//
// A common exponent keeps the digits of a part only down to its unit.  So a site takes the FP64
// multiply-adds (fp64_site) when the non-zero parts that it multiplies span more than kFixSpan bits,
// when anything it reads is infinite or NaN, and when the result could leave the normal range.
#pragma once

namespace qcu {
namespace detail {

// the FP64 SU(N) hops that run in fixed point; from SU(5) on only in the split form (a thread cannot hold
// the sums of 8N parts)
__host__ __device__ constexpr bool fix_hop(int prec, int N) { return prec == PREC_DOUBLE && N >= 3 && N <= 8; }
__host__ __device__ constexpr bool fix_split_only(int N) { return N > 4; }

// A part 31 bits below the largest keeps 25 digits of its own.  One site in FP64 multiply-adds takes a
// warp 27 us, as long as a small launch: at 24 bits, where 1e-5 of random sites span more, SU(3)
// 14x10x6x18 nrhs 5 took 54 us against 27.
constexpr int kFixSpan = 31;

// Parts |F| < 2^59 as limbs F = hi 2^31 + lo, |hi| <= 2^28, |lo| < 2^31.  Over a component's 2N products:
//   high  |sum uh hh|            <= 2N 2^56     (N = 4: 2^59)
//   mid   |sum uh hl + ul hh|    <= 2N 2 2^28 (2^31 - 1)   (N = 4: 2^63 - 2^32, so the rounding bit fits)
// A hop's sum in the accumulator's unit is high + (mid >> 31), below 2^59 + 2^32 at N = 4; eight of
// them stay below 2^63.  From SU(5) on |F| < 2^58, which bounds N = 8 by the same sums, and lo is
// balanced, |lo| <= 2^30: the 2N products low x low that are left out would otherwise cost 2e-16.
template <int N>
constexpr uint32_t kFixShift = N <= 4 ? 5 : 6;  // right shift of a mantissa whose top bit is bit 63

struct Limbs {
  int32_t hi, lo;
};

__device__ __forceinline__ uint32_t biased_exp(double x) { return ((uint32_t)__double2hiint(x) >> 20) & 0x7ffu; }

// x over the biased exponent es - kFixShift of the largest part; flip 0x80000000 negates
template <int N>
__device__ __forceinline__ Limbs to_limbs(double x, uint32_t es, uint32_t flip) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mh = __funnelshift_l(lo, hi, 11) | 0x80000000u, ml = lo << 11;
  const uint32_t s = es - ((hi >> 20) & 0x7ffu);  // a zero's is es, above 63
  unsigned long long f;
  asm("shr.u64 %0, %1, %2;" : "=l"(f) : "l"(((unsigned long long)mh << 32) | ml), "r"(s));  // shifts above 63 give 0
  const int32_t sign = ((int32_t)(hi ^ flip) >> 31) | 1;
  if constexpr (fix_split_only(N)) {
    const uint32_t top = (uint32_t)((f + (1u << 30)) >> 31);
    return Limbs{(int32_t)top * sign, (int32_t)((uint32_t)f - (top << 31)) * sign};
  }
  return Limbs{(int32_t)(uint32_t)(f >> 31) * sign, (int32_t)((uint32_t)f & 0x7fffffffu) * sign};
}

// v >> s for s up to 31, which a site's shifts are while its span holds (kFixSpan); with larger ones, whose
// sites take FP64, it is any value (a 64-bit shift instruction pair costs 1.5% of the hop)
__device__ __forceinline__ long long asr(long long v, uint32_t s) {
  const int32_t h = (int32_t)(v >> 32);
  const uint32_t lo = __funnelshift_r((uint32_t)v, (uint32_t)h, s);
  return (long long)(((unsigned long long)(uint32_t)(h >> (s & 31u)) << 32) | lo);
}

// a sum T over hops of largest exponent E is T 2^(E - 2110 + 2 kFixShift): from_fix(T, E + kFixBias)
template <int N>
constexpr int kFixBias = 2 * (int)kFixShift<N> - 1025;
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
// instead of the 12 projected ones, against 1685): [site][hop] records of the N^2 elements (int4), their
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
  int E = 0, Emin = 8191;
  bool bad = false;
};

// s = +1 / -1 of hop h as a sign bit, and the sign s g(u_perm) with which the product of row i enters the lower row
__device__ __forceinline__ uint32_t fix_sign(const DslashArgs& A, int h) {
  return ((h & 1) != (A.dagger != 0)) ? 0u : 0x80000000u;
}
__device__ __forceinline__ long long fix_lower_sign(const DslashArgs& A, int h, int i) {  // 0 or -1
  const int mu = h >> 1;
  const uint32_t g = fix_sign(A, h) ^ ((i ? mu == 0 : mu != 3) ? 0x80000000u : 0u);
  return (long long)(int32_t)g >> 31;
}

// Hop h: out.begin(exponent, smallest exponent, not for fixed point), then out.put(a, i, re, im) for the
// products of colour a and projected row i in the hop's own unit.
template <int N, bool SHARED, typename Out>
__device__ __forceinline__ void fix_hop_products(Out& out, const DslashArgs& A, const SiteXyzt& X, uint32_t rhs,
                                                 const int4* links, int h) {
  const int mu = h >> 1;
  const bool imag = !(mu & 1);
  const uint32_t nrhs = (uint32_t)A.nrhs;
  const double2* __restrict__ in = static_cast<const double2*>(A.in);
  const uint32_t cs_bytes = (uint32_t)A.geo.vh * nrhs * 16u;
  const uint32_t nb = X.neighbour(A, h);

  // the neighbour's spinor; rows 2 and 3 in the order in which rows 0 and 1 meet them
  double2 x[2][N], y[2][N];
  {
    const char* base = reinterpret_cast<const char*>(in + (nb * nrhs + rhs));
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

  // h_u = x_u + s g(u) y_u, into x
  const uint32_t sgn = fix_sign(A, h);
  const double k0 = __hiloint2double((int)(0x3ff00000u | (sgn ^ (mu == 1 ? 0x80000000u : 0u))), 0);
  const double k1 = __hiloint2double((int)(0x3ff00000u | (sgn ^ (mu == 2 ? 0x80000000u : 0u))), 0);
  uint32_t ep = 0, mn = 0xffffffffu;  // exponents: largest; smallest of the non-zero parts, less one
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int a = 0; a < N; a++) {
      const double k = i ? k1 : k0;
      x[i][a].x = fma(imag ? -k : k, imag ? y[i][a].y : y[i][a].x, x[i][a].x);
      x[i][a].y = fma(k, imag ? y[i][a].x : y[i][a].y, x[i][a].y);
      const uint32_t q0 = biased_exp(x[i][a].x), q1 = biased_exp(x[i][a].y);
      ep = max(ep, max(q0, q1));
      mn = min(mn, min(q0 - 1u, q1 - 1u));
    }
  bool bad = ep == 0x7ffu || eu == 0x7ffu || eu < 200u;
  int eh = (int)(ep + eu);
  uint32_t es = ep + kFixShift<N>;
  bad |= ep != 0 && es < 64;  // a zero's shift, es, would leave its implicit leading bit (to_limbs)
  if (ep == 0) {  // zeros add nothing; subnormal parts: FP64
    long long any = 0;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int a = 0; a < N; a++) any |= __double_as_longlong(x[i][a].x) | __double_as_longlong(x[i][a].y);
    bad |= (any << 1) != 0;
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

  out.begin(eh, (int)min(mn, 4095u) + 1 + (int)eu, bad);

#pragma unroll fix_split_only(N) ? 1 : N
  for (int a = 0; a < N; a++) {
    long long H[2][2], M[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int c = 0; c < 2; c++) H[i][c] = 0, M[i][c] = 1ll << 30;
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
#pragma unroll
    for (int i = 0; i < 2; i++) out.put(a, i, H[i][0] + (M[i][0] >> 31), H[i][1] + (M[i][1] >> 31));
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
  __device__ __forceinline__ void begin(int eh, int emin, bool bad) {
    S.bad |= bad;
    S.Emin = min(S.Emin, emin);
    if (eh > S.E) {
      const uint32_t up = (uint32_t)(eh - S.E);
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int a = 0; a < N; a++)
#pragma unroll
          for (int c = 0; c < 2; c++) {
            S.up[i][a][c] = asr(S.up[i][a][c], up);
            S.lo[i][a][c] = asr(S.lo[i][a][c], up);
          }
      S.E = eh;
    }
    d = (uint32_t)(S.E - eh);
  }
  // lower rows: lo(u) += s g(u_perm) (im ? i : 1) t_u
  __device__ __forceinline__ void put(int a, int i, long long re, long long im) {
    const long long t0 = asr(re, d), t1 = asr(im, d), m = fix_lower_sign(A, h, i);
    S.up[i][a][0] += t0;
    S.up[i][a][1] += t1;
    const bool imag = !((h >> 1) & 1);
    const long long mr = m ^ (imag ? -1ll : 0ll);
    S.lo[i][a][0] += ((imag ? t1 : t0) ^ mr) - mr;
    S.lo[i][a][1] += ((imag ? t0 : t1) ^ m) - m;
  }
};

template <int N, bool SHARED>
__device__ __forceinline__ void fix_hop_into(FixAcc<N>& S, const DslashArgs& A, const SiteXyzt& X, uint32_t rhs,
                                             const int4* links, int h) {
  FixAdd<N> add{S, A, h};
  fix_hop_products<N, SHARED>(add, A, X, rhs, links, h);
}

// whether a site's sums hold: E, Emin the largest and smallest exponents of its hops
__device__ __forceinline__ bool fix_holds(bool bad, int E, int Emin) {
  return !bad && (E == 0 || (E >= 1100 && E <= 3000 && E - Emin <= kFixSpan));
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
  // real gammas the instruction cache cost more than the selects, 1720 against 1685 us at SU(3) 24^3x48
  // nrhs 12, and 914 against 772 at SU(4) 16^3x32 nrhs 16, 128 registers
#pragma unroll 1
  for (int h = 0; h < 8; h++) {
    fix_hop_into<N, SHARED>(S, A, X, rhs, links, h);
    if (h == 3) {
#pragma unroll
      for (int a = 0; a < N; a++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const long long v = S.lo[0][a][c];
          S.lo[0][a][c] = S.lo[1][a][c];
          S.lo[1][a][c] = v;
        }
    }
  }

  if (!fix_holds(S.bad, S.E, S.Emin)) {
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
// thread a site and RHS / eight, us: SU(3) 8^4 nrhs 1 22 / 7.6, nrhs 4 22 / 11.7, 12^3x24 nrhs 1 27 / 19,
// 14x10x6x18 nrhs 5 27 / 29, 24^3x48 nrhs 12 1685 / 2369; SU(4) 8^4 nrhs 2 37 / 10.7.  The autotuner
// times both.
template <int N>
constexpr uint32_t kFixSplitUnit = 8 * (4 * N * 8 + 8);  // bytes of a site and RHS
// the largest block up to `block` whose products stay within 48 KB
template <int N>
int fix_split_block_size(int block) {
  while (block > 32 && (uint32_t)block / 8 * kFixSplitUnit<N> > 48u * 1024u) block -= 32;
  return block;
}

template <int N>
struct FixShare {
  long long* v;  // [4 N][U] of this hop: part (2 i N + 2 a + c)
  int2* e;       // exponent, smallest exponent
  uint32_t U;
  static constexpr int kBad = -(1 << 20);
  __device__ __forceinline__ void begin(int eh, int emin, bool bad) { *e = make_int2(eh, bad ? kBad : emin); }
  __device__ __forceinline__ void put(int a, int i, long long re, long long im) {
    v[(2 * (i * N + a)) * U] = re;
    v[(2 * (i * N + a) + 1) * U] = im;
  }
};

template <int N>
__device__ __forceinline__ void fix_split_block(const DslashArgs& A, uint32_t blk) {
  extern __shared__ int4 fix_smem[];
  const uint32_t U = blockDim.x / 8, h = threadIdx.x / U, u = threadIdx.x - h * U;
  long long* vals = reinterpret_cast<long long*>(fix_smem);
  int2* exps = reinterpret_cast<int2*>(vals + 8 * 4 * N * U);
  const uint32_t vh = (uint32_t)A.geo.vh, nrhs = (uint32_t)A.nrhs, cs = vh * nrhs;
  uint32_t site, rhs;
  A.div_groups.divmod(blk * U + u, site, rhs);
  const bool live = site < vh && (!A.mask || A.mask[rhs]);
  const SiteXyzt X = decode_site(A, live ? site : 0);
  const uint32_t o = X.site * nrhs + rhs;
  constexpr int K = (4 * N + 7) / 8;
  double2 xv[K];
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
  if (!live) return;

  int E = 0, Emin = 8191;
#pragma unroll
  for (int g = 0; g < 8; g++) {
    const int2 e = exps[g * U + u];
    E = max(E, e.x);
    Emin = min(Emin, e.y);
  }
  if (!fix_holds(Emin <= FixShare<N>::kBad, E, Emin)) {
    if (h == 0) fp64_site<N>(A, X, rhs);
    return;
  }
  const double ca = A.a_rhs_d ? A.a_rhs_d[rhs] : A.a;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const uint32_t comp = h + 8 * k;
    if (comp >= 4 * N) break;
    const int row = (int)comp / N, a = (int)comp - row * N;
    long long s0 = 0, s1 = 0;
    int Es = 0;
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const int mu = g >> 1, eg = exps[g * U + u].x;
      if (eg > Es) {
        s0 = asr(s0, (uint32_t)(eg - Es));
        s1 = asr(s1, (uint32_t)(eg - Es));
        Es = eg;
      }
      const int i = row < 2 ? row : mu < 2 ? 3 - row : row - 2;  // the projected row that feeds this one
      const long long* v = vals + ((g * 4 * N + 2 * (i * N + a)) * U + u);
      const long long t0 = asr(v[0], (uint32_t)(Es - eg)), t1 = asr(v[U], (uint32_t)(Es - eg));
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
    double2 r = make_double2(from_fix(s0, Es + kFixBias<N>), from_fix(s1, Es + kFixBias<N>));
    // store_out's operations
    if (A.x) {
      if (A.b == 1.0)
        r = make_double2(fma(ca, r.x, xv[k].x), fma(ca, r.y, xv[k].y));
      else
        r = make_double2(fma(A.b, xv[k].x, ca * r.x), fma(A.b, xv[k].y, ca * r.y));
    } else if (A.a_rhs_d || A.a != 1.0) {
      r = make_double2(r.x * ca, r.y * ca);
    }
    static_cast<double2*>(A.out)[o + comp * cs] = r;
  }
}

}  // namespace detail
}  // namespace qcu
