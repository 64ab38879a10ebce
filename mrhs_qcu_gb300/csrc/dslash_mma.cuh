// MRHS Wilson hop with the link product on register-fragment matrix
// instructions (mma.sync m16n8k16, FP32 accumulation) for 16-bit storage,
// SU(N) for N = 3..8.
//
// One warp = S consecutive output sites x 16 MT right-hand sides, on its own:
// no barrier joins it to other warps.  Per hop it multiplies the neighbour
// spinors (A: 16 RHS x 16 real components, one packed (Re, Im) word per
// colour) by the link (B, 16 x 8: four output colours), W = U_mu(x) or
// U_mu(x - mu)^dag as its real 2 x 2 blocks [[Re, Im], [-Im, Re]].  Lane
// (g = lane / 4, t = lane % 4) holds the word of colour t (+ 4) of RHS rows
// 2g and 2g + 1, used as the operand untouched, and receives the complex
// output colour t (+ 4) of the same RHS.
//
// The neighbour words go through shared memory: the warp copies the rows of
// its S neighbour sites, [4N][S x RHS], with cp.async in the field's own
// contiguous order, NST - 1 hops ahead, and reads the fragments from there.
// Reading them from global memory in fragment order touches a 128-byte line
// per colour in every quarter-warp pass: that form kept the L1 data pipe 97%
// busy at 7 wavefronts per 8-byte load and gave 0.7x of the register kernel
// at SU(3).  Rows are padded to 8 or 24 words modulo 32, so both sides are
// free of bank conflicts.
//
// The spin projection is exact: it is not rounded to 16 bits but folded into
// the products, t_u = W psi_u + c_u W psi_pu with c_u = +-1 or +-i, which
// only permutes the halves of B's words and flips their signs.  N <= 4: the
// two spins fill the K dimension of one MMA.  N > 4: two MMAs per output
// colour group.  BF16 fields with N <= 4 accumulate all hops in the MMA
// accumulators; N > 4 and FP16 (whose per-(site, RHS) scale multiplies t)
// form t_u once and add it to the two spin rows it contributes to.
//
// The eight links of a site come from 16-bit records [parity][site][hop][N][N]
// (layout.h gauge_site_records) that hold W itself, copied to shared memory
// with the first hop.
#pragma once

#include <type_traits>

#include "dslash_kernel.cuh"

namespace qcu {

struct MmaDslashArgs {
  DslashArgs A;
  FastDiv div_chunks;   // RHS chunks of 16 MT per site group
  uint32_t warps;       // site groups x chunks
  uint32_t cstr, sstr;  // component and site strides of the fields in complex elements (either layout)
};

namespace mma {

constexpr int kWarps = 4;  // per CTA

template <int P>
__device__ __forceinline__ void op(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (P == PREC_HALF)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
        "%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, "
        "%2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16 bytes global -> shared, through L1 or past it
template <bool L1>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src) {
  if constexpr (L1)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_groups() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int P>
__device__ __forceinline__ float2 unpack(uint32_t w) {
  return Store<P>::to_c(*reinterpret_cast<const typename Store<P>::elem*>(&w));
}
template <int P>
__device__ __forceinline__ uint32_t pack(float re, float im) {
  const typename Store<P>::elem e = Store<P>::from_c(make_float2(re, im));
  return *reinterpret_cast<const uint32_t*>(&e);
}

// Shared memory of a warp, in words: the link records of its S sites, then
// NST stages of 4N rows (FP16: and one of scales).  A row holds S sites x 16 MT
// RHS, padded to 8 or 24 modulo 32.
__host__ __device__ constexpr uint32_t rec_words(int N, int S) { return (uint32_t)(S * 8 * N * N); }
__host__ __device__ constexpr uint32_t row_pitch(int S, int MT) { return (uint32_t)(S * 16 * MT + 8); }
__host__ __device__ constexpr uint32_t stage_words(int P, int N, int S, int MT) {
  return (4u * N + (P == PREC_HALF ? 1u : 0u)) * row_pitch(S, MT);
}
__host__ __device__ constexpr uint32_t warp_words(int P, int N, int S, int MT, int NST) {
  return rec_words(N, S) + NST * stage_words(P, N, S, MT);
}

}  // namespace mma

// S sites x 16 MT RHS per warp, NST stages; L1: the copies go through L1 (RHS
// counts whose rows are not whole 32-byte sectors: neighbouring sites then
// share sectors).
template <int P, int N, int S, int MT, int NST, bool L1>
__global__ void __launch_bounds__(32 * mma::kWarps) wilson_mma_kernel(const __grid_constant__ MmaDslashArgs T) {
  using namespace detail;
  constexpr int CG = N <= 4 ? 1 : 2;  // groups of four colours
  constexpr bool kNorm = Store<P>::has_norm;
  constexpr bool kDirect = N <= 4 && !kNorm;  // hops accumulate in the MMA accumulators
  constexpr uint32_t kWidth = 16 * MT, kPitch = mma::row_pitch(S, MT), kStage = mma::stage_words(P, N, S, MT);
  constexpr uint32_t kRow = S * kWidth / 4;  // 16-byte vectors per row
  constexpr uint32_t kStep = 32 / kRow;      // rows per copy instruction of the warp
  constexpr uint32_t kCopies = (4 * N + kStep - 1) / kStep;
  constexpr bool kEven = (4 * N) % kStep == 0;
  static_assert(32 % kRow == 0 && kPitch % 16 == 8, "row shape");
  const DslashArgs& A = T.A;
  const uint32_t wid = blockIdx.x * mma::kWarps + (threadIdx.x >> 5);
  if (wid >= T.warps) return;
  const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
  const uint32_t nrhs = (uint32_t)A.nrhs, vh = (uint32_t)A.geo.vh, p = (uint32_t)A.parity;
  uint32_t group, chunk;
  T.div_chunks.divmod(wid, group, chunk);
  const uint32_t rhs0 = chunk * kWidth;           // the warp's first RHS
  const uint32_t count = min(nrhs - rhs0, kWidth);  // and how many
  if (A.mask) {
    if (!__any_sync(0xffffffffu, lane < count && A.mask[rhs0 + lane] != 0)) return;
  }

  extern __shared__ __align__(16) uint32_t mma_smem[];
  uint32_t* const ws = mma_smem + (threadIdx.x >> 5) * mma::warp_words(P, N, S, MT, NST);
  uint32_t* const rows = ws + mma::rec_words(N, S);

  // launch position -> site (slab order, dslash_kernel.cuh); positions past the end repeat the last site
  auto place = [&](uint32_t j) {
    const uint32_t pos = min(group * S + j, vh - 1u);
    if (A.zb) {
      EoSite e(A.geo, 0u);
      uint32_t q, r, q2, zz, slab;
      A.div_plane.divmod(pos, q, r);
      A.div_zb.divmod(q, q2, zz);
      A.div_lt.divmod(q2, slab, e.t);
      e.z = slab * A.zb + zz;
      A.geo.div_hx.divmod(r, e.y, e.xh);
      e.site = (e.t * (uint32_t)A.geo.L[2] + e.z) * (uint32_t)A.geo.plane + r;
      e.eo = (e.y + e.z + e.t) & 1u;
      return e;
    }
    return EoSite(A.geo, pos);
  };

  // this lane's part of every copy: vector cv of site cj in rows r0, r0 + kStep, ...
  const uint32_t r0 = lane / kRow, cj = lane % kRow / (kWidth / 4), cr = 4u * (lane % (kWidth / 4));
  const EoSite cs = place(cj);
  const bool copies = cr < count;
  const uint32_t src0 = r0 * T.cstr + rhs0 + cr;
  const uint64_t src_step = (uint64_t)(kStep * T.cstr);
  const uint32_t lane_word = r0 * kPitch + cj * kWidth + cr;
  const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(rows) + 4u * lane_word;
  const uint32_t* __restrict__ in = static_cast<const uint32_t*>(A.in);
  const uint32_t* __restrict__ xin = static_cast<const uint32_t*>(A.x);
  auto copy_rows = [&](const uint32_t* f, const float* norms, uint32_t site, int stage) {
    const uint32_t* src = f + (site * T.sstr + src0);
    const uint32_t dst = dst0 + 4u * kStage * stage;
    if (copies) {
#pragma unroll
      for (uint32_t k = 0; k < kCopies; k++, src += src_step)
        if (kEven || r0 + k * kStep < 4u * N) mma::copy_async<L1>(dst + 4u * k * kStep * kPitch, src);
      if (kNorm && r0 == 0)  // the scale row
        mma::copy_async<L1>(dst + 16u * N * kPitch, norms + (site * nrhs + rhs0 + cr));
    }
  };
  // hop d = 0..7, then the xpay field of the sites themselves (d = 8), each as one group
  auto issue = [&](int d) {
    if (d < 8)
      copy_rows(in, A.in_norm, cs.nb(A.geo, p, d), d % NST);
    else if (d == 8 && xin)
      copy_rows(xin, A.x_norm, cs.site, 8 % NST);
    mma::commit();
  };

  uint32_t edge = 0u;  // bits 2 j, 2 j + 1: site j at the last, first time slice
#pragma unroll
  for (int j = 0; j < S; j++) {
    const EoSite e = place((uint32_t)j);
    if (e.t == (uint32_t)A.geo.L[3] - 1u) edge |= 1u << (2 * j);
    if (e.t == 0u) edge |= 2u << (2 * j);
    const uint32_t* rec = static_cast<const uint32_t*>(A.gauge_rec) + (uint64_t)(p * vh + e.site) * (8u * N * N);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ws) + 4u * j * 8u * N * N;
#pragma unroll
    for (uint32_t k = 0; k < 8u * N * N; k += 128u)
      if (k + 4u * lane < 8u * N * N) mma::copy_async<false>(dst + 4u * (k + 4u * lane), rec + k + 4u * lane);
  }
#pragma unroll
  for (int d = 0; d < NST - 1; d++) issue(d);

  float acc[S][4][CG][MT][4];
#pragma unroll
  for (int j = 0; j < S; j++)
#pragma unroll
    for (int s = 0; s < 4; s++)
#pragma unroll
      for (int c = 0; c < CG; c++)
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
          for (int k = 0; k < 4; k++) acc[j][s][c][i][k] = 0.f;

  // Fragment addresses.  K and output columns past colour N - 1 (their link
  // words are zero) read the last colour's words again: no lane reads
  // memory that the copies have not written, and a non-finite spinor spreads
  // to nothing its hop does not already reach.
  const bool odd = g & 1u, dag = A.dagger != 0;
  constexpr int kLast = (N - 1) % 4;  // the last colour's lane in its group
  const uint32_t t_hi = min(t, (uint32_t)kLast);  // this lane's colour in the last group
  const uint32_t frag[2] = {(CG == 1 ? t_hi : t) * kPitch + 2u * g, t_hi * kPitch + 2u * g};
  const uint32_t one_sel = odd ? 0x1032u : 0x3210u, eye_sel = odd ? 0x3210u : 0x1032u;
  const uint32_t one_sign = odd ? 0u : 0x80000000u, eye_sign = odd ? 0x80000000u : 0x80008000u;

  auto hop = [&](auto dc) {
    constexpr int D = decltype(dc)::value;
    constexpr int MU = D >> 1;
    constexpr bool FWD = (D & 1) == 0;
    constexpr bool IM = gimag(MU);
    __syncwarp();  // stage (D - 1) % NST has been read
    issue(D + NST - 1);
    mma::wait_groups<NST - 1>();
    __syncwarp();
    const uint32_t* const st = rows + (D % NST) * kStage;
    // projector 1 + sigma g, sigma = -f (forward) or +f (backward)
    const uint32_t flip_s = (FWD != dag) ? 0x80008000u : 0u;
#pragma unroll
    for (int j = 0; j < S; j++) {
      uint32_t flip_b = 0u;  // the boundary sign, on W
      if constexpr (MU == 3) {
        if (A.antiperiodic_t && (edge >> (2 * j + (FWD ? 0 : 1)) & 1u)) flip_b = 0x80008000u;
      }
      // B words of W, [Wr, -Wi] (even columns: real part) or [Wi, Wr], and of sigma W (real gamma)
      // or sigma i W (imaginary gamma), per (output group, input group)
      uint32_t one[CG][CG], sig[CG][CG];
#pragma unroll
      for (int na = 0; na < CG; na++)
#pragma unroll
        for (int nk = 0; nk < CG; nk++) {
          const uint32_t a = (g >> 1) + 4u * na, b = t + 4u * nk;
          const bool has = (4 * na + 3 < N || a < (uint32_t)N) && (4 * nk + 3 < N || b < (uint32_t)N);
          const uint32_t w = has ? ws[(j * 8 + D) * N * N + a * N + b] : 0u;
          one[na][nk] = __byte_perm(w, 0u, one_sel) ^ (one_sign ^ flip_b);
          sig[na][nk] = IM ? __byte_perm(w, 0u, eye_sel) ^ (eye_sign ^ flip_b ^ flip_s) : one[na][nk] ^ flip_s;
        }
#pragma unroll
      for (int i = 0; i < MT; i++) {
        if (MT > 1 && 16u * i >= count) continue;  // a short last chunk
        // neighbour words w[spin][colour group]: rows g, g + 8 of the M tile are RHS 2 g, 2 g + 1
        uint2 w[4][CG];
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
          for (int c = 0; c < CG; c++)
            w[s][c] = *reinterpret_cast<const uint2*>(st + frag[c] + (uint32_t)(s * N + 4 * c) * kPitch +
                                                      j * kWidth + 16 * i);
        float nr[2];
        if constexpr (kNorm) {
          const uint2 q = *reinterpret_cast<const uint2*>(st + 4u * N * kPitch + 2u * g + j * kWidth + 16 * i);
          nr[0] = __uint_as_float(q.x);
          nr[1] = __uint_as_float(q.y);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          constexpr int pm[2] = {gperm(MU, 0), gperm(MU, 1)};
          constexpr int sg[2] = {gsign(MU, 0), gsign(MU, 1)};
          const int low = pm[u];  // the partner row, and the lower row that t_u feeds
          const uint32_t fu = sg[u] < 0 ? 0x80008000u : 0u;
          if constexpr (kDirect) {
            const uint32_t a[4] = {w[u][0].x, w[u][0].y, w[low][0].x, w[low][0].y};
            mma::op<P>(acc[j][u][0][i], a, one[0][0], sig[0][0] ^ fu);
            // row low: conj(c_u) W psi_u + W psi_low, conj(c) = c for real, -c for imaginary gammas
            mma::op<P>(acc[j][low][0][i], a, sig[0][0] ^ fu ^ (IM ? 0x80008000u : 0u), one[0][0]);
          } else {
#pragma unroll
            for (int c = 0; c < CG; c++) {
              float r[4] = {0.f, 0.f, 0.f, 0.f};
              if constexpr (CG == 1) {
                const uint32_t a[4] = {w[u][0].x, w[u][0].y, w[low][0].x, w[low][0].y};
                mma::op<P>(r, a, one[0][0], sig[0][0] ^ fu);
              } else {
                const uint32_t au[4] = {w[u][0].x, w[u][0].y, w[u][CG - 1].x, w[u][CG - 1].y};
                const uint32_t al[4] = {w[low][0].x, w[low][0].y, w[low][CG - 1].x, w[low][CG - 1].y};
                mma::op<P>(r, au, one[c][0], one[c][CG - 1]);
                mma::op<P>(r, al, sig[c][0] ^ fu, sig[c][CG - 1] ^ fu);
              }
              if constexpr (kNorm) r[0] *= nr[0], r[1] *= nr[0], r[2] *= nr[1], r[3] *= nr[1];
              float(&up)[4] = acc[j][u][c][i];
              float(&lo)[4] = acc[j][low][c][i];
#pragma unroll
              for (int k = 0; k < 4; k++) up[k] += r[k];
              // row low += conj(c_u) t_u, c_u = sigma g_u
              const float k0 = __uint_as_float(0x3f800000u ^ ((flip_s ^ fu) & 0x80000000u));
              if constexpr (IM) {  // -i k0 (x + i y) = k0 (y - i x)
                lo[0] = fmaf(k0, r[1], lo[0]);
                lo[1] = fmaf(-k0, r[0], lo[1]);
                lo[2] = fmaf(k0, r[3], lo[2]);
                lo[3] = fmaf(-k0, r[2], lo[3]);
              } else {
#pragma unroll
                for (int k = 0; k < 4; k++) lo[k] = fmaf(k0, r[k], lo[k]);
              }
            }
          }
        }
      }
    }
  };
  hop(std::integral_constant<int, 0>{});
  hop(std::integral_constant<int, 1>{});
  hop(std::integral_constant<int, 2>{});
  hop(std::integral_constant<int, 3>{});
  hop(std::integral_constant<int, 4>{});
  hop(std::integral_constant<int, 5>{});
  hop(std::integral_constant<int, 6>{});
  hop(std::integral_constant<int, 7>{});
  mma::wait_groups<0>();
  __syncwarp();

  // epilogue: out = a_r acc + b x in the storage precision, through the stage
  // that held x (in place), then stored in the field's contiguous order
  uint32_t* const st = rows + (8 % NST) * kStage;
#pragma unroll
  for (int i = 0; i < MT; i++) {
    float ca[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t r = 16u * i + 2u * g + h;
      ca[h] = A.a_rhs_f ? (r < count ? A.a_rhs_f[rhs0 + r] : 0.f) : A.af;
    }
#pragma unroll
    for (int j = 0; j < S; j++) {
      float bx[2] = {A.bf, A.bf};
      if constexpr (kNorm) {
        if (xin) {
          const uint2 q = *reinterpret_cast<const uint2*>(st + 4u * N * kPitch + 2u * g + j * kWidth + 16 * i);
          bx[0] *= __uint_as_float(q.x);
          bx[1] *= __uint_as_float(q.y);
        }
      }
      float mx[2] = {0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 4; s++)
#pragma unroll
        for (int c = 0; c < CG; c++) {
          const bool colour = (4 * c + 3 < N) || t + 4u * c < (uint32_t)N;
          uint32_t* const d = st + frag[c] + (uint32_t)(s * N + 4 * c) * kPitch + j * kWidth + 16 * i;
          uint2 x = make_uint2(0u, 0u);
          if (xin) x = *reinterpret_cast<const uint2*>(d);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float& re = acc[j][s][c][i][2 * h];
            float& im = acc[j][s][c][i][2 * h + 1];
            re *= ca[h];
            im *= ca[h];
            if (xin) {
              const float2 xc = mma::unpack<P>(h ? x.y : x.x);
              re = fmaf(bx[h], xc.x, re);
              im = fmaf(bx[h], xc.y, im);
            }
            if constexpr (kNorm) {
              if (colour) mx[h] = fmaxf(mx[h], fmaxf(fabsf(re), fabsf(im)));
            }
          }
        }
      float inv[2] = {1.f, 1.f};
      if constexpr (kNorm) {
        const uint32_t pos = group * S + j;
        const uint32_t osite = __shfl_sync(0xffffffffu, cs.site, j * (kWidth / 4));
#pragma unroll
        for (int h = 0; h < 2; h++) {  // the four lanes of an RHS row hold its colours
          mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
          mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
          inv[h] = mx[h] > 0.f ? 1.0f / mx[h] : 0.f;
          const uint32_t r = 16u * i + 2u * g + h;
          if (t == 0 && r < count && pos < vh && (!A.mask || A.mask[rhs0 + r]))
            A.out_norm[osite * nrhs + rhs0 + r] = mx[h];
        }
      }
      __syncwarp();  // the last colour's words of x have been read by every lane that repeats them
#pragma unroll
      for (int s = 0; s < 4; s++)
#pragma unroll
        for (int c = 0; c < CG; c++) {
          uint32_t w[2];
#pragma unroll
          for (int h = 0; h < 2; h++)
            w[h] = mma::pack<P>(acc[j][s][c][i][2 * h] * inv[h], acc[j][s][c][i][2 * h + 1] * inv[h]);
          if ((4 * c + 3 < N) || t + 4u * c < (uint32_t)N)
            *reinterpret_cast<uint2*>(st + frag[c] + (uint32_t)(s * N + 4 * c) * kPitch + j * kWidth + 16 * i) =
                make_uint2(w[0], w[1]);
        }
    }
  }
  __syncwarp();
  if (!copies || group * S + cj >= vh) return;
  uint32_t live = 15u;  // RHS of this lane's vectors that are not masked
  if (A.mask) {
    live = 0u;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) live |= A.mask[rhs0 + cr + k] != 0 ? 1u << k : 0u;
  }
  uint32_t* dst = static_cast<uint32_t*>(A.out) + (cs.site * T.sstr + src0);
  const uint32_t* src = st + lane_word;
#pragma unroll
  for (uint32_t k = 0; k < kCopies; k++, dst += src_step) {
    if (!kEven && r0 + k * kStep >= 4u * N) break;
    const uint4 w = *reinterpret_cast<const uint4*>(src + k * kStep * kPitch);
    if (live == 15u) {
      if (A.stream_out)
        __stcs(reinterpret_cast<uint4*>(dst), w);
      else
        *reinterpret_cast<uint4*>(dst) = w;
    } else {  // masked RHS keep their values
      if (live & 1u) dst[0] = w.x;
      if (live & 2u) dst[1] = w.y;
      if (live & 4u) dst[2] = w.z;
      if (live & 8u) dst[3] = w.w;
    }
  }
}

}  // namespace qcu
