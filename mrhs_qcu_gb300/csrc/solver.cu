// Even-odd preconditioned Krylov solves of M x = b, M = 1 - kappa D, for many
// right-hand sides at once.  The reference has no solver: cg_inverter is an
// empty stub (src/qcu.cu:173 of the reference); this is new work built on the
// MRHS hopping kernel.
//
// Schur system on the even sites, per RHS r with its own kappa_r:
//   Mhat_r = 1 - kappa_r^2 D_eo D_oe,   bhat_r = b_e + kappa_r D_eo b_o,
//   x_o    = b_o + kappa_r D_oe x_e,    bhat_r - Mhat_r x_e = (b_e - x_e) + kappa_r D_eo x_o,
// and Mhat^dag = 1 - kappa^2 D_eo^- D_oe^- (the dagger flag f = -1), because
// D^dag = gamma5 D gamma5 is the hop with f = -1.  With x_o reconstructed
// that way, |b - M x| over the full lattice equals |bhat - Mhat x_e|.
// With a clover field (M = A - kappa D, A Hermitian and block diagonal in
// chirality, so A commutes with gamma5):
//   Mhat_r = A_ee - kappa_r^2 D_eo A_oo^-1 D_oe,  bhat_r = b_e + kappa_r D_eo A_oo^-1 b_o,
//   x_o    = A_oo^-1 (b_o + kappa_r D_oe x_e),   Mhat^dag = Mhat with f = -1.
//
// CG  : CG on Mhat^dag Mhat that also tracks s = bhat - Mhat x (the residual
//       of the actual system), so convergence is tested on |s| / |b|.
// BiCGStab on Mhat directly.
//
// Mixed precision: the Krylov vectors live in FP32 (or FP64 for the plain
// FP64 solve) and the operator runs in the inner precision (FP64, FP32,
// FP16 or BF16 storage).  FP64 is used for exactly three things: the solution
// accumulator x, the true residual bhat - Mhat x recomputed at each reliable
// update, and every inner product / norm (FP64 accumulation in the BLAS
// reductions).
//
// Slots.  The engine owns `capacity` RHS slots.  A slot is admitted (its
// source packed, its state initialised), iterates, and is retired (its
// solution unpacked) independently of the others: every per-RHS scalar
// (alpha, beta, kappa, tolerance, ...) and the activity mask live in device
// arrays, and every per-slot initialisation / update is a masked operation.
// Reliable updates are per slot too: slot r is updated when its own iterated
// residual has dropped by delta since its last update or reached its
// tolerance.  A slot's arithmetic therefore depends only on its own data and
// iteration count, not on which other slots are occupied.  Iterations run in
// chunks of 8 with no host round trip; a chunk is captured once as a CUDA
// graph and replayed.  Between chunks the host retires finished slots and
// admits new ones (continuous batching, used by the serving loop).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "solver.h"

namespace qcu {
namespace {

// The per-RHS scalar kernels sum the block partials of the reduction before
// them (one warp per RHS, 4 per block) and its lane 0 updates the slot.
constexpr int kScalarThreads = 128;
__device__ __forceinline__ int scalar_rhs() { return blockIdx.x * (kScalarThreads / 32) + (threadIdx.x >> 5); }

// alpha = |r|^2 / |q|^2
__global__ void cg_alpha_kernel(SolverScalars S, int nrhs, Partials P) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double q = sum_partials(P.norm, P.blocks, nrhs, r, lane);
  if (lane) return;
  double a = 0.0;
  if (S.active[r]) {
    if (q > 0.0 && isfinite(q)) {
      a = S.rr[r] / q;
    } else {
      S.active[r] = 0;
      S.upd[r] = 1;
    }
  }
  S.alpha[r] = make_double2(a, 0.0);
}

// the slot's residual ss: tolerance reached (or NaN) -> verify in FP64; dropped by delta -> reliable update
__device__ __forceinline__ void test_residual(const SolverScalars& S, int r, double ss, double delta2) {
  if (!(ss > S.stop2[r])) {
    S.active[r] = 0;
    S.upd[r] = 1;
  } else if (ss < delta2 * S.maxss[r]) {
    S.upd[r] = 1;
  }
}

// beta, convergence and reliable-update test per slot
__global__ void cg_beta_kernel(SolverScalars S, int nrhs, Partials P, double delta2) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double ss = sum_partials(P.norm, P.blocks, nrhs, r, lane);
  const double rr = sum_partials(P.norm2, P.blocks, nrhs, r, lane);
  if (lane) return;
  double b = 0.0;
  if (S.active[r]) {
    b = rr / S.rr[r];
    S.rr[r] = rr;
    test_residual(S, r, ss, delta2);
  }
  S.beta[r] = make_double2(b, 0.0);
}

// BiCGStab: alpha = rho / <r0, v>
__global__ void bicg_alpha_kernel(SolverScalars S, int nrhs, Partials P) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double2 d = sum_partials(P.dot, P.blocks, nrhs, r, lane);
  if (lane) return;
  double2 a = make_double2(0.0, 0.0);
  if (S.active[r]) {
    const double2 rho = S.rho[r];
    const double den = d.x * d.x + d.y * d.y;
    if (den > 0.0 && isfinite(den)) {
      a = make_double2((rho.x * d.x + rho.y * d.y) / den, (rho.y * d.x - rho.x * d.y) / den);
    } else {
      S.active[r] = 0;
      S.upd[r] = 1;
    }
  }
  S.alpha[r] = a;
  S.nalpha[r] = make_double2(-a.x, -a.y);
}

// omega = <t, s> / <t, t>
__global__ void bicg_omega_kernel(SolverScalars S, int nrhs, Partials P) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double2 ts = sum_partials(P.dot, P.blocks, nrhs, r, lane);
  const double tt = sum_partials(P.norm, P.blocks, nrhs, r, lane);
  if (lane) return;
  double2 w = make_double2(0.0, 0.0);
  if (S.active[r]) {
    if (tt > 0.0 && isfinite(tt)) {
      w = make_double2(ts.x / tt, ts.y / tt);
    } else {
      S.active[r] = 0;
      S.upd[r] = 1;
    }
  }
  S.omega[r] = w;
}

// beta = (rho_new / rho) (alpha / omega), rho_new = <r0, r>; test |r|
__global__ void bicg_beta_kernel(SolverScalars S, int nrhs, Partials P, double delta2) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double2 rn = sum_partials(P.dot, P.blocks, nrhs, r, lane);
  const double ss = sum_partials(P.norm, P.blocks, nrhs, r, lane);
  if (lane) return;
  double2 b = make_double2(0.0, 0.0), nbo = make_double2(0.0, 0.0);
  if (S.active[r]) {
    const double2 ro = S.rho[r], a = S.alpha[r], w = S.omega[r];
    const double d1 = ro.x * ro.x + ro.y * ro.y, d2 = w.x * w.x + w.y * w.y;
    if (d1 > 0.0 && d2 > 0.0 && isfinite(d1) && isfinite(d2)) {
      const double2 q1 = make_double2((rn.x * ro.x + rn.y * ro.y) / d1, (rn.y * ro.x - rn.x * ro.y) / d1);
      const double2 q2 = make_double2((a.x * w.x + a.y * w.y) / d2, (a.y * w.x - a.x * w.y) / d2);
      b = make_double2(q1.x * q2.x - q1.y * q2.y, q1.x * q2.y + q1.y * q2.x);
      nbo = make_double2(-(b.x * w.x - b.y * w.y), -(b.x * w.y + b.y * w.x));
      S.rho[r] = rn;
    } else {
      S.active[r] = 0;
      S.upd[r] = 1;
    }
    if (S.active[r]) test_residual(S, r, ss, delta2);
  }
  S.beta[r] = b;
  S.nbo[r] = nbo;
}

// after a (re)start of the selected slots: rr, maxss from the fresh residuals;
// the CG invariant <r, p> = |r|^2 restored by p += c r with
// c = 1 - <r, p> / |r|^2 (fresh slots have p = 0, so p becomes r).  The
// update p += c r runs over every slot, so c = 0 for the slots not restarted.
__global__ void restart_kernel(SolverScalars S, int nrhs, Partials P) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double rr = sum_partials(P.norm, P.blocks, nrhs, r, lane);
  const double2 rp = sum_partials(P.dot, P.blocks, nrhs, r, lane);
  if (lane) return;
  double2 c = make_double2(0.0, 0.0);
  if (S.sel[r]) {
    S.rr[r] = rr;
    S.maxss[r] = S.ss_true[r];
    S.upd[r] = 0;
    if (rr > 0.0 && isfinite(rr)) c = make_double2(1.0 - rp.x / rr, -rp.y / rr);
  }
  S.tmp2[r] = c;
}

// BiCGStab restart of the selected slots: r0 = r, so rho = <r0, r> = |r|^2
__global__ void bicg_restart_kernel(SolverScalars S, int nrhs, Partials P) {
  const int r = scalar_rhs(), lane = threadIdx.x & 31;
  if (r >= nrhs) return;
  const double rr = sum_partials(P.norm, P.blocks, nrhs, r, lane);
  if (lane || !S.sel[r]) return;
  S.maxss[r] = S.ss_true[r];
  S.upd[r] = 0;
  S.rho[r] = make_double2(rr, 0.0);
}

}  // namespace

FieldRef SlotEngine::ref(const FieldView& f) const {
  FieldRef r;
  r.data = f.data;
  r.prec = f.prec;
  r.nrhs = f.nrhs;
  r.n = (int64_t)s_.geo.vh * 4 * s_.N * f.nrhs;
  return r;
}

// (an upper bound by two FP64 fields; admission keeps it, so a budget admits what it always did)
size_t SlotEngine::bytes_needed(const Session& s, int capacity, int inner_prec) {
  const int kp = inner_prec == PREC_DOUBLE ? PREC_DOUBLE : PREC_SINGLE;
  size_t b = 8 * s.field_bytes(PREC_DOUBLE, capacity) + 7 * s.field_bytes(kp, capacity);
  if (s.has_clover()) b += s.field_bytes(PREC_DOUBLE, capacity) + s.field_bytes(inner_prec, capacity) +
                           s.norm_bytes(inner_prec, capacity);
  if (inner_prec != kp) b += 3 * (s.field_bytes(inner_prec, capacity) + s.norm_bytes(inner_prec, capacity));
  b += s.field_bytes(inner_prec, capacity) + s.norm_bytes(inner_prec, capacity);
  return b;
}

SlotEngine::SlotEngine(Session& s, int capacity, const SolveRequest& q, const std::string& tag)
    : s_(s), n_(capacity), q_(q) {
  inject_failure("solver");
  QCU_REQUIRE(capacity >= 1 && capacity <= QCU_MAX_RHS, QCU_ERR_INVALID_ARGUMENT, "slot capacity must be in 1..256");
  QCU_REQUIRE(q.solver == 0 || q.solver == 1, QCU_ERR_INVALID_ARGUMENT, "unknown solver");
  QCU_REQUIRE(prec_valid(q.inner_prec), QCU_ERR_INVALID_ARGUMENT, "bad inner precision");
  QCU_REQUIRE(!(q.clover && prec_site_major(q.inner_prec)), QCU_ERR_UNSUPPORTED,
              "clover: site-major BF16 fields are not supported");
  QCU_REQUIRE(!prec_site_major(q.inner_prec) || capacity % 4 == 0, QCU_ERR_UNSUPPORTED,
              "site-major BF16 inner fields take the tensor-core dslash: the RHS count must be a multiple of 4");
  kp_ = q.inner_prec == PREC_DOUBLE ? PREC_DOUBLE : PREC_SINGLE;
  op_ = q.inner_prec;
  delta2_ = (q.inner_prec == PREC_DOUBLE) ? 0.0 : q.delta * q.delta;
  st_ = s.stream();
  const std::string t = tag + ".";
  be_ = s.alloc_field(t + "be", PREC_DOUBLE, n_);
  bo_ = s.alloc_field(t + "bo", PREC_DOUBLE, n_);
  xh_ = s.alloc_field(t + "xh", PREC_DOUBLE, n_);
  xo_ = s.alloc_field(t + "xo", PREC_DOUBLE, n_);
  sh_ = s.alloc_field(t + "sh", PREC_DOUBLE, n_);
  dh_ = s.alloc_field(t + "dh", PREC_DOUBLE, n_);
  xl_ = s.alloc_field(t + "xl", kp_, n_);
  sl_ = s.alloc_field(t + "sl", kp_, n_);
  rl_ = s.alloc_field(t + "rl", kp_, n_);
  pl_ = s.alloc_field(t + "pl", kp_, n_);
  ql_ = s.alloc_field(t + "ql", kp_, n_);
  wl_ = s.alloc_field(t + "wl", kp_, n_);
  if (q.solver == 1) r0l_ = s.alloc_field(t + "r0l", kp_, n_);
  if (op_ != kp_) {
    pop_ = s.alloc_field(t + "pop", op_, n_);
    qop_ = s.alloc_field(t + "qop", op_, n_);
    wop_ = s.alloc_field(t + "wop", op_, n_);
  }
  tmpop_ = s.alloc_field(t + "tmpop", op_, n_);
  // BF16 operator fields are internal: they take the site-major layout where
  // the tensor-core dslash on it is measured faster (same bytes either way)
  if (op_ == PREC_BF16 && !q.clover && s.prefer_site_major(pop_, qop_)) {
    op_ = PREC_BF16S;
    for (FieldView* f : {&pop_, &qop_, &wop_, &tmpop_}) f->prec = PREC_BF16S;
  }
  cl_ = q.clover;
  QCU_REQUIRE(!cl_ || s.has_clover(), QCU_ERR_NO_OPERATOR, "clover solve requested but no clover field loaded");
  if (cl_) {
    tmp64b_ = s.alloc_field(t + "tmp64b", PREC_DOUBLE, n_);
    tmpopb_ = s.alloc_field(t + "tmpopb", op_, n_);
  }
  // per-slot device scalars
  const int R = QCU_MAX_RHS;
  const size_t scalar_bytes = (size_t)R * (8 * sizeof(double) + 8 * sizeof(double2) + sizeof(float) + 3 * sizeof(int));
  char* d = static_cast<char*>(s.ws.get(t + "scalars", scalar_bytes));
  auto take = [&](auto*& p) {
    p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(d);
    d += R * sizeof(*p);
  };
  char* const base = d;
  for (double2** p : {&S_.alpha, &S_.nalpha, &S_.beta, &S_.omega, &S_.rho, &S_.tmp2, &S_.nbo, &S_.one}) take(*p);
  for (double** p : {&S_.rr, &S_.ss_true, &S_.maxss, &S_.stop2, &S_.bb, &S_.bo2, &S_.kap_d, &S_.nk2_d}) take(*p);
  take(S_.nk2_f);
  for (int** p : {&S_.active, &S_.upd, &S_.sel}) take(*p);
  host_.assign(n_, SlotState{});
  // The fields stay as they are: a slot's fields are written (moves, never
  // products with a zero coefficient) when it is admitted, and no operation
  // mixes slots.
  QCU_CHECK_CUDA(cudaMemsetAsync(base, 0, scalar_bytes, st_));
  std::vector<double> one(2 * n_, 0.0);
  for (int r = 0; r < n_; r++) one[2 * r] = 1.0;
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.one, one.data(), sizeof(double2) * n_, cudaMemcpyHostToDevice, st_));
  s.blas();  // BLAS scratch, before any graph capture
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
}

SlotEngine::~SlotEngine() {
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
}

std::vector<int> SlotEngine::free_slots() const {
  std::vector<int> f;
  for (int r = 0; r < n_; r++)
    if (host_[r].phase == SlotState::FREE) f.push_back(r);
  return f;
}

int SlotEngine::active_slots() const {
  int k = 0;
  for (int r = 0; r < n_; r++) k += host_[r].phase == SlotState::ACTIVE;
  return k;
}

void SlotEngine::upload_sel(const std::vector<int>& slots) {
  std::vector<int> m(n_, 0);
  for (int r : slots) m[r] = 1;
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.sel, m.data(), sizeof(int) * n_, cudaMemcpyHostToDevice, st_));
  // the upload reads host memory asynchronously: keep it alive until done
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
}

void SlotEngine::upload_kappa() {
  std::vector<double> k(n_), nk2(n_);
  std::vector<float> nk2f(n_);
  for (int r = 0; r < n_; r++) {
    k[r] = host_[r].kappa;
    nk2[r] = -host_[r].kappa * host_[r].kappa;
    nk2f[r] = (float)nk2[r];
  }
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.kap_d, k.data(), sizeof(double) * n_, cudaMemcpyHostToDevice, st_));
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.nk2_d, nk2.data(), sizeof(double) * n_, cudaMemcpyHostToDevice, st_));
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.nk2_f, nk2f.data(), sizeof(float) * n_, cudaMemcpyHostToDevice, st_));
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
}

// out = Mhat in (dagger 0) or Mhat^dag in (dagger 1) for the slots in mask,
// fields in precision `prec` with per-slot kappa
void SlotEngine::apply_mhat(const FieldView& out, const FieldView& in, const FieldView& tmp, const FieldView& tmp2,
                            int dagger, const int* mask) {
  s_.hop(tmp, in, FieldView{}, 1, dagger, 1.0, 0.0, mask);
  FieldView hop_in = tmp, x = in;
  if (cl_) {  // A_oo^-1 D_oe in, and A_ee in for the xpay term
    s_.clover_apply(tmp2, tmp, FieldView{}, 1, true, 1.0, 0.0, mask);
    s_.clover_apply(tmp, in, FieldView{}, 0, false, 1.0, 0.0, mask);
    hop_in = tmp2;
    x = tmp;
  }
  if (in.prec == PREC_DOUBLE)
    s_.hop(out, hop_in, x, 0, dagger, 0.0, 1.0, mask, nullptr, S_.nk2_d);
  else
    s_.hop(out, hop_in, x, 0, dagger, 0.0, 1.0, mask, S_.nk2_f, nullptr);
}

// Krylov-precision out = Mhat in (or Mhat^dag) for the slots in mask
void SlotEngine::op_apply(const FieldView& out_kp, const FieldView& in_kp, int dagger, const int* mask) {
  if (op_ == kp_) {
    apply_mhat(out_kp, in_kp, tmpop_, tmpopb_, dagger, mask);
  } else {
    convert_field(kp_, in_kp.data, nullptr, op_, pop_.data, pop_.norm, s_.geo.vh, 4 * s_.N, n_, st_, mask);
    apply_mhat(qop_, pop_, tmpop_, tmpopb_, dagger, mask);
    convert_field(op_, qop_.data, qop_.norm, kp_, out_kp.data, nullptr, s_.geo.vh, 4 * s_.N, n_, st_, mask);
  }
}

void SlotEngine::cg_iteration() {
  Blas& B = s_.blas();
  if (op_ == kp_) {
    apply_mhat(ql_, pl_, tmpop_, tmpopb_, 0, S_.active);
    apply_mhat(wl_, ql_, tmpop_, tmpopb_, 1, S_.active);
  } else {
    convert_field(kp_, pl_.data, nullptr, op_, pop_.data, pop_.norm, s_.geo.vh, 4 * s_.N, n_, st_, S_.active);
    apply_mhat(qop_, pop_, tmpop_, tmpopb_, 0, S_.active);
    apply_mhat(wop_, qop_, tmpop_, tmpopb_, 1, S_.active);
    convert_field(op_, qop_.data, qop_.norm, kp_, ql_.data, nullptr, s_.geo.vh, 4 * s_.N, n_, st_, S_.active);
    convert_field(op_, wop_.data, wop_.norm, kp_, wl_.data, nullptr, s_.geo.vh, 4 * s_.N, n_, st_, S_.active);
  }
  const Partials qq = B.norm2_partials(ref(ql_), st_);
  cg_alpha_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, qq);
  // s -= a q, r -= a w with their norms; then x += a p, p = r + b p in one pass over p
  const Partials sr = B.cg_update(S_.alpha, ref(ql_), ref(sl_), ref(wl_), ref(rl_), st_);
  cg_beta_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, sr, delta2_);
  B.cg_direction(S_.alpha, S_.beta, ref(rl_), ref(pl_), ref(xl_), st_);
}

void SlotEngine::bicg_iteration() {
  Blas& B = s_.blas();
  op_apply(ql_, pl_, 0, S_.active);  // v = Mhat p
  const Partials rv = B.dot_partials(ref(r0l_), ref(ql_), st_);
  bicg_alpha_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, rv);
  B.axpby(S_.nalpha, ref(ql_), nullptr, ref(sl_), st_);  // s = r - alpha v (sl holds r)
  op_apply(wl_, sl_, 0, S_.active);                       // t = Mhat s
  const Partials ts = B.dot_norm(ref(wl_), ref(sl_), st_);
  bicg_omega_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, ts);
  // x += alpha p + omega s, r = s - omega t, with |r|^2 and <r0, r>
  const Partials rr = B.bicg_update(S_.alpha, S_.omega, ref(pl_), ref(sl_), ref(wl_), ref(r0l_), ref(xl_), st_);
  bicg_beta_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, rr, delta2_);
  B.axpbypcz(S_.one, ref(sl_), S_.nbo, ref(ql_), S_.beta, ref(pl_), st_);  // p = r + beta p - beta omega v
}

void SlotEngine::run_chunk(int k) {
  if (q_.use_graph && k == chunk_) {
    if (!graph_exec_) {
      // kernel shapes are tuned in the first (eager) chunk; later chunks replay a graph
      if (!warm_) {
        for (int i = 0; i < k; i++) q_.solver == 0 ? cg_iteration() : bicg_iteration();
        warm_ = true;
        return;
      }
      cudaGraph_t g;
      QCU_CHECK_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
      try {
        for (int i = 0; i < k; i++) q_.solver == 0 ? cg_iteration() : bicg_iteration();
      } catch (...) {
        cudaGraph_t dummy = nullptr;
        cudaStreamEndCapture(st_, &dummy);
        if (dummy) cudaGraphDestroy(dummy);
        throw;
      }
      QCU_CHECK_CUDA(cudaStreamEndCapture(st_, &g));
      QCU_CHECK_CUDA(cudaGraphInstantiate(&graph_exec_, g, 0));
      QCU_CHECK_CUDA(cudaGraphDestroy(g));
    }
    QCU_CHECK_CUDA(cudaGraphLaunch(graph_exec_, st_));
  } else {
    for (int i = 0; i < k; i++) q_.solver == 0 ? cg_iteration() : bicg_iteration();
  }
}

// out = M_oo^-1 (b_o + kappa D_oe x_e): x_o of the slots in sel
void SlotEngine::odd_solution() {
  if (cl_) {
    s_.hop(tmp64b_, xh_, bo_, 1, 0, 0.0, 1.0, S_.sel, nullptr, S_.kap_d);
    s_.clover_apply(xo_, tmp64b_, FieldView{}, 1, true, 1.0, 0.0, S_.sel);
  } else {
    s_.hop(xo_, xh_, bo_, 1, 0, 0.0, 1.0, S_.sel, nullptr, S_.kap_d);
  }
}

// (Re)start the slots in `slots`: fold x_lo into x, recompute the true
// residual in FP64, decide convergence, and restart the Krylov recurrence of
// the slots that go on.  With x_o = b_o + kappa D_oe x_e the residual is
//   s = bhat - Mhat x_e = (b_e - x_e) + kappa D_eo x_o
// (clover: x_o = A_oo^-1 (..), s = (b_e - A_ee x_e) + kappa D_eo x_o), so a
// reliable update also leaves the odd half of the solution, and bhat itself
// is never formed.  `fresh` slots start from x = 0 with p = r.
void SlotEngine::restart(const std::vector<int>& slots, bool fresh) {
  if (slots.empty()) return;
  Blas& B = s_.blas();
  upload_sel(slots);
  if (fresh) {
    // s = b_e + kappa D_eo b_o (clover: b_e + kappa D_eo A_oo^-1 b_o)
    for (const FieldView* f : {&xl_, &xh_, &pl_}) B.select_copy(S_.sel, FieldRef{}, ref(*f), FieldRef{}, st_);
    FieldView odd = bo_;
    if (cl_) {
      s_.clover_apply(tmp64b_, bo_, FieldView{}, 1, true, 1.0, 0.0, S_.sel);
      odd = tmp64b_;
    }
    s_.hop(sh_, odd, be_, 0, 0, 0.0, 1.0, S_.sel, nullptr, S_.kap_d);
  } else {
    B.fold(S_.sel, ref(xl_), ref(xh_), ref(be_), cl_ ? FieldRef{} : ref(dh_), st_);
    odd_solution();
    if (cl_) s_.clover_apply(dh_, xh_, be_, 0, false, -1.0, 1.0, S_.sel);
    s_.hop(sh_, xo_, dh_, 0, 0, 0.0, 1.0, S_.sel, nullptr, S_.kap_d);
  }
  B.residual(S_.sel, ref(sh_), ref(sl_), S_.ss_true, st_);  // |s|^2, and s_lo = s
  std::vector<double> ss(n_);
  QCU_CHECK_CUDA(cudaMemcpyAsync(ss.data(), S_.ss_true, sizeof(double) * n_, cudaMemcpyDeviceToHost, st_));
  std::vector<int> act(n_);
  QCU_CHECK_CUDA(cudaMemcpyAsync(act.data(), S_.active, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
  std::vector<int> go_on;
  for (int r : slots) {
    SlotState& h = host_[r];
    h.true_res2 = ss[r];
    h.updates += fresh ? 0 : 1;
    if (verbose_)
      fprintf(stderr, "qcu solver: slot %d %s after %d iterations, true |s|/|b| %.3e\n", r,
              fresh ? "admitted" : "reliable update", h.iterations, std::sqrt(ss[r] / h.bb));
    if (ss[r] <= h.stop2) {
      h.phase = SlotState::DONE;
      h.converged = 1;
      act[r] = 0;
    } else if (h.iterations >= q_.max_iter || !std::isfinite(ss[r])) {
      h.phase = SlotState::DONE;
      h.converged = 0;
      act[r] = 0;
    } else {
      h.phase = SlotState::ACTIVE;
      act[r] = 1;
      go_on.push_back(r);
    }
  }
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.active, act.data(), sizeof(int) * n_, cudaMemcpyHostToDevice, st_));
  if (go_on.empty()) {
    QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
    return;
  }
  if (go_on.size() != slots.size()) upload_sel(go_on);
  if (q_.solver == 0) {
    op_apply(rl_, sl_, 1, S_.sel);  // r = Mhat^dag s
    const Partials rp = B.dot_norm(ref(rl_), ref(pl_), st_);
    restart_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, rp);
    B.axpby(S_.tmp2, ref(rl_), nullptr, ref(pl_), st_);  // p += c r
  } else {
    B.select_copy(S_.sel, ref(sl_), ref(r0l_), ref(pl_), st_);  // shadow residual r0 = r, p = r
    const Partials rr = B.norm2_partials(ref(sl_), st_);
    bicg_restart_kernel<<<scalar_blocks(), kScalarThreads, 0, st_>>>(S_, n_, rr);
  }
  QCU_CHECK_CUDA(cudaGetLastError());
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
}

void SlotEngine::admit(const std::vector<int>& slots, void* const* b, const double* kappa, const double* tol,
                       int src_mode) {
  if (slots.empty()) return;
  Blas& B = s_.blas();
  PtrArray pb{};
  for (size_t i = 0; i < slots.size(); i++) {
    const int r = slots[i];
    QCU_REQUIRE(r >= 0 && r < n_ && host_[r].phase == SlotState::FREE, QCU_ERR_INVALID_ARGUMENT,
                "admit: slot is not free");
    QCU_REQUIRE(tol[i] > 0 && kappa[i] > 0, QCU_ERR_INVALID_ARGUMENT, "kappa and tol must be positive");
    pb.p[r] = b[i];
    SlotState& h = host_[r];
    h = SlotState{};
    h.kappa = kappa[i];
    h.tol = tol[i];
    h.phase = SlotState::ACTIVE;
  }
  upload_kappa();
  pack_fermions(PREC_DOUBLE, s_.N, pb, src_mode, 0, be_.data, nullptr, s_.geo, n_, st_);
  pack_fermions(PREC_DOUBLE, s_.N, pb, src_mode, 1, bo_.data, nullptr, s_.geo, n_, st_);
  // |b|^2 over both parities; the slot stops when |s|^2 <= tol^2 |b|^2
  B.norm2(ref(be_), S_.bb, st_);
  B.norm2(ref(bo_), S_.bo2, st_);
  std::vector<double> bb(n_), bo2(n_), stop2(n_);
  QCU_CHECK_CUDA(cudaMemcpyAsync(bb.data(), S_.bb, sizeof(double) * n_, cudaMemcpyDeviceToHost, st_));
  QCU_CHECK_CUDA(cudaMemcpyAsync(bo2.data(), S_.bo2, sizeof(double) * n_, cudaMemcpyDeviceToHost, st_));
  QCU_CHECK_CUDA(cudaMemcpyAsync(stop2.data(), S_.stop2, sizeof(double) * n_, cudaMemcpyDeviceToHost, st_));
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
  for (int r : slots) {
    SlotState& h = host_[r];
    const double b2 = bb[r] + bo2[r];
    // a non-finite source is not solved: its true residual is non-finite, so
    // restart() finishes the slot unconverged, and the caller is told why
    h.bad_source = std::isfinite(b2) ? 0 : 1;
    h.bb = (b2 > 0 && std::isfinite(b2)) ? b2 : 1.0;  // a zero source: x = 0 is exact
    h.stop2 = h.tol * h.tol * h.bb;
    stop2[r] = h.stop2;
  }
  QCU_CHECK_CUDA(cudaMemcpyAsync(S_.stop2, stop2.data(), sizeof(double) * n_, cudaMemcpyHostToDevice, st_));
  restart(slots, true);
}

std::vector<int> SlotEngine::step() {
  std::vector<int> finished;
  for (int r = 0; r < n_; r++)
    if (host_[r].phase == SlotState::DONE && !host_[r].reported) {
      host_[r].reported = true;
      finished.push_back(r);
    }
  if (active_slots() == 0) return finished;
  const int k = chunk_;
  run_chunk(k);
  std::vector<int> act(n_), upd(n_);
  QCU_CHECK_CUDA(cudaMemcpyAsync(act.data(), S_.active, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
  QCU_CHECK_CUDA(cudaMemcpyAsync(upd.data(), S_.upd, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
  s_.sync();
  std::vector<int> sel;
  for (int r = 0; r < n_; r++) {
    if (host_[r].phase != SlotState::ACTIVE) continue;
    host_[r].iterations += k;
    if (upd[r] || !act[r] || host_[r].iterations >= q_.max_iter) sel.push_back(r);
  }
  restart(sel, false);
  for (int r : sel)
    if (host_[r].phase == SlotState::DONE && !host_[r].reported) {
      host_[r].reported = true;
      finished.push_back(r);
    }
  return finished;
}

void SlotEngine::retire(const std::vector<int>& slots, void* const* x, int src_mode) {
  if (slots.empty()) return;
  PtrArray px{};
  for (size_t i = 0; i < slots.size(); i++) {
    const int r = slots[i];
    QCU_REQUIRE(r >= 0 && r < n_ && host_[r].phase == SlotState::DONE, QCU_ERR_INVALID_ARGUMENT,
                "retire: slot has not finished");
    px.p[r] = x[i];
  }
  // x_o is the last reliable update's; a slot that finished without one has x = 0, so x_o is still to be formed
  std::vector<int> untouched;
  for (int r : slots)
    if (host_[r].updates == 0) untouched.push_back(r);
  if (!untouched.empty()) {
    upload_sel(untouched);
    odd_solution();
  }
  unpack_fermions(PREC_DOUBLE, s_.N, px, src_mode, 0, xh_.data, nullptr, s_.geo, n_, st_);
  unpack_fermions(PREC_DOUBLE, s_.N, px, src_mode, 1, xo_.data, nullptr, s_.geo, n_, st_);
  QCU_CHECK_CUDA(cudaStreamSynchronize(st_));
  for (int r : slots) host_[r].phase = SlotState::FREE;
}

SolveResult solve(Session& s, void* const* x, void* const* b, int nrhs, const SolveRequest& req) {
  QCU_REQUIRE(nrhs >= 1 && nrhs <= QCU_MAX_RHS, QCU_ERR_INVALID_ARGUMENT, "nrhs must be in 1..256");
  QCU_REQUIRE(req.tol > 0 && req.max_iter > 0, QCU_ERR_INVALID_ARGUMENT, "tol and max_iter must be positive");
  QCU_REQUIRE(req.src_mode == SRC_EO_FULL || req.src_mode == SRC_LEX, QCU_ERR_INVALID_ARGUMENT,
              "solver fields must be full eo or lexicographic");
  auto t0 = std::chrono::steady_clock::now();
  SlotEngine eng(s, nrhs, req, "sv");
  std::vector<int> slots(nrhs);
  std::vector<double> kap(nrhs, req.kappa), tol(nrhs, req.tol);
  for (int r = 0; r < nrhs; r++) slots[r] = r;
  eng.admit(slots, b, kap.data(), tol.data(), req.src_mode);
  int chunks = 0;
  while (eng.active_slots() > 0) {
    eng.step();
    chunks++;
  }
  eng.retire(slots, x, req.src_mode);
  SolveResult res;
  res.true_residual.resize(nrhs);
  res.converged.resize(nrhs);
  res.bad_source.resize(nrhs);
  for (int r = 0; r < nrhs; r++) {
    const SlotState& h = eng.slot(r);
    res.true_residual[r] = std::sqrt(h.true_res2 / h.bb);
    res.converged[r] = h.converged;
    res.bad_source[r] = h.bad_source;
    res.iterations = std::max(res.iterations, h.iterations);
    res.reliable_updates = std::max(res.reliable_updates, h.updates);
  }
  res.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  (void)chunks;
  return res;
}

}  // namespace qcu
