"""The work that users of this library have it do, as measurable cases.

A program that uses the library initialises a session for its lattice, loads a
gauge configuration, and then works on many fields with it: the hop term on
resident multi-RHS fields, the reference's queue of caller fields, layout
transforms, whole solves.  The configuration is therefore what such a program
keeps: it depends on the lattice and the colour count only.  The fields
(sources, spinors) and, where a call takes the links themselves, the links
come from the seed.

Case fields: kind, n (colours), x, y, z, t, nrhs, and per kind

  hop       precision, parity, dagger, xpay    resident MRHS fields
  queue     precision, parity, dagger          pushBackFermions / startDslash
  full      dagger                             fullDslashQcu (links and field in one call)
  layout    precision                          lexicographic <-> resident, both parities
  segments  count                              one work list of small lattices
  solve     solver, inner, kappa, tol          even-odd Krylov solve
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mrhs_qcu_gb300 as Q

PRECISIONS = {"fp64": Q.QCU_DOUBLE_PRECISION, "fp32": Q.QCU_SINGLE_PRECISION, "fp16": Q.QCU_HALF_PRECISION,
              "bf16": Q.QCU_BF16_PRECISION, "bf16_site": Q.QCU_BF16_SITE_PRECISION}
COMPLEX_BYTES = {"fp64": 16, "fp32": 8, "fp16": 4, "bf16": 4, "bf16_site": 4}
REALS = {"fp64": torch.float64, "fp32": torch.float32, "bf16": torch.bfloat16, "bf16_site": torch.bfloat16}
SOLVERS = {"cg": Q.QCU_SOLVER_CG, "bicgstab": Q.QCU_SOLVER_BICGSTAB}
ANTIPERIODIC = True
XPAY = (-0.12 * 0.12, 1.0)  # out = a D in + b x, the second half of 1 - kappa^2 D D


# ---- the cases -------------------------------------------------------------
def _lattice(x, y, z, t):
    return {"x": x, "y": y, "z": z, "t": t}


def listed():
    return [
        # the smallest call: one hop on a test-size lattice, where the launch is the cost
        {"name": "hop_fp32_su3_8x8x8x8_r4", "kind": "hop", "n": 3, **_lattice(8, 8, 8, 8), "nrhs": 4,
         "precision": "fp32", "parity": 0, "dagger": 0, "xpay": False},
        # the headline: the FP32 hop on a production lattice, a full set of 12 spin-colour sources
        {"name": "hop_fp32_su3_32x32x32x64_r12", "kind": "hop", "n": 3, **_lattice(32, 32, 32, 64), "nrhs": 12,
         "precision": "fp32", "parity": 0, "dagger": 0, "xpay": False},
        # the 16-bit hop of a mixed-precision solve, its second half (dagger, xpay)
        {"name": "hop_bf16_su3_24x24x24x48_r12", "kind": "hop", "n": 3, **_lattice(24, 24, 24, 48), "nrhs": 12,
         "precision": "bf16", "parity": 0, "dagger": 1, "xpay": True},
        # SU(N) at a modest batch, component-major 16-bit fields
        {"name": "hop_bf16_su6_16x16x16x32_r16", "kind": "hop", "n": 6, **_lattice(16, 16, 16, 32), "nrhs": 16,
         "precision": "bf16", "parity": 1, "dagger": 0, "xpay": False},
        # SU(N) at a large batch, the tensor-core field layout
        {"name": "hop_bf16_site_su8_16x16x16x32_r64", "kind": "hop", "n": 8, **_lattice(16, 16, 16, 32), "nrhs": 64,
         "precision": "bf16_site", "parity": 0, "dagger": 0, "xpay": False},
        # SU(N) in FP32, as the inner hop of an FP32 SU(N) solve
        {"name": "hop_fp32_su6_16x16x16x32_r32", "kind": "hop", "n": 6, **_lattice(16, 16, 16, 32), "nrhs": 32,
         "precision": "fp32", "parity": 1, "dagger": 0, "xpay": True},
        # the reference's call sequence on caller fields, an uneven lattice and an odd queue, FP64
        {"name": "queue_fp64_su3_14x10x6x18_r5", "kind": "queue", "n": 3, **_lattice(14, 10, 6, 18), "nrhs": 5,
         "precision": "fp64", "parity": 1, "dagger": 1},
        # the reference's one-call operator: links and one full field, both parities
        {"name": "full_fp64_su3_12x12x12x24", "kind": "full", "n": 3, **_lattice(12, 12, 12, 24), "nrhs": 1,
         "dagger": 0},
        # lexicographic caller fields to resident ones and back, as around a chain of hops
        {"name": "layout_fp32_su3_24x24x24x48_r12", "kind": "layout", "n": 3, **_lattice(24, 24, 24, 48),
         "nrhs": 12, "precision": "fp32"},
        # many small lattices in one work list
        {"name": "segments_fp32_su3_16_of_8x8x8x8_r4", "kind": "segments", "n": 3, **_lattice(8, 8, 8, 8),
         "nrhs": 4, "count": 16},
        # the mixed-precision propagator solve, 12 sources to 1e-10
        {"name": "solve_cg_su3_24x24x24x48_r12", "kind": "solve", "n": 3, **_lattice(24, 24, 24, 48), "nrhs": 12,
         "solver": "cg", "inner": "fp32", "kappa": 0.12, "tol": 1e-10},
        # the SU(N) solve of a batch of sources, BiCGStab
        {"name": "solve_bicgstab_su4_16x16x16x32_r16", "kind": "solve", "n": 4, **_lattice(16, 16, 16, 32),
         "nrhs": 16, "solver": "bicgstab", "inner": "fp32", "kappa": 0.11, "tol": 1e-10},
    ]


def _dims(rng, low, high):
    """A lattice of about 2^low .. 2^high sites (spread over the logarithm); extents even, as the
    even-odd split wants them, and mostly no powers of two."""
    want = 2.0 ** rng.uniform(low, high)
    shape = [rng.uniform(0.7, 1.4) for _ in range(3)] + [rng.uniform(1.0, 2.2)]
    f = (want / math.prod(shape)) ** 0.25
    return _lattice(*(max(4, 2 * round(s * f / 2)) for s in shape))


def _cost(c):
    """About the seconds that the work of a case takes: FP64 arithmetic runs at about 1 TFLOP/s."""
    w = work(c)
    fp64 = c["kind"] == "full" or c.get("precision") == "fp64"
    return max(w["bytes"] / 6.5e12, w["flops"] / (1e12 if fp64 else 4e13))


def _draw(rng):
    kind = rng.choice(["hop", "hop", "hop", "queue", "full", "layout", "segments", "solve"])
    c = {"kind": kind}
    if kind == "hop":
        p = rng.choice(["fp32", "fp32", "bf16", "bf16_site", "fp64"])
        n = rng.choice([3, 4, 5, 6, 7, 8]) if p == "bf16_site" else rng.choice([3, 3, 4, 5, 6, 8])
        if p == "bf16_site":
            nrhs = 4 * rng.randint(1, 16)
        else:
            nrhs = min(64 if n > 3 else 24, round(2.0 ** rng.uniform(0.0, 6.0)))
        c.update(n=n, **_dims(rng, 11, 21 if n == 3 else 17), nrhs=nrhs, precision=p, parity=rng.randint(0, 1),
                 dagger=rng.randint(0, 1), xpay=rng.random() < 0.4)
    elif kind == "queue":
        c.update(n=rng.choice([3, 3, 4]), **_dims(rng, 11, 18), nrhs=rng.randint(1, 24), precision="fp64",
                 parity=rng.randint(0, 1), dagger=rng.randint(0, 1))
    elif kind == "full":
        c.update(n=3, **_dims(rng, 11, 19), nrhs=1, dagger=rng.randint(0, 1))
    elif kind == "layout":
        c.update(n=rng.choice([3, 3, 4, 6]), **_dims(rng, 12, 18), nrhs=rng.randint(1, 24),
                 precision=rng.choice(["fp32", "fp64", "bf16"]))
    elif kind == "segments":
        c.update(n=3, **_dims(rng, 10, 13), nrhs=2 * rng.randint(1, 6), count=rng.randint(2, 16))
    else:
        inner = rng.choice(["fp32", "fp32", "fp16", "bf16"])
        c.update(n=rng.choice([3, 3, 4]), **_dims(rng, 12, 18), nrhs=rng.randint(1, 16),
                 solver=rng.choice(["cg", "bicgstab"]), inner=inner, kappa=round(rng.uniform(0.10, 0.12), 3),
                 tol=rng.choice([1e-10, 1e-12]))
    return c


def draw(rng):
    """One more case of the same kinds and ranges; none larger than the headline or the listed solve."""
    largest = {"solve": "solve_cg_su3_24x24x24x48_r12"}
    most = {c["name"]: _cost(c) for c in listed()}
    while True:
        c = _draw(rng)
        if _cost(c) <= most[largest.get(c["kind"], "hop_fp32_su3_32x32x32x64_r12")]:
            return c


def work(case):
    """Bytes: each input read and each output written once (links of both parities once per call).
    Flops: 128 N^2 + 56 N per hop, output site and RHS (projection, link product, reconstruction)."""
    n, nrhs, kind = case["n"], case["nrhs"], case["kind"]
    vh = case["x"] * case["y"] * case["z"] * case["t"] // 2
    units = vh * nrhs
    hop = (128 * n * n + 56 * n) * units
    links = 8 * vh * n * n  # complex numbers
    spinor = 4 * n * units
    if kind == "hop":
        c = COMPLEX_BYTES[case["precision"]]
        return {"bytes": (links + (3 if case["xpay"] else 2) * spinor) * c,
                "flops": hop + (24 * n * units if case["xpay"] else 0)}
    if kind == "queue":  # caller fields are FP64, the links resident
        return {"bytes": 2 * spinor * 16 + links * COMPLEX_BYTES[case["precision"]], "flops": hop}
    if kind == "full":
        return {"bytes": 4 * spinor * 16 + links * 16, "flops": 2 * hop}
    if kind == "layout":  # caller field in, resident field out and in, caller field out
        return {"bytes": 4 * spinor * 16 + 4 * spinor * COMPLEX_BYTES[case["precision"]], "flops": 0}
    if kind == "segments":
        return {"bytes": case["count"] * (links + 2 * spinor) * 8, "flops": case["count"] * hop}
    # a solve: sources in, solutions out, the links; four hops per iteration, about 2.2 iterations
    # per decimal digit on these configurations
    iterations = round(-2.2 * math.log10(case["tol"]))
    return {"bytes": 4 * spinor * 16 + links * 16, "flops": 4 * iterations * hop}


# ---- inputs ----------------------------------------------------------------
def _generator(seed, *more):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.SeedSequence([int(seed), *map(int, more)]).generate_state(1, np.uint64)[0] >> 1))
    return g


def _shape(case):
    return [case["x"], case["y"], case["z"], case["t"]]


def _vh(case):
    return math.prod(_shape(case)) // 2


def _links(gen, count, n):
    """count Haar-random SU(n) matrices [count, n, n]: the phase-fixed QR of complex Gaussian ones, det = 1."""
    out = torch.empty((count, n, n), dtype=torch.complex128, device="cuda")
    for s in range(0, count, 1 << 20):
        m = min(1 << 20, count - s)
        a = torch.randn((m, n, n), dtype=torch.complex128, device="cuda", generator=gen)
        q = torch.empty_like(a)
        for k in range(n):
            v = a[:, :, k].clone()
            for j in range(k):
                v -= (q[:, :, j].conj() * v).sum(1, keepdim=True) * q[:, :, j]
            for j in range(k):  # once more: unitary to rounding, as a configuration is
                v -= (q[:, :, j].conj() * v).sum(1, keepdim=True) * q[:, :, j]
            q[:, :, k] = v / torch.linalg.vector_norm(v, dim=1, keepdim=True)
        if n == 3:
            det = (torch.linalg.cross(q[:, :, 0], q[:, :, 1], dim=1) * q[:, :, 2]).sum(1)
        else:
            det = torch.linalg.det(q)
        # |det q| = 1: dividing by the n-th root of its phase leaves det = 1
        q /= torch.polar(torch.ones_like(det.real), det.angle() / n)[:, None, None]
        out[s:s + m] = q
    return out


def _gauge(case, seed):
    """[mu 4][parity 2][Vh][n][n] complex double, the caller layout."""
    vh, n = _vh(case), case["n"]
    return _links(_generator(seed, 1, n, *_shape(case)), 8 * vh, n).view(4, 2, vh, n, n)


CONFIGURATION = 20  # the seed of the configuration that a program keeps
_resident = None    # what the library's session holds: (lattice, colours)


def _session(case):
    """The session of the case's lattice with its configuration, as a program sets it up once."""
    global _resident
    key = (*_shape(case), case["n"])
    if _resident != key:
        _resident = None
        Q.initGridSize(_shape(case), case["n"])
        Q.set_antiperiodic_t(ANTIPERIODIC)
        gauge = _gauge(case, CONFIGURATION)
        torch.cuda.synchronize()
        Q.loadQcuGauge(gauge.data_ptr())
        _resident = key


def _normal(shape, dtype, gen):
    """Gaussian reals of variance 1/2 (complex components of unit variance), made in pieces of modest size."""
    out = torch.empty(shape, dtype=dtype, device="cuda")
    flat = out.view(-1)
    for s in range(0, flat.numel(), 1 << 27):
        m = min(1 << 27, flat.numel() - s)
        made = torch.float64 if dtype == torch.float64 else torch.float32
        flat[s:s + m] = torch.randn(m, dtype=made, device="cuda", generator=gen) * math.sqrt(0.5)
    return out


def _fields(case, seed, parities):
    """Caller fields of every RHS, complex double: [nrhs][Vh][4][n], or [nrhs][2 Vh][4][n] for both parities."""
    r = _normal((case["nrhs"], parities * _vh(case), 4, case["n"], 2), torch.float64, _generator(seed, 2))
    return torch.view_as_complex(r)


def _resident_shape(case):
    vh, n, nrhs = _vh(case), case["n"], case["nrhs"]
    return (vh, 4 * n, nrhs, 2) if case.get("precision") == "bf16_site" else (4 * n, vh, nrhs, 2)


def prepare(case, seed):
    kind, nrhs = case["kind"], case["nrhs"]
    state = {"case": case}
    if kind == "hop":
        _session(case)
        prec, shape, real = PRECISIONS[case["precision"]], _resident_shape(case), REALS[case["precision"]]
        state["in"] = _normal(shape, real, _generator(seed, 3))
        state["x"] = _normal(shape, real, _generator(seed, 4)) if case["xpay"] else None
        state["out"] = torch.empty(shape, dtype=real, device="cuda")
        Q.tune_dslash(nrhs, prec)
    elif kind == "queue":
        _session(case)
        state["in"] = _fields(case, seed, 1)
        state["out"] = torch.empty_like(state["in"])
        Q.getDslash(Q.DSLASH_WILSON, 0.0, case["n"], nrhs, PRECISIONS[case["precision"]])
        Q.tune_dslash(nrhs, PRECISIONS[case["precision"]])
    elif kind == "full":
        Q.set_antiperiodic_t(ANTIPERIODIC)
        state["gauge"] = _gauge(case, seed)
        state["in"] = _fields(case, seed, 2)
        state["out"] = torch.empty_like(state["in"])
    elif kind == "layout":
        _session(case)
        state["in"] = _fields(case, seed, 2)
        state["out"] = torch.empty_like(state["in"])
        state["resident"] = [torch.empty(_resident_shape(case), dtype=REALS[case["precision"]], device="cuda")
                             for _ in range(2)]
    elif kind == "segments":
        vh, n, gen = _vh(case), case["n"], _generator(seed, 5)
        state["gauges"], state["in"], state["out"] = [], [], []
        for _ in range(case["count"]):
            u = _links(gen, 8 * vh, n).view(8, vh, n * n).transpose(1, 2).contiguous()  # [8][n n][Vh]
            state["gauges"].append(u.to(torch.complex64))
            state["in"].append(_normal((4 * n, vh, nrhs, 2), torch.float32, gen))
            state["out"].append(torch.empty((4 * n, vh, nrhs, 2), dtype=torch.float32, device="cuda"))
        state["list"] = [dict(lattice=_shape(case), gauge=g.data_ptr(), in_=i.data_ptr(), out=o.data_ptr(),
                              nrhs=nrhs, parity=k % 2, dagger=0, antiperiodic_t=ANTIPERIODIC)
                         for k, (g, i, o) in enumerate(zip(state["gauges"], state["in"], state["out"]))]
    else:
        _session(case)
        state["b"] = _fields(case, seed, 2)
        state["x"] = torch.zeros_like(state["b"])
        for p in (case["inner"], "fp64"):
            Q.tune_dslash(nrhs, PRECISIONS[p])
    return state


def run(state):
    case = state["case"]
    kind, nrhs = case["kind"], case["nrhs"]
    if kind == "hop":
        prec = PRECISIONS[case["precision"]]
        if case["xpay"]:
            Q.dslash_xpay_mrhs(state["out"].data_ptr(), None, state["in"].data_ptr(), None, state["x"].data_ptr(),
                               None, nrhs, case["parity"], case["dagger"], prec, *XPAY)
        else:
            Q.dslash_mrhs(state["out"].data_ptr(), None, state["in"].data_ptr(), None, nrhs, case["parity"],
                          case["dagger"], prec)
        return state["out"]
    if kind == "queue":
        for r in range(nrhs):
            Q.pushBackFermions(state["out"][r].data_ptr(), state["in"][r].data_ptr())
        Q.startDslash(case["parity"], case["dagger"])
        return state["out"]
    if kind == "full":
        Q.fullDslashQcu(state["out"].data_ptr(), state["in"].data_ptr(), state["gauge"].data_ptr(), _shape(case),
                        case["dagger"])
        return state["out"]
    if kind == "layout":
        prec = PRECISIONS[case["precision"]]
        for p in range(2):
            Q.pack_fermions(state["resident"][p].data_ptr(), None, [f.data_ptr() for f in state["in"]],
                            Q.QCU_SRC_LEX, p, prec)
        for p in range(2):
            Q.unpack_fermions([f.data_ptr() for f in state["out"]], state["resident"][p].data_ptr(), None,
                              Q.QCU_SRC_LEX, p, prec)
        return {"even": state["resident"][0], "odd": state["resident"][1], "back": state["out"]}
    if kind == "segments":
        Q.dslash_segments(state["list"], case["n"], Q.QCU_SINGLE_PRECISION)
        return state["out"]
    params = Q.solver_params(solver=SOLVERS[case["solver"]], inner_precision=PRECISIONS[case["inner"]],
                             kappa=case["kappa"], tol=case["tol"])
    Q.invert([f.data_ptr() for f in state["x"]], [f.data_ptr() for f in state["b"]], params)
    return state["x"]


# ---- the same in 64 bits, by torch alone -------------------------------------
# gamma_mu row r has one non-zero, in column PERM[mu][r], of value PHASE[mu][r] (DeGrand-Rossi basis)
PERM = ((3, 2, 1, 0), (3, 2, 1, 0), (2, 3, 0, 1), (2, 3, 0, 1))
PHASE = ((1j, 1j, -1j, -1j), (-1, 1, 1, -1), (1j, -1j, -1j, 1j), (1, 1, 1, 1))


def _coordinates(case, parity):
    """Coordinates (X, y, z, t) of the half-sites of one parity, in index order."""
    x, y, z, t = _shape(case)
    s = torch.arange(_vh(case), device="cuda")
    xh, s = s % (x // 2), s // (x // 2)
    yy, s = s % y, s // y
    zz, tt = s % z, s // z
    return 2 * xh + ((parity + yy + zz + tt) & 1), yy, zz, tt


def _index(case, c):
    """Half-site index of coordinates (within their own parity)."""
    x, y, z, _ = _shape(case)
    return ((c[3] * z + c[2]) * y + c[1]) * (x // 2) + c[0] // 2


def _hop(case, psi, gauge, parity, dagger):
    """D_parity psi: psi [4, n, Vh, R] complex double of the other parity, gauge [4, 2, Vh, n, n]."""
    n, f = case["n"], -1.0 if dagger else 1.0
    here, dims = _coordinates(case, parity), _shape(case)
    out = torch.zeros_like(psi)
    for mu in range(4):
        for step in (1, -1):
            to = list(here)
            to[mu] = (here[mu] + step) % dims[mu]
            nb = _index(case, to)
            if step > 0:
                u = gauge[mu, parity]
                s = -f
            else:
                u = gauge[mu, 1 - parity].index_select(0, nb).conj().transpose(1, 2)
                s = f
            if mu == 3 and ANTIPERIODIC:
                edge = here[3] == (dims[3] - 1 if step > 0 else 0)
                u = u * torch.where(edge, -1.0, 1.0)[:, None, None]
            p = psi.index_select(2, nb)
            for r in range(2):  # rows 2, 3 of the projected spinor follow from rows 0, 1
                h = p[r] + s * PHASE[mu][r] * p[PERM[mu][r]]
                low = PERM[mu][r]  # row `low` of 1 + s g is s g[low][r] times row r
                for a in range(n):
                    w = u[:, a, 0, None] * h[0]
                    for b in range(1, n):
                        w = torch.addcmul(w, u[:, a, b, None], h[b])
                    out[r, a] += w
                    out[low, a] += s * PHASE[mu][low] * w
            del p
    return out


def _by_component(fields):
    """Caller fields [nrhs, Vh, 4, n] -> [4, n, Vh, nrhs]."""
    return fields.permute(2, 3, 1, 0).contiguous()


def _to_caller(psi):
    return psi.permute(3, 2, 0, 1).contiguous()


def _solve(case, b, gauge, kappa):
    """x of M x = b, M = 1 - kappa D over both parities, by conjugate gradients on the even-odd normal equations."""
    vh = _vh(case)
    be, bo = _by_component(b[:, :vh]), _by_component(b[:, vh:])

    def schur(v, dagger):
        return v - kappa ** 2 * _hop(case, _hop(case, v, gauge, 1, dagger), gauge, 0, dagger)

    def dot(u, v):
        return (u.conj() * v).sum((0, 1, 2)).real

    rhs = be + kappa * _hop(case, bo, gauge, 0, 0)
    x, s = torch.zeros_like(rhs), rhs.clone()
    r = schur(s, 1)
    p, rr = r.clone(), dot(r, r)
    stop = 1e-15 ** 2 * dot(rhs, rhs)
    for _ in range(200):
        q = schur(p, 0)
        a = rr / dot(q, q)
        x += a * p
        s -= a * q
        r = schur(s, 1)
        new = dot(r, r)
        if bool((dot(s, s) < stop).all()):
            break
        p = r + (new / rr) * p
        rr = new
    xo = bo + kappa * _hop(case, x, gauge, 1, 0)
    return torch.cat([_to_caller(x), _to_caller(xo)], 1)


def exact(case, seed):
    kind, n, nrhs, vh = case["kind"], case["n"], case["nrhs"], _vh(case)
    if kind == "hop":
        shape, real = _resident_shape(case), REALS[case["precision"]]
        site = case["precision"] == "bf16_site"

        def load(tag):
            f = torch.view_as_complex(_normal(shape, real, _generator(seed, tag)).double())
            return (f.permute(1, 0, 2) if site else f).reshape(4, n, vh, nrhs)

        out = _hop(case, load(3), _gauge(case, CONFIGURATION), case["parity"], case["dagger"])
        if case["xpay"]:
            out = XPAY[0] * out + XPAY[1] * load(4)
        out = out.view(4 * n, vh, nrhs)
        return torch.view_as_real((out.permute(1, 0, 2) if site else out).contiguous())
    if kind == "queue":
        gauge = _gauge(case, CONFIGURATION)
        return _to_caller(_hop(case, _by_component(_fields(case, seed, 1)), gauge, case["parity"], case["dagger"]))
    if kind == "full":
        gauge, psi = _gauge(case, seed), _fields(case, seed, 2)
        half = [_by_component(psi[:, :vh]), _by_component(psi[:, vh:])]
        return torch.cat([_to_caller(_hop(case, half[1 - p], gauge, p, case["dagger"])) for p in range(2)], 1)
    if kind == "layout":
        x, y, z, _ = _shape(case)
        psi = _fields(case, seed, 2)
        got = {"back": None}  # 16-bit storage: rounded once, which torch does not offer from 64 bits
        if case["precision"] != "bf16":
            got["back"] = psi if case["precision"] == "fp64" else psi.to(torch.complex64).to(torch.complex128)
        for p, name in enumerate(("even", "odd")):
            c = _coordinates(case, p)
            lex = ((c[3] * z + c[2]) * y + c[1]) * x + c[0]
            half = _by_component(psi.index_select(1, lex)).view(4 * n, vh, nrhs)
            got[name] = torch.view_as_real(half)
        return got
    if kind == "segments":
        gen, outs = _generator(seed, 5), []
        for k in range(case["count"]):
            u = _links(gen, 8 * vh, n).to(torch.complex64).to(torch.complex128).view(4, 2, vh, n, n)
            psi = torch.view_as_complex(_normal((4 * n, vh, nrhs, 2), torch.float32, gen).double())
            out = _hop(case, psi.view(4, n, vh, nrhs), u, k % 2, 0)
            outs.append(torch.view_as_real(out.view(4 * n, vh, nrhs).contiguous()))
        return outs
    return _solve(case, _fields(case, seed, 2), _gauge(case, CONFIGURATION), case["kappa"])
