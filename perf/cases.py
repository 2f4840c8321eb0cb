"""What a user of the framework has it do, as measurable cases.

The framework's path is Dirac operators on a lattice gauge field and the
linear solves, link smearing and link gradients built on them.  A case is one
call (or one short sequence of calls) of that path through the package's
public entry points, on synthetic fields: links near exp(i a H) with H random
traceless Hermitian, Gaussian sources, antiperiodic in t.

`listed()` spans the sizes the path is used at: an 8^4 solve where latency and
launches count, single operator applications, the 32^3x64 production solves,
odd extents, forward operators and backward link gradients, FP64 and the FP32
and int16 storage of the mixed solvers.  `draw()` gives further cases of the
same kinds.  `exact()` restates every kind in plain torch in 64 bits.
"""
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "latticematrices.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lmb200 as lmb  # noqa: E402

PHASES = (1, 1, 1, -1)
EPS_NAIK = -0.083
CSW = 1.0

# Parameters of the operators as the configurations and the benchmark use
# them: amplitude a of the links, the mass-like parameter, and about how many
# conjugate-gradient iterations a solve to 1e-10 takes with them.
OPS = {
    "wilson": dict(amplitude=0.3, kappa=0.125, iterations=130),
    "clover": dict(amplitude=0.2, kappa=0.1355, iterations=450),
    "staggered": dict(amplitude=0.25, mass=0.05, iterations=180),
    "hisq": dict(amplitude=0.25, mass=0.01, iterations=280),
    "domainwall": dict(amplitude=0.2, mass=0.1, M=-1.0, b=2.0, c=1.0, iterations=500),
}
BATCH = dict(amplitude=0.2, kappa=0.12, iterations=210)
EVENODD_ITERATIONS = 141
FORCE_MASS = 0.02


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest solve: the plain Wilson configuration, 8^4, FP64; every
        # iteration is a handful of microseconds
        dict(name="wilson_cg_8", kind="cg", op="wilson", L="8x8x8x8", precision="double"),
        # the headline production solve: Wilson-clover, int16 inner iterations
        # with FP64 reliable updates
        dict(name="clover_cg_32x64_half", kind="cg", op="clover", L="32x32x32x64", precision="half"),
        # the same operator in plain FP64 on a middle lattice
        dict(name="clover_cg_24x48_double", kind="cg", op="clover", L="24x24x24x48", precision="double"),
        # D and D^+ applied once each by a user's own Krylov loop, odd extents
        dict(name="clover_apply_odd", kind="apply", op="clover", L="21x15x17x27", precision="double"),
        # D x = b for a propagator, even/odd preconditioned, int16 inner
        dict(name="evenodd_24x48_half", kind="evenodd", op="clover", L="24x24x24x48", precision="half"),
        # many right-hand sides on lattices of uneven size in one call, FP32
        dict(name="batched_16_8_single", kind="batched", L="16x16x16x16:8,8x8x8x8:4", precision="single"),
        # one HISQ application with the refresh of the output's halo: the
        # protocol of the published Dslash study
        dict(name="hisq_apply_16", kind="apply", op="hisq", L="16x16x16x16", precision="double"),
        # staggered-type solve on smeared links, FP32 inner iterations
        dict(name="hisq_cg_32x64_single", kind="cg", op="hisq", L="32x32x32x64", precision="single"),
        # a gauge update of molecular dynamics: smear the new links, apply D
        dict(name="hisq_smear_24x48", kind="smear", op="hisq", L="24x24x24x48", precision="double"),
        # the link gradients of the fermion force, back through the smearing
        # and through the clover leaves
        dict(name="hisq_pullback_24", kind="pullback", op="hisq", L="24x24x24x24", precision="double"),
        dict(name="clover_pullback_24", kind="pullback", op="clover", L="24x24x24x24", precision="double"),
        # five-dimensional domain-wall solve, int16 inner iterations
        dict(name="domainwall_cg_16x32_half", kind="cg", op="domainwall", L="16x16x16x32x12", precision="half"),
    ]


def _extents(rng, lo, hi, even, most):
    """Four extents spread over the logarithm of lo..hi, at most `most` sites."""
    while True:
        L = [math.exp(rng.uniform(math.log(lo), math.log(hi + 1))) for _ in range(4)]
        L[3] *= rng.choice((1, 1, 1.5, 2))
        L = [2 * max(1, int(v / 2)) if even else int(v) for v in L]
        if math.prod(L) <= most and min(L) >= lo:
            return L


def draw(rng):
    kind = rng.choice(("cg", "cg", "cg", "apply", "apply", "evenodd", "batched", "smear", "pullback"))
    case = dict(kind=kind)
    if kind == "batched":
        sizes = []
        for _ in range(rng.choice((1, 2, 3))):
            L = _extents(rng, 4, 20, True, 1 << 16)
            sizes.append("%s:%d" % ("x".join(map(str, L)), rng.randint(1, 8)))
        return dict(case, L=",".join(sizes), precision=rng.choice(("single", "half")))
    if kind == "cg":
        op = rng.choice(("wilson", "clover", "staggered", "hisq", "domainwall"))
        precision = rng.choice(("double", "single", "half"))
        most = {"wilson": 1 << 20, "clover": 600000, "staggered": 1 << 20, "hisq": 1 << 20, "domainwall": 60000}[op]
        L = _extents(rng, 4, 32, True, most)
    elif kind == "apply":
        op = rng.choice(("wilson", "clover", "staggered", "hisq", "domainwall"))
        precision = rng.choice(("double", "double", "single", "half"))
        L = _extents(rng, 4, 32, False, 1 << 17 if op == "domainwall" else 1 << 20)
    elif kind == "evenodd":
        op, precision = rng.choice(("wilson", "clover")), rng.choice(("double", "single", "half"))
        L = _extents(rng, 4, 32, True, 1 << 20)
    elif kind == "smear":
        op, precision = "hisq", "double"
        L = _extents(rng, 4, 32, False, 600000)
    else:
        op, precision = rng.choice(("hisq", "clover")), "double"
        L = _extents(rng, 4, 24, False, 300000)
    if op == "domainwall":
        L.append(rng.choice((4, 7, 8, 10, 12, 16)))
    return dict(case, op=op, L="x".join(map(str, L)), precision=precision)


def _size(case):
    return tuple(int(v) for v in case["L"].split("x"))


def _batch(case):
    """[(extents, right-hand sides)] of a batched case."""
    out = []
    for part in case["L"].split(","):
        L, n = part.split(":")
        out.append((tuple(int(v) for v in L.split("x")), int(n)))
    return out


# ---------------------------------------------------------------------------
# inputs, from the seed alone (plain torch)
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _gaussian(gen, *shape):
    return torch.complex(torch.randn(shape, generator=gen, device=_device(), dtype=torch.float64),
                         torch.randn(shape, generator=gen, device=_device(), dtype=torch.float64)) * math.sqrt(0.5)


def _mm(a, b):
    """3x3 products of fields with the matrix indices leading."""
    return torch.stack([torch.stack([a[i, 0] * b[0, j] + a[i, 1] * b[1, j] + a[i, 2] * b[2, j]
                                     for j in range(3)]) for i in range(3)])


def _dagger(a):
    return a.transpose(0, 1).conj()


def _su3(gen, sites, amplitude):
    """SU(3) matrices (3, 3, *sites) near exp(i amplitude H), H traceless
    Hermitian with unit-variance Gaussian entries."""
    h = _gaussian(gen, 3, 3, *sites)
    h = (h + _dagger(h)) * math.sqrt(0.5)
    trace = (h[0, 0] + h[1, 1] + h[2, 2]) / 3
    for i in range(3):
        h[i, i] -= trace
    h *= 1j * amplitude
    # exp(h) to second order, then reunitarised: rows 0 and 1 by
    # Gram-Schmidt (twice, to rounding), row 2 from them
    u = _mm(h, h) * 0.5 + h
    for i in range(3):
        u[i, i] += 1
    del h
    r0, r1 = u[0], u[1]
    for _ in range(2):
        r0 = r0 / torch.linalg.vector_norm(r0, dim=0)
        r1 = r1 - r0 * (r0.conj() * r1).sum(0)
        r1 = r1 / torch.linalg.vector_norm(r1, dim=0)
    r2 = torch.linalg.cross(r0, r1, dim=0).conj()
    return torch.stack([r0, r1, r2])


def _links(gen, L, amplitude):
    sites = tuple(L[:4])[::-1]
    return [_su3(gen, sites, amplitude) for _ in range(4)]


def _spinor(gen, L, spins):
    """Gaussian field (spins, 3, *sites), sites slowest coordinate first."""
    return _gaussian(gen, spins, 3, *tuple(L)[::-1])


def _link_fields(U, L, nw):
    out = []
    for u in U:
        f = lmb.LatticeMatrix(3, 3, 4, L[:4], nw=nw)
        f.core_view().copy_(u.permute(2, 3, 4, 5, 1, 0))
        lmb.mark_halo_dirty_(f)
        out.append(f)
    return out


def _spinor_field(psi, L, nw):
    dim = len(L)
    f = lmb.LatticeMatrix(3, psi.shape[0], dim, L, nw=nw, phases=PHASES + (1,) * (dim - 4))
    f.core_view().copy_(psi.permute(*range(2, 2 + dim), 0, 1))
    lmb.mark_halo_dirty_(f)
    return f


def _spins(op):
    return 1 if op in ("staggered", "hisq") else 4


def _halo(op):
    return 3 if op == "hisq" else 1


def _operator(op, U, L):
    p = OPS[op]
    if op == "wilson":
        return lmb.WilsonDiracOperator4D(U, p["kappa"])
    if op == "clover":
        return lmb.WilsonDiracCloverOperator4D(U, p["kappa"], CSW)
    if op == "staggered":
        return lmb.StaggeredDiracOperator4D(U, p["mass"])
    if op == "hisq":
        return lmb.HISQDiracCache4D(U, p["mass"], EPS_NAIK)
    n = L[4]
    return lmb.D5DW_GeneralizedDomainwallOperator5D(U, n, p["mass"], p["M"], [1.0] * n, [(p["b"] + p["c"]) / 2] * n,
                                                    [(p["b"] - p["c"]) / 2] * n)


def prepare(case, seed):
    """The gauge field, the source and the operator a user's program holds."""
    gen = _generator(seed)
    if case["kind"] == "batched":
        systems = []
        for L, n in _batch(case):
            D = lmb.WilsonDiracOperator4D(_link_fields(_links(gen, L, BATCH["amplitude"]), L, 1), BATCH["kappa"])
            pairs = []
            for _ in range(n):
                b = _spinor_field(_spinor(gen, L, 4), L, 1)
                pairs.append((b.similar(), b))
            systems.append((D, pairs))
        return dict(case=case, systems=systems)
    op, L = case["op"], _size(case)
    nw = _halo(op)
    U = _link_fields(_links(gen, L, OPS[op]["amplitude"]), L, nw)
    state = dict(case=case, U=U, b=_spinor_field(_spinor(gen, L, _spins(op)), L, nw))
    state["x"] = state["b"].similar()
    if case["kind"] == "pullback":
        state["chi"] = _spinor_field(_spinor(gen, L, _spins(op)), L, nw)
        state["dU"] = [u.similar() for u in U]
    if case["kind"] in ("cg", "apply"):
        state["temp"] = state["b"].similar()
    D = state["D"] = _operator(op, U, L)
    if case["kind"] == "apply" and op == "hisq":
        links = lmb.hisq_links_from_thin(U, EPS_NAIK)
        state["D"] = lmb.HISQDiracOperator4D(links, D.mass, EPS_NAIK)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batched":
        for _, pairs in state["systems"]:
            for x, _ in pairs:
                lmb.clear_matrix_(x)
        results, _ = lmb.cg_batched_(state["systems"], rtol=1e-10, precision=case["precision"])
        out = [x.core_view() for _, pairs in state["systems"] for x, _ in pairs]
        return dict(x=out, converged=all(r.converged for r in results))
    D, x, b = state["D"], state["x"], state["b"]
    if kind == "cg":
        lmb.clear_matrix_(x)
        result = lmb.cg_(x, lmb.DdagDOp(D, state["temp"]), b, rtol=1e-10, precision=case["precision"])
        return dict(x=x.core_view(), converged=result.converged)
    if kind == "evenodd":
        result = lmb.solve_evenodd_(x, D, b, rtol=1e-10, precision=case["precision"])
        return dict(x=x.core_view(), converged=result.converged)
    if kind == "apply":
        if case["op"] == "hisq":
            lmb.mul_(x, D, b, precision=case["precision"])
            lmb.set_halo_(x)
            return x.A
        temp = state["temp"]
        lmb.mul_(temp, D, b, precision=case["precision"])
        lmb.mul_(x, lmb.adjoint(D), temp, precision=case["precision"])
        return temp.core_view(), x.core_view()
    if kind == "smear":
        for u in state["U"]:
            lmb.mark_halo_dirty_(u)
        lmb.mul_cached_hisq_(x, D, *state["U"], b)
        return x.core_view()
    dU = state["dU"]
    for d in dU:
        lmb.clear_matrix_(d)
    if case["op"] == "hisq":
        lmb.hisq_link_pullback_(dU, D, state["U"], state["chi"], b)
    else:
        lmb.wilson_clover_link_pullback_(dU, D, state["U"], state["chi"], b)
    return [d.core_view() for d in dU]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _per_site(op, precision, sites5=1):
    """Bytes and flops of one application per (4D or 5D) site: links and site
    terms once, the spinor read and written once; and of a spinor."""
    real = {"double": 8, "single": 4, "half": 2}[precision]
    spinor = 24 if _spins(op) == 4 else 6
    links = {"wilson": 48, "clover": 48 + 72, "staggered": 48, "hisq": 144, "domainwall": 48 / sites5}[op]
    flops = {"wilson": 1368, "clover": 1872, "staggered": 570, "hisq": 1146, "domainwall": 1464}[op]
    norm = 4 if precision == "half" else 0
    return real * links + 2 * (real * spinor + norm), flops, real * spinor + norm, spinor


def _cg_work(op, precision, V, iterations, sites5=1):
    apply, flops, vector, reals = _per_site(op, precision, sites5)
    low = reals * (8 if precision == "double" else 4)  # the accumulated solution
    # two applications, then x += a p and r -= a Ap (p, x, r read, x, r
    # written beside the application's own) and p = r + b p
    bytes_ = 2 * apply + 2 * vector + 2 * low + 3 * vector
    return iterations * V * bytes_, iterations * V * (2 * flops + 14 * reals)


def work(case):
    kind = case["kind"]
    if kind == "batched":
        done = [0, 0]
        for L, n in _batch(case):
            b, f = _cg_work("wilson", case["precision"], math.prod(L), BATCH["iterations"])
            links = BATCH["iterations"] * math.prod(L) * 2 * 48 * {"single": 4, "half": 2}[case["precision"]]
            done[0] += n * (b - links) + links  # the links once for all right-hand sides
            done[1] += n * f
        return dict(bytes=done[0], flops=done[1])
    op, L = case["op"], _size(case)
    V = math.prod(L)
    L5 = L[4] if len(L) == 5 else 1
    if kind == "cg":
        b, f = _cg_work(op, case["precision"], V, OPS[op]["iterations"], L5)
        return dict(bytes=b, flops=f)
    if kind == "evenodd":
        # per iteration four half-lattice hops: the links once each, A and
        # A^-1 once per pair, half the sites' vectors
        b, f = _cg_work(op, case["precision"], V, EVENODD_ITERATIONS)
        real = {"double": 8, "single": 4, "half": 2}[case["precision"]]
        return dict(bytes=b / 2 + EVENODD_ITERATIONS * V * real * 48, flops=f)
    if kind == "apply":
        reals = 24 if _spins(op) == 4 else 6
        links = {"wilson": 48, "clover": 120, "staggered": 48, "hisq": 144, "domainwall": 48 / L5}[op]
        passes = 1 if op == "hisq" else 2
        real = {"double": 8, "single": 4, "half": 2}[case["precision"]]
        out = reals * 16 * (math.prod(v + 6 for v in L) - V) / 2 if op == "hisq" else 0
        return dict(bytes=passes * V * (real * links + 16 * reals) + out, flops=passes * V * _per_site(op, "double", L5)[1])
    if kind == "smear":
        # thin links in, fat and long links out, D on them; two Fat7 levels
        # of about 4 x 12 transports of 4 products, projections, Naik
        return dict(bytes=V * 8 * (72 + 2 * 144 + 12), flops=V * (2 * 4 * 12 * 4 * 198 + 4 * 1500 + 4 * 2 * 198 + 1146))
    if op == "hisq":
        return dict(bytes=V * 8 * (3 * 72 + 12), flops=3 * V * (2 * 4 * 12 * 4 * 198 + 4 * 1500))
    # hopping outer products, six cotangents, four leaves of each plane
    return dict(bytes=V * 8 * (3 * 72 + 48), flops=V * (8 * 400 + 6 * 600 + 6 * 16 * 3 * 198))


def tolerance(case):
    """About four to six times the largest distance from exact() that the
    kinds' operators and precisions show."""
    kind, precision = case["kind"], case["precision"]
    if kind in ("cg", "evenodd", "batched"):
        # the solves stop at a relative residual of 1e-10; the solution's
        # error is that times a factor of up to 30 (domain wall)
        return dict(rel=2e-8, max=2e-7)
    if kind == "apply":
        return {"double": dict(rel=5e-15, max=1e-13), "single": dict(rel=4e-7, max=3e-6),
                "half": dict(rel=4e-4, max=2e-3)}[precision]
    return dict(rel=6e-15, max=2e-13)


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
# fields: links (3, 3, *sites), spinors (spin, colour, *sites), sites ordered
# (t, z, y, x), for domain-wall fields (s, t, z, y, x); direction mu is the
# mu-th axis from the end

# gamma_mu psi: row s of gamma_mu has the one entry VALUE at column COLUMN
_GAMMA = (((3, -1j), (2, -1j), (1, 1j), (0, 1j)), ((3, -1), (2, 1), (1, 1), (0, -1)),
          ((2, -1j), (3, 1j), (0, 1j), (1, -1j)), ((2, -1), (3, -1), (0, -1), (1, -1)))
_PLANES = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))


def _gamma(mu, psi):
    return torch.stack([psi[c] * v for c, v in _GAMMA[mu]])


def _gamma5(psi):
    return _gamma(0, _gamma(1, _gamma(2, _gamma(3, psi))))


def _shift(field, mu, by):
    """field(x + by mu), periodic."""
    return torch.roll(field, -by, -1 - mu)


def _hop(field, mu, by):
    """field(x + by mu) with the boundary phases of the fermions."""
    out = _shift(field, mu, by)
    if PHASES[mu] != 1:
        n, axis = out.shape[-1 - mu], out.ndim - 1 - mu
        wrapped = out.narrow(axis, n - by if by > 0 else 0, abs(by))
        wrapped *= PHASES[mu] if by > 0 else 1 / PHASES[mu]
    return out


def _mv(u, psi):
    return torch.stack([u[i, 0] * psi[:, 0] + u[i, 1] * psi[:, 1] + u[i, 2] * psi[:, 2] for i in range(3)], 1)


def _hopping(U, psi, dagger):
    """sum_mu (1 -+ gamma) U psi(x + mu) + (1 +- gamma) U^+ psi(x - mu)."""
    sign = -1 if dagger else 1
    total = 0
    for mu in range(4):
        f = _mv(U[mu], _hop(psi, mu, 1))
        b = _hop(_mv(_dagger(U[mu]), psi), mu, -1)
        total = total + f + b - sign * _gamma(mu, f - b)
    return total


def _field_strength(U):
    fields = []
    for mu, nu in _PLANES:
        m, n = U[mu], U[nu]
        a = _mm(m, _shift(n, mu, 1))  # U_mu(x) U_nu(x + mu)
        b = _mm(n, _shift(m, nu, 1))  # U_nu(x) U_mu(x + nu)
        side = _mm(_shift(_dagger(m), mu, -1), _shift(n, mu, -1))  # U_mu(x - mu)^+ U_nu(x - mu)
        end = _shift(_shift(m, mu, -1), nu, 1)  # U_mu(x + nu - mu)
        q = _mm(a, _dagger(b)) + _mm(_mm(n, _dagger(end)), _dagger(side))
        bb, aa = _shift(_shift(b, mu, -1), nu, -1), _shift(_shift(a, mu, -1), nu, -1)
        q = q + _mm(_dagger(bb), aa)
        down = _mm(_shift(_dagger(n), nu, -1), _shift(m, nu, -1))  # U_nu(x - nu)^+ U_mu(x - nu)
        corner = _shift(_shift(n, nu, -1), mu, 1)  # U_nu(x + mu - nu)
        q = q + _mm(_mm(down, corner), _dagger(m))
        fields.append((q - _dagger(q)) / 8)
    return fields


def _wilson(U, F, kappa, psi, dagger=False):
    out = psi - kappa * _hopping(U, psi, dagger)
    if F is not None:  # Hermitian: the same in D^+
        for (mu, nu), f in zip(_PLANES, F):
            out = out - kappa * CSW * _mv(f, _gamma(mu, _gamma(nu, psi)))
    return out


def _eta(mu, sites, device):
    """(-1)^(x_0 + .. + x_(mu-1)) over (t, z, y, x)."""
    total = torch.zeros(sites, device=device, dtype=torch.float64)
    for nu in range(mu):
        n = sites[3 - nu]
        total = total + torch.arange(n, device=device, dtype=torch.float64).reshape((n,) + (1,) * nu)
    return 1 - 2 * (total % 2)


def _staggered(terms, mass, psi, dagger=False):
    """m psi + sum eta c [W psi(x + d mu) - W^+ psi(x - d mu)] over the terms
    (links W, coefficient c, distance d)."""
    out = mass * psi
    for mu in range(4):
        eta = _eta(mu, psi.shape[2:], psi.device) * (-1 if dagger else 1)
        for W, c, d in terms:
            hop = _mv(W[mu], _hop(psi, mu, d)) - _hop(_mv(_dagger(W[mu]), psi), mu, -d)
            out = out + (c * eta) * hop
    return out


def _chiral(psi, mass, adjoint=False):
    """Spins 1, 2 from s - 1 and 3, 4 from s + 1 (adjoint: the reverse), with
    -mass across the walls; s is the first site axis."""
    up, down = torch.roll(psi[:2], 1 if not adjoint else -1, 2), torch.roll(psi[2:], -1 if not adjoint else 1, 2)
    first, last = (0, -1) if not adjoint else (-1, 0)
    up[:, :, first] *= -mass
    down[:, :, last] *= -mass
    return torch.cat([up, down])


def _domainwall(U, p, psi, dagger=False):
    b, c = (p["b"] + p["c"]) / 2, (p["b"] - p["c"]) / 2

    def dw(v):
        return (4 + p["M"]) * v - 0.5 * _hopping(U, v, dagger)

    if not dagger:
        f = _chiral(psi, p["mass"])
        return psi - f + dw(b * psi + c * f)
    q = dw(psi)
    return psi - _chiral(psi, p["mass"], True) + b * q + _chiral(c * q, p["mass"], True)


def _transport(M, U, mu, nu, steps=3):
    """U_nu(x) M(x + nu) U_nu(x + mu)^+ (bit 0 of steps) and
    U_nu(x - nu)^+ M(x - nu) U_nu(x - nu + mu) (bit 1)."""
    u = U[nu]
    ahead = _shift(u, mu, 1)
    out = 0
    if steps & 1:
        out = out + _mm(_mm(u, _shift(M, nu, 1)), _dagger(ahead))
    if steps & 2:
        out = out + _shift(_mm(_mm(_dagger(u), M), ahead), nu, -1)
    return out


def _fat7_mu(mu, c1, c3, c5, c7, lepage, *U):
    axes = [d for d in range(4) if d != mu]
    three = {a: _transport(U[mu], U, mu, a) for a in axes}
    out = c1 * U[mu]
    for a in axes:
        b, c = [d for d in axes if d != a]
        five = _transport(three[c], U, mu, b) + _transport(three[b], U, mu, c)
        out = out + c3 * three[a] + c5 * five + c7 * _transport(five, U, mu, a)
        if lepage:
            for s in (1, 2):
                out = out + lepage * _transport(_transport(U[mu], U, mu, a, s), U, mu, a, s)
    return out


def _fat7(U, coefficients):
    if not U[0].requires_grad:
        return [_fat7_mu(mu, *coefficients, *U) for mu in range(4)]
    from torch.utils.checkpoint import checkpoint
    return [checkpoint(_fat7_mu, mu, *coefficients, *U, use_reentrant=False) for mu in range(4)]


def _unitary(V):
    """The unitary factor of V's polar decomposition: X <- (X + X^-+) / 2."""
    for _ in range(9):
        cof = torch.stack([torch.linalg.cross(V[1], V[2], dim=0), torch.linalg.cross(V[2], V[0], dim=0),
                           torch.linalg.cross(V[0], V[1], dim=0)])
        det = (V[0] * cof[0]).sum(0)
        V = 0.5 * (V + (cof / det).conj())
    return V


def _smeared(U):
    first = _fat7(U, (1 / 8, 1 / 16, 1 / 64, 1 / 384, 0.0))
    W = [_unitary(v) for v in first]
    fat = _fat7(W, (1 + EPS_NAIK / 8, 1 / 16, 1 / 64, 1 / 384, -1 / 8))
    long = [_mm(_mm(W[mu], _shift(W[mu], mu, 1)), _shift(W[mu], mu, 2)) for mu in range(4)]
    return fat, long


def _dirac(op, U):
    """D(psi, dagger) of the operator."""
    p = OPS[op]
    if op == "wilson":
        return lambda v, dagger=False: _wilson(U, None, p["kappa"], v, dagger)
    if op == "clover":
        F = _field_strength(U)
        return lambda v, dagger=False: _wilson(U, F, p["kappa"], v, dagger)
    if op == "staggered":
        return lambda v, dagger=False: _staggered([(U, 0.5, 1)], p["mass"], v, dagger)
    if op == "hisq":
        fat, long = _smeared(U)
        terms = [(fat, 0.5, 1), (long, -(1 + EPS_NAIK) / 48, 3)]
        return lambda v, dagger=False: _staggered(terms, p["mass"], v, dagger)
    return lambda v, dagger=False: _domainwall(U, p, v, dagger)


def _solve(D, b, least=1e-13, most=4000):
    """(D^+ D)^-1 b by conjugate gradient."""
    def dot(u, v):
        return torch.vdot(u.reshape(-1), v.reshape(-1)).real
    x, r, p = torch.zeros_like(b), b, b
    rr = dot(r, r)
    stop = least * least * rr
    for k in range(most):
        q = D(D(p), True)
        a = rr / dot(p, q)
        x, r = x + a * p, r - a * q
        new = dot(r, r)
        if k % 10 == 9 and bool(new <= stop):
            break
        p, rr = r + (new / rr) * p, new
    return x


def _out(psi, L):
    """A spinor in the order of a field's storage."""
    n = len(L)
    return psi.permute(*range(2, 2 + n), 0, 1)


def _padded(psi, nw):
    """The storage of a 4D field with its halo filled."""
    for mu in range(4):
        axis = psi.ndim - 1 - mu
        n = psi.shape[axis]
        psi = torch.cat([psi.narrow(axis, n - nw, nw) / PHASES[mu], psi, psi.narrow(axis, 0, nw) * PHASES[mu]], axis)
    return psi


def exact(case, seed):
    gen = _generator(seed)
    if case["kind"] == "batched":
        out = []
        for L, n in _batch(case):
            U = _links(gen, L, BATCH["amplitude"])
            for _ in range(n):
                out.append((U, _spinor(gen, L, 4), L))
        return dict(x=[_out(_solve(lambda v, dagger=False, U=U: _wilson(U, None, BATCH["kappa"], v, dagger), b), L)
                       for U, b, L in out], converged=None)
    op, L, kind = case["op"], _size(case), case["kind"]
    U = _links(gen, L, OPS[op]["amplitude"])
    b = _spinor(gen, L, _spins(op))
    V = math.prod(L)
    if kind in ("cg", "evenodd"):
        # the plain solve is some 20 times slower than the framework's
        if V * OPS[op]["iterations"] * _spins(op) > 1.3e9:
            return None
        D = _dirac(op, U)
        # D x = b by D^+ D x = D^+ b
        return dict(x=_out(_solve(D, D(b, True) if kind == "evenodd" else b), L), converged=None)
    if kind == "apply":
        D = _dirac(op, U)
        first = D(b)
        if op == "hisq":
            return _padded(first, _halo(op)).permute(2, 3, 4, 5, 0, 1)
        return _out(first, L), _out(D(first, True), L)
    if kind == "smear":
        return _out(_dirac(op, U)(b), L)
    chi = _spinor(gen, L, _spins(op))
    U = [u.requires_grad_() for u in U]
    value = (chi.conj() * _dirac(op, U)(b)).sum().real
    return [g.permute(2, 3, 4, 5, 1, 0) for g in torch.autograd.grad(value, U)]
