"""GPU: the kernels a size or storage rule selects, at the edges of their
ranges: Fat7 on ragged site blocks and on both sides of the one-launch limit,
the clover link gradient on odd extents, domain-wall slice pairs, even/odd
pairs, the one-launch solver of small lattices and the direct store of FP64
applications.

Bars: FP64 results against the oracle as the parity tests' (1e-13 relative
norm), FP32 5e-6, int16 2e-3 (one rounding of each operand per application);
finite differences 1e-8 (step 1e-5: 1e-10 truncation, 1e-11 rounding)."""
import numpy as np
import pytest

import refdata as rd

pytestmark = pytest.mark.gpu
PHASES = (1, 1, 1, -1)
TWISTED = tuple(np.exp(1j * a) for a in (0.13, -0.21, 0.34, np.pi - 0.17))


@pytest.fixture(scope="module")
def lmb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lmb200
    lmb200.load()
    return lmb200


def _links(lmb, U, nw):
    return [lmb.LatticeMatrix.from_array(u, nw=nw) for u in U]


def _directions(L, seed):
    rng = np.random.default_rng(seed)
    return [np.asfortranarray(rng.normal(size=(3, 3) + L) + 1j * rng.normal(size=(3, 3) + L)) for _ in range(4)]


# blocks of sites whose last ones are ragged in every extent; an extent below
# the block's; one site more than a whole block
@pytest.mark.parametrize("L", [(9, 5, 3, 7), (3, 4, 5, 4), (17, 3, 5, 3)])
def test_fat7_levels_on_ragged_blocks(lmb, orc, L):
    U = orc.random_su3_links(L, 0.25, 31)
    fat, long = orc.hisq_links_from_thin(U, -0.083)
    links = lmb.hisq_links_from_thin(_links(lmb, U, 3), -0.083)
    for got, want in zip(links.fat_links + links.long_links, fat + long):
        assert rd.rel_err(got.gather_matrix(), want) <= 1e-12


# 4096 sites: four directions per launch; 17 x 16^3 = 69632 > 65536: one
@pytest.mark.parametrize("L", [(9, 5, 3, 7), (8, 8, 8, 8), (17, 16, 16, 16)])
def test_hisq_link_gradient_matches_finite_differences(lmb, orc, L):
    eps, h = -0.083, 1e-5
    U = orc.random_su3_links(L, 0.2, 41)
    psi = lmb.LatticeMatrix.from_array(orc.gaussian_field(L, 3, 1, 42), nw=3, phases=PHASES)
    chi = lmb.LatticeMatrix.from_array(orc.gaussian_field(L, 3, 1, 43), nw=3, phases=PHASES)
    Ud = _links(lmb, U, 3)
    cache = lmb.HISQDiracCache4D(Ud, 0.07, eps)
    dU = [u.similar() for u in Ud]
    lmb.hisq_link_pullback_(dU, cache, Ud, chi, psi)
    V = _directions(L, 44)
    out = psi.similar()

    def loss(sign):
        links = _links(lmb, [np.asfortranarray(u + sign * h * v) for u, v in zip(U, V)], 3)
        lmb.mul_cached_hisq_(out, cache, *links, psi)
        return lmb.dot(chi, out).real
    fd = (loss(+1) - loss(-1)) / (2 * h)
    an = sum(np.vdot(d.gather_matrix(), v).real for d, v in zip(dU, V))
    assert abs(an - fd) <= 1e-8 * max(abs(fd), np.sqrt(np.prod(L)))


@pytest.mark.parametrize("L", [(9, 5, 3, 7), (4, 4, 6, 5)])
def test_clover_link_gradient_on_odd_extents(lmb, orc, L):
    kappa, csw, h = 0.13, 1.2, 1e-5
    U = orc.random_su3_links(L, 0.2, 51)
    psi, chi = orc.gaussian_field(L, 3, 4, 52), orc.gaussian_field(L, 3, 4, 53)
    Ud = _links(lmb, U, 1)
    D = lmb.WilsonDiracCloverOperator4D(Ud, kappa, csw)
    dU = [u.similar() for u in Ud]
    lmb.wilson_clover_link_pullback_(dU, D, Ud, lmb.LatticeMatrix.from_array(chi, nw=1, phases=TWISTED),
                                     lmb.LatticeMatrix.from_array(psi, nw=1, phases=TWISTED))
    V = _directions(L, 54)
    loss = [np.vdot(chi, orc.wilson_clover([np.asfortranarray(u + s * h * v) for u, v in zip(U, V)], psi, kappa,
                                           csw, TWISTED)).real for s in (+1, -1)]
    fd = (loss[0] - loss[1]) / (2 * h)
    an = sum(np.vdot(d.gather_matrix(), v).real for d, v in zip(dU, V))
    assert abs(an - fd) <= 1e-8 * max(abs(fd), np.sqrt(np.prod(L)))


# extents of 1 and 2, where a site is its own neighbour or the same one on both
# sides (the HISQ fields without a halo: it may not be wider than an extent)
@pytest.mark.parametrize("L", [(2, 2, 4, 2), (1, 2, 3, 2), (4, 1, 1, 2)])
def test_link_gradients_on_extents_of_one_and_two(lmb, orc, L):
    eps, h = -0.083, 1e-5
    U, V = orc.random_su3_links(L, 0.2, 46), _directions(L, 47)
    fat, long = orc.hisq_links_from_thin(U, eps)
    links = lmb.hisq_links_from_thin(_links(lmb, U, 0), eps)
    for got, want in zip(links.fat_links + links.long_links, fat + long):
        assert rd.rel_err(got.gather_matrix(), want) <= 1e-12
    for spins in (1, 4):
        psi, chi = orc.gaussian_field(L, 3, spins, 48), orc.gaussian_field(L, 3, spins, 49)
        nw = 0 if spins == 1 else 1
        pd, cd = (lmb.LatticeMatrix.from_array(f, nw=nw, phases=PHASES) for f in (psi, chi))
        Ud = _links(lmb, U, nw)
        dU = [u.similar() for u in Ud]
        if spins == 1:
            lmb.hisq_link_pullback_(dU, lmb.HISQDiracCache4D(Ud, 0.07, eps), Ud, cd, pd)
        else:
            lmb.wilson_clover_link_pullback_(dU, lmb.WilsonDiracCloverOperator4D(Ud, 0.13, 1.2), Ud, cd, pd)

        def loss(sign):
            W = [np.asfortranarray(u + sign * h * v) for u, v in zip(U, V)]
            if spins == 1:
                return np.vdot(chi, orc.hisq(*orc.hisq_links_from_thin(W, eps), psi, 0.07, eps, PHASES)).real
            return np.vdot(chi, orc.wilson_clover(W, psi, 0.13, 1.2, PHASES)).real
        fd = (loss(+1) - loss(-1)) / (2 * h)
        an = sum(np.vdot(d.gather_matrix(), v).real for d, v in zip(dU, V))
        assert abs(an - fd) <= 1e-8 * max(abs(fd), np.sqrt(np.prod(L)))


# lattices of at least 222 (int16) and 296 (FP32, and not between 444 and 592)
# blocks of 128 pairs, which take them on 148 SMs.  L5 = 2: a pair is its own
# neighbour on both sides; 128: the longest one-pass fifth dimension (FP32: 300
# blocks of it); 6: blocks of the adjoint that leave threads idle; and links that
# are not SU(3), which keep 18 reals
@pytest.mark.parametrize("L,L5,scale", [((15, 16, 14, 13), 2, 1.0), ((11, 12, 10, 11), 6, 1.0), ((6, 5, 6, 5), 128, 1.0),
                                        ((6, 5, 4, 5), 128, 1.0), ((11, 12, 10, 11), 6, 1.01)])
@pytest.mark.parametrize("precision,bar", [("single", 5e-6), ("half", 2e-3)])
def test_domainwall_slice_pairs(lmb, orc, L, L5, scale, precision, bar):
    rng = np.random.default_rng(61)
    U = [np.asfortranarray(scale * u) for u in orc.random_su3_links(L, 0.3, 62)]
    flat = orc.gaussian_field(L[:3] + (L[3] * L5,), 3, 4, 63)
    psi = np.asfortranarray(flat.reshape((3, 4) + L + (L5,), order="F"))
    a, b, c = (list(lo + w * rng.random(L5)) for lo, w in ((0.8, 0.4), (0.9, 0.6), (-0.3, 0.6)))
    D = lmb.D5DW_GeneralizedDomainwallOperator5D(_links(lmb, U, 1), L5, 0.07, -1.8, a, b, c)
    pd = lmb.LatticeMatrix.from_array(psi, 5, nw=1, phases=TWISTED + (1,))
    out = pd.similar()
    for dagger in (False, True):
        lmb.mul_(out, lmb.adjoint(D) if dagger else D, pd, precision=precision)
        ref = orc.domainwall(U, psi, 0.07, -1.8, a, b, c, TWISTED, dagger=dagger)
        assert rd.rel_err(out.gather_matrix(), ref) <= bar


# from 222 blocks of 128 pairs on (113664 sites on 148 SMs) rows of 2 (one pair),
# 4 and 12 checkerboard sites take pairs; a row of 3 or 9 stays at one site per
# thread, and so do the small ones
# An int16 solve on pairs takes about the iterations of one on single sites (a
# worse operator would show there, not in the residual that FP64 corrects).
@pytest.mark.parametrize("L,scale", [((4, 32, 30, 32), 1.0), ((8, 30, 20, 24), 1.0), ((24, 18, 16, 18), 1.0),
                                     ((18, 18, 20, 18), 1.0), ((6, 4, 2, 4), 1.0), ((8, 30, 20, 24), 1.01)])
@pytest.mark.parametrize("csw", [0.0, 1.0])
def test_evenodd_pairs(lmb, orc, monkeypatch, L, scale, csw):
    kappa = 0.125 / scale
    U, b = [np.asfortranarray(scale * u) for u in orc.random_su3_links(L, 0.3, 71)], orc.gaussian_field(L, 3, 4, 72)
    Ud = _links(lmb, U, 1)
    bd = lmb.LatticeMatrix.from_array(b, nw=1, phases=TWISTED)
    iterations = []
    for precision, adjacent in (("half", "1"), ("half", "0"), ("single", "1")):
        monkeypatch.setenv("LMB_ADJ_SITES", adjacent)
        D = lmb.WilsonDiracCloverOperator4D(Ud, kappa, csw) if csw else lmb.WilsonDiracOperator4D(Ud, kappa)
        x = bd.similar()
        res = lmb.solve_evenodd_(x, D, bd, rtol=1e-10, precision=precision)
        assert res.converged
        iterations.append(res.iterations)
        xs = np.asfortranarray(x.gather_matrix())
        Dx = orc.wilson_clover(U, xs, kappa, csw, TWISTED) if csw else orc.wilson(U, xs, kappa, TWISTED)
        assert rd.rel_err(Dx, b) <= 1.05e-10
    assert abs(iterations[0] - iterations[1]) <= max(3, iterations[1] // 20)


def _solver(lmb, orc, op, L, scale, precision, phases):
    """A solve of `op` on a new context: (result, solution, relative residual by
    the oracle's operator)."""
    U = [np.asfortranarray(scale * u) for u in orc.random_su3_links(L, 0.25, 81)]
    nw, spins = (3 if op == "hisq" else 1), (1 if op in ("staggered", "hisq") else 4)
    Ud = _links(lmb, U, nw)
    if op == "domainwall":
        flat = orc.gaussian_field(L[:3] + (L[3] * 5,), 3, 4, 82)
        b0 = np.asfortranarray(flat.reshape((3, 4) + L + (5,), order="F"))
        b = lmb.LatticeMatrix.from_array(b0, 5, nw=1, phases=phases + (1,))
        D = lmb.D5DW_MobiusDomainwallOperator5D(Ud, 5, 0.2, -1.4, 1.5, 0.5)
    else:
        b0 = orc.gaussian_field(L, 3, spins, 82)
        b = lmb.LatticeMatrix.from_array(b0, nw=nw, phases=phases)
        D = {"wilson": lambda: lmb.WilsonDiracOperator4D(Ud, 0.12),
             "clover": lambda: lmb.WilsonDiracCloverOperator4D(Ud, 0.12, 1.0),
             "evenodd": lambda: lmb.WilsonDiracOperator4D(Ud, 0.12),
             "evenodd-clover": lambda: lmb.WilsonDiracCloverOperator4D(Ud, 0.12, 1.0),
             "staggered": lambda: lmb.StaggeredDiracOperator4D(Ud, 0.2),
             "hisq": lambda: lmb.HISQDiracCache4D(Ud, 0.2, -0.083)}[op]()
    x = b.similar()
    if op.startswith("evenodd"):
        res = lmb.solve_evenodd_(x, D, b, rtol=1e-9, maxiter=400, precision=precision)
    else:
        res = lmb.cg_(x, lmb.DdagDOp(D, b.similar()), b, rtol=1e-9, maxiter=400, precision=precision)
    xs = np.asfortranarray(x.gather_matrix())

    def apply(v, dagger):
        if op == "domainwall":
            a, bb, cc = [1.0] * 5, [1.0] * 5, [0.5] * 5  # Mobius b = 1.5, c = 0.5: (b + c) / 2 and (b - c) / 2
            return orc.domainwall(U, v, 0.2, -1.4, a, bb, cc, phases, dagger=dagger)
        if op in ("wilson", "evenodd"):
            return orc.wilson(U, v, 0.12, phases, dagger=dagger)
        if op in ("clover", "evenodd-clover"):
            return orc.wilson_clover(U, v, 0.12, 1.0, phases, dagger=dagger)
        if op == "staggered":
            return orc.staggered(U, v, 0.2, phases, dagger=dagger)
        return orc.hisq(*orc.hisq_links_from_thin(U, -0.083), v, 0.2, -0.083, phases, dagger=dagger)
    Ax = apply(xs, False)
    if not op.startswith("evenodd"):
        Ax = apply(np.asfortranarray(Ax), True)
    return res, xs, rd.rel_err(Ax, b0)


# the one-launch solver against one launch per stage (LMB_PERSISTENT=0): a
# lattice below one tile of 32 sites per block, ragged last tiles, links that
# are not SU(3) (18 reals).  The launches tell which of the two ran; both solve
# the oracle's equation.
@pytest.mark.parametrize("op", ["wilson", "clover", "staggered", "hisq", "evenodd", "evenodd-clover", "domainwall"])
@pytest.mark.parametrize("L,scale", [((3, 3, 3, 4), 1.0), ((5, 3, 7, 6), 1.0), ((4, 6, 4, 8), 1.01)])
@pytest.mark.parametrize("precision", ["double", "single", "half"])
def test_small_lattice_solver(lmb, orc, monkeypatch, op, L, scale, precision):
    if op in ("staggered", "hisq") or op.startswith("evenodd"):  # even extents: signs, parity
        L = {(3, 3, 3, 4): (4, 4, 4, 4), (5, 3, 7, 6): (6, 6, 6, 6)}.get(L, L)
    out = []
    for stages in ("1", "0"):
        monkeypatch.setenv("LMB_PERSISTENT", stages)
        out.append(_solver(lmb, orc, op, L, scale, precision, TWISTED))
    (ra, xa, ea), (rb, xb, eb) = out
    assert ra.reason == rb.reason
    assert abs(ra.iterations - rb.iterations) <= (1 if precision == "double" else max(3, rb.iterations // 20))
    assert ra.kernel_launches < 3 * ra.iterations <= rb.kernel_launches + 9
    assert ra.converged
    assert max(ea, eb) <= 1.05e-9
    assert rd.rel_err(xa, xb) <= 1e-6  # both within 1e-9 of the same equation


def test_small_lattice_solver_stops_as_the_staged_one(lmb, orc, monkeypatch):
    L = (4, 4, 4, 4)
    U = orc.random_su3_links(L, 0.3, 91)
    b = lmb.LatticeMatrix.from_array(orc.gaussian_field(L, 3, 4, 92), nw=1, phases=PHASES)
    for precision in ("double", "half"):
        for maxiter in (0, 1, 7):
            got = []
            for stages in ("1", "0"):
                monkeypatch.setenv("LMB_PERSISTENT", stages)
                D = lmb.WilsonDiracOperator4D(_links(lmb, U, 1), 0.12)
                res = lmb.cg_(b.similar(), lmb.DdagDOp(D, b.similar()), b, maxiter=maxiter, precision=precision)
                got.append((res.reason, res.iterations))
                assert res.iterations <= maxiter
            assert got[0] == got[1] == ("maximum_iterations", maxiter)


# FP64: the one launch up to 4 tiles per resident block, 37888 sites on 148 SMs
@pytest.mark.parametrize("L", [(16, 16, 12, 12), (16, 16, 12, 14)])
def test_solvers_on_both_sides_of_the_limit(lmb, orc, L):
    U = lmb.random_su3_links(L, 0.25, 95)
    b = lmb.gaussian_fermion(L, 3, 4, 96, phases=PHASES)
    D = lmb.WilsonDiracOperator4D(U, 0.12)
    for precision in ("double", "half"):
        x = b.similar()
        res = lmb.cg_(x, lmb.DdagDOp(D, b.similar()), b, rtol=1e-10, precision=precision)
        t, y = b.similar(), b.similar()
        lmb.DdagDOp(D, t).mul_(y, x)
        r = (y.core_view() - b.core_view()).norm() / b.core_view().norm()
        assert res.converged and float(r) <= 1.1e-10


@pytest.mark.parametrize("L,nw,phases", [((3, 5, 4, 7), 1, TWISTED), ((8, 4, 4, 2), 0, PHASES), ((1, 1, 2, 3), 1, PHASES)])
@pytest.mark.parametrize("scale", [1.0, 1.01])
def test_fp64_wilson_small_and_odd(lmb, orc, L, nw, phases, scale):
    """Reconstructed (scale 1) and 18-real links, extents down to 1."""
    U = [np.asfortranarray(scale * u) for u in orc.random_su3_links(L, 0.3, 101)]
    psi = orc.gaussian_field(L, 3, 4, 102)
    Ud, pd = _links(lmb, U, nw), lmb.LatticeMatrix.from_array(psi, nw=nw, phases=phases)
    out = pd.similar()
    for csw in (0.0, 1.1):
        D = lmb.WilsonDiracCloverOperator4D(Ud, 0.13, csw) if csw else lmb.WilsonDiracOperator4D(Ud, 0.13)
        for dagger in (False, True):
            lmb.mul_(out, lmb.adjoint(D) if dagger else D, pd)
            ref = orc.wilson_clover(U, psi, 0.13, csw, phases, dagger=dagger) if csw else \
                orc.wilson(U, psi, 0.13, phases, dagger=dagger)
            assert rd.rel_err(out.gather_matrix(), ref) <= 1e-13


def test_direct_store_leaves_the_halo_and_takes_any_alignment(lmb, orc):
    """An output whose storage starts 16 bytes off a 32-byte boundary takes
    128-bit stores; the ghosts stay as they were."""
    import torch
    L, nw = (4, 3, 5, 2), 1
    U, psi = orc.random_su3_links(L, 0.3, 111), orc.gaussian_field(L, 3, 4, 112)
    pd = lmb.LatticeMatrix.from_array(psi, nw=nw, phases=PHASES)
    out = pd.similar()
    shape = out.A.shape
    store = torch.zeros(out.A.numel() + 1, dtype=out.A.dtype, device="cuda")
    out.A = store[1:].view(shape)
    out.A.fill_(7.0)
    assert out.data_ptr() % 32 == 16
    lmb.mul_(out, lmb.WilsonDiracOperator4D(_links(lmb, U, nw), 0.13), pd)
    assert rd.rel_err(out.gather_matrix(), orc.wilson(U, psi, 0.13, PHASES)) <= 1e-13
    ghosts = out.A.clone()
    ghosts[1:-1, 1:-1, 1:-1, 1:-1] = 7.0
    assert bool((ghosts == 7.0).all()) and complex(store[0]) == 0


def _cg_iterates(apply, b, n):
    x, r = np.zeros_like(b), b.copy()
    p, rr = r.copy(), np.vdot(r, r).real
    for _ in range(n):
        q = apply(np.asfortranarray(p))
        alpha = rr / np.vdot(p, q).real
        x, r = x + alpha * p, r - alpha * q
        beta, rr = np.vdot(r, r).real / rr, np.vdot(r, r).real
        p = r + beta * p
        yield x


# x after n iterations of the staged solver, whose updates of x wait for each
# other: every number of them that can still wait at the end, and (mixed) a
# reliable update between them.  Bars: the rounding of the stored fields in each
# iteration (2^-53, 2^-24, 2^-16 of a site's largest component) times the growth
# of five CG steps; a direction left out or added twice shows at 0.45 in the second
# iteration and 0.08 in the fifth.
@pytest.mark.parametrize("op", ["clover", "staggered"])
@pytest.mark.parametrize("precision,bar", [("double", 1e-12), ("single", 1e-5), ("half", 5e-3)])
def test_iterate_when_the_solve_stops(lmb, orc, monkeypatch, op, precision, bar):
    monkeypatch.setenv("LMB_PERSISTENT", "0")
    L, nw, spins = (6, 4, 4, 8), (1 if op == "clover" else 3), (4 if op == "clover" else 1)
    U, b = orc.random_su3_links(L, 0.25, 97), orc.gaussian_field(L, 3, spins, 98)
    Ud, bd = _links(lmb, U, nw), lmb.LatticeMatrix.from_array(b, nw=nw, phases=PHASES)
    if op == "clover":
        D = lmb.WilsonDiracCloverOperator4D(Ud, 0.12, 1.0)
        ref = orc.Operator(orc.OP_CLOVER, U, L, kappa=0.12, csw=1.0, F=orc.clover_field_strength(U))
    else:
        D, ref = lmb.StaggeredDiracOperator4D(Ud, 0.5), orc.Operator(orc.OP_STAGGERED, U, L, mass=0.5)
    for n, xs in enumerate(_cg_iterates(ref.ddagd, b, 5), 1):
        x = bd.similar()
        res = lmb.cg_(x, lmb.DdagDOp(D, bd.similar()), bd, rtol=1e-14, maxiter=n, precision=precision)
        assert res.iterations == n
        assert rd.rel_err(x.gather_matrix(), xs) <= bar
