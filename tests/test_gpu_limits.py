"""GPU: the ways round a refused allocation or launch, taken under bounds that
LMB_LIMITS sets (lmb_create reads it), and the results on them.

A bound on the workspaces refuses on the host what the device would refuse when
it is full; nothing here fills the device."""
import numpy as np
import pytest

import refdata as rd

pytestmark = pytest.mark.gpu
PHASES = (1, 1, 1, -1)


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


def _field(lmb, orc, L, spins, seed, nw):
    return lmb.LatticeMatrix.from_array(orc.gaussian_field(L, 3, spins, seed), nw=nw, phases=PHASES)


def _clover_solve(lmb, orc, precision, **kw):
    L = (6, 4, 4, 8)
    D = lmb.WilsonDiracCloverOperator4D(_links(lmb, orc.random_su3_links(L, 0.25, 11), 1), 0.12, 1.0)
    b = _field(lmb, orc, L, 4, 12, 1)
    x = b.similar()
    return lmb.cg_(x, lmb.DdagDOp(D, b.similar()), b, precision=precision, **kw), [x.gather_matrix()]


def _staggered_solve(lmb, orc, precision, **kw):
    L = (6, 4, 4, 8)
    D = lmb.StaggeredDiracOperator4D(_links(lmb, orc.random_su3_links(L, 0.25, 13), 3), 0.3)
    b = _field(lmb, orc, L, 1, 14, 3)
    x = b.similar()
    return lmb.cg_(x, lmb.DdagDOp(D, b.similar()), b, precision=precision, **kw), [x.gather_matrix()]


def _evenodd_solve(lmb, orc, precision, **kw):
    L = (4, 4, 4, 6)
    D = lmb.WilsonDiracCloverOperator4D(_links(lmb, orc.random_su3_links(L, 0.25, 15), 1), 0.12, 1.0)
    b = _field(lmb, orc, L, 4, 16, 1)
    x = b.similar()
    return lmb.solve_evenodd_(x, D, b, precision=precision, **kw), [x.gather_matrix()]


def _domainwall_solve(lmb, orc, precision, **kw):
    L, L5 = (4, 4, 4, 4), 6
    D = lmb.D5DW_MobiusDomainwallOperator5D(_links(lmb, orc.random_su3_links(L, 0.25, 17), 1), L5, 0.2, -1.4, 1.5, 0.5)
    flat = orc.gaussian_field(L[:3] + (L[3] * L5,), 3, 4, 18)
    b = lmb.LatticeMatrix.from_array(np.asfortranarray(flat.reshape((3, 4) + L + (L5,), order="F")), 5, nw=1,
                                     phases=PHASES + (1,))
    x = b.similar()
    return lmb.cg_(x, lmb.DdagDOp(D, b.similar()), b, precision=precision, **kw), [x.gather_matrix()]


def _hisq_force(lmb, orc, precision, **kw):
    L = (4, 4, 4, 4)
    U = _links(lmb, orc.random_su3_links(L, 0.2, 19), 3)
    dU = [u.similar() for u in U]
    res = lmb.hisq_fermion_force_(dU, lmb.HISQDiracCache4D(U, 0.3), _field(lmb, orc, L, 1, 20, 3), precision=precision,
                                  **kw)
    return res, [d.gather_matrix() for d in dU]


def _clover_force(lmb, orc, precision, **kw):
    L = (4, 4, 4, 4)
    U = _links(lmb, orc.random_su3_links(L, 0.2, 21), 1)
    dU = [u.similar() for u in U]
    res = lmb.wilson_clover_fermion_force_(dU, lmb.WilsonDiracCloverOperator4D(U, 0.12, 1.0),
                                           _field(lmb, orc, L, 4, 22, 1), precision=precision, **kw)
    return res, [d.gather_matrix() for d in dU]


def _least(fits):
    """The smallest number of bytes, to 4 KiB, for which fits(bytes) holds."""
    lo, hi = 0, 1 << 16
    while not fits(hi):
        lo, hi = hi, 2 * hi
        assert hi < 1 << 34
    while hi - lo > 4096:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid) else (mid, hi)
    return hi


def _fits(lmb, call):
    try:
        call()
    except lmb.LMBError as e:
        assert "out of device memory" in str(e)
        return False
    return True


# Every number of directions, and every number of updates of x that still wait
# when the solve pauses or stops: the same sum in the same order.  A solve that
# stops with some of them waiting launches one kernel more, which shows how many
# directions it ran with (storages whose solves take no extra ones: one).
@pytest.mark.parametrize("solve,storages", [(_clover_solve, ("double", "single", "half")),
                                            (_evenodd_solve, ("double", "half")),
                                            (_domainwall_solve, ("single", "half")), (_staggered_solve, ("double",))])
@pytest.mark.parametrize("precision", ["double", "single", "half"])
def test_solution_does_not_depend_on_the_directions(lmb, orc, monkeypatch, solve, storages, precision):
    monkeypatch.setenv("LMB_PERSISTENT", "0")
    for maxiter in (2, 3, 4, 300):
        out = []
        for n in (1, 2, 3, 4):
            monkeypatch.setenv("LMB_LIMITS", f"directions={n}")
            out.append(solve(lmb, orc, precision, rtol=1e-9 if maxiter == 300 else 1e-14, maxiter=maxiter))
        assert out[0][0].converged == (maxiter == 300)
        for res, (x,) in out[1:]:
            assert (res.iterations, res.reason) == (out[0][0].iterations, out[0][0].reason)
            np.testing.assert_array_equal(x, out[0][1][0])
        if maxiter < 300 and out[0][0].reliable_updates == 0:
            more = [res.kernel_launches - out[0][0].kernel_launches for res, _ in out]
            assert more == [1 if precision in storages and maxiter % n else 0 for n in (1, 2, 3, 4)]


# Which solves take the extra directions, by the device memory that is gone
# after them: three more fields of 16 V NC bytes (FP64) from 16 MiB a field on,
# none below, as many as LMB_LIMITS says where it does.
@pytest.mark.parametrize("L,limits,extra", [((16, 16, 16, 16), "", 0), ((16, 16, 16, 24), "", 3),
                                            ((16, 16, 16, 16), "directions=4", 3), ((16, 16, 16, 24), "directions=2", 1)])
def test_who_takes_extra_directions(lmb, monkeypatch, L, limits, extra):
    import torch
    U, b = lmb.random_su3_links(L, 0.25, 23), lmb.gaussian_fermion(L, 3, 4, 24, phases=PHASES)
    x, t = b.similar(), b.similar()

    def taken(limits):
        monkeypatch.setenv("LMB_LIMITS", limits)
        D = lmb.WilsonDiracOperator4D(U, 0.12)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        lmb.cg_(x, lmb.DdagDOp(D, t), b, maxiter=2)
        return before - torch.cuda.mem_get_info()[0]
    monkeypatch.setenv("LMB_PERSISTENT", "0")
    taken("directions=1")  # what the process allocates once
    got = taken(limits) - taken("directions=1")
    assert abs(got - extra * 192 * np.prod(L)) <= 1 << 22  # device pages of 2 MiB


# The extra directions are no reason for a call to run out of memory: neither
# what the solve itself asks for after them (the workspaces of its FP64 updates)
# nor what follows on the same context (the gradient of a force, the residual of
# an even/odd solve) is refused because of them.
@pytest.mark.parametrize("call", [_domainwall_solve, _evenodd_solve, _hisq_force, _clover_force])
@pytest.mark.parametrize("precision", ["double", "half"])
def test_directions_take_no_memory_that_is_needed(lmb, orc, monkeypatch, call, precision):
    monkeypatch.setenv("LMB_PERSISTENT", "0")
    monkeypatch.setenv("LMB_DW_TWO_PASS", "1")

    def run(limits):
        monkeypatch.setenv("LMB_LIMITS", limits)
        return call(lmb, orc, precision, rtol=1e-9)
    least = _least(lambda n: _fits(lmb, lambda: run(f"directions=1,workspace={n}")))
    (one, want), (res, got) = run(f"directions=1,workspace={least}"), run(f"workspace={least}")
    assert one.converged and res.converged and res.iterations == one.iterations
    for g, w in zip(got, want):
        assert rd.rel_err(g, w) <= 1e-12
    monkeypatch.setenv("LMB_LIMITS", "workspace=4096")
    assert not _fits(lmb, lambda: call(lmb, orc, precision))


def _hisq_gradient(lmb, orc, L):
    U = _links(lmb, orc.random_su3_links(L, 0.2, 31), 3)
    dU = [u.similar() for u in U]
    lmb.hisq_link_pullback_(dU, lmb.HISQDiracCache4D(U, 0.3, -0.083), U, _field(lmb, orc, L, 1, 32, 3),
                            _field(lmb, orc, L, 1, 33, 3))
    return [d.gather_matrix() for d in dU]


def _hisq_smearing(lmb, orc, L):
    U, psi = _links(lmb, orc.random_su3_links(L, 0.2, 34), 3), _field(lmb, orc, L, 1, 35, 3)
    out = psi.similar()
    lmb.mul_cached_hisq_(out, lmb.HISQDiracCache4D(U, 0.3, -0.083), *U, psi)
    return [out.gather_matrix()]


def _clover_gradient(lmb, orc, L):
    U = _links(lmb, orc.random_su3_links(L, 0.2, 36), 1)
    dU = [u.similar() for u in U]
    lmb.wilson_clover_link_pullback_(dU, lmb.WilsonDiracCloverOperator4D(U, 0.12, 1.0), U, _field(lmb, orc, L, 4, 37, 1),
                                     _field(lmb, orc, L, 4, 38, 1))
    return [d.gather_matrix() for d in dU]


# The first call on a new context makes each workspace once, at the size of its
# largest stage: none is freed, which would wait for the device, to be made anew.
@pytest.mark.parametrize("call", [_hisq_smearing, _hisq_gradient, _clover_gradient,
                                  lambda lmb, orc, L: _hisq_force(lmb, orc, "double")],
                         ids=["smearing", "gradient", "clover", "force"])
def test_first_call_grows_no_workspace(lmb, orc, monkeypatch, call):
    monkeypatch.setenv("LMB_LIMITS", "growths=0")
    call(lmb, orc, (4, 4, 4, 4))


# One direction's (one plane's) workspace where those of all four (six) find no
# memory: bytes per site of the fields a call cannot do without, and 64 KiB of
# small ones.  All together would take 5184, 10368 - 2592 and 1440 more.  The
# stages are the same; the sums into a link run in another order.
@pytest.mark.parametrize("call,site", [(_hisq_smearing, 2 * 576 + 1296 + 2 * 48),
                                       (_hisq_gradient, 8 * 576 + 2592 + 2 * 48),
                                       (_clover_gradient, 2 * 576 + 2 * 192 + 480 + 288)])
@pytest.mark.parametrize("L", [(4, 4, 6, 8), (5, 3, 7, 9)])
def test_gradients_in_less_memory(lmb, orc, monkeypatch, call, site, L):
    want = call(lmb, orc, L)
    monkeypatch.setenv("LMB_LIMITS", f"workspace={int(np.prod(L)) * site + 65536}")
    for g, w in zip(call(lmb, orc, L), want):
        assert rd.rel_err(g, w) <= 1e-13


# The one-launch solver of small lattices, with a grid larger than the device can
# hold at once (refused by the host before anything runs) and with no memory for
# its barrier: the solve takes the staged kernels, three launches an iteration.
@pytest.mark.parametrize("limits", ["blocks=64", "workspace"])
def test_refused_cooperative_launch(lmb, orc, monkeypatch, limits):
    L, rtol = (16, 12, 12, 12), 1e-9
    U, b = orc.random_su3_links(L, 0.25, 41), orc.gaussian_field(L, 3, 4, 42)
    bd = lmb.LatticeMatrix.from_array(b, nw=1, phases=PHASES)

    def run():
        x, D = bd.similar(), lmb.WilsonDiracOperator4D(_links(lmb, U, 1), 0.12)
        return lmb.cg_(x, lmb.DdagDOp(D, bd.similar()), bd, rtol=rtol), x
    one, _ = run()
    assert one.kernel_launches < one.iterations
    if limits == "workspace":  # what the staged kernels take, to 4 KiB
        def staged(n):
            monkeypatch.setenv("LMB_LIMITS", f"directions=1,workspace={n}")
            return _fits(lmb, run)
        monkeypatch.setenv("LMB_PERSISTENT", "0")
        limits = f"directions=1,workspace={_least(staged)}"
        monkeypatch.setenv("LMB_PERSISTENT", "1")
    monkeypatch.setenv("LMB_LIMITS", limits)
    res, x = run()
    assert res.converged and res.iterations == one.iterations
    assert res.kernel_launches >= 3 * res.iterations
    op = orc.Operator(orc.OP_WILSON, U, L, kappa=0.12)
    assert rd.rel_err(op.ddagd(np.asfortranarray(x.gather_matrix())), b) <= 1.05 * rtol


# Which solver runs, told by the launches: one for all iterations up to a reliable
# update, or three an iteration.
@pytest.mark.parametrize("tiles", [0, 100])
@pytest.mark.parametrize("solve", [_clover_solve, _staggered_solve, _evenodd_solve, _domainwall_solve])
@pytest.mark.parametrize("precision", ["double", "half"])
def test_tiles_choose_the_solver(lmb, orc, monkeypatch, solve, precision, tiles):
    monkeypatch.setenv("LMB_LIMITS", f"tiles={tiles}")
    res, _ = solve(lmb, orc, precision, rtol=1e-9)
    assert res.converged and res.iterations > 20
    assert (res.kernel_launches < 3 * res.iterations) == bool(tiles)
