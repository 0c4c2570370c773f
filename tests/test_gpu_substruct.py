"""The substructured solver (shared elimination of the nodes off the mixed
boundary, one dense root per system) against the oracle's band solution, at
the sizes where its tiles and chains end: a mesh with a handful of interior
nodes, electrode counts around the 32-wide tiles, separators beyond one
front's 64 nodes, jittered triangles, and rectangles of systems cut by the
memory budget.  Tolerances as in test_gpu_forward.py: complex128 1e-10,
complex64 + FP64 refinement 1e-6."""
import numpy as np
import pytest

from conftest import relerr

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(nx, nz, ne, tri=False, seed=3):
    from titatest_gb300 import synth
    rng = np.random.default_rng(seed)
    grid, surface, _, _ = synth._quad_grid(np.arange(nx + 1, dtype=float), np.arange(nz + 1) * 0.7, triangles=tri,
                                           jitter=0.2 if tri else 0.0, rng=rng)
    mag, pha = synth.random_model(grid, rng)
    enodes = np.linspace(1, nx - 1, ne).astype(int)
    return synth._finish("sub", grid, surface, enodes, synth.dipole_dipole(ne, [1], [1, 2]), mag, pha, nx, nz)


@pytest.mark.parametrize("nx,nz,ne,tri", [(5, 4, 4, False), (24, 9, 16, True), (66, 13, 31, False),
                                          (67, 20, 33, False), (72, 70, 6, False), (40, 30, 32, True),
                                          (12, 5, 5, False), (150, 5, 20, False)])
def test_forward_and_adjoint_match_oracle(gpu_lib, nx, nz, ne, tri):
    from titatest_gb300 import MIXED, PLAIN, CRMod
    s = _case(nx, nz, ne, tri)
    P = O.Problem(s.grid, s.survey)
    kwn, kwnwi = P.rwaven()
    kp = P.forward(s.sigma, kwn, kwnwi)
    volt, _ = P.bvolt(P.rtrafo(kp, kwnwi), 0, None)
    g = np.random.default_rng(1).normal(size=(s.survey.nanz, 2)) @ np.array([1.0, 1j])
    grads = {}
    for prec, tol in ((PLAIN, 1e-10), (MIXED, 1e-6)):
        with CRMod(s.grid, s.survey, kwn, kwnwi, precision=prec) as m:
            out = m.forward(s.sigma, kpot=True)
            grads[prec] = m.adjoint(g)
            assert relerr(out["kpot"], kp) < tol
            assert relerr(out["volt"], volt) < tol
    assert relerr(grads[MIXED], grads[PLAIN]) < 1e-6


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("systems", [5, 33, 70])
def test_rectangles_of_a_small_memory_budget(gpu_lib, prec, systems):
    """Fewer systems than one wavenumber has electrodes, and whole
    wavenumbers that do not divide their count: the same voltages and
    adjoint as one batch."""
    from titatest_gb300 import CRMod
    s = _case(45, 16, 33)
    g = np.random.default_rng(2).normal(size=(s.survey.nanz, 2)) @ np.array([1.0, 1j])
    with CRMod(s.grid, s.survey, precision=prec) as m:
        v1 = m.forward(s.sigma)["volt"]
        a1 = m.adjoint(g)
        assert m.stats()["nbatches"] == 1
    nb = 45 + 2 * 16 + 1
    mp = (nb + 31) // 32 * 32
    esz = 16 if prec == 0 else 8
    per = mp * (mp + 32) * esz + s.grid.sanz * (3 * esz + (32 if prec else 0))
    with CRMod(s.grid, s.survey, precision=prec) as m:
        m.set_memory_budget(int(per * systems * 1.35))
        v2 = m.forward(s.sigma)["volt"]
        assert m.stats()["nbatches"] > 1
        a2 = m.adjoint(g)
    assert relerr(v2, v1) < 1e-12 and relerr(a2, a1) < 1e-12


@pytest.mark.parametrize("prec", [0, 1])
def test_memory_need_covers_the_root_factors(gpu_lib, prec):
    """The bytes a batch would still allocate: the root factors of every
    system before a forward, the Jacobian alone after it."""
    from titatest_gb300 import CRMod
    s = _case(60, 20, 20)
    with CRMod(s.grid, s.survey, precision=prec) as m:
        roots = m.kwnanz * 20 * (60 + 2 * 20 + 1) ** 2 * (16 if prec == 0 else 8)
        sens = s.survey.nanz * s.grid.elanz * 16
        assert m.memory_need() > roots + sens
        m.forward(s.sigma)
        assert m.memory_need() == sens


@pytest.mark.parametrize("where", ["interior", "corner"])
def test_fictitious_sink_is_a_source(gpu_lib, where):
    """The right-hand sides with a fictitious sink, inside the mesh and on the
    mixed boundary (a root node): only fronts above a source take part in
    their upward sweep."""
    from titatest_gb300 import MIXED, PLAIN, CRMod
    s = _case(36, 14, 9)
    g = s.grid
    x, y = g.node_xy()
    nsink = int(np.argmin(np.hypot(x - 18, y + 5)) if where == "interior" else np.argmax(x - y)) + 1
    P = O.Problem(g, s.survey)
    kwn, kwnwi = P.rwaven()
    kp = P.forward(s.sigma, kwn, kwnwi, lsink=True, nsink=nsink)
    for prec, tol in ((PLAIN, 1e-10), (MIXED, 1e-6)):
        with CRMod(g, s.survey, kwn, kwnwi, lsink=True, nsink=nsink, precision=prec) as m:
            assert relerr(m.forward(s.sigma, kpot=True)["kpot"], kp) < tol


@pytest.mark.parametrize("maxit,tol", [(0, 1e-10), (1, 1e-10), (2, 0.0), (8, 1e-2), (8, 1e-10), (64, 1e-10)])
def test_refinement_stops_alike_on_every_route(gpu_lib, maxit, tol):
    """Steps launched as the host learns of the systems left (forward, and
    several contexts in turn) and steps that a graph's loop repeats: the same
    bits and the same count of steps, from no step at all to the most."""
    import torch

    from titatest_gb300 import MIXED, CRMod, crmod
    cases = [_case(24, 9, 16), _case(36, 33, 9, True)]
    mods = [CRMod(s.grid, s.survey, precision=MIXED) for s in cases]
    try:
        for m in mods:
            m.set_refinement(maxit, tol)
        one = [(m.forward(s.sigma)["volt"], m.stats()["refine_iterations"]) for m, s in zip(mods, cases)]
        both = crmod.forward_sens_batch(mods, [s.sigma for s in cases])
        for m, (v, n), w in zip(mods, one, both):
            assert np.array_equal(v, w) and m.stats()["refine_iterations"] == n <= maxit
        s, m = cases[0], mods[0]
        sig = torch.from_numpy(s.sigma.view(np.float64).copy()).cuda()
        volt = torch.zeros(2 * s.survey.nanz, dtype=torch.float64, device="cuda")
        sens = torch.zeros(2 * s.survey.nanz * s.grid.elanz, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(3):  # record, then replay twice
            volt.zero_()
            torch.cuda.synchronize()
            m.forward_sens_graph(sig.data_ptr(), volt.data_ptr(), 0, sens.data_ptr())
            assert np.array_equal(volt.cpu().numpy().view(np.complex128), one[0][0])
            assert m.stats()["refine_iterations"] == one[0][1]
    finally:
        for m in mods:
            m.close()


def test_long_mesh_with_a_large_root_matches_the_band(gpu_lib):
    """2700 x 60 cells in complex128: a root of 2821 nodes is more than its
    solve's shared memory holds, so the default route is the pinned band's."""
    from titatest_gb300 import PLAIN, CRMod
    s = _case(2700, 60, 6)
    with CRMod(s.grid, s.survey, [0.05], [0.1], precision=PLAIN) as m:
        v = m.forward(s.sigma)["volt"]
        m.set_tune(1)  # complex128 has one band factor; any choice pins the band
        w = m.forward(s.sigma)["volt"]
    assert np.all(w != 0) and np.array_equal(v, w)
