"""The Jacobian's passes and dipole tables (post.cu) against the oracle's
bsens and bsensi, both precisions: more measurements than a pass holds, more
distinct dipoles on both sides than a table holds, poles (absent electrodes),
triangles and quadrilaterals.  Tolerances as in test_gpu_forward.py."""
import numpy as np
import pytest

from conftest import relerr

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _survey(ne, nanz, poles, seed):
    """Random four-electrode configurations: hardly any dipole twice."""
    rng = np.random.default_rng(seed)
    q = np.array([rng.choice(ne, 4, replace=False) + 1 for _ in range(nanz)])
    if poles:
        q[::3, 0] = 0  # A absent
        q[1::5, 3] = 0  # N absent
    return (q[:, 0] * 10000 + q[:, 1]).astype(np.int32), (q[:, 2] * 10000 + q[:, 3]).astype(np.int32)


@pytest.mark.parametrize("ne,nanz,poles,tri", [(4, 5, False, False), (24, 700, True, True), (48, 2600, False, False),
                                               (20, 4500, True, False)])
def test_sensitivities_match_oracle(gpu_lib, ne, nanz, poles, tri):
    from titatest_gb300 import MIXED, PLAIN, CRMod, formats
    from test_gpu_substruct import _case
    s = _case(50, 6, ne, tri)
    st, vn = _survey(ne, nanz, poles, 5)
    sv = formats.Survey(enr=s.survey.enr, strnr=st, vnr=vn, strom=np.linspace(0.5, 2.0, nanz))
    P = O.Problem(s.grid, sv)
    kwn, kwnwi = P.rwaven()
    kp = P.forward(s.sigma, kwn, kwnwi)
    volt, _ = P.bvolt(P.rtrafo(kp, kwnwi), 0, None)
    ref = [P.bsens(kp, kwn, kwnwi, s.sigma, volt, mode=m) for m in (0, 1)]
    for prec, tol in ((PLAIN, 1e-10), (MIXED, 1e-5)):
        with CRMod(s.grid, sv, kwn, kwnwi, precision=prec) as m:
            if prec == MIXED:
                m.set_tune(0, 0, 2)  # the direct form
            m.forward(s.sigma)
            # bsensi divides by V: compared times |V|, which random configurations spread over decades
            v = np.abs(volt)[:, None]
            assert relerr(m.bsens(), ref[0]) < tol
            assert relerr(m.bsensi() * v, ref[1] * v) < tol


@pytest.mark.parametrize("ne,parts,poles", [(90, (1300, 1500, 2300), False), (70, (2100,), True), (90, (33, 4096), False)])
def test_passes_with_and_without_tables_match_oracle(gpu_lib, ne, parts, poles):
    """Surveys that repeat their dipoles in parts only: stretches of random
    configurations (passes without tables) between stretches of 40 dipoles
    (passes with tables), and lengths around a pass and a warp."""
    from titatest_gb300 import MIXED, PLAIN, CRMod, formats
    from test_gpu_substruct import _case
    s = _case(100, 4, ne)
    rng = np.random.default_rng(8)
    st, vn = [], []
    for q, n in enumerate(parts):
        a, b = _survey(ne, n, poles, 5 + q)
        if q % 2:
            a, b = rng.choice(a[:40], n), rng.choice(b[:40], n)
            same = {(x, y) for x, y in zip(a, b) if {x // 10000, x % 10000} & {y // 10000, y % 10000} - {0}}
            keep = np.array([(x, y) not in same for x, y in zip(a, b)])  # no shared electrode
            a, b = a[keep], b[keep]
        st.append(a)
        vn.append(b)
    st, vn = np.concatenate(st).astype(np.int32), np.concatenate(vn).astype(np.int32)
    sv = formats.Survey(enr=s.survey.enr, strnr=st, vnr=vn, strom=np.linspace(0.5, 2.0, len(st)))
    P = O.Problem(s.grid, sv)
    kwn, kwnwi = np.array([0.02, 0.1, 0.5]), np.array([0.1, 0.2, 0.3])
    kp = P.forward(s.sigma, kwn, kwnwi)
    volt, _ = P.bvolt(P.rtrafo(kp, kwnwi), 0, None)
    ref = [P.bsens(kp, kwn, kwnwi, s.sigma, volt, mode=m) for m in (0, 1)]
    v = np.abs(volt)[:, None]
    for prec, tol in ((PLAIN, 1e-10), (MIXED, 1e-5)):
        with CRMod(s.grid, sv, kwn, kwnwi, precision=prec) as m:
            if prec == MIXED:
                m.set_tune(0, 0, 2)  # the direct form
            m.forward(s.sigma)
            assert relerr(m.bsens(), ref[0]) < tol
            assert relerr(m.bsensi() * v, ref[1] * v) < tol


def test_jacobian_to_pinned_memory_leaves_the_updates_jacobian(gpu_lib):
    """CRMod's Jacobian into page-locked memory, in chunks of a buffer beside the
    device array: the bits of the pageable one, and crgpu_update still reads the
    Jacobian of log V that the device holds."""
    import ctypes as C

    import torch

    from titatest_gb300 import MIXED, CRMod
    from test_gpu_substruct import _case
    s = _case(200, 30, 150)
    nanz, manz = s.survey.nanz, s.grid.elanz
    assert nanz * manz * 16 > 3 * (4 << 20)  # several chunks
    with CRMod(s.grid, s.survey, precision=MIXED) as m:
        m.set_tune(0, 0, 2)  # the direct form, with tables
        v = m.forward(s.sigma)["volt"]
        ref = m.bsens()
        reg = np.zeros((3, manz))  # smatm(manz, 3), column-major
        reg[0] = 1.0

        def update():
            return m.update(np.ones(nanz), np.ones(nanz, np.int32), -np.log(v) * 1.01, -np.log(v), 0,
                            reg, nx=200, lam=300.0, ncgmax=5)

        m.bsensi()
        before = update()
        host = torch.zeros(2 * nanz * manz, dtype=torch.float64).pin_memory()
        assert gpu_lib.crgpu_sens(m._h, 0, C.cast(host.data_ptr(), C.POINTER(C.c_double))) == 0
        got = host.numpy().view(np.complex128).reshape(manz, nanz).T
        assert np.array_equal(got, ref)
        for x, y in zip(before, update()):
            assert np.array_equal(np.asarray(x), np.asarray(y))
