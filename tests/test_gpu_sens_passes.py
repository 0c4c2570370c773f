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
