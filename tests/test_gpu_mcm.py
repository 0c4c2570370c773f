"""Model uncertainty and resolution (crgpu_mcm: src/bmcm_mod.f90 bata,
bata_reg, bmcm, bres, bmcm2) on the library's own dense FP64 kernels, against
the oracle's restatement, on config 1's Jacobian (1200 cells: 19 blocks of
the blocked Cholesky factor and inverse, the last one partial).

Both sides are FP64 with different summation orders; the diagonals agree to
1e-9 relative (the resolution diagonal relative to its largest entry)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ltri", [0, 1])
def test_mcm_dense_kernels_match_oracle(gpu_lib, ltri):
    from titatest_gb300 import PLAIN, CRMod, synth
    from titatest_gb300 import regularization as R
    s = synth.config1()
    g = s.grid
    rng = np.random.default_rng(71)
    with CRMod(g, s.survey, precision=PLAIN) as m:
        m.forward(s.sigma, volt_mode=1)
        J = m.sens(1)  # also kept on the device for crgpu_mcm
        nanz, manz = J.shape
        wmatd = rng.uniform(0.5, 2.0, size=nanz) / 0.03 ** 2
        wdfak = np.ones(nanz, np.int32)
        if ltri == 0:
            smatm, nach = R.bsmatmreg(g, s.nx, s.nz), None
        else:
            nach = R.bnachbar(g)
            smatm = R.bsmatmtri(g, nach)
        d = m.mcm(wmatd, wdfak, ltri, smatm, nx=s.nx, nachbar=nach, lam=30.0)
    o = O.mcm(J, wmatd, wdfak, ltri, smatm, nx=s.nx, nachbar=nach, maxnk=g.maxnk, lam=30.0)
    assert manz == 1200
    for key in ("ata", "reg", "cov1", "cov2"):
        err = np.max(np.abs(d[key] / o[key] - 1))
        assert err < 1e-9, (key, err)
    assert np.max(np.abs(d["res"] - o["res"])) / np.max(np.abs(o["res"])) < 1e-9


def test_more_data_than_cells_by_chunks_of_rows(gpu_lib):
    """12000 data on 1000 cells: the product with the covariance goes through S
    by chunks of rows, within the work space of a covariance matrix, and the
    diagonals are those of plain FP64 matrices."""
    from test_gpu_memory import _Peak
    from test_gpu_sens_passes import _survey
    from test_gpu_substruct import _case
    from titatest_gb300 import PLAIN, CRMod, formats
    s = _case(50, 20, 40)
    n, m = 1000, 12000
    st, vn = _survey(40, m, False, 5)
    sv = formats.Survey(enr=s.survey.enr, strnr=st, vnr=vn, strom=np.ones(m))
    reg = np.zeros((n, 3), order="F")
    reg[:, 0] = 1.0
    w, one = np.linspace(0.5, 2.0, m), np.ones(m, np.int32)
    with CRMod(s.grid, sv, np.array([0.05, 0.4]), np.array([0.1, 0.2]), precision=PLAIN) as c:
        c.forward(s.sigma)
        J = c.sens(0)
        w /= np.abs(J).max() ** 2
        with _Peak() as peak:
            d = c.mcm(w, one, 0, reg.ravel(order="F"), nx=50, lam=1.0)
    S = np.concatenate([np.sqrt(w)[:, None] * J.real, np.sqrt(w)[:, None] * J.imag])
    ata = S.T @ S
    cov = np.linalg.inv(ata + np.eye(n))
    res = cov @ ata
    assert peak.bytes < 8 * (2 * m * n + 4 * n * n) + (48 << 20)
    for key, ref in (("ata", np.diag(ata)), ("cov1", np.diag(cov)), ("res", np.diag(res)), ("cov2", np.diag(res @ cov))):
        assert np.max(np.abs(d[key] - ref)) / np.max(np.abs(ref)) < 1e-9, key
