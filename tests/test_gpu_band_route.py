"""The band path, pinned (crgpu_set_tune): ordinary forwards run on the
substructured solver, but singularity removal, DC mode, prescribed Dirichlet
values and long meshes keep the band, so its kernels are run here in every
setting that the other files run on the default route.  Tolerances as in
test_gpu_forward.py: mixed against complex128 1e-6 (voltages) and 1e-5
(Jacobian), complex128 against complex128 1e-10."""
import numpy as np
import pytest

from conftest import load_case, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [(0, 1, 2, 3), (1, 3), (2,)])
def test_batch_of_band_and_substructured_contexts(gpu_lib, pinned):
    """One persistent tensor-core launch for the pinned problems, the others
    beside it: each as alone on its route, and as complex128."""
    from titatest_gb300 import MIXED, PLAIN, CRMod, synth
    from titatest_gb300.crmod import forward_sens_batch
    shapes = synth.config5_shapes()
    by_size = sorted(range(len(shapes)), key=lambda q: shapes[q][0] * shapes[q][1])
    probs = synth.config5(indices=[by_size[q] for q in (0, 60, 90, 128)])

    def model(q, p):
        m = CRMod(p.grid, p.survey, precision=MIXED)
        m.set_refinement(8, 1e-10)
        if q in pinned:
            m.set_tune(1)
        return m

    models = [model(q, p) for q, p in enumerate(probs)]
    try:
        volts = forward_sens_batch(models, [p.sigma for p in probs], sens_mode=0)
        for q, (m, p, v) in enumerate(zip(models, probs, volts)):
            assert m.stats()["refine_iterations"] >= 1
            J = m.bsens()
            with model(q, p) as m1:
                assert relerr(v, m1.forward(p.sigma)["volt"]) < 1e-9
                assert relerr(J, m1.bsens()) < 1e-8
            with CRMod(p.grid, p.survey, precision=PLAIN) as mp:
                assert relerr(v, mp.forward(p.sigma)["volt"]) < 1e-6
    finally:
        for m in models:
            m.close()


def test_graph_replay_on_the_band(gpu_lib):
    """Config 3 on the tensor-core factor: two full rounds of systems and a
    partial third on the second stream, recorded and replayed bit for bit."""
    import torch

    from titatest_gb300 import MIXED, CRMod, synth
    s = synth.config3()
    nanz, manz = s.survey.nanz, s.grid.elanz
    sig = torch.from_numpy(s.sigma.view(np.float64).copy()).cuda()
    volt = torch.zeros(2 * nanz, dtype=torch.float64, device="cuda")
    sens = torch.zeros(2 * nanz * manz, dtype=torch.float64, device="cuda")
    with CRMod(s.grid, s.survey, precision=MIXED) as m:
        m.set_stream(torch.cuda.current_stream().cuda_stream)
        m.set_refinement(8, 1e-2)
        d = m.forward(s.sigma)["volt"]
        m.set_tune(1)

        def ordinary():
            m.forward_device(sig.data_ptr(), volt.data_ptr())
            m.sens_device(0, sens.data_ptr())
            torch.cuda.synchronize()
            return volt.clone(), sens.clone()

        v0, j0 = ordinary()
        assert relerr(v0.cpu().numpy().view(np.complex128), d) < 1e-3  # refined to 1e-2 of the potentials only
        for _ in range(3):  # record, then replay twice
            m.forward_sens_graph(sig.data_ptr(), volt.data_ptr(), 0, sens.data_ptr())
            torch.cuda.synchronize()
            assert torch.equal(volt, v0) and torch.equal(sens, j0)
        sig.mul_(1.25)
        m.forward_sens_graph(sig.data_ptr(), volt.data_ptr(), 0, sens.data_ptr())
        torch.cuda.synchronize()
        v1, j1 = volt.clone(), sens.clone()
        v2, j2 = ordinary()
        assert torch.equal(v1, v2) and torch.equal(j1, j2) and not torch.equal(v1, v0)


@pytest.mark.parametrize("prec,tol", [(0, 1e-10), (1, 1e-6)])
def test_adjoint_on_the_band_resident_and_refactored(gpu_lib, prec, tol):
    from titatest_gb300 import CRMod
    g_, sv, sig, _, _ = load_case("testmodinv")
    g = np.random.default_rng(3).normal(size=(sv.nanz, 2)) @ np.array([1.0, 1j])
    grads = []
    for budget in (None, (g_.sanz * (g_.mb + 1) * 16 + g_.sanz * 16 * 40) * 7):
        with CRMod(g_, sv, precision=prec) as m:
            m.set_tune(1)
            if budget:
                m.set_memory_budget(budget)  # a handful of systems per batch
            m.forward(sig)
            assert (m.stats()["nbatches"] > 1) == bool(budget)
            grads.append(m.adjoint(g))
    with CRMod(g_, sv, precision=0) as m:  # the substructured solver's
        m.forward(sig)
        ref = m.adjoint(g)
    for got in grads:
        assert relerr(got, ref) < tol


@pytest.mark.parametrize("tune,wide", [((1, 0), False), ((2, 1), False), ((2, 2), False), ((2, 4), False),
                                       ((4, 0), False), ((3, 1), True), ((3, 2), True)])
def test_forward_on_every_factor_kernel(gpu_lib, tune, wide):
    """Each kernel that the autotuner may choose, in a whole forward: config 1,
    and a band of 192 in the grid's own order."""
    from test_gpu_forward import _wide_band_case
    from titatest_gb300 import MIXED, PLAIN, CRMod, synth
    if wide:
        g, sv, sig = _wide_band_case()
    else:
        s = synth.config1()
        g, sv, sig = s.grid, s.survey, s.sigma
    with CRMod(g, sv, precision=PLAIN) as m:
        m.set_tune(1)
        ref = m.forward(sig, kpot=True)
        J = m.bsens()
    with CRMod(g, sv, precision=MIXED, band_order=0 if wide else 1) as m:
        m.set_tune(*tune)
        m.set_refinement(10, 1e-10)
        out = m.forward(sig, kpot=True)
        assert relerr(out["kpot"], ref["kpot"]) < 1e-6 and relerr(out["volt"], ref["volt"]) < 1e-6
        assert relerr(m.bsens(), J) < 1e-5


def test_band_in_geometric_order(gpu_lib):
    """The strip of band 192 in its nodes' geometric order (band 8)."""
    from test_gpu_forward import _wide_band_case
    from titatest_gb300 import MIXED, PLAIN, CRMod
    g, sv, sig = _wide_band_case()
    with CRMod(g, sv, precision=PLAIN) as m:
        ref = m.forward(sig, kpot=True, hpot=True)
    for kind in (1, 4):
        with CRMod(g, sv, precision=MIXED) as m:
            m.set_tune(kind)
            m.set_refinement(10, 1e-10)
            out = m.forward(sig, kpot=True, hpot=True)
        for key in ("kpot", "hpot", "volt"):
            assert relerr(out[key], ref[key]) < 1e-6
