"""Calls while device memory is short: the rest of it is held by a tensor."""
import ctypes as C

import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


def _trim():
    """Gives what the library's pool keeps back to the device."""
    cu = C.CDLL("libcuda.so.1")
    dev, pool = C.c_int(0), C.c_void_p()
    assert cu.cuDeviceGet(C.byref(dev), 0) == 0 and cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    assert cu.cuMemPoolTrimTo(pool, C.c_size_t(0)) == 0


class _Short:
    """with _Short(nbytes): only about nbytes of device memory are free."""

    def __init__(self, nbytes):
        self.nbytes = nbytes

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        _trim()
        free, _ = torch.cuda.mem_get_info()
        assert free > self.nbytes
        self.hold = torch.empty(free - self.nbytes, dtype=torch.uint8, device="cuda")

    def __exit__(self, *a):
        import torch
        del self.hold
        torch.cuda.empty_cache()


def test_failed_allocation_leaves_no_error_behind(gpu_lib):
    """A context whose arrays do not fit reports 94, and the next call on the
    same thread is not blamed for it."""
    from test_gpu_substruct import _case
    from titatest_gb300 import PLAIN, CRMod
    from titatest_gb300._lib import CRGPUError
    small, big = _case(24, 9, 16), _case(260, 60, 64)
    with CRMod(small.grid, small.survey, precision=PLAIN) as m:
        v = m.forward(small.sigma)["volt"]
        with _Short(128 << 20):
            with pytest.raises(CRGPUError) as ei:
                CRMod(big.grid, big.survey, precision=PLAIN)
            assert ei.value.errnr == 94
            assert np.array_equal(m.forward(small.sigma)["volt"], v)


def test_batch_whose_second_problem_does_not_fit(gpu_lib):
    """The first problem's work on its two streams is over before its buffers
    are given back: the call fails with 94, and problems that reuse the
    memory at once get the voltages of a run alone."""
    from test_gpu_substruct import _case
    from titatest_gb300 import MIXED, CRMod
    from titatest_gb300._lib import CRGPUError
    from titatest_gb300.crmod import forward_sens_batch
    one, two = _case(200, 50, 48), _case(260, 60, 64)
    ms = [CRMod(s.grid, s.survey, precision=MIXED) for s in (one, two)]
    need = ms[0].memory_need()
    assert ms[1].memory_need() > 1.5 * need
    with _Short(need + (256 << 20)):
        with pytest.raises(CRGPUError) as ei:
            forward_sens_batch(ms, [one.sigma, two.sigma], sens_mode=-1)
        assert ei.value.errnr == 94
        ms[0].close()
        with CRMod(one.grid, one.survey, precision=MIXED) as m:
            v = m.forward(one.sigma)["volt"]
    ms[1].close()
    with CRMod(one.grid, one.survey, precision=MIXED) as m:
        assert relerr(v, m.forward(one.sigma)["volt"]) < 1e-12


class _Peak:
    """Most bytes that the library's pool had handed out, beyond those at the
    start of the block."""

    def __enter__(self):
        self.cu = C.CDLL("libcuda.so.1")
        dev, self.pool = C.c_int(0), C.c_void_p()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0
        zero = C.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, 8, C.byref(zero)) == 0  # USED_MEM_HIGH
        self.start = self._get(7)  # USED_MEM_CURRENT
        return self

    def _get(self, attr):
        v = C.c_uint64(0)
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value

    def __exit__(self, *a):
        self.bytes = self._get(8) - self.start


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-10)])
@pytest.mark.parametrize("share", [0.6, 0.3])
def test_memory_budget_holds_the_shared_arrays_too(gpu_lib, prec, tol, share):
    """Forward and adjoint within a share of what one batch takes: some of the
    wavenumbers at a time, the results of one batch (tolerance: rounding in
    complex128, the refinement's in mixed precision)."""
    from test_gpu_substruct import _case
    from titatest_gb300 import CRMod
    s = _case(120, 40, 12)
    kwn, kwnwi = np.geomspace(0.01, 2.0, 10), np.full(10, 0.1)
    g = np.random.default_rng(2).normal(size=(s.survey.nanz, 2)) @ np.array([1.0, 1j])
    with CRMod(s.grid, s.survey, kwn, kwnwi, precision=prec) as m:
        whole = m.memory_need() - s.survey.nanz * s.grid.elanz * 16
        v, a = m.forward(s.sigma)["volt"], m.adjoint(g)
    with CRMod(s.grid, s.survey, kwn, kwnwi, precision=prec) as m:
        m.set_memory_budget(int(share * whole))
        with _Peak() as peak:
            w = m.forward(s.sigma)["volt"]
        assert m.stats()["nbatches"] > 1
        b = m.adjoint(g)
    assert peak.bytes <= share * whole + (1 << 20)  # small change: counters and roundings of the pool
    assert relerr(w, v) < tol and relerr(b, a) < tol


@pytest.mark.parametrize("leave", [0.7, 0.25, 0.05])
def test_forward_where_memory_is_short(gpu_lib, leave):
    """Less room than the default budget assumes: rectangles shrink until they
    fit, and where not even one wavenumber's shared arrays do, the band takes
    the problem in batches.  Same voltages and gradient."""
    from test_gpu_substruct import _case
    from titatest_gb300 import MIXED, CRMod
    s = _case(900, 60, 8)
    kwn, kwnwi = np.geomspace(0.01, 2.0, 6), np.full(6, 0.1)
    g = np.random.default_rng(2).normal(size=(s.survey.nanz, 2)) @ np.array([1.0, 1j])
    with CRMod(s.grid, s.survey, kwn, kwnwi, precision=MIXED) as m:
        need = m.memory_need() - s.survey.nanz * s.grid.elanz * 16
        v, a = m.forward(s.sigma)["volt"], m.adjoint(g)
    with CRMod(s.grid, s.survey, kwn, kwnwi, precision=MIXED) as m:
        m.forward(s.sigma)
        m.adjoint(g)  # the gradient's own arrays are there
        m.set_memory_budget(0)  # and the solver's are given back
        with _Short(int(leave * need)):
            w = m.forward(s.sigma)["volt"]
            assert m.stats()["nbatches"] > 1
            b = m.adjoint(g)
    assert relerr(w, v) < 1e-10 and relerr(b, a) < 1e-9


@pytest.mark.parametrize("nx,nz,same", [(120, 40, False), (400, 10, True)])
def test_contexts_on_the_band_keep_no_elimination_plan(gpu_lib, nx, nz, same):
    """Forwards with singularity removal run on the band, so such a context
    has no tables of the dissection; nor has one that the rule leaves on the
    band (400 x 10 cells in complex128)."""
    from test_gpu_substruct import _case
    from titatest_gb300 import PLAIN, CRMod
    s = _case(nx, nz, 12)
    kwn, kwnwi = np.geomspace(0.01, 2.0, 4), np.full(4, 0.1)
    held = []
    for lsr in (False, True):
        with _Peak() as peak:
            with CRMod(s.grid, s.survey, kwn, kwnwi, lsr=lsr, precision=PLAIN):
                pass
        held.append(peak.bytes)
    assert held[1] == held[0] if same else held[1] < held[0] - 4 * s.grid.sanz  # one position a node at least


def test_refused_context_takes_no_device_memory(gpu_lib):
    """A mixed context in a band of 258 is refused (1002) before its arrays are
    allocated and filled."""
    from test_gpu_substruct import _case
    from titatest_gb300 import MIXED, CRMod
    from titatest_gb300._lib import CRGPUError
    s = _case(160, 150, 8)
    assert s.grid.mb > 207
    with _Peak() as peak:
        with pytest.raises(CRGPUError) as ei:
            CRMod(s.grid, s.survey, precision=MIXED, band_order=0)
    assert ei.value.errnr == 1002 and peak.bytes == 0
