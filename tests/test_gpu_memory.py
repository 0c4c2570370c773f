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
