"""Which problems the substructured solver takes (sub_fits, sub_plan.cpp): the
rule by its numbers, on the host."""
import ctypes as C

import pytest

ROOT_MAX = {0: 48 * 1024 // 16 - 16 - 8 * 33, 1: 48 * 1024 // 8 - 32 - 8 * 33}  # complex128, complex64


@pytest.fixture(scope="module")
def fits():
    from titatest_gb300 import build
    f = C.CDLL(build.build()).crgpu_sub_fits
    f.argtypes = [C.c_int32] * 7 + [C.c_double] * 2

    def call(mixed, n, mb, m, mp, eanz=96, c_factor=1e8, c_apply=1e6):
        return f(mixed, n, mb, m, mp, ROOT_MAX[mixed], eanz, c_factor, c_apply)
    return call


@pytest.mark.parametrize("mixed,block", [(0, 16), (1, 32)])
def test_root_beyond_one_blocks_shared_memory_keeps_the_band(fits, mixed, block):
    """A mesh as deep as it is wide, where operation counts alone favour the
    root by far, at the last padded root that fits and one block beyond it."""
    mp = ROOT_MAX[mixed] // block * block
    n, mb = (mp // 3) ** 2, mp // 3 + 1
    assert fits(mixed, n, mb, mp, mp)
    assert not fits(mixed, n, mb, mp + 1, mp + block)
