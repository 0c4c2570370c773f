"""Which problems the substructured solver takes (sub_fits, sub_plan.cpp): the
rule by its numbers, on the host."""
import ctypes as C

import pytest

ROOT_MAX = {0: 48 * 1024 // 16 - 16 - 8 * 33, 1: 48 * 1024 // 8 - 32 - 8 * 33}  # complex128, complex64


@pytest.fixture(scope="module")
def fits():
    from titatest_gb300 import build
    f = C.CDLL(build.build()).crgpu_sub_fits
    f.argtypes = [C.c_int32] * 8 + [C.c_double] * 2

    def call(mixed, n, mb, m, mp, eanz=96, kwn=13, c_factor=1e8, c_apply=1e6):
        return f(mixed, n, mb, m, mp, ROOT_MAX[mixed], eanz, kwn, c_factor, c_apply)
    return call


@pytest.mark.parametrize("mixed,block", [(0, 16), (1, 32)])
def test_root_beyond_one_blocks_shared_memory_keeps_the_band(fits, mixed, block):
    """A mesh as deep as it is wide, where operation counts alone favour the
    root by far, at the last padded root that fits and one block beyond it."""
    mp = ROOT_MAX[mixed] // block * block
    n, mb = (mp // 3) ** 2, mp // 3 + 1
    assert fits(mixed, n, mb, mp, mp)
    assert not fits(mixed, n, mb, mp + 1, mp + block)


# columns x rows of cells, electrodes, wavenumbers, plan's counts, and the times in
# ms of a forward on the band and on the substructured solver (GB300)
MEASURED = [
    (1, 1000, 20, 96, 13, 22, 1.07e8, 2.14e6, 50.0, 61.1), (1, 500, 20, 96, 13, 22, 3.75e7, 1.03e6, 25.7, 13.9),
    (1, 1500, 30, 96, 13, 32, 2.39e8, 4.94e6, 110, 182), (1, 800, 30, 96, 13, 32, 1.22e8, 2.64e6, 58.4, 41.1),
    (1, 2000, 60, 96, 13, 62, 8.32e8, 1.48e7, 313, 448), (1, 1250, 60, 96, 13, 62, 4.4e8, 9.0e6, 196, 139),
    (1, 2600, 60, 24, 10, 62, 1.08e9, 1.92e7, 286, 486), (1, 2000, 60, 24, 10, 62, 8.32e8, 1.48e7, 220, 243), (1, 2000, 60, 8, 4, 62, 8.32e8, 1.48e7, 208, 77),
    (1, 2000, 100, 96, 13, 102, 1.57e9, 2.57e7, 1531, 516), (1, 200, 60, 96, 13, 62, 3.9e7, 1.36e6, 32.0, 9.6),
    (0, 600, 20, 24, 4, 41, 2.81e7, 1.03e6, 49.7, 63.9), (0, 300, 20, 24, 4, 41, 1.17e7, 4.98e5, 25.0, 13.2),
    (0, 1000, 30, 24, 10, 61, 1.04e8, 2.97e6, 287, 766), (0, 600, 30, 24, 4, 61, 5.12e7, 1.70e6, 91, 69),
    (0, 2000, 60, 24, 4, 121, 6.92e8, 1.36e7, 1298, 1819), (0, 800, 60, 96, 8, 121, 2.0e8, 5.2e6, 3021, 861),
    (0, 600, 20, 48, 8, 41, 2.81e7, 1.03e6, 137, 261), (0, 60, 20, 30, 10, 41, 2.5e6, 1.0e5, 8.8, 2.2),
]


@pytest.mark.parametrize("case", MEASURED)
def test_choice_follows_the_measured_times(fits, case):
    """The faster side by a tenth at least, from shallow to deep meshes and from
    few systems to many."""
    mixed, nx, nz, ne, kwn, mb, c_factor, c_apply, band, sub = case
    assert max(band, sub) > 1.1 * min(band, sub)
    m, block = nx + 2 * nz + 1, 32 if mixed else 16
    got = fits(mixed, (nx + 1) * (nz + 1), mb, m, -(-m // block) * block, ne, kwn, c_factor, c_apply)
    assert bool(got) == (sub < band)
