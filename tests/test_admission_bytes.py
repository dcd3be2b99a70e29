"""The bytes that admission counts for a lattice (host calls, no GPU): the array
that two-step launches work with is in them where creation takes it."""
import ctypes

import pytest


def desc(kind, bcase, l, m, n, pattern=0):
    from bgk3d_gpu_b200._lattice_abi import LatticeDesc
    from bgk3d_gpu_b200._lib import lib
    d = LatticeDesc()
    lib().bgk_lattice_desc_init(ctypes.byref(d), kind, bcase, l, m, n, 1.0)
    d.pattern = pattern
    return d


def figures(d):
    from bgk3d_gpu_b200._lib import lib
    return lib().bgk_lattice_device_bytes(ctypes.byref(d)), lib().bgk_lattice_least_bytes(ctypes.byref(d))


@pytest.mark.parametrize("kind,bcase,shape,pattern,arrays", [
    (1, 1, (256, 256, 256), 0, 38), (0, 0, (128, 128, 128), 0, 38), (1, 3, (512, 256, 256), 0, 38),
    (4, 1, (40, 150, 110), 0, 38), (4, 1, (256, 256, 256), 0, 38), (1, 1, (32, 32, 32), 0, 37), (2, 1, (256, 256, 256), 0, 37), (1, 1, (256, 256, 256), 1, 19),
    (1, 1, (1200, 1000, 900), 0, 37),            # an array of 4 GB or more takes single steps
])
def test_arrays_counted(kind, bcase, shape, pattern, arrays):
    full, least = figures(desc(kind, bcase, *shape, pattern=pattern))
    base = 19 if pattern else 37
    assert least % base == 0
    assert full == least // base * arrays


@pytest.mark.parametrize("kind,bcase", [(1, -1), (0, 9), (4, -1), (7, 1)])
def test_figures_of_descriptions_that_creation_refuses(kind, bcase):
    full, least = figures(desc(kind, bcase, 256, 256, 256))
    assert full == least > 0


def test_requests_count_the_table_of_solid_links():
    from bgk3d_gpu_b200.serve import Request, _bytes, lattice_bytes
    big = Request(0, 0.0, "sphere", 128, 10, 0.6, "f32")
    full, least = _bytes(big)
    array = least // 37
    assert lattice_bytes(big) == full
    assert array < full - least < array + 4 * (128 // 6 + 4) ** 3
    small = Request(1, 0.0, "sphere", 32, 10, 0.6, "f32")
    assert _bytes(small)[0] == _bytes(small)[1]
