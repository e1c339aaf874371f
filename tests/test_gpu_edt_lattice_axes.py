"""Lattice passes chosen axis by axis: power-of-two voxels that are coarser along
the earlier axes, and volumes with one long axis, against the oracle (values
equal), and which kernels took the passes."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(img, **kw):
    from pmmoto_gb300._lib import lib
    from pmmoto_gb300.filters import distance as D

    import bench

    L = lib()
    L.pmg_prof_reset()
    L.pmg_prof_enable(1)
    try:
        got = D.edt3d(img, squared=True, **kw)
    finally:
        L.pmg_prof_enable(0)
    return got, set(bench.prof_read(L))


def _media(shape, seed):
    rng = np.random.default_rng(seed)
    yield (rng.random(shape) >= 0.2).astype(np.uint8)
    yield (rng.random(shape) >= 0.002).astype(np.uint8)
    far = np.ones(shape, np.uint8)  # heights beyond the packed range, and lines without a solid
    far[0, shape[1] // 2, :: 7] = 0
    yield far


# the last two: a ratio of the sizes at the largest shift, and beyond it
@pytest.mark.parametrize("res", [(2.0, 1.0, 1.0), (1.0, 0.5, 0.25), (4.0, 4.0, 0.5), (1.0, 1.0, 2.0), (1.0, 2.0, 1.0),
                                 (2.0 ** 16, 1.0, 1.0), (2.0 ** 17, 1.0, 1.0)])
@pytest.mark.parametrize("shape", [(40, 33, 70), (300, 20, 64), (9, 130, 257)])
def test_unequal_powers_of_two_vs_oracle(shape, res):
    small = 2.0 ** 16
    for img in _media(shape, 3):
        for per in ((False,) * 3, (True,) * 3, (True, False, True)):
            got, ran = _run(img, periodic=per, resolution=res)
            np.testing.assert_array_equal(got, O.edt3d(img, periodic=per, resolution=res, squared=True))
            assert ("k_par_cols" in ran) == (res[1] <= res[0] <= small * res[1])
            assert ("k_par_rows" in ran) == (res[2] <= min(res[:2]) and max(res[:2]) <= small * res[2])


@pytest.mark.parametrize("shape", [(1025, 6, 40), (2048, 5, 8), (2049, 4, 33), (30, 1025, 9), (20, 9, 1025)])
def test_one_long_axis_vs_oracle(shape):
    for img in _media(shape, 4):
        for per in ((False,) * 3, (True,) * 3):
            got, ran = _run(img, periodic=per)
            np.testing.assert_array_equal(got, O.edt3d(img, periodic=per, squared=True))
            assert ("k_par_cols" in ran) == (shape[1] <= 1024)
            assert ("k_par_rows" in ran) == (shape[2] <= 1024)
