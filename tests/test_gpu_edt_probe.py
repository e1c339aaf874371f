"""Periodic lines of voxels that are powers of two but not equal: the probe sends
wide pores to the float envelope and narrow ones to the scan, pass by pass;
both, and media that differ between the axes, against the oracle (values
equal)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _balls(shape, n, r, seed):
    rng = np.random.default_rng(seed)
    g = np.indices(shape)
    img = np.ones(shape, np.uint8)
    for c, rad in zip(rng.random((n, 3)) * np.array(shape), rng.uniform(0.7, 1.3, n) * r):
        img[sum((g[d] - c[d]) ** 2 for d in range(3)) <= rad * rad] = 0
    return img


@pytest.mark.parametrize("shape", [(24, 70, 90), (61, 37, 128), (3, 150, 33)])
@pytest.mark.parametrize("kind", ["wide", "narrow", "plates"])
def test_periodic_media_vs_oracle(shape, kind):
    from pmmoto_gb300.filters import distance as D

    if kind == "wide":
        img = _balls(shape, 3, 5.0, 5)
    elif kind == "narrow":
        img = (np.random.default_rng(6).random(shape) >= 0.2).astype(np.uint8)
    else:  # solid planes far apart: wide along one axis only
        img = np.ones(shape, np.uint8)
        img[:, :: 35, :] = 0
    for res in ((2.0, 1.0, 1.0), (1.0, 0.5, 2.0)):
        for per in ((True,) * 3, (False, True, True), (True, True, False)):
            got = D.edt3d(img, periodic=per, resolution=res, squared=True)
            np.testing.assert_array_equal(got, O.edt3d(img, periodic=per, resolution=res, squared=True))
