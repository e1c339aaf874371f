"""Distance transforms of wide pores (solids far apart, or none): the scan's cost
grows with the distances, so its passes are handed to the float envelope, whose
cost does not; both choices give the oracle's values."""

import time

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _ball(shape, r):
    g = np.indices(shape)
    return (sum((g[d] - shape[d] / 2) ** 2 for d in range(3)) > r * r).astype(np.uint8)


def _points(shape, p, seed):
    return (np.random.default_rng(seed).random(shape) >= p).astype(np.uint8)


MEDIA = {
    "one_ball": lambda s: _ball(s, 0.1 * min(s)),
    "points": lambda s: _points(s, 2e-5, 3),
    "no_solid": lambda s: np.ones(s, np.uint8),
}


def _kernels():
    import bench
    from pmmoto_gb300._lib import lib

    return bench.prof_read(lib())


@pytest.mark.parametrize("medium", sorted(MEDIA))
@pytest.mark.parametrize("res,n", [((2.25,) * 3, 256), ((1.0, 1.0, 2.0), 256), ((1.0,) * 3, 512)])
def test_wide_pores_cost_no_more_than_the_float_envelope(medium, res, n):
    """No more than twice its time (scans of this size alone take 5 to 30 times as
    long, all steps of the lattice up to 3 times)."""
    import torch

    from pmmoto_gb300 import tune
    from pmmoto_gb300.filters import distance as D

    img = torch.as_tensor(MEDIA[medium]((n, n, n)), device="cuda")
    best, got = {}, {}
    try:
        for path in (0, 2):
            tune._set_lib("edt.path", path)
            got[path] = D.edt3d(img, resolution=res, squared=True)
            best[path] = np.inf
            for _ in range(4):
                torch.cuda.synchronize()
                t = time.perf_counter()
                D.edt3d(img, resolution=res, squared=True)
                torch.cuda.synchronize()
                best[path] = min(best[path], time.perf_counter() - t)
    finally:
        tune._set_lib("edt.path", -1)
    assert torch.equal(got[0], got[2])
    assert best[0] <= 2.0 * best[2]


# passes of few and of many lines, lines shorter than the probe's reach and
# longer, fewer lines than its groups
@pytest.mark.parametrize("shape", [(24, 70, 90), (61, 37, 128), (3, 150, 33), (2, 3, 300), (1, 1, 9)])
@pytest.mark.parametrize("per", [(False,) * 3, (True,) * 3])
def test_both_choices_vs_oracle(shape, per):
    from pmmoto_gb300 import tune
    from pmmoto_gb300._lib import lib
    from pmmoto_gb300.filters import distance as D

    L = lib()
    try:
        for img in (_points(shape, 0.002, 5), _points(shape, 0.2, 6), np.ones(shape, np.uint8)):
            for res in ((1.0, 1.0, 2.0), (2.25,) * 3):
                want = O.edt3d(img, periodic=per, resolution=res, squared=True)
                for k in (0, 8193):
                    tune._set_lib("edt.wide", k)
                    L.pmg_prof_reset()
                    L.pmg_prof_enable(1)
                    got = D.edt3d(img, periodic=per, resolution=res, squared=True)
                    L.pmg_prof_enable(0)
                    np.testing.assert_array_equal(got, want)
                    # (periodic lines of the other size have no scan; with the knob at
                    # 8193 nothing has to be probed)
                    ran = set(_kernels())
                    if res[0] == 1.0:
                        assert {"k_scan_rows", "k_envelope_whole"} <= ran and ("k_pore_probe" in ran) == (k == 0)
    finally:
        L.pmg_prof_enable(0)
        tune._set_lib("edt.wide", -1)


@pytest.mark.parametrize("res", [(2.25,) * 3, (1.0, 1.0, 2.0), (30.0, 0.75, 0.75)])
def test_far_near_ties_on_long_lines_vs_oracle(res):
    """Scans of distances where the envelope's rounding may order values more than
    half a step apart: solids hundreds of voxels away, in pairs that nearly tie."""
    from pmmoto_gb300 import tune
    from pmmoto_gb300.filters import distance as D

    rng = np.random.default_rng(12)
    img = np.ones((40, 3, 1024), np.uint8)
    for i in range(40):
        lo, hi = rng.integers(0, 200), rng.integers(824, 1024)
        img[i, rng.integers(0, 3), lo] = img[i, rng.integers(0, 3), hi] = 0
    want = O.edt3d(img, resolution=res, squared=True)
    try:
        tune._set_lib("edt.wide", 8193)
        np.testing.assert_array_equal(D.edt3d(img, resolution=res, squared=True), want)
        np.testing.assert_array_equal(D.edt3d(img.transpose(0, 2, 1).copy(), resolution=(res[0], res[2], res[1]), squared=True),
                                      O.edt3d(img.transpose(0, 2, 1).copy(), resolution=(res[0], res[2], res[1]), squared=True))
    finally:
        tune._set_lib("edt.wide", -1)


@pytest.mark.parametrize("shape", [(5, 300, 520), (7, 520, 299), (300, 260, 12)])
@pytest.mark.parametrize("per", [(False,) * 3, (True,) * 3, (False, True, False)])
def test_lattice_lines_left_to_the_envelope_vs_oracle(shape, per):
    """Power-of-two voxels: lines longer than a lattice pass reaches with few solids
    or none, beside lines with many, so that blocks give up their lines early, late
    or not at all."""
    from pmmoto_gb300.filters import distance as D

    rng = np.random.default_rng(sum(shape))
    media = [_points(shape, 1e-4, 7), _points(shape, 3e-6, 8), np.ones(shape, np.uint8)]
    half = np.ones(shape, np.uint8)  # dense in one corner, a single solid in the far half
    half[:, : shape[1] // 4, : shape[2] // 3] = rng.random((shape[0], shape[1] // 4, shape[2] // 3)) >= 0.1
    half[shape[0] // 2, -2, -3] = 0
    for img in media + [half]:
        for res in ((1.0,) * 3, (2.0, 1.0, 1.0)):
            for squared in (True, False):
                np.testing.assert_array_equal(D.edt3d(img, periodic=per, resolution=res, squared=squared),
                                              O.edt3d(img, periodic=per, resolution=res, squared=squared))
