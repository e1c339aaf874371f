"""Erosions and dilations beyond the capped pipeline's thresholds (radii above 31
voxels of a power-of-two size) on the lattice pass, against the oracle."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vox", [(100, 77, 90), (41, 100, 131)])
@pytest.mark.parametrize("radius", [32.0, 37.3, 60.1])
@pytest.mark.parametrize("kinds", [("wall",) * 3, ("end", "wall", "periodic"), ("periodic",) * 3])
def test_wide_radii_vs_oracle(vox, radius, kinds):
    import bench
    import pmmoto_gb300 as P
    from pmmoto_gb300._lib import lib
    from pmmoto_gb300.filters import morphological_operators as M

    if any(np.ceil(radius) > n for n in vox):
        pytest.skip("refused: wider than an axis")
    h = 0.125
    kw = dict(box=tuple((0.0, v * h) for v in vox), boundary_types=tuple((k, k) for k in kinds))
    sd, g = P.initialize(vox, **kw), O.Geom(vox, **kw)
    rng = np.random.default_rng(int(radius))
    img = O.update_buffer(g, (rng.random(sd.voxels) >= 2e-5).astype(np.uint8))
    r = radius * h
    L = lib()
    L.pmg_prof_reset()
    L.pmg_prof_enable(1)
    try:
        eroded, dilated = M.erode(sd, img, r), M.dilate(sd, 1 - img, r)
    finally:
        L.pmg_prof_enable(0)
    np.testing.assert_array_equal(eroded, O.subtraction(g, img, r))
    np.testing.assert_array_equal(dilated, O.addition(g, 1 - img, r))
    ran = set(bench.prof_read(L))
    assert "k_par_cols" in ran and not any(k.startswith("k_scan") for k in ran)
