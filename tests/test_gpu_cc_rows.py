"""Row runs of the labelling (tiles of 4 x 8 rows of 32 elements) at tile edges
and remainders, dense and sparse, one value and several, against the oracle
(labels and their numbering equal)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# voxel extents around the tile sizes of the voxel (4 x 8 x 32) and the block
# (8 x 16 x 64) labelling, odd ones, single planes and lines
SHAPES = [(4, 8, 32), (5, 9, 33), (8, 16, 64), (9, 17, 65), (7, 15, 63), (16, 33, 130), (3, 40, 200), (33, 2, 97)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fill", [0.12, 0.35, 0.97])
def test_labels_vs_oracle(shape, fill):
    from pmmoto_gb300.core import initialize
    from pmmoto_gb300.filters import connected_components as C

    rng = np.random.default_rng(int(1000 * fill) + shape[2])
    sd, g = initialize(shape), O.Geom(shape)
    one = (rng.random(shape) < fill).astype(np.uint8)
    # checkerboards touch by edges and corners only
    idx = np.indices(shape).sum(0)
    several = one * rng.integers(1, 4, shape).astype(np.uint8)
    for img in (one, one * 7, one * (idx % 2 == 0), several, several.astype(np.int32), several.astype(np.int64)):
        lbl, n = C.connect_components(np.ascontiguousarray(img), sd)
        want, wn = O.connect_components(np.ascontiguousarray(img), g)
        np.testing.assert_array_equal(lbl, want)
        assert n == wn


@pytest.mark.parametrize("kinds", [("periodic",) * 3, ("end", "wall", "periodic")])
def test_periodic_labels_of_long_seams_vs_oracle(kinds):
    """Seams whose rows mostly repeat the key of the row before."""
    from pmmoto_gb300.core import initialize
    from pmmoto_gb300.filters import connected_components as C

    vox = (30, 26, 70)
    bts = tuple((k, k) for k in kinds)
    sd, g = initialize(vox, boundary_types=bts), O.Geom(vox, boundary_types=bts)
    rng = np.random.default_rng(8)
    for img in (np.ones(sd.voxels, np.uint8), (rng.random(sd.voxels) < 0.9).astype(np.uint8),
                np.kron(rng.random(tuple(-(-v // 4) for v in sd.voxels)) < 0.5, np.ones((4, 4, 4)))
                [tuple(slice(0, v) for v in sd.voxels)].astype(np.uint8)):
        img = O.update_buffer(g, np.ascontiguousarray(img))
        lbl, n = C.connect_components(img, sd)
        want, wn = O.connect_components(img, g)
        np.testing.assert_array_equal(lbl, want)
        assert n == wn
