"""The lattice and scan passes of the distance transform at the sizes where
their tiles, segments and line classes change, against the oracle (whole
numbers times a power of two, or the reference's float steps: no tolerance)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# lines of one chunk, one segment, several, the longest of each class (and one
# more voxel), odd extents beside even ones and multiples of four
SHAPES = [(15, 64, 64), (17, 65, 66), (128, 63, 129), (129, 256, 5), (33, 257, 128), (1024, 3, 8), (1025, 4, 6),
          (2, 1024, 33), (3, 1025, 4), (5, 2, 1024), (7, 3, 1023), (2049, 2, 3), (1, 1, 1), (2, 513, 512), (16, 1, 257)]


def _media(shape, seed):
    rng = np.random.default_rng(seed)
    p0 = (0.4, 0.05, 0.003, 0.0)[seed % 4]
    img = (rng.random(shape) >= p0).astype(np.uint8)
    if seed % 3 == 2:
        img = np.where(img > 0, rng.integers(1, 4, shape), 0).astype(np.uint8)
    return img


@pytest.mark.parametrize("i", range(len(SHAPES)))
@pytest.mark.parametrize("res", [(0.5, 0.5, 0.5), (2.25, 2.25, 2.25), (5.0, 2.25, 0.01)])
def test_edt3d_sizes_vs_oracle(i, res):
    from pmmoto_gb300.filters import distance as D

    shape = SHAPES[i]
    for k, per in enumerate(((False,) * 3, (True,) * 3, (False, True, True))):
        img = _media(shape, i + k)
        got = D.edt3d(img, periodic=per, resolution=res, squared=True)
        np.testing.assert_array_equal(got, O.edt3d(img, periodic=per, resolution=res, squared=True),
                                      err_msg=f"{shape} {per} {res}")


@pytest.mark.parametrize("per", [(False,) * 3, (True,) * 3])
def test_edt3d_far_solids_vs_oracle(per):
    """Distances beyond the packed heights' range (245 voxels) on lines that
    hold a solid voxel, and lines without one."""
    from pmmoto_gb300.filters import distance as D

    img = np.ones((260, 6, 600), np.uint8)
    img[3, 2, 5] = img[250, 4, 590] = 0
    for squared in (True, False):
        np.testing.assert_array_equal(D.edt3d(img, periodic=per, squared=squared),
                                      O.edt3d(img, periodic=per, squared=squared))


@pytest.mark.parametrize("seed", range(6))
def test_periodic_imports_vs_oracle(seed):
    """Line ends that depend on the imported hulls: solids a few voxels to
    half a line away from the seams, and balls whose hulls keep more entries
    than are imported."""
    from pmmoto_gb300.filters import distance as D

    rng = np.random.default_rng(70 + seed)
    shape = [(64, 64, 64), (40, 130, 72), (30, 24, 340)][seed % 3]
    idx = np.indices(shape)
    img = np.ones(shape, np.uint8)
    for _ in range(6 + 4 * seed):
        c, r = rng.random(3) * shape, rng.uniform(2, 9)
        img[((idx - c[:, None, None, None]) ** 2).sum(0) <= r * r] = 0
    for res in ((1.0,) * 3, (0.3,) * 3):
        np.testing.assert_array_equal(D.edt3d(img, periodic=(True,) * 3, resolution=res, squared=True),
                                      O.edt3d(img, periodic=(True,) * 3, resolution=res, squared=True))


@pytest.mark.parametrize("radius", [1.0, 2.3, 6.0, 11.7])
@pytest.mark.parametrize("bc", ["periodic", "wall"])
def test_erosion_of_other_voxel_sizes_vs_oracle(radius, bc):
    """Morphology on the scan passes: values beyond the radius are cut off,
    values at it compared as the reference's floats."""
    import pmmoto_gb300 as P
    from pmmoto_gb300.filters import morphological_operators as M

    vox, h = (50, 41, 66), 0.01
    kw = dict(box=tuple((0.0, v * h) for v in vox), boundary_types=((bc, bc),) * 3)
    sd, g = P.initialize(vox, **kw), O.Geom(vox, **kw)
    rng = np.random.default_rng(5)
    img = O.update_buffer(g, (rng.random(sd.voxels) >= 0.002).astype(np.uint8))
    r = radius * h
    np.testing.assert_array_equal(M.erode(sd, img, r), O.subtraction(g, img, r))
    np.testing.assert_array_equal(M.dilate(sd, 1 - img, r), O.addition(g, 1 - img, r))
