"""Pore sizes of unequal voxel edges, and drainage curves of more radii than the
step volume counts, against the oracle (values equal)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# (entry points refuse three different edges)
@pytest.mark.parametrize("edges", [(0.5, 0.25, 0.25), (0.25, 0.25, 0.5), (0.3, 0.3, 0.2), (5.0, 2.25, 2.25)])
@pytest.mark.parametrize("kind", ["periodic", "mixed"])
def test_pore_sizes_of_unequal_voxels(edges, kind):
    import pmmoto_gb300 as P

    vox = (27, 30, 34)
    bts = {"periodic": (("periodic", "periodic"),) * 3,
           "mixed": (("end", "end"), ("wall", "wall"), ("periodic", "periodic"))}[kind]
    box = tuple((0.0, v * e) for v, e in zip(vox, edges))
    sd, g = P.initialize(vox, box=box, boundary_types=bts), O.Geom(vox, box=box, boundary_types=bts)
    rng = np.random.default_rng(7)
    sph = np.c_[rng.random((40, 3)) * np.array([b[1] for b in box]), rng.uniform(2.0, 5.0, 40) * min(edges)]
    pm = P.domain_generation.gen_pm_spheres_domain(sd, sph)
    h = np.array(g.resolution, dtype=float)
    odd = min(h) * np.array([1.1, 2.3, 3.7, 5.2])
    # distances between voxel centres: decided by a radius's own field
    lattice = [float(v) for v in (h[0], 2 * h[1], np.hypot(h[0], h[1]), np.sqrt((h ** 2).sum()), 2 * h[2])]
    for radii in (np.array(sorted(lattice + list(odd))), odd, np.array(lattice[::-1])):
        # (the ball modes measure in voxels of the first axis, which unequal edges do not suit)
        got = P.filters.porosimetry.pore_size_distribution(sd, pm, radii=radii.copy(), mode="distance")
        np.testing.assert_array_equal(got, O.pore_size_distribution(g, pm.img, radii.copy(), mode="distance"))


@pytest.mark.parametrize("n", [254, 255, 260])
@pytest.mark.parametrize("scale", [32, 30])
def test_drainage_of_many_radii(n, scale):
    import pmmoto_gb300 as P

    vox = (28, 20, 23)
    bts = (("end", "end"), ("wall", "wall"), ("wall", "wall"))
    box = tuple((0.0, v / scale) for v in vox)
    kw = dict(box=box, boundary_types=bts, inlet=((True, False), (False, False), (False, False)),
              outlet=((False, True), (False, False), (False, False)))
    sd, g = P.initialize(vox, **kw), O.Geom(vox, **kw)
    rng = np.random.default_rng(n + scale)
    sph = np.c_[rng.random((40, 3)) * np.array([b[1] for b in box]), rng.uniform(0.05, 0.14, 40)]
    pm = P.domain_generation.gen_pm_spheres_domain(sd, sph)
    pcs = sorted(float(p) for p in 2.0 / (np.linspace(0.9, 7.0, n) / scale))
    mp = P.domain_generation.gen_mp_constant(pm, 2)
    sat = P.filters.equilibrium_distribution.drainage(mp, list(pcs), mode="distance")
    want, state = O.drainage(g, pm.img, list(pcs))
    np.testing.assert_array_equal(sat, want)
    np.testing.assert_array_equal(mp.img, state)
