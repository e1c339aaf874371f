"""Pore size distributions whose openings share one erosion distance field:
voxel sizes with and without exact fields, periodic extensions, walls, radii on
lattice distances (decided by their own fields), both comparison types, with and
without the inlet filter, against the oracle (values equal)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

KINDS = {
    "periodic": (("periodic", "periodic"),) * 3,
    "mixed": (("end", "end"), ("wall", "wall"), ("periodic", "periodic")),
    "closed": (("wall", "wall"),) * 3,
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("scale", [32, 30])
@pytest.mark.parametrize("mode", ["distance", "hybrid", "morph"])
def test_sizes_vs_oracle(kind, scale, mode):
    import pmmoto_gb300 as P

    vox = (37, 30, 46) if scale == 32 else (36, 30, 42)
    box = tuple((0.0, v / scale) for v in vox)
    inlet = ((kind == "mixed", False), (False, False), (False, False))
    sd = P.initialize(vox, box=box, boundary_types=KINDS[kind], inlet=inlet)
    g = O.Geom(vox, boundary_types=KINDS[kind], box=box, inlet=inlet)
    rng = np.random.default_rng(scale + len(kind))
    sph = np.c_[rng.random((70, 3)) * np.array([b[1] for b in box]), rng.uniform(0.06, 0.16, 70)]
    pm = P.domain_generation.gen_pm_spheres_domain(sd, sph)
    res = float(min(g.resolution))
    odd = list(res * np.array([1.1, 2.3, 3.7, 4.45, 5.2]))
    lattice = list(res * np.array([1.0, 2.0, 3.0]) * np.sqrt(2.0)) + [2 * res, 3 * res]
    for radii in (np.array(odd + lattice), odd, lattice, odd[:1]):
        for use_inlet in {False, kind == "mixed"}:
            got = P.filters.porosimetry.pore_size_distribution(sd, pm, radii=radii.copy(), inlet=use_inlet, mode=mode)
            want = O.pore_size_distribution(g, pm.img, radii.copy(), inlet=use_inlet, mode=mode)
            np.testing.assert_array_equal(got, want)
