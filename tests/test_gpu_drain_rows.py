"""Drainage on row words (32 blocks of 2x2x2 voxels to a word): extents around
the pieces and tiles, odd and even rows, wall planes on every axis, a reservoir,
probes wider than the small-window dilation, steps that change nothing, and a
second curve from the state of the first, against the oracle (saturations and
final phases equal)."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (voxels, boundary types, reservoir voxels, voxels per unit length, spheres, probe radii in voxels)
END, WALL = ("end", "end"), ("wall", "wall")
CASES = {
    "odd": ((37, 35, 69), (END, WALL, WALL), 0, 32, 90, np.linspace(1, 8, 12)),
    "even_rows": ((40, 33, 130), (END, WALL, END), 0, 32, 160, np.linspace(1, 7, 9)),
    "one_piece": ((40, 18, 64), (END, WALL, WALL), 3, 32, 60, np.linspace(1, 6, 8)),
    "thin_rows": ((48, 30, 7), (END, WALL, WALL), 2, 32, 40, np.linspace(1, 5, 6)),
    "walls_along": ((34, 26, 66), (END, WALL, END), 0, 32, 70, np.linspace(1, 6, 7)),
    "wide_probe": ((96, 80, 72), (END, END, END), 0, 32, 26, [3.0, 10.0, 14.0, 17.0, 19.5, 21.5, 23.0]),
    "float_scale": ((37, 30, 50), (END, WALL, WALL), 0, 30, 80, np.linspace(1, 7, 7)),
    "float_reservoir": ((37, 30, 66), (END, WALL, WALL), 4, 30, 80, np.linspace(1, 7, 7)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_curves_vs_oracle(name):
    import pmmoto_gb300 as P

    vox, bts, rv, scale, n, radii = CASES[name]
    rng = np.random.default_rng(len(name) + vox[2])
    box = tuple((0.0, v / scale) for v in vox)
    inlet, outlet = ((True, False), (False, False), (False, False)), ((False, True), (False, False), (False, False))
    sd = P.initialize(vox, box=box, boundary_types=bts, inlet=inlet, outlet=outlet, reservoir_voxels=rv)
    g = O.Geom(vox, boundary_types=bts, box=box, inlet=inlet, outlet=outlet, reservoir_voxels=rv)
    sph = np.c_[rng.random((n, 3)) * np.array([b[1] for b in box]), rng.uniform(0.05, 0.14, n)]
    pm = P.domain_generation.gen_pm_spheres_domain(sd, sph)
    # radii below a voxel and above the largest pore change nothing
    pcs = sorted(list(2.0 / (np.r_[0.4, radii, radii[-1], 500.0] / scale)))
    mp = P.domain_generation.gen_mp_constant(pm, 2)
    half = len(pcs) // 2
    state = None
    for part in (pcs[:half], pcs[half:]):
        sat = P.filters.equilibrium_distribution.drainage(mp, list(part), mode="distance")
        want, state = O.drainage(g, pm.img, list(part), mp_img=state)
        np.testing.assert_array_equal(sat, want)
        np.testing.assert_array_equal(mp.img, state)
