"""Halo update and maximum of volumes with short rows (fewer voxels than a warp has
lanes): values against the oracle or numpy, and no more time than a small multiple
of a copy of the volume."""

import time

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

KINDS = ("end", "wall", "periodic")


@pytest.mark.parametrize("n2", [2, 3, 5, 7, 8, 13, 16, 17, 31, 33, 70])
def test_halo_update_vs_oracle(n2):
    import torch

    import pmmoto_gb300 as P
    from pmmoto_gb300 import _ops
    from pmmoto_gb300.core.geometry import geo_of

    vox = (5, 9, n2)
    rng = np.random.default_rng(n2)
    for kinds in ((a, b, c) for a in KINDS for b in KINDS for c in KINDS):
        bts = tuple((k, k) for k in kinds)
        sd, g = P.initialize(vox, boundary_types=bts), O.Geom(vox, boundary_types=bts)
        for dtype in (np.uint8, np.float32):
            img = rng.integers(0, 200, sd.voxels).astype(dtype)
            got = _ops.update_buffer_device(torch.as_tensor(img, device="cuda"), geo_of(sd)).cpu().numpy()
            np.testing.assert_array_equal(got, O.update_buffer(g, img))


@pytest.mark.parametrize("shape", [(3, 5, 1), (7, 2, 4), (40, 30, 6), (1, 1, 500), (9, 1, 17), (2, 900, 33)])
def test_maximum_vs_numpy(shape):
    import torch

    from pmmoto_gb300 import _ops

    x = np.random.default_rng(sum(shape)).normal(size=shape).astype(np.float32)
    t = torch.as_tensor(x, device="cuda")
    assert _ops.max_f32_device(t) == x.max()
    box = np.array([v for n in shape for v in (n // 3, n)], np.int64)
    assert _ops.max_f32_device(t, box) == x[shape[0] // 3:, shape[1] // 3:, shape[2] // 3:].max()


def _best(fn):
    import torch

    fn()
    best = np.inf
    for _ in range(5):
        torch.cuda.synchronize()
        t = time.perf_counter()
        fn()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


def test_short_rows_cost_like_the_copy_of_the_volume():
    import torch

    import pmmoto_gb300 as P
    from pmmoto_gb300 import _ops
    from pmmoto_gb300.core.geometry import geo_of

    vox = (4000, 2000, 4)
    g = geo_of(P.initialize(vox, boundary_types=(("periodic", "periodic"),) * 3))
    x = torch.ones(tuple(n + 2 for n in vox), dtype=torch.float32, device="cuda")
    copy = _best(lambda: x.clone())
    assert _best(lambda: _ops.update_buffer_device(x, g)) <= 15 * copy
    assert _best(lambda: _ops.max_f32_device(x)) <= 10 * copy
