"""Pore sizes report a failure of the shared distance field: only a failed
allocation makes every radius erode by itself."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_failed_launch_is_reported():
    import torch

    import pmmoto_gb300 as P
    from pmmoto_gb300._lib import PmgError, lib
    from pmmoto_gb300.filters import porosimetry

    vox = (30, 26, 34)
    sd = P.initialize(vox, box=tuple((0.0, float(v)) for v in vox), boundary_types=(("periodic", "periodic"),) * 3)
    img = np.ones(sd.voxels, np.uint8)
    img[:, 8:12] = 0
    pm = P.domain_generation.gen_pm(sd, torch.as_tensor(img, device="cuda"))
    radii = [1.5, 2.5, 3.5]
    want = porosimetry.pore_size_distribution(sd, pm, radii=radii)
    # the runtime refuses a copy from no address (nothing runs on the device) and
    # keeps the error for the next launch check of this thread, which is the field's
    L = lib()
    L.pmg_cnn_check.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert L.pmg_cnn_check(None, None) != 0
    with pytest.raises(PmgError):
        porosimetry.pore_size_distribution(sd, pm, radii=radii)
    assert torch.equal(porosimetry.pore_size_distribution(sd, pm, radii=radii), want)
