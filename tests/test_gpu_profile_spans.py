"""nif_profile_kernels: the row kernels' times add up to the row phase's, on a
mesh whose rows all go to k_rows_general, and launches are counted by kernel."""
import ctypes

import numpy as np
import pytest
import torch

import natinterp3d_b200 as ni
from natinterp3d_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('scale', [1.0, 1e-7])
def test_times_add_up(cuda_device, scale):
    rng = np.random.default_rng(3)
    it = ni.Interpolator(rng.uniform(0, scale, (5000, 3)), constructor='gpu')
    q = torch.from_numpy(rng.uniform(0.1 * scale, 0.9 * scale, (400_000, 3))).to(cuda_device)
    v = torch.from_numpy(rng.standard_normal((5000, 1))).to(cuda_device)
    lib = N.cuda_lib()
    it.interpolate_device(q, v)
    phases, ms, launches = (ctypes.c_double * 4)(), (ctypes.c_double * 5)(), (ctypes.c_double * 5)()
    N.check(lib.nif_profile_enable(1), 'enable')
    try:
        for _ in range(3):
            it.interpolate_device(q, v)
        N.check(lib.nif_profile_read(phases), 'read')
        N.check(lib.nif_profile_kernels(ms, launches), 'kernels')
    finally:
        lib.nif_profile_enable(0)
    assert list(launches) == [1.0] * 5
    # the events of a phase enclose those of its kernels, a few us of launches apart
    assert 0.9 * phases[1] <= sum(ms) <= phases[1]
