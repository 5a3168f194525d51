"""The table of corner terms against a chunk's terms (k_rows_terms), which are
evaluated one by one: the same bits on meshes whose tet count leaves every kind of
last group of eight tets, with cavities whose tets take copies of all faces."""
import numpy as np
import pytest
import torch

from natinterp3d_b200 import device as nd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [5, 6, 7, 8, 9, 10, 11, 12, 40, 41, 300])
def test_same_bits(cuda_device, n):
    rng = np.random.default_rng(n)
    keys = rng.uniform(0, 1, (n, 3))
    c = keys.mean(axis=0)
    packed, _ = nd.gpu_delaunay(keys - c, cuda_device)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(nd, '_room', lambda *a: 0)
        lean = nd.DeviceMesh(*packed, device=cuda_device)
    full = nd.DeviceMesh(*packed, device=cuda_device)
    assert lean.table_bytes == 0 < full.table_bytes
    q = torch.from_numpy(rng.uniform(-0.2, 1.2, (4000, 3))).to(cuda_device)
    for a, b in zip(full.weights_csr(q, c, return_totals=True), lean.weights_csr(q, c, return_totals=True)):
        assert torch.equal(a, b)
