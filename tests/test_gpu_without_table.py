"""Meshes without the table of corner terms (above 2^26 tets, or where device
memory has no room for it): the terms of a chunk's rows are written beside
their records.  Bit for bit against the same mesh with the table, on calls of
one row, on both sides of the row kernels' spreading and of a chunk, with rows
of the general and the wide kind, through every kind of call and a batch of
both kinds of mesh."""
import numpy as np
import pytest
import torch

from natinterp3d_b200 import batch as nb
from natinterp3d_b200 import device as nd

pytestmark = pytest.mark.gpu


def _lean(mesh, n_tets, monkeypatch):
    """The mesh again, as if its buffer had no room for the table."""
    empty = torch.empty

    def refuse(*a, **k):
        if a and isinstance(a[0], int) and a[0] > 512 * n_tets:
            raise torch.cuda.OutOfMemoryError('no room')
        return empty(*a, **k)
    with monkeypatch.context() as m:
        m.setattr(nd.torch, 'empty', refuse)
        dm = nd.DeviceMesh(*mesh, device='cuda:0')
    assert dm._buf.numel() < 512 * n_tets
    return dm


@pytest.fixture(scope='module')
def meshes(cuda_device):
    rng = np.random.default_rng(81)
    d = rng.standard_normal((60, 3))
    keys = np.concatenate([rng.uniform(0, 1, (3000, 3)),  # and a hole of wide cavities
                           0.5 + 0.06 * rng.uniform(1, 1.001, (60, 1)) *
                           d / np.linalg.norm(d, axis=1, keepdims=True)])
    c = keys.mean(axis=0)
    mesh, _ = nd.gpu_delaunay(keys - c)
    mesh = tuple(x.cpu().numpy() for x in mesh)
    mp = pytest.MonkeyPatch()
    return nd.DeviceMesh(*mesh, device=cuda_device), _lean(mesh, len(mesh[1]), mp), c, len(keys)


def _bits(x):
    return x.contiguous().view(torch.int64 if x.element_size() == 8 else torch.int32)


@pytest.mark.parametrize('m', [1, 63, 4097, 16385, (1 << 20) + 5])
@pytest.mark.parametrize('dt', [torch.float64, torch.float32])
def test_same_bits(meshes, cuda_device, m, dt):
    full, lean, c, n = meshes
    rng = np.random.default_rng(m)
    q = rng.uniform(-0.05, 1.05, (m, 3))
    q[::3] = 0.5 + 0.08 * (q[::3] - 0.5)
    q = torch.from_numpy(q).to(cuda_device, dt)
    v = torch.from_numpy(rng.standard_normal((n, 3))).to(cuda_device, dt)
    assert torch.equal(_bits(full.interpolate(q, v, c)), _bits(lean.interpolate(q, v, c)))
    for a, b in zip(full.weights_csr(q, c, return_totals=True), lean.weights_csr(q, c, return_totals=True)):
        assert torch.equal(_bits(a), _bits(b))


def test_gradient_and_batch(meshes, cuda_device):
    full, lean, c, n = meshes
    rng = np.random.default_rng(5)
    q = torch.from_numpy(rng.uniform(0.1, 0.9, (7001, 3))).to(cuda_device)
    v = torch.from_numpy(rng.standard_normal((n, 2))).to(cuda_device)
    grads = []
    for dm in (full, lean):
        rowptr, cols, w, tot, _, rec = dm.weights_csr(q, c, return_totals=True, return_summary=True,
                                                      keep_records=True)
        g = torch.ones(q.shape[0], 2, dtype=torch.float64, device=cuda_device)
        grads.append(dm.query_grad(q, v, g, c, rowptr, w, tot, records=rec))
    assert torch.equal(_bits(grads[0]), _bits(grads[1]))

    class One:
        def __init__(self, dm):
            self.device_mesh, self.centroid = dm, c

        def close(self):
            pass
    made = iter([One(full), One(lean), One(full)])
    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(nb, 'Interpolator', lambda *a, **k: next(made))
        batch = nb.BatchInterpolator([np.zeros((4, 3))] * 3, device=cuda_device, threads=1)
    out = batch.interpolate_device(q, batch.query_offsets([2000, 3000, 2001]), torch.cat([v, v, v]))
    assert torch.equal(_bits(out), _bits(full.interpolate(q, v, c)))
