"""Calls on a mesh without the table of corner terms need no more scratch than on
one with it, but for the terms of a short call; at the edges of the chunks that
this takes, and with records kept for the gradient, the same bits."""
import numpy as np
import pytest
import torch

from natinterp3d_b200 import _native as N
from natinterp3d_b200 import device as nd

pytestmark = pytest.mark.gpu

CUT = 1 << 16  # rows up to which a call is one chunk
TERMS = 48 * 32  # bytes of a row's corner terms


@pytest.fixture(scope='module')
def meshes(cuda_device):
    keys = np.random.default_rng(83).uniform(0, 1, (1500, 3))
    c = keys.mean(axis=0)
    packed, _ = nd.gpu_delaunay(keys - c)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(nd, '_room', lambda *a: 0)
        lean = nd.DeviceMesh(*packed, device=cuda_device)
    full = nd.DeviceMesh(*packed, device=cuda_device)
    assert lean.table_bytes == 0 < full.table_bytes
    return full, lean, c, len(keys)


@pytest.mark.parametrize('mode', [N.NIF_MODE_WEIGHTS, N.NIF_MODE_INTERP])
@pytest.mark.parametrize('M', [1, 1000, CUT, CUT + 1, 3 * CUT + 1, 1 << 20, 5_000_000])
def test_scratch(meshes, mode, M):
    full, lean, _, _ = meshes
    more = lean.workspace_bytes(M, mode) - full.workspace_bytes(M, mode)
    assert more <= TERMS * min(M, CUT) + 4096
    if M >= 1 << 20:  # a third of the rows' records and terms against all records
        assert more <= 4096


@pytest.mark.parametrize('M', [CUT - 1, CUT, CUT + 1, 2 * CUT + 1, 3 * CUT + 2, (1 << 20) + 3])
def test_chunk_edges(meshes, cuda_device, M):
    full, lean, c, n = meshes
    rng = np.random.default_rng(M)
    q = torch.from_numpy(rng.uniform(0.0, 1.0, (M, 3))).to(cuda_device)
    v = torch.from_numpy(rng.standard_normal((n, 2))).to(cuda_device)
    assert torch.equal(full.interpolate(q, v, c), lean.interpolate(q, v, c))
    g = torch.from_numpy(rng.standard_normal((M, 2))).to(cuda_device)
    grads = []
    for dm in (full, lean):
        rowptr, cols, w, tot, rec = dm.weights_csr(q, c, return_totals=True, keep_records=True)
        grads.append(dm.query_grad(q, v, g, c, rowptr, w, tot, records=rec))
        grads.append(dm.query_grad(q, v, g, c, rowptr, w, tot))
    assert all(torch.equal(grads[0], x) for x in grads[1:])
