"""The query gradient of every route a row can take -- common, general, wide (the
fused kernel) and large rows -- on a Qhull mesh, which needs no constructor of
natinterp3d's: from kept records, recomputed and called again the same bits, and
central differences of the interpolation; weights bit for bit against the oracle."""
import numpy as np
import pytest
import torch
from scipy.spatial import Delaunay

import natinterp3d_b200 as ni
from natinterp3d_b200.autograd import interpolate
from oracle import oracle

pytestmark = pytest.mark.gpu


def qhull_interpolator(keys):
    """Delaunay tets of the keys and a super-simplex in the packed layout: positive
    tets (orient3d of their vertices), face i's neighbour opposite vertex 3 - i."""
    c = keys.mean(axis=0)
    r = 40 * np.abs(keys - c).max()
    corners = r * np.array([[-1.0, -1, -1], [3, -1, -1], [-1, 3, -1], [-1, -1, 3]])
    v = np.concatenate([keys - c, corners])
    d = Delaunay(v)
    assert len(np.unique(d.simplices)) == len(v)
    p, opposite = d.simplices.copy(), d.neighbors.copy()
    negative = np.linalg.det(v[p[:, :3]] - v[p[:, 3:]]) < 0
    for x in (p, opposite):
        x[negative, :2] = x[negative, 1::-1]
    return ni.Interpolator.from_mesh(c, v, p, opposite[:, ::-1])


def _sphere(rng, centre, n):
    s = rng.standard_normal((n, 3))
    s /= np.linalg.norm(s, axis=1, keepdims=True)
    return centre + 0.09 * s * (1 + 1e-3 * rng.standard_normal((n, 1)))


CENTRES = {12: (0.2, 0.2, 0.2), 26: (0.2, 0.8, 0.2), 40: (0.8, 0.2, 0.2), 300: (0.8, 0.8, 0.8)}


@pytest.fixture(scope='module')
def case(cuda_device):
    rng = np.random.default_rng(17)
    keys = rng.uniform(0, 1, (1500, 3))
    for centre in CENTRES.values():  # holes of 0.1 around them, but for the spheres' keys
        keys = keys[np.linalg.norm(keys - centre, axis=1) > 0.12]
    keys = np.concatenate([keys] + [_sphere(rng, np.array(c), n) for n, c in CENTRES.items()])
    near = [np.array(c) + 0.03 * rng.uniform(-1, 1, (150, 3)) for c in CENTRES.values()]
    q = np.concatenate(near + [rng.uniform(0.1, 0.9, (600, 3)), keys[:30]])
    it = qhull_interpolator(keys)
    v = torch.from_numpy(rng.standard_normal((len(keys), 3))).to(cuda_device)
    return it, q, v, rng


def test_weights_equal_oracle_on_every_route(case):
    it, q, v, _ = case
    W = it.get_weights(q)
    ref, stats, _ = oracle.OracleMesh(*it.mesh_arrays).weights(q - it.centroid, with_stats=True)
    assert np.array_equal(W.indptr, ref.indptr) and np.array_equal(W.indices, ref.indices)
    assert np.array_equal(W.data.view(np.uint8), ref.data.view(np.uint8))
    s = it.device_mesh.last_summary
    assert s['rows_wide'] > 100 and s['rows_large'] > 100
    assert np.diff(W.indptr).max() > 200


@pytest.mark.parametrize('M', [1380, (1 << 20) + 2760])
@pytest.mark.parametrize('dt', [torch.float64, torch.float32])
def test_same_bits(case, cuda_device, M, dt):
    it, qn, v, rng = case
    dm = it.device_mesh
    qn = np.concatenate([qn, rng.uniform(0.05, 0.95, (150, 3))])
    assert len(qn) == 1380
    many = np.concatenate([qn, rng.uniform(0.05, 0.95, (M - 2 * len(qn), 3)), qn]) if M > len(qn) else qn
    q = torch.from_numpy(many).to(cuda_device, dt)
    g = torch.from_numpy(rng.standard_normal((M, 3))).to(cuda_device)
    rowptr, cols, w, totals, rec = dm.weights_csr(q, it.centroid, return_totals=True, keep_records=True)
    grads = [dm.query_grad(q, v, g, it.centroid, rowptr, w, totals, records=r) for r in (rec, rec, None, None)]
    assert all(torch.equal(grads[0], x) for x in grads[1:])
    assert bool(torch.isfinite(grads[0]).all())
    s = dm.last_summary
    assert s['rows_wide'] > 100 and s['rows_large'] > 100


def test_central_differences(case, cuda_device):
    it, qn, v, rng = case
    qn = qn[:1200]
    q = torch.from_numpy(qn).to(cuda_device).requires_grad_(True)
    g = torch.from_numpy(rng.standard_normal((len(qn), 3))).to(cuda_device)
    gq, = torch.autograd.grad(interpolate(it, q, v), q, g)
    h = 1e-6
    num = torch.empty_like(gq)
    for a in range(3):
        e = torch.zeros(3, dtype=torch.float64, device=cuda_device)
        e[a] = h
        num[:, a] = ((it.interpolate_device(q.detach() + e, v) -
                      it.interpolate_device(q.detach() - e, v)) * g).sum(1) / (2 * h)
    # h^2 / 6 times the third derivative (the weights vary over a key spacing, at
    # least 1e-2) and rounding, 1e-15 / 1e-6 times the values' sum: below 1e-6 of a
    # row's gradient, but where a step crosses a neighbour change
    err = (gq - num).abs().amax(1)
    scale = num.abs().amax(1) + num.abs().amax(1).median()
    for k in range(0, 600, 150):  # each kind of row by itself
        assert float((err / scale)[k:k + 150].quantile(0.95)) < 1e-6
    assert float((err / scale)[600:].quantile(0.95)) < 1e-6
