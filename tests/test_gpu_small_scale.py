"""Keys so close that triangles of the rows' virtual tets fall below natinterp3d's
threshold (twice the area 1e-15): rows around a tet of a squared radius below
4e-15 go to the general kernel straight away, the others through the common one.
Weights bit for bit against the oracle on both sides of that size and on meshes
with rows of both kinds; gradients (facets, and dual numbers where natinterp3d's
fallbacks are met) against central differences, and the same bits from kept
records as from a new search."""
import numpy as np
import pytest
import torch

import natinterp3d_b200 as ni
from natinterp3d_b200.autograd import interpolate
from oracle import oracle

pytestmark = pytest.mark.gpu


def _case(kind):
    rng = np.random.default_rng(93)
    if kind == 'mixed':  # a cluster of keys some 1e-7 apart in a cloud some 0.1 apart
        keys = np.concatenate([rng.uniform(0, 1, (1000, 3)), 0.5 + 5e-7 * rng.standard_normal((600, 3))])
        q = np.concatenate([rng.uniform(0.05, 0.95, (600, 3)), 0.5 + 4e-7 * rng.standard_normal((900, 3))])
    else:
        keys = rng.uniform(0, kind, (2500, 3))
        q = np.concatenate([rng.uniform(0.1 * kind, 0.9 * kind, (1500, 3)), keys[:40]])
    it = ni.Interpolator(keys, constructor='gpu')
    assert it.construction['constructor'] == 'gpu'
    return it, keys, q, rng


KINDS = [4e-6, 1e-6, 5e-7, 1e-7, 1e-8, 1e-9, 'mixed']


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('mode', ['fast', 'exact'])
def test_weights_equal_oracle(cuda_device, kind, mode):
    it, keys, q, rng = _case(kind)
    it.set_predicates(mode)
    W = it.get_weights(q)
    om = oracle.OracleMesh(*it.mesh_arrays)
    om.set_predicates(mode)
    ref = om.weights(q - it.centroid)
    assert np.array_equal(W.indptr, ref.indptr) and np.array_equal(W.indices, ref.indices)
    assert np.array_equal(W.data.view(np.uint8), ref.data.view(np.uint8))
    v = rng.standard_normal((len(keys), 3))
    assert np.array_equal(it.interpolate(q, v), W @ v)


@pytest.mark.parametrize('kind', KINDS)
def test_gradient(cuda_device, kind):
    it, keys, qn, rng = _case(kind)
    dm = it.device_mesh
    v = torch.from_numpy(rng.standard_normal((len(keys), 2))).to(cuda_device)
    g = torch.from_numpy(rng.standard_normal((len(qn), 2))).to(cuda_device)
    q = torch.from_numpy(qn).to(cuda_device).requires_grad_(True)
    gq, = torch.autograd.grad(interpolate(it, q, v), q, g)
    q = q.detach()
    rowptr, cols, vals, totals, rec = dm.weights_csr(q, it.centroid, return_totals=True, keep_records=True)
    for records in (rec, None):
        assert torch.equal(gq, dm.query_grad(q, v, g, it.centroid, rowptr, vals, totals, records=records))
    if kind == 'mixed':
        h = torch.where((q - 0.5).abs().amax(1) < 1e-5, 1e-13, 1e-6)
    else:
        h = torch.full((len(qn),), 1e-6 * kind, dtype=torch.float64, device=cuda_device)
    num = torch.empty_like(gq)
    for a in range(3):
        e = torch.zeros_like(q)
        e[:, a] = h
        lo, hi = q - e, q + e  # the steps that are taken, as rounded
        num[:, a] = ((it.interpolate_device(hi, v) - it.interpolate_device(lo, v)) * g).sum(1) / \
            (hi[:, a] - lo[:, a])
    rows = slice(0, len(qn) - 40) if kind != 'mixed' else slice(0, 600)
    # as for unit keys: h^2 / 6 times the third derivative, and rounding, 1e-15 / 1e-6,
    # below 1e-6 of a row's gradient but where a step crosses a neighbour change or one
    # of natinterp3d's thresholds.  (In the cluster of 'mixed' a step is a thousand ulp
    # of the coordinates: its rows are compared by the bits above alone.)
    err = (gq - num)[rows].abs().amax(1)
    scale = num[rows].abs().amax(1) + num[rows].abs().amax(1).median()
    assert float((err - 1e-6 * scale).quantile(0.95)) <= 0.0
