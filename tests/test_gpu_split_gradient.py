"""Query gradients of split rows (the facet polygons of the query's cell), on
meshes built on the GPU: against central differences of the interpolation, the
same bits from kept records as from a new point location, call after call, and
rows on both sides of the general kernel's limits."""
import numpy as np
import pytest
import torch

import natinterp3d_b200 as ni
from natinterp3d_b200.autograd import interpolate

pytestmark = pytest.mark.gpu


def _keys(kind, rng):
    if kind == 'sphere':  # many neighbours: the general kernel's rows
        s = rng.standard_normal((60, 3))
        s /= np.linalg.norm(s, axis=1, keepdims=True)
        return np.concatenate([s * (1 + 1e-2 * rng.standard_normal((60, 1))),
                               rng.uniform(-3, 3, (400, 3))])
    return rng.uniform(0, 1, (2000, 3))


@pytest.mark.parametrize('kind', ['uniform', 'sphere'])
@pytest.mark.parametrize('D', [1, 5])
def test_against_central_differences(cuda_device, kind, D):
    rng = np.random.default_rng(81)
    keys = _keys(kind, rng)
    it = ni.Interpolator(keys, constructor='gpu')
    c, ext = keys.mean(0), keys.max(0) - keys.min(0)
    qn = c + rng.uniform(-0.3, 0.3, (400, 3)) * ext * (0.3 if kind == 'sphere' else 1.0)
    v = torch.from_numpy(rng.standard_normal((len(keys), D))).to(cuda_device)
    g = torch.from_numpy(rng.standard_normal((400, D))).to(cuda_device)
    q = torch.from_numpy(qn).to(cuda_device).requires_grad_(True)
    gq, = torch.autograd.grad(interpolate(it, q, v), q, g)
    h = 1e-6 * float(ext.max())
    num = torch.empty_like(gq)
    for a in range(3):
        e = torch.zeros(3, dtype=torch.float64, device=cuda_device)
        e[a] = h
        num[:, a] = ((it.interpolate_device(q.detach() + e, v) -
                      it.interpolate_device(q.detach() - e, v)) * g).sum(1) / (2 * h)
    # h^2 / 6 times the third derivative (the weights vary over a key spacing,
    # at least 1e-2 ext) and rounding, 1e-15 / 1e-6: below 1e-6 of the scale of
    # a row's gradient, save where a step crosses a neighbour change (a jump in
    # the second derivative: h over the spacing)
    err = (gq - num).abs().amax(1)
    scale = num.abs().amax(1) + num.abs().amax(1).median()
    assert float((err / scale).max()) < 1e-3
    assert float((err / scale).quantile(0.98)) < 1e-6


@pytest.mark.parametrize('kind', ['uniform', 'sphere'])
def test_same_bits_from_records_and_again(cuda_device, kind):
    rng = np.random.default_rng(82)
    keys = _keys(kind, rng)
    it = ni.Interpolator(keys, constructor='gpu')
    dm = it.device_mesh
    q = torch.from_numpy(np.concatenate([
        rng.uniform(keys.min(0), keys.max(0), (3000, 3)), keys[:50],
        keys.mean(0) + 0.01 * rng.standard_normal((200, 3))])).to(cuda_device)
    v = torch.from_numpy(rng.standard_normal((len(keys), 3))).to(cuda_device)
    g = torch.from_numpy(rng.standard_normal((q.shape[0], 3))).to(cuda_device)
    rowptr, cols, vals, totals, rec = dm.weights_csr(q, it.centroid, return_totals=True,
                                                     keep_records=True)
    first = dm.query_grad(q, v, g, it.centroid, rowptr, vals, totals, records=rec)
    for records in (rec, None, None):
        again = dm.query_grad(q, v, g, it.centroid, rowptr, vals, totals, records=records)
        assert torch.equal(first, again)
    assert bool((first[3000:3050] == 0).all())  # on keys: no derivative
