"""Rows at the limits of the split row kernels, bit for bit against the oracle.

The common volume kernel takes rows of at most 32 neighbours and 42 boundary
faces, a general one the rest, and the tets whose triangles fall below
natinterp3d's degeneracy thresholds (1e-30) too; meshes are built on the GPU, and
the oracle runs on the same mesh."""
import numpy as np
import pytest
import torch

import natinterp3d_b200 as ni
from oracle import oracle

pytestmark = pytest.mark.gpu


def _keys(kind, rng):
    if kind == 'sphere':  # a query near the centre has most keys for neighbours
        s = rng.standard_normal((60, 3))
        s /= np.linalg.norm(s, axis=1, keepdims=True)
        return np.concatenate([s * (1 + 1e-4 * rng.standard_normal((60, 1))),
                               rng.uniform(-3, 3, (400, 3))])
    if kind == 'clusters':
        c = rng.uniform(0, 1, (6, 3))
        return c[rng.integers(0, 6, 4000)] + np.exp(rng.uniform(-7, -2, (4000, 1))) * \
            rng.standard_normal((4000, 3))
    if kind == 'flat':
        return rng.uniform(0, 1, (2000, 3)) * [1, 1, 1e-3]
    scale = {'five': 1.0, 'uniform': 1.0, 'micro': 1e-6, 'nano': 1e-9, 'mega': 1e8}[kind]
    return rng.uniform(0, scale, (5 if kind == 'five' else 1500, 3))


def _case(kind):
    rng = np.random.default_rng(71)
    keys = _keys(kind, rng)
    it = ni.Interpolator(keys, constructor='gpu')
    assert it.construction['constructor'] == 'gpu'
    lo, hi = keys.min(0), keys.max(0)
    ext = hi - lo
    q = np.concatenate([
        rng.uniform(lo - 0.05 * ext, hi + 0.05 * ext, (1500, 3)),
        rng.uniform(lo - 40 * ext, hi + 40 * ext, (60, 3)),      # some outside the super-simplex
        keys[rng.integers(0, len(keys), 100)],                   # exactly on keys
        keys.mean(0) + 0.02 * ext * rng.standard_normal((300, 3)),
    ])
    return it, keys, q, rng


KINDS = ['uniform', 'five', 'sphere', 'clusters', 'flat', 'micro', 'nano', 'mega']


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('mode', ['fast', 'audit', 'exact'])
def test_weights_equal_oracle(cuda_device, kind, mode):
    it, keys, q, _ = _case(kind)
    it.set_predicates(mode)
    W = it.get_weights(q)
    om = oracle.OracleMesh(*it.mesh_arrays)
    om.set_predicates(mode)
    ref, stats, _ = om.weights(q - it.centroid, with_stats=True)
    assert np.array_equal(W.indptr, ref.indptr) and np.array_equal(W.indices, ref.indices)
    assert np.array_equal(W.data.view(np.uint8), ref.data.view(np.uint8))
    if mode != 'fast':  # the sphere tests that the cached spheres decide are certified ones
        got = it.predicate_stats
        assert got['insphere_uncertain'] == stats['insphere_uncertain']
        assert got['insphere_flipped'] == stats['insphere_flipped']


@pytest.mark.parametrize('kind', ['sphere', 'clusters', 'nano'])
@pytest.mark.parametrize('D', [1, 4, 5, 8, 9, 33])
def test_interpolation_equals_weights_times_values(cuda_device, kind, D):
    it, keys, q, rng = _case(kind)
    v = rng.standard_normal((len(keys), D))
    W = oracle.OracleMesh(*it.mesh_arrays).weights(q - it.centroid)
    assert np.array_equal(it.interpolate(q, v), W @ v)
    # float32 queries: natinterp3d casts the weights and sorts the columns
    q32, v32 = q.astype(np.float32), v.astype(np.float32)
    W32 = oracle.OracleMesh(*it.mesh_arrays).weights(q32.astype(np.float64) - it.centroid)
    W32 = W32.astype(np.float32)
    W32.sort_indices()
    assert np.array_equal(it.interpolate(q32, v32), W32 @ v32)


@pytest.mark.parametrize('M', [1, 63, 4096, 16384, 16385, 16400])
def test_row_order_does_not_matter(cuda_device, M):
    """Calls of up to 16,384 rows run as they come, larger ones by bucket: the
    same rows have the same bits in one call and in two."""
    rng = np.random.default_rng(72)
    it = ni.Interpolator(rng.uniform(0, 1, (3000, 3)), constructor='gpu')
    q = rng.uniform(-0.02, 1.02, (M, 3))
    v = rng.standard_normal((3000, 2))
    whole = it.interpolate(q, v)
    cut = M // 3
    parts = [it.interpolate(p, v) for p in (q[:cut], q[cut:]) if len(p)]
    assert np.array_equal(whole.view(np.uint8), np.concatenate(parts).view(np.uint8))
    W = it.get_weights(q)
    assert np.array_equal(W @ v, whole)
