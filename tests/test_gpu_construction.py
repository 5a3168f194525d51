"""The GPU constructor's rounds on key sets of general position, against the
definition: every key is used, and no vertex lies in a tet's circumsphere
(brute force in exact arithmetic where rounding does not decide)."""
from fractions import Fraction

import numpy as np
import pytest

import natinterp3d_b200 as ni

pytestmark = pytest.mark.gpu


def _insphere(p):
    """Sign of the lifted determinant of 5 points (exact), positive inside for a
    positively oriented tet."""
    rows = [[Fraction(float(x)) for x in r] for r in p]
    e = rows[4]
    m = []
    for r in rows[:4]:
        d = [r[k] - e[k] for k in range(3)]
        m.append(d + [sum(x * x for x in d)])
    det = Fraction(1)
    for k in range(4):
        pivot = next((i for i in range(k, 4) if m[i][k] != 0), None)
        if pivot is None:
            return 0
        if pivot != k:
            m[k], m[pivot] = m[pivot], m[k]
            det = -det
        det *= m[k][k]
        for i in range(k + 1, 4):
            f = m[i][k] / m[k][k]
            m[i] = [m[i][j] - f * m[k][j] for j in range(4)]
    return (det > 0) - (det < 0)


@pytest.mark.parametrize('kind,n', [('uniform', 5), ('uniform', 33), ('uniform', 300), ('flat', 200),
                                    ('clusters', 300), ('line', 120)])
def test_delaunay_by_definition(cuda_device, kind, n):
    rng = np.random.default_rng(91)
    keys = rng.uniform(0, 1, (n, 3))
    if kind == 'flat':
        keys *= [1, 1, 1e-3]
    elif kind == 'clusters':
        keys = keys[rng.integers(0, 6, n)] + 1e-4 * rng.standard_normal((n, 3))
    elif kind == 'line':
        t = np.sort(rng.uniform(0, 1, n))
        keys = np.stack([t, t, t], 1) + 0.02 * rng.standard_normal((n, 3))
    it = ni.Interpolator(keys, constructor='gpu')
    c = it.construction
    assert c['constructor'] == 'gpu'
    assert c['bad_orientation'] == 0 and c['bad_adjacency'] == 0 and c['non_delaunay_faces'] == 0
    v, tv, _ = it.mesh_arrays
    assert np.array_equal(np.unique(tv), np.arange(n + 4))
    # rounded determinants of every tet against every vertex; near zero exactly
    P = v[tv]
    for i in range(n + 4):
        d = P - v[i]
        m = np.concatenate([d, (d * d).sum(2, keepdims=True)], 2)
        det = np.linalg.det(m)
        scale = np.prod(np.abs(m).sum(2), 1)
        orient = np.sign(np.linalg.det(P[:, :3] - P[:, 3:]))
        other = (tv != i).all(1)
        assert not (other & (det * orient > 1e-9 * scale)).any()
        for t in np.flatnonzero(other & (np.abs(det) <= 1e-9 * scale))[:2]:
            assert _insphere(np.concatenate([P[t], v[i:i + 1]])) * orient[t] <= 0


def test_many_keys_in_few_tets_and_duplicates(cuda_device):
    """All keys start in one tet; a duplicate key is refused after some rounds."""
    rng = np.random.default_rng(92)
    keys = rng.standard_normal((20_000, 3)) * 1e-3
    it = ni.Interpolator(keys, constructor='gpu')
    assert it.construction['constructor'] == 'gpu' and it.construction['rounds'] < 2000
    from natinterp3d_b200.device import GPUConstructionError, gpu_delaunay
    with pytest.raises(GPUConstructionError):
        gpu_delaunay(np.concatenate([keys[:500], keys[:1]]))
