"""The transpose product's column sort at the edges of its digits and tiles:
bit for bit scipy's W.T @ x (columns summed in ascending row order)."""
import numpy as np
import pytest
import scipy.sparse
import torch

import natinterp3d_b200 as ni

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def mesh(cuda_device):
    keys = np.random.default_rng(0).uniform(0, 1, (40, 3))
    return ni.Interpolator(keys, constructor='gpu').device_mesh


@pytest.mark.parametrize('cols', [1, 2, 3, 255, 256, 257, 65536, 65537, 70001])
@pytest.mark.parametrize('rows,per', [(1, 1), (2047, 1), (2048, 1), (2049, 1), (700, 9), (5000, 17)])
def test_equals_scipy(cuda_device, mesh, cols, rows, per):
    rng = np.random.default_rng(cols + rows)
    n = min(per, cols)
    # each row's columns distinct, in no order; the last rows empty
    ind = np.stack([rng.permutation(cols)[:n] if cols < 300 else
                    rng.choice(cols, n, replace=False) for _ in range(rows)]).astype(np.int32)
    ptr = np.concatenate([np.arange(rows + 1) * n, [rows * n] * 3]).astype(np.int32)
    data = rng.standard_normal(rows * n)
    W = scipy.sparse.csr_matrix((data, ind.ravel(), ptr), shape=(rows + 3, cols))
    x = rng.standard_normal((rows + 3, 2))
    dev = cuda_device
    y = mesh.spmm_t(torch.from_numpy(ptr).to(dev), torch.from_numpy(ind.ravel()).to(dev),
                    torch.from_numpy(data).to(dev), torch.from_numpy(x).to(dev), cols)
    assert np.array_equal(y.cpu().numpy(), W.T @ x)
