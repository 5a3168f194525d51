"""Device memory and the table of corner terms: a mesh takes it only where
enough memory stays free, so that the mesh, the uploads beside it and the calls
on it run wherever they run without it."""
import numpy as np
import pytest
import torch

from natinterp3d_b200 import device as nd

GB = 1 << 30


def test_rule():
    fits = nd._table_fits
    assert fits(3 * GB, 170 * GB, 0)
    assert not fits(3 * GB, 6 * GB, 0)             # too little left for a call's workspace
    assert not fits(GB // 4, 4 * GB, 0)
    assert fits(25 * GB, 100 * GB, 0) and not fits(26 * GB, 100 * GB, 0)
    # many meshes of 2 GB with tables of 4: a quarter at most, and all meshes still fit
    room, held, meshes = 178 * GB, 0, 0
    while room >= 2 * GB:
        room -= 2 * GB
        meshes += 1
        if fits(4 * GB, room, held):
            room, held = room - 4 * GB, held + 4 * GB
    assert held <= 178 * GB // 4 and meshes >= 178 // 2 * 3 // 4


def test_room_is_measured_once_and_kept_up(monkeypatch):
    """The free memory is asked for once a second; what the process's allocator
    takes and gives back, and its limit, are followed without."""
    clock = [100.0]
    monkeypatch.setattr(nd.time, 'monotonic', lambda: clock[0])
    now = {'free': 90 * GB, 'reserved': 10 * GB, 'used': 4 * GB, 'share': 1.0, 'asked': 0}

    def info(device):
        now['asked'] += 1
        return now['free'], 100 * GB
    monkeypatch.setattr(torch.cuda, 'mem_get_info', info)
    monkeypatch.setattr(torch.cuda, 'get_per_process_memory_fraction', lambda d: now['share'])
    monkeypatch.setattr(torch.cuda, 'memory_stats_as_nested_dict', lambda d: {
        'allocated_bytes': {'all': {'current': now['used']}},
        'reserved_bytes': {'all': {'current': now['reserved']}}})
    monkeypatch.setattr(nd, '_all_free', {})
    assert nd._room('d', False) == 96 * GB
    now.update(free=70 * GB, reserved=30 * GB, used=28 * GB)
    assert nd._room('d', False) == 72 * GB and now['asked'] == 1
    now.update(free=20 * GB)  # someone else took 50 GB
    assert nd._room('d', False) == 72 * GB and nd._room('d') == nd._room('d', False) == 22 * GB
    now.update(share=0.4)
    assert nd._room('d', False) == 12 * GB and now['asked'] == 2
    now.update(free=30 * GB, share=1.0)
    clock[0] += 1.5
    assert nd._room('d', False) == 32 * GB and now['asked'] == 3

    def none(device):
        raise RuntimeError
    monkeypatch.setattr(torch.cuda, 'memory_stats_as_nested_dict', none)
    assert nd._room('d', False) == 30 * GB


@pytest.fixture(scope='module')
def mesh(cuda_device):
    keys = np.random.default_rng(91).uniform(0, 1, (60_000, 3))
    c = keys.mean(axis=0)
    packed, _ = nd.gpu_delaunay(keys - c)
    return tuple(x.cpu().numpy() for x in packed), c, len(keys)


@pytest.mark.gpu
def test_upload_without_room_takes_the_mesh_without_table(mesh, cuda_device, monkeypatch):
    packed, c, n = mesh
    upload, refused = torch.from_numpy, []

    def refuse_once(x):
        if not refused:
            refused.append(1)
            raise torch.cuda.OutOfMemoryError('no room')
        return upload(x)
    with monkeypatch.context() as m:
        m.setattr(nd.torch, 'from_numpy', refuse_once)
        lean = nd.DeviceMesh(*packed, device=cuda_device)
    assert refused and lean.table_bytes == 0
    full = nd.DeviceMesh(*packed, device=cuda_device)
    assert full.nbytes - lean.nbytes == full.table_bytes == 512 * len(packed[1])
    q = torch.from_numpy(np.random.default_rng(1).uniform(0.1, 0.9, (5000, 3))).to(cuda_device)
    v = torch.from_numpy(np.random.default_rng(2).standard_normal((n, 2))).to(cuda_device)
    assert torch.equal(full.interpolate(q, v, c), lean.interpolate(q, v, c))


@pytest.mark.gpu
def test_calls_fit_where_the_mesh_just_fits(mesh, cuda_device):
    """A process limit that holds the mesh with its table and the uploads, but no
    call beside them: the mesh without the table leaves the call its room."""
    packed, c, n = mesh
    M = 40_000
    q = torch.from_numpy(np.random.default_rng(1).uniform(0.1, 0.9, (M, 3))).to(cuda_device)
    v = torch.from_numpy(np.random.default_rng(2).standard_normal((n, 2))).to(cuda_device)
    full = nd.DeviceMesh(*packed, device=cuda_device)
    expect = full.interpolate(q, v, c)
    nbytes = full.nbytes
    del full
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    uploads = 24 * len(packed[0]) + 32 * len(packed[1])
    total = torch.cuda.mem_get_info(cuda_device)[1]
    limit = torch.cuda.memory_reserved(cuda_device) + nbytes + uploads + (16 << 20)
    torch.cuda.set_per_process_memory_fraction(limit / total, cuda_device)
    try:
        dm = nd.DeviceMesh(*packed, device=cuda_device)
        assert dm.nbytes < nbytes
        assert torch.equal(dm.interpolate(q, v, c), expect)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, cuda_device)
