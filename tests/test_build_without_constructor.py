"""Without natinterp3d's sources and without a prebuilt constructor the CUDA
library is still built, and the host constructor alone raises."""
import os
import sys

import numpy as np
import pytest

from natinterp3d_b200 import _build, _native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


@pytest.fixture
def bare(tmp_path, monkeypatch):
    monkeypatch.setenv('NATINTERP3D_SRC', str(tmp_path))
    monkeypatch.setattr(_build, 'MESH_SO', str(tmp_path / 'libnif_mesh.so'))
    monkeypatch.setattr(_native, '_mesh_lib', None)
    built = []
    monkeypatch.setattr(_build, 'build_cuda_lib', lambda force=False: built.append(force))
    return built


def test_cuda_library_is_built(bare, capsys):
    assert not _build.have_mesh_lib()
    assert _build.build() is False
    assert bare == [False] and 'not built' in capsys.readouterr().err


def test_entry_point(bare, monkeypatch):
    import __graft_entry__ as entry
    monkeypatch.setattr(_native, 'cuda_lib', lambda: None)
    entry.build()
    assert bare == [False]


def test_host_constructor_raises(bare):
    with pytest.raises(RuntimeError, match='constructor sources not found'):
        _native.HostMesh(np.zeros((5, 3)))


def test_prebuilt_constructor_is_used(bare, tmp_path):
    (tmp_path / 'libnif_mesh.so').write_bytes(b'')
    assert _build.have_mesh_lib() and _build.build() is True
