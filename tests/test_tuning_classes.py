"""Calls of up to IDENTITY_ROWS queries are not bucketed: the tuner tries and
keeps no bucket resolution for them, and finds none that other calls' keys hold."""
import os
import re

import pytest
import torch

from natinterp3d_b200 import tuning

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_limit_is_the_librarys():
    with open(os.path.join(ROOT, 'natinterp3d_b200', 'csrc', 'nif_cuda.cu')) as f:
        assert re.search(r'constexpr int64_t IDENTITY_ROWS = (\d+);', f.read()).group(1) == \
            str(tuning.IDENTITY_ROWS)


class _Mesh:
    device = torch.device('cpu')

    def get_tuning(self):
        return {}


class _Interp:
    n_keys, predicates, device_mesh = 1000, 'fast', _Mesh()

    def __init__(self):
        self.set = []

    def set_tuning(self, t):
        self.set.append(t)

    def interpolate_device(self, q, v, check=True):
        return q


@pytest.fixture
def tuned(tmp_path, monkeypatch):
    monkeypatch.setenv('NATINTERP3D_B200_TUNING', str(tmp_path / 'tuning.json'))
    monkeypatch.setattr(torch.cuda, 'get_device_name', lambda d: 'gpu')
    monkeypatch.setattr(torch.cuda, 'device', lambda d: torch.no_grad())
    monkeypatch.setattr(torch.cuda, 'synchronize', lambda *a: None)
    # the bucket resolution of 1 seems the fastest, by chance
    monkeypatch.setattr(tuning, '_time', lambda run, reps: 2.0 - it.set[-1]['bucket_shift'])
    it = _Interp()

    def tune(M, **k):
        it.set = []
        return tuning.tune(it, torch.zeros(M, 3), torch.zeros(1000), **k)
    return tune


@pytest.mark.parametrize('M', [1, 64, 12_000, 16_384])
def test_small_calls_keep_the_default_resolution(tuned, M):
    rep = tuned(M)
    assert rep['tuning']['bucket_shift'] == 0 and len(rep['times_ms']) == 6


def test_neither_side_reads_the_other(tuned):
    assert tuned(12_000)['cached'] is False
    rep = tuned(20_000)
    assert rep['cached'] is False and rep['tuning']['bucket_shift'] == 1
    assert tuned(16_385)['cached'] is True
    rep = tuned(16_384)
    assert rep['cached'] is True and rep['tuning']['bucket_shift'] == 0


def test_small_sample_of_a_large_call(tuned):
    assert tuned(100_000, max_queries=5_000)['tuning']['bucket_shift'] == 0


def test_kept_entry_with_a_resolution_is_measured_again(tuned):
    tuning._store_cache('gpu|interpolate|k2^10|q2^12|float32|float32/D1|fast',
                        {'tuning': {'blocks_per_sm': 8, 'tile': 8, 'bucket_shift': -1}})
    rep = tuned(4_000)
    assert rep['cached'] is False and rep['tuning']['bucket_shift'] == 0
