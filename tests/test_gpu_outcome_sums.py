"""mean_infectious_duration on tensors that the kernel cannot take as they are: it reads its three
arrays to the first one's length."""
import pytest
import torch

from covasim_gb300 import _lib as L
from covasim_gb300.sim import mean_infectious_duration

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('sizes', [(8, 7, 8), (8, 8, 7), (8, 1, 8), (7, 8, 8), (8, 0, 8)])
def test_arrays_of_different_lengths_are_refused(monkeypatch, sizes):
    launched = []
    monkeypatch.setattr(L, 'call', lambda *a: launched.append(a))
    with pytest.raises((IndexError, RuntimeError)):
        mean_infectious_duration(*(torch.arange(float(n), device='cuda') for n in sizes))
    assert not launched


def test_negative_and_strided_views():
    x = torch.arange(20.0, device='cuda')
    rec, dead, inf = x[::2] + 7, torch.full((10,), float('nan'), device='cuda'), x[::2]
    want = mean_infectious_duration(rec.contiguous(), dead, inf.contiguous())
    assert want == 7.0
    assert mean_infectious_duration(torch._neg_view(-rec), dead, torch._neg_view(-inf)) == want
    assert mean_infectious_duration((x + 7)[::2], dead, x[::2]) == want
