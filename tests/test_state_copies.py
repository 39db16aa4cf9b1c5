"""What a state's one-launch copies may take (BatchState._spans): plain copies between arrays of
the state's device, each array written once; everything else goes through copy_, in order."""
from types import SimpleNamespace

import pytest
import torch

from covasim_gb300 import _lib as L
from covasim_gb300 import state as S


@pytest.fixture
def launched(monkeypatch):
    """The spans of the launches, as (destination, source, bytes, fill); nothing runs."""
    out = []
    monkeypatch.setattr(S.L, 'call', lambda name, spans, n, stream: out.extend(
        (s.dst, s.src, s.bytes, s.fill) for s in spans[:n]))
    monkeypatch.setattr(S, '_stream', lambda: None)
    return out


STATE = SimpleNamespace(res_all=torch.zeros(1))  # a state whose arrays are where the test's are


def spans(*args):
    S.BatchState._spans(STATE, *args)


def test_plain_copies_and_fills_are_launched(launched):
    a, b, c = torch.zeros(7), torch.arange(7.0), torch.zeros(3, dtype=torch.int64)
    spans([(a, b)], [c], [b[:0]])
    assert sorted(launched, key=lambda s: s[2]) == [(b[:0].data_ptr() or None, None, 0, 0xFF), (c.data_ptr(), None, 24, 0),
                                                    (a.data_ptr(), b.data_ptr(), 28, 0)]


@pytest.mark.parametrize('dst', ['another device', 'negative view', 'strided', 'subclass'])
def test_destinations_that_are_not_plain_arrays_of_the_device(launched, dst):
    """E.g. a checkpoint whose buffers were moved to host memory: a launch would write the
    device's bytes through a pointer of another device."""
    x = torch.zeros(8)
    d = {'another device': torch.empty(4, device='meta'), 'negative view': torch._neg_view(x[:4]), 'strided': x[::2],
         'subclass': torch.nn.Parameter(x[:4].clone(), requires_grad=False)}[dst]
    spans([(d, torch.arange(4.0))])
    assert not launched
    if dst != 'another device':
        assert d.tolist() == [0, 1, 2, 3]


def test_negative_view_as_a_source(launched):
    d = torch.zeros(4)
    spans([(d, torch._neg_view(torch.arange(4.0)))])
    assert not launched and d.tolist() == [0, -1, -2, -3]


def test_an_array_that_is_copied_and_then_cleared(launched):
    """Blocks of one launch run in any order: of the two writes only the last one may be in it."""
    d, e = torch.ones(4), torch.ones(4)
    spans([(d, torch.arange(4.0)), (e, torch.arange(4.0))], [d])
    assert [s[0] for s in launched].count(d.data_ptr()) == 1
    assert (d.data_ptr(), None, 16, 0) in launched and len(launched) == 2


def test_copies_among_the_destinations_themselves(launched):
    """b's old values go to a before b is overwritten, in the order of the pairs."""
    a, b, c = torch.zeros(4), torch.arange(4.0), torch.full((4,), 9.0)
    spans([(a, b), (b, c)])
    assert not launched and a.tolist() == [0, 1, 2, 3] and b.tolist() == [9] * 4
