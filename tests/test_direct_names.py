"""The straight calls ask torch by names of its own: without one of them, and while torch compiles,
a call goes through the operators."""
import pytest
import torch

from covasim_gb300 import utils

F32 = ((torch.float32,),)


@pytest.mark.parametrize('owner,name', [(torch._C, '_len_torch_dispatch_stack'), (torch._C, '_len_torch_function_stack'),
                                        (torch._C, '_get_tracing_state'), (torch._C._functorch, 'peek_interpreter_stack'),
                                        (torch.autograd.forward_ad, '_current_level'),
                                        (torch._C._autograd, '_profiler_enabled')])
def test_a_torch_without_one_of_the_names(monkeypatch, owner, name):
    x = torch.zeros(3)
    monkeypatch.delattr(owner, name)
    assert utils._direct((x,), F32, 5) is False


def test_compiled_callers_need_no_graph_break():
    f = torch.compile(lambda x: x + (1.0 if utils._direct((x,), F32, 5) else 2.0), backend='eager', fullgraph=True)
    assert f(torch.zeros(3)).tolist() == [2.0] * 3


@pytest.mark.gpu
def test_calls_on_the_current_stream_without_the_raw_name(monkeypatch):
    import covasim_gb300 as cv
    n = 1003
    args = (85, torch.full((n,), 80.0, device='cuda'), torch.full((n,), 95.0, device='cuda'),
            torch.full((n,), float('nan'), device='cuda'), 0.3, 2.0, 4.0)
    want = cv.compute_viral_load(*args)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        monkeypatch.delattr(torch._C, '_cuda_getCurrentRawStream')
        got = cv.compute_viral_load(*args)
        monkeypatch.undo()
    s.synchronize()
    assert torch.equal(got, want)
