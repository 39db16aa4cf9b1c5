"""compute_infections in one evaluation per edge (find, then emit) against the two-pass form."""
import ctypes as C

import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _inputs(n, E, frac, seed=3):
    g = torch.Generator(device='cuda').manual_seed(seed)
    r = lambda m: torch.rand(m, generator=g, device='cuda')  # noqa: E731
    p1 = torch.randint(0, n, (E,), generator=g, device='cuda', dtype=torch.int32)
    p2 = torch.randint(0, n, (E,), generator=g, device='cuda', dtype=torch.int32)
    return p1, p2, r(E), (r(n) < frac) * (0.2 + r(n)), (r(n) < 0.7) * (0.5 + r(n))


def _two_pass(beta, p1, p2, lb, rt, rs, seed, day):
    E = len(p1)
    out = torch.full((2, 2 * E), -1, dtype=torch.int32, device='cuda')
    count = torch.zeros(1, dtype=torch.int64, device='cuda')
    rc = L.lib().covgpu_infections_noalloc(
        beta, p1.data_ptr(), p2.data_ptr(), lb.data_ptr(), E, rt.data_ptr(), rs.data_ptr(), len(rt), None, seed, day,
        0, 0, out[0].data_ptr(), out[1].data_ptr(), 2 * E, count.data_ptr(), None,
        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == L.OK
    m = int(count)
    return out[0, :m], out[1, :m]


# sizes around a warp's round (128 edges) and a block's range, sparse and certain transmissions
@pytest.mark.parametrize('n,E', [(5, 1), (40, 127), (40, 129), (700, 304 * 128), (700, 304 * 128 + 1),
                                 (100_003, 20_011), (1_000_003, 400_001)])
@pytest.mark.parametrize('beta,frac', [(0.05, 0.15), (3.0, 1.0)])
def test_find_and_emit_match_two_passes(n, E, beta, frac):
    p1, p2, lb, rt, rs = _inputs(n, E, frac)
    want = _two_pass(beta, p1, p2, lb, rt, rs, 9, 4)
    got = cv.compute_infections(beta, p1, p2, lb, rt, rs, seed=9, day=4)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    if E > 130:  # lists off a 16-byte boundary
        want = _two_pass(beta, p1[1:], p2[1:], lb[1:], rt, rs, 9, 4)
        got = cv.compute_infections(beta, p1[1:], p2[1:], lb[1:], rt, rs, seed=9, day=4)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


# covgpu_infections at its scratch limits: the two-pass form's least, and find's
@pytest.mark.parametrize('scratch', ['two_pass', 'find'])
def test_infections_at_scratch_limits_and_capacity(scratch):
    n, E, beta = 3000, 10_007, 0.3
    p1, p2, lb, rt, rs = _inputs(n, E, 0.3)
    p1[77] = n  # outside: skipped and flagged
    lib = L.lib()
    nbytes = dict(two_pass=2 * ((E + 2047) // 2048) * 12 + 256, find=lib.covgpu_infections_scratch_bytes(E))[scratch]
    want = _two_pass(beta, p1, p2, lb, rt, rs, 2, 1)
    for cap in (2 * E, 100):
        out = torch.full((2, cap), -1, dtype=torch.int32, device='cuda')
        count = torch.full((1,), 7, dtype=torch.int64, device='cuda')
        status = torch.zeros(1, dtype=torch.int32, device='cuda')
        buf = torch.empty(nbytes, dtype=torch.uint8, device='cuda')
        args = (beta, p1.data_ptr(), p2.data_ptr(), lb.data_ptr(), E, rt.data_ptr(), rs.data_ptr(), n, None, 2, 1, 0,
                0, out[0].data_ptr(), out[1].data_ptr(), cap, count.data_ptr(), status.data_ptr(), buf.data_ptr())
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.covgpu_infections(*args, nbytes, stream) == L.OK
        m = min(int(count), cap)
        assert int(count) == len(want[0])
        assert int(status) == L.BADARG | (L.OVERFLOW if cap < int(count) else 0)
        assert torch.equal(out[0, :m], want[0][:m]) and torch.equal(out[1, :m], want[1][:m])
    with pytest.raises(IndexError):
        cv.compute_infections(beta, p1, p2, lb, rt, rs)
    assert lib.covgpu_infections(*args, 2 * ((E + 2047) // 2048) * 12 + 255, stream) == L.BADARG
