"""The reference's three numba kernels as GPU drop-ins (covasim/utils.py:38-128).

Same names, arguments and return values as ``cv.compute_viral_load``,
``cv.compute_trans_sus`` and ``cv.compute_infections``. numpy inputs give
numpy outputs (copied through the device); torch CUDA tensors stay on the
device. They are also registered as torch custom ops ``covgpu::*``.
"""
import numpy as np
import torch

from . import _lib as L

__all__ = ['compute_viral_load', 'compute_trans_sus', 'compute_infections']

_F32, _I32, _U8, _F64 = torch.float32, torch.int32, torch.uint8, torch.float64


def _dev(x, dtype):
    if torch.is_tensor(x):
        return x.to(device='cuda', dtype=dtype).contiguous()
    return torch.from_numpy(np.ascontiguousarray(np.asarray(x), dtype=torch.empty(0, dtype=dtype).numpy().dtype)).cuda()


def _ptr(t):
    return t.data_ptr() if t is not None and t.numel() else None


def _raw_stream(x):
    try:
        return torch._C._cuda_getCurrentRawStream(x.get_device())
    except AttributeError:  # a private name: the public way takes a microsecond more
        return torch.cuda.current_stream(x.device).cuda_stream


def _direct(xs, dtypes, *ints):
    """May the library be called on these arguments without going through the
    operators below? Only when no torch mechanism could want to see the call
    (dispatch and function modes, functorch and forward-mode levels, tracing,
    compilation, profiling, gradients) and every argument is a plain contiguous
    tensor of the current device in one of its dtypes (and the integers fit the
    operators' int64). The operators' Python machinery takes about 30 us a call:
    the viral load of 20,000 agents took 45.7 us through them and takes 14.2 us.
    torch's own (private) names are asked; without one of them the answer is no."""
    if torch.compiler.is_compiling():  # first: constant under compilation, which knows none of the names below
        return False
    try:
        if (torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack() or
                torch._C._get_tracing_state() is not None or
                torch._C._functorch.peek_interpreter_stack() is not None or
                torch.autograd.forward_ad._current_level >= 0 or torch._C._autograd._profiler_enabled()):
            return False
        dev = torch._C._cuda_getDevice() if torch.cuda.is_initialized() else -1
    except AttributeError:
        return False
    for i in ints:
        if not -(1 << 63) <= i < 1 << 63:
            return False
    for x, dtype in zip(xs, dtypes):
        if (type(x) is not torch.Tensor or x.dtype not in dtype or not x.is_cuda or x.get_device() != dev or
                x.requires_grad or not x.is_contiguous() or x.is_neg()):
            return False
    return True


# ---------------------------------------------------------------- the library's calls
def _viral_load_call(t, time_start, time_recovered, time_dead, frac_time, load_ratio, high_cap):
    n = time_start.numel()
    out = torch.empty(n, dtype=_F32, device=time_start.device)
    L.call('covgpu_viral_load', int(t), _ptr(time_start), _ptr(time_recovered), _ptr(time_dead), n, float(frac_time),
           float(load_ratio), float(high_cap), _ptr(out), _raw_stream(out))
    return out


def _trans_sus_call(rel_trans, rel_sus, inf, sus, beta_layer, viral_load, symp, iso, quar, asymp_factor, iso_factor,
                    quar_factor, immunity_factors):
    n = rel_trans.numel()
    a = torch.empty(n, dtype=_F32, device=rel_trans.device)
    b = torch.empty(n, dtype=_F32, device=rel_trans.device)
    # the scalars are rounded to float32 by the C call, as the reference's signature casts them
    L.call('covgpu_trans_sus', _ptr(rel_trans), _ptr(rel_sus), _ptr(inf), _ptr(sus), float(beta_layer),
           _ptr(viral_load), _ptr(symp), _ptr(iso), _ptr(quar), float(asymp_factor), float(iso_factor),
           float(quar_factor), _ptr(immunity_factors), n, _ptr(a), _ptr(b), _raw_stream(a))
    return a, b


def _infections_call(beta, p1, p2, layer_betas, rel_trans, rel_sus, uniforms, seed, day, variant, layer):
    E = p1.numel()
    dev = p1.device
    if E == 0:
        return torch.empty(0, dtype=_I32, device=dev), torch.empty(0, dtype=_I32, device=dev)
    n_agents = min(rel_trans.numel(), rel_sus.numel())
    count = torch.empty(2, dtype=torch.int64, device=dev)  # transmissions, status
    nbytes = int(L.lib().covgpu_infections_scratch_bytes(E))
    scratch = torch.empty(nbytes, dtype=_U8, device=dev)
    L.call('covgpu_infections_find', float(beta), _ptr(p1), _ptr(p2), _ptr(layer_betas), E, _ptr(rel_trans),
           _ptr(rel_sus), n_agents, _ptr(uniforms), int(seed) & 0xFFFFFFFFFFFFFFFF, int(day), int(variant), int(layer),
           count.data_ptr(), scratch.data_ptr(), nbytes, _raw_stream(count))
    n, status = count.tolist()
    if status & L.BADARG:
        raise IndexError('compute_infections: an edge index is outside the agent arrays')
    src = torch.empty(n, dtype=_I32, device=dev)
    tgt = torch.empty(n, dtype=_I32, device=dev)
    L.call('covgpu_infections_emit', _ptr(p1), _ptr(p2), E, scratch.data_ptr(), n, _ptr(src), _ptr(tgt),
           _raw_stream(count))
    return src, tgt


# ---------------------------------------------------------------- torch custom ops
@torch.library.custom_op('covgpu::compute_viral_load', mutates_args=())
def _viral_load_op(t: int, time_start: torch.Tensor, time_recovered: torch.Tensor, time_dead: torch.Tensor,
                   frac_time: float, load_ratio: float, high_cap: float) -> torch.Tensor:
    return _viral_load_call(t, time_start, time_recovered, time_dead, frac_time, load_ratio, high_cap)


@torch.library.custom_op('covgpu::compute_trans_sus', mutates_args=())
def _trans_sus_op(rel_trans: torch.Tensor, rel_sus: torch.Tensor, inf: torch.Tensor, sus: torch.Tensor,
                  beta_layer: float, viral_load: torch.Tensor, symp: torch.Tensor, iso: torch.Tensor,
                  quar: torch.Tensor, asymp_factor: float, iso_factor: float, quar_factor: float,
                  immunity_factors: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    return _trans_sus_call(rel_trans, rel_sus, inf, sus, beta_layer, viral_load, symp, iso, quar, asymp_factor,
                           iso_factor, quar_factor, immunity_factors)


@torch.library.custom_op('covgpu::compute_infections', mutates_args=())
def _infections_op(beta: float, p1: torch.Tensor, p2: torch.Tensor, layer_betas: torch.Tensor,
                   rel_trans: torch.Tensor, rel_sus: torch.Tensor, uniforms: torch.Tensor, seed: int, day: int,
                   variant: int, layer: int) -> tuple[torch.Tensor, torch.Tensor]:
    return _infections_call(beta, p1, p2, layer_betas, rel_trans, rel_sus, uniforms, seed, day, variant, layer)


# ---------------------------------------------------------------- reference-signature drop-ins
_FLOATS, _BOOLS, _INTS = (_F32,), (torch.bool, _U8), (_I32,)


def compute_viral_load(t, time_start, time_recovered, time_dead, frac_time, load_ratio, high_cap):
    """utils.py:39-79."""
    if _direct((time_start, time_recovered, time_dead), (_FLOATS,) * 3, int(t)):
        return _viral_load_call(t, time_start, time_recovered, time_dead, frac_time, load_ratio, high_cap)
    as_np = not torch.is_tensor(time_start)
    out = torch.ops.covgpu.compute_viral_load(int(t), _dev(time_start, _F32), _dev(time_recovered, _F32),
                                              _dev(time_dead, _F32), float(frac_time), float(load_ratio),
                                              float(high_cap))
    return out.cpu().numpy() if as_np else out


_TRANS_SUS = (_FLOATS, _FLOATS, _BOOLS, _BOOLS, _FLOATS, _BOOLS, _BOOLS, _BOOLS, _FLOATS)


def compute_trans_sus(rel_trans, rel_sus, inf, sus, beta_layer, viral_load, symp, iso, quar, asymp_factor,
                      iso_factor, quar_factor, immunity_factors):
    """utils.py:82-90."""
    if _direct((rel_trans, rel_sus, inf, sus, viral_load, symp, iso, quar, immunity_factors), _TRANS_SUS):
        # the kernel reads booleans as bytes, so boolean tensors need no conversion
        return _trans_sus_call(rel_trans, rel_sus, inf, sus, beta_layer, viral_load, symp, iso, quar, asymp_factor,
                               iso_factor, quar_factor, immunity_factors)
    as_np = not torch.is_tensor(rel_trans)
    b = lambda x: _dev(x, _U8) if not torch.is_tensor(x) else x.to('cuda').to(_U8).contiguous()  # noqa: E731
    a, c = torch.ops.covgpu.compute_trans_sus(_dev(rel_trans, _F32), _dev(rel_sus, _F32), b(inf), b(sus),
                                              float(beta_layer), _dev(viral_load, _F32), b(symp), b(iso), b(quar),
                                              float(asymp_factor), float(iso_factor), float(quar_factor),
                                              _dev(immunity_factors, _F32))
    return (a.cpu().numpy(), c.cpu().numpy()) if as_np else (a, c)


_INFECTIONS = (_INTS, _INTS, _FLOATS, _FLOATS, _FLOATS)


def compute_infections(beta, p1, p2, layer_betas, rel_trans, rel_sus, legacy=False, uniforms=None, seed=0, day=0,
                       variant=0, layer=0):
    """utils.py:93-128 (non-legacy). Returns (sources, targets): direction p1->p2
    in edge order, then p2->p1. ``uniforms`` ([2, E] float64 draws by direction
    and edge) replays given draws; otherwise Bernoullis come from Philox keyed
    by (seed, day, variant, layer, edge)."""
    if legacy:
        raise NotImplementedError('the legacy (pre-3.1.1) transmission path is not supported on the GPU')
    if uniforms is None and _direct((p1, p2, layer_betas, rel_trans, rel_sus), _INFECTIONS, int(seed),
                                    int(day), int(variant), int(layer)):
        return _infections_call(beta, p1, p2, layer_betas, rel_trans, rel_sus, None, seed, day, variant, layer)
    as_np = not torch.is_tensor(p1)
    uni = _dev(uniforms, _F64) if uniforms is not None else torch.empty(0, dtype=_F64, device='cuda')
    src, tgt = torch.ops.covgpu.compute_infections(float(beta), _dev(p1, _I32), _dev(p2, _I32), _dev(layer_betas, _F32),
                                                   _dev(rel_trans, _F32), _dev(rel_sus, _F32), uni, int(seed),
                                                   int(day), int(variant), int(layer))
    return (src.cpu().numpy(), tgt.cpu().numpy()) if as_np else (src, tgt)
