"""covgpu_version moves with the layout of the structures that callers fill."""
import ctypes as C

from covasim_gb300 import _lib as L

# version: sizes of sim_params, layer, agent_block, event, log_rec, state, testing, lik, span
LAYOUTS = {
    1: (2040, 112, 24, 16, 16, 512, 568, 72, None),
    2: (2208, 120, 24, 16, 16, 512, 568, 72, 32),
}


def test_version_of_the_present_layout():
    sizes = (C.sizeof(L.SimParams), C.sizeof(L.Layer), C.sizeof(L.AgentBlock), 16, 16, C.sizeof(L.State),
             C.sizeof(L.Testing), C.sizeof(L.Lik), C.sizeof(L.Span))
    version = L.lib().covgpu_version()
    assert version == L.ABI_VERSION
    assert LAYOUTS.get(version) == sizes, f'a changed layout takes the next version: {sizes}'
