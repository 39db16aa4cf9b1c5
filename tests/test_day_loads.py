"""The arrays that the day's kernels write are read with plain loads: a kernel launched as a
dependent can be resident while its predecessor still writes them, and the read-only path
(__ldg, ld.global.nc, a restricted pointer) is for data that does not change while the kernel lives."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'covasim_gb300', 'csrc')
# written by a kernel of a day: agent, infect, testing, post and the likelihood's passes
WRITTEN = ('flags', 'vstate', 'rel_trans', 'n_infections', 'n_breakthroughs', 'peak_nab', 'nab', 't_nab_event', 'sus_imm',
           'symp_imm', 'sev_imm', 'dates', 'durs', 'viral_load', 'roles', 'claim', 'src_rec', 'tgt_rec', 'events',
           'event_count', 'log', 'log_count', 'status', 'trace_bits', 'contact_bits', 'pending_quar', 'trace_count',
           'res_int', 'res_var', 'res_fx', 'logq', 'w', 'll', 'g_ll', 'g_exp', 'expected')


def _calls(text, name):
    """The argument text of every call of ``name``."""
    for m in re.finditer(r'\b' + name + r'\(', text):
        depth, k = 1, m.end()
        while depth:
            depth += {'(': 1, ')': -1}.get(text[k], 0)
            k += 1
        yield text[m.end():k - 1]


@pytest.mark.parametrize('name', ['covgpu.cu', 'covgpu_testing.cu', 'covgpu_device.cuh', 'covgpu_dropin.cu'])
def test_written_arrays_are_not_read_as_constant(name):
    text, header = (re.sub(r'//[^\n]*', '', open(os.path.join(CSRC, f)).read()) for f in (name, 'covgpu_device.cuh'))
    helpers = [m.group(1) for m in re.finditer(r'(\w+)\([^()]*\)\s*{[^{}]*(?:ld\.global\.nc|__ldg)', header)]
    assert 'ld_stream_v4' in helpers
    read_only = [a for f in ('__ldg', *helpers) for a in _calls(text, f)]
    bad = [a for a in read_only if any(re.search(r'\b(st|K|sp)\.' + w + r'\b', a) for w in WRITTEN)]
    # the bitmaps and their views, under the names they are passed by
    bad += [a for a in read_only if re.match(r'(?:const uint32_t\* ?)?(roles|bits|g4)\b', a)]
    assert not bad, bad
    assert not re.findall(r'__restrict__ (?:roles|bits)\b', text)
    if name == 'covgpu.cu':  # the rule sees the loads there are
        assert sum('rp1' in a for a in read_only) >= 2 and 'ld_stream_v4(' in text
