"""Rules of the device sources that keep memory accesses in their order, read off the text:
a compiler may move what it is not told about, and no run shows whether it will."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'boast-lig_gb300', 'csrc')
SOURCES = sorted(glob.glob(os.path.join(CSRC, '*.cu')) + glob.glob(os.path.join(CSRC, '*.cuh')))


def asm_statements(path):
    """(volatile, text) of every inline assembly statement."""
    text = open(path).read()
    for m in re.finditer(r'\basm\s*(volatile)?\s*\(', text):
        depth, i = 1, m.end()
        quoted = False
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != '\\':
                quoted = not quoted
            elif not quoted:
                depth += (c == '(') - (c == ')')
            i += 1
        yield m.group(1) is not None, text[m.end():i - 1]


@pytest.mark.parametrize('path', SOURCES, ids=os.path.basename)
def test_memory_instructions_are_ordered(path):
    """What reads or writes memory, barriers or tensor memory is volatile and clobbers memory:
    otherwise a load's result is a function of its address to the compiler, which may move it
    across a wait or a store."""
    for volatile, text in asm_statements(path):
        if re.search(r'\b(ld|st|red|atom|cp\.async|mbarrier|tcgen05\.(ld|mma|commit))\b', text):
            assert volatile and '"memory"' in text, text


@pytest.mark.parametrize('path', SOURCES, ids=os.path.basename)
def test_early_kernels_read_no_constant_memory_of_their_predecessors(path):
    """A kernel that starts before its predecessors end (griddepcontrol.wait) takes what those write
    through plain pointers: const __restrict__ lets the compiler load it before the wait.  The
    descriptors and prefix sums of a batch are written by no kernel."""
    text = open(path).read()
    for m in re.finditer(r'__global__[^;{]*?(\w+)\(([^{;]*?)\)\s*\{', text):
        body = text[m.end():].split('__global__')[0]
        if 'griddepcontrol.wait' in body:
            params = re.findall(r'__restrict__\s*(\w+)', m.group(2))
            assert set(params) <= {'descs', 'prefix'}, (m.group(1), params)


def test_sweep_prologue_reads_no_global_memory():
    """Before griddepcontrol.wait the tensor-core sweep touches parameters and its own memory only:
    nothing there goes through a pointer parameter, prefix sums and descriptors of a batch included."""
    text = open(os.path.join(CSRC, 'tc_kernel.cuh')).read()
    body = text[text.index('sweep_tc_kernel('):]
    prologue = body[body.index('{') + 1:body.index('griddepcontrol.wait')]
    prologue = re.sub(r'//[^\n]*', '', prologue)
    assert not re.search(r'\b(descs|prefix|lineE|status|locate|skip_inactive)\b', prologue)
    assert not re.search(r'S0\.(x|y|x2|active|dot_part|le_next|le_zero)\b', prologue)


def test_sweeps_and_self_test_share_the_bounded_wait():
    """One wait function, limited by the GPU's global timer; no loop of polls beside it."""
    for name in ('tc_kernel.cuh', 'libconv_api.cu'):
        text = open(os.path.join(CSRC, name)).read()
        assert 'mbarrier.try_wait' not in text and 'mbarrier.test_wait' not in text and 'bar_wait(' in text, name
    wait = open(os.path.join(CSRC, 'lcg_wait.cuh')).read()
    assert 'globaltimer' in wait and 'limit_ns' in wait
