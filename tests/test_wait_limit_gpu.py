"""The sweeps' wait function ends at its limit: the self-test waits by it on a barrier that nothing
completes (no fault, trap or hang), and its duration is the limit plus at most two runs of polls."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('limit_us', [1, 300, 20000])
def test_wait_ends_at_its_limit(pkg, limit_us):
    import torch
    L = pkg.lib()
    L.libconv_gb300_selftest_wait.argtypes = [ctypes.c_int, ctypes.c_void_p]
    L.libconv_gb300_check.argtypes = [ctypes.c_void_p]
    st = torch.cuda.current_stream()
    assert L.libconv_gb300_selftest_wait(1, st.cuda_stream) == 0        # first launch
    torch.cuda.synchronize()
    e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    e0.record(st)
    assert L.libconv_gb300_selftest_wait(limit_us, st.cuda_stream) == 0
    e1.record(st)
    torch.cuda.synchronize()
    us = 1e3 * e0.elapsed_time(e1)
    assert L.libconv_gb300_check(None) == -7 and L.libconv_gb300_check(None) == 0
    # two runs of polls (together less than 512 of 1 us and twice 64 ns), the timer's steps of
    # 1 us, and 100 us for the launch between two events
    assert limit_us <= us <= limit_us + 2 * 256 * 1.13 + 1 + 100
