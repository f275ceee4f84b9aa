"""GPU: what an expired barrier wait looks like to the caller.  A one-CTA self-test kernel of the library waits, with
the same helper the attention kernels use, on a barrier nobody arrives on and with nothing else in flight (no TMA, no
MMA, no cluster traffic); after the limit it writes the status words and returns normally - the context stays usable.
No wait is made to run out inside the attention kernels themselves."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_expired_wait_is_reported_and_the_context_survives():
    import flashmla_b200 as fm
    from flashmla_b200 import _capi, flash_mla_interface as fmi
    lib = _capi.lib()
    dev = torch.device(DEV)
    fm.check_status()                                # nothing pending from earlier tests
    status = fmi._status(dev)                        # the words every kernel launch of the Python API reports into
    flag = torch.full((2,), -1, dtype=torch.int32, device=dev)
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record()
    rc = lib.mla_selftest_bounded_wait(1_000_000, 77, _capi.ptr(status), _capi.ptr(flag), torch.cuda.current_stream().cuda_stream)
    t1.record()
    assert rc == 0
    torch.cuda.synchronize()                         # returns: the kernel ended by itself
    assert 0.2 <= t0.elapsed_time(t1) <= 50.0        # about 1e6 cycles at 1-2 GHz, far from the default limit of a second
    assert flag.tolist() == [1, 0]                   # the CTA's abort flag is raised, the wait reported failure
    vals = status.tolist()
    assert vals[0] == 77 and vals[1] == 64           # first code, and every one of the 64 threads counted
    with pytest.raises(RuntimeError, match="gave up a bounded wait \\(code 77, 64 threads\\)"):
        fm.check_status()
    fm.check_status()                                # cleared by the raise
    assert status.tolist()[:2] == [0, 0]
    # the context is intact: an ordinary launch still works
    x = torch.arange(8, device=dev)
    assert int((x * 2).sum()) == 56


def test_selftest_rejects_bad_arguments():
    from flashmla_b200 import _capi
    lib = _capi.lib()
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    assert lib.mla_selftest_bounded_wait(0, 1, _capi.ptr(status), None, None) == 1
    assert lib.mla_selftest_bounded_wait(3_000_000_000, 1, _capi.ptr(status), None, None) == 1
    assert lib.mla_selftest_bounded_wait(1000, 1, None, None, None) == 1


# A fresh process (the words are made once per process and device).  `words` are made by the first use of a device, on a stream
# that is busy, or inside a capture; another stream's kernel may report right away.
_FIRST_USE = """
import torch
from flashmla_b200 import _capi, flash_mla_interface as fmi
first, other = torch.cuda.Stream(), torch.cuda.Stream()
x = torch.zeros(8, device="cuda:0")
# (a kernel's first launch may wait for the device while its code is loaded)
assert _capi.lib().mla_selftest_bounded_wait(1000, 1, _capi.ptr(x), None, other.cuda_stream) == 0
torch.cuda._sleep(1000)
torch.zeros(4, dtype=torch.int32, device="cuda:0")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
if {capture}:
    with torch.cuda.graph(graph, stream=first):
        x.add_(1)
        words = fmi._status("cuda:0")
else:
    with torch.cuda.stream(first):
        torch.cuda._sleep(200_000_000)                 # about a tenth of a second
        words = fmi._status("cuda:0")
assert _capi.lib().mla_selftest_bounded_wait(100_000, 77, _capi.ptr(words), None, other.cuda_stream) == 0
torch.cuda.synchronize()
if {capture}:
    graph.replay()
torch.cuda.synchronize()
assert words.tolist() == [77, 64, 0, 0], words.tolist()
"""


@pytest.mark.parametrize("capture", [False, True])
def test_status_words_do_not_lose_a_report_of_another_stream(capture):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FIRST_USE.format(capture=capture)], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
