"""The package, its planners and the binding import on a torch that has no CUDA stream call (one built without
CUDA); a stream is looked up at a GPU call only."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import torch
if hasattr(torch._C, "_cuda_getCurrentRawStream"):
    del torch._C._cuda_getCurrentRawStream
import torchquantum_gb300
from torchquantum_gb300 import _lib, binding, fusion, program
assert _lib.expval_passes([1, 2], 10) == 1

class Stream:
    cuda_stream = 77

asked = []
torch.cuda.current_stream = lambda device=None: asked.append(str(device)) or Stream()
assert _lib._dstream(torch.device("cuda", 1)) == 77
assert binding._stream(torch.device("cuda", 2)) == 77
assert asked == ["cuda:1", "cuda:2"]
print("imported")
"""


def test_import_without_the_stream_call():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("imported"), r.stderr


def test_a_stream_of_no_cuda_device_is_refused_as_by_torch():
    import pytest
    import torch

    from torchquantum_gb300 import _lib

    with pytest.raises((ValueError, RuntimeError, AssertionError)):
        _lib._stream(torch.zeros(1))


def test_coset_groups_given_out_are_the_callers_own():
    from torchquantum_gb300 import _lib

    masks = [1 << 19, 3, 5, 1 << 7, 1 << 18, 9, 17, 33, 65]
    groups = _lib.coset_groups(masks, 20)
    passes = _lib.expval_passes(masks, 20)
    groups[0][0].clear()
    groups.pop()
    assert _lib.expval_passes(masks, 20) == passes and _lib.coset_groups(masks, 20)[0][0]
