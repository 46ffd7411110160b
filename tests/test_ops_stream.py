"""The operators' stream handle: torch's current stream, also where torch does not have the short way to it."""
import subprocess
import sys

import pytest
import torch


def test_import_without_the_short_way_to_the_stream():
    # as in a torch built without CUDA
    code = ("import torch\n"
            "for n in ('_cuda_getCurrentRawStream', '_cuda_getDevice'):\n"
            "    if hasattr(torch._C, n): delattr(torch._C, n)\n"
            "from teenygrad_b200 import ops\n"
            "torch.cuda.current_stream = lambda: type('Stream', (), {'cuda_stream': 41})\n"
            "assert ops._stream() == 41\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.gpu
def test_current_stream():
    from teenygrad_b200 import ops
    side = torch.cuda.Stream()
    assert ops._stream() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert ops._stream() == side.cuda_stream != 0
        y = ops.silu_forward(torch.full((1000,), 2.0, device="cuda"))
    side.synchronize()
    assert torch.allclose(y, torch.nn.functional.silu(torch.full((1000,), 2.0, device="cuda")))
