"""The stream's handle comes from calls private to torch where they are, and from the public ones where they are not."""
import subprocess
import sys

import pytest
import torch

from rustinfer_b200.ops import library as L


def test_the_package_loads_with_a_torch_without_cuda():
    code = ("import torch\n"
            "for name in ('_cuda_getDevice', '_cuda_getCurrentRawStream'):\n"
            "    if hasattr(torch._C, name): delattr(torch._C, name)\n"
            "import rustinfer_b200.engine.runner, rustinfer_b200.ops.library as L\n"
            "assert L._current_device is torch.cuda.current_device\n")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)


@pytest.mark.gpu
def test_both_name_the_same_stream():
    device, raw = L._stream_calls(object())
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            assert raw(device()) == L.stream_ptr() == stream.cuda_stream
