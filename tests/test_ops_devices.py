"""Only CUDA devices have a stream to launch on."""
import pytest
import torch

from hashpoint import ops


@pytest.mark.parametrize("device", ["cpu", "meta"])
def test_no_stream_off_the_gpu(device):
    """A launch for another device is refused before its (host) workspace reaches a kernel."""
    with pytest.raises(ValueError):
        ops._stream(torch.device(device))
