"""Host-side choices of an engine step's kernels, on the CPU."""
import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="a device answers")
def test_status_of_a_device_that_cannot_be_asked():
    """The worst status instead of an exception: failure detection reads a number."""
    from onecat_vllm.ops import _C
    assert _C.read_status(False) == 0x80000000 and _C.read_status(True) == 0x80000000
