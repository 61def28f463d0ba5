"""The stream that the library's calls get."""
import pytest

from agama_gpu_b200 import _lib


@pytest.mark.gpu
def test_stream_without_the_raw_number(monkeypatch):
    """A torch that does not give the stream's number itself: the same stream."""
    import torch
    import agama_gpu_b200 as agb
    dev = torch.device("cuda", torch.cuda.current_device())
    pot = agb.PlummerPotentialGPU(mass=1e10, scaleRadius=0.5)
    x = torch.randn(37, 3, dtype=torch.float64, device=dev)
    ref = pot.force(x)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for s in (torch.cuda.current_stream(), side):
        with torch.cuda.stream(s):
            want = _lib.raw_stream(dev)
            assert want == s.cuda_stream
            with monkeypatch.context() as m:
                m.setattr(_lib, "_current_raw", None)
                assert _lib.raw_stream(dev) == want
                assert torch.equal(pot.force(x), ref)
