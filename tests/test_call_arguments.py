"""How a call's arguments are formed: the packed leaf records against field-by-field writes,
and inputs that are taken as they are against those that are converted."""
import ctypes

import numpy as np
import pytest

from agama_gpu_b200 import _lib


@pytest.mark.parametrize("number", [float, np.float64, np.float32, int])
def test_packed_leaf_equals_field_writes(number):
    lf = _lib.AgbLeaf()
    vals = [number(v) for v in (2.0, -1.0, 3.0, 0.0, 5.0)]
    lf.comp, lf.sigma, lf.ampl = 7, vals[0], vals[4]
    lf.gamma[0], lf.gamma[1], lf.gamma[2] = vals[1:4]
    got = (_lib.AgbLeaf * 1).from_buffer_copy(_lib.pack_leaf(7, *vals))
    assert bytes(got) == bytes(lf) and ctypes.sizeof(got) == 48


@pytest.mark.gpu
def test_converted_points_give_the_same_bits():
    import torch
    import agama_gpu_b200 as agb
    pot = agb.PlummerPotentialGPU(mass=1e10, scaleRadius=0.5)
    x = torch.randn(37, 3, dtype=torch.float64, device="cuda")
    ref = pot.force(x)
    assert ref.shape == x.shape and ref.is_contiguous() and not ref.requires_grad
    wide = torch.zeros(37, 5, dtype=torch.float64, device="cuda")
    wide[:, 1:4] = x
    forms = [wide[:, 1:4], x.t().contiguous().t(), x.cpu(), x.cpu().numpy(), x.clone().requires_grad_(),
             torch.nn.Parameter(x.clone())]
    for form in forms:
        got = pot.force(form)
        assert torch.equal(got, ref) and got.is_contiguous() and not got.requires_grad
        assert type(got) is torch.Tensor
    assert torch.equal(pot.force(x[3]), ref[3])
    assert pot.force(x[:0]).shape == (0, 3)
    with pytest.raises(ValueError):
        pot.force(torch.zeros(4, 2, dtype=torch.float64, device="cuda"))
