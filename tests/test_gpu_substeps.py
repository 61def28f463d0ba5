"""Several steps in one call share the launch between the half-kick that ends a substep and
the kick and drift that begin the next: the same bits as one step per call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_time", [False, True])
@pytest.mark.parametrize("scheme", ["leapfrog", "yoshida4"])
@pytest.mark.parametrize("n", [1, 33])
def test_steps_together_equal_steps_alone(scheme, device_time, n):
    import torch
    import agama_gpu_b200 as agb
    from agama_gpu_b200.integrate import Leapfrog
    from agama_gpu_b200.synthetic import nfw_multipole
    halo = agb.MultipolePotentialGPU(nfw_multipole(lmax=4, n_nodes=30, seed=2, amp=0.3))
    prog = agb.PlummerPotentialGPU(mass=1e10, scaleRadius=0.5)
    if device_time:                            # a moving centre: leaves from the step counter
        prog = agb.ShiftedPotentialGPU(prog, np.column_stack(
            [np.linspace(0.0, 0.1, 9), np.cos(np.arange(9.0)), np.sin(np.arange(9.0)), np.arange(9.0)]))
    pot = agb.CompositePotentialGPU([halo, prog])
    gen = torch.Generator(device="cuda").manual_seed(4)
    x0 = torch.randn(n, 3, dtype=torch.float64, device="cuda", generator=gen) * 8
    v0 = torch.randn(n, 3, dtype=torch.float64, device="cuda", generator=gen) * 100
    ends = []
    for parts in ([5], [1] * 5, [2, 3]):
        it = Leapfrog(pot, 1e-3, precision="fp64", use_graph=False, scheme=scheme,
                      device_time=device_time)
        x, v, F = x0.clone(), v0.clone(), torch.empty_like(x0)
        it._set_step(x, 0)
        it._force_at(x, 0, 0.0, F)
        k = 0
        for m in parts:
            it._steps(x, v, F, k, m)
            k += m
        ends.append((x, v, F))
    for other in ends[1:]:
        for a, b in zip(ends[0], other):
            assert torch.equal(a, b)
