"""A point's result does not depend on the kernel that its call takes: one thread per point, a
block's warps sharing the harmonics, a warp loading its CylSpline records together, sorted or
not, leaves from the host or from the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _halo(lmax, every_l=False, seed=3):
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import nfw_multipole
    coefs = nfw_multipole(lmax=lmax, n_nodes=40, seed=seed, amp=0.3)
    if every_l:
        rng = np.random.default_rng(1)
        for c, (l, _) in enumerate(coefs.lm_labels):
            if l % 2:
                f = 0.1 * 10.0 ** (-l / 2.0) * rng.normal()
                coefs.phi[:, c] = coefs.phi[:, 0] * f
                coefs.dphi_dr[:, c] = coefs.dphi_dr[:, 0] * f
    return agb.MultipolePotentialGPU(coefs)


def _tree(name):
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import bar_cylspline
    mn = agb.MiyamotoNagaiPotentialGPU(mass=5e10, scaleRadius=3.0, scaleHeight=0.3)
    if name == "even":
        return _halo(32) + mn + agb.ShiftedPotentialGPU(_halo(8), [1.0, -2.0, 0.5])
    if name == "every_l":
        return _halo(9, True) + _halo(2)
    if name == "barred":
        return _halo(12) + agb.CylSplinePotentialGPU(bar_cylspline())
    if name == "disk":
        return agb.CylSplinePotentialGPU(bar_cylspline()) + mn
    if name == "moving_disk":
        t = np.arange(5.0)
        return mn + agb.ShiftedPotentialGPU(agb.CylSplinePotentialGPU(bar_cylspline()),
                                            np.column_stack([0.7 * t, np.sin(t), 0.1 * t * t, t]))
    # snapshots of unequal orders: the components in use change with time
    return mn + agb.EvolvingPotentialGPU([_halo(4, seed=1), _halo(12, seed=2), _halo(32, seed=3)],
                                         [0.0, 1.0, 2.0])


def _points(n):
    import torch
    from agama_gpu_b200.synthetic import hernquist_points
    x = hernquist_points(n, 10.0, n)
    odd = [(0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (1e-4, 0.0, 0.0), (0.0, 2e3, 1e3), (np.nan, 1.0, 1.0),
           (np.inf, 1.0, 1.0), (1.0, 1.0, -np.inf), (1e-12, 0.0, 5.0)]
    x[:min(n, len(odd))] = odd[:n]
    return torch.from_numpy(x).cuda()


def _all(pot, x, prec, flags, t=0.4):
    from agama_gpu_b200 import _lib
    base = type(pot)._flags
    pot._flags = lambda *a: base(pot, *a) | flags
    try:
        return [v for mode in (_lib.MODE_POT, _lib.MODE_GRAD, _lib.MODE_HESS, _lib.MODE_DENS)
                for v in pot._launch(x, t, mode, True, precision=prec) if v is not None]
    finally:
        del pot._flags


def _same(a, b):
    import torch
    return len(a) == len(b) and all(
        bool(((u == v) | (torch.isnan(u) & torch.isnan(v))).all()) for u, v in zip(a, b))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["even", "every_l", "barred", "disk", "snapshots"])
def test_every_kernel_gives_the_same_bits(name, prec):
    from agama_gpu_b200 import _lib
    pot = _tree(name)
    for n in (1, 31, 149, 2003, 10007, 40009):
        x = _points(n)
        one = _all(pot, x, prec, _lib.OUT_NO_BINNING | 1 << _lib.OUT_GRID_SHIFT)
        for flags in (0, _lib.OUT_NO_BINNING, _lib.OUT_BIN_ALWAYS):
            assert _same(_all(pot, x, prec, flags), one), (n, flags)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["snapshots", "moving_disk"])
def test_leaves_from_the_device_give_the_same_bits(name, prec):
    from agama_gpu_b200 import _lib
    pot = _tree(name)
    for n in (100, 3001, 20011):
        x = _points(n)
        for t in (0.0, 0.3, 1.0, 1.9, 2.5):
            for mode in (_lib.MODE_POT, _lib.MODE_GRAD, _lib.MODE_HESS, _lib.MODE_DENS):
                host = pot._launch(x, t, mode, True, precision=prec)
                dev = pot._launch_timed(x, None, t, 0.0, 0.0, mode, True, precision=prec)
                assert _same([v for v in host if v is not None],
                             [v for v in dev if v is not None]), (n, t, mode)


def test_points_of_a_call_do_not_matter():
    import torch
    pot = _tree("even")
    x = _points(40009)
    whole = pot.force(x)
    for lo, hi in ((0, 1), (5, 40), (100, 2100), (3000, 13007)):
        assert _same([pot.force(x[lo:hi])], [whole[lo:hi]])
    assert _same([pot.eval_host(x.cpu(), acc=True, chunk_points=9001).cuda()], [whole])
