"""Small calls: the kernel that splits the harmonics over a block's warps (split.cu) and the
one-launch sort (bin_small), against one thread per point on unsorted points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _halo(lmax, every_l, nodes=40):
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import nfw_multipole
    coefs = nfw_multipole(lmax=lmax, n_nodes=nodes, seed=lmax, amp=0.3)
    if every_l:
        rng = np.random.default_rng(1)
        for c, (l, _) in enumerate(coefs.lm_labels):
            if l % 2:
                f = 0.1 * 10.0 ** (-l / 2.0) * rng.normal()
                coefs.phi[:, c] = coefs.phi[:, 0] * f
                coefs.dphi_dr[:, c] = coefs.dphi_dr[:, 0] * f
    return agb.MultipolePotentialGPU(coefs)


def _points(n):
    import torch
    from agama_gpu_b200.synthetic import hernquist_points
    x = hernquist_points(n, 10.0, n)
    x[0] = (0.0, 0.0, 3.0)                    # on the pole
    if n > 3:
        x[1] = 0.0                            # the origin
        x[2] = (1e-4, 0.0, 0.0)               # inside and beyond the grid
        x[3] = (0.0, 2e3, 1e3)
    return torch.from_numpy(x).cuda()


def _all(pot, x, prec, flags):
    """Every mode's outputs at x with these flags."""
    from agama_gpu_b200 import _lib
    base = type(pot)._flags
    pot._flags = lambda *a: base(pot, *a) | flags
    try:
        out = []
        for mode in (_lib.MODE_POT, _lib.MODE_GRAD, _lib.MODE_HESS, _lib.MODE_DENS):
            out += [v for v in pot._launch(x, 0.3, mode, True, precision=prec) if v is not None]
        return out
    finally:
        del pot._flags


def _close(a, b):
    # the same operations per |m| group; only the FP64 sums of the groups differ in order
    for u, v in zip(a, b):
        scale = float(v[4:].abs().max()) if v.shape[0] > 4 else float(v.abs().max())
        assert float((u - v)[4:].abs().max() if v.shape[0] > 4 else (u - v).abs().max()) <= 1e-13 * scale
        assert bool(((u - v).abs() <= 1e-13 * v.abs() + 1e-13 * scale).all())


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("lmax,every_l", [(2, False), (3, True), (8, False), (9, True), (32, False)])
def test_split_equals_one_thread_per_point(lmax, every_l, prec):
    from agama_gpu_b200 import _lib
    import agama_gpu_b200 as agb
    pot = _halo(lmax, every_l) + agb.MiyamotoNagaiPotentialGPU(mass=5e10, scaleRadius=3.0,
                                                               scaleHeight=0.3) + \
        agb.ShiftedPotentialGPU(_halo(4, False, 30), [1.0, -2.0, 0.5])
    for n in (1, 31, 149, 148 * 32 + 1, 148 * 64 + 1):
        x = _points(n)
        one = _all(pot, x, prec, _lib.OUT_NO_BINNING | 1 << _lib.OUT_GRID_SHIFT)
        _close(_all(pot, x, prec, _lib.OUT_NO_BINNING), one)


@pytest.mark.parametrize("n", [1, 7, 1025, 8193, 32768, 32769])
def test_one_launch_sort(n):
    from agama_gpu_b200 import _lib
    pot = _halo(16, False, 100)
    x = _points(n)
    one = _all(pot, x, "fp64", _lib.OUT_NO_BINNING | 1 << _lib.OUT_GRID_SHIFT)
    _close(_all(pot, x, "fp64", _lib.OUT_BIN_ALWAYS), one)
    _close(_all(pot, x, "fp64", _lib.OUT_BIN_ALWAYS | 1 << _lib.OUT_GRID_SHIFT), one)


@pytest.mark.parametrize("n", [32768, 32769, 65569, 131072, 131073])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_sorted_in_slices_equals_unsorted(n, prec):
    """Edges of the slices and of their rule; the order of the points changes no bit."""
    from agama_gpu_b200 import _lib
    pot, x = _halo(6, True), _points(n)
    for a, b in zip(_all(pot, x, prec, _lib.OUT_NO_BINNING), _all(pot, x, prec, 4)):
        assert (a == b).all()
