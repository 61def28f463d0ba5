"""The CylSpline kernel that loads a warp's records together (cyl.cu) against the one-thread
loads of the general kernel, at sizes around a warp and a block, with points off the grid,
on cell edges and on the axis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_scaling", [True, False])
@pytest.mark.parametrize("mmax", [0, 6])
def test_warp_loads_equal_thread_loads(mmax, log_scaling):
    import torch
    import agama_gpu_b200 as agb
    from agama_gpu_b200 import _lib
    from agama_gpu_b200.synthetic import bar_cylspline, disk_points
    c = bar_cylspline(n_R=12, n_z=9, Rmin=0.0, mmax=mmax)
    if not log_scaling:
        c.phi[0] = c.phi[0] + 0.5 * abs(c.phi[0]).max()
    cs = agb.CylSplinePotentialGPU(c)
    pot = cs + agb.ShiftedPotentialGPU(agb.NFWPotentialGPU(mass=1e11, scaleRadius=9.0), [1.0, 0.0, 2.0]) \
        + agb.ScaledPotentialGPU(cs, 1.7, 0.4)
    t = cs.tables
    for n in (1, 31, 33, 128, 129, 4097):
        x = disk_points(n, seed=n)
        edge = t.Rscale * np.sinh(np.array([t.lR_grid[3], t.lz_grid[2]]))
        for i, p in enumerate([(0.0, 0.0, 1.0), (edge[0], 0.0, edge[1]), (400.0, 10.0, 3.0),
                               (1.0, 1.0, -500.0)]):
            if i < n - 1:
                x[i] = p
        x = torch.from_numpy(x).cuda()
        for mode in (_lib.MODE_POT, _lib.MODE_GRAD, _lib.MODE_HESS):
            base = type(pot)._flags
            got = pot._launch(x, 0.0, mode, True, precision="fp64")
            pot._flags = lambda *a: base(pot, *a) | 1 << _lib.OUT_GRID_SHIFT
            ref = pot._launch(x, 0.0, mode, True, precision="fp64")
            del pot._flags
            for u, v in zip(got, ref):
                if v is not None:
                    # the same operations on the same records
                    assert float((u - v).abs().max()) <= 1e-14 * float(v.abs().max())
