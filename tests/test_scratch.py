"""Scratch of the evaluation entries: what is asked for serves every smaller call and every
time, and calls that need none run without it."""
import pytest


def _descriptors(columns, nodes=50, n_leaves=1):
    """Multipoles of so many columns in one frame, described as far as sizes look at them."""
    from agama_gpu_b200 import _lib
    comps = (_lib.AgbComponent * n_leaves)()
    leaves = (_lib.AgbLeaf * n_leaves)()
    for i in range(n_leaves):
        comps[i].kind = _lib.KIND_MULTIPOLE
        comps[i].n_lm, comps[i].n_int = columns, nodes - 1
        leaves[i].comp, leaves[i].sigma, leaves[i].ampl = i, 1.0, 1.0
    return comps, n_leaves, leaves, n_leaves


SIZES = [1, 4999, 16383, 16384, 32768, 32769, 32868, 60000, 100003, 131072, 131073, 1 << 20,
         (1 << 23) + 1]


@pytest.mark.parametrize("lmax", [4, 6, 8, 10, 12, 16, 20, 32])
def test_workspace_of_the_largest_call_serves_smaller_ones(lmax):
    from agama_gpu_b200 import _lib
    columns = (lmax // 2 + 1) * (lmax + 1)
    one, two = _descriptors(columns), _descriptors(columns, n_leaves=2)
    most = 0
    for n in SIZES:
        # two snapshots in use, or one of them
        b = _lib.lib.agb_eval_workspace_bytes(*two, n, 0)
        assert b == _lib.lib.agb_eval_workspace_bytes(two[0], 2, two[2], 1, n, 0) >= most
        most = b
        for args in (one, two):
            for mode in range(5):
                for prec in (_lib.PREC_FP64, _lib.PREC_MIXED):
                    for flags in (0, _lib.OUT_BIN_ALWAYS):
                        assert _lib.lib.agb_eval_scratch_bytes(*args, n, mode, prec, flags) <= most
    assert _lib.lib.agb_eval_workspace_bytes(*two, 10**6, _lib.OUT_NO_BINNING) == 0
    assert _lib.lib.agb_eval_scratch_bytes(*two, 10**6, _lib.MODE_POT, 0, _lib.OUT_NO_BINNING) == 0


def test_fewest_points_never_sort():
    """The calls for which no scratch is asked (SORT_NEVER) are calls that need none."""
    from agama_gpu_b200 import _lib
    from itertools import product
    for columns, leaves in product((45, 64, 144, 560, 561, 1024, 1088, 1089), (1, 2, 7, _lib.MAX_LEAVES)):
        args = _descriptors(columns, nodes=200, n_leaves=leaves)
        for mode, prec in product(range(5), (_lib.PREC_FP64, _lib.PREC_MIXED)):
            for n in {1, _lib.SORT_NEVER // leaves}:
                assert _lib.lib.agb_eval_scratch_bytes(*args, n, mode, prec, 0) == 0
                # by flag they do
                assert _lib.lib.agb_eval_scratch_bytes(*args, n, mode, prec, _lib.OUT_BIN_ALWAYS) > 0


def _multipole(lmax, seed=3, nodes=50):
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import nfw_multipole
    return agb.MultipolePotentialGPU(nfw_multipole(lmax=lmax, n_nodes=nodes, seed=seed, amp=0.3))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [60000, 131072])
@pytest.mark.parametrize("lmax", [6, 8, 12])
def test_eval_host_at_a_snapshot_and_between(n, lmax):
    import torch
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import hernquist_points
    pot = agb.EvolvingPotentialGPU([_multipole(lmax, s) for s in (1, 2, 3)], [0.0, 1.0, 2.0])
    x = torch.from_numpy(hernquist_points(n, 10.0, 5))
    xd = x.cuda()
    for t in (0.0, 0.5, 1.0, 1.7, -1.0):
        for want in (dict(pot=True), dict(pot=True, acc=True), dict(der=True)):
            got, ref = pot.eval_host(x, t=t, **want), pot.eval(xd, t=t, **want)
            for a, b in zip(*((v if isinstance(v, tuple) else (v,)) for v in (got, ref))):
                # a chunk may take another kernel than the whole call: rounding
                assert float((a - b.cpu()).abs().max()) <= 1e-13 * float(b.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5000, 16383])
def test_small_calls_need_no_scratch(n):
    """Below the documented size a call runs without scratch, with too little or at an
    unaligned address; the order of the points changes no bit."""
    import torch
    from agama_gpu_b200 import _lib
    from agama_gpu_b200.synthetic import hernquist_points
    pot = _multipole(32, nodes=100)
    x = torch.from_numpy(hernquist_points(n, 10.0, 5)).cuda()
    cargs = pot._c_args(0.0, x.device)
    need = _lib.lib.agb_eval_scratch_bytes(*cargs, n, _lib.MODE_GRAD, 0, 0)
    ws = torch.empty(_lib.lib.agb_eval_workspace_bytes(*cargs, n, 0), dtype=torch.uint8, device="cuda")
    if n == 16383:
        assert 0 < need < ws.numel()
    out = []
    for p, room in ((ws.data_ptr(), ws.numel()), (None, 0), (ws.data_ptr(), 256), (ws.data_ptr() + 8, ws.numel() - 8)):
        F = torch.empty_like(x)
        assert _lib.lib.agb_eval_ws(*cargs, x.data_ptr(), n, _lib.MODE_GRAD, 0, None, F.data_ptr(),
                                    None, None, 0, p, room, None) == 0
        out.append(F)
    F = torch.empty_like(x)
    assert _lib.lib.agb_eval(*cargs, x.data_ptr(), n, _lib.MODE_GRAD, 0, None, F.data_ptr(), None,
                             None, 0, None) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(out[0], f) for f in out[1:] + [F])
    # asked for by flag, the sort needs its scratch as before
    assert _lib.lib.agb_eval_ws(*cargs, x.data_ptr(), n, _lib.MODE_GRAD, 0, None, F.data_ptr(), None,
                                None, _lib.OUT_BIN_ALWAYS, None, 0, None) == -1


def test_other_frames_and_cylsplines_count_for_the_sort():
    """Sorting by one Multipole's intervals helps Multipoles in other frames and CylSplines."""
    from agama_gpu_b200 import _lib
    frames = _descriptors(45, n_leaves=8)
    for i in range(8):
        frames[2][i].gamma[0] = float(i)
    barred = _descriptors(45, n_leaves=2)
    barred[0][1].kind, barred[0][1].n_lm = _lib.KIND_CYLSPLINE, 13
    alone = _descriptors(45)
    for n in (100003, 400003):
        for mode in (_lib.MODE_GRAD, _lib.MODE_HESS):
            # 691 -> 513 us (forces) of the eight, 341 -> 272 with the CylSpline at 400003 points
            assert _lib.lib.agb_eval_scratch_bytes(*frames, n, mode, _lib.PREC_FP64, 0) > 0
            assert _lib.lib.agb_eval_scratch_bytes(*barred, n, mode, _lib.PREC_FP64, 0) > 0
            # 62 -> 87 us: one small table is read from L1 in any order
            assert _lib.lib.agb_eval_scratch_bytes(*alone, n, mode, _lib.PREC_FP64, 0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tree,n,prec", [("analytic", 100003, "mixed"), ("four", 100003, "mixed"),
                                         ("analytic", 40009, "fp64"), ("frames", 131072, "fp64")])
def test_default_call_is_no_slower_than_one_thread_per_point(tree, n, prec):
    """Trees with many leaves: the kernel that the rules pick against one thread per point on
    sorted points (1.4 to 1.85 times as slow before the rules looked at all leaves)."""
    import torch
    import agama_gpu_b200 as agb
    from agama_gpu_b200 import _lib
    from agama_gpu_b200.synthetic import hernquist_points
    shift = lambda p, i: agb.ShiftedPotentialGPU(p, [float(i), 1.0, 0.0])  # noqa: E731
    leaves = {"analytic": lambda: [_multipole(16, nodes=64)] + [
                  shift(agb.PlummerPotentialGPU(mass=1e9, scaleRadius=0.5), i) for i in range(20)],
              "four": lambda: [_multipole(16, s, 64) for s in range(4)],
              "frames": lambda: [shift(_multipole(8, 3, 64), i) for i in range(8)]}[tree]()
    pot = agb.CompositePotentialGPU(leaves)
    x = torch.from_numpy(hernquist_points(n, 10.0, 5)).cuda()
    base = type(pot)._flags

    def time(flags):
        pot._flags = lambda *a: base(pot, *a) | flags
        best = 1e9
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(8):
                pot._launch(x, 0.0, _lib.MODE_POT if tree == "frames" else _lib.MODE_GRAD, False,
                            precision=prec)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        del pot._flags
        return best
    time(0)
    assert time(0) < 1.25 * time(_lib.OUT_BIN_ALWAYS | 2 << _lib.OUT_GRID_SHIFT)


@pytest.mark.gpu
def test_small_static_calls_may_overlap():
    """agb_eval_static's shared array is not used below the documented size: small calls on two
    streams at the same time give their own results."""
    import torch
    from agama_gpu_b200 import _lib
    from agama_gpu_b200.synthetic import hernquist_points
    pots = [_multipole(32, nodes=100), _multipole(24, 4, 60)]
    xs = [torch.from_numpy(hernquist_points(n, 10.0, n)).cuda() for n in (16383, 9001)]
    cargs = [p._c_args(0.0, x.device) for p, x in zip(pots, xs)]
    out = [[torch.empty_like(x) for _ in range(10)] for x in xs]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k in range(10):
        for i in (0, 1):
            assert _lib.lib.agb_eval_static(*cargs[i], xs[i].data_ptr(), xs[i].shape[0], _lib.MODE_GRAD,
                                            0, None, out[i][k].data_ptr(), None, None, _lib.OUT_NEGATE,
                                            streams[i].cuda_stream) == 0
    torch.cuda.synchronize()
    for p, x, fs in zip(pots, xs, out):
        ref = p.force(x)
        assert all(torch.equal(f, ref) for f in fs)
