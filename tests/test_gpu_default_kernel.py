"""Tuned calls and the host pipeline reach the library's own choice of kernel, not only the
shapes of the kernel with one thread per point."""
import json

import pytest

pytestmark = pytest.mark.gpu


def _galaxy():
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import nfw_multipole
    return (agb.MultipolePotentialGPU(nfw_multipole(lmax=16, n_nodes=64, seed=3, amp=0.3))
            + agb.MiyamotoNagaiPotentialGPU(mass=5e10, scaleRadius=3.0, scaleHeight=0.3))


def _disk():
    import agama_gpu_b200 as agb
    from agama_gpu_b200.synthetic import bar_cylspline
    return agb.CylSplinePotentialGPU(bar_cylspline())


def _ms(fn):
    import torch
    best = 1e9
    for _ in range(8):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        for _ in range(8):
            fn()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) / 8)
    return best


@pytest.mark.parametrize("tree,n", [(_galaxy, 2003), (_galaxy, 10007), (_disk, 1_000_000)])
def test_tuned_calls_are_no_slower(tree, n, tmp_path, monkeypatch):
    import torch
    from agama_gpu_b200 import autotune
    from agama_gpu_b200.synthetic import disk_points, hernquist_points
    monkeypatch.setenv("AGB_AUTOTUNE_CACHE", str(tmp_path / "cache.json"))
    pot = tree()
    x = torch.from_numpy(disk_points(n, seed=1) if tree is _disk else hernquist_points(n, 10.0, 4)).cuda()
    ref = pot.force(x)
    before = _ms(lambda: pot.force(x))
    res = autotune.autotune(pot, x, mode="force", reps=10)
    assert any(k.endswith("/default") for k in res["ms"])
    assert torch.equal(pot.force(x), ref)
    # 47 -> 180 us (galaxy, 10007 points) and 146 -> 284 (disk) when the shapes alone were tried
    assert _ms(lambda: pot.force(x)) < 1.25 * before


@pytest.mark.parametrize("n", [70000, (1 << 21) + 5])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_the_default_stands_for_the_shape_that_it_is(n, mode):
    from agama_gpu_b200 import autotune
    cands = autotune._candidates(n, mode)
    assert len(dict(cands)) == len(cands) == (32 if mode == 2 else 48)
    assert [f & ~6 for k, f in cands if k.endswith("/default")] == [0, 0]


def test_choices_among_other_candidates_are_not_applied(tmp_path, monkeypatch):
    from agama_gpu_b200 import _lib, autotune
    monkeypatch.setenv("AGB_AUTOTUNE_CACHE", str(tmp_path / "cache.json"))
    pot = _galaxy()
    key = json.loads(autotune.signature(pot, _lib.MODE_GRAD, _lib.PREC_FP64, 10007))
    rec = {"flags": 1 << _lib.OUT_GRID_SHIFT, "best": "sort/b256/grid1", "ms": {}}
    (tmp_path / "cache.json").write_text(json.dumps({json.dumps(key[:6]): rec}))
    assert not autotune.apply_cached(pot, 10007, precision="fp64")
    (tmp_path / "cache.json").write_text(json.dumps({json.dumps(key): rec}))
    assert autotune.apply_cached(pot, 10007, precision="fp64")


def test_host_pipeline_sets_no_shape_on_disks():
    import torch
    from agama_gpu_b200 import _lib
    from agama_gpu_b200.synthetic import disk_points
    x = torch.from_numpy(disk_points(1_000_000, seed=1))
    seen, inner = [], _lib.lib.agb_eval_ws
    bits = 15 << _lib.OUT_GRID_SHIFT

    def call(*args):
        seen.append(args[12])
        return inner(*args)
    for pot, prec, shaped in ((_disk(), "fp64", False), (_disk(), "mixed", True), (_galaxy(), "fp64", True)):
        pot.set_precision(prec)
        ref = pot.eval(x.cuda(), acc=True)
        del seen[:]
        _lib.lib.agb_eval_ws = call
        try:
            got = pot.eval_host(x, acc=True)
        finally:
            _lib.lib.agb_eval_ws = inner
        assert len(seen) > 2 and any(f & bits for f in seen) == shaped
        assert torch.equal(got, ref.cpu())
