"""node_vjp on CUDA gradients takes and refuses what it takes and refuses on the CPU: tables
edited in place, shapes that do not fit, degenerate l=0 nodes, batched gradients."""
import copy
import pickle

import numpy as np
import pytest
import torch


def _tables(nodes=20, lmax=2, seed=3):
    from agama_gpu_b200.prep_multipole import build_multipole_tables
    from agama_gpu_b200.synthetic import nfw_multipole
    return build_multipole_tables(nfw_multipole(lmax=lmax, n_nodes=nodes, seed=seed, amp=0.2))


def _degenerate(t, which):
    """l=0 nodes (values, dPhi/dr) where the builder's fits divide by zero."""
    p0, d0 = t.node_phi[:, 0].copy(), t.node_dphi_dr[:, 0].copy()
    r1, r2 = t.r_grid[0], t.r_grid[1]
    if which == "zeros":                # equal values, a slope
        p0[:2] = 0.0
    if which == "w":                    # the cubic's W = P1 - r1 d1 / 2 vanishes
        p0[0], p0[1] = -2.0, -3.0
        d0[0] = 2.0 * p0[0] / r1
        p0[0] = 0.5 * (r1 * d0[0])
        d0[1] = (r2 / r1 * (6.0 * r1 * (p0[1] - p0[0]) / (r2 - r1) - d0[0] * (2 * r1 + r2))) / (2 * r2 + r1)
    if which == "outer":                # equal denominators beyond the grid
        p0[-1] = p0[-2] = 0.0
    if which == "nan":
        p0[0] = np.nan
    return p0, d0


@pytest.mark.parametrize("which", ["zeros", "w", "outer", "nan"])
def test_degenerate_nodes_divide_as_tensors_do(which):
    from agama_gpu_b200.diff_tables import consts_and_jacobian, multipole_consts_from_nodes
    t = _tables()
    p0, d0 = _degenerate(t, which)
    phi, dphi = torch.from_numpy(t.node_phi.copy()), torch.from_numpy(t.node_dphi_dr.copy())
    phi[:, 0], dphi[:, 0] = torch.from_numpy(p0), torch.from_numpy(d0)
    ref = multipole_consts_from_nodes(t, phi, dphi).numpy()
    v, J = consts_and_jacobian(t, p0, d0)
    assert J.shape == (8, 6)
    assert np.allclose(v, ref, rtol=1e-12, atol=0.0, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("const", [False, True])
def test_tables_edited_in_place(const):
    from agama_gpu_b200.diff_tables import _node_vjp_torch, node_vjp
    t = _tables()
    rng = np.random.default_rng(1)
    g = torch.from_numpy(rng.normal(size=t.poly.shape))
    gc = torch.from_numpy(rng.normal(size=8)) if const else None
    on = lambda a: None if a is None else a.cuda()  # noqa: E731
    node_vjp(t, g.cuda(), None, grad_const=on(gc))
    for tab in (t, copy.deepcopy(t)):
        tab.node_phi *= 1.25
        tab.node_dphi_dr[3] *= 0.75
        got, ref = node_vjp(tab, g.cuda(), None, grad_const=on(gc)), _node_vjp_torch(tab, g, None, gc)
        for u, w in zip(got, ref):
            assert bool(((u.cpu() - w).abs() <= 1e-11 * w.abs().amax(0) + 1e-300).all())
    # nothing of the device stays on the tables
    back = pickle.loads(pickle.dumps(t))
    assert set(vars(back)) == set(vars(_tables()))


@pytest.mark.gpu
def test_shapes_that_do_not_fit_are_refused():
    from agama_gpu_b200.diff_tables import node_vjp
    t = _tables()
    g = torch.zeros(t.poly.shape, dtype=torch.float64)
    phi, dphi = torch.from_numpy(t.node_phi), torch.from_numpy(t.node_dphi_dr)
    bad = [dict(grad_poly=g[:-1]), dict(grad_poly=g[:, :-1]), dict(grad_poly=g[..., :5]),
           dict(grad_poly=g.reshape(-1)), dict(nodes=(phi[:, :-1], dphi[:, :-1])),
           dict(nodes=(phi[:-1], dphi[:-1])), dict(nodes=(phi, dphi[:-1])),
           dict(grad_const=torch.zeros(7, dtype=torch.float64)),
           dict(grad_const=torch.zeros(1, 8, dtype=torch.float64))]
    for kw in bad:
        for dev in ("cpu", "cuda"):
            args = dict(grad_poly=g, nodes=None, grad_const=None)
            args.update(kw)
            put = lambda a: a.to(dev) if torch.is_tensor(a) else None if a is None else tuple(q.to(dev) for q in a)  # noqa: E731
            with pytest.raises((RuntimeError, ValueError, IndexError)):
                node_vjp(t, put(args["grad_poly"]), None, nodes=put(args["nodes"]),
                         grad_const=put(args["grad_const"]))


@pytest.mark.gpu
def test_batched_gradients():
    from agama_gpu_b200.diff_tables import node_vjp
    t = _tables()
    G = torch.from_numpy(np.random.default_rng(2).normal(size=(3,) + t.poly.shape)).cuda()
    got = torch.func.vmap(lambda g: node_vjp(t, g, None))(G)
    for k in range(3):
        for u, w in zip((got[0][k], got[1][k]), node_vjp(t, G[k], None)):
            assert bool(((u - w).abs() <= 1e-11 * w.abs().amax(0) + 1e-300).all())
