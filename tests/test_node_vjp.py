"""The transposed table builder on the GPU (nodes.cu) and the builder's scalars with their
derivatives in plain numbers, against the differentiable restatement in torch."""
import numpy as np
import pytest


def _tables(nodes, lmax, kind, seed=3):
    from agama_gpu_b200.prep_multipole import build_multipole_tables
    from agama_gpu_b200.synthetic import nfw_multipole
    c = nfw_multipole(lmax=lmax, n_nodes=nodes, seed=seed, amp=0.2,
                      rmin=5.0 if kind == "steep" else 1e-2)
    if kind == "positive":              # no log-scaling: Phi_00 changes sign
        c.phi[:, 0] += 0.5 * abs(c.phi[0, 0])
    if kind == "core":                  # a flat centre: constant density inside
        r = c.R_grid
        c.phi[:, 0] = -1e5 / np.sqrt(1.0 + (r / 5.0) ** 2)
        c.dphi_dr[:, 0] = 1e5 * (r / 25.0) / (1.0 + (r / 5.0) ** 2) ** 1.5
    return build_multipole_tables(c, prune_threshold=0.0 if kind == "positive" else 1e-16)


def _rounding(v):
    """The builder's inner fit took the root s = (A - A) / lnr, which is rounding, and divided
    by it (U = g / s): its derivatives are rounding too, in either implementation."""
    return abs(v[2]) > 1e6 * abs(v[6])


@pytest.mark.parametrize("kind", ["nfw", "steep", "positive", "core"])
def test_consts_and_jacobian_match_the_torch_restatement(kind):
    import torch
    from agama_gpu_b200.diff_tables import consts_and_jacobian, multipole_consts_from_nodes
    for nodes in (2, 3, 20, 64):
        t = _tables(nodes, 2, kind)
        phi = torch.tensor(t.node_phi, requires_grad=True)
        dphi = torch.tensor(t.node_dphi_dr, requires_grad=True)
        k = multipole_consts_from_nodes(t, phi, dphi)
        v, J = consts_and_jacobian(t, t.node_phi[:, 0], t.node_dphi_dr[:, 0])
        # the same formulas: rounding only
        assert np.allclose(v, k.detach().numpy(), rtol=1e-13, atol=0.0)
        assert v[0] == pytest.approx(t.invPhi0, rel=1e-14)
        if _rounding(v):
            continue
        # contracted with a cotangent, as it is used; the powers are A - A to rounding and so
        # are their rows
        gk = np.random.default_rng(nodes).normal(size=8)
        gk[1] *= abs(v[1]) > 1e-6
        gk[4] *= abs(v[4]) > 1e-6
        ref = torch.autograd.grad(k, (phi, dphi), grad_outputs=torch.from_numpy(gk),
                                  allow_unused=True)
        ref = np.stack([np.zeros(nodes) if g is None else g[:, 0].numpy() for g in ref])
        got = np.zeros((2, nodes))
        for e, at in enumerate([(0, 0), (0, 1), (0, nodes - 2), (0, nodes - 1), (1, 0),
                                (1, nodes - 1)]):
            got[at] += gk @ J[:, e]
        for u, w in zip(got, ref):
            assert np.allclose(u, w, rtol=1e-9, atol=1e-12 * np.abs(w).max())


@pytest.mark.gpu
@pytest.mark.parametrize("const", [False, True])
@pytest.mark.parametrize("kind,nodes,lmax", [("nfw", 2, 2), ("nfw", 3, 0), ("nfw", 31, 4),
                                             ("core", 33, 4), ("positive", 64, 3), ("nfw", 65, 8),
                                             ("steep", 256, 6), ("nfw", 257, 2)])
def test_node_vjp_matches_the_torch_restatement(kind, nodes, lmax, const):
    import torch
    from agama_gpu_b200.diff_tables import _node_vjp_torch, consts_and_jacobian, node_vjp
    t = _tables(nodes, lmax, kind)
    rng = np.random.default_rng(nodes)
    g = torch.from_numpy(rng.normal(size=t.poly.shape))
    gc = torch.from_numpy(rng.normal(size=8) * abs(t.node_phi[0, 0])) if const else None
    moved = [torch.from_numpy(a * (1.0 + 1e-3 * rng.normal(size=a.shape)))
             for a in (t.node_phi, t.node_dphi_dr)]
    for src in (None, moved):
        p0, d0 = ((t.node_phi, t.node_dphi_dr) if src is None else [a.numpy() for a in src])
        if const and _rounding(consts_and_jacobian(t, p0[:, 0], d0[:, 0])[0]):
            continue
        ref = _node_vjp_torch(t, g, src, gc)
        got = node_vjp(t, g.cuda(), None, nodes=None if src is None else [a.cuda() for a in src],
                       grad_const=None if gc is None else gc.cuda())
        for u, w in zip(got, ref):
            # a well-conditioned solve (diagonally dominant) and a few dozen products: 1e-11
            # of the largest entry of the column
            w = w.detach()
            assert bool(((u.cpu() - w).abs() <= 1e-11 * w.abs().amax(0) + 1e-300).all())


@pytest.mark.gpu
def test_node_vjp_rejects_what_it_cannot_do():
    from agama_gpu_b200 import _lib
    assert _lib.lib.agb_multipole_node_vjp(257, 1, 0, 0.1, 0.0, 8, 8, 8, 8, None, None, 8, 8, None) == -1
    assert _lib.lib.agb_multipole_node_vjp(9, 1, 0, 0.1, 0.0, None, 8, 8, 8, None, None, 8, 8, None) == -1
