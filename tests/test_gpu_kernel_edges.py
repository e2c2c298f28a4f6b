"""The kernels of the main path at the sizes where their tilings change:
decompositions and decouplings of small to very large boxes (leaf sizes that
reach every launch group and class), dense solves at the edges of the 16-row
blocks, operator and domain sums at the edges of the 128- and 256-row tiles.

Bars: ranks and skeletons equal to the oracle's and solutions within 1e-10 of
it (as in test_gpu_parity.py); dense solves of these well-conditioned systems
(condition below 1e3) within 1e3 * 768 * 2^-53 < 1e-10; sums of at most 4096
terms within 4096 * 2^-53 * 8 < 1e-11 of the exact entries' sum, relative to
the largest."""
import numpy as np
import pytest

import domain as D
import helpers as H
import ki_geometry as G
import kinterp
import kioracle as K

pytestmark = pytest.mark.gpu


def _cover(make, **kw):
    return lambda leaf: make(leaf_points=leaf, **kw)


BOXES = [("star", leaf) for leaf in (4, 16, 48, 100, 128, 190, 330, 700)] + \
        [("stokes", leaf) for leaf in (8, 64, 150, 260)]
MAKE = {"star": _cover(G.star_case, n=4096), "stokes": _cover(G.stokes_holes_case, n_total=2048)}


@pytest.mark.parametrize("name,leaf", BOXES)
def test_boxes_of_every_size_match_oracle(name, leaf):
    import torch
    H.ensure_oracle()
    pr = MAKE[name](leaf)
    s = kinterp.Solver(pr)
    o = K.PortSolver(pr)
    d = H.compare_solvers(s, o)
    assert not any(d[k] for k in ("partition", "rank", "skel", "redundant")), d
    mu, alpha = s.solve(pr.f)
    mu_o, alpha_o = o.solve(pr.f)
    assert H.rel(mu, mu_o) < 1e-10
    # the sketched decompositions of the same boxes: the refined solution's
    # residual, by the operator with exact entries (its own error: at most
    # 4096 * 2^-53 |A| |x| / |f|, below 1e-11)
    p = kinterp.Solver(pr, id_tol=3e-8, mode=1)
    mu_p, alpha_p = p.solve_refined(pr.f, rel_tol=1e-12)[:2]
    x = torch.tensor(np.concatenate([mu_p, alpha_p]), device="cuda", dtype=torch.float64)
    y = torch.empty_like(x)
    p.apply_device(x.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    f = np.concatenate([pr.f, np.zeros(len(alpha_p))])
    assert H.rel(y.cpu().numpy(), f) < 1e-11


@pytest.mark.parametrize("n", [1, 15, 16, 17, 32, 33, 48, 49, 300, 511, 752, 753, 767, 768, 769])
def test_dense_solve_at_block_edges(n):
    pr = G.star_case(n=n, leaf_points=2048, n_targets=4)
    s = kinterp.Solver(pr)
    mu, _ = s.solve(pr.f)
    dofs = np.arange(n)
    ref = np.linalg.solve(s.kernel_block(dofs, dofs), pr.f)
    assert H.rel(mu, ref) < 1e-10


@pytest.mark.parametrize("make", [lambda n: G.star_case(n=n, n_targets=4),
                                  lambda n: G.stokes_holes_case(n_total=n, n_holes=1)])
@pytest.mark.parametrize("n", [255, 256, 257, 384, 1000])
def test_sums_at_tile_edges(make, n):
    import torch
    pr = make(n)
    s = kinterp.Solver(pr)
    rng = np.random.default_rng(n)
    x = torch.tensor(rng.standard_normal(s.n_dofs + s.n_border), device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    s.apply_device(x.data_ptr(), y.data_ptr())
    s.matvec_device(x.data_ptr(), z.data_ptr())
    torch.cuda.synchronize()
    assert (y - z).abs().max() <= 1e-11 * y.abs().max()
    # points: inside ones (listed) among outside ones (zero), ragged counts
    mu, alpha = s.solve(pr.f)
    al = alpha if s.n_border else None
    for nt in (1, 31, 127, 129, 257, 700):
        tg = rng.uniform(-1.5, 1.5, 2 * nt)
        tg[:2] = pr.targets[:2]
        out = s.eval_domain(tg, mu, al, "nodes")
        exact = s.eval_targets(tg, mu, al)
        inside = np.repeat(D.in_domain_nodes(pr.points, pr.holes, tg).astype(bool), pr.sol_dim)
        assert np.all(out[~inside] == 0.0)
        if inside.any():
            assert np.abs(out[inside] - exact[inside]).max() <= 1e-11 * np.abs(exact[inside]).max()
