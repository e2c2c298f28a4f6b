"""Operator and domain sums on both sides of the line between one target per
thread and two (on 148 SMs: 148 blocks of 256 targets for the operator, 296
for the domain sums), and of full launches, against sums of the exact entries: within 8 units in the last place per term, relative to the
largest."""
import numpy as np
import pytest

import ki_geometry as G
import kinterp

pytestmark = pytest.mark.gpu

MAKE = {"laplace": lambda n: G.star_case(n=n, n_targets=4),
        "stokes": lambda n: G.stokes_holes_case(n_total=n, n_holes=1, n_targets=4)}


@pytest.mark.parametrize("pde", list(MAKE))
@pytest.mark.parametrize("n", [3071, 3072, 3073, 4096, 8704, 8960, 16384])
def test_operator(pde, n):
    import torch
    s = kinterp.Solver(MAKE[pde](n), id_tol=1e-3)
    x = torch.tensor(np.random.default_rng(n).standard_normal(s.n_dofs + s.n_border),
                     device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    s.apply_device(x.data_ptr(), y.data_ptr())
    s.matvec_device(x.data_ptr(), z.data_ptr())
    torch.cuda.synchronize()
    assert (y - z).abs().max() <= 8 * 2.0**-53 * s.n_dofs * y.abs().max()


@pytest.mark.parametrize("pde", list(MAKE))
@pytest.mark.parametrize("nt", [148 * 256, 148 * 256 + 1, 592 * 256, 592 * 256 + 1])
def test_domain(pde, nt):
    pr = MAKE[pde](1000)  # two splits of the sources
    s = kinterp.Solver(pr, id_tol=1e-3)
    mu, alpha = s.solve(pr.f)
    al = alpha if s.n_border else None
    tg = np.random.default_rng(1).uniform(-1.5, 1.5, 2 * nt)
    out, exact = s.eval_domain(tg, mu, al, "all"), s.eval_targets(tg, mu, al)
    assert np.abs(out - exact).max() <= 8 * 2.0**-53 * s.n_dofs * np.abs(exact).max()


@pytest.mark.parametrize("sizes", [(17, 300, 257, 6000), (256, 256), (512, 700, 8192)])
def test_operator_of_uneven_problems(sizes):
    """More source splits than a small problem has tiles: the rest are empty."""
    import torch
    rng = np.random.default_rng(sizes[0])
    b = kinterp.BatchSolver([G.random_star(rng, n, 64) for n in sizes], id_tol=1e-3)
    x = torch.tensor(rng.standard_normal(b.n_dofs), device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    b.apply_device(x.data_ptr(), y.data_ptr())
    kinterp.Solver.matvec_device(b, x.data_ptr(), z.data_ptr())
    torch.cuda.synchronize()
    for n, p, q in zip(sizes, b.split(y), b.split(z)):
        assert (p - q).abs().max() <= 8 * 2.0**-53 * n * p.abs().max()
