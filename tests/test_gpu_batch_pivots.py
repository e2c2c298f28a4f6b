"""A problem keeps in a batch the ranks and skeletons it has alone, where only
rounding decides: circles, whose columns' norms tie in pairs, and random stars
decomposed down to 1e-14, whose last pivots are chosen among rounding errors.
Both are equal only if a column's sums are formed in the same order in both
calls.  The solutions then differ by the rounding of the solves: 3e-13 for
sums of 3,000 terms (3,000 * 2^-53)."""
import numpy as np
import pytest

import helpers as H
import ki_geometry as G
import kinterp

pytestmark = pytest.mark.gpu


def _circle(n):
    pts, nrm, kap, w, holes = G.reference_shape("circle", n)
    return G.Problem("circle", G.LAPLACE, pts, nrm, kap, w, holes, G.single_electron(pts),
                     np.zeros(0), np.zeros(0), 64, 1e-10)


def _star(n):
    return G.random_star(np.random.default_rng(7 + n), n, 64)


def _skeletons(s, start, end):
    """(level, skeleton) of each compressed box whose dofs are start .. end."""
    out = set()
    for l in range(s.levels()):
        for i in range(s.nodes(l)):
            b = s.node(l, i)
            if b["compressed"] and start <= b["skel"][0] < end:
                out.add((l, tuple(np.sort(b["skel"] - start))))
    return out


@pytest.mark.parametrize("make,tol", [(_circle, 1e-5), (_circle, 1e-10), (_star, 1e-10),
                                      (_star, 1e-14)])
def test_batch_keeps_each_problems_skeletons(make, tol):
    prs = [make(n) for n in range(1000, 3000, 80)]
    b = kinterp.BatchSolver(prs, id_tol=tol)
    mu = b.split(b.solve())
    for p, pr in enumerate(prs):
        s = kinterp.Solver(pr, id_tol=tol)
        alone = _skeletons(s, 0, s.n_dofs)
        assert alone and alone == _skeletons(b, b.offsets[p], b.offsets[p + 1])
        assert H.rel(mu[p], s.solve(pr.f)[0]) < 3e-13
        s.close()
