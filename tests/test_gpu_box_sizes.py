"""Boxes of every size: device scratch, launch groups, and solutions where the
kernels for a box change with its size.

Solutions are compared with the oracle's at the same tolerance, within 1e-10
plus 100 times the tolerance (test_gpu_parity.py's bar, and the compression's
own error where a loose tolerance lets rounding change a skeleton)."""
import ctypes as C
import gc

import pytest

import helpers as H
import ki_geometry as G
import kinterp
import kioracle as K

pytestmark = pytest.mark.gpu


def _cached(mode, pr):
    """Bytes that one factorization leaves in an empty cache, and the bytes of
    X_rr of the level with the largest sum."""
    lib = kinterp.load()
    lib.ki_cached_bytes.restype = C.c_longlong
    gc.collect()
    lib.ki_release_cache()
    s = kinterp.Solver(pr, mode=mode)
    x = max(sum(len(b["redundant"]) ** 2 for b in level if b["compressed"])
            for level in s.all_nodes())
    s.close()
    return lib.ki_cached_bytes(), 8 * x


def test_decoupling_keeps_no_copy_of_the_redundant_blocks():
    """Reference mode corrects L with X_rr itself, which waits in the place of
    its inverse: beside preconditioner mode it takes the workspace of its
    larger decompositions, less than 1.25 times (what a scratch buffer is
    grown by) the level's X_rr."""
    pr = G.star_case(n=65536, n_targets=4)
    ref, x = _cached(0, pr)
    pre, _ = _cached(1, pr)
    assert ref - pre < 1.25 * x


def _in_shared_memory(n, k):
    """K_BN (row stride 4 mod 8), a node record per dof and the pivot column
    in 227 KB, and X_rr in the widest register tile."""
    ld = n + (4 - n) % 8
    return n - k <= 160 and 8 * (n * ld + 8 * n + 320) + 4 * (5 * n + 4) <= 227 * 1024


@pytest.mark.parametrize("make,leaf", [(lambda l: G.star_case(leaf_points=l), 160),
                                       (lambda l: G.stokes_holes_case(n_total=4096,
                                                                      leaf_points=l), 80)])
def test_boxes_that_fit_are_decoupled_together(make, leaf):
    """Only boxes whose K_BN does not fit a CTA's shared memory take a launch
    sequence of their own."""
    s = kinterp.Solver(make(leaf), timed=True)
    alone = {int(r[0]): int(r[2]) for r in s.launch_log() if int(r[1]) == 1}
    for level, boxes in enumerate(s.all_nodes()):
        done = [(len(b["active"]), len(b["skel"])) for b in boxes if b["compressed"]]
        if done:
            assert alone[level] == sum(not _in_shared_memory(n, k) for n, k in done)


@pytest.mark.parametrize("shape,leaf", [("star", 152), ("star", 158), ("star", 164),
                                        ("stokes", 76), ("stokes", 82)])
@pytest.mark.parametrize("tol", [1e-5, 1e-10, 1e-14])
def test_boxes_whose_t_stays_in_global_memory(shape, leaf, tol):
    """149 to 164 dofs, ranks low to high: each register tile."""
    H.ensure_oracle()
    pr = (G.star_case(n=4096, leaf_points=leaf) if shape == "star" else
          G.stokes_holes_case(n_total=2048, leaf_points=leaf))
    s = kinterp.Solver(pr, id_tol=tol)
    assert any(149 <= len(b["active"]) <= 164 for v in s.all_nodes() for b in v
               if b["compressed"])
    mu, _ = s.solve(pr.f)
    ref, _ = K.PortSolver(pr, id_tol=tol).solve(pr.f)
    assert H.rel(mu, ref) < 1e-10 + 100 * tol
    p = kinterp.Solver(pr, id_tol=max(tol, 1e-8), mode=1)
    assert p.solve_refined(pr.f, rel_tol=1e-12)[3] <= 1e-12
