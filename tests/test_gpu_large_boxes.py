"""Boxes whose factors do not fit shared memory: the transposed solve by
clusters of CTAs, and which kernels the problems of test_gpu_kernel_edges.py
run.

Bar of the solve: |A^T x - b| <= 1e-9 |b| at id_tol 1e-10 (as in
test_gpu_adjoint.py)."""
import numpy as np
import pytest

import ki_geometry as G
import kinterp
import test_gpu_kernel_edges as E

pytestmark = pytest.mark.gpu


def _compressed(s):
    """(dofs, rank) of the compressed boxes, by level."""
    return [[(len(b["active"]), len(b["skel"])) for b in v if b["compressed"]]
            for v in s.all_nodes()]


def _swept_by_clusters(boxes):
    """A level of at most 64 boxes whose two factors of a sweep, beside the
    vector, take more than 100 KB."""
    return (0 < len(boxes) <= 64 and
            8 * (max(n for n, _ in boxes) + 2 * max(k * (n - k) for n, k in boxes)) > 100 * 1024)


@pytest.mark.parametrize("leaf,tol", [(190, 1e-10), (190, 1e-14), (330, 1e-13), (700, 1e-10),
                                      (700, 1e-14)])
def test_transposed_solve_of_large_boxes(leaf, tol):
    import torch
    s = kinterp.Solver(G.star_case(n=4096, leaf_points=leaf), id_tol=tol)
    levels = _compressed(s)
    assert any(n - k > 104 for v in levels for n, k in v)  # the diagonal step's
    assert leaf < 700 or any(_swept_by_clusters(v) for v in levels)
    b = np.random.default_rng(leaf).standard_normal(s.n_dofs)
    bd = torch.tensor(b, device="cuda")
    x = torch.empty_like(bd)
    s.solve_transpose_device(bd.data_ptr(), x.data_ptr())
    torch.cuda.synchronize()
    idx = np.arange(s.n_dofs, dtype=np.int32)
    r = s.kernel_block(idx, idx).T @ x.cpu().numpy() - b
    assert np.linalg.norm(r) <= 1e-9 * np.linalg.norm(b)


def _decoupling(n, k):
    """Register tile of the redundant block (r <= 64, 96, 160), + 3 where T
    does not fit shared memory beside K_BN; -1: neither fits."""
    def smem(t):
        ld = n + (4 - n) % 8
        return 8 * (n * ld + (max(t, 8 * n) + 1) // 2 * 2 + 320) + 4 * (5 * n + 4) <= 227 * 1024
    tile = next((i for i, r in enumerate((64, 96, 160)) if n - k <= r), -1)
    if tile < 0 or not smem(0):
        return -1
    return tile if smem((k + (4 - k) % 8) * (n - k)) else tile + 3


def test_edge_problems_reach_every_kernel():
    """Decompositions in registers (nine of the ten tiles; the tenth serves
    ellipses), in shared memory, sketched in shared memory, spilled, and every
    class of decoupling, beside levels of more CTAs than the GPU holds."""
    groups, classes, ctas = set(), set(), 0
    for name, leaf in E.BOXES + [("ellipse", 64)]:
        pr = (G.ellipse_case(n=3000, leaf_points=leaf) if name == "ellipse" else
              E.MAKE[name](leaf))
        for kw in ({}, {"id_tol": 3e-8, "mode": 1}):
            s = kinterp.Solver(pr, timed=True, **kw)
            ids = [r for r in s.launch_log() if int(r[1]) == 0]
            groups |= {int(r[2]) for r in ids}
            ctas = max([ctas] + [int(r[2]) % 100 * int(r[3]) for r in ids])
            classes |= {_decoupling(n, k) for v in _compressed(s) for n, k in v}
    assert {g // 100 - 10 for g in groups if g >= 1000} == set(range(10))
    slabs = {100: (1, 2, 4, 8, 16), 200: (1, 2, 8, 16), 300: (16,)}
    assert {g for g in groups if g < 1000} == {c + n for c in slabs for n in slabs[c]}
    assert classes == {-1, 0, 1, 2, 3, 4, 5}
    assert ctas > 148
