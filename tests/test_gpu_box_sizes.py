"""What a factorization takes beside its result: device scratch and launches
over the sizes of a leaf."""
import ctypes as C

import pytest

import ki_geometry as G
import kinterp

pytestmark = pytest.mark.gpu


def _cached(mode, pr):
    """Bytes that one factorization leaves in an empty cache, and the bytes of
    X_rr of the level with the largest sum."""
    lib = kinterp.load()
    lib.ki_cached_bytes.restype = C.c_longlong
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
