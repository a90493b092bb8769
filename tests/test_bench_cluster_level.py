"""The coarse-level rule of bench.py's byte model against the library's: the levels that a cluster of blocks takes on the
grids of the bench, on flat levels whose cells are few but whose ghost rings are not, and below the smallest hierarchy.
"""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _bench():
    sys.path.insert(0, os.path.dirname(HERE))
    import bench
    return bench


@pytest.mark.parametrize("n,elem,first", [(256, 4, 32), (256, 8, 16), (128, 4, 32), (128, 8, 16), (64, 4, 32), (16, 8, 8)])
def test_cubes(n, elem, first):
    b = _bench()
    lev = b.mg_levels(n)
    assert lev[b.mg_cluster_level(lev, elem)] == (first, first, first)


def test_flat_levels_need_their_rings():
    b = _bench()
    # 2 x 128 x 128: 2^15 cells, not cut (fewer than 4 planes), 3 * 4 * 130 * 130 * 4 = 811 KB
    lev = [(4, 256, 256), (2, 128, 128), (1, 64, 64)]
    assert b.mg_cluster_level(lev, 4) == len(lev)
    # 1 x 2 x 2 under 2 x 4 x 4 fits
    assert b.mg_cluster_level([(4, 8, 8), (2, 4, 4), (1, 2, 2)], 4) == 1


def test_two_levels_at_least_and_never_level_0():
    b = _bench()
    assert b.mg_cluster_level([(4, 4, 4), (2, 2, 2)], 4) == 2
    assert b.mg_cluster_level([(2, 2, 2)], 8) == 1


def test_roofline_of_the_cluster_form():
    b = _bench()
    # FP64, 256^3: 4 grid levels above 16^3, one bracketed call per smoothing and the coarse solve
    sm = b.roofline("mg_smooth", {"mg_smooth": {"count": 9 * 4, "ms": 8.0}}, 256, 8, 6778.0, "measured", None, cluster=True)
    assert sm["vcycles"] == pytest.approx(4.0)
