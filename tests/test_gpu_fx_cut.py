"""One V-cycle of FP64 multigrid levels that the integer sums' 32 x 8 x 8 tiles do not divide: cut along x, along
y and z, and levels without a whole tile, in doubles of one and of eight cells per thread. Oracle, fields
and bar as for whole tiles.
"""
import pytest

import test_gpu_fx as whole

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["smooth", "spread", "point"])
@pytest.mark.parametrize("topology,n", [("closed", (80, 80, 80)), ("perio_xyz", (64, 68, 124)), ("perio_x", (48, 104, 104)),
                                        ("perio_xy", (16, 120, 104)), ("perio_y", (6, 258, 250)),
                                        ("perio_xyz", (258, 6, 250)), ("closed", (2, 2, 70000))])
def test_cut_tiles_against_oracle(topology, n, kind):
    whole.test_fx_vcycle_against_oracle(topology, n, kind)
