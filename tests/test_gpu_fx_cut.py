"""One V-cycle of FP64 multigrid levels that the integer sums' 32 x 8 x 8 tiles cut off, large enough
(500000 cells) that they are summed in integers all the same: cut along x, along y and z, and every tile
cut. Oracle, fields and bar as for whole tiles.
"""
import pytest

import test_gpu_fx as whole

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["smooth", "spread", "point"])
@pytest.mark.parametrize("topology,n", [("closed", (80, 80, 80)), ("perio_xyz", (64, 68, 124)), ("perio_xy", (16, 200, 160)),
                                        ("perio_x", (48, 104, 104))])
def test_cut_tiles_against_oracle(topology, n, kind):
    whole.test_fx_vcycle_against_oracle(topology, n, kind)
