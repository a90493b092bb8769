"""One V-cycle of the mixed solver on narrow grids, where level 0 takes four planes per thread whatever its size:
more planes than a grid of blocks has along z, and more blocks than one plane per thread pays for. Oracle and
bar as for small level 0.
"""
import pytest

import test_gpu_small_level0 as small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topology,n", [("closed", (4, 2, 70000)), ("perio_xyz", (4, 2, 131068)), ("perio_xy", (4, 4, 16384)),
                                        ("perio_y", (8, 64, 256))])
def test_cycle_against_oracle(topology, n):
    small.test_cycle_against_oracle(topology, n)
