"""The cluster kernel of the coarse multigrid levels: V-cycles on grids whose coarse levels are cut
into slabs that fill the blocks evenly, leave some empty or the last one short, and on ones
that block 0 holds alone, against the oracle, FP64 and FP32.

Bars: FP64 1e-13 of max|x| per V-cycle from zero (as the grid kernels' test); FP32 V-cycles in
a refinement stopped after one cycle: about 60 operations per value of 6e-8 each, 4e-6.
"""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOPO = {"closed": 1, "perio_x": 2, "perio_y": 3, "perio_xy": 5, "perio_xyz": 6}


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-13), ("mixed", 4e-6)])
@pytest.mark.parametrize("topology,n", [
    ("closed", (32, 32, 32)), ("perio_xyz", (32, 32, 32)),     # 16^3 in 8 slabs of 2 planes
    ("perio_xyz", (48, 48, 48)), ("closed", (24, 24, 48)),     # 24 planes: 6 slabs of 4
    ("perio_xy", (64, 64, 64)), ("perio_x", (16, 32, 40)),     # two levels cut; 20 planes: 5 slabs of 4
    ("perio_y", (32, 64, 16)), ("closed", (16, 16, 72)),       # 36 planes: 6 slabs of 6, two slabs cut twice
    ("closed", (20, 12, 28)), ("perio_xy", (8, 8, 8)), ("closed", (64, 16, 8))])
def test_cluster_levels_against_oracle(topology, n, precision, bar):
    from nyles_gb300.multigrid import MG
    nx, ny, nz = n
    mg = MG(nx, ny, nz, topology=topology, precision=precision)
    o = oracle.OracleMG(nx, ny, nz, TOPO[topology])
    rng = np.random.Generator(np.random.PCG64(nx + 100 * ny + 10000 * nz))
    b = rng.standard_normal((nz, ny, nx))
    b -= b.mean()
    mg.set(1, 2, torch.from_numpy(b))
    full = b
    for axis, key in ((2, "x"), (1, "y"), (0, "z")):     # mgfor's ghosts: periodic image, or 0
        pad = [(0, 0)] * 3
        pad[axis] = (3, 3)
        full = np.pad(full, pad, mode="wrap" if key in topology[5:] else "constant")
    o.set(2, full)
    mg.set_params(1e-30, 1, 0.9)
    o.params(1e-30, 1, 0.9)
    for cycle in range(2 if precision == "fp64" else 1):
        x, _ = mg.solve()
        torch.cuda.synchronize()
        o.solve()
        ref = o.get(1)[3:-3, 3:-3, 3:-3]
        assert np.max(np.abs(x.cpu().numpy() - ref)) <= bar * np.max(np.abs(ref)), cycle
