"""The FP64 multigrid levels summed in integers (levels of 2^18 cells and more): one
V-cycle through the C ABI against the oracle, on extents that fill the 32 x 8 x 8 tiles and on
ones that cut them off, with fields that keep a tile's exponents together, spread them (tiles
summed in doubles), and are zero over whole tiles.

Bar: 1e-13 of max|x| after one V-cycle, as for the levels summed in doubles: the sums are
exact to 2^-59 of a tile's largest value, and a V-cycle is about ten operations per level on
the solution (10 x 1.1e-16 x 7 levels, growing by the smoother's factor below 2 per sweep).
"""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOPO = {"closed": 1, "perio_x": 2, "perio_y": 3, "perio_xy": 5, "perio_xyz": 6}   # mgfor's topology numbers


def _rhs(kind, shape, rng):
    z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in shape], indexing="ij")
    b = np.cos(np.pi * x) * np.cos(2 * np.pi * y) * np.cos(np.pi * z) + 1e-2 * rng.standard_normal(shape)
    if kind == "spread":        # magnitudes over 40 powers of two within tiles
        b = b * np.exp2(rng.uniform(-40, 0, size=shape))
    elif kind == "point":       # zero outside a few cells
        b = np.where((np.abs(x - 0.3) < 0.02) & (np.abs(y - 0.6) < 0.03) & (np.abs(z - 0.4) < 0.03), b, 0.0)
    return b - b.mean() if kind != "point" else b


@pytest.mark.parametrize("topology,n,kind", [
    ("closed", (64, 64, 64), "smooth"), ("perio_xyz", (64, 64, 64), "spread"), ("perio_xy", (64, 64, 64), "point"),
    ("perio_x", (128, 40, 56), "smooth"), ("closed", (48, 104, 56), "spread"), ("perio_xyz", (80, 60, 60), "smooth"),
    ("perio_y", (32, 128, 128), "point"),
    # 8 coarse planes per thread in the prolongation into level 0, the last thread 4
    ("perio_xyz", (264, 264, 152), "smooth"), ("closed", (264, 264, 152), "smooth")])
def test_fx_vcycle_against_oracle(topology, n, kind):
    from nyles_gb300.multigrid import MG
    nx, ny, nz = n
    mg = MG(nx, ny, nz, topology=topology, precision="fp64")
    o = oracle.OracleMG(nx, ny, nz, TOPO[topology])
    rng = np.random.Generator(np.random.PCG64(nx + 1000 * ny))
    b = _rhs(kind, (nz, ny, nx), rng)
    x0 = 0.1 * _rhs("smooth", (nz, ny, nx), rng)
    for var, a in ((1, x0), (2, b)):
        mg.set(1, var, torch.from_numpy(a))
        for axis, key in ((2, "x"), (1, "y"), (0, "z")):     # mgfor's ghosts: periodic image, or 0
            pad = [(0, 0)] * 3
            pad[axis] = (3, 3)
            a = np.pad(a, pad, mode="wrap" if key in topology[5:] else "constant")
        o.set(var, a)
    mg.set_params(1e-30, 1, 0.9)
    o.params(1e-30, 1, 0.9)
    x, _ = mg.solve()
    torch.cuda.synchronize()
    o.solve()
    ref = o.get(1)[3:-3, 3:-3, 3:-3]
    assert np.max(np.abs(x.cpu().numpy() - ref)) <= 1e-13 * np.max(np.abs(ref))
