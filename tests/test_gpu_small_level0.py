"""Level-0 kernels of the mixed solver on small and on narrow grids: the half-sweeps and transfers
with one plane per thread (extents that the four-plane kernels do not take among them), and the
Krylov sums where level 0 has more blocks than the workspace has slots for their partials.

Bars: one V-cycle in FP32 from zero, about 60 operations per value of 6e-8 each, 4e-6 of max|x|;
a solve to sum(r^2) < 1e-20 sum(b^2): the residual in FP64, 1.1e-20 (storing x as float pairs moves r
by about 1e-14 |x|, below 1e-11 of |b| on these grids).
"""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOPO = {"closed": 1, "perio_x": 2, "perio_y": 3, "perio_xy": 5, "perio_xyz": 6}


def _rhs(nx, ny, nz):
    b = np.random.Generator(np.random.PCG64(nx + 100 * ny + 10000 * nz)).standard_normal((nz, ny, nx))
    return b - b.mean()


@pytest.mark.parametrize("topology,n", [
    ("closed", (12, 6, 6)), ("perio_xyz", (12, 22, 10)),     # planes that are no multiple of 4
    ("perio_xy", (100, 36, 44)), ("perio_x", (132, 20, 4)),  # idle lanes, two blocks along x
    ("perio_y", (64, 64, 128)), ("closed", (10, 12, 8))])    # nx % 4: the scalar kernels
def test_cycle_against_oracle(topology, n):
    from nyles_gb300.multigrid import MG
    nx, ny, nz = n
    b = _rhs(nx, ny, nz)
    mg = MG(nx, ny, nz, topology=topology, precision="mixed")
    o = oracle.OracleMG(nx, ny, nz, TOPO[topology])
    mg.set(1, 2, torch.from_numpy(b))
    full = b
    for axis, key in ((2, "x"), (1, "y"), (0, "z")):
        pad = [(0, 0)] * 3
        pad[axis] = (3, 3)
        full = np.pad(full, pad, mode="wrap" if key in topology[5:] else "constant")
    o.set(2, full)
    mg.set_params(1e-30, 1, 0.9)
    o.params(1e-30, 1, 0.9)
    x, _ = mg.solve()
    torch.cuda.synchronize()
    o.solve()
    ref = o.get(1)[3:-3, 3:-3, 3:-3]
    assert np.max(np.abs(x.double().cpu().numpy() - ref)) <= 4e-6 * np.max(np.abs(ref))


def _laplacian(x, topology):
    """sum of the wet neighbours minus their number times x"""
    out = np.zeros_like(x)
    for axis, key in ((2, "x"), (1, "y"), (0, "z")):
        d = np.roll(x, -1, axis) - x      # towards the next cell; the last one's is the wrap
        if key not in topology[5:]:
            d[tuple(slice(-1, None) if a == axis else slice(None) for a in range(3))] = 0.0
        out += d - np.roll(d, 1, axis)
    return out


@pytest.mark.parametrize("topology,n", [("perio_xyz", (32, 32, 64)), ("closed", (16, 16, 64)), ("perio_xy", (8, 8, 32)),
                                        ("closed", (4, 4, 16)), ("perio_x", (32, 30, 60)), ("closed", (128, 32, 32))])
def test_krylov_on_narrow_grids(topology, n):
    from nyles_gb300.multigrid import MG
    nx, ny, nz = n
    b = _rhs(nx, ny, nz)
    mg = MG(nx, ny, nz, topology=topology, precision="mixed")
    mg.set_params(1e-20, 400, 0.9)
    mg.set_krylov(True)
    x, st = mg.solve(b)
    assert st["nite"] < 400
    r = b - _laplacian(x.double().cpu().numpy(), topology)
    assert np.sum(r * r) <= 1.1e-20 * np.sum(b * b)
