"""Local accuracy of the FP64 multigrid levels summed in integers (levels of 2^18 cells and more):
the coarse right-hand side after one pre-smoothing and restriction, cell by cell against the
same operations in extended precision, relative to the largest |x| and |b| that reach the cell.

Bar: 1.2e-13 of that largest value M. A double sum of seven values up to M rounds partial sums of up
to 13 M, at most 40 M 2^-53 in all; a half-sweep scales that by omega/diag (8 M 2^-53), and each of two
half-sweeps enters a residual with at most 12 times its error: 232 M 2^-53 a child, 8 children times
0.5: 928 M 2^-53 = 1.03e-13 M, with max|x| growing by at most a sixth of max|b|.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TILE = (8, 8, 32)


def _shift(a, axis, step, periodic):
    """neighbour values along axis (0 outside a closed box)"""
    s = np.roll(a, -step, axis)
    if not periodic:
        edge = [slice(None)] * 3
        edge[axis] = -1 if step > 0 else 0
        s[tuple(edge)] = 0
    return s


def _coarse_rhs(x, b, per, omega=0.9):
    ld = np.longdouble
    x, b = x.astype(ld), b.astype(ld)
    dirs = [(axis, step) for axis in range(3) for step in (-1, 1)]
    diag = sum(_shift(np.ones_like(x), axis, step, per[axis]) for axis, step in dirs)
    nsum = lambda a: sum(_shift(a, axis, step, per[axis]) for axis, step in dirs)
    om = ld(omega)
    for _ in range(2):
        x = (1 - om) * x + (nsum(x) - b) * (om / diag)
    r = b + diag * x - nsum(x)
    nz, ny, nx = r.shape
    return r.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2).sum(axis=(1, 3, 5)) / 2


def _reach(x, b, per):
    """largest |x|, |b| within the four cells that reach a coarse cell's children"""
    m = np.maximum(np.abs(x), np.abs(b))
    for axis in range(3):
        for _ in range(4):
            m = np.maximum(m, np.maximum(_shift(m, axis, -1, per[axis]), _shift(m, axis, 1, per[axis])))
    nz, ny, nx = m.shape
    return m.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2).max(axis=(1, 3, 5))


def _tiles(a, op):
    (nz, ny, nx), (tz, ty, tx) = a.shape, TILE
    return op(a.reshape(nz // tz, tz, ny // ty, ty, nx // tx, tx), axis=(1, 3, 5))


def _magnitude(kind, shape):
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    if kind == "planes":                    # one large plane in 16: most cells of its tile are small
        return np.where(z % 16 == 0, 1.0, 2.0 ** -40)
    if kind == "decay_z":
        return 2.0 ** (-3.0 * z)
    if kind == "decay_y":
        return 2.0 ** (-3.0 * y)
    if kind == "decay_x":
        return 2.0 ** (-1.0 * x)
    if kind == "smooth":
        return np.ones(shape)
    corner = (z < 3) & (y < 5) & (x < 7)
    return np.where(corner, 1.0, {"zero": 0.0, "small": 2.0 ** -45, "tiny": 2.0 ** -950}[kind])


@pytest.mark.parametrize("topology", ["closed", "perio_xyz"])
@pytest.mark.parametrize("kind", ["planes", "decay_z", "decay_y", "decay_x", "smooth", "zero", "small", "tiny"])
def test_coarse_rhs_cell_by_cell(kind, topology):
    from nyles_gb300.multigrid import MG
    nx, ny, nz = 64, 64, 64
    per = [key in topology[5:] for key in "zyx"]
    mg = MG(nx, ny, nz, topology=topology, precision="fp64")
    rng = np.random.Generator(np.random.PCG64(7))
    mag = _magnitude(kind, (nz, ny, nx))
    x, b = (rng.uniform(-1, 1, mag.shape) * mag for _ in range(2))
    top = _tiles(np.maximum(np.abs(x), np.abs(b)), np.max)      # the case is what its name says
    if kind == "zero":
        assert (top == 0.0).any()
    elif kind == "tiny":
        assert ((top > 0.0) & (top < 2.0 ** -895)).any()
    elif kind != "smooth":
        assert (_tiles(_reach(x, b, per).repeat(2, 0).repeat(2, 1).repeat(2, 2), np.min) < 2.0 ** -6 * top).any()
    mg.set(1, 1, torch.from_numpy(x))
    mg.set(1, 2, torch.from_numpy(b))
    mg.set_params(1e-30, 1, 0.9)
    mg.solve()
    torch.cuda.synchronize()
    got = mg.get(2, 2).cpu().numpy()
    err = np.abs(got - _coarse_rhs(x, b, per)).astype(float)
    bar = 1.2e-13 * _reach(x, b, per)
    worst = np.unravel_index(np.argmax(err - bar), err.shape)
    assert (err <= bar).all(), (worst, err[worst], bar[worst])
