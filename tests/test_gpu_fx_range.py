"""The FP64 multigrid levels summed in integers at the ends of the double range: a sum that overflows in
doubles, infinities and NaN end the solve with an error, as on levels summed in doubles.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(64, 64, 64), (32, 32, 32)])     # integer sums, double sums
@pytest.mark.parametrize("kind", ["overflow", "nan", "inf"])
def test_solve_reports_values_beyond_the_range(kind, n):
    from nyles_gb300._native import BlowUp
    from nyles_gb300.multigrid import MG
    nx, ny, nz = n
    mg = MG(nx, ny, nz, topology="perio_xyz", precision="fp64")
    rng = np.random.Generator(np.random.PCG64(3))
    b = rng.standard_normal((nz, ny, nx))
    x = np.zeros((nz, ny, nx))
    if kind == "overflow":
        x[...] = 1.5 * 2.0 ** 1022          # 6 x is beyond the doubles
    else:
        x[nz // 2, ny // 2, nx // 2] = float(kind)
    mg.set(1, 1, torch.from_numpy(x))
    mg.set(1, 2, torch.from_numpy(b - b.mean()))
    mg.set_params(1e-30, 1, 0.9)
    with pytest.raises(BlowUp):
        mg.solve()
