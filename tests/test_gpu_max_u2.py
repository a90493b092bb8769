"""max(U^2 + V^2 + W^2) of FP32 velocities, whose kernel forms a cell's sum in double only where
its FP32 sum may be the largest: equal to the FP64 maximum of the same values, bit for bit.
"""
import numpy as np
import pytest

import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (64, 32, 16), (128, 128, 64)])
@pytest.mark.parametrize("kind", ["random", "ties", "growing", "huge", "tiny", "denormal", "zero", "nan", "inf"])
def test_max_u2(kind, n):
    from nyles_gb300._native import BlowUp
    from nyles_gb300.nyles import Nyles
    m = Nyles(helpers.make_params(geometry="perio_xy", n=n, precision="mixed")).model
    rng = np.random.Generator(np.random.PCG64(n[0]))
    shape = tuple(m.state.get("U_i").view("i").shape)
    v = rng.standard_normal((3,) + shape).astype(np.float32)
    flat = v.reshape(3, -1)
    if kind == "ties":          # sums equal to a few units of FP32 rounding, in any order
        t = rng.uniform(0, 6.3, flat.shape[1])
        flat[:] = np.stack([np.cos(t), np.sin(t), 0 * t]) * (1 + 1e-7 * rng.standard_normal(t.size))
    elif kind == "growing":     # every cell a new maximum
        flat[:] = np.linspace(0.5, 1.5, flat.shape[1])
    elif kind in ("huge", "tiny", "denormal"):
        flat *= {"huge": 1e25, "tiny": 1e-25, "denormal": 1e-40}[kind]
    elif kind == "zero":
        flat[:] = 0.0
    elif kind in ("nan", "inf"):
        flat[1, -1] = np.float32(kind)
    for a, name in zip(v, ("U_i", "U_j", "U_k")):
        m.state.get(name).view("i")[...] = torch.from_numpy(a).cuda()
    d = v.astype(np.float64)
    ref = np.max((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])
    if not np.isfinite(ref):
        with pytest.raises(BlowUp):
            m.max_U2()
        return
    assert float(m.max_U2()) == ref
