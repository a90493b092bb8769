"""The line-marching FP64 right-hand side on fields with NaN, infinities and large values: a register is finite where
the oracle's is, and equal to it there within 1e-13 of the register's largest finite value (as for ordinary fields:
the operations are the same).
"""
import ctypes

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FIELDS = ["b", "p", "ke", "div", "u_i", "u_j", "u_k", "U_i", "U_j", "U_k", "vor_i", "vor_j", "vor_k", "work"]


@pytest.mark.parametrize("geometry,n", [("closed", (33, 18, 21)), ("perio_xyz", (14, 9, 24))])
@pytest.mark.parametrize("kind", ["nan", "inf", "large"])
def test_values(kind, geometry, n):
    from nyles_gb300 import _native as nat
    nx, ny, nz = n
    h = 0.1
    o = oracle.OracleModel(dict(nx=nx, ny=ny, nz=nz, nh=3, geometry=geometry, n_tracers=1, modelname="LES",
                                timestepping="RK3_SSP", dx=h, dy=h, dz=h, idx2=h ** -2, idy2=h ** -2, idz2=h ** -2,
                                fparam=0.0, visc=0.0, tracer_diffusion=None, tracer_order=0, vf_order=0))
    d = nat.NylesDesc()
    d.nx, d.ny, d.nz, d.nh, d.n_tracers = nx, ny, nz, 3, 1
    d.periodic_x = d.periodic_y = d.periodic_z = int(geometry == "perio_xyz")
    d.dx = d.dy = d.dz = h
    d.idx2 = d.idy2 = d.idz2 = h ** -2
    d.dx2 = h ** 2
    rng = np.random.Generator(np.random.PCG64(11))
    dev = []
    for name in FIELDS + ["t0"]:
        a = rng.standard_normal(o.field(name).shape)
        if name in ("b", "t0", "vor_i", "vor_j", "vor_k"):
            if kind in ("nan", "inf"):
                at = tuple(rng.integers(0, m, 3) for m in a.shape)      # inside, and on a face
                a[at] = float(kind)
                a[0, at[1][0], at[2][1]] = -float(kind)
            else:
                a *= 1e15
        o.field(name)[...] = a
        dev.append(torch.from_numpy(a).cuda())
    out = [torch.full_like(dev[0], 7.0) for _ in range(5)]
    nat.check(nat.lib().nyles_rhs_f64(ctypes.byref(d), nat.ptr_array([t.data_ptr() for t in dev]),
                                      nat.ptr_array([t.data_ptr() for t in out]), 0, nat.stream_ptr()))
    torch.cuda.synchronize()
    o.rhs(1, False)
    for q, name in enumerate(["b", "u_i", "u_j", "u_k", "t0"]):
        ref, got = o.register(1, q), out[q].cpu().numpy()
        ok = np.isfinite(ref)
        assert ok.any() and (kind == "large" or not ok.all())
        np.testing.assert_array_equal(np.isfinite(got), ok, err_msg=name)
        err = np.max(np.abs(got[ok] - ref[ok])) / np.max(np.abs(ref[ok]))
        assert err < 1e-13, (name, err)
