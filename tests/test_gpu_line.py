"""The line-marching FP64 right-hand side (nyles_rhs_f64) at extents that end inside a
thread's chunk, at its edges and at the shortest lines, closed and periodic, with tracer
diffusion and viscosity, against the oracle.

Bar: 1e-13 of a field's max-norm. A register sums at most nine fluxes and six diffusion
terms of the field's own size; a flux is about 30 operations on positive weights and on
differences, each rounding to 1.1e-16 of its result: 15 x 30 x 1.1e-16 = 5e-14.
"""
import ctypes

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FIELDS = ["b", "p", "ke", "div", "u_i", "u_j", "u_k", "U_i", "U_j", "U_k", "vor_i", "vor_j", "vor_k", "work"]


@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("geometry,n", [("closed", (5, 6, 7)), ("closed", (33, 5, 9)), ("closed", (8, 65, 5)),
                                        ("closed", (12, 7, 67)), ("closed", (67, 34, 31)), ("perio_xy", (11, 27, 6)),
                                        ("perio_xyz", (6, 7, 8)), ("perio_x", (26, 33, 5))])
def test_rhs_f64_any_extents(geometry, n, last):
    from nyles_gb300 import _native as nat
    nx, ny, nz = n
    ntr, h, visc = 1, 0.1, 2e-3
    kd = {"b": 3e-3, "t0": 5e-3}
    o = oracle.OracleModel(dict(nx=nx, ny=ny, nz=nz, nh=3, geometry=geometry, n_tracers=ntr, modelname="LES",
                                timestepping="RK3_SSP", dx=h, dy=h, dz=h, idx2=h ** -2, idy2=h ** -2, idz2=h ** -2,
                                fparam=0.0, visc=visc, tracer_diffusion=kd, tracer_order=0, vf_order=0))
    d = nat.NylesDesc()
    d.nx, d.ny, d.nz, d.nh, d.n_tracers = nx, ny, nz, 3, ntr
    d.periodic_x, d.periodic_y, d.periodic_z = (int(a in geometry[5:]) if geometry != "closed" else 0 for a in "xyz")
    d.dx = d.dy = d.dz = h
    d.idx2 = d.idy2 = d.idz2 = h ** -2
    d.dx2 = h ** 2
    d.add_viscosity, d.viscosity = 1, visc
    d.tracer_diffusion = 3
    d.tracer_diffusivity[0], d.tracer_diffusivity[1] = kd["b"], kd["t0"]
    rng = np.random.Generator(np.random.PCG64(nx * 10000 + ny * 100 + nz))
    dev = []
    for name in FIELDS + ["t0"]:
        a = rng.standard_normal(o.field(name).shape)
        if name.startswith("vor"):
            a *= np.exp(rng.uniform(-6, 0, size=a.shape))
        if name in ("b", "vor_j"):
            a[: a.shape[0] // 2] = 0.75          # constant lines: every indicator at its floor
        if name == "U_j":
            a[:, :, ::3] = 0.0                   # no upwind side
        o.field(name)[...] = a
        dev.append(torch.from_numpy(a).cuda())
    out = [torch.full_like(dev[0], 7.0) for _ in range(5)]
    nat.check(nat.lib().nyles_rhs_f64(ctypes.byref(d), nat.ptr_array([t.data_ptr() for t in dev]),
                                      nat.ptr_array([t.data_ptr() for t in out]), int(last), nat.stream_ptr()))
    torch.cuda.synchronize()
    o.rhs(1, last)
    for q, name in enumerate(["b", "u_i", "u_j", "u_k", "t0"]):
        ref = o.register(1, q)
        err = np.max(np.abs(out[q].cpu().numpy() - ref)) / np.max(np.abs(ref))
        assert err < 1e-13, (name, err)
