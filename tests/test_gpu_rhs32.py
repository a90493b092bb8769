"""The FP32 right-hand side (nyles_rhs_f32) at extents that end inside a block's 32 x 8 columns and
inside a thread's planes, at their edges and at the shortest lines, with a tracer and
viscosity, against the FP64 oracle on the same (FP32) inputs.

Bar: 2e-5 of a field's max-norm. A register sums at most nine fluxes and three diffusion terms of
the field's own size; a flux is about 30 operations of 6e-8 each: 12 x 30 x 6e-8 = 2.2e-5 if all
errors added up.
"""
import ctypes

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FIELDS = ["b", "p", "ke", "div", "u_i", "u_j", "u_k", "U_i", "U_j", "U_k", "vor_i", "vor_j", "vor_k", "work"]


@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("geometry,n", [("closed", (5, 6, 7)), ("closed", (33, 5, 9)), ("closed", (32, 17, 5)),
                                        ("closed", (65, 8, 35)), ("perio_xy", (26, 35, 6)),
                                        ("perio_xyz", (7, 6, 9)), ("perio_x", (59, 16, 18)),
                                        ("closed", (1201, 35, 26)), ("perio_xy", (27, 200, 190)),
                                        ("perio_xyz", (130, 101, 79))])
def test_rhs_f32_any_extents(geometry, n, last):
    from nyles_gb300 import _native as nat
    nx, ny, nz = n
    h, visc = 0.1, 2e-3
    o = oracle.OracleModel(dict(nx=nx, ny=ny, nz=nz, nh=3, geometry=geometry, n_tracers=1, modelname="LES",
                                timestepping="RK3_SSP", dx=h, dy=h, dz=h, idx2=h ** -2, idy2=h ** -2, idz2=h ** -2,
                                fparam=0.0, visc=visc, tracer_diffusion=None, tracer_order=0, vf_order=0))
    d = nat.NylesDesc()
    d.nx, d.ny, d.nz, d.nh, d.n_tracers = nx, ny, nz, 3, 1
    d.periodic_x, d.periodic_y, d.periodic_z = (int(a in geometry[5:]) if geometry != "closed" else 0 for a in "xyz")
    d.dx = d.dy = d.dz = h
    d.idx2 = d.idy2 = d.idz2 = h ** -2
    d.dx2 = h ** 2
    d.add_viscosity, d.viscosity = 1, visc
    rng = np.random.Generator(np.random.PCG64(nx * 10000 + ny * 100 + nz))
    dev = []
    for name in FIELDS + ["t0"]:
        a = rng.standard_normal(o.field(name).shape).astype(np.float32)
        if name in ("b", "vor_j"):
            a[: a.shape[0] // 2] = 0.75          # constant lines: every indicator at its floor
        if name == "U_j":
            a[:, :, ::3] = 0.0                   # no upwind side
        o.field(name)[...] = a
        dev.append(torch.from_numpy(a).cuda())
    out = [torch.full_like(dev[0], 7.0) for _ in range(5)]
    nat.check(nat.lib().nyles_rhs_f32(ctypes.byref(d), nat.ptr_array([t.data_ptr() for t in dev]),
                                      nat.ptr_array([t.data_ptr() for t in out]), int(last), nat.stream_ptr()))
    torch.cuda.synchronize()
    o.rhs(1, last)
    for q, name in enumerate(["b", "u_i", "u_j", "u_k", "t0"]):
        ref = o.register(1, q)
        err = np.max(np.abs(out[q].cpu().numpy() - ref)) / np.max(np.abs(ref))
        assert err < 2e-5, (name, err)
