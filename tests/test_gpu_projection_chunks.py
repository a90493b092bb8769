"""The projection (divergence, pressure solve, correction) at grids where its columns hold one,
two, four and eight planes, the last column short: against the oracle in FP64, against the FP64
model in mixed precision.

Bars: 1e-12 as a step of the FP64 model against the oracle; mixed: a float-pair divergence, a
solve to sum(r^2) < 1e-6 sum(b^2) that stops at the same iteration, and velocities stored in FP32
(6e-8 each): 1e-5, as the mixed steps'.
"""
import pytest

import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry,n", [("closed", (48, 32, 16)), ("perio_xy", (64, 128, 64)), ("perio_xyz", (96, 96, 96)),
                                        ("perio_xyz", (128, 128, 128))])
def test_projection(geometry, n):
    from nyles_gb300.nyles import Nyles
    names = ["u_i", "u_j", "u_k", "p"]
    L = tuple(float(k) / n[2] for k in n)
    nyl = Nyles(helpers.make_params(geometry=geometry, n=n, L=L))
    o = helpers.oracle_for(nyl)
    fields = helpers.seeded_state(nyl, "noise", 5)
    helpers.load_state(nyl, o, fields)
    nyl.model.diagnose_var(nyl.model.state)
    o.diagnose()
    errs = helpers.parity_errors(lambda s: nyl.model.state.get(s).view("i").cpu().numpy(), o.field, names)
    assert max(errs.values()) < 1e-12, errs
    mix = Nyles(helpers.make_params(geometry=geometry, n=n, L=L, precision="mixed"))
    for k, v in fields.items():
        mix.model.state.get(k).view("i")[...] = torch.from_numpy(v)
    mix.model.diagnose_var(mix.model.state)
    assert mix.model.mg_stats()["nite"] == nyl.model.mg_stats()["nite"]
    errs = helpers.parity_errors(lambda s: mix.model.state.get(s).view("i").double().cpu().numpy(), o.field, names)
    assert max(errs.values()) < 1e-5, errs
