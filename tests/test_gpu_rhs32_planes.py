"""The FP32 right-hand side on planes so large that a block's reach in bytes leaves 32 bits (offsets in cells), and in
cells too (fewer planes per thread): equal, bit for bit, to the right-hand side of a small grid of which the large one is
the repetition in x and y (away from the walls, where every cell's stencil is the small grid's).
"""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

USED = ["b", "ke", "U_i", "U_j", "U_k", "vor_i", "vor_j", "vor_k", "t0"]
ORDER = ["b", "p", "ke", "div", "u_i", "u_j", "u_k", "U_i", "U_j", "U_k", "vor_i", "vor_j", "vor_k", "work", "t0"]


def _rhs(fields):
    from nyles_gb300 import _native as nat
    nz, ny, nx = fields["b"].shape
    d = nat.NylesDesc()
    d.nx, d.ny, d.nz, d.nh, d.n_tracers = nx, ny, nz, 3, 1
    d.dx = d.dy = d.dz = 0.1
    d.idx2 = d.idy2 = d.idz2 = 100.0
    d.dx2 = 0.01
    out = [torch.full_like(fields["b"], 7.0) for _ in range(5)]
    nat.check(nat.lib().nyles_rhs_f32(ctypes.byref(d), nat.ptr_array([fields.get(k, fields["b"]).data_ptr() for k in ORDER]),
                                      nat.ptr_array([t.data_ptr() for t in out]), 0, nat.stream_ptr()))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("ny,nx,rep_y,rep_x,nz", [(100, 96, 80, 63, 11),      # 48.4 M cells: bytes, 16 planes
                                                  (100, 96, 82, 64, 11),      # 50.4 M: cells
                                                  (100, 96, 164, 90, 6),      # 141.7 M
                                                  (100, 96, 160, 167, 5)])    # 256.5 M: 8 planes
def test_large_planes_equal_the_small_grid(ny, nx, rep_y, rep_x, nz):
    need = 4 * 15 * nz * ny * nx * rep_y * rep_x
    if torch.cuda.mem_get_info()[0] < 1.2 * need:
        pytest.skip("needs %.0f GB" % (1.2e-9 * need))
    gen = torch.Generator("cuda").manual_seed(nz)
    tile = {k: torch.randn((nz, ny, nx), device="cuda", generator=gen) for k in USED}
    mid = _rhs({k: v.repeat(1, 3, 3) for k, v in tile.items()})
    big = _rhs({k: v.repeat(1, rep_y, rep_x) for k, v in tile.items()})
    for q in range(5):
        ref = mid[q].view(nz, 3, ny, 3, nx)[:, 1, :, 1, :]
        got = big[q].view(nz, rep_y, ny, rep_x, nx)
        for j in range(1, rep_y - 1):
            assert torch.equal(got[:, j, :, 1:-1, :], ref[:, :, None, :].expand(nz, ny, rep_x - 2, nx)), (q, j)
