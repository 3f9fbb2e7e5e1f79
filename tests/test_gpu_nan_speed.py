"""A cell whose velocity is not a number takes no part in a patch's CFL (GPU
required): the largest speed of the other faces is reported, whichever faces
a thread happens to solve."""
import numpy as np
import pytest

import geoflood_gb300 as gf

pytestmark = pytest.mark.gpu


def cfl_of(ctx, q, aux, m):
    lev = gf.Level(ctx, q.shape[0], m, 1)
    lev.set_geometry(1.0, 1.0)
    lev.upload(q, aux)
    cfl = lev.step(0.0, 0.01)
    out = cfl, lev.patch_cfl()
    lev.close()
    return out


@pytest.mark.parametrize("m", [8, 16, 32])
@pytest.mark.parametrize("side", ["x", "y"])
def test_a_nan_speed_is_left_out_of_the_cfl(ctx, m, side):
    """Calm water with one fast cell in every patch and NaN momenta in half of
    it, away from the fast cell: the CFLs of the patches without the NaN."""
    n = m + 4
    q = np.zeros((24, n, n, 3))
    q[..., 0] = 2.0
    for k in range(len(q)):
        j, i = 3 + k % (m - 2), m // 2 + 6 if m > 8 else 9
        q[k, j, i] = (2.0, 16.0 + k, 0.0)
    bad = q.copy()
    bad[:, :, : m // 2 + (4 if m > 8 else 2), 1] = np.nan
    if side == "y":
        q, bad = (np.ascontiguousarray(a.transpose(0, 2, 1, 3)[..., [0, 2, 1]]) for a in (q, bad))
    aux = np.zeros(q.shape[:3] + (1,))
    ctx.set_phys(0, gf.Phys())
    keep = gf.Context.tile(m, 0)
    try:
        for v in range(gf.Context.tile_count(m)):
            gf.Context.set_tile(m, 0, v)
            want, got = cfl_of(ctx, q, aux, m), cfl_of(ctx, bad, aux, m)
            assert want[0] > 0.0 and got[0] == want[0]
            assert np.array_equal(got[1], want[1])
    finally:
        gf.Context.set_tile(m, 0, keep)
