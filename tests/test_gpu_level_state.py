"""A level before its first step (GPU required)."""
import numpy as np
import pytest

import geoflood_gb300 as gf
from geoflood_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [8, 16])
def test_a_wait_before_the_first_step_finds_no_cfl_and_no_error(ctx, m):
    """Levels made where others were, with their CFLs and sums in the memory they
    left: a ghost fill and a wait report no error, no CFL and a still state."""
    n = 8
    q, aux, py, px = synth.uniform_dam_break_level(4, 2, m, 1.0, seed=3, x_dam=2.0 * m)
    nbr, xl, yl = synth.brick_layout(py, px, m, 1.0)
    ctx.set_phys(0, gf.Phys())
    for k in range(6):
        used = [gf.Level(ctx, n, m, 1) for _ in range(k + 1)]
        for lev in used:
            lev.set_geometry(1.0, 1.0)
            lev.upload(q, aux)
            assert lev.step(0.0, 0.05) > 0.0
        for lev in used:
            lev.close()
        fresh = [gf.Level(ctx, n, m, 1) for _ in range(k + 1)]
        for lev in fresh:
            lev.set_geometry(1.0, 1.0)
            lev.set_layout(nbr, xl, yl)
            lev.ghost_fill_async(0.0)
            assert lev.sync() == 0.0
            assert not lev.patch_cfl().any()
            assert not lev.download().any() and not lev.download_aux().any()
        for lev in fresh:
            lev.close()
