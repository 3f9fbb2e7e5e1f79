"""A level before its first step (GPU required)."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import geoflood_gb300 as gf
from geoflood_gb300 import synth

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


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


WORKER = """
import sys
import numpy as np
import geoflood_gb300 as gf

ctx = gf.Context(0, gf.Phys())
r = np.random.default_rng(int(sys.argv[1]))
for k in range(120):
    m, n = (8, 16, 32)[k % 3], int(r.integers(1, 100))
    q = np.zeros((n, m + 4, m + 4, 3))
    q[..., 0] = 1.0
    aux = r.random((n, m + 4, m + 4, 1 + k % 3))
    lev = gf.Level(ctx, n, m, 1 + k % 3)
    lev.set_geometry(1.0, 1.0)
    lev.upload(q, aux)
    lev.step(0.0, 1e-9)
    assert np.array_equal(lev.download_aux(), aux), k
    assert (lev.download()[..., 0] > 0.99).all(), k
    lev.close()
"""


def test_an_upload_into_a_new_level_stays_on_a_shared_device(gpu_lib):
    """Four programs share the device and make level after level: each finds the
    state that it uploaded."""
    run = [subprocess.Popen([sys.executable, "-c", WORKER, str(k)], cwd=ROOT) for k in range(4)]
    assert [p.wait(timeout=300) for p in run] == [0] * 4
