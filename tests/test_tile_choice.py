"""The choice of a launch's tile (gf_tile_set, gf_tile_of): a variant pinned by
hand is the one that every launch takes, the variants that launches take by
themselves included."""
import pytest

import geoflood_gb300 as gf

COUNTS = (1, 12, 19, 20, 36, 153, 400, 1073, 6000)


@pytest.mark.parametrize("m", [8, 16, 32])
@pytest.mark.parametrize("goal", [0, 1])
def test_a_pinned_tile_is_taken_by_every_launch(gpu_lib, m, goal):
    keep = gf.Context.tile(m, goal)
    try:
        for v in range(gf.Context.tile_count(m)):
            gf.Context.set_tile(m, goal, v)
            assert gf.Context.tile(m, goal) == v
            assert [gf.Context.tile_of(m, n, goal) for n in COUNTS] == [v] * len(COUNTS)
    finally:
        gf.Context.set_tile(m, goal, keep)


@pytest.mark.parametrize("m", [8, 16, 32])
def test_a_choice_by_hand_is_taken_back(gpu_lib, m):
    gf.Context.set_tile(m, 0, gf.TILE_AUTO)
    auto = [gf.Context.tile_of(m, n) for n in COUNTS]
    gf.Context.set_tile(m, 0, 1)
    gf.Context.set_tile(m, 0, gf.TILE_AUTO)
    assert gf.Context.tile(m, 0) == gf.TILE_AUTO
    assert [gf.Context.tile_of(m, n) for n in COUNTS] == auto


def test_tile_arguments(gpu_lib):
    for bad in (-1, 9, gf.TILE_AUTO - 1):
        with pytest.raises(gf.GeoFloodError):
            gf.Context.set_tile(8, 0, bad)
    with pytest.raises(gf.GeoFloodError):
        gf.Context.tile_of(12, 1)
    with pytest.raises(gf.GeoFloodError):
        gf.Context.tile_of(8, 0)
    with pytest.raises(gf.GeoFloodError):
        gf.Context.tile_shape(8, 99)
    assert gf.Context.tile_shape(32, 1) == (256, 4, 1)
