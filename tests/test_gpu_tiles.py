"""Tile shapes of the patch kernel (GPU required): every variant of every
patch size meets the same parity bar against the oracle, and the autotuner
measures them and installs a choice per goal."""
import numpy as np
import pytest

import geoflood_gb300 as gf
from geoflood_gb300 import synth

from test_gpu_patch import compare, level_vs_oracle, random_state

pytestmark = pytest.mark.gpu


def variants(m):
    return range(gf.Context.tile_count(m))


@pytest.mark.parametrize("m", [8, 16, 32])
def test_every_tile_meets_the_parity_bar(ctx, m):
    keep = gf.Context.tile(m, 0)
    try:
        for v in variants(m):
            gf.Context.set_tile(m, 0, v)
            q, aux = random_state(24, m, 40 + v)
            out, ref, cg, cr, pg, pr = level_vs_oracle(ctx, q, aux, m, 2.0, 0.04, gf.Phys())
            compare(q, out, ref, cg, cr, m, pcfl_gpu=pg, pcfl_ref=pr)
            q, aux, _, _ = synth.uniform_dam_break_level(4, 4, m, 1.0, seed=v, x_dam=1.5 * m)
            out, ref, cg, cr, pg, pr = level_vs_oracle(ctx, q, aux, m, 1.0, 0.05, gf.Phys())
            compare(q, out, ref, cg, cr, m, pcfl_gpu=pg, pcfl_ref=pr)
    finally:
        gf.Context.set_tile(m, 0, keep)


@pytest.mark.parametrize("m", [8, 16, 32])
def test_tile_shapes_give_the_same_bits(ctx, m):
    """Threads per patch, slices per band and the split of one patch over a
    thread-block cluster change the work split, not the sums: every
    variant's step equals variant 0's bit for bit."""
    keep = gf.Context.tile(m, 0)
    outs = []
    try:
        for v in variants(m):
            gf.Context.set_tile(m, 0, v)
            q, aux, _, _ = synth.uniform_dam_break_level(4, 4, m, 1.0, seed=7, x_dam=1.5 * m)
            out, _, cg, _, pg, _ = level_vs_oracle(ctx, q, aux, m, 1.0, 0.05, gf.Phys())
            outs.append((out, cg, pg))
    finally:
        gf.Context.set_tile(m, 0, keep)
    for out, cg, pg in outs[1:]:
        assert np.array_equal(out, outs[0][0]) and cg == outs[0][1]
        assert np.array_equal(pg, outs[0][2])


@pytest.mark.parametrize("m,npx", [(16, 1), (16, 38), (16, 39), (16, 76), (16, 77), (16, 152), (16, 153),
                                   (32, 19), (32, 20), (32, 38), (32, 39), (32, 76), (32, 77)])
def test_tile_by_the_number_of_patches_gives_the_same_bits(ctx, m, npx):
    """Without a choice by hand the tile follows the launch's number of
    patches: either side of each switch gives the bits of one fixed tile."""
    keep, other = gf.Context.tile(m, 0), 2
    q, aux, _, _ = synth.uniform_dam_break_level(npx, 1, m, 1.0, seed=npx, x_dam=0.4 * m * npx)
    assert keep != other
    auto = level_vs_oracle(ctx, q, aux, m, 1.0, 0.05, gf.Phys())
    try:
        gf.Context.set_tile(m, 0, other)
        one = level_vs_oracle(ctx, q, aux, m, 1.0, 0.05, gf.Phys())
    finally:
        gf.Context.set_tile(m, 0, keep)
    compare(q, auto[0], auto[1], auto[2], auto[3], m, pcfl_gpu=auto[4], pcfl_ref=auto[5])
    assert np.array_equal(auto[0], one[0]) and auto[2] == one[2] and np.array_equal(auto[4], one[4])


@pytest.mark.parametrize("m,npx", [(8, 38), (8, 39), (16, 304), (16, 305), (32, 266), (32, 267), (32, 304), (32, 305)])
def test_tile_switches_of_wider_launches_give_the_same_bits(ctx, m, npx):
    """Either side of the remaining switches: the bits of one fixed tile."""
    keep, other = gf.Context.tile(m, 0), 2 if m == 16 else 0
    assert keep != other
    q, aux, _, _ = synth.uniform_dam_break_level(npx, 1, m, 1.0, seed=npx, x_dam=0.4 * m * npx)
    ctx.set_phys(0, gf.Phys())
    outs = []
    try:
        for v in (keep, other):
            gf.Context.set_tile(m, 0, v)
            lev = gf.Level(ctx, npx, m, 1)
            lev.set_geometry(1.0, 1.0)
            lev.upload(q, aux)
            cfl = lev.step(0.0, 0.05)
            outs.append((lev.download(), cfl, lev.patch_cfl()))
            lev.close()
    finally:
        gf.Context.set_tile(m, 0, keep)
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
    assert np.array_equal(outs[0][2], outs[1][2])


@pytest.mark.parametrize("m", [8, 16, 32])
def test_every_switch_of_the_tile_gives_the_same_bits(ctx, m):
    """The numbers of patches at which the tile changes, clusters resident at
    once on this device among them: either side has the bits of one fixed tile."""
    keep = gf.Context.tile(m, 0)
    gf.Context.set_tile(m, 0, gf.TILE_AUTO)
    try:
        of = [gf.Context.tile_of(m, n) for n in range(1, 1001)]
        counts = [n + d for n in range(1, 1000) if of[n - 1] != of[n] for d in (0, 1)]
        assert len(counts) >= 2
        q, aux, _, _ = synth.uniform_dam_break_level(32, -(-max(counts) // 32), m, 1.0, seed=m, x_dam=12.8 * m)
        ctx.set_phys(0, gf.Phys())
        for n in counts:
            outs = []
            for v in (gf.TILE_AUTO, 2 if m == 16 else 0):
                gf.Context.set_tile(m, 0, v)
                lev = gf.Level(ctx, n, m, 1)
                lev.set_geometry(1.0, 1.0)
                lev.upload(np.ascontiguousarray(q[:n]), np.ascontiguousarray(aux[:n]))
                cfl = lev.step(0.0, 0.05)
                outs.append((lev.download(), cfl, lev.patch_cfl()))
                lev.close()
            assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
            assert np.array_equal(outs[0][2], outs[1][2])
    finally:
        gf.Context.set_tile(m, 0, keep)


@pytest.mark.parametrize("m", [8, 16, 32])
@pytest.mark.parametrize("kind", ["band", "row", "thin"])
def test_dry_rows_and_windows(ctx, m, kind):
    """Water in some rows only (a band of rows at every height, a single row at
    every place from ghost to ghost, depths below the tolerance with momentum):
    rows that a tile passes over, or windows of a split patch without water,
    come out as the oracle's, and as the same bits from every tile."""
    n = m + 4
    q, aux = random_state(n, m, 60 + m)
    for k in range(n):
        lo, hi = (k, min(k + 1, n)) if kind == "row" else (k // 2, min(k // 2 + 1 + k % 7, n))
        if kind == "thin":
            q[k, :lo, :, 0] = np.minimum(q[k, :lo, :, 0], 5e-4)
            q[k, hi:, :, 0] = np.minimum(q[k, hi:, :, 0], 1e-3)
        else:
            q[k, :lo] = 0.0
            q[k, hi:] = 0.0
    keep = gf.Context.tile(m, 0)
    outs = []
    try:
        for v in variants(m):
            gf.Context.set_tile(m, 0, v)
            out, ref, cg, cr, pg, pr = level_vs_oracle(ctx, q, aux, m, 2.0, 0.02, gf.Phys())
            compare(q, out, ref, cg, cr, m, pcfl_gpu=pg, pcfl_ref=pr)
            outs.append((out, cg, pg))
    finally:
        gf.Context.set_tile(m, 0, keep)
    for out, cg, pg in outs[1:]:
        assert np.array_equal(out, outs[0][0]) and cg == outs[0][1]
        assert np.array_equal(pg, outs[0][2])


def test_autotune_measures_and_selects(ctx):
    ctx.set_phys(0, gf.Phys())
    res = ctx.autotune(reps=2)
    assert [r["mx"] for r in res] == [8, 16, 32]
    for r in res:
        assert len(r["tiles"]) == len(variants(r["mx"]))
        assert all(v > 0 for v in r["throughput"]) and all(v > 0 for v in r["latency_us"])
        assert r["best_throughput"] == int(np.argmax(r["throughput"]))
        assert r["best_latency"] == int(np.argmin(r["latency_us"]))
        assert gf.Context.tile(r["mx"], 0) == r["best_throughput"]
        assert gf.Context.tile(r["mx"], 1) == r["best_latency"]
    with pytest.raises(gf.GeoFloodError):
        gf.Context.set_tile(8, 0, 9)


def test_autotune_leaves_smaller_launches_to_their_number_of_patches(ctx):
    """The throughput choice is that of a level of 4M cells: it serves launches of
    that size, and smaller ones take the tiles they take without it."""
    counts = (1, 100, 247, 300, 400, 760, 911, 1073, 4095)
    try:
        for m in (8, 16, 32):
            for goal in (0, 1):
                gf.Context.set_tile(m, goal, gf.TILE_AUTO)
        before = [[gf.Context.tile_of(m, n) for n in counts] for m in (8, 16, 32)]
        ctx.set_phys(0, gf.Phys())
        res = ctx.autotune(reps=1)
        assert [[gf.Context.tile_of(m, n) for n in counts] for m in (8, 16, 32)] == before
        for r in res:
            assert gf.Context.tile_of(r["mx"], (4 << 20) // r["mx"] ** 2) == r["best_throughput"]
            assert gf.Context.tile_of(r["mx"], 8, 1) == r["best_latency"]
    finally:
        for m in (8, 16, 32):
            for goal in (0, 1):
                gf.Context.set_tile(m, goal, gf.TILE_AUTO)


@pytest.mark.parametrize("m", [8, 16, 32])
def test_small_host_batches_take_the_latency_tile_with_the_same_bits(ctx, m):
    """gf_patch_update_batch on a handful of patches runs the latency
    choice (a patch split over a cluster for the window tiles): every
    variant installed there gives the bits of the one-CTA kernel."""
    keep = gf.Context.tile(m, 1)
    q, aux, _, _ = synth.uniform_dam_break_level(2, 2, m, 1.0, seed=5, x_dam=1.0 * m)
    outs = []
    try:
        for v in variants(m):
            gf.Context.set_tile(m, 1, v)
            qs = [np.array(q[k]) for k in range(4)]
            cfl, mc = ctx.patch_update_batch(qs, [np.ascontiguousarray(aux[k]) for k in range(4)],
                                             1.0, 1.0, 0.0, 0.05)
            outs.append((np.stack(qs), cfl, mc))
    finally:
        gf.Context.set_tile(m, 1, keep)
    for out, cfl, mc in outs[1:]:
        assert np.array_equal(out, outs[0][0])
        assert np.array_equal(cfl, outs[0][1]) and mc == outs[0][2]
