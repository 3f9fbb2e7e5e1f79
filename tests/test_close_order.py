"""Levels and forests are destroyed before their context, each once, in whatever
order the program or the collector lets go of them (no GPU: a library that
records the calls)."""
import gc

import pytest

import geoflood_gb300 as gf
from geoflood_gb300 import _lib


class Recorder:
    def __init__(self):
        self.calls, self.made = [], 0

    def _make(self, ref):
        self.made += 1
        ref._obj.value = self.made
        return 0

    def gf_ctx_create(self, device, ref):
        return self._make(ref)

    def gf_ctx_set_phys(self, *a):
        return 0

    def gf_level_create(self, ctx, n, mx, my, maux, ref):
        return self._make(ref)

    def gf_level_destroy(self, h):
        self.calls.append("level")

    def gf_ctx_destroy(self, h):
        self.calls.append("ctx")


@pytest.fixture
def rec(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(_lib, "load", lambda: r)
    return r


def test_collected_together(rec):
    ctx = gf.Context(0)
    box = [ctx, gf.Level(ctx, 1, 8), gf.Level(ctx, 1, 16)]
    box.append(box)
    del box, ctx
    gc.collect()
    assert rec.calls == ["level", "level", "ctx"]


@pytest.mark.parametrize("order", ["level first", "context first", "twice"])
def test_closed_by_hand(rec, order):
    ctx = gf.Context(0)
    lev = gf.Level(ctx, 1, 8)
    if order != "context first":
        lev.close()
    ctx.close()
    if order != "level first":
        lev.close()
        ctx.close()
    del lev, ctx
    gc.collect()
    assert rec.calls == ["level", "ctx"]
