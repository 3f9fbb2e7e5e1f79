"""The bench's counter figures belong to the tile that ran (no GPU)."""
import json
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

from tests.test_bench_line import _full_result  # noqa: E402


@pytest.fixture
def bench():
    import bench

    return bench


def test_a_tile_without_a_capture_has_no_counts(bench):
    assert all(v > 0 for tile in ([256, 4, 1], [384, 9, 1]) for v in bench.ncu_counts(tile))
    for tile in ((256, 7, 1), (384, 7, 1), (384, 10, 2)):
        assert bench.ncu_counts(tile) == (None, None)


def test_the_line_says_so(bench):
    r = _full_result(bench)
    r["roofline"]["traffic"] = None
    r["fp64"]["frac_of_measured_dfma"] = None
    d = json.loads(json.dumps(bench.compact(r)))
    assert d["roofline"]["traffic"] is None and d["fp64"]["frac_of_measured_dfma"] is None
