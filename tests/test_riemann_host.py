"""The single-precision face classes of the contracted build (gf_riemann.cuh),
compiled for the host: wherever a class allows a shorter solve (smooth, edge,
wall), it gives the full solve's speeds and f-waves bit for bit."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
# kind of faces -> least share of each class (smooth, edge, edge with its flag):
# smooth flow, anything, near critical, thin water on a high bed, random dry
# tolerance, lake at rest, edge of the steady-state bounds, one side dry twice
KINDS = {0: (0.5, 0, 0.005), 1: (0.05, 0.05, 0.1), 2: (0.001, 0.001, 0.1), 3: (0.01, 0.05, 0.2),
         4: (0.05, 0.05, 0.1), 5: (0.5, 0, 0.05), 6: (0.05, 0.05, 0.1), 7: (0, 0.2, 0.1), 8: (0, 0.2, 0.1)}


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    out = tmp_path_factory.mktemp("riemann") / "riemann_host"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT}/geoflood_gb300/csrc",
                    f"-I{ROOT}/include", str(ROOT / "tests" / "riemann_host.cpp"), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_shorter_solves_give_the_same_bits(prog, kind):
    n = 300000
    r = subprocess.run([str(prog), str(kind), str(n)], check=True, capture_output=True, text=True)
    *count, differ = (int(v) for v in r.stdout.split())
    assert sum(count) == n and all(c >= share * n for c, share in zip(count, KINDS[kind]))
    assert differ == 0
