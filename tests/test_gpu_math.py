"""Reciprocal, roots and 2/3 power of the device code (gf_cmp.cuh, gf_ghost.cu)
against long double, over every exponent of their range (GPU required)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from geoflood_gb300 import build

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
L = np.longdouble


def two_thirds(x):
    """x to the double 2.0 / 3.0, the exponent of the reference's power."""
    return np.exp(L(2.0 / 3.0) * np.log(x))


# (operation, lowest and highest exponent of its argument, exact value, bound in
# units of the result's last place). One rounding is half a unit. The reciprocal
# adds its remainder alone (below 1/100). The roots' residual is that of a rounded
# product a y, half of whose relative error (2^-53) stays: up to half a unit
# more. pow23 takes the product's rounding up and so adds its remainder alone.
OPS = {"rcp": (0, -1022, 1022, lambda x: 1 / x, 0.55), "rsqrt": (1, -1022, 1024, lambda x: 1 / np.sqrt(x), 1.05),
       "sqrt": (2, -1022, 1024, np.sqrt, 1.05), "pow23": (3, -99, 99, two_thirds, 0.55)}


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    so = tmp_path_factory.mktemp("cmp") / "cmp_device.so"
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-shared", str(ROOT / "tests" / "cmp_device.cu"),
                    "-o", str(so), "-lcudart"], check=True)
    lib = C.CDLL(str(so))
    dp = C.POINTER(C.c_double)
    lib.eval.argtypes = [C.c_int, dp, dp, C.c_int]

    def run(op, x):
        y = np.empty_like(x)
        assert lib.eval(op, x.ctypes.data_as(dp), y.ctypes.data_as(dp), x.size) == 0
        return y

    return run


@pytest.mark.parametrize("name", sorted(OPS))
def test_refined_operations_meet_their_bounds(evaluate, name):
    op, lo, hi, exact, bound = OPS[name]
    r = np.random.default_rng(op)
    man = np.concatenate([r.uniform(1.0, 2.0, 160), 1.0 + 2.0 ** -np.arange(1.0, 53.0), [1.0, 2.0 - 2.0**-52]])
    x = np.ldexp(man[:, None], np.arange(lo, hi)[None, :]).ravel()
    if name == "rcp":
        x = np.concatenate([x, -x])
    y = evaluate(op, x)
    want = exact(L(x))
    err = np.abs((L(y) - want) / L(np.spacing(np.abs(want.astype(np.float64))))).astype(np.float64)
    print(name, "largest error", err.max(), "mean", err.mean())
    assert err.max() <= bound
