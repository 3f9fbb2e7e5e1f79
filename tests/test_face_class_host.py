"""The single-precision face classes (gf_riemann.cuh) are spelled out: a compiler
that may fuse products into sums and one that may not give every face the same
class, and so would two kernels that hold the function."""
import platform
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def fused_flags():
    """Flags of a host that has fused instructions, or None."""
    if platform.machine() == "aarch64":
        return ["-ffp-contract=fast"]
    info = Path("/proc/cpuinfo")
    if platform.machine() == "x86_64" and info.exists() and " fma " in info.read_text():
        return ["-ffp-contract=fast", "-mfma"]
    return None


def test_fusing_products_changes_no_class(tmp_path):
    fused = fused_flags()
    if fused is None:
        pytest.skip("host without fused instructions")
    out = []
    for name, flags in (("plain", ["-ffp-contract=off"]), ("fused", fused)):
        exe = tmp_path / name
        subprocess.run(["g++", "-O2", "-std=c++17", *flags, f"-I{ROOT}/geoflood_gb300/csrc", f"-I{ROOT}/include",
                        str(ROOT / "tests" / "face_class_host.cpp"), "-o", str(exe)], check=True)
        out.append(subprocess.run([str(exe), "20000000"], check=True, capture_output=True, text=True).stdout)
    print(out)
    assert min(int(v) for v in out[0].split()[:4]) > 0
    assert out[0] == out[1]
