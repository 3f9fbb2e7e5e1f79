"""Copies and fills of device memory name the stream whose kernels read it (no
GPU): the library's streams do not wait for the default one, so a plain
cudaMemset, or the tail of a plain cudaMemcpy from pageable memory, may come
after the kernel that needs it."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "geoflood_gb300" / "csrc"
# its kernels run on the default stream themselves
DEFAULT_STREAM = {"gf_probe.cu"}


def test_no_copy_or_fill_on_the_default_stream():
    found = []
    for f in sorted(CSRC.iterdir()):
        if f.suffix in (".cu", ".cpp", ".cuh", ".h") and f.name not in DEFAULT_STREAM:
            for k, line in enumerate(f.read_text().splitlines(), 1):
                if re.search(r"\bcudaMem(cpy|set)(2D|3D|ToSymbol|FromSymbol)?\(", line):
                    found.append(f"{f.name}:{k}: {line.strip()}")
    assert not found, found
