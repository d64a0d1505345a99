"""The library allocates no device memory, as its header promises: every buffer is the caller's. No GPU needed."""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "wadi2d_b200" / "csrc"
DEVICE_MEMORY = re.compile(r"\bcu(?:da)?(?:Malloc|MemAlloc|MemCreate|Free|MemFree)(?!Host|_?Host)\w*\s*\(")


def test_no_call_allocates_or_frees_device_memory():
    sources = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))
    assert len(sources) >= 8
    for path in sources:
        for number, line in enumerate(path.read_text().splitlines(), 1):
            code = line.split("//")[0]
            assert not DEVICE_MEMORY.search(code), f"{path.name}:{number}: {line.strip()}"
