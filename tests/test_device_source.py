"""What the compiler must not do with the device code's inline assembly, read from the source (no GPU)."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "webgpu_b200" / "csrc"


def _function(text, name):
    start = re.search(r"__device__ __forceinline__ \w+ " + name + r"\(", text).start()
    return text[start:text.index("\n}", start)]


@pytest.mark.parametrize("path,name", [("common.cuh", "load32")])
def test_loads_used_behind_a_programmatic_wait_stay_behind_it(path, name):
    """A load of what the kernel before may still be writing is volatile and clobbers memory, so that it cannot move above
    griddepcontrol.wait, and is no read of constant data."""
    body = _function((CSRC / path).read_text(), name)
    loads = re.findall(r"asm\s+(volatile)?\s*\((.*?)\);", body, re.S)
    assert loads
    for volatile, rest in loads:
        assert "ld.global" in rest
        assert volatile == "volatile" and '"memory"' in rest and ".nc" not in rest
