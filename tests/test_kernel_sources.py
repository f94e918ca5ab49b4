"""What every CUDA source has to keep to, read from the text of the sources (no GPU)."""
import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).resolve().parent.parent / "qwen_triton_b200" / "csrc").glob("*.cu*"))
# operands that are written once, when a model is loaded
WEIGHTS = ("norm_w", "wr[r]", "bias", "p.skip", "p.weight", "p.read", "p.out_weight", "p.mix")


@pytest.mark.parametrize("source", SOURCES, ids=lambda path: path.name)
def test_what_earlier_kernels_write_is_read_by_ordinary_loads(source):
    """A kernel starts while the one before it still runs.  Reads through ``__ldg`` or through a restricted const parameter may be moved ahead of
    the wait for it (nobody writes there while the kernel runs, they say), so they are left to weights."""
    text = source.read_text()
    for start in (match.start() for match in re.finditer("__global__", text)):
        signature = text[start:text.index("{", start)]
        assert not re.search(r"const \w+\s*\*\s*__restrict__", signature), signature
    for call in re.finditer(r"__ldg\(", text):
        assert text[call.end():].startswith(WEIGHTS), text[call.start():call.start() + 80]


@pytest.mark.parametrize("source", SOURCES, ids=lambda path: path.name)
def test_what_the_runtime_keeps_per_device_is_not_kept_per_process(source):
    """A kernel's limit of dynamic shared memory belongs to a device: raised once in a process, it is missing on the second device."""
    assert not re.search(r"static bool \w+ = false;", source.read_text())
