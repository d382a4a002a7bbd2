"""What the built library holds."""

import os
import zlib

import pytest

from sundog_b200 import build


@pytest.mark.parametrize("path", [build.LIB, build.LIB_CW8])
def test_device_code_is_not_compressed(path):
    """Compressed device code costs a process's first render 11 ms. Plain
    machine code deflates to about a third; what was compressed already hardly
    shrinks, so no MiB of the library may be such."""
    if not os.path.isfile(path):
        build.build_all()
    with open(path, "rb") as f:
        data = f.read()
    block = 1 << 20
    for at in range(0, len(data) - block + 1, block):
        part = data[at:at + block]
        assert len(zlib.compress(part, 1)) < 0.7 * block, "block at %d MiB" % (at >> 20)
