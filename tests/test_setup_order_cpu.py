"""An engine's stream does not wait for the legacy default stream, so every fill
and copy of engine memory has to be issued on the engine's own stream: a fill on
the default one may land after the kernel that writes the buffer."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afqmclab_b200", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_no_fill_or_copy_on_the_default_stream(name):
    with open(os.path.join(CSRC, name)) as f:
        found = [i for i, line in enumerate(f, 1) if re.search(r"\bcuda(Memset|Memcpy)\(", line.split("//")[0])]
    assert found == []
