"""Every copy and fill of the CUDA library names its stream.  A handle's streams are non-blocking, so
work on the legacy stream is not ordered with theirs: a copy from pageable memory may return before
its data is on the device, and a fill before it has run."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "coupled_cluster_doubles_b200", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_copies_and_fills_are_on_a_stream(name):
    with open(os.path.join(CSRC, name)) as f:
        for number, line in enumerate(f, 1):
            assert not re.search(r"\bcuda(Memcpy|Memset)(2D|3D)?\(", line), f"{name}:{number}"
