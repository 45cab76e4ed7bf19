"""Device work of the library runs on the calls' own non-blocking streams, which nothing orders after
the legacy default stream. A clear on that stream is not done when a call's kernels start: it waits
behind whatever the caller has queued there. So no source writes device memory on it.
"""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "minirender_b200", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_no_clear_on_the_legacy_stream(name):
    with open(os.path.join(CSRC, name)) as f:
        source = f.read()
    assert not re.findall(r"\bcudaMemset\s*\(", source)
    # A stream argument that is a literal 0 is the legacy stream too.
    assert not re.findall(r"\bcudaMemsetAsync\s*\([^;]*,\s*(?:0|nullptr)\s*\)", source)
