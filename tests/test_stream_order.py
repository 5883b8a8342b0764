"""Device memory that a context's kernels read is written on the context's stream.  That stream is a non-blocking one,
so a copy or fill on the default stream (the calls without ``Async``) is not ordered before its kernels.  The window in
which such a copy is still on its way is too short to meet in a run, so the sources are read instead."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amber_b200", "csrc")


@pytest.mark.parametrize("name", sorted(os.listdir(CSRC)))
def test_no_copy_or_fill_on_the_default_stream(name):
    src = open(os.path.join(CSRC, name), encoding="utf-8").read()
    assert re.findall(r"\bcudaMem(?:cpy|set)(?:2D|3D|ToSymbol|FromSymbol)?\s*\(", src) == []
