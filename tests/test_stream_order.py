"""Host: a context's kernels run in its own non-blocking stream, so what they read is
written in that stream: no source file uploads or clears device memory by the
calls of the legacy stream, which a non-blocking stream does not wait for and
whose copies may return before the last bytes have arrived."""
from __future__ import annotations

import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "mini-fem-pic-main_b200", "csrc")


def test_uploads_are_in_the_contexts_stream():
    found = []
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"cudaMemset\s*\(|cudaMemcpy(?:2D)?\s*\([^;]*?cudaMemcpyHostToDevice", text):
            found.append((name, text.count("\n", 0, m.start()) + 1))
    assert not found, found
