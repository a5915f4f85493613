"""Every kernel that is launched as part of a chain (launch_after.cuh) waits for the launch ahead before anything
else: one that does not overtakes it."""
from __future__ import annotations

import re
import sys


def test_every_chained_kernel_waits_first(pkg):
    b = sys.modules[pkg.__name__ + ".build"]
    text = "\n".join((b.CSRC / f).read_text() for f in ("adjoint.cu", "sliced_gemm.cuh", "sytrd.cu"))
    chained = set(re.findall(r"launch_after\((?:\w+::)?(\w+),", text))
    assert len(chained) >= 11
    for name in chained:
        body = re.search(r"\b%s\([^)]*\)\s*\{(.*?)\n\}" % name, text, re.S).group(1)
        declarations, _, rest = body.partition("wait_previous_launch();")
        assert rest, name
        # before it only shared memory and indices of the block
        for line in filter(None, map(str.strip, declarations.splitlines())):
            assert re.match(r"(extern )?__shared__ [^=]*;$|const int64_t \w+ = blockIdx\.\w;$", line), (name, line)
