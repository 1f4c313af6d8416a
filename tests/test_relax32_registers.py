"""The FP32C relaxation of a single scan keeps its state in registers: a spill
costs several percent of a small scan.  Reads the compiler's own report."""
import os
import re
import tempfile

import pytest

from mechafm_gb300 import build


def test_single_scan_kernels_do_not_spill():
    try:
        cmd = next(c for c, o in build._units() if o == "relax32.o")
    except RuntimeError:
        pytest.skip("no nvcc")
    with tempfile.TemporaryDirectory() as tmp:
        log = build._run(cmd + ["-Xptxas", "-v", "-o", os.path.join(tmp, "relax32.o")])
    spills = {}
    for name, stores in re.findall(r"Compiling entry function '\S*relax32_kernelILi(\d+)ELb0E\S*'.*?(\d+) bytes spill stores",
                                   log, re.S):
        spills[int(name)] = int(stores)
    assert sorted(spills) == [1, 2, 4, 8, 16, 32]
    # one lane a column: a store of 8 bytes and a load outside the term loop
    assert all(spills[g] <= (8 if g == 1 else 0) for g in spills), spills
