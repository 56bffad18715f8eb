"""NERVA_B200_GEMM_TIMELINE=1: the block projections' stamps, on whichever kernel the shape goes to."""
import os
import re
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

RUN = """
from nerva_b200 import ops, synth
rows, cols, tokens = {rows}, {cols}, {tokens}
w = ops.synth_normal_bf16(0, 77, rows * cols, 0.02)
x = ops.synth_normal_bf16(0, synth.T_ACTIVATION, tokens * cols, 1.0)
ops.projection_sustained(w, x, rows, cols, tokens=tokens, copies=2, warmup=2, iterations=4)
"""


@pytest.mark.parametrize("rows,cols,tokens", [(1024, 1024, 32), (14080, 1024, 100)])  # gemm_tc.cu, pairs of SMs
def test_stamps_are_written_in_order(built_lib, rows, cols, tokens):
    out = subprocess.run([sys.executable, "-c", RUN.format(rows=rows, cols=cols, tokens=tokens)], cwd=ROOT, text=True,
                         capture_output=True, timeout=120, env=dict(os.environ, NERVA_B200_GEMM_TIMELINE="1"))
    assert out.returncode == 0, out.stderr
    stamps = {}
    for launch, block, name, ns in re.findall(r"launch (\d) (\w+) block (\w+): (-?\d+) ns", out.stderr):
        stamps.setdefault((launch, block), []).append(int(ns))
    assert set(stamps) == {(launch, block) for launch in "01" for block in ("first", "last")}
    for s in stamps.values():
        assert len(s) == 4 and s == sorted(s) and s[3] > s[0]
