"""CPU: the host-side plan of the weight-gradient kernel (how blocks of weight rows and token tiles are dealt to CTAs)."""
import subprocess
import sys

import pytest

from tests.conftest import ROOT

# dims (B, H, S, d_h, Hkuv, E, d_e) whose plans differ although they have the same number of weight blocks and token tiles
PAIRS = [((5, 4, 100, 64, 4, 9, 64), (5, 4, 100, 64, 4, 10, 64)), ((2, 8, 1500, 96, 8, 1, 64), (2, 8, 1500, 96, 8, 2, 64)),
         ((2, 8, 333, 96, 8, 9, 64), (2, 8, 333, 96, 8, 10, 64))]


def _bytes_in_fresh_process(shapes):
    src = ("import ctypes as C, sys\nfrom flashmhf_b200 import _lib\nlib = _lib.load()\n"
           f"for s in {shapes!r}: print(lib.flashmhf_backward_workspace_bytes(C.byref(_lib.Dims(*s, 0))))")
    r = subprocess.run([sys.executable, "-c", src], cwd=ROOT, capture_output=True, text=True, check=True)
    return [int(v) for v in r.stdout.split()]


@pytest.mark.parametrize("a,b", PAIRS)
def test_plan_does_not_depend_on_the_calls_before(a, b):
    ab, ba = _bytes_in_fresh_process([a, b]), _bytes_in_fresh_process([b, a])
    assert ab == ba[::-1]
