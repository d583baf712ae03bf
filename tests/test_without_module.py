"""The array interface without the compiled module, whose absence costs time alone."""
import subprocess
import sys

import pytest

CODE = """
import sys
sys.modules["libmolgrid_b200.molgrid_native"] = None      # importing it raises ImportError
import torch, libmolgrid_b200 as lmg
from libmolgrid_b200 import api
assert api._fast() is False
if %d:
    gm = lmg.GridMaker(0.5, 5.5)
    out = torch.empty(gm.grid_dimensions(2), device="cuda")
    gm.forward((0., 0., 0.), torch.zeros(3, 3, device="cuda"), torch.zeros(3, device="cuda"), torch.ones(3, device="cuda"), out)
    assert float(out.max()) > 0
    gi, b = lmg.GridInterpolater(0.5, 5.5, 0.5, 5.5), torch.empty_like(out)
    gi.forward(out, lmg.Transform(), b)
    assert torch.equal(out, b)
print("fine")
"""


def run(gpu):
    assert subprocess.run([sys.executable, "-c", CODE % gpu], capture_output=True, text=True, check=True).stdout.strip() == "fine"


def test_import():
    run(0)


@pytest.mark.gpu
def test_calls():
    run(1)
