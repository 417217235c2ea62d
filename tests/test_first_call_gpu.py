"""GPU: the first operator call of a process, which loads the compiled code, is served like every later one."""

import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent

SETUP = """
import torch
from sage_b200 import SAGELinear, _lib, sage, synthetic_sage

packed = {key: value.cuda() for key, value in synthetic_sage(256, 48, seed=1).items()}
x = torch.randn(3, 256, generator=torch.Generator().manual_seed(0)).half().cuda()
layer = SAGELinear(packed, 48)
assert _lib._native is None
"""
CHECK = """
want = x.float() @ layer.dequantize().float().T
assert ((y.float() - want).norm() / want.norm()) < 1e-3
"""
FIRST = {
    "operator": "y = sage(x, *packed.values(), 48)",
    "inference_mode": """
with torch.inference_mode():
    y = sage(x, *packed.values(), 48)
""",
    "gradient": """
y = sage(x.requires_grad_(), *packed.values(), 48)
try:
    y.sum().backward()
except RuntimeError as error:
    assert "no autograd formula" in str(error), error
else:
    raise AssertionError("differentiated")
y, x = y.detach(), x.detach()
""",
    "compiled": "y = torch.compile(layer, fullgraph=True)(x)",
}


@pytest.mark.parametrize("name", FIRST)
def test_first_call_of_a_process(name):
    done = subprocess.run([sys.executable, "-c", SETUP + FIRST[name] + CHECK], cwd=ROOT, capture_output=True, text=True)
    assert done.returncode == 0, done.stdout + done.stderr
    assert "overrid" not in done.stderr.lower(), done.stderr  # (no kernel is registered over another one)
