"""Dynamic and static shared memory together may pass 48 KB where the dynamic part alone does not: widths between 2950 and 4060
in the one-token expert product.  In a process of its own, because the permission stays with a kernel once it is given."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch, tilert_b200
from tilert_b200 import gqa_ops as ops
tilert_b200.load_backend("ralasun")
dim, e, top, ff = %d, 4, 2, 8
x, z = torch.ones(dim, device="cuda"), torch.arange(4.0, device="cuda")
w = torch.ones(e, 2, ff, dim, dtype=torch.bfloat16, device="cuda") / dim
hidden, ids, sw = torch.zeros(top * ff, device="cuda"), torch.zeros(top, dtype=torch.int32, device="cuda"), torch.zeros(top, device="cuda")
ops.vec_gate_up(x, dim, z, top, w, None, ff, 0, 7.0, 7.0, 1.702, hidden, ids, sw)
assert sorted(ids.tolist()) == [2, 3] and abs(float(hidden[0]) - 2 / (1 + 2.718281828 ** -1.702)) < 1e-2, hidden
assert tilert_b200.device_status(0, "ralasun") == 0
"""


@pytest.mark.parametrize("dim", [2944, 2952, 3736, 4056, 4064])
def test_expert_product(dim):
    done = subprocess.run([sys.executable, "-c", PROGRAM % dim], cwd=Path(__file__).parent.parent, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
