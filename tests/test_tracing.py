"""The layer operators under torch.compile and the checks of torch.library: traced whole, shape functions as the kernels allocate."""
import subprocess
import sys

import pytest
import torch

import llsa_b200
from llsa_b200 import ops, synth

DEV = "cuda:0"

# a fresh process: the first call of the library is the traced one
_FIRST_CALL = """
import torch, llsa_b200
from llsa_b200 import synth
q, k, v, do = [t.cuda() for t in synth.gaussian_qkv(1, 1, 2, 4096, 64, dtype=torch.bfloat16)]
table = torch.ones(4096, 64, device="cuda", dtype=torch.bfloat16)
w = torch.ones(64, device="cuda", requires_grad=True)
for call in (lambda *x: llsa_b200.llsa_l2(*x), lambda *x: llsa_b200.llsa_l1_rope(*x, table), lambda *x: llsa_b200.llsa_l2_rms_rope(*x, w, w, table)):
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    o = torch.compile(lambda *x: call(*x) * 2, fullgraph=True, backend="aot_eager")(*x)
    want = call(*x) * 2
    assert torch.equal(o, want)
    got, want = [torch.autograd.grad(t, x, do) for t in (o, want)]
    # dq and dv repeat exactly or up to the order of fp32 sums in front of a rounding to bf16
    assert all(float((a.float() - b.float()).norm() / b.float().norm()) < 1e-3 for a, b in zip(got, want))
"""


@pytest.mark.gpu
def test_whole_graph_compile_of_a_first_call():
    r = subprocess.run([sys.executable, "-c", _FIRST_CALL], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
