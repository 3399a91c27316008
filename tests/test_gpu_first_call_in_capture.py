"""Calls whose first use of the library in a process is inside a stream capture: what needs no warm-up call, and what says so."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gptq-2d_b200")
SCRIPT = r"""
import functools, sys
sys.path.insert(0, sys.argv[1])
import torch
import _abi, gptq_2d as G, kron_factors as K, quantizer_int as Q
what, m, n, batch, dtype = sys.argv[2], int(sys.argv[3]), int(sys.argv[4]), int(sys.argv[5]), getattr(torch, sys.argv[6])
lead = (batch,) if batch else ()
gen = torch.Generator(device="cuda").manual_seed(m)
rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)
w, l, u = 3 * rand(*lead, m, n), torch.tril(rand(m, m) * (.3 / m ** .5), -1), torch.triu(rand(n, n) * (.3 / n ** .5), 1)
g = rand(2 * m, m); g = g.T @ g / (2 * m) + torch.eye(m, device="cuda", dtype=dtype)
_abi.status_word(w.device)
run = (lambda: G.gptq_2d(w, l, u)) if what == "sweep" else (lambda: K.ldl_of_inverse(g, check=False))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
try:
    with torch.cuda.graph(graph):
        out = run()
except RuntimeError as refused:
    assert "unsupported combination" in str(refused), refused
    print("refused")
    sys.exit(0)
out.fill_(7)
graph.replay()
torch.cuda.synchronize()
if dtype == torch.float32 and what == "sweep" and not batch:
    G.SWEEP_SCHEDULE = 1  # in capture, such a call takes the tile schedule
want = run()
assert torch.equal(out, want), (out - want).abs().max()
print("equal")
"""


@pytest.mark.parametrize("what, m, n, batch, dtype, answer", [
    ("sweep", 301, 402, 0, "float32", "equal"), ("sweep", 301, 400, 0, "float32", "equal"), ("sweep", 200, 300, 2, "float32", "equal"),
    ("sweep", 200, 300, 0, "float64", "equal"), ("factors", 700, 1, 0, "float32", "equal"), ("factors", 300, 1, 0, "float64", "equal"),
    ("sweep", 300, 400, 0, "float32", "refused")])  # the pipelined schedule: after one call outside capture
def test_first_call(what, m, n, batch, dtype, answer):
    done = subprocess.run([sys.executable, "-c", SCRIPT, PACKAGE, what, str(m), str(n), str(batch), dtype], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and done.stdout.split() == [answer], done.stdout + done.stderr


@pytest.mark.parametrize("m, n", [(130, 200), (65, 64)])
def test_y_off_a_16_byte_boundary(m, n):
    """A matrix rounded in place that starts at an odd element: columns a multiple of 4, rows not."""
    sys.path.insert(0, PACKAGE)
    import torch

    import gptq_2d as G

    gen = torch.Generator(device="cuda").manual_seed(m)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    l, u = torch.tril(rand(m, m) * (.3 / m ** .5), -1), torch.triu(rand(n, n) * (.3 / n ** .5), 1)
    w = 3 * rand(m, n)
    y = torch.empty(m * n + 1, device="cuda")[1:].view(m, n).copy_(w)
    assert y.data_ptr() % 16
    G.SWEEP_SCHEDULE = 1
    try:
        want = G.gptq_2d(w, l, u)
    finally:
        G.SWEEP_SCHEDULE = 0
    assert torch.equal(G.gptq_2d(y, l, u, inplace=True), want)
