"""CG sweep against the oracle where its kernels change form: the basis passes by TMA (even widths) and element-wise
(odd ones), every s-step order, the Gram matrix's second off-diagonal as dots (FP64, and FP32 up to 65536 points) and
from the recurrence (FP32 above: 41^3 and 42^3), the literal preconditioner above it, no preconditioner, no line step, and bands that come in unnormalised
(the first step then takes its dots from H x, not from g)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from rsdft_b200 import api
from rsdft_b200.cell import Workload, build_cell

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 form's bar; measured 1e-14 .. 2e-13


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("n,nb,mloop,ncg,scale", [
    (12, 16, 3, 4, 1.0), (12, 5, 1, 3, 1.0), (12, 3, 2, 2, 30.0), (16, 7, 4, 4, 1.0), (15, 9, 3, 4, 1.0),
    (13, 1, 4, 2, 1.0), (12, 4, 5, 3, 1.0), (12, 4, 0, 3, 1.0), (14, 6, 3, 0, 1.0), (15, 2, 2, 1, 30.0),
    (40, 2, 4, 2, 1.0), (41, 2, 3, 2, 1.0), (42, 2, 4, 2, 1.0),
])
def test_cg_forms(gpu, n, nb, mloop, ncg, scale):
    c = build_cell(Workload("cg_forms", 1, n, nb, nb, 0.03, 2000 + n))
    gpu.setup(c)
    o = O.Oracle(c)
    q = np.linalg.qr(c.psi0(nb))[0] * (scale / np.sqrt(c.dV))
    q = np.asfortranarray(q)
    ru, resp, rres, _ = o.conjugate_gradient(q, ncg, mloop)
    u = api.fortran_empty(c.ML, nb)
    u.copy_(torch.from_numpy(q))
    esp = torch.zeros(nb, dtype=torch.float64, device="cuda")
    res = torch.zeros_like(esp)
    gpu.conjugate_gradient(1, c.ML, nb, 1, 1, u, esp, res, ncg=ncg, mloop=mloop)
    gpu.synchronize()
    assert rel(u.cpu().numpy(), ru) <= TOL
    assert rel(esp.cpu().numpy(), resp) <= TOL
    assert rel(res.cpu().numpy(), rres) <= TOL
    # the FP32 form of the same sweep: eps(FP32) = 6e-8 per operation, a few line steps.  Measured: x 2.0e-6, esp 7.2e-6
    # (eigenvalues far below the kinetic energies they are sums of), res 6.7e-6; four times that
    x = api.fortran_empty(c.ML, nb)
    x.copy_(torch.from_numpy(q))
    gpu.conjugate_gradient(1, c.ML, nb, 1, 1, x, esp, res, ncg=ncg, mloop=mloop, mode=api.MODE_MIXED_BF16X3)
    gpu.synchronize()
    assert rel(x.cpu().numpy(), ru) <= 8e-6
    assert rel(esp.cpu().numpy(), resp) <= 3e-5
    assert rel(res.cpu().numpy(), rres) <= 3e-5


def test_captured_calls(gpu):
    """H psi and the CG sweep in a CUDA graph (their launches are then ordinary ones): a replay gives the call's bits."""
    c = build_cell(Workload("cap", 1, 16, 12, 12, 0.03, 2500))
    gpu.setup(c)
    q = np.asfortranarray(np.linalg.qr(c.psi0(12))[0] / np.sqrt(c.dV))
    start, u, h = (api.fortran_empty(c.ML, 12) for _ in range(3))
    start.copy_(torch.from_numpy(q))
    esp = torch.zeros(12, dtype=torch.float64, device="cuda")
    res = torch.zeros_like(esp)

    def calls():
        u.copy_(start)
        gpu.hamiltonian(1, 1, u, h, 1, c.ML, 1, 12)
        gpu.conjugate_gradient(1, c.ML, 12, 1, 1, u, esp, res, ncg=2, mloop=3)

    calls()  # allocates the workspaces
    gpu.synchronize()
    want = [t.clone() for t in (h, u, esp, res)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=gpu._torch_stream):
        calls()
    for t in (h, u, esp, res):
        t.fill_(float("nan"))
    graph.replay()
    gpu.synchronize()
    for got, ref in zip((h, u, esp, res), want):
        assert torch.equal(got, ref)
    del graph
