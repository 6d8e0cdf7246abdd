"""H psi where the march kernel, its tile and its z split change: odd widths (k_stencil_row), widths below the
finite-difference order, few and many bands, several projector tails per band, every order's register layout; FP32
through the CG sweep at widths of an odd multiple of two."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from rsdft_b200 import api
from rsdft_b200.cell import Workload, build_cell

pytestmark = pytest.mark.gpu


def dev(a):
    t = api.fortran_empty(a.shape[0], a.shape[1])
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t


@pytest.mark.parametrize("n,nb,md", [
    (5, 3, 6), (7, 1, 8), (9, 2, 6), (13, 5, 6), (15, 40, 4), (17, 3, 8), (21, 2, 7), (27, 9, 6), (45, 3, 6), (12, 1, 6),
    (12, 200, 6), (20, 7, 2), (26, 3, 6), (36, 5, 6), (40, 30, 8),
    (36, 100, 6), (48, 20, 5), (48, 3, 6),
])
def test_hpsi_widths(gpu, n, nb, md):
    c = build_cell(Workload("w", 1, n, nb, nb, 0.03, 5000 + n, md))
    gpu.setup(c)
    o = O.Oracle(c)
    u = np.asfortranarray(c.psi0(nb))
    ref = o.hamiltonian(u)
    out = api.fortran_empty(c.ML, nb)
    out.fill_(np.nan)
    gpu.hamiltonian(1, 1, dev(u), out, 1, c.ML, 1, nb)
    gpu.synchronize()
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n,nb", [(14, 5), (18, 3), (22, 40), (16, 4)])
def test_fp32_widths(gpu, n, nb):
    c = build_cell(Workload("w32", 1, n, nb, nb, 0.03, 6000 + n))
    gpu.setup(c)
    o = O.Oracle(c)
    q = np.asfortranarray(np.linalg.qr(c.psi0(nb))[0] / np.sqrt(c.dV))
    ru, resp, rres, _ = o.conjugate_gradient(q, 3, 3)
    u = dev(q)
    esp = torch.zeros(nb, dtype=torch.float64, device="cuda")
    res = torch.zeros_like(esp)
    gpu.conjugate_gradient(1, c.ML, nb, 1, 1, u, esp, res, ncg=3, mloop=3, mode=api.MODE_MIXED_BF16X3)
    gpu.synchronize()
    # FP32 storage and arithmetic: 2^-24 per operation, kinetic energies of white noise 40 times the result's
    assert np.abs(u.cpu().numpy() - ru).max() <= 2e-5 * np.abs(ru).max()
    assert np.abs(esp.cpu().numpy() - resp).max() <= 2e-4 * np.abs(resp).max()
    assert np.abs(res.cpu().numpy() - rres).max() <= 2e-4 * np.abs(rres).max()
