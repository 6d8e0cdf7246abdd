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
    (36, 100, 6), (48, 20, 5), (48, 3, 6), (27, 1, 6), (33, 2, 8), (39, 1, 5),
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


def smooth_bands(n, nb, a, seed):
    """Rows of Gaussian noise damped above 1 Ha, as bands are after the first iterations."""
    rng = np.random.default_rng(seed)
    k = 2.0 * np.pi * np.fft.fftfreq(n, 1.0 / n) / a
    e = 0.5 * (k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2)
    noise = np.fft.fftn(rng.normal(size=(nb, n, n, n)), axes=(1, 2, 3))
    return np.fft.ifftn(noise / (1.0 + e * e), axes=(1, 2, 3)).real


@pytest.mark.parametrize("n,md", [(15, 2), (15, 6), (21, 4), (27, 5), (33, 6), (45, 4), (45, 6), (45, 8)])
def test_odd_width_rounding(gpu, n, md):
    """The stencil at odd widths rounds no worse than the register-queue kernel's sum: the centre, then for each distance
    the three axes' symmetric pairs by one multiply-add each, then Vloc."""
    ld = np.longdouble
    c = build_cell(Workload("w", max(1, round(n / 24)), n, 2, 2, 0.02, 1003, md))
    c.uv[:] = 0.0
    gpu.setup(c)
    x = smooth_bands(n, 2, c.a, n)
    v = c.vloc.reshape(-1)[:c.ML].reshape(n, n, n)

    def pair(f, axis, m):
        return np.roll(f, m, 3 - axis) + np.roll(f, -m, 3 - axis)

    xl = x.astype(ld)
    ref = (ld(c.coef_lap0) + v.astype(ld)) * xl
    q = c.coef_lap0 * x
    for m in range(1, md + 1):
        for axis in range(3):
            w = c.coef_lap[axis, m - 1]
            ref += ld(w) * pair(xl, axis, m)
            q = (ld(w) * pair(x, axis, m) + q).astype(np.float64)
    q = (v.astype(ld) * x + q).astype(np.float64)
    out = api.fortran_empty(c.ML, 2)
    gpu.hamiltonian(1, 1, dev(x.reshape(2, -1).T), out, 1, c.ML, 1, 2)
    gpu.synchronize()
    got = out.cpu().numpy().T.reshape(x.shape)
    assert np.sqrt(((got - ref) ** 2).sum()) <= np.sqrt(((q - ref) ** 2).sum())
