"""The FP64 products of tall blocks (Gram, rotation) and the overlap's Cholesky factor where their kernels change form:
tile edges, remainders, the INT8-slice form against the DMMA one, and values that the slices cannot hold."""
import ctypes

import numpy as np
import pytest
import torch

from rsdft_b200 import _lib, api
from rsdft_b200.cell import Workload, build_cell

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def sliced(ml, nb):
    """Whether the library takes the INT8 slices for a product of this size."""
    f = getattr(_lib.load(), "_ZN5rsdft10imma_suitsEli")
    f.restype, f.argtypes = ctypes.c_bool, [ctypes.c_long, ctypes.c_int]
    return f(ml, nb)


def dev(a):
    t = api.fortran_empty(a.shape[0], a.shape[1])
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t


@pytest.mark.parametrize("ml,m,n,sym", [
    (5, 1, 1, 0), (300, 31, 32, 0), (4099, 33, 64, 0), (1000, 65, 130, 0), (777, 32, 32, 1), (513, 64, 64, 1),
    (129, 97, 97, 1), (640, 160, 160, 1),
])
def test_gram(gpu, ml, m, n, sym):
    rng = np.random.default_rng(ml + m)
    a, b = rng.normal(size=(ml, m)), rng.normal(size=(ml, n))
    c = api.fortran_empty(m, n)
    gpu.gram(dev(a), dev(b), c, alpha=0.5, sym=sym)
    gpu.synchronize()
    ref = 0.5 * (a.astype(np.longdouble).T @ b.astype(np.longdouble))
    if sym:
        ref = 0.5 * (ref + ref.T)
    # ml products and additions per element, each within EPS of sum |a b|
    bound = ml * EPS * 0.5 * (np.abs(a).T @ np.abs(b)).max()
    assert np.abs(c.cpu().numpy() - ref).max() <= bound


@pytest.mark.parametrize("ml,nb", [
    (4096, 96), (4097, 97), (4160, 127), (5000, 128), (4159, 129), (8192, 192), (4500, 200), (4095, 96), (5000, 95),
    (30001, 129), (13824, 191), (13000, 197), (100001, 96), (100000, 97), (100002, 127), (100063, 128), (4096, 352),
    (29000, 192),
])
def test_rotate(gpu, ml, nb):
    """The second half of the sizes takes the INT8 slices, the others the DMMA kernel.  Bands of very different scale."""
    assert sliced(ml, nb) == (ml * nb * nb >= 5e8)
    rng = np.random.default_rng(nb)
    u = rng.normal(size=(ml, nb)) * 10.0 ** rng.uniform(-6, 6, nb)
    u[:, nb // 2] = 0.0
    v = rng.normal(size=(nb, nb)) * 10.0 ** rng.uniform(-3, 3, nb)
    t = dev(u)
    gpu.rotate(t, dev(v))
    gpu.synchronize()
    ref = u.astype(np.longdouble) @ v.astype(np.longdouble)
    # nb terms and additions, each within EPS of sum_m |u(i, m)| |v(m, n)|; the slices: within 2^-60 of the bands' largest
    bound = nb * EPS * (np.abs(u) @ np.abs(v))
    if sliced(ml, nb):
        bound += nb * 2.0 ** -60 * (np.abs(u).max(0) @ np.abs(v))
    assert (np.abs(t.cpu().numpy() - ref) <= bound).all()


@pytest.mark.parametrize("kind", ["vacuum", "slab", "localised", "one band"])
@pytest.mark.parametrize("ml,nb", [(4096, 96), (30000, 130), (13824, 200), (4096, 352), (100000, 96)])
def test_rotate_decaying_bands(gpu, kind, ml, nb):
    """Bands that fall off by many decades keep the digits of their tails: every element within FP64's own bound."""
    rng = np.random.default_rng(nb)
    u, i, m = rng.normal(size=(ml, nb)), np.arange(ml)[:, None], np.arange(nb)[None, :]
    v = np.linalg.qr(rng.normal(size=(nb, nb)))[0]
    assert sliced(ml, nb) == (ml * nb * nb >= 5e8)
    if kind == "vacuum":    # the whole set, along the grid
        u *= 10.0 ** (-20.0 * i / ml)
    elif kind == "slab":    # the whole set, a few points of every row of 64
        u *= 10.0 ** (-1.5 * np.maximum(0, i % 64 - 52))
    elif kind == "localised":  # each band about a point of its own; hardly mixed
        u *= 10.0 ** (-20.0 * np.abs(i / ml - m / nb))
        v = np.eye(nb) + 1e-14 * v
    else:
        u[:, 70] *= 10.0 ** (-20.0 * i[:, 0] / ml)
        v[:, :] = 0.0
        v[(m[0] + 1) % nb, m[0]] = 1.0
    t = dev(u)
    gpu.rotate(t, dev(v))
    gpu.synchronize()
    ref = u.astype(np.longdouble) @ v.astype(np.longdouble)
    assert (np.abs(t.cpu().numpy() - ref) <= nb * EPS * (np.abs(u) @ np.abs(v))).all()


@pytest.mark.parametrize("ml,nb", [(30000, 130), (13824, 200), (20000, 290)])
@pytest.mark.parametrize("mix", [1e-14, 1e-6, 1e-2])
@pytest.mark.parametrize("inplace", [True, False])
def test_rotate_tail_bands(gpu, ml, nb, mix, inplace):
    """A few bands that fall to 2^-17 among bands that do not: columns made of them keep FP64's bound, by tiles of 128
    columns from the DMMA kernel, the others by either form.  Out of place through the Gram-Schmidt of nearly
    orthonormal bands, whose second rotation is by I + rounding."""
    rng = np.random.default_rng(nb)
    u, i = rng.normal(size=(ml, nb)), np.arange(ml) / ml
    tails = np.array([1, nb - 2])
    u[:, tails] = rng.uniform(0.5, 1.5, size=(ml, 2)) * 2.0 ** (-24.0 * np.abs(i[:, None] - np.array([0.3, 0.6])))
    v = np.eye(nb) + mix * np.linalg.qr(rng.normal(size=(nb, nb)))[0]
    assert sliced(ml, nb)
    if inplace:
        t = dev(u)
        gpu.rotate(t, dev(v))
        gpu.synchronize()
        ref = u.astype(np.longdouble) @ v.astype(np.longdouble)
        err, bound = np.abs(t.cpu().numpy() - ref), nb * EPS * (np.abs(u) @ np.abs(v))
        assert (err[:, tails] <= bound[:, tails]).all()
        assert (err <= bound + nb * 2.0 ** -60 * (np.abs(u).max(0) @ np.abs(v))).all()
        return
    n = round(ml ** (1 / 3))
    c = build_cell(Workload("tails", 1, n, nb, nb, 0.03, 3300 + n))
    gpu.setup(c)
    w = np.linalg.qr(np.column_stack([u[:n ** 3, tails], np.delete(u[:n ** 3], tails, 1)]))[0] / np.sqrt(c.dV)
    t = dev(w)
    gpu.gram_schmidt(1, nb, 1, 1, t)
    gpu.synchronize()
    g = t.cpu().numpy()
    assert np.abs(g.T @ g * c.dV - np.eye(nb)).max() <= 1e-14
    # the first two columns stay themselves, to the rounding of a norm and of the pair's overlap
    err = np.abs(g[:, :2] - w[:, :2])
    assert (err <= 1e-14 * (np.abs(w[:, :1]) + np.abs(w[:, :2]))).all()


def test_second_block_decays(gpu):
    """subspace_diag where only H psi leaves the slices' range: both products go to the DMMA kernel."""
    c = build_cell(Workload("sd", 1, 24, 192, 192, 0.03, 3100))
    assert sliced(c.ML, 192)
    c.coef_lap[:], c.coef_lap0, c.uv[:] = 0.0, 0.0, 0.0
    c.vloc[:] = (10.0 ** (-20.0 * np.arange(c.vloc.size) / c.vloc.size)).reshape(c.vloc.shape)
    gpu.setup(c)
    u = np.linalg.qr(np.random.default_rng(1).normal(size=(c.ML, 192)))[0] / np.sqrt(c.dV)
    t, esp = dev(u), torch.zeros(192, dtype=torch.float64, device="cuda")
    gpu.subspace_diag(1, 1, t, esp)
    gpu.synchronize()
    h = u.T @ (c.vloc.reshape(-1, 1)[:c.ML] * u) * c.dV
    w, z = np.linalg.eigh(0.5 * (h + h.T))
    assert np.abs(esp.cpu().numpy() - w).max() <= 192 * EPS * np.abs(w).max()
    g = t.cpu().numpy()
    assert np.abs(g.T @ g * c.dV - np.eye(192)).max() <= 1e-13
    assert np.abs(np.abs((u @ z * g).sum(0) * c.dV) - 1.0).max() <= 1e-10


@pytest.mark.parametrize("ml,nb", [(4096, 96), (4096, 352)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300, 1e-300])
def test_rotate_out_of_range(gpu, bad, ml, nb):
    """A value the slices cannot hold sends the whole product to the DMMA kernel, on the device."""
    rng = np.random.default_rng(5)
    u = rng.normal(size=(ml, nb))
    if abs(bad) < 1.0:
        u[:, 3] *= bad
    else:
        u[17, 3] = bad
    v = rng.normal(size=(nb, nb))
    t = dev(u)
    gpu.rotate(t, dev(v))
    gpu.synchronize()
    with np.errstate(all="ignore"):
        ref = u @ v
    got = t.cpu().numpy()
    rows = np.arange(ml) != 17
    assert np.isfinite(got[rows]).all() and np.abs(got[rows] - ref[rows]).max() <= nb * EPS * np.abs(ref).max(where=rows[:, None], initial=0) * 8
    np.testing.assert_array_equal(np.isnan(got[17]), np.isnan(ref[17]))
    np.testing.assert_array_equal(np.isinf(got[17]), np.isinf(ref[17]))


@pytest.mark.parametrize("n,nb", [(16, 96), (17, 128), (18, 131), (20, 190), (16, 352), (24, 191), (25, 180), (26, 200)])
def test_gram_schmidt_slices(gpu, n, nb):
    c = build_cell(Workload("gs", 1, n, nb, nb, 0.03, 3000 + n))
    gpu.setup(c)
    rng = np.random.default_rng(nb)
    q = np.linalg.qr(rng.normal(size=(c.ML, nb)))[0]
    u = q + 0.1 * rng.normal(size=q.shape) / np.sqrt(c.ML)
    t = dev(u)
    gpu.gram_schmidt(1, nb, 1, 1, t)
    gpu.synchronize()
    g = t.cpu().numpy()
    r = np.linalg.cholesky(u.T @ u * c.dV).T
    ref = np.linalg.solve(r.T, u.T).T
    assert np.abs(g.T @ g * c.dV - np.eye(nb)).max() <= 1e-14
    # condition of the overlap times EPS, a small factor for the two orders of summation
    assert np.abs(g - ref).max() <= 50 * EPS * np.linalg.cond(u) ** 2 * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 100])
def test_cholesky(gpu, n):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, 2 * n + 1))
    s = a @ a.T / n
    rinv = api.fortran_empty(n, n)
    gpu.overlap_cholesky(dev(s), rinv)
    gpu.synchronize()
    ref = np.linalg.inv(np.linalg.cholesky(s).T)
    cond = np.linalg.cond(s)
    assert np.abs(rinv.cpu().numpy() - ref).max() <= 20 * n * EPS * cond * np.abs(ref).max()


def test_cholesky_not_positive(gpu):
    s = np.eye(70)
    s[40, 40] = -1.0
    with pytest.raises(api.RsdftError, match="info=41"):
        gpu.overlap_cholesky(dev(s), api.fortran_empty(70, 70))


@pytest.mark.parametrize("nb,zero", [(1, False), (31, False), (33, True), (70, True)])
def test_adjoint_bands(gpu, nb, zero):
    """Force and potential gradient at the edges of the band chunks, with empty bands (whose values are not read)."""
    c = build_cell(Workload("adj", 1, 14, nb, nb, 0.03, 4000 + nb))
    gpu.setup(c)
    rng = np.random.default_rng(nb)
    u, x = rng.normal(size=(c.ML, nb)), rng.normal(size=(c.ML, nb))
    occ = rng.uniform(0.5, 2.0, nb)
    if zero:
        occ[::3] = 0.0
        u[:, ::3] = np.nan
    used = np.flatnonzero(occ)

    def tables(values):
        t = np.zeros((c.nzlma, c.ML))
        for m in range(c.nzlma):
            s = slice(c.lma_ptr[m], c.lma_ptr[m + 1])
            np.add.at(t[m], c.jjp[s], values[s])
        return t

    uv, duv = tables(c.uv), [tables(c.duv[:, k]) for k in range(3)]
    force = torch.zeros(3 * c.natom, dtype=torch.float64, device="cuda")
    dv = torch.zeros(c.ML, dtype=torch.float64, device="cuda")
    gpu.calc_force_ps_nloc2(c.natom, force, dev(u), torch.from_numpy(occ).cuda())
    gpu.hpsi_adjoint(dev(u), occ=torch.from_numpy(occ).cuda(), dl_dv=dv)
    gpu.synchronize()
    w = u[:, used]
    per = np.stack([-2.0 * c.dV ** 2 * c.iuv * ((uv @ w) * (d @ w) * occ[used]).sum(1) for d in duv], 1)
    ref = np.zeros((c.natom, 3))
    np.add.at(ref, c.amap, per)
    assert np.abs(force.cpu().numpy().reshape(-1, 3) - ref).max() <= 1e-12 * np.abs(ref).max()
    rdv = c.dV * (occ[used] * w * w).sum(1)
    assert np.abs(dv.cpu().numpy() - rdv).max() <= 1e-13 * rdv.max()
    if zero:
        return
    dr = torch.zeros(3 * c.natom, dtype=torch.float64, device="cuda")
    gpu.hpsi_adjoint(dev(u), chi=dev(x), dl_dv=dv, dl_dr=dr)
    gpu.synchronize()
    per = np.stack([c.dV * c.iuv * ((d @ x) * (uv @ u) + (uv @ x) * (d @ u)).sum(1) for d in duv], 1)
    ref = np.zeros((c.natom, 3))
    np.add.at(ref, c.amap, per)
    assert np.abs(dr.cpu().numpy().reshape(-1, 3) - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.abs(dv.cpu().numpy() - (u * x).sum(1)).max() <= 1e-13 * np.abs(u * x).sum(1).max()
