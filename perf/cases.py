"""The timed cases of the framework: what a Kohn-Sham program calls, over the sizes it calls it at.

Every case is one public call of ``rsdft_b200.api.RsdftGpu`` (the calls the
Fortran shim forwards) on a periodic silicon cell of ``rsdft_b200.cell``:

======== =====================================================================
kind     call
======== =====================================================================
hpsi     ``hamiltonian``: H psi of a band block
cg       ``conjugate_gradient``: one CG sweep (4 line steps, mloop 3, IPC 4)
gs       ``gram_schmidt`` on bands as a CG sweep leaves them
sd       ``subspace_diag`` of orthonormal bands
sweep    ``eigensolver_iteration``: CG, Gram-Schmidt and subspace_diag
adjoint  ``hpsi_adjoint`` (potential and positions) and ``calc_force_ps_nloc2``
======== =====================================================================

``n`` is the number of grid points per axis, ``bands`` the band count, ``md``
the finite-difference order and ``mode`` the precision form: ``fp64``, or
``bf16x3`` (FP32 CG, split-BF16 contractions).  The cell (potential, projector
tables) of a size is the program's set-up and is uploaded once; the bands are
made from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rsdft_b200 import api
from rsdft_b200.cell import Workload, build_cell

NCG, MLOOP = 4, 3
MODES = {"fp64": api.MODE_FP64, "bf16x3": api.MODE_MIXED_BF16X3}
# bands whose kinetic energy is well above this (Ha) are damped in the start bands
SMOOTH_HA = 1.0
# the smallest and largest numbers of bands of a drawn case
BANDS = (8, 640)


def _case(name, kind, n, bands, mode="fp64", md=6):
    return {"name": name, "kind": kind, "n": n, "bands": bands, "mode": mode, "md": md}


def listed():
    return [
        # H psi alone: the call of a residual or energy evaluation.  The 8-atom
        # cell is launch-bound; the 216-atom cell is the size quoted for the
        # framework; the 45-point grid with 101 bands is an odd width, as user
        # input often gives.
        _case("hpsi 24^3 x 32", "hpsi", 24, 32),
        _case("hpsi 45^3 x 101", "hpsi", 45, 101),
        _case("hpsi 72^3 x 480", "hpsi", 72, 480),
        # One CG sweep: what calc_sweep spends most of its time on, in the plain
        # form on the 64-atom cell and in the mixed form on the 216-atom cell.
        _case("cg 48^3 x 160", "cg", 48, 160),
        _case("cg 72^3 x 480 mixed", "cg", 72, 480, "bf16x3"),
        # The dense steps by themselves, as a program calls them that has its
        # own minimiser: orthonormalisation of the large band set and
        # Rayleigh-Ritz of the middle one.
        _case("gs 72^3 x 480", "gs", 72, 480),
        _case("sd 48^3 x 160", "sd", 48, 160),
        # Whole iterations of calc_sweep: the smallest cell (an interactive
        # run), the headline cell in both precision forms and the largest cell.
        _case("sweep 24^3 x 32", "sweep", 24, 32),
        _case("sweep 72^3 x 480", "sweep", 72, 480),
        _case("sweep 72^3 x 480 mixed", "sweep", 72, 480, "bf16x3"),
        _case("sweep 96^3 x 1088 mixed", "sweep", 96, 1088, "bf16x3"),
        # The backward direction: gradients of the band energy with respect to
        # the local potential and the atoms, and the nonlocal force.
        _case("adjoint 72^3 x 480", "adjoint", 72, 480),
    ]


def draw(rng):
    kind = rng.choice(["hpsi", "cg", "cg", "gs", "sd", "sweep", "sweep", "adjoint"])
    n = round(math.exp(rng.uniform(math.log(16), math.log(80))))
    if rng.random() < 0.75:
        n += n % 2  # even grids are the rule, odd ones come too
    ml = n ** 3
    lo, hi = max(BANDS[0], ml / 2000), min(BANDS[1], ml / 200, 480 * 72 ** 3 / ml)
    bands = max(BANDS[0], round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))
    mode = rng.choice(["fp64", "bf16x3"]) if kind in ("cg", "sweep", "gs", "sd") else "fp64"
    mode = mode if n % 2 == 0 else "fp64"  # the mixed contractions take grids of a multiple of 8 points
    return {"kind": kind, "n": n, "bands": bands, "mode": mode, "md": rng.choice([4, 6, 6, 6, 8])}


# ----------------------------------------------------------------- set-up
@functools.lru_cache(maxsize=4)
def _cell(n, bands, md):
    ncell = max(1, round(n / 24))  # 0.43 bohr spacing, as the framework's own cells have
    nocc = max(1, round(0.9 * bands))
    return build_cell(Workload(f"si{8 * ncell ** 3}_{n}", ncell, n, bands, nocc, 0.02, 1003, md))


class _Session:
    """The one library context of the process, on a stream shared with torch."""

    def __init__(self):
        self.gpu = api.RsdftGpu(0)
        self.stream = torch.cuda.Stream()
        self.gpu.set_stream(self.stream.cuda_stream)
        self.cell = None

    def use(self, cell):
        torch.cuda.set_stream(self.stream)
        if self.cell is not cell:
            self.gpu.setup(cell)
            self.cell = cell
        return self.gpu


@functools.lru_cache(maxsize=1)
def _session():
    return _Session()


def _smooth(cell, nb, gen):
    """nb rows of Gaussian noise, damped above SMOOTH_HA as bands are after the first iterations."""
    n = cell.ngrid[0]
    k = 2.0 * math.pi * torch.fft.fftfreq(n, d=1.0 / n, dtype=torch.float64, device="cuda") / cell.a
    kr = k[: n // 2 + 1].abs()
    e = 0.5 * (k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2)
    damp = 1.0 / (1.0 + (e / SMOOTH_HA) ** 2)
    out = torch.empty((nb, cell.ML), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // cell.ML)
    for b in range(0, nb, step):
        m = min(step, nb - b)
        w = torch.randn((m, n, n, n), dtype=torch.float64, device="cuda", generator=gen)
        out[b:b + m] = torch.fft.irfftn(torch.fft.rfftn(w, dim=(1, 2, 3)) * damp, s=(n, n, n), dim=(1, 2, 3)).view(m, -1)
    return out


def _orthonormal(x, dv):
    chol = torch.linalg.cholesky((x @ x.t()) * dv)
    return torch.linalg.solve_triangular(chol, x, upper=False).contiguous()


def _bands(case, seed):
    """(nb, ML) rows: orthonormal smooth bands; for Gram-Schmidt, with the overlaps of a CG sweep."""
    cell = _cell(case["n"], case["bands"], case["md"])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = _orthonormal(_smooth(cell, case["bands"], gen), cell.dV)
    if case["kind"] == "gs":
        y = _smooth(cell, case["bands"], gen)
        x += y * (0.2 / torch.sqrt((y * y).sum(1, keepdim=True) * cell.dV))
    return x


def prepare(case, seed):
    cell = _cell(case["n"], case["bands"], case["md"])
    gpu = _session().use(cell)
    nb, kind = case["bands"], case["kind"]
    start = _bands(case, seed).t()  # column-major (ML, nb)
    s = {"kind": kind, "gpu": gpu, "cell": cell, "mode": MODES[case["mode"]], "start": start}
    if kind in ("hpsi", "cg", "gs", "sd", "sweep"):
        s["out"] = api.fortran_empty(cell.ML, nb)
    if kind in ("cg", "sd", "sweep"):
        s["esp"] = torch.zeros(nb, dtype=torch.float64, device="cuda")
        s["res"] = torch.zeros(nb, dtype=torch.float64, device="cuda")
        s["gauge"] = _gauge(cell)
    if kind == "adjoint":
        s["occ"] = torch.from_numpy(cell.occupations()).cuda()
        s["dv"] = torch.zeros(cell.ML, dtype=torch.float64, device="cuda")
        s["dr"] = torch.zeros(3 * cell.natom, dtype=torch.float64, device="cuda")
        s["force"] = torch.zeros(3 * cell.natom, dtype=torch.float64, device="cuda")
    torch.cuda.current_stream().synchronize()
    return s


# -------------------------------------------------------------------- run
def _gauge(cell):
    i = torch.arange(min(cell.ML, 4096), dtype=torch.float64, device="cuda")
    return torch.cos(1.7 * i + 0.3 * i * i)


def _fix_sign(u, gauge):
    """Each band's sign, which an eigenvector leaves open, from a fixed functional (as a restart needs it)."""
    sign = torch.sign(u[: gauge.numel()].t() @ gauge)
    return u.mul_(sign + (sign == 0))


def run(state):
    """One call.  CG, Gram-Schmidt and subspace_diag work in place, so they get the start bands anew."""
    s = state
    cell, kind = s["cell"], s["kind"]
    gpu = _session().use(cell)
    nb = s["start"].shape[1]
    if kind == "hpsi":
        gpu.hamiltonian(1, 1, s["start"], s["out"], 1, cell.ML, 1, nb)
        return s["out"]
    if kind == "adjoint":
        gpu.hpsi_adjoint(s["start"], occ=s["occ"], dl_dv=s["dv"], dl_dr=s["dr"])
        gpu.calc_force_ps_nloc2(cell.natom, s["force"], s["start"], s["occ"])
        return s["dv"], s["dr"], s["force"]
    u = s["out"]
    u.copy_(s["start"])
    if kind == "gs":
        gpu.gram_schmidt(1, nb, 1, 1, u, mode=s["mode"])
        return u
    if kind == "cg":
        gpu.conjugate_gradient(1, cell.ML, nb, 1, 1, u, s["esp"], s["res"], ncg=NCG, mloop=MLOOP, mode=s["mode"])
        return u, s["esp"], s["res"]
    if kind == "sd":
        gpu.subspace_diag(1, 1, u, s["esp"], mode=s["mode"])
        return _fix_sign(u, s["gauge"]), s["esp"]
    gpu.eigensolver_iteration(u, s["esp"], s["res"], ncg=NCG, mloop=MLOOP, mode=s["mode"])
    return _fix_sign(u, s["gauge"]), s["esp"], s["res"]


# ------------------------------------------------------------------- work
def work(case):
    """Bytes: bands read and written once, potential and projector tables once.
    Flops: the finite-difference, projector, preconditioner and dense products."""
    cell = _cell(case["n"], case["bands"], case["md"])
    ml, nb, nnz = cell.ML, case["bands"], int(cell.lma_ptr[-1])
    tables = 8.0 * ml + 12.0 * nnz
    bands = 8.0 * ml * nb
    h = nb * (ml * (9.0 * case["md"] + 3.0) + 4.0 * nnz)
    gram, rot = 1.0 * ml * nb * nb, 2.0 * ml * nb * nb  # a symmetric Gram matrix, a rotation
    solve = 9.0 * nb ** 3
    cg = (NCG + 1) * h + NCG * nb * ml * (MLOOP * 18.0 + 40.0)
    kind = case["kind"]
    if kind == "hpsi":
        return {"bytes": 2 * bands + tables, "flops": h}
    if kind == "cg":
        return {"bytes": 2 * bands + tables, "flops": cg}
    if kind == "gs":
        return {"bytes": 2 * bands, "flops": 2 * (gram + rot)}
    if kind == "sd":
        return {"bytes": 2 * bands + tables, "flops": h + gram + rot + solve}
    if kind == "sweep":
        return {"bytes": 2 * bands + tables, "flops": cg + 2 * gram + rot + solve}
    occ = case["bands"] * 8.0 * ml
    return {"bytes": occ + 8.0 * ml + 36.0 * nnz, "flops": nb * (3.0 * ml + 16.0 * nnz)}


def tolerance(case):
    """About four times the distance from ``exact`` seen over these sizes."""
    kind, mixed = case["kind"], case["mode"] != "fp64"
    if kind in ("hpsi", "adjoint"):
        return {"rel": 1e-14, "max": 1e-12}
    if kind == "gs":
        return {"rel": 1e-6, "max": 1e-5} if mixed else {"rel": 2e-14, "max": 1e-12}
    if kind == "cg":
        return {"rel": 1e-4, "max": 1e-3} if mixed else {"rel": 5e-13, "max": 5e-12}
    # Rayleigh-Ritz: a band is determined up to (error of Hsub) / (gap to the next Ritz value)
    if kind == "sd":
        return {"rel": 1e-5, "max": 1e-4} if mixed else {"rel": 2e-12, "max": 1e-10}
    return {"rel": 1e-4, "max": 2e-2} if mixed else {"rel": 5e-11, "max": 5e-9}


# --------------------------------------- the same results in plain 64 bits
class _Exact:
    """H, the CG sweep and the dense steps in plain torch, 64 bits, bands as rows."""

    def __init__(self, cell):
        self.cell, self.shape = cell, tuple(reversed(cell.ngrid))
        self.v = torch.from_numpy(cell.vloc).cuda()
        lma = np.repeat(np.arange(cell.nzlma), np.diff(cell.lma_ptr))
        at = torch.from_numpy(np.stack([lma, cell.jjp.astype(np.int64)])).cuda()

        def table(values):
            t = torch.from_numpy(np.ascontiguousarray(values)).cuda()
            return torch.sparse_coo_tensor(at, t, (cell.nzlma, cell.ML)).coalesce()

        self.uv = table(cell.uv)
        self.uvt = self.uv.t().coalesce()
        self.duv = [table(cell.duv[:, k]) for k in range(3)]
        self.iuv = torch.from_numpy(cell.iuv.astype(np.float64)).cuda()

    def _taps(self, x, weights, centre):
        f = x.view(-1, *self.shape)
        out = centre * f
        for axis in range(3):
            for m, w in enumerate(weights[axis], 1):
                out += w * (torch.roll(f, m, 3 - axis) + torch.roll(f, -m, 3 - axis))
        return out.view(x.shape)

    def h(self, x):
        c, out = self.cell, torch.empty_like(x)
        step = max(1, (1 << 25) // c.ML)
        for b in range(0, x.shape[0], step):
            y = x[b:b + step]
            t = self._taps(y, c.coef_lap, c.coef_lap0) + self.v * y
            p = self.iuv[:, None] * c.dV * torch.sparse.mm(self.uv, y.t().contiguous())
            out[b:b + step] = t + torch.sparse.mm(self.uvt, p).t()
        return out

    def a(self, x):  # the 7-point operator of the preconditioner
        g = [1.0 / float(h) ** 2 for h in self.cell.h]
        return self._taps(x, [[-0.5 * v] for v in g], sum(g))

    def dot(self, x, y):
        return (x * y).sum(1)

    def precondition(self, g):
        z, r = g.clone(), g - self.a(g)
        q, rr = r.clone(), self.dot(r, r)
        live = (rr >= 1e-24)
        for it in range(MLOOP):
            f = self.a(q)
            al = torch.where(live, rr / self.dot(q, f), 0.0)
            z += al[:, None] * q
            if it + 1 < MLOOP:
                r = r - al[:, None] * f
                rn = self.dot(r, r)
                q = r + torch.where(live, rn / rr, 0.0)[:, None] * q
                rr = rn
        return z

    def cg(self, x, tol=1e-15):
        dv = self.cell.dV
        hx = self.h(x)
        e = self.dot(x, hx) * dv
        e1 = torch.full_like(e, 1e10)
        g = -2.0 * (hx - e[:, None] * x)
        rb = self.dot(g, g) * dv
        res, gkgk, p = torch.zeros_like(e), torch.ones_like(e), None
        on = torch.ones_like(e, dtype=torch.bool)
        for icg in range(NCG + 1):
            res = torch.where(on, rb / 4.0, res)
            on = on & ((e - e1).abs() >= tol)
            if icg == NCG:
                break
            z = self.precondition(g)
            rb = self.dot(z, g) * dv
            p = z if p is None else z + (rb / gkgk)[:, None] * p
            gkgk = rb
            hp = self.h(p)
            pairs = ((x, x), (p, x), (p, p), (x, hx), (p, hx), (p, hp))
            b11, b12, b22, a11, a12, a22 = (self.dot(u, w) * dv for u, w in pairs)
            chol = torch.linalg.cholesky(torch.stack([b11, b12, b12, b22], 1).view(-1, 2, 2))
            amat = torch.stack([a11, a12, a12, a22], 1).view(-1, 2, 2)
            m = torch.linalg.solve_triangular(chol, amat, upper=False)
            m = torch.linalg.solve_triangular(chol, m.mT, upper=False)
            w, z2 = torch.linalg.eigh(0.5 * (m + m.mT))
            u = torch.linalg.solve_triangular(chol.mT, z2, upper=True)
            pick = ((w[:, 0] - e).abs() > 1e-1) & ((w[:, 1] - e).abs() <= 1e-1)
            u = torch.where(pick[:, None], u[:, :, 1], u[:, :, 0])
            u = u * torch.where(u[:, :1] < 0, -1.0, 1.0)
            wn = torch.where(pick, w[:, 1], w[:, 0])
            e1, e = torch.where(on, e, e1), torch.where(on, wn, e)
            u11 = torch.where(on, u[:, 0], 1.0)[:, None]
            u21 = torch.where(on, u[:, 1], 0.0)[:, None]
            hx = u11 * hx + u21 * hp
            x = u11 * x + u21 * p
            g = -2.0 * (hx - e[:, None] * x)
            rb = self.dot(g, g) * dv
        return x, e, res

    def ritz(self, x):
        dv = self.cell.dV
        x = _orthonormal(x, dv)
        hs = (x @ self.h(x).t()) * dv
        e, v = torch.linalg.eigh(0.5 * (hs + hs.t()))
        return v.t() @ x, e


def exact(case, seed):
    if case["n"] ** 3 * case["bands"] > 480 * 72 ** 3:
        return None  # the 512-atom cell: over 20 seconds
    cell = _cell(case["n"], case["bands"], case["md"])
    x, ref, kind = _bands(case, seed), _Exact(cell), case["kind"]
    mixed = case["mode"] != "fp64"
    if kind == "hpsi":
        return ref.h(x).t()
    if kind == "gs":
        return _orthonormal(_orthonormal(x, cell.dV), cell.dV).t()
    if kind == "adjoint":
        occ = torch.from_numpy(cell.occupations()).cuda()
        dv = cell.dV * (occ[:, None] * x * x).sum(0)
        xt = x.t().contiguous()
        t = torch.sparse.mm(ref.uv, xt)
        lma = [2.0 * cell.dV ** 2 * (occ * t * torch.sparse.mm(d, xt)).sum(1) * ref.iuv for d in ref.duv]
        dr = torch.zeros((cell.natom, 3), dtype=torch.float64, device="cuda")
        dr.index_add_(0, torch.from_numpy(cell.amap.astype(np.int64)).cuda(), torch.stack(lma, 1))
        return dv, dr.view(-1), -dr.view(-1)
    if kind == "cg":
        x, e, res = ref.cg(x)
        return x.t(), e, res
    gauge = _gauge(cell)
    res = None
    if kind == "sweep":
        x, _, res = ref.cg(x)
    x, e = ref.ritz(x)
    # in the mixed form the distance of near-degenerate bands from these is chance, so they have no such value
    u = None if mixed else _fix_sign(x.t(), gauge)
    return (u, e, res) if kind == "sweep" else (u, e)
