"""The INT8 slices of the FP64 products are optional memory: the products do without them where they would take more than
half of what is free, and they give way to any other allocation.  In a process of its own, whose device memory a torch
tensor fills up to a given rest."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import numpy as np, torch
from rsdft_b200 import api
from rsdft_b200.cell import Workload, build_cell
path, rest = sys.argv[1], float(sys.argv[2])
g = api.RsdftGpu(0)
st = torch.cuda.Stream()
torch.cuda.set_stream(st)
g.set_stream(st.cuda_stream)
c = build_cell(Workload("mem", 2, 48, 160, 144, 0.02, 1002))
g.setup(c)
gen = torch.Generator(device="cuda")
gen.manual_seed(7)
block = 8 * c.ML * 160
x = torch.randn((160, c.ML), dtype=torch.float64, device="cuda", generator=gen).t()
esp = torch.zeros(160, dtype=torch.float64, device="cuda")
res = torch.zeros_like(esp)
g.esp_calc(1, 1, x, 1, c.ML, 1, 1, esp)  # the kernels' code is loaded on first use
g.synchronize()
torch.cuda.empty_cache()
free = torch.cuda.mem_get_info()[0]
if rest > 0:
    fill = torch.empty(int(free - rest * block), dtype=torch.uint8, device="cuda")
g.gram_schmidt(1, 160, 1, 1, x)
g.synchronize()
u = x.cpu().numpy()
g.conjugate_gradient(1, c.ML, 160, 1, 1, x, esp, res, ncg=1, mloop=3)
g.synchronize()
np.savez(path, u=u, x=x.cpu().numpy(), esp=esp.cpu().numpy())
"""


def run(tmp_path, rest):
    out = str(tmp_path / f"r{rest}.npz")
    r = subprocess.run([sys.executable, "-c", CHILD, out, str(rest)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(out)


def test_slices_give_way(gpu, tmp_path):
    """Rests in units of the band block.  9.8: Gram-Schmidt takes its copy (1) and the slices (2), the CG's vectors (7 and
    partial sums) only fit without those.  2.6: no room for slices, the DMMA form runs; then the CG does not fit, as
    it never did."""
    free = run(tmp_path, 0)
    tight = run(tmp_path, 9.8)
    for k in ("u", "x", "esp"):
        np.testing.assert_array_equal(tight[k], free[k])
    with pytest.raises(AssertionError, match="ENOMEM"):
        run(tmp_path, 2.6)


def test_products_without_slices(gpu, tmp_path):
    """The same bands with the slices refused: equal to rounding (condition of 160 random bands about 1.1)."""
    free = run(tmp_path, 0)
    global CHILD
    child = CHILD
    try:
        CHILD = child.split("g.conjugate_gradient")[0] + "np.savez(path, u=u)\n"
        none = run(tmp_path, 2.6)
    finally:
        CHILD = child
    assert not np.array_equal(none["u"], free["u"])
    assert np.abs(none["u"] - free["u"]).max() <= 1e-14 * np.abs(free["u"]).max()
