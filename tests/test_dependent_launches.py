"""The rules that programmatic dependent launches rest on, read off the CUDA sources (common.cuh, grid_dependency): every
kernel waits for its predecessor first and lets its successor in only then, launches go through launch_as, and a kernel
that may be a dependent reads only the cell's tables, and what its predecessor does not write, through const
__restrict__ parameters or __ldg."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rsdft_b200", "csrc")

# uploaded by rsdft_gpu_set_nonlocal, which returns after the copies
TABLES = {"grp_lma0", "grp_cnt", "lma_ptr", "jjp", "uv", "iuv", "duv", "nl_pts", "nl_ptr", "gpt_grp", "gpt_uv4",
          "atom_ptr", "atom_lma"}
# written by kernels, but not by the launch before: k_ss_p follows s_sstep, which writes per-band scalars (g and hx come
# from the line step before); k_nl_scatter follows the stencil, which writes H psi (uVunk is the projection's, the band
# flags the line step's; rsdft_gpu_op_nonlocal_add, where uVunk may be the launch before's, makes an ordinary launch)
EARLIER = {"k_ss_p": {"g", "hx"}, "k_nl_scatter": {"uvunk", "band_active"}}
ORDINARY = {"k_convert", "k_imma", "k_nl_project", "k_stencil", "k_sytrd", "k_widen"}  # never dependents


def _sources():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        out[os.path.basename(path)] = re.sub(r"//[^\n]*", "", text)
    return out


def _closing(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _kernels(text):
    """(name, parameter list, body) of every __global__ function defined in text."""
    for m in re.finditer(r"__global__", text):
        head = re.compile(r"\b([ks]_\w+)\s*\(").search(text, m.end())
        p0 = head.end() - 1
        p1 = _closing(text, p0, "()")
        b0 = text.index("{", p1)
        yield head.group(1), text[p0 + 1:p1], text[b0 + 1:_closing(text, b0, "{}")]


def test_every_kernel_waits_first():
    names = []
    for name, text in _sources().items():
        for kernel, _, body in _kernels(text):
            assert body.lstrip().startswith("grid_dependency();"), (name, kernel)
            names.append(kernel)
    assert len(names) > 50
    wait = _sources()["common.cuh"].split("void grid_dependency()")[1].split("}")[0]
    assert wait.index("griddepcontrol.wait") < wait.index("griddepcontrol.launch_dependents")


def test_launches_go_through_one_place():
    text = "".join(_sources().values())
    assert text.count("cudaLaunchAttributeProgrammaticStreamSerialization") == 1 and "<<<" not in text
    # k_sytrd's cluster launch is the one other, without that attribute
    assert text.count("cudaLaunchKernelEx(&cfg") == 2
    for kernel in ORDINARY - {"k_sytrd"}:
        assert re.search(r"\blaunch_ordinary\(%s\b" % kernel, text) and not re.search(r"\blaunch\(%s\b" % kernel, text)


def test_dependents_read_coherently():
    for name, text in _sources().items():
        for kernel, params, body in _kernels(text):
            if kernel in ORDINARY:
                continue
            allowed = TABLES | EARLIER.get(kernel, set())
            assert set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)) <= allowed, (name, kernel)
            if kernel not in EARLIER:
                assert set(re.findall(r"__ldg\(\s*(\w+)", body)) <= allowed, (name, kernel)
