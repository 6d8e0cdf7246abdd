"""The rules that programmatic dependent launches rest on, read off the CUDA sources (common.cuh, grid_dependency): every
kernel waits for its predecessor first and lets its successor in only then, only launch_dependent makes a dependent, and a
kernel launched that way reads what its predecessor writes coherently, that is not through const __restrict__ parameters
or __ldg."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rsdft_b200", "csrc")

# const __restrict__ parameters of dependents, none written by the launch before: k_ss_p follows s_sstep, which writes
# per-band scalars (g and hx come from the line step before); k_nl_scatter follows the stencil, which writes H psi (the
# tables are the cell's, uVunk the projection's, the band flags the line step's)
READ_ONLY = {
    "k_ss_p": {"g", "hx"},
    "k_nl_scatter": {"nl_pts", "nl_ptr", "gpt_grp", "gpt_uv4", "uvunk", "band_active"},
}


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


def _dependents(text):
    for m in re.finditer(r"\blaunch_(?:dependent|as)\(", text):
        args = text[m.end():_closing(text, m.end() - 1, "()")]
        yield from re.findall(r"\b([ks]_[a-z]\w*)\b", args.split("vg,")[0].split("dim3")[0][:160])


def test_every_kernel_waits_first():
    names = []
    for name, text in _sources().items():
        for kernel, _, body in _kernels(text):
            assert body.lstrip().startswith("grid_dependency();"), (name, kernel)
            names.append(kernel)
    assert len(names) > 50
    wait = _sources()["common.cuh"].split("void grid_dependency()")[1].split("}")[0]
    assert wait.index("griddepcontrol.wait") < wait.index("griddepcontrol.launch_dependents")


def test_only_asked_for_launches_are_dependents():
    text = _sources()["common.cuh"]
    plain = text.split("inline void launch(")[1].split("inline void")[0]
    assert "launch_as(false," in plain and "numAttrs" not in plain
    uses = sum(t.count("cudaLaunchAttributeProgrammaticStreamSerialization") for t in _sources().values())
    assert uses == 1


def test_dependents_read_coherently():
    kernels, dependents = {}, set()
    for text in _sources().values():
        kernels.update({k: (p, b) for k, p, b in _kernels(text)})
        dependents.update(_dependents(text))
    dependents &= set(kernels)
    assert {"s_step", "s_eig", "s_sstep", "k_ss_p", "k_pc_tma", "k_cg_upd1", "k_stencil_tma", "k_nl_scatter"} <= dependents
    dependents.add("k_stencil_row")  # launched through a function pointer
    for k in dependents:
        params, body = kernels[k]
        nc = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
        assert nc <= READ_ONLY.get(k, set()), (k, nc)
        assert "__ldg" not in body or k in READ_ONLY, k
