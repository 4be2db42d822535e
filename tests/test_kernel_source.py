"""Rules of the CUDA source that no run can show to be kept: a kernel launched
while its predecessor still runs must not read through the read-only path what
that predecessor writes, and an iteration that gives up leaves no step length
for the grouped solution update."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pot3d_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _functions(src):
    """name -> parameters and body, of the __global__ and __device__ functions."""
    out = {}
    for m in re.finditer(r"__(?:global|device)__[^;{]*?\b(\w+)\(", src):
        if m.group(1) == "__launch_bounds__":
            m = re.compile(r"[^;{]*?\b(\w+)\(").match(src, src.index(")", m.end()) + 1)
        start = src.index("{", m.end())
        depth, end = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
        out[m.group(1)] = src[m.end():end]
    return out


def test_overlapped_kernels_read_only_setup_data_through_the_read_only_path():
    src = _source("pcg.cu")
    fn = _functions(src)
    launched = {k for call in re.findall(r"launch_pdl\(([^;]*);", src) for k in re.findall(r"\bk_\w+\b(?!\")", call)}
    assert launched == {"k_stencil", "k_update", "k_update_x_group"}
    for k in launched:
        bodies = [fn[k]] + [fn[c] for c in re.findall(r"\b(\w+_body)\b", fn[k])]
        text = "".join(bodies)
        assert "pdl_wait();" in text, k
        for arg in re.findall(r"__ldg\((.*?)\)\)?;", text):
            assert re.search(r"\(a\.ai\b", arg), (k, arg)
        for par in re.findall(r"const [^,()]*__restrict__[^,()]*", text):
            assert "BatchInst" in par, (k, par)
        assert "ld.global.nc" not in text


def test_every_early_exit_of_the_stencil_clears_its_step_length():
    body = _functions(_source("pcg.cu"))["stencil_body"]
    exits = [body[:m.start()].rsplit("if (", 2) for m in re.finditer(r"\breturn;", body)]
    assert len(exits) == 2  # not running any more; a wait that ran out
    for e in exits:
        assert re.search(r"if \(a\.xslot1\b[^;]*a\.st->xa\[a\.xslot1 - 1\] = 0\.0;", "if (" + "if (".join(e[1:])), e[1:]
