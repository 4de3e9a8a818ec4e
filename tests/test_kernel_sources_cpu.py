"""Rules of the CUDA sources that no run shows reliably, checked by reading them."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jgpt_b200", "csrc")

# Written before the chain of early launches begins: a step's descriptors (copies in front of its first launch), weights and their factors.
WRITTEN_BEFORE = {"seq", "pos", "tok", "segs", "list", "tiles", "entries", "singles", "chunks", "longs", "rowsel", "embed", "pos_table", "gamma", "r"}
# Read by bulk copies and cp.async alone, which are no loads that the compiler could move or mark.
COPIED = {("gemm_umma_kernel", "Aimg"), ("gemm_tc_small_kernel", "A")}


def _closing(s, at, pair):
    depth = 1
    while depth:
        depth += (s[at] == pair[0]) - (s[at] == pair[1])
        at += 1
    return at


def _kernels():
    """(name, parameters, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            s = f.read()
        for m in re.finditer(r"__global__ void ", s):
            at = m.end()
            if s.startswith("__launch_bounds__(", at):
                at = _closing(s, at + len("__launch_bounds__("), "()")
            name = re.compile(r"\s*(\w+)\(").match(s, at)
            end = _closing(s, name.end(), "()")
            body = s.index("{", end)
            yield name[1], s[name.end():end - 1], s[body:_closing(s, body + 1, "{}")]


def test_what_is_read_behind_a_wait_is_not_promised_to_be_read_only():
    """A kernel that is launched early is resident while the launch in front still writes its operands.  As const __restrict__ parameters they
    could be read past the coherent caches, or ahead of the wait."""
    early = [(n, p) for n, p, body in _kernels() if "griddep_wait()" in body]
    assert len(early) >= 28 and "rmsnorm_pack_half_kernel" in dict(early)
    found = {(n, q) for n, p in early for q in re.findall(r"const [^,]*?\*\s*__restrict__ (\w+)", p)}
    assert len(found) >= 30
    assert not {(n, q) for n, q in found if q not in WRITTEN_BEFORE} - COPIED
