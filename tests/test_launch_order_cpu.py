"""Order of the dependent-launch calls in the kernel sources.

A kernel that lets its successor begin before it holds its tensor memory can wait
for good: the successor may take the columns and then waits for the kernel's end.
Neither wait has a bound, so the order is checked here, where nothing runs.  And what
a caller's kernel may have written just before a step is read after the wait.
"""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "ionosphere_fdtd_b200" / "csrc"


def kernels() -> dict[str, str]:
    """Body of every __global__ function, by name, without comments."""

    out = {}
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            brace = text.index("{", m.end())
            if ";" in text[m.end():brace]:
                continue
            depth, at = 1, brace + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            head = re.sub(r"__(launch_bounds|maxnreg)__\s*\([^()]*\)", "", text[m.end():brace])
            out[re.search(r"(\w+)\s*\(", head).group(1)] = text[brace:at]
    return out


def test_tensor_memory_is_held_before_the_next_launch_begins():
    both = {n: b for n, b in kernels().items() if "tcgen05.alloc" in b and "launch_next()" in b}
    assert "layer_gemm" in both
    for name, body in both.items():
        held = body.index("__syncthreads()", body.index("tcgen05.alloc"))
        assert body.index("launch_next()") > held, name


def test_source_currents_are_read_after_the_wait():
    both = {n: b for n, b in kernels().items() if "R.cur[" in b and "wait_previous()" in b}
    assert {"ke_tma", "ke_tma_batch"} <= both.keys()
    for name, body in both.items():
        assert body.rindex("wait_previous()", 0, body.index("R.cur[")) > 0, name
        assert "wait_previous()" not in body[body.index("R.cur["):], name
