"""What only the kernels' source shows."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "brian2cuda_b200", "csrc")


def _body(source: str, name: str) -> str:
    """The braces of the first definition of function `name` and what is between them."""
    at = source.index("{", re.search(rf"\b{name}\(", source).start())
    depth = 0
    for k in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[k], 0)
        if depth == 0:
            return source[at:k + 1]
    raise AssertionError(f"{name} has no end")


def test_split_update_has_one_barrier_outside_its_roles():
    """The warps of a CTA take different roles there; __syncthreads() is defined only where all
    threads of the block reach the same one."""
    with open(os.path.join(CSRC, "neuron.cu")) as f:
        body = _body(f.read(), "hh_split_body")
    body = re.sub(r"//[^\n]*", "", body)
    barriers = [m.start() for m in re.finditer(r"__syncthreads\w*\(", body)]
    assert len(barriers) == 1
    before = body[:barriers[0]]
    assert before.count("{") - before.count("}") == 1
