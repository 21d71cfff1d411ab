"""A cluster barrier of the aligned form is executed by the threads of a warp together.  Behind code that lanes leave one by one that is
not a matter of course: there a __syncwarp() (or a barrier of the CTA) stands in front of it in the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cnet_b200", "csrc")


def _body(text, name):
    """The text of the kernel `name`, by its braces."""
    at = text.index("{", re.search(r"\b%s\s*\(" % name, text).end())
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at:i]


def test_a_product_of_a_cluster_ends():
    with open(os.path.join(CSRC, "cgemm_tc.cu")) as f:
        lines = [re.sub(r"//.*", "", line).strip() for line in f]
    last = max(i for i, line in enumerate(lines) if "cluster_reduce<8, VEC, TN>" in line)
    i = next(i for i in range(last, len(lines)) if lines[i] == "cluster_sync();")
    assert lines[i - 1] == "__syncwarp();"


def test_packing_by_a_cluster():
    with open(os.path.join(CSRC, "cgemm_tc.cu")) as f:
        lines = [re.sub(r"//.*", "", line).strip() for line in _body(f.read(), "pack_one_k").split("\n")]
    lines = [line for line in lines if line]
    barriers = [i for i, line in enumerate(lines) if "barrier.cluster" in line or line == "cluster_sync();"]
    assert len(barriers) == 3
    for i in barriers:
        assert lines[i - 1] in ("__syncwarp();", "__syncthreads();"), lines[i - 2:i + 1]
