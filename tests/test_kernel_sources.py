"""Rules of the device code that no run shows, read from its source (CPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ggbtddft_b200", "csrc")


def _kernels():
    """{name: body} of every __global__ function."""
    out = {}
    for fn in sorted(os.listdir(CSRC)):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, fn)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", src):
            i = src.index("{", m.end())
            depth, j = 0, i
            while True:
                depth += {"{": 1, "}": -1}.get(src[j], 0)
                j += 1
                if depth == 0:
                    break
            out[m.group(1)] = src[i:j]
    return out


def test_products_are_committed_by_the_lane_that_issued_them():
    """tcgen05.commit covers the MMAs of the executing thread only: a kernel that issues them from the
    elected lane commits from it everywhere, the drain after a timed-out wait included."""
    elected = {n: b for n, b in _kernels().items() if re.search(r"tc_mma\w*_if\(", b)}
    assert "k_angular_i8" in elected
    for name, body in elected.items():
        assert "tc_commit_if(" in body, name
        assert not re.search(r"\btc_commit\(", body), name
