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


def _body(src, head):
    i = src.index("{", src.index(head))
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        j += 1
        if depth == 0:
            return src[i:j]


def test_a_context_configures_the_kernels_of_its_groups_only():
    """A kernel's first mention in a process loads it, so what every context runs through names none, and a
    group's set-up takes the kernels from the functions that choose them for its launches."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "ggb_kernels_fp64.cu")).read())
    assert not re.search(r"\bk_\w+", _body(src, "cudaError_t configure_kernels_fp64("))
    group = _body(src, "cudaError_t configure_group_fp64(")
    assert not re.search(r"\bk_(angular|radial)_\w+", group)
    for choice, launch in (("angular_launch(g)", "void launch_angular_fp64("), ("radial_tile_of(", "void launch_radial_fp64(")):
        assert choice in group and choice in _body(src, launch)
