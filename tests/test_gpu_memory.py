"""Device memory that a form does not need is not allocated."""
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation

pytestmark = pytest.mark.gpu


def test_int8_form_holds_fp64_chain_matrices_only_for_fp64_angular_products():
    """The FP64 MMA fragments of the chain matrices (ten matrices of two m, N_l 220: 8 MB) belong to the
    FP64 angular products."""
    import torch
    run = P.reference_like(20, 220, 2, "Ne3", r_mask=8.0, dt_as=10.0)

    def held(angular_fp64):
        tp = TimePropagation([run], precision="split_int8", angular_fp64=angular_fp64)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        tp.step(1)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        tp.close()
        return used

    held(False)                       # module loading and the like
    held(True)
    fragments = 2 * 5 * 2 * 28 * 28 * 64 * 8
    assert held(True) - held(False) > fragments - (4 << 20)
