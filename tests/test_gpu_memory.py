"""Device memory that a form does not need is not allocated."""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import inputs as I
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


def test_fp64_form_holds_the_chain_matrices_in_fragment_order_only():
    """Ten matrices of eight m, N_l 220: 32 MB as fragments, 32 MB more as plain matrices."""
    import torch
    n_l, n_m = 220, 8
    run = P.reference_like(20, n_l, 2, "Ne3", r_mask=8.0, dt_as=10.0)
    ang = I.angular_eigensystems(n_l, n_m)
    m = np.array([0, 1, n_m - 1], np.int32)
    run = dataclasses.replace(run, V={c: ang[c][0] for c in I.COUPLINGS}, D={c: ang[c][1] for c in I.COUPLINGS}, l_active=m, m_active=m)

    def held():
        tp = TimePropagation([run], precision="fp64")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        tp.step(1)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        tp.close()
        return used

    held()                            # module loading and the like
    fragments = 2 * 5 * n_m * 28 * 28 * 64 * 8
    assert held() < fragments + (16 << 20)
