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


def test_steps_at_radii_that_need_more_shared_memory_than_the_default():
    """3500 radii: the potentials' rows take 56 KB; each form's kernels are configured by its own groups."""
    rng = np.random.default_rng(1)
    base = P.reference_like(40, 4, 2, "Ne3", r_mask=12.0, dt_as=10.0)
    n_r = 3500
    grid = I.make_grid(n_r, 0.5 * n_r, I.zeta_physical_to_ref(0.5, 0.5 * n_r))
    w = np.zeros((4, n_r, n_r), np.complex128)
    w[:, np.arange(n_r), np.arange(n_r)] = 1.0
    x = rng.standard_normal((4, 3, n_r)) + 0j
    x[0, base.m_active == 1] = 0
    run = dataclasses.replace(base, grid=grid, W=w, x0=x / np.linalg.norm(x), rho_frozen=np.zeros(n_r), angular="theta")
    for precision in ("fp64", "split_int8"):
        tp = TimePropagation([run], precision=precision)
        tp.step(2)
        assert np.allclose(tp.observables(0)["norm"].sum(axis=0), 1.0, atol=1e-6) and tp.status()[0] == 0
        tp.close()
