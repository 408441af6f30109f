"""The int8 kernels at the edges of their tiles, bit for bit between shapes that must agree and against
the oracle.

The products accumulate exactly in int32, so a run must give the same bits alone, grouped (another number
of orbital columns per tile, a last tile of 16 to 64 columns) and with any tile width.  Against the FP64
product one step is within 1e-6 of the vector norm (operands of 31 bits, as the other int8 tests).
"""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation

pytestmark = pytest.mark.gpu


def _random(run, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(run.x0.shape) + 1j * rng.standard_normal(run.x0.shape)
    return dataclasses.replace(run, x0=x / np.linalg.norm(x))


@pytest.mark.parametrize("n_r,n_l,cols", [(7, 5, 1), (33, 17, 17), (64, 31, 33), (65, 32, 47), (128, 33, 48), (129, 40, 65),
                                          (136, 64, 90), (137, 65, 96), (31, 97, 3), (40, 128, 20), (33, 129, 5), (50, 145, 2),
                                          (17, 160, 66), (35, 161, 3), (30, 193, 2), (21, 220, 1)])
@pytest.mark.parametrize("angular", ["theta", "reference"])
def test_one_step_is_the_radial_product_at_every_tile_edge(n_r, n_l, cols, angular):
    """E = 0: both angular halves multiply to the identity.  Rows and columns that do not fill a stage,
    one to seven 32-wide k steps (images of pitch 32, 64, 128; one or several rounds of the stages)."""
    base = dataclasses.replace(P.reference_like(n_r, n_l, 2, "H", r_mask=10.0).with_field(np.zeros(2)), angular=angular)
    runs = [_random(base, i) for i in range(cols)]
    tp = TimePropagation(runs, precision="split_int8", groups=[list(range(cols))])
    tp.step(1)
    got = [tp.orbitals(i) for i in range(cols)]
    st, msg = tp.status()
    tp.close()
    assert st == 0, msg
    for i in sorted({0, cols // 2, cols - 1}):
        want = np.einsum("lba,lkb->lka", base.W, runs[i].x0)
        assert np.linalg.norm(got[i] - want) < 1e-6 * np.linalg.norm(want)
        one = TimePropagation([runs[i]], precision="split_int8")
        one.step(1)
        assert np.array_equal(one.orbitals(0), got[i])
        one.close()


@pytest.mark.parametrize("n_l,n_orb_runs", [(33, 1), (97, 12), (161, 4)])
def test_observables_partials_match_the_orbitals(n_l, n_orb_runs):
    """The per-l dipole, acceleration and norm of a step against sums over the orbitals read back: every
    share of the radii (several threads per l), rows per warp and the totals' counters, on two steps."""
    base = P.reference_like(70, n_l, 3, "Ne3", r_mask=15.0, dt_as=10.0, perturb=0.05, seed=9)
    base = dataclasses.replace(base, angular="theta")
    runs = [base.with_field(base.E * (1.0 + 0.1 * i)) for i in range(n_orb_runs)]
    tp = TimePropagation(runs, precision="split_int8")
    tp.step(2)
    r = base.grid.r
    l, m = np.arange(n_l)[:, None], base.m_active[None].astype(float)
    c = np.sqrt(np.where(l >= m, ((l + 1.0) ** 2 - m ** 2) / ((2 * l + 1.0) * (2 * l + 3.0)), 0.0))[..., None]
    for i in (0, n_orb_runs - 1):
        x, got, tot = tp.orbitals(i), tp.observables(i), tp.observables(i, per_l=False)
        z = np.zeros_like(x)
        z[:-1] += c[:-1] * x[1:]
        z[1:] += c[:-1] * x[:-1]
        for key, q in (("dipole", r), ("acceleration", r ** -2.0)):
            want, scale = (x.conj() * z * q).sum(-1), (np.abs(x) * np.abs(z) * q).sum(-1).max()
            assert np.abs(got[key][:, :, 1] - want).max() <= 1e-13 * scale      # 70 terms of FP64
            assert np.abs(tot[key][:, 1] - want.sum(0)).max() <= 1e-13 * scale * n_l
        assert np.allclose(got["norm"][:, 1], (np.abs(x) ** 2).sum(axis=(0, 2)), rtol=1e-13, atol=0)
    tp.close()


@pytest.mark.parametrize("n_r", [511, 512, 513, 1023, 1024, 1025])
def test_slices_of_rows_at_the_register_limits(n_r):
    """Rows of one and two quads per thread and longer ones (read twice): the radial product of a short
    l range against the FP64 product."""
    base = P.reference_like(n_r, 2, 2, "H", r_mask=10.0).with_field(np.zeros(2))
    run = _random(base, n_r)
    tp = TimePropagation([run], precision="split_int8")
    tp.step(1)
    got = tp.orbitals(0)
    tp.close()
    want = np.einsum("lba,lkb->lka", run.W, run.x0)
    assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)
