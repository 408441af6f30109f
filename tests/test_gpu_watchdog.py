"""The NaN / Inf watchdog (status bit 0) of observables that leave the range of FP64."""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split_int8"])
@pytest.mark.parametrize("scale,status", [(1.0, 0), (1e153, 1)])
def test_a_dipole_that_overflows_while_the_norm_does_not_is_flagged(precision, scale, status):
    """Two rows on the last radius, W = 1 and E = 0: at 1e153 the norm is 2e306 and the dipole, some
    hundreds of radii times that, is out of range."""
    base = P.reference_like(40, 6, 2, "H", r_mask=10.0).with_field(np.zeros(2))
    r = base.grid.r * (1000.0 / base.grid.r[-1])
    w = np.zeros_like(base.W)
    w[:, np.arange(40), np.arange(40)] = 1.0
    x = np.zeros_like(base.x0)
    x[:2, 0, -1] = scale
    run = dataclasses.replace(base, grid=dataclasses.replace(base.grid, r=r), W=w, x0=x, angular="theta")
    tp = TimePropagation([run], precision=precision)
    tp.step(1)
    norm, st = tp.observables(0)["norm"][0, 0], tp.status()[0]
    tp.close()
    assert abs(norm / scale / scale - 2.0) < 1e-6
    assert st == status
