"""ggb_set_grid after the first step: the exchange potential follows the grid with the next step, with and
without a density that acts back."""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation, _ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,angular", [("fp64", "theta"), ("split_int8", "theta"), ("split_bf16", "reference")])
def test_frozen_exchange_potential_follows_another_grid(precision, angular):
    base = P.reference_like(40, 12, 8, "Ne3", r_mask=12.0, dt_as=10.0, perturb=0.05, seed=1)
    base = dataclasses.replace(base, angular=angular, use_hartree=0, rho_frozen=0.01 * np.exp(-base.grid.r))
    grid = dataclasses.replace(base.grid, drdx=np.ascontiguousarray(0.5 * base.grid.drdx))
    other = dataclasses.replace(base, grid=grid)
    tp, fresh = TimePropagation([base], precision=precision), TimePropagation([other], precision=precision)
    tp.step(2)
    fresh.step(2)
    old = tp.potentials(0)
    tp._call("ggb_set_grid", 0, _ptr(grid.r), _ptr(grid.drdx), _ptr(grid.P), 40)
    tp.step(3)
    new, want = tp.potentials(0), fresh.potentials(0)
    assert not np.array_equal(old["vexc"], want["vexc"])
    assert np.array_equal(new["vexc"], want["vexc"])
    assert np.array_equal(new["vexc0"], old["vexc0"])        # the t = 0 potential stays
    assert tp.observables(0)["norm"].shape[-1] == 5 and tp.status()[0] == 0
    tp.set_orbitals(0, base.x0)
    tp.step(1)
    assert np.array_equal(tp.potentials(0)["vexc0"], want["vexc0"])
    tp.close()
    fresh.close()
