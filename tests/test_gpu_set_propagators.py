"""ggb_set_radial_propagators after the first step: every form takes the new propagators."""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation, _ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,angular,n_l,n_har", [("fp64", "theta", 12, 4), ("split_int8", "theta", 12, 4),
                                                         ("split_int8", "theta", 14, 17), ("split_int8", "reference", 131, 4),
                                                         ("split_bf16", "reference", 12, 4)])
def test_new_propagators_equal_a_fresh_context(precision, angular, n_l, n_har):
    """Steps with one W, then another W, back to the initial orbitals and steps again: the same bits as a
    context that had the second W from the start; without the restart the state goes on from where it was."""
    base = P.reference_like(40, n_l, 12, "Ne3", r_mask=12.0, dt_as=10.0, perturb=0.05, seed=1)
    base = dataclasses.replace(base, angular=angular, n_har=n_har)
    other = dataclasses.replace(base, W=np.ascontiguousarray(0.5 * base.W[::-1]))
    tp, fresh = TimePropagation([base], precision=precision), TimePropagation([other], precision=precision)
    tp.step(4)
    before = tp.orbitals(0)
    tp._call("ggb_set_radial_propagators", 0, _ptr(other.W))
    assert np.array_equal(tp.orbitals(0), before)
    tp.step(1)                                     # W is half as large
    assert abs(np.linalg.norm(tp.orbitals(0)) / np.linalg.norm(before) - 0.5) < 0.1
    tp.set_orbitals(0, base.x0)
    tp.step(6)
    fresh.step(6)
    assert np.array_equal(tp.orbitals(0), fresh.orbitals(0))
    a, b, u, v = tp.observables(0), fresh.observables(0), tp.potentials(0), fresh.potentials(0)
    assert all(np.array_equal(a[k], b[k]) for k in a) and all(np.array_equal(u[k], v[k]) for k in u)
    tp.close()
    fresh.close()
