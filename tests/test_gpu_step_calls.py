"""One call of n steps equals n calls of one step, every series, orbital and potential, where steps fork
(k_finalize beside the exact multipoles) and where they do not, in one grid group and in several."""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation

pytestmark = pytest.mark.gpu


def _run(n_r, n_l, n_har, seed):
    run = P.reference_like(n_r, n_l, 64, "Ne3", r_mask=12.0, dt_as=10.0, perturb=0.05, seed=seed)
    return dataclasses.replace(run, angular="theta", n_har=n_har)


@pytest.mark.parametrize("precision", ["fp64", "split_int8"])
@pytest.mark.parametrize("groups", [[(37, 9, 4)], [(37, 9, 17)], [(37, 9, 17), (45, 12, 23)], [(37, 9, 17), (45, 12, 4), (33, 33, 65)],
                                    [(40, 131, 9), (37, 9, 17)]])
def test_steps_in_one_call_equal_single_steps(precision, groups):
    """The same kernels on the same data: the same bits, with calls on both sides of the long graph's length.
    Every run of several groups also equals the run stepped alone."""
    runs = [_run(*g, seed=i) for i, g in enumerate(groups)]
    one, many = (TimePropagation(runs, precision=precision, per_l=True) for _ in range(2))
    assert len(one.groups) == len(groups)
    for n in (0, 1, 7, 8, 9, 33):
        many.step(n)
        for _ in range(n):
            one.step(1)
    for i, r in enumerate(runs):
        alone = TimePropagation([r], precision=precision, per_l=True)
        alone.step(58)
        for other in (one, alone):
            k = i if other is one else 0
            assert np.array_equal(many.orbitals(i), other.orbitals(k))
            a, b, u, v = many.observables(i), other.observables(k), many.potentials(i), other.potentials(k)
            assert a["dipole"].shape[-1] == 58
            for key in a:
                assert np.array_equal(a[key], b[key]), key
            for key in u:
                assert np.array_equal(u[key], v[key]), key
        alone.close()
    assert many.status()[0] == 0
    one.close()
    many.close()
