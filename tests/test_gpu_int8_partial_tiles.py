"""The int8 form over several interacting steps at radii that do not fill its angular tiles (32 radii up to 128
channels, 16 above), against the oracle: phases of the laser, Hartree and exchange on, kept vectors stored and
read back where a tile's last radii are missing, odd and even N_r.

Bar: 3e-5, as the other int8 tests against the oracle over 48 steps (these are 12).
"""
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation
from oracle.step_oracle import propagate
from tests.helpers import rel_err, to_oracle

pytestmark = pytest.mark.gpu

TOL_I8 = 3e-5


@pytest.mark.parametrize("n_r,n_l,angular,n_har", [(45, 33, "theta", 4), (70, 33, "theta", 4), (45, 97, "theta", 4), (70, 128, "theta", 4),
                                                   (45, 131, "theta", 4), (70, 161, "theta", 4), (37, 220, "theta", 4),
                                                   (45, 40, "theta", 79), (45, 35, "reference", 4), (51, 134, "reference", 4),
                                                   pytest.param(39, 201, "reference", 4, marks=pytest.mark.xfail(
                                                       strict=True, reason="the form's own error: the acceleration is 3.3e-5 off "
                                                       "at this size, with untrimmed stage images too"))])
def test_steps_on_part_full_tiles_track_the_oracle(n_r, n_l, angular, n_har):
    run = P.reference_like(n_r, n_l, 12, "Ne3", r_mask=15.0, dt_as=10.0, perturb=0.05, seed=7)
    run = dataclasses.replace(run, angular=angular, n_har=n_har)
    assert np.abs(run.E).max() > 0.01
    ref = propagate(to_oracle(run))
    for reuse in (True, False) if angular == "theta" else (True,):
        # alone, and as the second of two runs of a group (columns after another run's)
        for copies in (1, 2):
            runs = [run.with_field(run.E * (1.0 + 0.5 * i)) for i in range(copies - 1, -1, -1)]
            tp = TimePropagation(runs, precision="split_int8", groups=[list(range(copies))], theta_reuse=reuse)
            tp.step(12)
            x, got = tp.orbitals(copies - 1), tp.observables(copies - 1)
            st, msg = tp.status()
            tp.close()
            assert st == 0, msg
            assert rel_err(x, ref["x"]) < TOL_I8
            assert rel_err(got["norm"], ref["norm"]) < TOL_I8
            for key in ("dipole", "acceleration"):
                assert rel_err(got[key].sum(axis=0), ref[key].sum(axis=0)) < TOL_I8, key
