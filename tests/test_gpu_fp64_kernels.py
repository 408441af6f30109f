"""The FP64 kernels at the edges of their tiles, against NumPy in FP64.

Tolerances: a sum of n products in FP64 is off by at most n eps of the sum of the terms' magnitudes;
the vectors are normalised, so 1e-12 covers n <= 1000 with the angular chain's V V^T on both sides.
"""
import ctypes
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import inputs as I
from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation, load_library

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("n_r,cols", [(5, 1), (31, 2), (32, 3), (33, 4), (37, 5), (64, 6), (65, 7), (100, 8), (129, 9),
                                      (70, 10), (33, 13), (45, 17)])
def test_fp64_radial_product_at_every_column_count(n_r, cols):
    """E = 0 and no Hartree: one step is x <- A x.  Column counts on both sides of the row form's limit,
    radii at the edges of its 32-radius blocks, k slices and 16-wide chunks (down to empty slices)."""
    base = P.reference_like(n_r, 6, 2, "H", r_mask=10.0).with_field(np.zeros(2))
    rng = np.random.default_rng(cols)
    runs = []
    for _ in range(cols):
        x = rng.standard_normal((6, 1, n_r)) + 1j * rng.standard_normal((6, 1, n_r))
        runs.append(dataclasses.replace(base, x0=x / np.linalg.norm(x)))
    tp = TimePropagation(runs, precision="fp64", groups=[list(range(cols))])
    tp.step(1)
    got = [tp.orbitals(i) for i in range(cols)]
    tp.close()
    for r, g in zip(runs, got):
        want = np.einsum("lba,lkb->lka", base.W, r.x0)
        assert np.linalg.norm(g - want) < TOL * np.linalg.norm(want)


@pytest.mark.parametrize("n_r,n_l", [(650, 45), (1001, 33)])
def test_fp64_radial_product_of_few_columns_on_large_grids(n_r, n_l):
    """One, two and six columns where the tiles of 128 radii fill the GPU (the tile form's own column
    counts), the last tile and k chunk part full, and three, which stay on the row form."""
    rng = np.random.default_rng(n_r)
    grid, ang = I.make_grid(n_r, 0.5 * n_r, I.zeta_physical_to_ref(0.5, 0.5 * n_r)), I.angular_eigensystems(n_l, 1)
    w = rng.standard_normal((n_l, n_r, n_r, 2)).view(np.complex128)[..., 0] / np.sqrt(2.0 * n_r)
    for cols in (1, 2, 3, 6):
        x = rng.standard_normal((n_l, cols, n_r)) + 1j * rng.standard_normal((n_l, cols, n_r))
        m = np.zeros(cols, np.int32)
        run = P.RunInputs(grid=grid, n_l=n_l, dt=0.02, W=w, V={c: ang[c][0] for c in I.COUPLINGS},
                          D={c: ang[c][1] for c in I.COUPLINGS}, x0=x / np.linalg.norm(x), l_active=m, m_active=m, occ=m + 1,
                          rho_frozen=np.zeros(n_r), E=np.zeros(1), use_hartree=0, angular="theta")
        tp = TimePropagation([run], precision="fp64")
        tp.step(1)
        got = tp.orbitals(0)
        tp.close()
        want = np.matmul(run.x0, w)
        assert np.linalg.norm(got - want) < TOL * np.linalg.norm(want)


@pytest.mark.parametrize("n_l,n_orb,n_r", [(2, 1, 1), (5, 2, 127), (9, 3, 128), (17, 1, 129), (33, 4, 600)])
def test_observables_noalloc_at_the_edges(n_l, n_orb, n_r):
    """Rows of fewer radii than threads, of one more than a multiple, m from 0 to N_l - 1 and an m
    outside 0 .. N_l - 1, which contributes nothing."""
    import torch
    rng = np.random.default_rng(n_r)
    x = rng.standard_normal((n_l, n_orb, n_r)) + 1j * rng.standard_normal((n_l, n_orb, n_r))
    r = np.sort(rng.uniform(0.1, 50.0, n_r))
    m = np.array(([0, n_l - 1, -1, n_l + 3] * 2)[:n_orb], dtype=np.int32)
    l = np.arange(n_l)[:, None]
    keep = (l >= m[None]) & (m >= 0)[None] & (m < n_l)[None]
    for k in range(n_orb):
        x[~keep[:, k], k] = 0.0
    mf = np.clip(m, 0, n_l - 1)[None].astype(float)
    c = np.sqrt(np.where(l >= mf, ((l + 1.0) ** 2 - mf ** 2) / ((2 * l + 1.0) * (2 * l + 3.0)), 0.0))[..., None]
    z = np.zeros_like(x)
    z[:-1] += c[:-1] * x[1:]
    z[1:] += c[:-1] * x[:-1]
    p = x.conj() * z
    dev = torch.device("cuda", 0)
    xd, rd, md = torch.from_numpy(x).to(dev), torch.from_numpy(r).to(dev), torch.from_numpy(m).to(dev)
    dip = torch.full((n_l, n_orb), float("nan"), dtype=torch.complex128, device=dev)
    acc, norm = torch.full_like(dip, float("nan")), torch.full((n_orb,), float("nan"), dtype=torch.float64, device=dev)
    rc = load_library().ggb_observables_noalloc(xd.data_ptr(), rd.data_ptr(), md.data_ptr(), n_l, n_orb, n_r, dip.data_ptr(),
                                                acc.data_ptr(), norm.data_ptr(), ctypes.c_void_p(None))
    assert rc == 0
    torch.cuda.synchronize()
    for got, q in ((dip, r), (acc, r ** -2.0)):
        scale = (np.abs(x) * np.abs(z) * q).sum(-1).max() + 1e-300
        assert np.abs(got.cpu().numpy() - (p * q).sum(-1)).max() <= TOL * scale
    assert np.allclose(norm.cpu().numpy(), (np.abs(x) ** 2).sum(axis=(0, 2)), rtol=TOL, atol=0)


@pytest.mark.parametrize("n_l,n_orb,n_r", [(7, 3, 3), (3, 2, 31), (129, 1, 32), (31, 7, 33)])
def test_observables_noalloc_rows_that_do_not_fill_a_block(n_l, n_orb, n_r):
    """Several short rows a block, the last block part full."""
    test_observables_noalloc_at_the_edges(n_l, n_orb, n_r)


@pytest.mark.parametrize("n_r,n_l,n_har", [(9, 8, 5), (13, 9, 17), (37, 33, 65), (45, 40, 33), (66, 36, 71)])
def test_fp64_multipole_kernels_at_their_edges(n_r, n_l, n_har):
    """The theta form's exact multipoles at radii that do not fill a block's four, nodes and multipoles
    around the table chunk (32 rows) and the eight partial sums, against the oracle."""
    from oracle.step_oracle import propagate
    from tests.helpers import rel_err, to_oracle
    run = P.reference_like(n_r, n_l, 6, "Ne3", r_mask=15.0, dt_as=10.0, perturb=0.05, seed=3)
    run = dataclasses.replace(run, angular="theta", n_har=n_har)
    ref = propagate(to_oracle(run))
    tp = TimePropagation([run], precision="fp64")
    tp.step(6)
    x, pot, got = tp.orbitals(0), tp.potentials(0), tp.observables(0)
    st, msg = tp.status()
    tp.close()
    assert st == 0, msg
    assert rel_err(x, ref["x"]) < 1e-10          # the FP64 form's bar against the oracle
    assert rel_err(pot["v"], ref["v"][:4]) < 1e-10
    assert rel_err(got["norm"], ref["norm"]) < 1e-10


@pytest.mark.parametrize("n_har", [4, 17])
def test_steps_in_one_call_equal_single_steps(n_har):
    """Calls on both sides of the long graph's length, with and without the forked potentials: the same
    kernels on the same data, so the same bits as one step at a time."""
    run = P.reference_like(37, 9, 64, "Ne3", r_mask=15.0, dt_as=10.0, perturb=0.05, seed=3)
    run = dataclasses.replace(run, angular="theta", n_har=n_har)
    one, many = (TimePropagation([run], precision="fp64", per_l=True) for _ in range(2))
    done = 0
    for n in (0, 1, 7, 8, 9, 33):
        many.step(n)
        for _ in range(n):
            one.step(1)
        done += n
        assert np.array_equal(many.orbitals(0), one.orbitals(0)), done
    for a, b in zip(many.observables(0), one.observables(0)):
        assert np.array_equal(np.asarray(a), np.asarray(b))
    one.close()
    many.close()


@pytest.mark.parametrize("n_r,n_l,angular", [(7, 5, "reference"), (41, 8, "reference"), (33, 9, "theta"), (50, 65, "reference"),
                                             (130, 129, "theta"), (21, 193, "theta")])
def test_fp64_angular_tiles_at_their_edges(n_r, n_l, angular):
    """Channel tiles of 8 and row groups of 64 (N_l 5 .. 193), radii that do not fill a tile, m = 0 and 1,
    every coupling or the theta phase: one step against the oracle."""
    from oracle.step_oracle import propagate
    from tests.helpers import rel_err, to_oracle
    run = P.reference_like(n_r, n_l, 3, "Ne3", r_mask=12.0, dt_as=10.0, perturb=0.05, seed=4)
    run = dataclasses.replace(run, angular=angular)
    for copies in (1, 30):                       # few tiles and many: another number of radii per tile
        ref = propagate(to_oracle(run))
        runs = [run.with_field(run.E) for _ in range(copies)]
        tp = TimePropagation(runs, precision="fp64", groups=[list(range(copies))])
        tp.step(3)
        x, pot = tp.orbitals(copies - 1), tp.potentials(copies - 1)
        st, msg = tp.status()
        tp.close()
        assert st == 0, msg
        assert rel_err(x, ref["x"]) < 1e-10
        assert rel_err(pot["v"], ref["v"][:4]) < 1e-10


@pytest.mark.parametrize("n_r,n_l,angular", [(90, 17, "reference"), (90, 24, "theta"), (50, 31, "reference"), (51, 88, "theta"),
                                             (49, 89, "reference"), (50, 104, "reference")])
def test_fp64_angular_tiles_of_many_columns(n_r, n_l, angular):
    """Sizes at which 90 columns take the four-warp blocks of 16 radii (one column the larger ones): odd
    numbers of 8-channel tiles, part-full radii, two, three and four blocks an SM."""
    test_fp64_angular_tiles_at_their_edges(n_r, n_l, angular)
