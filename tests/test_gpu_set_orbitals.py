"""ggb_set_orbitals sends again only what changed (by value): restarts with other quantum numbers,
occupations or frozen densities, from host and from device memory, equal a fresh context's."""
import ctypes
import dataclasses

import numpy as np
import pytest

from ggbtddft_b200 import problems as P
from ggbtddft_b200.engine import TimePropagation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split_int8"])
def test_restarts_equal_a_fresh_context(precision):
    import torch
    base = P.reference_like(40, 12, 6, "Ne3", r_mask=12.0, dt_as=10.0, perturb=0.05, seed=1)
    base = dataclasses.replace(base, angular="theta")
    rho = 0.01 * np.exp(-base.grid.r)
    x1 = base.x0[:, [1, 0, 2]].copy()
    variants = [base, dataclasses.replace(base, occ=np.array([2, 1, 3], np.int32)),
                dataclasses.replace(base, rho_frozen=rho), dataclasses.replace(base, x0=x1, l_active=base.l_active[[1, 0, 2]]),
                dataclasses.replace(base, m_active=np.array([0, 1, 1], np.int32), x0=_from_m(base.x0, 1)), base]
    tp = TimePropagation([base], precision=precision)
    for n, v in enumerate(variants):
        args = [v.x0, v.l_active, v.m_active, v.occ, v.rho_frozen]
        if n % 2:                      # every other restart from device memory
            args = [torch.from_numpy(np.ascontiguousarray(a).view(np.float64) if a.dtype == np.complex128 else
                                     np.ascontiguousarray(a)).cuda() for a in args]
            ptr = [ctypes.c_void_p(a.data_ptr()) for a in args]
        else:
            args = [np.ascontiguousarray(a) for a in args]
            ptr = [ctypes.c_void_p(a.ctypes.data) for a in args]
        assert tp.lib.ggb_set_orbitals(tp.ctx, 0, *ptr) == 0
        assert np.array_equal(tp.potentials(0)["vexc"], np.zeros(40))
        tp.step(6)
        fresh = TimePropagation([dataclasses.replace(v, V=base.V, D=base.D)], precision=precision)
        fresh.step(6)
        assert np.array_equal(tp.orbitals(0), fresh.orbitals(0)), n
        assert np.array_equal(tp.potentials(0)["vexc"], fresh.potentials(0)["vexc"]), n
        assert np.array_equal(tp.observables(0)["dipole"], fresh.observables(0)["dipole"]), n
        fresh.close()
    tp.close()


def _blocking_stream():
    """A stream that the legacy stream waits for (torch's own side streams are not)."""
    import torch
    handle = ctypes.c_ulonglong(0)
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    return torch.cuda.ExternalStream(handle.value)


@pytest.mark.parametrize("blocking", [False, True])
def test_pinned_arrays_are_read_after_the_copies_that_fill_them(blocking):
    """Asynchronous copies into pinned arrays, queued before the call behind some milliseconds of work on
    the legacy stream or a blocking one: the call sees what they bring, as the copies it makes on the
    legacy stream do."""
    import torch
    base = P.reference_like(40, 12, 4, "Ne3", r_mask=12.0, dt_as=10.0, perturb=0.05, seed=1)
    base = dataclasses.replace(base, angular="theta")
    new = dataclasses.replace(base, occ=np.array([2, 1, 3], np.int32), rho_frozen=0.01 * np.exp(-base.grid.r),
                              m_active=np.array([0, 1, 1], np.int32), x0=_from_m(base.x0, 1))
    def arrays(r):
        return [torch.from_numpy(np.ascontiguousarray(a).view(np.float64) if a.dtype == np.complex128 else
                                 np.ascontiguousarray(a)) for a in (r.x0, r.l_active, r.m_active, r.occ, r.rho_frozen)]
    pinned, source = [a.pin_memory() for a in arrays(base)], [a.cuda() for a in arrays(new)]
    a = torch.rand((2048, 2048), dtype=torch.float64, device="cuda")
    b = a @ a
    tp = TimePropagation([base], precision="fp64")
    tp.step(4)
    torch.cuda.synchronize()
    with torch.cuda.stream(_blocking_stream() if blocking else torch.cuda.default_stream()):
        for _ in range(40):
            torch.matmul(a, a, out=b)
        for p, s in zip(pinned, source):
            p.copy_(s, non_blocking=True)
    assert tp.lib.ggb_set_orbitals(tp.ctx, 0, *(ctypes.c_void_p(p.data_ptr()) for p in pinned)) == 0
    tp.step(4)
    fresh = TimePropagation([new], precision="fp64")
    fresh.step(4)
    assert np.array_equal(tp.orbitals(0), fresh.orbitals(0))
    assert np.array_equal(tp.potentials(0)["vexc0"], fresh.potentials(0)["vexc0"])
    assert np.array_equal(tp.observables(0)["dipole"], fresh.observables(0)["dipole"])
    fresh.close()
    tp.close()


def _from_m(x0, m):
    """Orbital 1 without components below l = m, renormalised."""
    x = x0.copy()
    x[:m, 1] = 0.0
    return x
