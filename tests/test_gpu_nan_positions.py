"""GPU: particles without a finite position lie in no cell.

A run that blows up leaves NaN or infinite positions behind.  Every kernel
that turns a position into a cell has to treat them as it treats a particle
far outside the grid: nothing deposited, no force, and no effect on the other
particles."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOST = {0: np.nan, 1: np.inf, 2: -np.inf}  # particle -> its position


def _particles(hv, w, dtype, lost):
    """The workload's particles with some (protons and neutrons) lost: to the
    values above, or to a finite place far outside the grid."""
    p = [a.copy() for a in hv.workload_particles(w, dtype)]
    for i, v in LOST.items():
        for at in (5 * i + 3, w.protons + 7 * i + 1):
            for axis in range(3):
                # one axis lost is enough; the three kinds take different ones
                if axis == i or i == 0:
                    p[axis][at] = v if lost else 1e6
    return p


@pytest.mark.parametrize("path", ["plain", "fused"])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", ["sorted", "atomic"])
def test_lost_particles_act_as_particles_far_outside(hv, path, prec, mode):
    """The sorted deposit repeats bit for bit, so the fields of both runs are
    the same bits; the atomic one's order moves them by rounding only."""
    w = replace(hv.CA40_SMALL, ppn=40, deposit_mode=hv.HV_DEPOSIT_SORTED if mode == "sorted" else hv.HV_DEPOSIT_ATOMIC)
    dtype, precision = (np.float32, hv.HV_F32) if prec == "f32" else (np.float64, hv.HV_F64)
    fields = []
    for lost in (True, False):
        with hv.Session.from_workload(w, precision) as s:
            s.set_fast_options(sort_every=2)
            s.upload_particles(*_particles(hv, w, dtype, lost))
            if path == "plain":
                s.initial_solve()
            s.run(4, hv.HV_PATH_PLAIN if path == "plain" else hv.HV_PATH_FUSED)
            fields.append([s.download_field(f) for f in (hv.HV_FIELD_DENSITY_RAW, hv.HV_FIELD_COULOMB, hv.HV_FIELD_FORCE_X)])
    for a, b in zip(*fields):
        assert np.all(np.isfinite(a))
        if mode == "sorted":
            assert np.array_equal(a, b)
        else:
            assert np.abs(a - b).max() <= (1e-4 if prec == "f32" else 1e-9) * np.abs(b).max()


@pytest.mark.parametrize("path", ["plain", "fused"])
def test_lost_particles_leave_the_gradient(hv, path):
    """A particle lost along x keeps its z, so D(t) and the gradient are those
    of the run with it far outside."""
    from hv_b200.adjoint import AdjointRun
    w = replace(hv.CA40_SMALL, ppn=40, deposit_mode=hv.HV_DEPOSIT_SORTED)
    grads = []
    for value in (np.nan, 1e6):
        p = [a.copy() for a in hv.workload_particles(w, np.float64)]
        p[0][[3, w.protons + 1]] = value
        run = AdjointRun(w, p, 4, 2, path=hv.HV_PATH_PLAIN if path == "plain" else hv.HV_PATH_FUSED)
        try:
            run.forward((w.t0, w.t3, w.sigma, w.a_sym))
            grads.append(run.backward(np.arange(1.0, 5.0)))
        finally:
            run.close()
    assert np.all(np.isfinite(grads[0]))
    assert np.abs(grads[0] - grads[1]).max() <= 1e-6 * np.abs(grads[1]).max()
