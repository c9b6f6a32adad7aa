"""GPU: a batch whose contexts changed after it was planned: other particles,
other parameters, other options.  Its waves hold the contexts' buffers and
options, so it plans anew; its runs are those of a batch created after the
change."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(hv, **kw):
    return replace(hv.CA40_SMALL, ppn=40, dt=0.25, deposit_mode=hv.HV_DEPOSIT_SORTED, **kw)


def _sessions(hv, ws, seeds, options=({}, {})):
    out = []
    for w, seed, o in zip(ws, seeds, options):
        s = hv.Session.from_workload(w, hv.HV_F32)
        s.set_fast_options(**o)
        s.upload_particles(*hv.workload_particles(replace(w, seed=seed), np.float32))
        out.append(s)
    return out


def _run(hv, sessions, steps, change=None, before=0):
    from hv_b200.batch import Batch
    try:
        with Batch(sessions) as b:
            if before:
                b.run(before)
            if change:
                change(sessions)
            obs = b.run(steps)
            return obs, [s.download_field(hv.HV_FIELD_COULOMB) for s in sessions]
    finally:
        for s in sessions:
            s.close()


def _same(a, b, tol):
    for x, y in zip(a[0], b[0]):
        assert np.abs(x["dipole"] - y["dipole"]).max() <= tol * np.abs(y["dipole"]).max()
    for x, y in zip(a[1], b[1]):
        assert np.abs(x - y).max() <= tol * np.abs(y).max()


def test_particles_uploaded_after_the_plan(hv):
    """Their fields are solved before the first step: solves at 1e-6 from
    different starts, in float."""
    ws = [_workload(hv), _workload(hv, n=40, h=0.8)]

    def change(ss):
        for s, w, seed in zip(ss, ws, (3, 4)):
            s.upload_particles(*hv.workload_particles(replace(w, seed=seed), np.float32))

    _same(_run(hv, _sessions(hv, ws, (1, 2)), 12, change), _run(hv, _sessions(hv, ws, (3, 4)), 12), 1e-5)


def test_parameters_changed_after_the_plan(hv):
    """A change of parameters releases the buffers that the waves held."""
    ws = [_workload(hv), _workload(hv, n=40, h=0.8)]
    new = [replace(w, t0=w.t0 * 0.98, sigma_r=0.7) for w in ws]

    def change(ss):
        for s, w, seed in zip(ss, new, (1, 2)):
            s.set_params(w.run_params())
            s.upload_particles(*hv.workload_particles(replace(w, seed=seed), np.float32))

    _same(_run(hv, _sessions(hv, ws, (1, 2)), 12, change), _run(hv, _sessions(hv, new, (1, 2)), 12), 1e-5)


def test_options_changed_after_the_plan(hv):
    """One instance goes from the direct solve to sweeps and back; the other
    runs on its own between two batched runs."""
    from hv_b200.batch import Batch
    ws = [_workload(hv), _workload(hv, n=40, h=0.8)]
    ss = _sessions(hv, ws, (1, 2))
    try:
        with Batch(ss) as b:
            runs = [b.run(9)]
            ss[0].set_fast_options(sor_coarse=0)
            runs.append(b.run(9))
            ss[0].set_fast_options(sor_coarse=1)
            ss[1].autotune(1)
            runs.append(b.run(9))
    finally:
        for s in ss:
            s.close()
    its = [[r[i]["sor_iterations"] for r in runs] for i in (0, 1)]
    assert np.all(its[0][0] <= 3) and np.all(its[0][1] >= 8) and np.all(its[0][2] <= 3), its[0]
    assert all(np.all(x <= 3) for x in its[1]), its[1]
    for r in runs:
        assert not np.any(r["flags"] & 1) and np.all(np.isfinite(r["dipole"]))
    # the first instance's D(t) goes on through the three runs
    t = np.concatenate([r[0]["t"] for r in runs])
    assert np.allclose(t, np.arange(27) * ws[0].dt, rtol=1e-6)
    with _sessions(hv, ws[:1], (1,))[0] as s:
        alone = s.run(27, hv.HV_PATH_FUSED)["dipole"]
    d = np.concatenate([r[0]["dipole"] for r in runs])
    assert np.abs(d - alone).max() <= 1e-4 * np.abs(alone).max()
