"""GPU: the sweeps of the fused Coulomb solve, where the direct form does not
run: coarse-corrected cycles on planes past its shared memory, plain cycles,
and batches of both.

Which solver ran shows in the iterations: a correction of the direct form
counts as one, a coarse-corrected cycle as sor_coarse_sweeps, and a plain
cycle as sor_inner_min at least."""
from dataclasses import replace

import numpy as np
import pytest
from conftest import max_rel

pytestmark = pytest.mark.gpu

# y-z planes past the direct form's; every axis divides by the coarse factor
# 16, and a block's tile fits the staged sweeps (two forms)
BOXES = [((32, 128, 256), (8.0, 16.0, 32.0)), ((32, 256, 128), (8.0, 32.0, 16.0))]
# a tile that does not: the generic sweep's plain cycles
LARGE = (32, 256, 256), (8.0, 32.0, 32.0)


def _world(n, d_max):
    from hv_b200 import _lib as L
    world = L.hv_world()
    for a in range(3):
        world.n[a], world.d_max[a] = n[a], d_max[a]
    return world


def _run(hv, w, box, steps, **opts):
    with hv.Session(_world(*box), w.protons, w.neutrons, w.run_params(), hv.HV_F32) as s:
        s.set_fast_options(**opts)
        s.upload_particles(*hv.workload_particles(w, np.float32))
        s.run(0, hv.HV_PATH_FUSED)
        obs = s.run(steps, hv.HV_PATH_FUSED)
        return obs, s.download_field(hv.HV_FIELD_DENSITY), s.download_field(hv.HV_FIELD_COULOMB)


@pytest.mark.parametrize("box", BOXES)
def test_coarse_corrected_cycles_on_large_planes(hv, box):
    """Three settings of the sweeps end at the same FP64 rule: D(t) and the
    potential within the solves' tolerance of each other, and the potential
    within it of the exact solution of its density.  Corrected cycles take
    fewer iterations than plain ones; on these flat boxes, whose coarse grid
    has one node along x, those of 16 sweeps at the run's omega fewest."""
    w = replace(hv.CA40_SMALL, dt=0.25)
    res = [_run(hv, w, box, 10, **o) for o in ({}, dict(sor_coarse_sweeps=16, sor_coarse_omega=w.sor_omega),
                                               dict(sor_coarse=0))]
    for obs, *_ in res:
        assert not np.any(obs["flags"] & 1)
    its = [obs["sor_iterations"] for obs, *_ in res]
    assert np.all(its[0] >= 12) and np.all(its[0] % 12 == 0), its[0]
    assert np.all(its[1] >= 16) and np.all(its[1] % 16 == 0), its[1]
    assert its[0][2:].sum() < its[2][2:].sum() and its[1][2:].sum() < its[2][2:].sum(), its
    for obs, _, phi in res[1:]:
        assert max_rel(obs["dipole"], res[0][0]["dipole"]) < 1e-6
        assert max_rel(phi, res[0][2]) < 1e-6
    _within_the_rule(w, box, res[0])


def _within_the_rule(w, box, run):
    """|r|_2 <= 1e-6 |b|_2: phi within that over the smallest eigenvalue of
    -lap of the exact solution of its density, and a rounding to float."""
    import test_gpu_poisson as poisson
    n, d_max = box
    _, rho, phi = run
    rho = rho.reshape(2, *n)[0].astype(np.float64)
    old = poisson.HALF_BOX
    try:
        poisson.HALF_BOX = d_max
        ref = poisson.exact_phi(n, w.Z, rho)
    finally:
        poisson.HALF_BOX = old
    lam = sum((2.0 - 2.0 * np.cos(np.pi / (m - 1))) * (m / (2.0 * d)) ** 2 for m, d in zip(n, d_max))
    b = 4.0 * np.pi * 1.44 * np.linalg.norm(rho[1:-1, 1:-1, 1:-1])
    assert np.abs(phi.reshape(n) - ref).max() <= 1e-6 * b / lam + 1.2e-7 * np.abs(ref).max()


def test_plain_cycles_on_larger_planes(hv):
    w = replace(hv.CA40_SMALL, dt=0.25)
    run = _run(hv, w, LARGE, 3)
    assert not np.any(run[0]["flags"] & 1) and np.all(run[0]["sor_iterations"] >= 8)
    _within_the_rule(w, LARGE, run)


@pytest.mark.parametrize("n,direct", [((6, 194, 194), True), ((6, 195, 195), False), ((6, 194, 196), False),
                                      ((4, 200, 16), True)])
def test_edge_of_the_direct_form(hv, n, direct):
    """Planes of 194 x 194 nodes are the largest square ones whose transforms
    fit in a block's shared memory; the next ones take plain cycles."""
    w = replace(hv.CA40_SMALL, dt=0.25)
    obs, _, _ = _run(hv, w, (n, (10.0, 10.0, 10.0)), 3)
    assert not np.any(obs["flags"] & 1)
    if direct:
        assert np.all(obs["sor_iterations"] <= 3), obs["sor_iterations"]
    else:
        assert np.all(obs["sor_iterations"] >= 8), obs["sor_iterations"]


def _workloads(hv):
    from hv_b200.workloads import batch_workloads
    return [replace(w, ppn=min(w.ppn, 100)) for w in batch_workloads(5, seed=7)]


@pytest.mark.parametrize("cap", [0, 8])
@pytest.mark.parametrize("coarse", [(0, 0, 0, 0, 0), (1, 0, 1, 0, 1)])
def test_batched_sweeps_match_the_instances_own_runs(hv, cap, coarse):
    """Waves of plain cycles, and batches in which some instances sweep and
    some solve directly."""
    from hv_b200.batch import Batch
    ws, steps = _workloads(hv), 12
    alone, sessions = [], []
    for w, c in zip(ws, coarse):
        for keep in (False, True):
            s = hv.Session.from_workload(w, hv.HV_F32)
            s.set_fast_options(sor_coarse=c)
            s.upload_particles(*hv.workload_particles(w, np.float32))
            if keep:
                sessions.append(s)
            else:
                with s:
                    alone.append(s.run(steps, hv.HV_PATH_FUSED))
    try:
        with Batch(sessions) as b:
            b.plan(cap)
            obs = np.concatenate([b.run(5), b.run(steps - 5)], axis=1)
    finally:
        for s in sessions:
            s.close()
    for c, o, a in zip(coarse, obs, alone):
        assert not np.any(o["flags"] & 1) and np.allclose(o["t"], a["t"])
        assert np.abs(o["dipole"] - a["dipole"]).max() <= 1e-4 * np.abs(a["dipole"]).max()
        assert np.all(o["sor_iterations"] <= 3) if c else np.all(o["sor_iterations"][2:] >= 8), (c, o["sor_iterations"])


@pytest.mark.parametrize("box", BOXES)
def test_batched_coarse_cycles(hv, box):
    """A coarse-corrected instance (large planes) beside a direct one."""
    from hv_b200.batch import Batch
    w = replace(hv.CA40_SMALL, dt=0.25)
    p = hv.workload_particles(w, np.float32)
    alone, _, _ = _run(hv, w, box, 8)
    sessions = [hv.Session(_world(*box), w.protons, w.neutrons, w.run_params(), hv.HV_F32),
                hv.Session.from_workload(w, hv.HV_F32)]
    try:
        for s in sessions:
            s.upload_particles(*p)
        with Batch(sessions) as b:
            obs = b.run(8)
    finally:
        for s in sessions:
            s.close()
    assert not np.any(obs["flags"] & 1)
    assert np.all(obs[0]["sor_iterations"] % 12 == 0) and np.all(obs[0]["sor_iterations"] >= 12), obs[0]["sor_iterations"]
    assert np.all(obs[1]["sor_iterations"] <= 3)
    assert np.abs(obs[0]["dipole"] - alone["dipole"]).max() <= 1e-4 * np.abs(alone["dipole"]).max()
