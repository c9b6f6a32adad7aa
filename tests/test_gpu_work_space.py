"""GPU: what the solvers and the deposit need beyond a context's own buffers.

A context that fits in memory has to run: work space that a later call adds is
either found among the buffers that exist or done without."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_plain_solve_takes_no_memory(hv, prec):
    """The solve's saved values are a field's worth of words (17 MB here in
    double): they lie in a buffer that the context has anyway.  A small context
    comes first, so that the kernels are loaded."""
    dtype, precision = (np.float64, hv.HV_F64) if prec == "f64" else (np.float32, hv.HV_F32)
    for n in (32, 64, 128):
        w = replace(hv.CA40_SMALL, n=n, h=32.0 / n, sor_tol=1e-2)
        with hv.Session.from_workload(w, precision) as s:
            s.upload_particles(*hv.workload_particles(w, dtype))
            s.deposit()
            s.smooth()
            s.coulomb_boundary()
            before = _free()
            s.coulomb_sor()
            used = before - _free()
    assert used < 2 ** 21, used


def test_plain_solve_between_sorted_deposits(hv):
    """The shared buffer is written anew by every deposit: raw densities before
    and after a solve are the same bits."""
    w = replace(hv.CA40_SMALL, deposit_mode=hv.HV_DEPOSIT_SORTED)
    with hv.Session.from_workload(w, hv.HV_F64) as s:
        s.upload_particles(*hv.workload_particles(w, np.float64))
        raw = []
        for _ in range(2):
            s.deposit()
            raw.append(s.download_field(hv.HV_FIELD_DENSITY_RAW))
            s.smooth()
            s.coulomb_boundary()
            s.coulomb_sor()
    assert np.array_equal(*raw) and raw[0].sum() > 0.0


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_slot_re_sort_takes_no_memory(hv, prec):
    """A re-sort moves six arrays and the permutation (12 or 22 MB here)
    through buffers that are free between steps, and keeps every particle."""
    dtype, precision = (np.float64, hv.HV_F64) if prec == "f64" else (np.float32, hv.HV_F32)
    for ppn in (10, 2000):
        w = replace(hv.PB208_104K, ppn=ppn, deposit_mode=hv.HV_DEPOSIT_SORTED)
        p = hv.workload_particles(w, dtype)
        out = []
        for every in (0, 1):
            with hv.Session.from_workload(w, precision) as s:
                s.set_fast_options(sort_every=0, graph_steps=0)
                s.upload_particles(*p)
                s.run(1, hv.HV_PATH_FUSED)
                s.set_fast_options(sort_every=every)
                before = _free()
                s.run(1, hv.HV_PATH_FUSED)
                used = before - _free()
                out.append(s.download_particles() + [s.download_array(f) for f in ("fx", "fy", "fz")])
        # the re-sorted run steps the same particles (the sorted deposit sums a
        # node's particles in another slot order: rounding)
        for a, b in zip(*out):
            assert np.abs(a - b).max() <= (1e-4 if prec == "f32" else 1e-11) * max(1.0, np.abs(a).max())
    assert used < 2 ** 21, used
