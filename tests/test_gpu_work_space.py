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


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_sorted_deposit_without_room_for_its_entries(hv, prec):
    """The deterministic mode asked for on a full device: the deposit goes
    without its entries and gives the same bits, as do a fused step's fields."""
    import torch
    from hv_b200 import _lib as L
    dtype, precision = (np.float64, hv.HV_F64) if prec == "f64" else (np.float32, hv.HV_F32)
    path = hv.HV_PATH_PLAIN if prec == "f64" else hv.HV_PATH_FUSED
    w = replace(hv.PB208_104K, ppn=20000, n=64)  # 4.16 M particles: 67 or 133 MB of entries
    p = hv.workload_particles(w, dtype)
    atomic = w.run_params()
    ordered = replace(w, deposit_mode=hv.HV_DEPOSIT_SORTED).run_params()
    with hv.Session(w.world(), w.protons, w.neutrons, atomic, precision) as s:
        s.upload_particles(*p)
        s.deposit()
        full, size = [], 2 ** 36
        while size >= 2 ** 22:
            if _free() > size + 2 ** 25:
                full.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            else:
                size //= 2
        assert _free() < 60e6
        try:
            L.check(s.lib.hv_ctx_set_params(s.handle, L.C.byref(ordered)), "hv_ctx_set_params")
            s.deposit()
            without = s.download_field(hv.HV_FIELD_DENSITY_RAW)
        finally:
            del full
            torch.cuda.empty_cache()
        s.run(2, path)
        again = [s.download_field(hv.HV_FIELD_DENSITY_RAW), s.download_field(hv.HV_FIELD_FORCE_Z)]
    with hv.Session(w.world(), w.protons, w.neutrons, ordered, precision) as s:
        s.upload_particles(*p)
        s.deposit()
        assert np.array_equal(without, s.download_field(hv.HV_FIELD_DENSITY_RAW))
        s.run(2, path)
        kept = [s.download_field(hv.HV_FIELD_DENSITY_RAW), s.download_field(hv.HV_FIELD_FORCE_Z)]
    assert all(np.array_equal(a, b) for a, b in zip(again, kept))


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_pair_sums_give_their_work_space_back_to_a_run(hv, prec):
    """The pair sums keep 28 to 56 bytes a particle (12 or 23 MB here) for the
    next call, but not when the context plans a run: it then holds as much
    memory as one that never made them, and they can be made again."""
    dtype, precision = (np.float64, hv.HV_F64) if prec == "f64" else (np.float32, hv.HV_F32)
    used = {}
    for ppn in (10, 2000):  # a small context first loads the kernels
        w = replace(hv.PB208_104K, ppn=ppn)
        p = hv.workload_particles(w, dtype)
        for sums in (False, True):
            with hv.Session.from_workload(w, precision) as s:
                s.set_fast_options(graph_steps=0)
                s.upload_particles(*p)
                before = _free()
                first = s.particle_densities() if sums else None
                s.run(1, hv.HV_PATH_FUSED)
                used[sums] = before - _free()
                if sums:
                    s.upload_particles(*p)
                    again = s.particle_densities()
                    for a, b in zip(first, again):
                        assert np.abs(a - b).max() <= (1e-5 if prec == "f32" else 1e-12) * np.abs(a).max()
    assert abs(used[True] - used[False]) < 2 ** 21, used
