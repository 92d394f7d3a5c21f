"""The four-warps-per-unit BM kernel, which runs tables of few units: bit for
bit the results of the oracle and of the warp-per-unit kernel, at the edges of
its rule (sweep counts against its halo, unit counts against the SMs)."""
import numpy as np
import pytest

from cochlearmodel_gb300 import model, native
from oracle import oracle as orc
from tests import cases

pytestmark = pytest.mark.gpu

HALO = 32  # most sweeps of one solve that the kernel takes; longer ones go to the other


def _case(mv, ms, fast, slow, max_outer, seed):
    cfg, sc, gamma, units, x, rows = cases.framed_batch(mv, [ms, 0.6 * ms, 1.3 * ms], seed=seed,
                                                       block_ms=0.5, overlap_ms=0.2)
    sc = native.BMScalars.from_buffer_copy(sc)
    sc.jacobi_fast, sc.jacobi_slow, sc.max_outer = fast, slow, max_outer
    return cfg, sc, gamma, units, x, rows


@pytest.mark.parametrize("controller", [0, 1])
@pytest.mark.parametrize("fast,slow,max_outer", [(2, 20, 10), (0, 1, 10), (3, 5, 3), (4, 31, 10),
                                                 (2, HALO, 1), (HALO, 20, 2), (2, HALO + 1, 10)])
def test_sweep_counts_against_oracle(mv, bm_solver, controller, fast, slow, max_outer):
    cfg, sc, gamma, units, x, rows = _case(mv, 0.7, fast, slow, max_outer, seed=3)
    sc.controller = controller
    o_v, o_f, o_st = orc.bm_run(mv.section_params(), gamma, sc, units, x, rows)
    v, f, st = bm_solver.run(sc, gamma, units, x, rows)
    assert np.array_equal(v.view(np.uint32), o_v.view(np.uint32))
    assert np.array_equal(f, o_f)
    for k in ("substeps", "iterations", "sweeps", "failed_samples", "written_samples", "status"):
        assert np.array_equal(st[k], o_st[k]), k


@pytest.mark.parametrize("controller,arith", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("extra", [0, 1])
def test_both_sides_of_the_unit_rule(mv, bm_solver, controller, arith, extra):
    """The same units once alone and once in a table just at (extra 0) or just
    past (extra 1: the warp-per-unit kernel) the most units of the rule: one an
    SM for controller 0, two for controller 1."""
    import torch
    sms = torch.cuda.get_device_properties(bm_solver.device).multi_processor_count
    cfg, sc, gamma, units, x, rows = _case(mv, 0.5, 2, 20, 10, seed=5)
    sc.controller, sc.arith = controller, arith
    v, f, st = bm_solver.run(sc, gamma, units, x, rows)
    assert np.abs(v).max() > 0
    n = (2 if controller else 1) * sms + extra
    copies = -(-n // len(units))
    table = np.concatenate([units] * copies)[:n].copy()
    table["out_base"] += np.repeat(np.arange(copies), len(units))[:n] * rows
    vv, ff, ss = bm_solver.run(sc, gamma, table, x, rows * copies)
    whole = n // len(units)
    assert np.array_equal(vv[:whole * rows].view(np.uint32).reshape(whole, rows, 256),
                          np.broadcast_to(v.view(np.uint32), (whole, rows, 256)))
    assert np.array_equal(ff[:whole * rows].reshape(whole, rows), np.broadcast_to(f, (whole, rows)))
    for k in ("substeps", "iterations", "sweeps", "failed_samples"):
        assert np.array_equal(ss[k], np.resize(st[k], n)), k


@pytest.mark.parametrize("controller,arith", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("value", [np.inf, 3e38])
def test_infinite_pressure_at_the_ends(mv, bm_solver, controller, arith, value):
    """An input that drives the pressure out of range: the sections outside a
    unit stay zero in both kernels, so the iterations are the same too."""
    import torch
    sms = torch.cuda.get_device_properties(bm_solver.device).multi_processor_count
    cfg, sc, gamma, units, x, rows = _case(mv, 0.5, 2, 20, 10, seed=7)
    sc.controller, sc.arith = controller, arith
    x = x.copy()
    u = units[0]  # (a sample in the middle of a unit)
    x[u["in_base"] + (u["start"] + u["end"]) // 2] = value
    v, f, st = bm_solver.run(sc, gamma, units, x, rows)
    assert not np.isfinite(v).all()
    copies = -(-(2 * sms + 1) // len(units))
    table = np.concatenate([units] * copies)
    table["out_base"] += np.repeat(np.arange(copies), len(units)) * rows
    vv, ff, ss = bm_solver.run(sc, gamma, table, x, rows * copies)
    assert np.array_equal(vv[:rows], v, equal_nan=True) and np.array_equal(ff[:rows], f)
    for k in ("substeps", "iterations", "sweeps", "failed_samples"):
        assert np.array_equal(ss[k][:len(units)], st[k]), k
