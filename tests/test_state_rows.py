"""Padded node-state rows (metadata only, no GPU): rows hold whole walk vectors, and a budget that
the padding would overrun is planned as if there were none."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import artifact_path
from grg_spmv_b200 import RuntimeRequirements, scan_grg_spmv
from grg_spmv_b200.backends.b200.plan import B200PlanPair, plan_layout_from_scans, state_ld


@pytest.mark.parametrize("itemsize,expected", [(8, {1: 1, 2: 2, 3: 4, 4: 4, 5: 8, 8: 8, 33: 36, 64: 64}),
                                               (4, {1: 1, 2: 2, 3: 4, 4: 4, 5: 8, 8: 8, 9: 16, 33: 40})])
def test_rows_hold_whole_vectors(itemsize, expected):
    assert {k: state_ld(k, itemsize) for k in expected} == expected


def _plan(budget):
    req = RuntimeRequirements(5, 5, True, False, False, False, False)
    path = artifact_path("synth_haploid")
    return plan_layout_from_scans(scans=(scan_grg_spmv(path),), paths=(path,), dtype=np.float64, requirements=req, requested_budget=budget,
                                  requested_ring=1, allow_residency=True, device_id=0, stream_ptr=0, stream_owner=None, pair=B200PlanPair())


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
def test_tight_budgets_plan_without_padding():
    full = _plan(0)
    nodes = full.max_num_nodes
    padding = nodes * 3 * 8
    assert full.state_ld == 8 and full.bytes_by_category["state"] == nodes * 8 * 8
    assert _plan(full.bytes_total).state_ld == 8
    tight = _plan(full.bytes_total - 1)  # overrun only by padding: every level stays resident
    assert tight.state_ld == 5 and tight.bytes_total == full.bytes_total - padding
    assert all(lp.resident for lp in tight.level_plans())
    assert _plan(full.bytes_total - padding).bytes_total == full.bytes_total - padding


def test_quad_rows_locate_narrow_lists():
    """``quad_rows`` of default-order padded lists gives every narrow list's extent by arithmetic; it
    is zero where the order or a longer list rules that out."""
    from grg_spmv_b200.backends.b200 import _native as nat
    from grg_spmv_b200.backends.b200.structures import _finish

    rng = np.random.default_rng(4)
    lengths = np.concatenate((rng.integers(0, 33, 500), [40, 33, 0, 32, 29, 28]))
    rows = np.repeat(np.arange(lengths.size), lengths)
    ids, z = rng.integers(0, 1000, rows.size), np.zeros(rows.size, dtype=np.int64)
    level = _finish(0, 0, lengths.size, rows, ids, z, z, 32, pad=True)
    narrow = lengths.size - 2
    more = np.asarray(level.quad_rows())
    assert more.size == nat.QUAD_CLASSES and more[0] == (lengths > 0).sum() - 2 and more[7] == ((lengths > 28) & (lengths < 33)).sum()
    pos = np.arange(narrow)[:, None]
    start = np.minimum(pos, more[None, :]).sum(1)
    np.testing.assert_array_equal(4 * start, level.row_ptr[:narrow])
    np.testing.assert_array_equal(4 * (start + (pos < more[None, :]).sum(1)), level.row_ptr[1:narrow + 1])
    for other in (dict(pad=False), dict(pad=True, quad_order=False), dict(pad=True, long_first=False)):
        assert _finish(0, 0, lengths.size, rows, ids, z, z, 32, **other).quad_rows() == [0] * nat.QUAD_CLASSES
    assert _finish(0, 0, lengths.size, rows, ids, z, z, 36, pad=True).quad_rows() == [0] * nat.QUAD_CLASSES  # 33 entries: 9 quads
