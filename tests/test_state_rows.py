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
