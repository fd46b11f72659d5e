"""The calls that users make, without bounds checks: the row walk in every mode.

The first part runs the suites of the checked kernels again with checks off, as they stand, with their
own inputs and tolerances.  The second part holds what they lack: recorded calls with new inputs, node
states that a tight budget leaves without padding, infinities and NaN, and the mixed words bit by bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from conftest import ATOL_F32, ATOL_F64, RTOL_F32, RTOL_F64, artifact_path  # noqa: E402
from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402
from grg_spmv_b200.backends.b200 import B200Plan, B200PlanPair, B200Runtime, plan_b200_layout  # noqa: E402
from grg_spmv_b200.backends.b200 import _native as nat  # noqa: E402
from test_gpu_adaptor import artifact, test_captured_grg_matches_oracle_exactly_on_integer_inputs  # noqa: E402,F401
from test_gpu_batch import test_batch_autotune_picks_a_tile_and_stays_correct, test_batch_matches_oracle, two_artifacts  # noqa: E402,F401
from test_gpu_mixed import (  # noqa: E402,F401
    synth_artifact, test_mixed_against_oracle, test_mixed_large_integers_stay_exact, test_mixed_prepared_ops_and_graph_replay)
from test_gpu_parity import GROUPS, _run_case, test_golden_mixed_precision  # noqa: E402,F401
from test_gpu_runtime import (  # noqa: E402,F401
    test_float32_runtime, test_foreign_stream_ordering, test_graphs_off_matches_graphs_on, test_hybrid_budget_is_exact,
    test_k_below_max_with_matrix_and_emit_vector, test_lean_mixed_streamed_layout, test_multi_grg_single_graph_mixed_heights,
    test_one_sided_layouts, test_prepared_chain_captures_in_a_cuda_graph, test_programmatic_dependent_launch_is_bit_identical,
    test_repeated_calls_are_deterministic, test_streamed_levels_are_exact)
from test_gpu_xtx import diploid_artifact, test_kinship_cg_solve, test_standardized_xtx_matches_cpu_model  # noqa: E402,F401
from test_mixed_words import decode, encode  # noqa: E402
from test_zz_no_alloc import small_artifact, test_static_state_entry_point_matches_traverse  # noqa: E402,F401


@pytest.fixture(autouse=True)
def unchecked(monkeypatch):
    init = B200Runtime.__init__
    monkeypatch.setattr(B200Runtime, "__init__", lambda self, layout, *, check_bounds=None, use_graphs=None: init(
        self, layout, check_bounds=False, use_graphs=use_graphs))


def _layout(path, k, dtype=np.float64, budget=0, **kw):
    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=True, need_up_miss_output=True, need_init_vector=True,
                              need_init_matrix=True, need_init_xtx=True)
    return plan_b200_layout(artifacts=[str(path)], dtype=dtype, requirements=req, vram_budget_bytes=budget, ring_buffer_size=0,
                            device=0, stream=0, **kw)


@pytest.mark.parametrize("heavy", [128, 2], ids=["narrow", "heavy-rows"])
@pytest.mark.parametrize("group", sorted(GROUPS), ids=[f"{a}-{d}" for a, d in sorted(GROUPS)])
def test_golden_default_plans(group, heavy, golden_data):
    """Golden cases on default plans: exact for integer-valued inputs, else to reassociation."""
    name, dtype = group
    pair = B200PlanPair(plan_up=B200Plan(heavy_threshold=heavy), plan_down=B200Plan(heavy_threshold=heavy))
    rtol, atol = (RTOL_F64, ATOL_F64) if dtype == "float64" else (RTOL_F32, ATOL_F32)
    with B200Runtime(_layout(artifact_path(name), 8, np.dtype(dtype), pair=pair)) as runtime:
        (grg,) = runtime.grgs
        for case in GROUPS[group]:
            out, miss = _run_case(grg, case, golden_data)
            expected = golden_data[case["key"] + "|out"]
            if any(tag in case["case"] for tag in ("pm1", "ones", "zeros")) and case["init"] is None:
                np.testing.assert_array_equal(out, expected, err_msg=case["key"])
                if case["miss"] and case["direction"] == "up":
                    np.testing.assert_array_equal(miss, golden_data[case["key"] + "|miss_out"], err_msg=case["key"])
            else:
                np.testing.assert_allclose(out, expected, rtol=rtol, atol=atol * max(1.0, np.abs(expected).max()), err_msg=case["key"])


@pytest.mark.parametrize("precision,dtype", [("plain", np.float64), ("plain", np.float32), ("mixed", np.float64)])
@pytest.mark.parametrize("k", [1, 2, 3, 8, 33])
def test_recorded_calls_with_new_inputs(synth_artifact, k, precision, dtype):
    """Every recorded op, several times with other inputs each time.  Integers: exact in any order
    (sums below 2^24, the exact range of FP32)."""
    oracle = OracleGRG(synth_artifact)
    rng = np.random.default_rng(80 + k)
    with B200Runtime(_layout(synth_artifact, k, dtype, precision=precision)) as runtime:
        (grg,) = runtime.grgs
        for direction in ("up", "down"):
            for by_individual, use_miss in ((False, False), (True, False), (False, True)):
                op = grg.prepare_matmul_cuda(direction=direction, k=k, by_individual=by_individual, use_miss=use_miss)
                assert op._graph is not None
                for _ in range(3):
                    x = rng.integers(-3, 4, size=tuple(op.input.shape)).astype(np.float64)
                    miss = rng.integers(-3, 4, size=(k, grg.num_mutations)).astype(np.float64) if use_miss else None
                    op.input.copy_(torch.from_numpy(x))
                    if use_miss and direction == "down":
                        op.miss_input.copy_(torch.from_numpy(miss))
                    op()
                    torch.cuda.synchronize()
                    total = None if miss is None else (miss.copy() if direction == "down" else np.zeros_like(miss))
                    expected = oracle.matmul(x, direction, by_individual=by_individual, miss=total)
                    np.testing.assert_array_equal(op.output.cpu().numpy(), expected)
                    if use_miss and direction == "up":
                        np.testing.assert_array_equal(op.miss_output.cpu().numpy(), total)


@pytest.mark.parametrize("dtype,ks", [(np.float64, (3, 5, 7, 9)), (np.float32, (3, 5, 7, 9, 17))])
def test_states_without_padding(synth_artifact, dtype, ks):
    """A budget that padded rows would overrun: rows of k values, whatever vectors they hold."""
    oracle = OracleGRG(synth_artifact)
    rng = np.random.default_rng(4)
    for k in ks:
        layout = _layout(synth_artifact, k, dtype, budget=_layout(synth_artifact, k, dtype).bytes_total - 1)
        assert layout.state_ld == k
        with B200Runtime(layout) as runtime:
            (grg,) = runtime.grgs
            for direction, cols in (("up", grg.num_samples), ("down", grg.num_mutations)):
                x = rng.integers(-3, 4, size=(k, cols))
                miss = rng.integers(-3, 4, size=(k, grg.num_mutations))
                for kw in ({}, {"by_individual": True}, {"emit_all_nodes": True}, {"miss": miss}):
                    y = x[:, :grg.num_individuals] if direction == "up" and kw.get("by_individual") else x
                    got = grg.matmul(y.astype(dtype), direction, **{n: v.astype(dtype) if n == "miss" else v for n, v in kw.items()})
                    ref = oracle.matmul(y.astype(np.float64), direction, **{n: v.astype(np.float64) if n == "miss" else v for n, v in kw.items()})
                    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("precision,dtype", [("plain", np.float64), ("plain", np.float32), ("mixed", np.float64)])
@pytest.mark.parametrize("k", [1, 4, 8])
def test_infinities_and_nan(synth_artifact, k, precision, dtype):
    """Infinite and NaN inputs reach exactly the outputs that depend on them, the others stay exact."""
    oracle = OracleGRG(synth_artifact)
    rng = np.random.default_rng(6)
    with B200Runtime(_layout(synth_artifact, k, dtype, precision=precision)) as runtime:
        (grg,) = runtime.grgs
        for direction, cols in (("up", grg.num_samples), ("down", grg.num_mutations)):
            for values in ((np.inf,), (-np.inf,), (np.nan,), (np.inf, -np.inf, np.nan)):
                x = rng.integers(-3, 4, size=(k, cols)).astype(np.float64)
                for v in values:
                    x[rng.integers(0, k, 3), rng.integers(0, cols, 3)] = v
                for kw in ({}, {"emit_all_nodes": True}):
                    with np.errstate(invalid="ignore"):
                        ref = oracle.matmul(x, direction, **kw)
                    assert not np.isfinite(ref).all()
                    np.testing.assert_array_equal(grg.matmul(x.astype(dtype), direction, **kw), ref)


def _word_values() -> np.ndarray:
    rng = np.random.default_rng(9)
    one = np.asarray([1.0, -1.0])
    ties = np.concatenate([one * (1 + 2.0**-40), one * (1 + 3 * 2.0**-40), one * (2 - 2.0**-40)])
    top = np.asarray([2.0**128 * (1 - 2.0**-40), -(2.0**128) * (1 - 2.0**-41), 2.0**128 * (1 - 2.0**-42), 2.0**128, -1e300])
    low = np.asarray([2.0**-126, 2.0**-126 * (1 - 2.0**-39), 2.0**-149 * 1.75, 2.0**-165, -(2.0**-165) * 1.5, 2.0**-166, 2.0**-180, -1e-300])
    special = np.asarray([np.inf, -np.inf, np.nan])
    return np.concatenate([ties, top, low, special, rng.standard_normal(12), rng.standard_normal(6) * 1e30, rng.standard_normal(6) * 1e-42])


def test_mixed_words_bit_by_bit(synth_artifact):
    """One input value and zeros: every node that it reaches once holds exactly its stored words, which
    pass through the seed or encode kernel, the walk (its decoding and its rounding) and the output kernel."""
    values = _word_values()
    k = values.size
    hi, lo = encode(values)
    expected = decode(hi, lo)
    oracle = OracleGRG(synth_artifact)
    with B200Runtime(_layout(synth_artifact, k, precision="mixed")) as runtime:
        (grg,) = runtime.grgs
        N, S, M, ld = grg.num_nodes, grg.num_samples, grg.num_mutations, nat.mix_ld(k)
        for direction, cols in (("up", S), ("down", M)):
            for col in (0, cols // 2, cols - 1):
                unit = np.zeros((1, cols))
                unit[0, col] = 1.0
                reached = oracle.matmul(unit, direction, emit_all_nodes=True)[0]
                x = np.zeros((k, cols))
                x[:, col] = values
                got = grg.matmul(x, direction, emit_all_nodes=True)
                once = reached == 1.0
                assert once.sum() > 1
                np.testing.assert_array_equal(got[:, once], np.broadcast_to(expected[:, None], (k, int(once.sum()))))
                assert not got[:, reached == 0.0].any()
        op = grg.prepare_matmul_cuda(direction="up", k=k)  # the words themselves: level 0 holds the inputs
        x = np.zeros((k, S))
        x[:, 5] = values
        op.input.copy_(torch.from_numpy(x))
        op()
        torch.cuda.synchronize()
        raw = runtime._state.cpu().numpy()
        got_hi = raw[: N * ld * 4].view(np.uint32).reshape(N, ld)[5, :k]
        got_lo = raw[nat.mix_plane(N * ld * 4):][: N * ld * 2].view(np.uint16).reshape(N, ld)[5, :k]
        nan = np.isnan(values)
        np.testing.assert_array_equal(got_hi[~nan], hi[~nan])
        np.testing.assert_array_equal(got_lo[~nan], lo[~nan].astype(np.uint16))
        assert np.isnan(decode(got_hi[nan], got_lo[nan].astype(np.uint32))).all()
