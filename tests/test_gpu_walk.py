"""The library-chosen row walk of default plans (``level_walk.cu``) against the FP64 oracle: widths
around every chunk and warp boundary, input rows that are and are not aligned to a chunk, rows long
enough for the cluster kernel, and short, narrow and heavy rows in one level.

Integer-valued inputs are exact in any order of additions (sums stay below 2^24 in FP32).  Real
inputs differ by reassociation only: at most n eps times the sum of magnitudes of a row's n leaf
terms, with n below 2^16 here, so 2^16 * 2^-53 < 1e-11 in FP64 and, for FP32 against FP64, a
square-root law on n <= 2^16 random signs gives 2^8 * 2^-24 < 2e-5 of the result's norm."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402


@pytest.fixture(scope="module")
def artifact(tmp_path_factory):
    """60k nodes with random ids; thousands of its mutations sit on one node."""
    from grg_spmv_b200.synth import SynthSpec, write_synthetic_artifact

    path = tmp_path_factory.mktemp("walk") / "walk.grg_spmv"
    write_synthetic_artifact(SynthSpec(num_samples=1200, num_levels=12, num_nodes=60_000, num_mutations=40_000, children=(2, 14),
                                       miss_fraction=0.02, random_ids=True, seed=41), path)
    return path


@pytest.mark.parametrize("k,spare", [(1, 0), (1, 2), (2, 0), (2, 1), (3, 0), (4, 0), (5, 0), (7, 0), (8, 0), (8, 1), (12, 0), (20, 0),
                                     (33, 0), (64, 0), (65, 0), (84, 0), (84, 1), (128, 0), (132, 0), (257, 0)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_walk_against_oracle(artifact, dtype, k, spare):
    """``spare``: columns that the runtime's buffers hold beyond k (they move the input rows off
    their alignment)."""
    from grg_spmv_b200.backends.b200 import B200Runtime, plan_b200_layout
    from grg_spmv_b200.backends.b200 import _native as nat

    oracle = OracleGRG(artifact)
    req = RuntimeRequirements(max_k_up=k + spare, max_k_down=k + spare, need_down_miss_input=True, need_up_miss_output=False,
                              need_init_vector=False, need_init_matrix=False, need_init_xtx=False)
    layout = plan_b200_layout(artifacts=[str(artifact)], dtype=dtype, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                              device=0, stream=0)
    rng = np.random.default_rng(1000 + k)
    with B200Runtime(layout, check_bounds=False) as runtime:
        (grg,) = runtime.grgs
        levels = runtime._artifacts[0].levels["down"].array
        assert any(lv.long_rows[2] > 0 for lv in levels) and any(lv.short_rows > 0 for lv in levels)
        S, M = grg.num_samples, grg.num_mutations
        for direction, cols, use_miss in (("up", S, False), ("down", M, False), ("down", M, True)):
            x = rng.choice(np.asarray([-1.0, 0.0, 1.0]), size=(k, cols))
            miss = rng.choice(np.asarray([-1.0, 1.0]), size=(k, M)) if use_miss else None
            got = grg.matmul(x.astype(dtype), direction, miss=None if miss is None else miss.astype(dtype))
            np.testing.assert_array_equal(got, oracle.matmul(x, direction, miss=None if miss is None else miss.copy()))
            x = rng.standard_normal((k, cols)).astype(dtype)
            ref = oracle.matmul(x.astype(np.float64), direction)
            assert np.linalg.norm(grg.matmul(x, direction) - ref) <= (1e-11 if dtype == np.float64 else 2e-5) * np.linalg.norm(ref)
        with grg.prepare_matmul_cuda(direction="down", k=k) as op:
            assert op._args.launch_flags & nat.LAUNCH_WALK
