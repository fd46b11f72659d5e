"""Which kernels a call is launched with: what autotuning times and keeps, and early launches."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402
from grg_spmv_b200.backends.b200 import B200Plan, B200PlanPair, B200Runtime, plan_b200_layout  # noqa: E402
from grg_spmv_b200.backends.b200 import _native as nat  # noqa: E402


@pytest.fixture(scope="module")
def artifact(tmp_path_factory):
    from grg_spmv_b200.synth import SynthSpec, write_synthetic_artifact

    path = tmp_path_factory.mktemp("choice") / "mid.grg_spmv"
    write_synthetic_artifact(SynthSpec(num_samples=3000, num_levels=14, num_nodes=60_000, num_mutations=15_000, children=(2, 16),
                                       miss_fraction=0.02, ploidy=2, with_coalescence=True, random_ids=True, seed=21), path)
    return path


def _layout(path, k, **kw):
    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=True, need_up_miss_output=True, need_init_vector=True,
                              need_init_matrix=True, need_init_xtx=True)
    return plan_b200_layout(artifacts=[str(path)], dtype=np.float64, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                            device=0, stream=0, **kw)


class _Recording(B200Runtime):
    """Keeps the launch flags and kernel shapes of every launch."""

    def __init__(self, *args, **kw) -> None:
        super().__init__(*args, **kw)
        self.launched = []

    def _launch(self, args, recording=None) -> None:
        self.launched.append((int(args.direction), bool(args.launch_flags & nat.LAUNCH_WALK), int(args.narrow_variant), int(args.heavy_variant)))
        super()._launch(args, recording)


@pytest.mark.parametrize("checked", [False, True], ids=["plain", "checked"])
def test_autotune_times_what_later_calls_run(artifact, checked):
    """Every kernel shape is timed by itself, and the library's row walk beside them where it serves;
    what was kept is what calls run, and calls that the walk does not serve run the best shape."""
    k = 4
    oracle = OracleGRG(artifact)
    pair = B200PlanPair(plan_up=B200Plan(autotune=True), plan_down=B200Plan(autotune=True))
    rng = np.random.default_rng(13)
    with _Recording(_layout(artifact, k, pair=pair), check_bounds=checked) as runtime:
        (grg,) = runtime.grgs
        tuning = list(runtime.launched)
        for direction, code, cols in (("up", nat.UP, grg.num_samples), ("down", nat.DOWN, grg.num_mutations)):
            timed = [(walk, narrow) for d, walk, narrow, _ in tuning if d == code]
            assert {narrow for walk, narrow in timed if not walk} == set(runtime.TUNE_VARIANTS)
            assert any(walk for walk, _ in timed) == (not checked)
            runtime.launched.clear()
            x = rng.integers(-3, 4, size=(k, cols)).astype(np.float64)
            np.testing.assert_array_equal(grg.matmul(x, direction), oracle.matmul(x, direction))
            init = rng.integers(-3, 4, size=(k, grg.num_nodes)).astype(np.float64)
            np.testing.assert_array_equal(grg.matmul(x, direction, init=init), oracle.matmul(x, direction, init=init))
            plain, with_init = runtime.launched
            assert plain[1] == (not checked and runtime._row_walk[direction])
            for call in (plain, with_init):
                assert call[2:] == (runtime._variant[direction], runtime._heavy_variant[direction])


@pytest.mark.parametrize("precision,checked", [("plain", False), ("plain", True), ("mixed", False), ("mixed", True)])
def test_early_launches_below_8_columns_where_the_row_walk_serves(artifact, precision, checked):
    """Calls below k = 8 start levels early with the row walk only; from 8 on, and as a plan says, with any kernel."""
    for pdl in (None, True, False):
        pair = B200PlanPair(plan_up=B200Plan(pdl=pdl), plan_down=B200Plan(pdl=pdl))
        with B200Runtime(_layout(artifact, 8, pair=pair, precision=precision), check_bounds=checked) as runtime:
            (grg,) = runtime.grgs
            for k in (1, 2, 7, 8):
                for init, emit in (("none", False), ("none", True), ("matrix", False), ("vector", True)):
                    op = grg.prepare_matmul_cuda(direction="up", k=k, init_mode=init, emit_all_nodes=emit)
                    serves = precision == "mixed" or (init == "none" and not checked)
                    assert bool(op._args.launch_flags & nat.LAUNCH_PDL) == (k >= 8 or serves if pdl is None else pdl)
