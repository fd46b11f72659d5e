"""The eager call's result: an array of its own, brought to the host without device memory beside the layout's."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402
from grg_spmv_b200.backends.b200 import B200Runtime, plan_b200_layout  # noqa: E402


def _artifact(tmp_path, **kw):
    from grg_spmv_b200.synth import SynthSpec, write_synthetic_artifact

    spec = dict(num_samples=1200, num_levels=12, num_nodes=60_000, num_mutations=40_000, children=(2, 14), miss_fraction=0.02,
                ploidy=2, with_coalescence=True, random_ids=True, seed=41)
    return write_synthetic_artifact(SynthSpec(**{**spec, **kw}), tmp_path / "matmul.grg_spmv")


def _runtime(path, k, dtype, precision):
    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=False, need_up_miss_output=True, need_init_vector=False,
                              need_init_matrix=False, need_init_xtx=False)
    layout = plan_b200_layout(artifacts=[str(path)], dtype=dtype, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                              device=0, stream=0, precision=precision)
    return B200Runtime(layout, check_bounds=False)


@pytest.mark.parametrize("dtype,precision", [(np.float64, "plain"), (np.float32, "plain"), (np.float64, "mixed")])
@pytest.mark.parametrize("k", [1, 3, 8])
def test_result_arrays(tmp_path, k, dtype, precision):
    path = _artifact(tmp_path)
    oracle = OracleGRG(path)
    rng = np.random.default_rng(k)
    with _runtime(path, 8, dtype, precision) as runtime:
        (grg,) = runtime.grgs
        for direction, cols, kw in (("up", grg.num_samples, {}), ("up", grg.num_samples, {"emit_all_nodes": True}),
                                    ("down", grg.num_mutations, {}), ("down", grg.num_mutations, {"by_individual": True})):
            x = rng.integers(-3, 4, size=(k, cols)).astype(dtype)
            got = grg.matmul(x, direction, **kw)  # once for the library's one-time allocations
            del got
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            got = grg.matmul(x, direction, **kw)
            # the input may pass through a device copy of its own size
            assert torch.cuda.max_memory_allocated() - before <= x.nbytes + 1024
            assert got.dtype == dtype and got.flags.c_contiguous and got.flags.owndata and got.flags.writeable
            np.testing.assert_array_equal(got, oracle.matmul(x.astype(np.float64), direction, **kw))
        x = rng.integers(-3, 4, size=(k, grg.num_samples)).astype(dtype)
        miss, expected = np.ones((k, grg.num_mutations), dtype=dtype), np.ones((k, grg.num_mutations))
        np.testing.assert_array_equal(grg.matmul(x, "up", miss=miss), oracle.matmul(x.astype(np.float64), "up", miss=expected))
        np.testing.assert_array_equal(miss, expected)


def test_result_rows_longer_than_the_node_state(tmp_path):
    """More mutations than node values: the result comes back in pieces."""
    path = _artifact(tmp_path, num_samples=64, num_levels=4, num_nodes=300, num_mutations=5_000, miss_fraction=0.0, children=(2, 4))
    oracle = OracleGRG(path)
    x = np.arange(3 * 64, dtype=np.float64).reshape(3, 64)
    with _runtime(path, 3, np.float64, "plain") as runtime:
        (grg,) = runtime.grgs
        assert runtime._state.numel() < grg.num_mutations
        np.testing.assert_array_equal(grg.matmul(x, "up"), oracle.matmul(x, "up"))
