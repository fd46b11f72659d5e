"""Padded node states are given up where the device has little room, and results stay as they are."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402
from grg_spmv_b200.backends.b200 import B200Runtime, plan_b200_layout  # noqa: E402


@pytest.fixture(scope="module")
def artifact(tmp_path_factory):
    from grg_spmv_b200.synth import SynthSpec, write_synthetic_artifact

    path = tmp_path_factory.mktemp("room") / "room.grg_spmv"
    write_synthetic_artifact(SynthSpec(num_samples=1200, num_levels=12, num_nodes=60_000, num_mutations=40_000, children=(2, 14),
                                       random_ids=True, seed=41), path)
    return path


@pytest.mark.parametrize("dtype,k,padded", [(np.float64, 5, 8), (np.float64, 3, 4), (np.float32, 9, 16)])
@pytest.mark.parametrize("full", [False, True], ids=["room", "full"])
def test_states_without_padding_on_a_full_device(artifact, monkeypatch, full, dtype, k, padded):
    oracle = OracleGRG(artifact)
    rng = np.random.default_rng(k)
    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=False, need_up_miss_output=False,
                              need_init_vector=False, need_init_matrix=False, need_init_xtx=False)
    layout = plan_b200_layout(artifacts=[str(artifact)], dtype=dtype, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                              device=0, stream=0)
    if full:  # what is free and cached would not hold the layout twice
        monkeypatch.setattr(torch.cuda, "memory_reserved", torch.cuda.memory_allocated)
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (2 * layout.bytes_by_category["state"] - 1, 1 << 37))
    ld = k if full else padded
    with B200Runtime(layout, check_bounds=False) as runtime:
        (grg,) = runtime.grgs
        N = grg.num_nodes
        assert runtime._state.numel() == N * ld
        x = rng.integers(-3, 4, size=(k, grg.num_samples)).astype(dtype)
        y = rng.integers(-3, 4, size=(k, grg.num_mutations)).astype(dtype)
        refs = oracle.matmul(x.astype(np.float64), "up"), oracle.matmul(y.astype(np.float64), "down")
        np.testing.assert_array_equal(grg.matmul(x, "up"), refs[0])
        np.testing.assert_array_equal(grg.matmul(y, "down"), refs[1])
        with runtime.prepare_batch([(grg, "up", k), (grg, "down", k)]) as batch:
            assert [t.state.numel() for g in batch._groups for t in g.tiles] == [N * ld] * 2
            for view, values in zip(batch.inputs, (x, y)):
                view.copy_(torch.from_numpy(values))
            batch()
            torch.cuda.synchronize()
            for view, ref in zip(batch.outputs, refs):
                np.testing.assert_array_equal(view.cpu().numpy(), ref)
