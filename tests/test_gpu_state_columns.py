"""Whose columns of the node state a call may touch, through the C interface: [0, k) only, unless
GRG_B200_STATE_PADDING says that the rest of each row is scratch too.  Integer inputs, exact results."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402


@pytest.fixture(scope="module")
def artifact(tmp_path_factory):
    """Rows of every kind: short, narrow, heavy and (down, from the mutation hub) a cluster's."""
    from grg_spmv_b200.synth import SynthSpec, write_synthetic_artifact

    path = tmp_path_factory.mktemp("columns") / "columns.grg_spmv"
    write_synthetic_artifact(SynthSpec(num_samples=1200, num_levels=12, num_nodes=60_000, num_mutations=40_000, children=(2, 14),
                                       miss_fraction=0.02, random_ids=True, seed=41), path)
    return path


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k,first,ld", [(1, 0, 8), (3, 0, 8), (3, 4, 8), (5, 0, 8), (6, 8, 16), (8, 8, 24), (9, 0, 16)])
@pytest.mark.parametrize("direction", ["up", "down"])
def test_columns_beside_the_call_keep_their_values(artifact, direction, k, first, ld, dtype):
    """Node states in columns [first, first + k) of wider rows; the last row ends with the call's columns."""
    from grg_spmv_b200.backends.b200 import B200Runtime, plan_b200_layout
    from grg_spmv_b200.backends.b200 import _native as nat

    oracle = OracleGRG(artifact)
    rng = np.random.default_rng(60 + k)
    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=True, need_up_miss_output=False,
                              need_init_vector=False, need_init_matrix=False, need_init_xtx=False)
    layout = plan_b200_layout(artifacts=[str(artifact)], dtype=dtype, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                              device=0, stream=0)
    with B200Runtime(layout, check_bounds=False) as runtime:
        (grg,) = runtime.grgs
        op = grg.prepare_matmul_cuda(direction=direction, k=k)
        args, N = op._args, grg.num_nodes
        assert args.launch_flags & nat.LAUNCH_WALK
        x = rng.integers(-3, 4, size=tuple(op.input.shape))
        ref = oracle.matmul(x.astype(np.float64), direction)
        tail = 64  # behind the last row's columns: another owner's
        state = torch.full((N * ld + tail,), -7.0, device="cuda:0", dtype=torch.float64 if dtype == np.float64 else torch.float32)
        for padding in (False, True):
            state.fill_(-7.0)
            op.input.copy_(torch.from_numpy(x))
            args.state = state.data_ptr() + first * state.element_size()
            args.ld_state = ld
            args.launch_flags = (args.launch_flags & ~nat.STATE_PADDING) | (nat.STATE_PADDING if padding and first == 0 else 0)
            torch.cuda.synchronize()
            nat.check(runtime._lib, runtime._lib.grg_b200_traverse(ctypes.byref(args), ctypes.c_void_p(runtime.stream_ptr)), "traverse")
            torch.cuda.synchronize()
            np.testing.assert_array_equal(op.output.cpu().numpy(), ref)
            got = state.cpu().numpy()
            assert (got[N * ld:] == -7.0).all()
            if not padding or first:
                rows = got[: N * ld].reshape(N, ld)
                assert (rows[:, :first] == -7.0).all() and (rows[:, first + k:] == -7.0).all()
