"""Mixed storage on the paths that ordinary calls take: no bounds checks, recorded and captured calls.

Integer-valued inputs are exact (sums stay below 2^40).  Real ones: each node is rounded to within
2^-40 of itself, a path has at most 12 nodes here, and the FP64 sums add less than 1e-11 (2^16 terms),
so a result is within 1e-10 of the largest magnitude sum."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from grg_oracle import OracleGRG  # noqa: E402
from grg_spmv_b200 import RuntimeRequirements  # noqa: E402


@pytest.fixture(scope="module")
def artifact(tmp_path_factory):
    """Diploid, random ids, thousands of mutations on one node (rows of every kind of walk)."""
    from grg_spmv_b200.synth import SynthSpec, write_synthetic_artifact

    path = tmp_path_factory.mktemp("mixed_paths") / "mixed.grg_spmv"
    write_synthetic_artifact(SynthSpec(num_samples=1200, num_levels=12, num_nodes=60_000, num_mutations=40_000, children=(2, 14),
                                       miss_fraction=0.02, ploidy=2, with_coalescence=True, random_ids=True, seed=41), path)
    return path


def _runtime(path, k, stream=0, **kw):
    from grg_spmv_b200.backends.b200 import B200Runtime, plan_b200_layout

    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=True, need_up_miss_output=True,
                              need_init_vector=True, need_init_matrix=False, need_init_xtx=True)
    layout = plan_b200_layout(artifacts=[str(path)], dtype=np.float64, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                              device=0, stream=stream, precision="mixed")
    return B200Runtime(layout, check_bounds=False, **kw)


@pytest.mark.parametrize("k", [1, 8])
@pytest.mark.parametrize("init", ["none", "vector"])
def test_mixed_up_captured_after_the_kernel_that_writes_its_input(artifact, init, k):
    """The caller's graph: a kernel writes the input, the traversal reads it, another kernel
    overwrites it (and so on, twice), all in one capture."""
    oracle = OracleGRG(artifact)
    rng = np.random.default_rng(17)
    stream = torch.cuda.Stream(device=0)
    with _runtime(artifact, k, stream) as runtime:
        (grg,) = runtime.grgs
        xs = [rng.integers(-4, 5, size=(k, grg.num_samples)).astype(np.float64) for _ in range(2)]
        v = rng.integers(-4, 5, size=k).astype(np.float64)
        op = grg.prepare_matmul_cuda(direction="up", k=k, init_mode=init)
        halves = [torch.from_numpy(x / 2).to("cuda:0") for x in xs]
        outs = [torch.empty((k, grg.num_mutations), device="cuda:0", dtype=torch.float64) for _ in xs]
        if init == "vector":
            op.init_vector.copy_(torch.from_numpy(v))
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for half, out in zip(halves, outs):
                torch.add(half, half, out=op.input)
                op()
                out.copy_(op.output)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        for x, out in zip(xs, outs):
            np.testing.assert_array_equal(out.cpu().numpy(), oracle.matmul(x, "up", init=v if init == "vector" else None))


def test_mixed_down_with_a_state_wider_than_k(artifact):
    """ld_state > k through the C interface: the encoded copies hold zeros from column k on, and no
    column past a source row is read (what follows the inputs is NaN here)."""
    import ctypes

    from grg_spmv_b200.backends.b200 import _native as nat

    k, ld = 8, 16
    oracle = OracleGRG(artifact)
    rng = np.random.default_rng(29)
    with _runtime(artifact, k) as runtime:
        (grg,) = runtime.grgs
        M, N = grg.num_mutations, grg.num_nodes
        args = grg.prepare_matmul_cuda(direction="down", k=k, use_miss=True)._args
        x, miss = (rng.integers(-4, 5, size=(M, k)).astype(np.float64) for _ in range(2))
        buffers = []
        for values in (x, miss):
            buf = torch.full((M + 2, k), float("nan"), device="cuda:0", dtype=torch.float64)
            buf[:M] = torch.from_numpy(values)
            buffers.append(buf)
        state = torch.zeros(nat.mix_bytes(N, ld), device="cuda:0", dtype=torch.uint8)
        scratch = torch.full((2 * nat.mix_bytes(M, ld),), 0x55, device="cuda:0", dtype=torch.uint8)
        out = torch.empty((grg.num_samples, k), device="cuda:0", dtype=torch.float64)
        args.input, args.miss, args.output = (t.data_ptr() for t in (*buffers, out))
        args.ld_input = args.ld_miss = args.ld_output = k
        args.state, args.ld_state = state.data_ptr(), ld
        args.mix_scratch, args.mix_scratch_bytes = scratch.data_ptr(), scratch.numel()
        torch.cuda.synchronize()
        nat.check(runtime._lib, runtime._lib.grg_b200_traverse(ctypes.byref(args), ctypes.c_void_p(runtime.stream_ptr)), "traverse")
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy().T, oracle.matmul(x.T.copy(), "down", miss=miss.T.copy()))
        for part in scratch.cpu().numpy().reshape(2, -1):
            hi = part[: M * ld * 4].view(np.uint32).reshape(M, ld)
            lo = part[nat.mix_plane(M * ld * 4):][: M * ld * 2].view(np.uint16).reshape(M, ld)
            assert not hi[:, k:].any() and not lo[:, k:].any()


@pytest.mark.parametrize("k", [(1 << 24) - 4, 1 << 24, (1 << 24) + 129])
def test_mixed_widths_around_2_to_the_24(k):
    """The widest calls: a graph of two nodes and as many columns as wanted."""
    from conftest import artifact_path
    from grg_spmv_b200.backends.b200 import B200Runtime, plan_b200_layout

    path = artifact_path("sparse_selector")
    oracle = OracleGRG(path)
    req = RuntimeRequirements(max_k_up=k, max_k_down=k, need_down_miss_input=False, need_up_miss_output=False,
                              need_init_vector=False, need_init_matrix=False, need_init_xtx=False)
    layout = plan_b200_layout(artifacts=[str(path)], dtype=np.float64, requirements=req, vram_budget_bytes=0, ring_buffer_size=0,
                              device=0, stream=0, precision="mixed", emit_all_nodes=False)
    with B200Runtime(layout, check_bounds=False) as runtime:
        (grg,) = runtime.grgs
        for direction, cols in (("up", grg.num_samples), ("down", grg.num_mutations)):
            weights = torch.from_numpy(oracle.matmul(np.eye(cols), direction)).to("cuda:0")
            op = grg.prepare_matmul_cuda(direction=direction, k=k)
            x = torch.arange(k * cols, device="cuda:0", dtype=torch.float64).remainder_(1021.0).view(k, cols)
            op.input.copy_(x)
            op()
            assert torch.equal(op.output, x @ weights)
