"""The workloads that the framework's speed is followed on.

A case is a dict of plain values: the shape of a synthetic genotype graph (the fields of
``SynthSpec``) and one call on it.  ``op`` names the entry point that the case goes through:

* ``prepared``: ``grg.prepare_matmul_cuda(...)``, whose op is called over and over (the inner
  loop of PCA, of association scans and of conjugate gradients);
* ``matmul``: ``grg.matmul`` on NumPy arrays, the eager call of a script;
* ``gram``: ``StandardizedXTX.apply``, the operator of randomized PCA;
* ``batch``: ``runtime.prepare_batch``, many blocks of right-hand sides on one graph.

A graph is fixed by its case, as a user's artifact is; the values that are multiplied come from
the seed.  Artifacts are generated once and kept in the system's temporary folder.
"""

from __future__ import annotations

import functools
import hashlib
import math
import os
from pathlib import Path
import tempfile

import numpy as np
import torch

from grg_spmv_b200 import RuntimeRequirements
from grg_spmv_b200.artifact import scan_grg_spmv
from grg_spmv_b200.backends.b200 import B200PlanPair, B200Plan, B200Runtime, BatchItem, plan_b200_layout
from grg_spmv_b200.synth import CONFIG1, CONFIG2, SynthSpec, write_synthetic_artifact
from grg_spmv_b200.xtx import StandardizedXTX


def _graph(spec: SynthSpec) -> dict:
    return {"num_samples": spec.num_samples, "num_levels": spec.num_levels, "num_nodes": spec.num_nodes,
            "num_mutations": spec.num_mutations, "children_min": spec.children[0], "children_max": spec.children[1],
            "miss_fraction": spec.miss_fraction, "ploidy": spec.ploidy, "with_coalescence": spec.with_coalescence,
            "random_ids": spec.random_ids, "graph_seed": spec.seed}


# The graph of the smoke test, the CPU-sized and the plain-FP64 configurations, the benchmark's
# small graph (diploid, no missing data) and its medium one (diploid, 1% missing, coalescences).
_SMOKE = _graph(SynthSpec(num_samples=512, num_levels=8, num_nodes=6_000, num_mutations=2_000, children=(2, 10),
                          miss_fraction=0.02, random_ids=True, seed=7))
_CPU_SIZED = _graph(CONFIG1)
_PLAIN = _graph(CONFIG2)
_SMALL = _graph(SynthSpec(num_samples=20_000, num_levels=20, num_nodes=600_000, num_mutations=100_000, children=(2, 28),
                          ploidy=2, seed=0))
_MEDIUM = _graph(SynthSpec(num_samples=30_000, num_levels=40, num_nodes=1_500_000, num_mutations=300_000, children=(2, 22),
                           miss_fraction=0.01, ploidy=2, with_coalescence=True, seed=0))


def _case(graph: dict, op: str = "prepared", **call) -> dict:
    base = {"op": op, "direction": "up", "k": 1, "dtype": "float64", "precision": "plain", "init": "none", "use_miss": False,
            "by_individual": False, "streamed": 0.0}
    return {**graph, **base, **call}


def listed() -> list[dict]:
    return [
        # the smallest call there is: one vector through a graph of a few thousand nodes
        {"name": "smoke up k1", **_case(_SMOKE)},
        # one vector the other way through the configuration that a CPU still runs comfortably
        {"name": "cpu-sized down k1", **_case(_CPU_SIZED, direction="down")},
        # a script's eager call with host arrays in and out, a handful of vectors
        {"name": "cpu-sized matmul k4", **_case(_CPU_SIZED, "matmul", k=4)},
        # the headline workload, each direction by itself (the down step with missing data)
        {"name": "plain up k8", **_case(_PLAIN, k=8)},
        {"name": "plain down k8", **_case(_PLAIN, direction="down", k=8, use_miss=True)},
        # one phenotype or one power-iteration vector on an ordinary graph
        {"name": "medium up k1", **_case(_MEDIUM, by_individual=True)},
        # a few covariates: a width that no vector load divides, with missing data, per individual
        {"name": "medium down k3", **_case(_MEDIUM, direction="down", k=3, use_miss=True, by_individual=True)},
        # single precision, a block of vectors
        {"name": "medium down f32 k16", **_case(_MEDIUM, direction="down", k=16, dtype="float32")},
        # the precision configuration: mixed node state, diploid, coalescence initialisation
        {"name": "medium up mixed k32", **_case(_MEDIUM, k=32, precision="mixed", init="xtx")},
        # randomized PCA's operator, both directions and the centring and scaling around them
        {"name": "small gram k64", **_case(_SMALL, "gram", k=64)},
        # uneven blocks, both directions, one call
        {"name": "small batch 1+3+16+64", **_case(_SMALL, "batch", k=84)},
        # conjugate gradients' block on a device budget that half of the gather lists exceed
        {"name": "medium up streamed k16", **_case(_MEDIUM, k=16, streamed=0.5)},
    ]


def _log_between(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    """One more call: a graph of any size up to the medium one, any direction, width, type and option,
    with at most the node values of the listed batch."""
    nodes = _log_between(rng, 6_000, 1_500_000)
    widest = max(8, min(96, 50_000_000 // nodes))
    graph = {"num_samples": max(64, nodes // rng.randint(12, 60)), "num_levels": rng.randint(8, 40), "num_nodes": nodes,
             "num_mutations": max(100, nodes // rng.randint(3, 6)), "children_min": 2, "children_max": rng.randint(8, 28),
             "miss_fraction": rng.choice([0.0, 0.01, 0.02]), "ploidy": 2, "with_coalescence": True,
             "random_ids": rng.random() < 0.3, "graph_seed": rng.randint(0, 1_000_000)}
    graph["num_samples"] -= graph["num_samples"] % 2
    op = rng.choice(["prepared"] * 6 + ["matmul", "batch", "gram"])
    if op == "gram":
        return _case({**graph, "miss_fraction": 0.0}, op, k=_log_between(rng, 2, min(64, widest)))
    if op == "batch":
        return _case(graph, op, k=_log_between(rng, 8, max(9, widest)))
    direction = rng.choice(["up", "down"])
    if op == "matmul":
        return _case({**graph, "num_nodes": min(graph["num_nodes"], 100_000), "num_mutations": min(graph["num_mutations"], 25_000),
                      "num_samples": min(graph["num_samples"], 5_000)}, op, direction=direction, k=_log_between(rng, 1, 16))
    kind = rng.choice(["float64", "float64", "float64", "float32", "mixed"])
    use_miss = rng.random() < 0.3
    return _case(graph, direction=direction, k=_log_between(rng, 1, min(64, widest)), dtype="float32" if kind == "float32" else "float64",
                 precision="mixed" if kind == "mixed" else "plain", use_miss=use_miss,
                 init="none" if use_miss else rng.choice(["none", "none", "vector", "xtx"]), by_individual=rng.random() < 0.4)


# -- inputs ----------------------------------------------------------------------------------------

def _artifact(case: dict) -> Path:
    spec = SynthSpec(num_samples=case["num_samples"], num_levels=case["num_levels"], num_nodes=case["num_nodes"],
                     num_mutations=case["num_mutations"], children=(case["children_min"], case["children_max"]),
                     miss_fraction=case["miss_fraction"], ploidy=case["ploidy"], with_coalescence=case["with_coalescence"],
                     random_ids=case["random_ids"], seed=case["graph_seed"])
    folder = Path(tempfile.gettempdir()) / f"grg_spmv_perf_{os.getuid()}"
    path = folder / (hashlib.sha256(repr(spec).encode()).hexdigest()[:24] + ".grg_spmv")
    if not path.exists():
        write_synthetic_artifact(spec, path)
    return path


def _blocks(k: int) -> list[int]:
    """Uneven block widths that add up to k: 1, 3, 16 and the rest, as far as they go."""
    widths, left = [], k
    for w in (1, 3, 16):
        if left > w:
            widths.append(w)
            left -= w
    return widths + [left]


def _input_cols(case: dict) -> int:
    if case["direction"] == "down":
        return case["num_mutations"]
    return case["num_samples"] // case["ploidy"] if case["by_individual"] else case["num_samples"]


def _values(case: dict, seed: int) -> dict:
    """The call's dense inputs, one row per vector and node-major in memory (the layout of a
    prepared op's views), in the case's type."""
    dtype = torch.float32 if case["dtype"] == "float32" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(cols, k):
        return torch.randn((cols, k), generator=gen, device="cuda", dtype=dtype).T

    k = case["k"]
    if case["op"] == "gram":
        return {"v": normal(case["num_mutations"], k).T}
    if case["op"] == "batch":
        return {"up": [normal(case["num_samples"], w) for w in _blocks(k)], "down": [normal(case["num_mutations"], w) for w in _blocks(k)]}
    values = {"x": normal(_input_cols(case), k)}
    if case["use_miss"] and case["direction"] == "down":
        values["miss"] = normal(case["num_mutations"], k)
    if case["init"] == "vector":
        values["init"] = normal(k, 1)[0].contiguous()
    return values


class _State:
    """An entered runtime with what the case calls on it; released with the state."""

    def __init__(self, case: dict, seed: int) -> None:
        self.op = case["op"]
        both = self.op in ("gram", "batch")
        up, down = both or case["direction"] == "up", both or case["direction"] == "down"
        req = RuntimeRequirements(max_k_up=case["k"], max_k_down=case["k"],
                                  need_down_miss_input=case["use_miss"] and case["direction"] == "down",
                                  need_up_miss_output=case["use_miss"] and case["direction"] == "up",
                                  need_init_vector=case["init"] == "vector", need_init_matrix=False,
                                  need_init_xtx=case["init"] == "xtx")
        call = dict(artifacts=[_artifact(case)], dtype=np.dtype(case["dtype"]), requirements=req, device=0, stream=0,
                    precision=case["precision"], pair=B200PlanPair(plan_up=B200Plan() if up else None, plan_down=B200Plan() if down else None),
                    emit_all_nodes=False)
        layout = plan_b200_layout(vram_budget_bytes=0, ring_buffer_size=0, **call)
        if case["streamed"] > 0.0:
            budget = layout.required_budget_for_full_residency - int(case["streamed"] * layout.bytes_by_category["resident_sparse"])
            layout = plan_b200_layout(vram_budget_bytes=budget, ring_buffer_size=4, **call)
        values = _values(case, seed)
        self.direction = case["direction"]
        self.runtime = B200Runtime(layout)
        self.runtime.__enter__()
        (self.grg,) = self.runtime.grgs
        if self.op == "matmul":
            self.x = values["x"].cpu().contiguous().numpy()
            self.options = {"by_individual": case["by_individual"]}
        elif self.op == "gram":
            self.gram = StandardizedXTX(self.runtime, self.grg, case["k"])
            self.v = values["v"]
        elif self.op == "batch":
            widths = _blocks(case["k"])
            self.batch = self.runtime.prepare_batch([BatchItem(self.grg, d, w) for d in ("up", "down") for w in widths])
            for view, x in zip(self.batch.inputs, values["up"] + values["down"]):
                view.copy_(x)
        else:
            self.prepared = self.grg.prepare_matmul_cuda(direction=case["direction"], k=case["k"], by_individual=case["by_individual"],
                                                         init_mode=case["init"], use_miss=case["use_miss"])
            self.x = values["x"]
            self.miss_output = case["use_miss"] and case["direction"] == "up"
            if "miss" in values:
                self.prepared.miss_input.copy_(values["miss"])
            if "init" in values:
                self.prepared.init_vector.copy_(values["init"])

    def __del__(self) -> None:
        runtime = getattr(self, "runtime", None)
        if runtime is not None and torch is not None:
            if self.op == "batch":
                self.batch.close()
            runtime.__exit__(None, None, None)


def prepare(case: dict, seed: int) -> _State:
    return _State(case, seed)


def run(state: _State):
    if state.op == "matmul":
        return state.grg.matmul(state.x, state.direction, **state.options)
    if state.op == "gram":
        return state.gram.apply(state.v)
    if state.op == "batch":
        state.batch()
        return list(state.batch.outputs)
    op = state.prepared
    op.input.copy_(state.x)  # a prepared op's output shares the buffer of its input
    op()
    return {"out": op.output, "miss": op.miss_output} if state.miss_output else {"out": op.output}


def work(case: dict) -> dict:
    """Every edge's index once, the dense inputs once and the dense outputs once; one addition per edge and vector."""
    scan = scan_grg_spmv(_artifact(case))
    size = 4 if case["dtype"] == "float32" else 8
    k, samples, mutations, edges = case["k"], case["num_samples"], case["num_mutations"], scan.num_edges
    individuals = samples // case["ploidy"]
    if case["op"] == "gram":
        return {"bytes": 2 * 4 * edges + 2 * size * mutations * k, "flops": 2 * edges * k}
    if case["op"] == "batch":
        return {"bytes": 2 * 4 * edges + 2 * size * (samples + mutations) * k, "flops": 2 * edges * k}
    ends = mutations * (2 if case["use_miss"] else 1) + (individuals if case["by_individual"] else samples)
    selected = scan.selector_mut_nnz + (scan.selector_miss_nnz if case["use_miss"] else 0)
    return {"bytes": 4 * (edges + selected) + size * ends * k, "flops": edges * k}


# -- the same products in 64 bits --------------------------------------------------------------------

@functools.lru_cache(maxsize=1)
def _edges(path: Path):
    """The artifact's edges, selectors and maps as tensors, read without the framework: per parent
    level the parent and child of every edge, in the artifact's node order."""
    def dev(a):
        return torch.from_numpy(np.asarray(a, dtype=np.int64)).cuda()

    with np.load(path) as data:
        offsets = np.asarray(data["level_offsets"], dtype=np.int64)
        levels = []
        for level in range(len(offsets) - 1):
            parents, children = [], []
            for below in range(level):
                indptr = np.asarray(data[f"A_blocks_{level}_{below}_indptr"], dtype=np.int64)
                parents.append(np.repeat(np.arange(offsets[level], offsets[level + 1]), np.diff(indptr)))
                children.append(np.asarray(data[f"A_blocks_{level}_{below}_indices"], dtype=np.int64) + offsets[below])
            levels.append((dev(np.concatenate(parents)), dev(np.concatenate(children))) if parents else None)
        selectors = {}
        for name in ("mut", "miss"):
            indptr = np.asarray(data[f"sel_{name}_indptr"], dtype=np.int64)
            selectors[name] = (dev(np.repeat(np.arange(indptr.size - 1), np.diff(indptr))), dev(data[f"sel_{name}_indices"]))
        coal = dev(data["coalescence_counts"]) if "coalescence_counts" in data.files else None
        return levels, selectors, dev(data["sample_to_individual"]), coal, int(data["num_nodes"]), int(data["num_mutations"])


def _exact_product(path: Path, x, direction: str, by_individual: bool, miss=None, init=None, miss_out: bool = False):
    """(input columns, k) -> (output columns, k) in FP64, and the miss rows of an up product (or None)."""
    levels, selectors, individual, coal, num_nodes, num_mutations = _edges(path)
    x = x.double()
    k = x.shape[1]
    nodes = torch.zeros((num_nodes, k), dtype=torch.float64, device="cuda")
    if init is not None:
        nodes += 2.0 * coal.double()[:, None] if isinstance(init, str) else init.double()[None, :]
    if direction == "up":
        nodes[: individual.numel()] += x[individual] if by_individual else x
        for edges in levels:
            if edges is not None:
                nodes.index_add_(0, edges[0], nodes[edges[1]])
        outs = []
        for name in ("mut", "miss") if miss_out else ("mut",):
            rows, at = selectors[name]
            outs.append(torch.zeros((num_mutations, k), dtype=torch.float64, device="cuda").index_add_(0, rows, nodes[at]))
        return outs[0], outs[1] if miss_out else None
    for name, rows_in in (("mut", x), ("miss", miss)):
        if rows_in is not None:
            rows, at = selectors[name]
            nodes.index_add_(0, at, rows_in.double()[rows])
    for edges in reversed(levels):
        if edges is not None:
            step = 1 << 23  # edges per gather, to bound its buffer
            for lo in range(0, edges[0].numel(), step):
                nodes.index_add_(0, edges[1][lo:lo + step], nodes[edges[0][lo:lo + step]])
    out = nodes[: individual.numel()]
    if by_individual:
        out = torch.zeros((int(individual.max()) + 1, k), dtype=torch.float64, device="cuda").index_add_(0, individual, out)
    return out, None


def exact(case: dict, seed: int):
    path = _artifact(case)
    values = _values(case, seed)
    if case["op"] == "gram":
        v = values["v"]
        individuals = case["num_samples"] // case["ploidy"]
        counts = _exact_product(path, torch.ones((individuals, 1), device="cuda"), "up", True)[0][:, 0]
        freq = counts / case["num_samples"]
        sigma = torch.sqrt(case["ploidy"] * freq * (1.0 - freq))
        sigma = torch.where(sigma == 0.0, 1.0, sigma)[:, None]
        centre = case["ploidy"] * freq[:, None]
        scaled = v / sigma
        u = _exact_product(path, scaled, "down", True)[0] - (centre * scaled).sum(0)
        return (_exact_product(path, u, "up", True)[0] - centre * u.sum(0)) / sigma
    if case["op"] == "batch":
        return [_exact_product(path, x.T, d, False)[0].T for d in ("up", "down") for x in values[d]]
    init = None if case["init"] == "none" else "xtx" if case["init"] == "xtx" else values["init"]
    up_miss = case["use_miss"] and case["direction"] == "up"
    miss_in = values["miss"].T if "miss" in values else None
    out, miss = _exact_product(path, values["x"].T, case["direction"], case["by_individual"], miss_in, init, up_miss)
    if case["op"] == "matmul":
        return out.T.cpu().numpy()
    return {"out": out.T, "miss": miss.T} if up_miss else {"out": out.T}
