"""Kernels that may start while the previous one runs (programmatic dependent launch), by their source:
each has to wait for the previous grid before it touches what other kernels write."""

from __future__ import annotations

from pathlib import Path
import re

CSRC = Path(__file__).resolve().parents[1] / "grg_spmv_b200" / "csrc"


def _closing(text: str, start: int, pair: str) -> int:
    """Index after the bracket that closes the one at ``start``."""
    depth, i = 1, start + 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
    return i


def _source() -> str:
    text = "\n".join(p.read_text() for p in sorted(CSRC.glob("*.cu*")))
    text = re.sub(r"//[^\n]*", "", text)
    while (m := re.search(r"__(?:launch_bounds|cluster_dims|align)__\s*(?=\()", text)):
        text = text[:m.start()] + text[_closing(text, m.end(), "()"):]
    return text


def _functions(text: str) -> dict[str, str]:
    """Bodies of the device functions and kernels, by name (overloads joined)."""
    bodies: dict[str, str] = {}
    for m in re.finditer(r"__(?:device|global)__\b[^;{}()]*?\b(\w+)\s*(?=\()", text):
        end = _closing(text, m.end(), "()")
        body = re.compile(r"\s*\{").match(text, end)
        if body:
            bodies[m.group(1)] = bodies.get(m.group(1), "") + text[end:_closing(text, body.end() - 1, "{}")]
    return bodies


def _launched_early(text: str) -> set[str]:
    """Kernels launched through the helpers that take the launch attribute."""
    return {m.group(1) for m in re.finditer(r"launch_(?:smem_)?k\((?!bool)[^;]*?\b(\w+_kernel)\b", text)}


def test_kernels_launched_early_wait_for_the_previous_grid():
    text = _source()
    bodies, kernels = _functions(text), _launched_early(text)
    assert {"seed_up_kernel", "seed_up_mx_kernel", "level_walk_kernel", "level_hub_kernel", "gather_out_mx_kernel"} <= kernels

    def waits(name: str, seen: frozenset = frozenset()) -> bool:
        body = bodies.get(name, "")
        return "pdl_wait()" in body or any(
            waits(callee, seen | {name}) for callee in bodies if callee not in seen | {name} and re.search(rf"\b{callee}\b", body))

    assert sorted(k for k in kernels if not waits(k)) == []
    assert sorted(k for k, body in bodies.items() if "pdl_trigger()" in body and k != "pdl_trigger" and not waits(k)) == []


def test_read_only_loads_name_static_arrays():
    """A read-only load may be served by a line from before the previous grid's writes, and may be
    moved ahead of the wait: only lists, selectors, permutations and per-row constants take it."""
    text = _source()
    assert "ld.global.nc" not in text
    static = r"(?:[aL]\.)?(?:row_ptr|row_ids|entries|heavy_rows|codes4?|ptr|idx|node_perm|s2i|xtx_node|bias|(?:pre|sub|post|miss|miss_out)_scale|sum_weight)"
    loads = [text[m.end():_closing(text, m.end() - 1, "()") - 1] for m in re.finditer(r"__ldg\(", text)]
    assert len(loads) > 20
    unknown = [arg for arg in loads if not re.match(static + r"\b", re.sub(r"^(?:static_cast|reinterpret_cast)<[^>]*>+\(", "", arg))]
    assert unknown == []
