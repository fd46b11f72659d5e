"""``grg_b200_rowop`` against the same steps in PyTorch FP64: every product and sum of an element is
rounded separately on both sides, so elements are equal bit for bit; a column sum of n terms
differs by the order of additions, at most n eps times the sum of magnitudes."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,k", [(1, 1), (31, 2), (32, 64), (33, 3), (1000, 130), (40_000, 6), (100_000, 5), (2_500, 600)])
@pytest.mark.parametrize("terms", ["", "pre sums weight", "miss_in pre sub scale post miss_out sums", "sub sums", "miss_in pre sub scale"])
def test_rowop_matches_torch(rows, k, terms):
    from grg_spmv_b200.backends.b200 import _native as nat

    lib = nat.load_library()
    on = set(terms.split())
    gen = torch.Generator(device="cuda").manual_seed(rows + k)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)

    src, miss, col = rand(rows, k), rand(rows, k), rand(k)
    vec = {name: rand(rows) for name in ("miss_scale", "pre", "sub", "post", "miss_out", "weight")}
    dst, miss_out, sums = torch.empty_like(src), torch.empty_like(src), torch.zeros(k, device="cuda", dtype=torch.float64)
    partials = torch.empty((nat.rowop_blocks(rows), k), device="cuda", dtype=torch.float64)

    def ptr(t, name):
        return int(t.data_ptr()) if name in on else None

    args = nat.RowopArgs(rows=rows, k=k, ld=k, src=int(src.data_ptr()), dst=int(dst.data_ptr()), miss_in=ptr(miss, "miss_in"),
                         miss_scale=ptr(vec["miss_scale"], "miss_in"), pre_scale=ptr(vec["pre"], "pre"), col_sub=ptr(col, "sub"),
                         sub_scale=ptr(vec["sub"], "scale"), post_scale=ptr(vec["post"], "post"), miss_out=ptr(miss_out, "miss_out"),
                         miss_out_scale=ptr(vec["miss_out"], "miss_out"), col_sums=int("sums" in on),
                         sum_weight=ptr(vec["weight"], "weight"), partials=int(partials.data_ptr()), sums=int(sums.data_ptr()))
    nat.check(lib, lib.grg_b200_rowop(ctypes.byref(args), None), "grg_b200_rowop")
    torch.cuda.synchronize()
    want = src.clone()
    if "miss_in" in on:
        want = want + miss * vec["miss_scale"][:, None]
    if "pre" in on:
        want = want * vec["pre"][:, None]
    if "sub" in on:
        want = want - (col[None, :] * vec["sub"][:, None] if "scale" in on else col[None, :])
    if "post" in on:
        want = want * vec["post"][:, None]
    assert torch.equal(dst, want)
    if "miss_out" in on:
        assert torch.equal(miss_out, want * vec["miss_out"][:, None])
    if "sums" in on:
        weighted = want * vec["weight"][:, None] if "weight" in on else want
        bound = rows * 2.0**-53 * weighted.abs().sum(0) + 1e-300
        assert bool(((sums - weighted.sum(0)).abs() <= 2 * bound).all())
