"""32-bit products on the tensor cores in bfloat16 pieces (csrc/gemm_split_tcgen05.cu) against 64 bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def bound(x, w):
    """Of sum |x w|: the three products of pieces that are left out (2^-22); four additions of a block of 64 of k in an
    accumulator that rounds towards zero (2^-23 each); the small products, 2^-6 of the whole, over a segment of K / 8 in
    such accumulators (3 K / 128 additions); then up to K / 512 + 6 rounded additions of 2^-24."""
    k = x.shape[1]
    return (2.0 ** -22 + 4 * 2.0 ** -23 + (3 * k / 128 + 12) * 2.0 ** -29 + (k / 512 + 6) * 2.0 ** -24) \
        * (x.double().abs() @ w.double().abs().t())


@pytest.mark.parametrize("m,k", [(1, 512), (130, 516), (1024, 1024), (200, 2060), (6144, 1024), (40, 3072)])
def test_split_product_is_the_same_however_it_is_cut(m, k):
    """Every number of rows, every number of CTAs per tile and every height of the tiles gives the bits of the largest
    product, within the bound, and closer to 64 bits than one chain of fused multiply-adds."""
    from inferrs_b200 import kernels as K
    x, w = rand((130, k), 1), rand((m, k), 2)
    want, limit = x.double() @ w.double().t(), bound(x, w)
    whole = torch.full((130, m), float("nan"), device="cuda")
    K.gemm_tn_split(x, w, whole)
    err = (whole.double() - want).abs()
    assert bool((err <= limit).all())
    chain = torch.empty_like(whole)
    K.gemm_tn_simt(x, w, chain, torch.float32)
    assert float(err.norm()) <= float((chain.double() - want).norm())
    for n in (1, 16, 17, 32, 33, 64, 65, 130):
        for splits, tile_rows in ((0, 0), (1, 128), (2, 40), (4, 96), (8, 16), (8, 128)):
            out = torch.full((n, m), float("nan"), device="cuda")
            K.gemm_tn_split(x[:n], w, out, splits, tile_rows)
            assert torch.equal(out, whole[:n]), (n, splits, tile_rows)
    assert K.gemm_split_error() == 0


def test_split_product_of_infinities_nan_and_the_range_ends():
    """What is no finite number comes out as the chain makes it; large and small numbers keep their precision."""
    from inferrs_b200 import kernels as K
    x, w = rand((20, 1024), 3), rand((200, 1024), 4)
    x[3, 7], x[5, 9], w[11, 100] = float("inf"), float("nan"), -float("inf")
    x[6], w[20] = 1e38, 3e38
    x[8] *= 1e-30
    x[9, 1:] = 0.0
    out, chain = torch.empty((20, 200), device="cuda"), torch.empty((20, 200), device="cuda")
    K.gemm_tn_split(x, w, out)
    K.gemm_tn_simt(x, w, chain, torch.float32)
    odd = ~chain.isfinite()
    assert torch.equal(out.isfinite(), chain.isfinite()) and bool(odd.any())
    assert torch.equal(out[odd].nan_to_num(1.0, 2.0, 3.0), chain[odd].nan_to_num(1.0, 2.0, 3.0))
    rows = torch.tensor([8, 9], device="cuda")
    cols = torch.tensor([c for c in range(200) if c not in (11, 20)], device="cuda")
    want = x[rows].double() @ w[cols].double().t()
    assert bool(((out[rows][:, cols].double() - want).abs() <= bound(x[rows], w[cols])).all())


def test_linear_takes_the_split_product_by_its_width_alone():
    from inferrs_b200 import kernels as K
    for k in (508, 512, 514, 1024):
        x, w = rand((70, k), 5), rand((96, k), 6)
        out = [torch.empty((n, 96), device="cuda") for n in (70, 3)]
        for o in out:
            K.linear(x[:o.shape[0]], w, o, torch.float32)
        ref = torch.empty((70, 96), device="cuda")
        (K.gemm_tn_split if k >= 512 and k % 4 == 0 else lambda a, b, c: K.gemm_tn_simt(a, b, c, torch.float32))(x, w, ref)
        assert torch.equal(out[0], ref) and torch.equal(out[1], ref[:3])
