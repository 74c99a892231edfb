"""32-bit products on the tensor cores in bfloat16 pieces (csrc/gemm_split_tcgen05.cu) against 64 bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def bound(x, w):
    """Of sum |x w|: the product of the two smallest pieces, which is left out (2^-34); four additions of a block of 64 of k in
    an accumulator that rounds towards zero (2^-23 each); the small products, 2^-6 of the whole, over a segment of K / 8 in
    such accumulators (7 K / 128 additions); then up to K / 512 + 5 rounded additions of 2^-24."""
    k = x.shape[1]
    return (2.0 ** -34 + 4 * 2.0 ** -23 + (7 * k / 128 + 12) * 2.0 ** -29 + (k / 512 + 5) * 2.0 ** -24) \
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


@pytest.mark.parametrize("n,m,k", [(3, 70, 512), (16, 130, 1000), (17, 70, 4096), (64, 130, 1024), (130, 70, 3072)])
def test_a_sum_of_one_product_is_rounded_once(n, m, k):
    """One number of a row of x that is not zero, at every place of a block of k and in every segment: the product in 64 bits
    rounded to 24 (2^-24; the small pieces' products, 2^-6 of it, meet five additions that round towards zero), no worse than the
    chain of multiply-adds.  And with numbers whose pieces are the largest that there can be."""
    from inferrs_b200 import kernels as K
    worst = torch.tensor([1 + 2.0 ** -7 - 2.0 ** -23, 1 + 2.0 ** -8 - 2.0 ** -23, 1 + 2.0 ** -8 + 2.0 ** -16, 2 - 2.0 ** -23], device="cuda")
    x, w = torch.zeros((n, k), device="cuda"), rand((m, k), 8)
    w[:4] = worst[:, None]
    at = torch.arange(n, device="cuda") * 61 % k
    x[torch.arange(n), at] = torch.cat([worst, rand((n,), 9)])[:n]
    out, chain = torch.empty((n, m), device="cuda"), torch.empty((n, m), device="cuda")
    K.gemm_tn_split(x, w, out)
    K.gemm_tn_simt(x, w, chain, torch.float32)
    want = x.double() @ w.double().t()
    err, err_chain = (out.double() - want).abs(), (chain.double() - want).abs()
    assert bool((err <= (2.0 ** -24 + 5 * 2.0 ** -29) * want.abs()).all())
    assert float(err.norm()) <= 1.01 * float(err_chain.norm())


@pytest.mark.parametrize("kind", ["worst", "positive", "one beyond the others"])
@pytest.mark.parametrize("n,k", [(8, 512), (70, 2048), (20, 4096)])
def test_numbers_of_one_sign_and_sums_that_few_products_make(kind, n, k):
    """No part of a product is left out on one side: where every product would lose the same, and where one makes the sum,
    the result is within the bound and nearer to 64 bits than the chain's."""
    from inferrs_b200 import kernels as K
    if kind == "worst":
        x, w = torch.full((n, k), 1 + 2.0 ** -7 - 2.0 ** -23, device="cuda"), torch.full((96, k), 1 + 2.0 ** -7 - 2.0 ** -23, device="cuda")
    elif kind == "positive":
        x, w = rand((n, k), 10).abs(), rand((96, k), 11).abs()
    else:
        x, w = 1e-4 * rand((n, k), 12), rand((96, k), 13)
        x[:, k // 2] = 1 + rand((n,), 14).abs()
    out, chain = torch.empty((n, 96), device="cuda"), torch.empty((n, 96), device="cuda")
    K.gemm_tn_split(x, w, out)
    K.gemm_tn_simt(x, w, chain, torch.float32)
    want = x.double() @ w.double().t()
    err, err_chain = (out.double() - want).abs(), (chain.double() - want).abs()
    assert bool((err <= bound(x, w)).all()) and float(err.norm()) <= float(err_chain.norm())


def test_numbers_whose_first_piece_would_be_an_infinity():
    """Beyond 3.39e38 a number rounded to bfloat16 is none: such results are made as the chain makes them."""
    from inferrs_b200 import kernels as K
    x, w = rand((5, 512), 15), rand((130, 512), 16)
    x[2], w[7] = 0.0, 0.0
    x[2, 3], w[7, 5] = 3.4e38, -3.4028234e38
    w[:, 3] = 0.5
    out, chain = torch.empty((5, 130), device="cuda"), torch.empty((5, 130), device="cuda")
    K.gemm_tn_split(x, w, out)
    K.gemm_tn_simt(x, w, chain, torch.float32)
    assert torch.equal(out[2], chain[2]) and bool(out[2].isfinite().all())
    assert torch.equal(out[:, 7].nan_to_num(1.0, 2.0, 3.0), chain[:, 7].nan_to_num(1.0, 2.0, 3.0))


@pytest.mark.parametrize("n,k", [(5, 512), (40, 1024), (70, 1024)])
def test_numbers_whose_pieces_are_too_small_for_bfloat16(n, k):
    """A result below 2^-90 is the chain's; one row of zeros among them stays zero."""
    from inferrs_b200 import kernels as K
    w = rand((96, k), 18)
    for power in (-96, -110, -120, -126):
        x = rand((n, k), 17) * 2.0 ** power
        x[n // 2] = 0.0
        out, chain = torch.empty((n, 96), device="cuda"), torch.empty((n, 96), device="cuda")
        K.gemm_tn_split(x, w, out)
        K.gemm_tn_simt(x, w, chain, torch.float32)
        small = chain.abs() < 2.0 ** -90
        assert bool(small.any()) and torch.equal(out[small], chain[small])
        want = x.double() @ w.double().t()
        assert bool(((out.double() - want).abs() <= torch.where(small, 2.0 ** -23 * k ** 0.5 * (x.double().abs() @ w.double().abs().t()),
                                                               bound(x, w)) + 2.0 ** -148).all())
