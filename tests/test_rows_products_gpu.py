"""bfloat16 products of a few rows by the kernel without clusters (csrc/gemm_tcgen05.cu) against 64 bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def close(got, want, terms):
    """Sums of ``terms`` exact products in float32 (2^-24 each of sum |x w|), then one rounding to the output's type."""
    half = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -24
    return bool(((got.double() - want).abs() <= half * want.abs() + terms).all())


FORMS = [(16, 1), (16, 3), (16, 16), (24, 1), (24, 8), (32, 8), (32, 13), (48, 5), (1024 + 16, 7), (1024 + 32, 16), (1024 + 32, 2)]


@pytest.mark.parametrize("r,n", FORMS)
@pytest.mark.parametrize("m,k", [(64, 8), (200, 72), (1000, 3080), (1024, 2048)])
def test_product_with_folded_norms_and_gate(r, n, m, k):
    from inferrs_b200 import kernels as K
    x, w = rand((n, k), 1), rand((m, k), 2, 0.05)
    dot = x.double() @ w.double().t()
    terms = k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((n, m), float("nan"), device="cuda", dtype=dtype)
        K.gemm_tn_tcgen05(x, w, out, split_k=-r)
        assert close(out, dot, terms)
    # rows scaled by the norm before, added to the stream, handed on times the weight of the norm after
    ssq = torch.rand(7, K.SSQ_LD, device="cuda")
    inv = 1.0 / torch.sqrt(ssq[:, :n].double().sum(0) / k + 1e-6)
    scaled = K.ScaledRows(x, ssq, 7, 1e-6, k)
    stream = torch.randn(n, m, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    weight, old = 0.5 + torch.rand(m, device="cuda"), stream.clone()
    out = torch.empty(n, m, dtype=torch.bfloat16, device="cuda")
    got = K.gemm_tn_tcgen05(scaled, w, out, split_k=-r, sink=K.ResidualSink(stream, weight, 1e-5))
    y = dot * inv[:, None]
    assert bool(((stream.double() - (old.double() + y)).abs() <= 2.0 ** -8 * y.abs() + terms * inv[:, None] + 1e-6).all())
    assert torch.equal(out, (stream * weight).to(torch.bfloat16))
    sums, want = got.ssq[:got.n_parts, :n].double().sum(0), (stream.double() ** 2).sum(1)
    assert got.n_parts == -(-m // (r % 1024)) and bool(((sums - want).abs() <= m * 2.0 ** -24 * want).all())
    if r <= (24 if n <= 8 else 16):
        inner = m // 2
        out = torch.full((n, inner), float("nan"), dtype=torch.bfloat16, device="cuda")
        K.gemm_swiglu_tcgen05(scaled, w[:2 * inner], out, rows_per_cta=r)
        g, u = y[:, :inner], y[:, inner:2 * inner]
        want = g / (1 + torch.exp(-g)) * u
        # both factors are rounded to bfloat16 first (2^-8 each; silu changes at most 1.1 times as much as its argument), the
        # result again
        off = terms * inv[:, None]                           # of the float32 sums
        off_g, off_u = off[:, :inner], off[:, inner:2 * inner]
        slack = 2.0 ** -8 * (1.11 * g.abs() * u.abs() + 2.1 * want.abs()) + 1.2 * (off_g * u.abs() + off_u * g.abs() + off_g * off_u)
        assert bool(((out.double() - want).abs() <= slack).all())
    assert K.gemm_tcgen05_error() == 0


@pytest.mark.parametrize("n", [1, 8, 9, 16])
@pytest.mark.parametrize("b,m,k", [(1, 40, 8), (3, 100, 72), (16, 512, 128), (16, 128, 512)])
def test_batch_of_products(n, b, m, k):
    """Heads of [rows, heads, k] and of [heads, rows, k], read and written in place; and rows that do not start on 16 bytes."""
    from inferrs_b200 import kernels as K
    w = rand((b, m, k), 4, 0.1)
    for x in (rand((n, b, k + 8), 5)[:, :, :k].transpose(0, 1), rand((b, n, k), 6), rand((n, b, k + 1), 7)[:, :, 1:].transpose(0, 1)):
        want = torch.einsum("bnk,bmk->bnm", x.double(), w.double())
        terms = k * 2.0 ** -24 * torch.einsum("bnk,bmk->bnm", x.double().abs(), w.double().abs())
        out = torch.full((n, b, m), float("nan"), dtype=torch.bfloat16, device="cuda")
        K.batched_linear(x, w, out.transpose(0, 1), torch.bfloat16)
        assert close(out.transpose(0, 1), want, terms)
        first = torch.empty((b, n, m), dtype=torch.bfloat16, device="cuda")
        K.batched_linear(x, w, first, torch.bfloat16)
        assert torch.equal(first, out.transpose(0, 1))


@pytest.mark.parametrize("n", [1, 16, 17])
def test_batch_of_empty_sums_is_zeros(n):
    from inferrs_b200 import kernels as K
    out = torch.full((2, n, 24), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.batched_linear(rand((2, n, 0), 4), rand((2, 24, 0), 5), out, torch.bfloat16)
    assert bool((out == 0).all())


@pytest.mark.parametrize("b,n,k", [(1, 1, 8), (3, 16, 72), (16, 9, 512)])
def test_batches_run_on_the_kernel_for_few_rows(b, n, k):
    """The library function itself takes whole rows of either layout, and leaves those that do not start on 16 bytes."""
    from inferrs_b200 import kernels as K
    lib, m = K._gemm_lib(), 40
    w, out = rand((b, m, k), 4, 0.1), torch.empty((b, n, m), dtype=torch.bfloat16, device="cuda")

    def call(x):
        out.fill_(float("nan"))
        return lib.ib_gemm_tn_rows_batched(x.data_ptr(), x.stride(1), x.stride(0), w.data_ptr(), out.data_ptr(), out.stride(1),
                                           out.stride(0), n, m, k, b, torch.cuda.current_stream().cuda_stream)

    for x in (rand((n, b, k + 8), 5)[:, :, :k].transpose(0, 1), rand((b, n, k), 6)):
        assert call(x) == 0
        terms = k * 2.0 ** -24 * torch.einsum("bnk,bmk->bnm", x.double().abs(), w.double().abs())
        assert close(out, torch.einsum("bnk,bmk->bnm", x.double(), w.double()), terms)
    assert call(rand((b, n, k + 1), 7)[:, :, 1:]) == -1 and bool(out.isnan().all())


@pytest.mark.parametrize("m,k", [(m, 72) for m in (8 * 148, 8 * 148 + 1, 32 * 148, 32 * 148 + 1, 32 * 296, 32 * 296 + 1, 48 * 296,
                                                   48 * 296 + 1, 4 * 48 * 296 - 1, 4 * 48 * 296)]
                         + [(m, k) for m in (8 * 148, 8 * 148 + 1, 32 * 148, 32 * 148 + 1) for k in (4096, 4104)])
def test_products_beside_the_lines_of_the_rule(m, k):
    """`linear` and `gated_linear` on both sides of every size and row count at which another form is chosen."""
    from inferrs_b200 import kernels as K
    x, w = rand((17, k), 1), rand((m, k), 2, 0.05)
    dot, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    for n in (1, 8, 9, 16, 17):
        for dtype in (torch.bfloat16, torch.float32):
            out = torch.full((n, m), float("nan"), dtype=dtype, device="cuda")
            if n <= 16:                                      # (more rows are the library's)
                K.linear(x[:n], w, out, torch.bfloat16)
                assert close(out, dot[:n], k * 2.0 ** -24 * size[:n])
        inner = m // 2
        out = torch.full((n, inner), float("nan"), dtype=torch.bfloat16, device="cuda")
        K.gated_linear(x[:n], w[:2 * inner], out, torch.bfloat16)
        g, u = dot[:n, :inner], dot[:n, inner:2 * inner]
        want = g / (1 + torch.exp(-g)) * u
        off = k * 2.0 ** -24 * size[:n]
        off_g, off_u = off[:, :inner], off[:, inner:2 * inner]
        # as above, and the gate's fast exponential and division of more rows (2^-20)
        slack = (2.0 ** -8 * 1.11 + 2.0 ** -20) * g.abs() * u.abs() + 2.0 ** -8 * 2.1 * want.abs() \
            + 1.2 * (off_g * u.abs() + off_u * g.abs() + off_g * off_u)
        assert bool(((out.double() - want).abs() <= slack).all())
    assert K.gemm_tcgen05_error() == 0
