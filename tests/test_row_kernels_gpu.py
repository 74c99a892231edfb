"""The forms of the row kernels that hold a row in registers (csrc/streams.cu), at the edges of their ranges."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed))


def near(got, want, terms=8):
    """``terms`` roundings of float32 of values up to the largest, and one of the output's type."""
    want = want.double()
    half = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -23
    slack = half * want.abs() + terms * 2.0 ** -23 * float(want.abs().max())
    return bool(((got.double().cpu() - want).abs() <= slack).all())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("streams,groups,width", [(1, 1, 128), (2, 4, 2048), (4, 2, 1024), (1, 3, 2688), (2, 1, 4096), (1, 8, 8192),
                                                  (4, 1, 8192), (2, 5, 640), (2, 2, 8320)])
def test_streams_update_and_norm(streams, groups, width, dtype):
    from inferrs_b200 import kernels as K
    n, eps = 5, 1e-5
    x, delta = rand((n, streams, width), 1), rand((n, width), 2).to(dtype)
    mix, gain, read = torch.eye(streams) + 0.3 * rand((streams, streams), 3), rand((streams,), 4), 0.5 + rand((streams,), 5).abs()
    weight = (1 + 0.2 * rand((width,), 6)).to(dtype)
    new = torch.einsum("st,nsw->ntw", mix.double(), x.double()) + gain.double()[None, :, None] * delta.double()[:, None, :]

    def normed(u):
        g = u.reshape(u.shape[0], groups, -1)
        return (g / (g.pow(2).mean(-1, keepdim=True) + eps).sqrt()).reshape(u.shape) * weight.double()

    res, out = x.cuda(), torch.empty((n, width), dtype=dtype, device="cuda")
    K.stream_add_norm(res, delta.cuda(), mix.cuda(), gain.cuda(), read.cuda(), weight.cuda(), groups, eps, out)
    assert near(res, new) and near(out, normed(torch.einsum("t,ntw->nw", read.double(), new)), 24)
    among = out
    rows, kept = torch.tensor([4, 0], dtype=torch.int32, device="cuda"), res.clone()
    out = torch.empty((2, width), dtype=dtype, device="cuda")
    K.stream_add_norm(res, None, None, None, None, weight.cuda(), groups, eps, out, rows)
    assert torch.equal(res, kept) and near(out, normed(new.sum(1)[[4, 0]]), 24)
    # one row alone has the bits of the row among others
    one, alone = x[2:3].cuda(), torch.empty((1, width), dtype=dtype, device="cuda")
    K.stream_add_norm(one, delta[2:3].cuda(), mix.cuda(), gain.cuda(), read.cuda(), weight.cuda(), groups, eps, alone)
    assert torch.equal(one[0], res[2]) and torch.equal(alone[0], among[2])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("e_dim", [4, 128, 132, 256, 260, 130])
@pytest.mark.parametrize("gate_act,normed,shared", [(0, True, True), (1, False, False), (0, True, False)])
def test_heads_normed_and_gated(e_dim, gate_act, normed, shared, dtype):
    from inferrs_b200 import kernels as K
    n, heads, eps = 7, 3, 1e-5
    for o_dtype in {torch.float32, dtype}:
        o, wide = rand((n, heads, e_dim), 7).to(o_dtype), rand((n, heads * e_dim + 8), 8).to(dtype)
        w = (1 + 0.2 * rand((e_dim if shared else heads * e_dim,), 9)).to(dtype)
        v = o.double()
        if normed:
            v = v / (v.pow(2).mean(-1, keepdim=True) + eps).sqrt()
        v = v * w.double().reshape((1, 1, -1) if shared else (1, heads, -1))
        for offset in (0, 3):                                # the second: rows that do not start on whole loads
            z = wide[:, offset:offset + heads * e_dim].double().reshape(n, heads, e_dim)
            want = (v * (torch.sigmoid(z) * (z if gate_act == 0 else 1))).reshape(n, -1)
            out = torch.empty((n, heads * e_dim), dtype=dtype, device="cuda")
            K.head_norm_gate(o.cuda(), wide.cuda()[:, offset:offset + heads * e_dim], w.cuda(), normed,
                             K.GATE_SILU if gate_act == 0 else K.GATE_SIGMOID, eps, out)
            assert near(out, want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,taps", [(128, 4), (516, 5), (2048, 6), (2052, 3), (4096, 4), (4096, 5), (4100, 2), (8192, 4)])
def test_kept_rows_of_the_norm_with_a_convolution(width, taps, dtype):
    """Taps below, at and beyond those that are fetched before the wait, in every number of groups a thread has: three layers
    a step, each on what the one before left, as a replayed graph with early starts, for three steps."""
    from inferrs_b200 import kernels as K
    n, layers, eps = 3, 3, 1e-5
    delta, weight = rand((layers, n, width), 1).to(dtype).cuda(), (1 + 0.2 * rand((layers, width), 2)).cuda()
    conv_w, start = 0.3 * rand((layers, taps, width), 3).cuda(), rand((n, width), 4).cuda()
    keep = (taps - 1) * width
    first = rand((n + 1, layers * keep), 5).cuda()
    slots, req = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in ([2, 0, 3], [1, 0, 2]))
    state, stream, out = first.clone(), torch.empty((n, width), device="cuda"), torch.empty((layers, n, width), dtype=dtype, device="cuda")

    def step():
        stream.copy_(start)
        for i in range(layers):
            K.sandwich_norm(stream, delta[i], None, 0.0, weight[i], eps, out[i], residual=stream,
                            conv=(conv_w[i], state, i * keep, slots, req))

    step()
    torch.cuda.synchronize()
    state.copy_(first)
    K.set_pdl(True, dtype)
    graph = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(graph):
            step()
    finally:
        K.set_pdl(False, dtype)
    at = [[2, 0, 3][r] for r in [1, 0, 2]]
    kept = first[at].double().cpu().reshape(n, layers, taps - 1, width)
    for _ in range(3):
        graph.replay()
        x = start.double().cpu()
        for i in range(layers):
            x = x + delta[i].double().cpu()
            want = x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt() * weight[i].double().cpu()
            h = state[at][:, i * keep:(i + 1) * keep].reshape(n, taps - 1, width)[:, -1].double().cpu()      # as it was rounded
            assert near(h.to(dtype), want, 24)
            w = conv_w[i].double().cpu()
            got = h * (1 + w[-1]) + (kept[:, i] * w[None, :-1]).sum(1)
            assert near(out[i], got, 24)
            kept[:, i] = torch.cat([kept[:, i, 1:], h[:, None]], 1)
    assert torch.equal(state[at].double().cpu().reshape(kept.shape), kept) and torch.equal(state[1], first[1])
