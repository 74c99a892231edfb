"""Decode attention that hands its CTAs out longest request first (csrc/attention_decode.cu)."""
from __future__ import annotations

import random

import pytest
import torch

import kernel_refs as R
from helpers import rel_err
from test_kernels_gpu import _paged_setup, rand

pytestmark = pytest.mark.gpu


def cut_in_two(tiles, nkv, min_tiles=8, resident=296):
    """The requests beyond five quarters of a resident CTA's even share, if both halves have min_tiles; none where more than
    a wave of CTAs has three quarters of the longest one's tiles."""
    if sum(4 * t > 3 * max(tiles) for t in tiles) * nkv > resident:
        return [False] * len(tiles)
    return [4 * resident * t > 5 * sum(tiles) * nkv and t >= 2 * min_tiles for t in tiles]


@pytest.mark.parametrize("n,nkv,window", [(2, 2, None), (37, 8, None), (64, 8, 300), (255, 1, None), (256, 2, None)])
def test_ranked_requests_give_what_the_list_gives(n, nkv, window):
    """Lengths around the tiles' edges, equal ones and one far beyond the others (which is cut in two where that pays), alone
    and as a list of rows with gaps: the reference's values, and the unranked kernel's bits for every request that stays in one
    slice."""
    from inferrs_b200 import kernels as K
    rng = random.Random(n)
    lens = [rng.choice([1, 63, 64, 65, 128, rng.randint(1, 200)]) for _ in range(n)]
    lens[n // 2] = 1500
    table, positions, row_request, k_pages, v_pages = _paged_setup(torch.bfloat16, nkv, 128, 16, lens, [1] * n, 7)
    q = rand((n, 2 * nkv, 128), torch.bfloat16, 8)
    ref = torch.empty((n, 2 * nkv * 128), dtype=torch.bfloat16, device="cuda")
    R.paged_attention_generic(q, k_pages, v_pages, table, row_request, positions, 128 ** -0.5, window, ref)
    plain, out = torch.empty_like(ref), torch.full_like(ref, float("nan"))
    K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, window, plain, 1)
    for _ in range(2):                                   # twice: the counters are back at zero
        K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, window, out, 2, min_tiles=8, ranked=True)
        assert K.attention_decode_error() == 0
        assert rel_err(out, ref) < 2e-2
        others = torch.tensor([i for i in range(n) if i != n // 2], device="cuda")
        assert torch.equal(out[others], plain[others])
    rows = torch.tensor([i if i % 3 else -1 for i in range(n)], dtype=torch.int32, device="cuda")
    some = torch.full_like(ref, 7.0)
    K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, window, some, 2, rows, rows, min_tiles=8,
                             ranked=True)
    kept = torch.tensor([i for i in range(n) if i % 3], dtype=torch.long, device="cuda")
    left = torch.tensor([i for i in range(n) if i % 3 == 0], dtype=torch.long, device="cuda")
    assert bool((some[left] == 7.0).all()) and rel_err(some[kept], ref[kept]) < 2e-2


@pytest.mark.parametrize("lens,nkv", [
    ([513, 575, 576, 577, 700, 960, 961, 1023, 1024, 1025] + [40] * 54, 8),      # 9 to 17 tiles: from 16 on in two
    ([2048] * 27 + [1] * 37, 8),                    # nearly as many in two as there can be
    ([2048] * 37 + [1200] * 27, 8), ([2048] * 38 + [1200] * 26, 8), ([3000] * 38 + [1] * 26, 8),       # a wave of long ones, and one more
    ([4000] * 14 + [64] * 50, 8), ([1500] * 200 + [3] * 20, 1), ([300] * 64, 8), ([2000] * 64, 8), ([3, 2000], 1)])
def test_two_slices_are_for_long_requests_beyond_the_even_share_alone(lens, nkv):
    """Every request in one slice has the unranked kernel's bits with one slice, every other one those with two."""
    from inferrs_b200 import kernels as K
    n = len(lens)
    order = random.Random(5).sample(range(n), n)
    lens = [lens[i] for i in order]
    table, positions, row_request, k_pages, v_pages = _paged_setup(torch.bfloat16, nkv, 128, 16, lens, [1] * n, 7)
    q = rand((n, 2 * nkv, 128), torch.bfloat16, 8)
    one, two, out = (torch.full((n, 2 * nkv * 128), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, None, one, 1)
    K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, None, two, 2, min_tiles=8)
    K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, None, out, 2, min_tiles=8, ranked=True)
    assert K.attention_decode_error() == 0
    cut = torch.tensor(cut_in_two([(x + 63) // 64 for x in lens], nkv), device="cuda")
    assert torch.equal(out, torch.where(cut[:, None], two, one))
    K.paged_attention_decode(q, k_pages, v_pages, table, positions, 128 ** -0.5, None, out, 1, ranked=True)
    assert torch.equal(out, one)                    # no slices to choose from


def test_more_requests_than_are_ranked_are_refused_and_the_plan_keeps_to_the_list():
    from inferrs_b200 import kernels as K
    assert K.decode_plan(64, 8, 4096) == {"max_splits": 2, "min_tiles": 8, "ranked": True}
    assert K.decode_plan(8, 8, 4096) == {"max_splits": 4, "min_tiles": 4}
    assert K.decode_plan(75, 8, 4096) == K.decode_plan(257, 8, 4096) == {"max_splits": 1, "min_tiles": 4}
    # up to a wave and a half, and where no request has two slices' tiles, the list is as it was
    for n, keys in ((40, 200), (48, 256), (55, 4096), (56, 512), (64, 256), (64, 960)):
        assert K.decode_plan(n, 8, keys) == dict(zip(("max_splits", "min_tiles"), K.decode_slices(n, 8, keys)))
    assert K.decode_plan(56, 8, 961)["ranked"] and K.decode_plan(74, 8, 961)["ranked"]
    table, positions, _, k_pages, v_pages = _paged_setup(torch.bfloat16, 1, 128, 16, [3] * 257, [1] * 257, 9)
    q = rand((257, 1, 128), torch.bfloat16, 10)
    with pytest.raises(K.KernelError):
        K.paged_attention_decode(q, k_pages, v_pages, table, positions, 0.1, None, torch.empty((257, 128), dtype=torch.bfloat16,
                                                                                              device="cuda"), 2, ranked=True)
