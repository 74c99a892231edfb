"""The penalties' windows and the seeds as native code reads them out of Python's lists (csrc/host_python.cpp)."""
from __future__ import annotations

import random

import numpy as np
import pytest

from inferrs_b200.csrc import build
from inferrs_b200.sampling import params
from inferrs_b200.sampling.params import host_python, uniform_for, uniforms_for
from inferrs_b200.sampling.sampler import Sampler


class Request:
    def __init__(self, tokens):
        self.tokens, self.n_tokens = tokens, len(tokens)

    def tail(self, n):
        return self.tokens[-n:]


def plain(last, histories, pend, width):
    rows, counts = [], []
    for k, h, x in zip(last, histories, pend):
        t = list(h.tokens if isinstance(h, Request) else h)
        row = ([-1] if x and k else []) + (t[-(k - x):] if k > x else [])
        counts.append(len(row))
        rows.append(row + [-1] * (width - len(row)))
    return rows, counts


@pytest.mark.skipif(host_python() is None, reason="the interpreter's headers are not installed")
@pytest.mark.parametrize("rows,longest", [(1, 0), (1, 1), (3, 5), (64, 100)])
def test_windows_are_those_of_the_lists(rows, longest):
    rng = random.Random(rows * 1000 + longest)
    for objects in (False, True):
        histories = [[rng.randrange(-2 ** 31, 2 ** 31) for _ in range(rng.randint(0, longest))] for _ in range(rows)]
        last, pend = [rng.choice([0, 1, 2, 64]) for _ in range(rows)], [rng.randint(0, 1) for _ in range(rows)]
        if objects:
            histories = [Request(h) if rng.random() < 0.5 else h for h in histories]
        lengths = [h.n_tokens if isinstance(h, Request) else len(h) for h in histories]
        width = max(1, max(min(k, n + x) for k, n, x in zip(last, lengths, pend)))
        words, counts = np.empty(rows * width, dtype=np.int32), np.empty(rows, dtype=np.int32)
        assert Sampler._windows_natively(last, histories, pend, width, words, counts)
        want, n = plain(last, histories, pend, width)
        assert words.reshape(rows, width).tolist() == want and counts.tolist() == n


@pytest.mark.parametrize("history", [(1, 2, 3), [1, 2.0, 3], [1, 2 ** 31, 3], [1, np.int64(2), 3], [True, 2, 3]])
def test_what_is_no_list_of_integers_is_left_to_the_general_way(history):
    words, counts = np.empty(4, dtype=np.int32), np.empty(1, dtype=np.int32)
    assert not Sampler._windows_natively([4], [history], [0], 4, words, counts)
    assert not Sampler._windows_natively([4.0], [[1, 2]], [0], 4, words, counts)
    assert not Sampler._windows_natively([2 ** 40], [[1, 2]], [0], 4, words, counts)
    assert not Sampler._windows_natively([4, 4], [[1, 2]] * 2, [0, 0], 4, words, counts)


@pytest.mark.parametrize("copies", [1, 3])
def test_seeds_of_every_kind_give_the_bits_of_the_plain_generator(copies):
    seeds, steps = [0, 1, -5, 2 ** 63 + 7, 2 ** 70 + 1] * copies, [3, 0, 2 ** 40, 7, 1] * copies
    want = [float(np.float32(uniform_for(a, b))) for a, b in zip(seeds, steps)]
    assert uniforms_for(seeds, steps).tolist() == want
    assert uniforms_for(tuple(seeds), np.array(steps)).tolist() == want
    assert uniforms_for([9], steps).tolist() == uniforms_for([9] * 5 * copies, steps).tolist()
    with pytest.raises(ValueError):
        uniforms_for([1, 2], steps)
    assert uniforms_for((s for s in seeds), iter(steps)).tolist() == want


@pytest.mark.parametrize("error", [build.BuildError("no compiler"), OSError("cannot be loaded")])
def test_without_the_native_functions_everything_goes_the_general_way(monkeypatch, error):
    """A library that cannot be built is asked for once, when a sampler is made, and no step fails for it."""
    asked = []

    def refuse(name):
        asked.append(name)
        raise error

    monkeypatch.setitem(build.LIBRARIES, "host_python", {})
    monkeypatch.setattr(build, "build_library", refuse)
    monkeypatch.setattr(params, "_NATIVE", [])
    torch = pytest.importorskip("torch")
    Sampler(torch.device("cpu"))
    assert asked == ["host_python"] and host_python() is None
    seeds, steps = list(range(20)), list(range(20, 40))
    assert uniforms_for(seeds, steps).tolist() == [float(np.float32(uniform_for(a, b))) for a, b in zip(seeds, steps)]
    words, counts = np.empty(4, dtype=np.int32), np.empty(1, dtype=np.int32)
    assert not Sampler._windows_natively([4], [[1, 2, 3, 4]], [0], 4, words, counts)
    assert asked == ["host_python"]
