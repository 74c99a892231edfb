"""Generation through the Python entry point on the CPU (plain kernel statements in the kernels' place)
against a plain loop: forward the whole sequence, pick the next token, append."""
import pytest
import torch

import kernel_refs
import plain_qwen3
import plain_sampler
from helpers import CONFIG_A, CONFIG_B, PAGE_SIZE, random_tokens
from inferrs_b200.engine.engine import Engine
from inferrs_b200.runtime import Runtime
from inferrs_b200.sampling.params import SamplingParams, uniform_for


def plain_generate(model_dir, prompt, n, **sampling):
    cfg, w = plain_qwen3.read_model(model_dir)
    toks = list(prompt)
    for _ in range(n):
        logits = plain_qwen3.forward(cfg, w, toks)[-1]
        toks.append(plain_sampler.sample_token(logits.numpy(), toks, **sampling))
    return toks[len(prompt):]


def cpu_engine(model_dir, name, **kw):
    return Engine(model_dir, block_size=PAGE_SIZE[name], runtime=Runtime(torch.device("cpu"), torch.float32), **kw)


def test_uniform_matches_the_plain_generator():
    for seed, step in [(0, 0), (4, 17), (2 ** 63 - 1, 5000), (123456789, 1)]:
        assert abs(uniform_for(seed, step) - float(plain_sampler.rand_f32(seed, step))) < 1e-7


def test_uniforms_of_many_rows_have_the_same_bits():
    import numpy as np
    from inferrs_b200.sampling.params import uniforms_for
    seeds = [0, 4, 2 ** 63 - 1, 2 ** 64 - 1, 2 ** 70 + 5, -1, -12345] + random_tokens(50, 10 ** 9, seed=3)
    steps = [0, 17, 5000, 1, 2 ** 31, 7, 0] + random_tokens(50, 10 ** 5, seed=4)
    want = np.array([uniform_for(a, b) for a, b in zip(seeds, steps)], dtype=np.float32)
    assert np.array_equal(uniforms_for(seeds, steps), want) and uniforms_for([], []).shape == (0,)


def _sampler_words(monkeypatch, params, seeds, histories, rows):
    """What a sampling call hands to its kernels: (temperatures, uniforms, windows)."""
    from inferrs_b200 import kernels
    from inferrs_b200.sampling.sampler import Sampler
    got = {"windows": []}
    monkeypatch.setattr(kernels, "sample", lambda l, t, k, p, m, u, out, act, **kw: got.update(t=t.tolist(), u=u.tolist()))
    monkeypatch.setattr(kernels, "penalties", lambda l, prev, n, *rest: got.update(
        windows=[sorted(row[:k]) for row, k in zip(prev.tolist(), n.tolist())]))
    Sampler(torch.device("cpu")).sample(torch.zeros(rows, 9), params, seeds, histories)
    return got["t"], got["u"], got["windows"]


def test_sampling_with_lists_of_other_lengths(monkeypatch):
    """One options object, seed or history counts for every row; any other length that is not the rows' is refused."""
    import numpy as np
    plain, window = SamplingParams(repetition_penalty=1.0), SamplingParams(repeat_last_n=3)
    u = lambda seed, step: float(np.float32(uniform_for(seed, step)))   # noqa: E731
    assert _sampler_words(monkeypatch, [plain] * 2, [4], [[1], [1, 2]], 2)[1] == [u(4, 1), u(4, 2)]
    assert _sampler_words(monkeypatch, [plain] * 3, [1, 2, 3], [[1, 2]], 3)[1] == [u(1, 2), u(2, 2), u(3, 2)]
    t, got, _ = _sampler_words(monkeypatch, [plain], [7, 8], [[1], [2]], 2)
    assert t == [t[0]] * 2 and got == [u(7, 1), u(8, 1)]
    # windows: of the rows with an options object and a history of their own; histories beyond the rows are not looked at
    assert _sampler_words(monkeypatch, [window], [1] * 3, [[1, 2, 3, 4]] * 3, 3)[2] == [[2, 3, 4], [], []]
    assert _sampler_words(monkeypatch, [window] * 3, [1] * 3, [[5]], 3)[2] == [[5], [], []]
    assert _sampler_words(monkeypatch, [window] * 2, [1] * 2, [[1], [2], [3]], 2)[2] == [[1], [2]]
    for params, seeds, histories in (([plain] * 4, [4, 5, 6], [[1]] * 5), ([plain] * 2, [1] * 4, [[1]] * 4),
                                     ([window] * 5, [1] * 4, [[1]] * 4), ([plain] * 4, [1] * 4, [[1]] * 3),
                                     ([plain] * 4, [], [[1]] * 4), ([plain] * 4, [1, 2], [[1]])):
        with pytest.raises(ValueError):
            _sampler_words(monkeypatch, params, seeds, histories, 4)


def test_options_shared_by_rows_or_not(monkeypatch):
    """Rows that share options objects in part, altogether or not at all hand over the same numbers."""
    from dataclasses import replace
    a, b, c = SamplingParams(top_k=3), SamplingParams.greedy(), SamplingParams(temperature=0.3, repeat_last_n=2)
    seeds, histories = [1, 2, 3, 4], [[1, 2, 3], [4], [5, 6, 7], [8, 9]]
    for params in ([a, b, a, c], [c, c, c, c], [b, a, c, SamplingParams(repeat_last_n=0)]):
        assert _sampler_words(monkeypatch, params, seeds, histories, 4) == \
            _sampler_words(monkeypatch, [replace(p) for p in params], seeds, histories, 4)


def test_windows_from_histories_of_every_kind(monkeypatch):
    import numpy as np
    for history in ([4, 6], (4, 6), torch.tensor([4, 6]), np.array([4, 6]), [4.0, 6.0], np.array([4.0, 6.0]),
                    torch.tensor([4.0, 6.0]), range(4, 8, 2)):
        words = _sampler_words(monkeypatch, [SamplingParams()] * 2, [1, 2], [history, [1]], 2)
        assert words[2] == [[4, 6], [1]]


@pytest.mark.parametrize("name", ["A", "B"])
def test_greedy_generation(model_dirs, monkeypatch, name):
    kernel_refs.install(monkeypatch)
    cfg = CONFIG_A if name == "A" else CONFIG_B
    prompts = [random_tokens(n, cfg["vocab_size"], seed=40 + n) for n in (5, 17, 33)]
    eng = cpu_engine(model_dirs[name], name, num_blocks=64, max_batch_size=4, max_tokens_per_step=24)
    got = eng.generate(prompts, SamplingParams.greedy(max_tokens=8))
    for p, g in zip(prompts, got):
        assert g == plain_generate(model_dirs[name], p, 8, temperature=0.0, repetition_penalty=1.0)
    assert eng.stats()["free_pages"] == eng.stats()["pages"]


def test_sampled_generation_matches_the_plain_sampler(model_dirs, monkeypatch):
    kernel_refs.install(monkeypatch)
    name, cfg = "B", CONFIG_B
    prompts = [random_tokens(n, cfg["vocab_size"], seed=50 + n) for n in (1, 9, 40)]
    opts = dict(temperature=0.8, top_k=20, top_p=0.95, repetition_penalty=1.1, repeat_last_n=16,
                frequency_penalty=0.2, presence_penalty=0.1, min_p=0.01)
    eng = cpu_engine(model_dirs[name], name, num_blocks=32, max_batch_size=4, max_tokens_per_step=7)
    got = eng.generate(prompts, SamplingParams(max_tokens=10, seed=4, **opts))
    for p, g in zip(prompts, got):
        assert g == plain_generate(model_dirs[name], p, 10, seed=4, **opts)


def test_preemption_gives_the_same_tokens(model_dirs, monkeypatch):
    kernel_refs.install(monkeypatch)
    name, cfg = "A", CONFIG_A
    prompts = [random_tokens(n, cfg["vocab_size"], seed=60 + n) for n in (9, 14, 11)]
    sp = SamplingParams(temperature=0.9, top_k=0, top_p=1.0, repetition_penalty=1.0, max_tokens=14, seed=7)
    roomy = cpu_engine(model_dirs[name], name, num_blocks=64, max_batch_size=4)
    want = roomy.generate(prompts, sp)
    tight = cpu_engine(model_dirs[name], name, num_blocks=14, max_batch_size=4)   # 14 pages of 4 tokens
    got = tight.generate(prompts, sp)
    assert tight.stats()["preemptions"] > 0
    assert got == want
