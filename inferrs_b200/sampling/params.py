"""Per-request sampling options, with the reference's names, meanings and defaults
(inferrs/src/sampler.rs:27-112)."""
from __future__ import annotations

import sys
from array import array
from dataclasses import dataclass, field
from typing import Optional, Tuple

GREEDY_EPS = 1e-5  # temperatures below this pick the largest logit (sampler.rs:114, :176-179)


@dataclass
class SamplingParams:
    temperature: float = 0.7
    top_p: float = 0.9
    top_k: int = 50                      # 0: off
    repetition_penalty: float = 1.1      # 1.0: off; logit / p if >= 0 else logit * p, once per distinct token
    repeat_last_n: int = 64              # window of previous tokens the penalties look at; 0: off
    frequency_penalty: float = 0.0       # logit -= f * (times seen in the window)
    presence_penalty: float = 0.0        # logit -= q for tokens seen in the window
    min_p: float = 0.0                   # keep p >= min_p * p_max; 0: off
    max_tokens: int = 2048
    stop_token_ids: Tuple[int, ...] = ()  # the reference's extra_stop_token_ids
    seed: Optional[int] = None           # None: a fresh random seed per request
    ignore_eos: bool = False             # the reference's bypass_stop_tokens

    def __post_init__(self):
        if self.temperature < 0:
            raise ValueError(f"temperature must be >= 0, got {self.temperature}")
        if not 0.0 < self.top_p <= 1.0:
            raise ValueError(f"top_p must be in (0, 1], got {self.top_p}")
        if self.top_k < 0:
            raise ValueError(f"top_k must be >= 0, got {self.top_k}")
        if not 0.0 <= self.min_p <= 1.0:
            raise ValueError(f"min_p must be in [0, 1], got {self.min_p}")
        if self.max_tokens <= 0:
            raise ValueError(f"max_tokens must be positive, got {self.max_tokens}")
        if self.repeat_last_n < 0:
            raise ValueError(f"repeat_last_n must be >= 0, got {self.repeat_last_n}")
        self.stop_token_ids = tuple(int(t) for t in self.stop_token_ids)

    @classmethod
    def greedy(cls, max_tokens: int = 2048, **kw) -> "SamplingParams":
        """Largest logit, no penalties."""
        return cls(temperature=0.0, top_p=1.0, top_k=0, repetition_penalty=1.0, max_tokens=max_tokens, **kw)

    @property
    def is_greedy(self) -> bool:
        return self.temperature < GREEDY_EPS

    @property
    def has_penalty(self) -> bool:
        return self.repeat_last_n > 0 and (self.repetition_penalty not in (1.0, 0.0) or self.frequency_penalty != 0.0
                                           or self.presence_penalty != 0.0)


_M64 = (1 << 64) - 1


def _splitmix(x: int) -> int:
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & _M64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & _M64
    return x ^ (x >> 31)


def uniform_for(seed: int, step: int) -> float:
    """The random number in [0, 1) for a request's seed and ``step`` = number of tokens it holds so far
    (prompt and generated): the reference's stateless generator (sampler.rs:370-397).  Being a function
    of (seed, step) only, a request's draws do not depend on what else is in the batch."""
    x = _splitmix((int(seed) + 0x9E3779B97F4A7C15) & _M64)
    x = (x + ((int(step) + 1) * 0x9E3779B97F4A7C15)) & _M64
    x = _splitmix(x)
    if x == 0:
        x = 0x1234567890ABCDEF
    x ^= (x << 13) & _M64
    x ^= x >> 7
    x ^= (x << 17) & _M64
    u = ((x * 0x2545F4914F6CDD1D) & _M64) >> 32
    return u / 4294967296.0


def uniforms_for(seeds, steps):
    """:func:`uniform_for` for many (seed, step) pairs at once, with the same bits, in native code.  One seed or one step
    goes with every entry of the other list.  Returns float32 [n]."""
    import numpy as np

    from ..cache.manager import host_library

    a = seeds if hasattr(seeds, "__len__") else list(seeds)
    b = steps if hasattr(steps, "__len__") else list(steps)
    if len(a) != len(b):
        if len(a) != 1 and len(b) != 1:
            raise ValueError(f"{len(a)} seeds for {len(b)} steps")
        a, b = (list(a) * len(b), b) if len(a) == 1 else (a, list(b) * len(a))
    n = len(a)
    native = host_python() if n >= NATIVE_ROWS else None
    words = None if native is None else np.empty((2 * n,), dtype=np.uint64)
    at = 0 if native is None else words.__array_interface__["data"][0]
    if native is None or native.ibh_low_words(a, n, at) or native.ibh_low_words(b, n, at + 8 * n):
        words = array("Q", [int(x) & _M64 for x in a] + [int(x) & _M64 for x in b])
        at = words.buffer_info()[0]
    out = np.empty((n,), dtype=np.float32)
    host_library().ibh_uniforms(at, at + 8 * n, n, out.__array_interface__["data"][0])
    return out


_NATIVE = []
NATIVE_ROWS = 12     # rows from which the calls into native code cost less than they save (a call and its arrays: about 5 us)


def host_python():
    """The native functions that read Python's lists (csrc/host_python.cpp), or None where they cannot be built or loaded
    (tried once: every caller has a way without them)."""
    if not _NATIVE:
        import ctypes

        from ..csrc.build import LIBRARIES, BuildError, build_library

        lib = None
        if "host_python" in LIBRARIES:
            try:
                lib = ctypes.PyDLL(build_library("host_python"))       # (called with the interpreter's lock held)
            except (BuildError, OSError) as e:
                print(f"[inferrs_b200] without native code for Python's lists: {str(e).splitlines()[0]}", file=sys.stderr, flush=True)
        if lib is not None:
            i, p, o = ctypes.c_int, ctypes.c_void_p, ctypes.py_object
            lib.ibh_windows.argtypes, lib.ibh_windows.restype = [o, p, p, i, i, p, p], i
            lib.ibh_low_words.argtypes, lib.ibh_low_words.restype = [o, i, p], i
        _NATIVE.append(lib)
    return _NATIVE[0]
