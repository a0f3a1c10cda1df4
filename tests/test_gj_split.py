"""The resident inversion's choice of launches (host only): one look at what every panel count holds gives what
trying one launch, then two, and so on did, each with every panel count again."""
import random

import pytest


def _by_trial(count, slots):
    parts, chunk = 1, count
    while True:
        for i, s in enumerate(slots):
            if chunk <= s:
                return i + 1, chunk
        if chunk == 1:
            return 0, 0
        parts += 1
        chunk = (count + parts - 1) // parts


@pytest.mark.parametrize("seed", range(4))
def test_split_is_what_trials_find(seed):
    from robinsolver_b200 import _lib
    rng = random.Random(seed)
    for _ in range(500):
        n = rng.randint(1, 28)
        slots = [rng.choice([0, 0, rng.randint(1, 8), rng.randint(1, 600)]) for _ in range(n)]
        if rng.random() < 0.5:
            slots.sort()
        count = rng.choice([1, 2, 3, rng.randint(1, 50), rng.randint(1, 4096)])
        chunk = _lib.C.c_int(0)
        ppc = _lib.lib.rb_test_gj_split(count, (_lib.C.c_int * n)(*slots), n, _lib.C.byref(chunk))
        want = _by_trial(count, slots)
        assert (ppc, chunk.value if ppc else 0) == want, (count, slots)
