"""Which kernels take a step's portions of prompts (ops.window_prompt_form, csrc/window_attn_mma.cu; on 148 SMs): what decides, and that the step's short way to the answer gives the same."""
import random

import pytest

from lia_b200 import ops

TCGEN05, MMA_SYNC, BOTH = 2, 3, 4


def portions_of(spec):
    out, row = [], 0
    for i, (past, n) in enumerate(spec):
        out.append((i, past, row, n))
        row += n
    return out, row


def form(spec, H=16, window=0, chunk=0, gated=False):
    p, rows = portions_of(spec)
    return ops.window_prompt_form(p, len(p), rows, H, window, chunk, gated)


def test_few_rows_and_long_histories():
    assert form([(0, 2)]) == form([(0, 33)]) == form([(0, 40)] * 32) == form([(0, 16)] * 64, 32) == MMA_SYNC
    assert form([(256, 2)]) == form([(0, 2048)]) == form([(2000, 1)] * 31 + [(0, 200)]) == form([(500, 64)] * 32) == form([(0, 128)] * 16) == TCGEN05
    assert form([(0, 40)] * 8) == MMA_SYNC and form([(0, 40)] * 8, gated=True) == TCGEN05
    assert form([(2000, 40)] * 32) == TCGEN05 and form([(2000, 40)] * 32, window=8) == MMA_SYNC and form([(2000, 40)] * 32, chunk=64) == MMA_SYNC        # what is hidden does not count
    both = form([(0, 200)] + [(30, 1)] * 62 + [(0, 130)])
    assert both & 7 == BOTH and both >> 3 & 16383 == 4 and both >> 17 == 62              # tiles of 128 rows of the long portions, of 64 of the short ones


@pytest.mark.parametrize("seed", range(4))
def test_long_portions_are_never_mma_syncs(seed):
    rng = random.Random(seed)
    for _ in range(300):
        spec = [(rng.choice((0, rng.randint(1, 2000))), rng.choice((rng.randint(1, 16), rng.randint(17, 128), rng.randint(129, 600)))) for _ in range(rng.randint(1, 40))]
        f = form(spec, rng.choice((1, 8, 32)), rng.choice((0, 64, 1024)), rng.choice((0, 0, 100)), rng.random() < 0.5)
        long = [n for _, n in spec if n > 128]
        assert f in (TCGEN05, MMA_SYNC) or (f & 7 == BOTH and long and f >> 3 & 16383 == sum(-(-n // 128) for n in long) and f >> 17 == sum(-(-n // 64) for _, n in spec if n <= 128))
        assert not (long and f == MMA_SYNC)


@pytest.mark.parametrize("seed", range(4))
def test_the_steps_short_way_is_the_same(seed):
    rng, short = random.Random(100 + seed), 0
    for _ in range(500):
        past, most = rng.choice((0, 10, 200)), rng.choice((20, 60, 300))
        spec = [(rng.randint(0, past), rng.choice((rng.randint(1, 40), rng.randint(1, 128), rng.randint(129, 300))) % most + 1) for _ in range(rng.randint(1, 18))]
        p, rows = portions_of(spec)
        lengths, ctx = (min(n for _, n in spec), max(n for _, n in spec)), max(a + n for a, n in spec)
        H, window, chunk, gated = rng.choice((1, 4, 8, 16, 32)), rng.choice((0, 64, 97, 1024)), rng.choice((0, 0, 50)), rng.random() < 0.5
        whole = ops.window_prompt_form(p, len(p), rows, H, window, chunk, gated)
        assert ops.window_step_form(p, lengths, rows, ctx, H, window, chunk, gated, 148) == whole, (spec, H, window, chunk, gated)
        short += ops.window_step_form(p, lengths, rows, ctx, H, window, chunk, gated, 0) != whole
    assert short == 0                                                # (without the shortcut for few tiles)


def test_portions_that_the_host_does_not_know():
    assert ops.window_prompt_form(None, 64, 64 * 16, 32, 0) == ops.window_prompt_form(None, 32, 32 * 128, 32, 0) == MMA_SYNC
    assert ops.window_prompt_form(None, 1, 5, 32, 0) == ops.window_prompt_form(None, 6, 751, 8, 0) == ops.window_prompt_form(None, 4, 4 * 300, 32, 0) == TCGEN05
