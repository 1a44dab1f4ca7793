"""Which portions of a step the latent attention expands (seq_layers.LatentAttentionMixer): the portion alone decides."""
import random

import pytest
import torch

from lia_b200.seq_layers import LatentAttentionMixer


def mixer(window=0):
    m = object.__new__(LatentAttentionMixer)
    m.w_ukv, m.window = object(), window
    return m


@pytest.mark.parametrize("H", [1, 4, 16, 32])
@pytest.mark.parametrize("window", [0, 1024])
def test_the_company_does_not_count(H, window):
    m, rng, q = mixer(window), random.Random(H), torch.empty(1, 64, dtype=torch.bfloat16)
    for _ in range(50):
        portions = [(i, rng.choice((0, rng.randint(1, 3000), rng.randint(1, 100000))), 0, rng.choice((1, rng.randint(2, 80), rng.randint(64, 4000)))) for i in range(rng.randint(1, 40))]
        assert list(m._expands_exactly(q, portions, H)) == [i for i, p in enumerate(portions) if m._expands_exactly(q, [p], H)]


def test_few_rows_behind_a_long_history_stay_in_the_latent_space():
    m, q = mixer(), torch.empty(1, 64, dtype=torch.bfloat16)
    expands = lambda H, n, past: bool(m._expands_exactly(q, [(0, past, 0, n)], H))
    assert all(not expands(H, n, past) for H in (4, 8, 16) for n in (1, 15, 16, 24) for past in (2000, 8000, 30000))
    assert all(expands(H, n, past) for H in (4, 8, 16, 32) for n in (33, 64, 256, 2048) for past in (0, 300))
    assert all(expands(16, n, 8000) for n in (64, 100, 2048)) and not expands(16, 33, 30000)
    assert expands(32, 2048, 30000) and not expands(32, 64, 30000)          # groups of heads: enough blocks in each, or none at all
    w = mixer(512)
    assert w._expands_exactly(q, [(0, 100000, 0, 33)], 16)                  # what a window hides does not count
