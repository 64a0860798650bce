"""Which tokens of a latent-attention step may share tiles of keys (on the host)."""
from types import SimpleNamespace

import pytest

from ginfer_b200.ops import latent


@pytest.mark.parametrize("window, portions, tokens", [
    (1024, [(0, 1000)], 1000), (1024, [(0, 2000)], 1024), (1024, [(900, 1100)], 124), (1024, [(1024, 1000)], 0),
    (1024, [(500, 1)] * 3 + [(600, 700), (1500, 200)], 3 + 424), (0, [(3000, 1000)], 1000), (512, [(100, 2000)], 0),
    (512, [(0, 600), (400, 1)], 513)])
def test_the_tokens_that_may_share_keys_are_those_whose_window_reaches_back_to_the_first(window, portions, tokens):
    T, keys = sum(n for _, n in portions), max(a + n for a, n in portions)
    ctx = SimpleNamespace(q_starts_host=[a for a, _ in portions], q_lens_host=[n for _, n in portions])
    assert latent.sharing_tokens(ctx, T, window, keys) == tokens
    for a, n in portions if len(portions) == 1 and keys <= 2 * window else ():   # one by one
        assert tokens == sum(p - window + 1 <= 0 for p in range(a, a + n))
    assert latent.sharing_tokens(SimpleNamespace(), T, window, keys) == (0 if 0 < 2 * window < keys else T)
