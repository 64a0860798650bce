"""Which steps with prompt portions are replayed from a graph, and which graph goes when there are too many:
the runner's book-keeping, without a GPU."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from ginfer_b200.engine import StepEntry, runner as R


@pytest.fixture
def books(monkeypatch):
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    return SimpleNamespace(enforce_eager=False, _graphs={}, _short_seen={}, _portion_seen={}, device=None,
                           graph_batch=R.ModelRunner.graph_batch)


def step(books, lens, starts=None, want=1, width=4):
    """One step of whole prompts (or from ``starts``): "eager", "captured" or "replayed"."""
    entries = [StepEntry(f"r{i}", [1] * n, list(range(n))[-want:]) for i, n in enumerate(lens)]
    facts = dict(B=len(lens), T=sum(lens), q_lens=np.array(lens), q_starts=np.array(starts or [0] * len(lens)),
                 width=width, max_q_len=max(lens))
    key = R.ModelRunner._graph_key(books, entries, facts)
    if key is None:
        return "eager"
    if key in books._graphs:
        return "replayed"
    if key[0] == "short":
        R.ModelRunner._make_room(books, key)
    books._graphs[key] = object()
    return "captured"


def test_the_short_graph_replayed_longest_ago_is_given_up(books):
    """Forty lengths, each until it is captured: every one is, there are never too many, and those that are
    still replayed stay."""
    for n in range(8, 48):
        assert [step(books, [n]) for _ in range(5)] == ["eager"] * 3 + ["captured", "replayed"]
        assert step(books, [8]) == "replayed"
        assert len(books._graphs) == min(n - 7, R.PORTION_GRAPH_LIMIT)
    assert step(books, [47]) == step(books, [33]) == "replayed"
    assert [step(books, [9]) for _ in range(4)] == ["eager"] * 3 + ["captured"]      # given up: counted anew


def test_short_steps_are_whole_prompts_with_few_wanted_rows(books):
    for _ in range(6):
        assert step(books, [1, 17], [4089, 0]) == "eager"            # beside a decoding request
        assert step(books, [17], [100]) == "eager"                   # a prompt's later portion
        assert step(books, [17], want=R.PORTION_GRAPH_SHORT_ROWS + 1) == "eager"
        assert step(books, [17] * (R.PORTION_GRAPH_MAX_SEQS + 1)) == "eager"
    assert [step(books, [1, 17, 3], want=1) for _ in range(4)][-1] == "captured"


def test_short_shapes_do_not_wipe_what_is_known_of_long_portions(books):
    assert step(books, [300]) == "eager"
    for n in range(6000):
        step(books, [1 + n % 200, 1 + n // 200])
    assert len(books._short_seen) <= R.PORTION_GRAPH_SHAPES
    assert step(books, [300]) == "captured" and step(books, [300], [300]) == "replayed"
