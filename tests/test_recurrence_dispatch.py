"""The host side of the recurrences: what a step asks for, without a GPU."""
import threading
from types import SimpleNamespace

import torch

from ginfer_b200.ops import decay


class Meeting:
    """Threads that ask for the same thing go on together, until the meeting is over."""

    def __init__(self, threads):
        self.barrier, self.over = threading.Barrier(threads), False

    def wait(self):
        if not self.over:
            self.barrier.wait(timeout=5)


class FakeLibrary:
    def __init__(self, meeting):
        self.meeting = meeting
        self.gf_decay_chunk_words = lambda chunks, H, G, D, Vd: chunks * H * D * Vd

    def gf_decay_chunk_tokens(self):
        self.meeting.wait()
        return 64


class Lengths(list):
    """Portion lengths that are read when both threads have got that far."""
    meeting = None

    def __getitem__(self, what):
        if isinstance(what, slice):
            self.meeting.wait()
        return list.__getitem__(self, what)


def test_two_threads_may_ask_for_the_first_chunked_recurrence_at_once(monkeypatch):
    """What the process keeps of the library is the same whichever thread is first, and one more call works."""
    meeting, calls, done = Meeting(2), [], []
    lib = FakeLibrary(meeting)
    monkeypatch.setattr(decay, "load_library", lambda name: lib)
    monkeypatch.setattr(decay, "_fn", lambda *a, **k: lambda *args: calls.append(args) or 0)
    monkeypatch.setattr(decay, "_p", lambda t: t)
    monkeypatch.setattr(decay, "_stream", lambda: 0)
    H, D, Vd, lens = 2, 4, 8, Lengths([65, 200])
    lens.meeting = meeting
    T = sum(lens)
    q, v, g, state = torch.zeros(T, H * D), torch.zeros(T, H * Vd), torch.zeros(T, H), torch.zeros(2, H * D * Vd)
    ctx = SimpleNamespace(num_seqs=2, q_lens_host=lens, cu_seqlens_q=torch.zeros(3), slot_ids=torch.zeros(2))

    def run():
        done.append(decay._chunked(q, q, v, g, state, ctx, 0, H, H, D, Vd, None, None, None, v, None))
    both = [threading.Thread(target=run) for _ in range(2)]
    for t in both:
        t.start()
    for t in both:
        t.join()
    meeting.over = True
    run()
    assert done == [True] * 3 and len(calls) == 3
    for args in calls:                               # 2 + 4 chunks, and their scratch
        assert any(isinstance(a, int) and a == 6 for a in args)
        assert any(torch.is_tensor(a) and a.numel() == 6 * 2 * 4 * 8 for a in args)
