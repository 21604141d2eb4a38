"""Entries of a step run shortest first, and the logits come back in the order of the entries.  A stand-in for the model, no GPU."""
import torch

from krasis_b200 import scheduler


class _Kv:
    def __init__(self, *a, **k):
        self.seq_len, self.pages = 0, []

    def ensure_capacity(self, n):
        self.pages = list(range((self.seq_len + n + 3) // 4))

    def advance(self, n):
        self.seq_len += n

    def free(self):
        pass


class _Model:
    device = torch.device("cpu")

    def __init__(self):
        self.layouts = []

    def make_caches(self, max_tokens, max_requests):
        free = list(range(max_requests))
        return None, type("P", (), {"alloc": lambda s: free.pop(0), "free": lambda s, i: free.append(i), "tensors": []})()

    def forward_step(self, tb, rows):
        self.layouts.append([(n, start) for _, n, start, _ in tb.layout])
        assert [int(v) for v in tb.slots] == [self.slot_of[int(tb.tokens[r])] for r, *_ in tb.layout]
        return None if rows is None else torch.stack([tb.tokens, tb.positions], 1).index_select(0, rows)


def test_mixed_entries(monkeypatch):
    monkeypatch.setattr(scheduler, "SequenceKVState", _Kv)
    m = _Model()
    s = scheduler.Scheduler(m, 1000, 8)
    m.slot_of = {100: 0, 200: 1, 300: 2, 400: 3, 150: 0, 250: 1, 350: 2, 450: 3, 151: 0}
    tok = lambda base, n: list(range(base, base + n))  # noqa: E731
    out = s.step([("a", tok(100, 9), [8, 0]), ("b", tok(200, 1), [0]), ("c", tok(300, 30), []), ("d", tok(400, 1), [0])])
    assert m.layouts[-1] == [(1, 0), (1, 0), (9, 0), (30, 0)]
    assert out.tolist() == [[108, 8], [100, 0], [200, 0], [400, 0]]
    out = s.step([("c", tok(350, 2), [1]), ("b", tok(250, 1), [0]), ("a", tok(150, 1), [0]), ("d", tok(450, 40), [0, 39])])
    assert m.layouts[-1] == [(1, 1), (1, 9), (2, 30), (40, 1)]                       # equal lengths keep their order
    assert out.tolist() == [[351, 31], [250, 1], [150, 9], [450, 1], [489, 40]]
    assert s.step([("a", [151], [])]) is None
