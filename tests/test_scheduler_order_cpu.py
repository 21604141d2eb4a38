"""Short portions of a step run first, and the logits come back in the order of the entries.  A stand-in for the model, no GPU."""
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
    m.slot_of = {1000: 0, 2000: 1, 3000: 2, 4000: 3, 5000: 4, 1500: 0, 2500: 1, 3500: 2, 4500: 3, 1600: 0}
    tok = lambda base, n: list(range(base, base + n))  # noqa: E731
    out = s.step([("a", tok(1000, 130), [129, 0]), ("b", tok(2000, 1), [0]), ("c", tok(3000, 300), []), ("d", tok(4000, 3), [0]), ("e", tok(5000, 64), [])])
    assert m.layouts[-1] == [(1, 0), (3, 0), (64, 0), (130, 0), (300, 0)]
    assert out.tolist() == [[1129, 129], [1000, 0], [2000, 0], [4000, 0]]
    out = s.step([("c", tok(3500, 127), [1]), ("b", tok(2500, 63), [0]), ("a", tok(1500, 1), [0]), ("d", tok(4500, 128), [0, 39])])
    assert m.layouts[-1] == [(63, 1), (1, 130), (127, 300), (128, 3)]                 # portions of one kind keep their order
    assert out.tolist() == [[3501, 301], [2500, 1], [1500, 130], [4500, 3], [4539, 42]]
    assert s.step([("a", [1600], [])]) is None
