"""Which form a recurrence takes, by the step's entries (no GPU)."""
from types import SimpleNamespace

from sparseengine_b200.csrc import ops
from sparseengine_b200.parts import recurrent


def test_choice(monkeypatch):
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)

    def takes(lens, heads=64, rows=128, columns=64, prepare=2e-4, least=16):
        step = SimpleNamespace(max_q_len=max(lens), num_tokens=sum(lens), num_seqs=len(lens))
        return recurrent.takes_chunks(SimpleNamespace(chunk_min_tokens=least), step, heads, rows, columns, prepare, "cuda:0")

    assert takes([2048]) and takes([128]) and takes([128] * 4) and takes([2048] + [1] * 8)
    assert not takes([1] * 64) and not takes([15]) and not takes([32]) and not takes([48] * 64) and not takes([64] * 16)
    assert not takes([2048], least=None) and not takes([2048], least=4096)
    delta = dict(heads=16, rows=128, columns=128, prepare=2.5e-3)
    assert takes([1500, 1037, 1323, 860], **delta) and not takes([64] * 64, **delta)
