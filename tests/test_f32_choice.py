"""Which kernel a step's 32-bit attention takes (no GPU)."""
from types import SimpleNamespace

import pytest
import torch

from sparseengine_b200.config.specs import AttentionSpec
from sparseengine_b200.csrc import ops
from sparseengine_b200.parts.base import make_mixer


@pytest.fixture(autouse=True)
def _sms(monkeypatch):
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)


def _takes(q_lens, held=0, heads=4, kv_heads=2, odd=None):
    part = make_mixer(AttentionSpec(hidden_size=64, num_heads=heads, num_kv_heads=kv_heads, head_dim=64, scale=0.125, position=None),
                      torch.float32)
    kv_lens = [held + n for n in q_lens]
    step = SimpleNamespace(num_tokens=sum(q_lens), num_seqs=len(q_lens), max_q_len=max(q_lens), max_kv_len=max(kv_lens), q_lens=q_lens,
                           kv_lens=kv_lens, q_starts=[held] * len(q_lens), max_kv_bound=None, extras={})
    t = {n: SimpleNamespace(dtype=torch.float32, device="cuda:0", data_ptr=lambda n=n: 4096 + 4 * (n == odd)) for n in ("q", "out", "kv")}
    return part.takes_f32_tiles(t["q"], t["out"], step, SimpleNamespace(kv=t["kv"]))


def test_addresses_and_grid():
    assert _takes([2048]) and not any(_takes([2048], odd=n) for n in ("q", "out", "kv"))
    # 65,535 tiles of 128 rows are the most
    most = 65535 * 128
    assert _takes([most // 64], heads=64, kv_heads=1) and not _takes([most // 64 + 1], heads=64, kv_heads=1)


@pytest.mark.parametrize("q_lens,held,heads,kv_heads,tiles", [
    # measured, a layer, us plain / tiles: 4,014 / 6,926, 2,355 / 6,282, 2,777 / 14,706, 9,511 / 7,154
    ([160] + [1] * 63, 4000, 16, 16, False), ([64] + [1] * 63, 4000, 16, 16, False), ([1] * 600, 1000, 16, 16, False),
    ([600] + [1] * 63, 4000, 16, 16, True),
    # 757 / 1,261, 5,567 / 1,421, 664 / 434, 119 / 124
    ([16], 4000, 48, 8, False), ([160], 4000, 48, 8, True), ([64], 1000, 48, 8, True), ([64], 0, 48, 8, False),
    # 5,048 / 1,331, 225 / 271, 9,910 / 1,408, 699 / 357
    ([1] * 600, 1000, 32, 1, True), ([1] * 600, 0, 32, 1, False), ([16] * 16, 4000, 48, 8, True), ([600], 0, 16, 16, True)])
def test_by_entries(q_lens, held, heads, kv_heads, tiles):
    assert _takes(q_lens, held, heads, kv_heads) is tiles


def test_windows_bound_the_keys():
    """600 single tokens of 1,000 keys pay with all keys in sight, with eight they do not."""
    lens = [1] * 600, [1001] * 600
    assert ops.attn_f32_tiles_pay(*lens, 32, 1, None, 148) and not ops.attn_f32_tiles_pay(*lens, 32, 1, 8, 148)
