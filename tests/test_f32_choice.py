"""Which kernel a step's 32-bit attention takes (no GPU)."""
from types import SimpleNamespace

import torch

from sparseengine_b200.config.specs import AttentionSpec
from sparseengine_b200.parts.base import make_mixer


def _takes(q_lens, held=0, heads=4, kv_heads=2, odd=None):
    part = make_mixer(AttentionSpec(hidden_size=64, num_heads=heads, num_kv_heads=kv_heads, head_dim=64, scale=0.125, position=None),
                      torch.float32)
    kv_lens = [held + n for n in q_lens]
    step = SimpleNamespace(num_tokens=sum(q_lens), num_seqs=len(q_lens), max_q_len=max(q_lens), max_kv_len=max(kv_lens), q_lens=q_lens,
                           kv_lens=kv_lens, q_starts=[held] * len(q_lens))
    t = {n: SimpleNamespace(dtype=torch.float32, device="cuda:0", data_ptr=lambda n=n: 4096 + 4 * (n == odd)) for n in ("q", "out", "kv")}
    return part.takes_f32_tiles(t["q"], t["out"], step, SimpleNamespace(kv=t["kv"]))


def test_addresses_and_grid():
    assert _takes([600]) and not any(_takes([600], odd=n) for n in ("q", "out", "kv"))
    # 65,535 tiles of 128 rows are the most
    most = 65535 * 128
    assert _takes([most // 64], heads=64, kv_heads=1) and not _takes([most // 64 + 1], heads=64, kv_heads=1)
