"""Which kernel a step's latent attention takes, by its entries' own tokens and keys (no GPU)."""
from types import SimpleNamespace

import pytest

from sparseengine_b200.csrc import ops


def _takes(lens, held, window=None, heads=32, rank=192, rot=64):
    return ops.latent_takes_tc(len(lens), max(lens), heads, rank, rot, 148, q_lens=lens, kv_lens=[held + n for n in lens], window=window)


@pytest.mark.parametrize("lens,held,window,tc", [
    # a portion beside decoding requests, which tcgen05 would walk unsplit: measured 121 / 168, 625 / 1,012 and 905 / 1,015 us
    ([64, 1, 1, 1], 4000, None, False), ([64, 1, 1, 1], 30000, None, False), ([128, 1, 1, 1], 30000, None, False),
    ([8] + [1] * 31, 30000, None, False), ([8] + [1] * 31, 4000, None, False),
    # small steps wait for the host, which the tiled kernel takes longer: a call 168 / 153, 157 / 152, 162 / 151, 167 / 153
    ([64, 1, 1, 1], 4000, 1024, True), ([64, 1, 1, 1], 0, None, True), ([8] + [1] * 31, 0, None, True), ([64], 500, None, True),
    # where the tiled kernel does not split either: 296 / 195, 1,765 / 1,058, 254 / 178
    ([512] + [1] * 7, 4000, None, True), ([512] + [1] * 7, 30000, None, True), ([32] + [1] * 63, 4000, None, True),
    ([512] + [1] * 7, 4000, 1024, True),
    # portions alone: 207 / 174, 123 / 166, 1,195 / 411
    ([256], 4000, None, True), ([128], 4000, None, False), ([2048], 4000, None, True), ([64] * 16, 4000, None, True),
    ([1] * 64, 4000, None, False)])
def test_by_entries(lens, held, window, tc):
    assert _takes(lens, held, window) is tc


def test_asked_once_per_step():
    from sparseengine_b200.config.specs import LatentAttentionSpec
    from sparseengine_b200.parts.base import make_mixer
    import torch
    part = make_mixer(LatentAttentionSpec(hidden_size=64, num_heads=32, head_dim=16, rot_dim=64, v_head_dim=16, q_rank=16, kv_rank=192,
                                          scale=0.1, position=None), torch.bfloat16)
    asked = []
    before, count = ops.latent_takes_tc, ops.sm_count
    ops.latent_takes_tc, ops.sm_count = lambda *a, **k: asked.append(k["kv_lens"]) or True, lambda device=None: 148
    try:
        step = SimpleNamespace(num_seqs=2, max_q_len=5, q_lens=[5, 1], kv_lens=[9, 1], max_kv_bound=None, extras={})
        assert part.takes_tc(step, "cuda:0") and part.takes_tc(step, "cuda:0") and asked == [[9, 1]]
        step = SimpleNamespace(num_seqs=2, max_q_len=1, q_lens=[1, 1], kv_lens=[9, 1], max_kv_bound=64, extras={})
        assert part.takes_tc(step, "cuda:0") and asked[1] == [64, 64]
    finally:
        ops.latent_takes_tc, ops.sm_count = before, count


def test_captured_steps_stay_in_the_latent_space(monkeypatch):
    """Keys per head take a workspace for the lengths that the host knows, a replayed graph may meet others: also where the same step has
    run before."""
    from sparseengine_b200.config.specs import LatentAttentionSpec
    from sparseengine_b200.parts.base import make_mixer
    import torch
    part = make_mixer(LatentAttentionSpec(hidden_size=64, num_heads=32, head_dim=64, rot_dim=64, v_head_dim=64, q_rank=16, kv_rank=192,
                                          scale=0.1, position=None), torch.bfloat16)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    step = SimpleNamespace(num_seqs=1, max_q_len=2048, q_lens=[2048], kv_lens=[2500], max_kv_bound=None, extras={})
    assert part.takes_heads(step, "cuda:0") == (2500, 2500)
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert part.takes_heads(step, "cuda:0") is None
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert part.takes_heads(step, "cuda:0") == (2500, 2500)
