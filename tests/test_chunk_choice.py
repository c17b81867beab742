"""Which form a recurrence takes, by the step's entries (no GPU)."""
from types import SimpleNamespace

import pytest

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


@pytest.mark.parametrize("lens,state_space,channel,head", [
    # short pieces beside a portion, a layer, us token by token / in chunks: 188/588, 244/367, 234/403; 594/752, 791/546, 753/577;
    # 360/422, 425/324, 415/338; 614/1,194, 512/720, 504/814
    ([300] + [1] * 31, False, False, False), ([1024] + [1] * 31, False, True, True), ([600] + [1] * 15, False, True, True),
    ([500] + [1] * 63, False, False, False), ([200] + [1] * 15, False, False, False), ([130] + [1] * 3, False, True, True),
    ([300] + [1] * 7, False, True, True), ([2048] + [1] * 31, True, True, True),
    # alone and side by side: 86/66, 109/64, 100/62; 238/195, 180/164, 177/152; 2,096/1,886, 1,335/1,457, 1,350/1,391
    ([128], True, True, True), ([192] * 4, True, True, True), ([128] * 64, True, False, False), ([64] * 64, False, False, False)])
def test_by_the_entries_own_tokens(monkeypatch, lens, state_space, channel, head):
    import torch

    from sparseengine_b200.config.specs import GatedDeltaSpec, StateSpaceSpec
    from sparseengine_b200.parts.base import make_mixer
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    step = SimpleNamespace(max_q_len=max(lens), num_tokens=sum(lens), num_seqs=len(lens), q_lens=lens)
    delta = dict(hidden_size=64, num_heads=16, num_kv_heads=16, head_dim=128, v_head_dim=128, conv_taps=4)
    specs = [StateSpaceSpec(hidden_size=64, num_heads=64, head_dim=64, state_size=128, groups=8, conv_taps=4, norm_groups=8),
             GatedDeltaSpec(**delta, decay_per="channel", gate_activation="sigmoid", decay_rank=8, gate_rank=8),
             GatedDeltaSpec(**delta, decay_per="head", gate_activation="silu")]
    assert [make_mixer(s, torch.bfloat16).in_chunks(step, "cuda:0") for s in specs] == [state_space, channel, head]


@pytest.mark.parametrize("lens,sixteen,thirty_two", [
    # a layer, us chunk at a time / walk, 16 and 32 heads: 434/491, 857/983; 484/516, 930/1,022; 631/575, 1,139/1,128; 286/301 at 32
    ([90] + [1] * 63, False, False), ([150, 150] + [1] * 62, False, False), ([600] + [1] * 63, True, True), ([90] + [1] * 15, True, False),
    # 1,045/914, 2,368/2,099; 300/260, 682/614; one chunk: 92/76 alone and 118 to 135 / 124 to 143 for four entries of 32 heads
    ([96] * 64, True, True), ([128] * 16, True, True), ([64], True, True), ([65] * 4, True, True), ([64] * 4, False, False)])
def test_retention_walk_by_the_entries_own_tokens(monkeypatch, lens, sixteen, thirty_two):
    import torch

    from sparseengine_b200.config.specs import RetentionSpec
    from sparseengine_b200.parts.base import make_mixer
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    step = SimpleNamespace(max_q_len=max(lens), num_tokens=sum(lens), num_seqs=len(lens), q_lens=lens)
    for heads, walk in ((16, sixteen), (32, thirty_two)):
        part = make_mixer(RetentionSpec(hidden_size=64, num_heads=heads, head_dim=128, v_head_dim=128, decays=(0.9,) * heads, position=None), torch.bfloat16)
        assert part.in_walk(step, "cuda:0") is walk


@pytest.mark.parametrize("lens,heads,hidden,tiles", [
    # device us of a layer without its projections, the walk / chunks side by side: 33/45, 41/45; 56/51, 56/53, 52/45; 44/45, 45/47, 117/78
    ([17], 32, 4096, False), ([128], 32, 4096, False), ([192], 32, 4096, False), ([257], 32, 4096, True), ([17], 64, 8192, True), ([40] * 2, 32, 4096, True),
    ([257], 16, 8192, True), ([17] * 4, 16, 8192, True), ([17] + [1] * 15, 16, 8192, True), ([8192], 32, 4096, True), ([130] * 2, 16, 8192, False),
    # calls one behind the other: 73/60, 72/60, 71/69; 71/78
    ([17], 16, 2048, True), ([17], 32, 2048, True), ([17], 24, 3072, True), ([17], 24, 4096, False)])
def test_retention_tiles_where_the_walk_is_not_ahead(monkeypatch, lens, heads, hidden, tiles):
    import torch

    from sparseengine_b200.config.specs import RetentionSpec
    from sparseengine_b200.parts.base import make_mixer
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    part = make_mixer(RetentionSpec(hidden_size=hidden, num_heads=heads, head_dim=128, v_head_dim=128, decays=(0.9,) * heads, position=None), torch.bfloat16)
    step = SimpleNamespace(max_q_len=max(lens), num_tokens=sum(lens), num_seqs=len(lens), q_lens=lens)
    assert part.in_tiles(step, sum(lens), 0, "cuda:0") is tiles
    # a captured step does not wait for the host
    if max(lens) <= 192 and len(lens) * heads * 4 <= 148:
        monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
        assert not part.in_tiles(step, sum(lens), 0, "cuda:0")


def _state_space(heads, groups):
    import torch

    from sparseengine_b200.config.specs import StateSpaceSpec
    from sparseengine_b200.parts.base import make_mixer
    return make_mixer(StateSpaceSpec(hidden_size=64, num_heads=heads, head_dim=64, state_size=128, groups=groups, conv_taps=4, norm_groups=groups), torch.bfloat16)


@pytest.mark.parametrize("lens,heads,groups,tiles", [
    # device us of a layer, the walk / chunks side by side: 42/46, 45/47, 43/47; 52/49, 65/45, 66/60, 84/67, 90/58
    ([128], 32, 8, False), ([96] * 2, 32, 8, False), ([130] * 2, 16, 8, False), ([128], 64, 8, True), ([128], 32, 1, True), ([257], 64, 8, True),
    ([512], 64, 8, True), ([1024], 16, 8, True),
    # token by token / side by side: 66/48, 185/138; 94/92 by tokens
    ([90], 64, 8, True), ([40] * 16, 64, 8, True), ([17] * 16, 64, 8, False)])
def test_state_space_tiles_by_all_three_estimates(monkeypatch, lens, heads, groups, tiles):
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    step = SimpleNamespace(max_q_len=max(lens), num_tokens=sum(lens), num_seqs=len(lens), q_lens=lens)
    assert bool(_state_space(heads, groups).in_tiles(step, "cuda:0")) is tiles


def test_state_space_chunks_from_a_number_of_tokens_on(monkeypatch):
    """What the engine's option sets: both forms of chunks from that many tokens on, whichever is estimated shorter."""
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    wide, narrow = _state_space(64, 8), _state_space(8, 8)
    wide.chunk_min_tokens, wide.chunks_by_estimate = 40, False
    narrow.chunk_min_tokens, narrow.chunks_by_estimate = 5, False

    def forms(part, lens):
        step = SimpleNamespace(max_q_len=max(lens), num_tokens=sum(lens), num_seqs=len(lens), q_lens=lens)
        return bool(part.in_tiles(step, "cuda:0")), part.in_chunks(step, "cuda:0")
    assert forms(wide, [2048]) == (True, True) and forms(wide, [40] * 4) == (True, True) and forms(wide, [39] * 400) == (False, False)
    assert forms(narrow, [5]) == (False, True) and forms(narrow, [4]) == (False, False) and forms(narrow, [1024]) == (True, True)
    wide.chunk_min_tokens = None
    assert forms(wide, [2048]) == (False, False)


def test_state_space_heads_a_block():
    heads = lambda *a: ops.ssm_tiles_plan(*a, 148)[1]      # noqa: E731
    # 257 tokens 72 us a layer with one head, 60 with two; 4,096 346 with four, 310 with eight; one block per SM and head at 128
    assert heads(3, 64, 8) == 2 and heads(32, 64, 8) == 8 and heads(1, 64, 8) == 1 and heads(95, 64, 8) == 8
    assert heads(10000, 11, 1) <= 8 and heads(1, 3, 3) == 1 and heads(50, 18, 2) <= 8
