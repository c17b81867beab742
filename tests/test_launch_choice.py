"""What launchers are told to choose by: the longest entry, the step's states, the device's SMs (no GPU)."""
import pytest

from sparseengine_b200.csrc import ops


@pytest.mark.parametrize("heads,size,lens,lanes", [
    # portions beside single tokens, measured us lane groups / tiles: 61/38, 62/56, 69/79, 125/148, 221/205, 84/49
    (64, 128, [64] + [1] * 3, 0), (64, 128, [64] + [1] * 15, 0), (64, 128, [64] + [1] * 31, 1), (64, 128, [90] + [1] * 63, 1),
    (64, 128, [200] + [1] * 63, 0), (64, 128, [90] + [1] * 3, 0),
    # 8.2/10.3, 43/33, 53/99, 265/302, and with fewer and more heads 41/29, 12/25, 186/257, 187/135
    (64, 128, [8], 1), (64, 128, [64], 0), (64, 128, [1] * 64, 1), (64, 128, [17] * 64, 1),
    (16, 64, [64] + [1] * 7, 0), (16, 64, [1] * 128, 1), (128, 128, [90] + [1] * 63, 1), (128, 128, [200] + [1] * 7, 0)])
def test_by_the_longest_entry(heads, size, lens, lanes):
    assert ops.library().se_ssm_scan_by_lanes(heads, 64, size, sum(lens), len(lens), max(lens), 148) == lanes


@pytest.fixture
def seen(monkeypatch):
    """The arguments that launchers are called with, on a device of 99 SMs."""
    calls = []
    monkeypatch.setattr(ops, "_fn", lambda name, types: lambda *args: calls.append(args) or 0)
    for name, value in (("sm_count", 99), ("_stream", None), ("_ptr", 0), ("error_word", None)):
        monkeypatch.setattr(ops, name, lambda *args, value=value: value)
    return calls


def test_the_scan_hears_of_the_longest_entry_and_the_device(seen):
    from types import SimpleNamespace

    import torch
    f, i = torch.zeros(4, 8), torch.zeros(3, dtype=torch.int32)
    step = SimpleNamespace(cu_q=i, seq_rows=i, num_seqs=2, max_q_len=3)
    ops.ssm_scan(f, f, 0, f[0], f[0], f[0], f, step, f.clone(), heads=1, head_dim=4, state_size=2, groups=1)
    assert seen[0][-4:-2] == (3, 99)


def test_plain_attention_hears_of_the_device(seen):
    import torch
    f, i = torch.zeros(4, 8), torch.zeros(4, dtype=torch.int32)
    ops.paged_attention_plain(f, f, i.view(2, 2), i, i, i, f.clone(), num_heads=2, num_kv_heads=1, head_dim=4, page_size=4, scale=1.0)
    assert seen[0][-3] == 99


def test_sm_counts_are_kept_by_device(monkeypatch):
    """A device with an index answers from memory; one without goes by the current device each time."""
    from types import SimpleNamespace

    import torch
    current, counts = [0], {0: 148, 1: 132}
    monkeypatch.setattr(ops, "_sm_counts", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[0])
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda key: SimpleNamespace(multi_processor_count=counts[key]))
    for _ in range(2):
        assert [ops.sm_count(d) for d in (torch.device("cuda", 1), "cuda:1", 1, torch.device("cuda", 0), "cuda:0")] == [132, 132, 132, 148, 148]
        for current[0] in (0, 1):
            assert ops.sm_count() == ops.sm_count("cuda") == ops.sm_count(torch.device("cuda")) == counts[current[0]]
