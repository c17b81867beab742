"""Prompt-portion attention on tcgen05 where a block's two query tiles see different key tiles, against 64-bit softmax: windows, chunks and kept
first keys whose ends fall into, before and behind key tiles, second query tiles with few rows and none."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hq,hkv", [(2, 2), (3, 1)])
@pytest.mark.parametrize("options", [{}, dict(window=1), dict(window=64), dict(window=100), dict(window=63, keep_first=70), dict(window=200, keep_first=3),
                                     dict(window=129, keep_first=500), dict(chunk=64), dict(chunk=150), dict(window=320, softcap=3.0)],
                         ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()) or "plain")
def test_against_64_bits(hq, hkv, options):
    from sparseengine_b200.csrc import ops
    page, D = 16, 128
    g = torch.Generator(device=DEV).manual_seed(hq)
    q_lens, kv_lens = [257, 1, 128, 255, 17, 600, 64], [257, 64, 129, 900, 17, 1000, 1000]
    entries, tokens = len(q_lens), sum(q_lens)
    most = -(-max(kv_lens) // page)
    table = torch.randperm(entries * most, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(entries, most).to(DEV)
    rows = torch.tensor([3, 0, 5, 4, 1, 2, 6], dtype=torch.int32, device=DEV)
    cache = torch.randn(entries * most, 2, hkv, page, D, generator=g, device=DEV).to(torch.bfloat16)
    q = torch.randn(tokens, hq, D, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((tokens, hq, D), float("nan"), dtype=torch.bfloat16, device=DEV)
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    scale = D ** -0.5 * 1.5
    ops.attn_prefill_tc(q, cache, table, rows, torch.tensor(cu, dtype=torch.int32, device=DEV),
                        torch.tensor(kv_lens, dtype=torch.int32, device=DEV), out, entries=entries, max_q_len=max(q_lens), num_heads=hq,
                        num_kv_heads=hkv, head_dim=D, page_size=page, scale=scale, **options)
    ops.error_check(DEV)
    window, chunk, keep, cap = (options.get(k) for k in ("window", "chunk", "keep_first", "softcap"))
    want = torch.empty(tokens, hq, D, dtype=torch.float64, device=DEV)
    for e, (n, kv) in enumerate(zip(q_lens, kv_lens)):
        k, v = cache[table[int(rows[e])].long()].permute(1, 2, 0, 3, 4).reshape(2, hkv, -1, D)[:, :, :kv].double().repeat_interleave(hq // hkv, 1)
        pos, at = torch.arange(kv - n, kv, device=DEV)[:, None], torch.arange(kv, device=DEV)[None]
        seen = at <= pos
        if window:
            seen = seen & ((at > pos - window) | (at < (keep or 0)))
        if chunk:
            seen = seen & (at >= pos // chunk * chunk)
        s = torch.einsum("thd,hkd->htk", q[cu[e]:cu[e + 1]].double(), k) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        want[cu[e]:cu[e + 1]] = torch.einsum("htk,hkd->thd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), v)
    # weights rounded to 16 bits (2^-9 of their sum's size), the result rounded once
    assert float((out.double() - want).abs().max()) < 8e-3 * float(want.abs().max())
