"""Latent attention over prompt portions on tcgen05 against 64-bit softmax: every number of 64-dim blocks it takes, row tiles
that are full, half full and nearly empty, windows that end inside key tiles, pages that must not be read."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("heads", [1, 5, 32])
@pytest.mark.parametrize("rank,rot,window,sinks", [(192, 64, 100, True), (192, 64, None, False), (192, 0, 64, True), (128, 128, None, True),
                                                   (128, 64, 65, True), (128, 0, 1, False), (64, 192, 130, True), (64, 64, None, False), (64, 0, 63, True)])
def test_against_64_bits(rank, rot, heads, window, sinks):
    from sparseengine_b200.csrc import ops
    assert ops.latent_attention_tc_supported(rank, rot) and bool(ops.library().se_latent_attention_tc_supported(rank, rot))
    D, page = rank + rot, 16
    g = torch.Generator(device=DEV).manual_seed(rank + rot + heads)
    q_lens, kv_lens = [37, 1, 130, 8, 64], [37, 64, 409, 140, 64]
    entries, tokens = len(q_lens), sum(q_lens)
    most = -(-max(kv_lens) // page)
    table = torch.randperm(entries * most, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(entries, most).to(DEV)
    rows = torch.tensor([3, 0, 4, 1, 2], dtype=torch.int32, device=DEV)
    cache = (torch.randn(entries * most, page, D, generator=g, device=DEV) * 0.7).to(torch.bfloat16)
    qfull = torch.randn(tokens, heads, D, generator=g, device=DEV).to(torch.bfloat16)
    sink = torch.linspace(-6.0, 4.0, heads, device=DEV) if sinks else None
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    scale = D ** -0.5 * 2.0
    args = (torch.tensor(cu, dtype=torch.int32, device=DEV), torch.tensor(kv_lens, dtype=torch.int32, device=DEV), sink)
    sizes = dict(entries=entries, max_q_len=max(q_lens), heads=heads, rank=rank, rot=rot, page_size=page, scale=scale, window=window)

    def run(cache, table):
        out = torch.full((tokens, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.latent_attention_tc(qfull, cache, table, rows, *args, out, **sizes)
        ops.error_check(DEV)
        return out

    out = run(cache, table)
    want = torch.empty(tokens, heads, rank, dtype=torch.float64, device=DEV)
    for e, (n, kv) in enumerate(zip(q_lens, kv_lens)):
        keys = cache[table[int(rows[e])].long()].reshape(-1, D)[:kv].double()
        pos, at = torch.arange(kv - n, kv, device=DEV)[:, None], torch.arange(kv, device=DEV)[None]
        hidden = (at > pos) | (at <= pos - window) if window else at > pos
        s = torch.einsum("thd,kd->thk", qfull[cu[e]:cu[e + 1]].double(), keys) * scale
        s = s.masked_fill(hidden[:, None], float("-inf"))
        if sinks:
            s = torch.cat([s, sink.double()[None, :, None].expand(n, -1, 1)], -1)
        want[cu[e]:cu[e + 1]] = torch.einsum("thk,kd->thd", torch.softmax(s, -1)[..., :kv], keys[:, :rank])
    # weights rounded to 16 bits (2^-9 of their sum's size), the result rounded once
    assert float((out.double() - want).abs().max()) < 8e-3 * float(want.abs().max())
    if window:          # what lies before every query's window may be anybody's
        dirty, wrong = cache.clone(), table.clone()
        for e, (n, kv) in enumerate(zip(q_lens, kv_lens)):
            first = kv - n - window + 1          # tiles start at multiples of 64 rows; a block spans all rows of short entries
            for i in range(max(0, first) // page):
                dirty[int(table[int(rows[e]), i])] = float("inf")
                wrong[int(rows[e]), i] = 10 ** 6
        assert torch.equal(run(dirty, wrong), out)


def test_a_bad_page_names_this_kernel():
    """An entry that names no page: left out, reported with a code that no other kernel has."""
    from sparseengine_b200.csrc import ops
    i32 = dict(dtype=torch.int32, device=DEV)
    table = torch.tensor([[0, 10 ** 6, 2, 3]], **i32)
    cache, q = torch.randn(4, 16, 128, device=DEV).to(torch.bfloat16), torch.randn(60, 4, 128, device=DEV).to(torch.bfloat16)
    out = torch.empty(60, 4, 64, dtype=torch.bfloat16, device=DEV)
    args = (torch.zeros(1, **i32), torch.tensor([0, 60], **i32), torch.tensor([60], **i32), None, out)
    sizes = dict(entries=1, max_q_len=60, heads=4, rank=64, rot=64, page_size=16, scale=0.1)
    for fn, name in ((ops.latent_attention_tc, "the tcgen05 latent"), (ops.latent_attention_tiled, "the tiled latent")):
        fn(q, cache, table, *args, **sizes)
        with pytest.raises(RuntimeError, match=name):
            ops.error_check(DEV)
    assert bool(torch.isfinite(out).all())


def test_choice_by_rows():
    from sparseengine_b200.csrc import ops
    assert ops.latent_takes_tc(1, 2048, 32, 192, 64, 148) and ops.latent_takes_tc(4, 512, 16, 128, 64, 148)
    assert not ops.latent_takes_tc(64, 1, 32, 192, 64, 148) and not ops.latent_takes_tc(1, 64, 32, 192, 64, 148)
    assert not ops.latent_takes_tc(1, 8192, 32, 256, 0, 148) and not ops.latent_takes_tc(1, 8192, 32, 80, 48, 148)
