"""Latent attention over keys and values formed per head against 64-bit softmax: query tiles that are full, nearly empty and empty, entries that
follow held rows, windows that end inside key tiles and leave whole tiles to one of a block's two query tiles, pages that must not be read."""
import pytest
import torch

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("heads,window,sinks", [(1, None, False), (3, 1, True), (2, 64, False), (5, 100, True), (2, 700, False), (32, None, True)])
def test_against_64_bits(heads, window, sinks):
    from sparseengine_b200.csrc import ops
    rank, page, D = 192, 16, 256
    g = torch.Generator(device=DEV).manual_seed(heads + (window or 0))
    q_lens, kv_lens = [257, 1, 128, 255, 17, 600], [257, 64, 129, 900, 17, 1000]
    entries, tokens = len(q_lens), sum(q_lens)
    most = -(-max(kv_lens) // page)
    table = torch.randperm(entries * most, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(entries, most).to(DEV)
    rows = torch.tensor([3, 0, 5, 4, 1, 2], dtype=torch.int32, device=DEV)
    cache = (torch.randn(entries * most, page, D, generator=g, device=DEV) * 0.7).to(torch.bfloat16)
    uk, uv = ((torch.randn(heads * 64, rank, generator=g, device=DEV) * rank ** -0.5).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(tokens, heads * 128 + 8, generator=g, device=DEV).to(torch.bfloat16)[:, :heads * 128]      # rows at a pitch
    sink = torch.linspace(-6.0, 4.0, heads, device=DEV) if sinks else None
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    cu_d, kv_d, scale = torch.tensor(cu, **i32), torch.tensor(kv_lens, **i32), 128 ** -0.5 * 2.0
    seen = ops.latent_seen_keys(q_lens, kv_lens, window)

    def run(cache, table):
        out = ops.latent_attention_heads(q, cache, table, rows, cu_d, kv_d, sink, uk, uv, rows=sum(seen), most_keys=max(seen), entries=entries,
                                         max_q_len=max(q_lens), heads=heads, rank=rank, page_size=page, scale=scale, window=window)
        ops.error_check(DEV)
        return out.view(tokens, heads, 64)

    out = run(cache, table)
    want = torch.empty(tokens, heads, 64, dtype=torch.float64, device=DEV)
    for e, (n, m) in enumerate(zip(q_lens, kv_lens)):
        at0 = m - seen[e]
        lat = cache[table[int(rows[e])].long()].reshape(-1, D)[at0:m]
        k, v = (torch.mm(lat[:, :rank], w.t()).double().view(-1, heads, 64) for w in (uk, uv))        # rounded to 16 bits there too
        k = torch.cat([k, lat[:, None, rank:].double().expand(-1, heads, -1)], -1)
        qs = q[cu[e]:cu[e + 1]].view(n, heads, 128).double()
        pos, at = torch.arange(m - n, m, device=DEV)[:, None], torch.arange(at0, m, device=DEV)[None]
        s = torch.einsum("thd,khd->thk", qs, k) * scale
        s = s.masked_fill(((at > pos) | (at <= pos - window) if window else at > pos)[:, None], float("-inf"))
        if sinks:
            s = torch.cat([s, sink.double()[None, :, None].expand(n, -1, 1)], -1)
        want[cu[e]:cu[e + 1]] = torch.einsum("thk,khd->thd", torch.softmax(s, -1)[..., :seen[e]], v)
    # weights rounded to 16 bits (2^-9 of their sum's size), the result rounded once
    assert float((out.double() - want).abs().max()) < 8e-3 * float(want.abs().max())
    if window:          # what lies before every query's window may be anybody's
        dirty, wrong = cache.clone(), table.clone()
        for e, n in enumerate(seen):
            for i in range((kv_lens[e] - n) // page):
                dirty[int(table[int(rows[e]), i])] = float("inf")
                wrong[int(rows[e]), i] = 10 ** 6
        assert torch.equal(run(dirty, wrong), out)


def _mixer_step(lens, held):
    from sparseengine_b200.parts.base import StepContext
    n, total, cu = len(lens), sum(lens), [0]
    for t in lens:
        cu.append(cu[-1] + t)
    i32 = dict(dtype=torch.int32, device=DEV)
    kv = [h + t for h, t in zip(held, lens)]
    return StepContext(num_tokens=total, num_seqs=n, token_ids=torch.zeros(total, **i32),
                       positions=torch.tensor([h + i for h, t in zip(held, lens) for i in range(t)], **i32),
                       token_seq=torch.tensor([j for j, t in enumerate(lens) for _ in range(t)], **i32),
                       seq_rows=torch.arange(n, **i32), cu_q=torch.tensor(cu, **i32), kv_len=torch.tensor(kv, **i32), q_lens=list(lens),
                       q_starts=list(held), kv_lens=kv, rows=list(range(n)), dtype=torch.bfloat16)


def _mixer(**options):
    from sparseengine_b200.config.specs import LatentAttentionSpec, RotarySpec
    from sparseengine_b200.parts.base import make_mixer
    part = make_mixer(LatentAttentionSpec(**dict(dict(hidden_size=256, num_heads=4, head_dim=64, rot_dim=64, v_head_dim=64, q_rank=128, kv_rank=192,
                                                      scale=128 ** -0.5, sink=True, position=RotarySpec(rotary_dim=64, theta=1e4)), **options)), torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(3)
    part.bind({n: (torch.randn(p.shape, generator=g, device=DEV) * (0.5 if "sink" in n else 0.06) + float("norm" in n)).to(
        torch.float32 if p.dtype == "float32" else torch.bfloat16) for n, p in part.parameters().items()})
    return part


def _mixer64(part, x, step, cache, table):
    """The mixer in 64 bits: cache [pages, 16, row] as it was before the step."""
    from sparseengine_b200.parts.position import as_rotary_args
    s, H = part.spec, part.spec.num_heads
    inv, split = as_rotary_args(part.position.kernel_args(torch.device(DEV))).inv_freq.double(), s.position.pairing == "split_half"
    angle = step.positions.double()[:, None] * inv

    def norm(t, w):
        return t / torch.sqrt((t * t).mean(-1, keepdim=True) + s.norm_eps) * w.double()

    def turn(t):                # [tokens, ..., 64]
        cs, sn = (f(angle).view(-1, *[1] * (t.dim() - 2), 32) for f in (torch.cos, torch.sin))
        a, b = (t[..., :32], t[..., 32:]) if split else (t[..., 0::2], t[..., 1::2])
        a, b = a * cs - b * sn, b * cs + a * sn
        return torch.cat([a, b], -1) if split else torch.stack([a, b], -1).flatten(-2)

    proj = x.double() @ (part.down if s.q_rank else part.in_proj).double().t()
    q = norm(proj[:, :s.q_rank], part.q_norm) @ part.uq.double().t() if s.q_rank else proj[:, :H * 128]
    q = q.view(-1, H, 128)
    q = torch.cat([q[..., :64], turn(q[..., 64:])], -1)
    lat = proj[:, s.q_rank or H * 128:]
    new = torch.cat([norm(lat[:, :s.kv_rank], part.kv_norm), turn(lat[:, s.kv_rank:s.kv_rank + 64])], -1)
    out, at = [], 0
    for e, (n, kv) in enumerate(zip(step.q_lens, step.kv_lens)):
        rows = torch.cat([cache[table[e].long()].reshape(-1, cache.shape[-1])[:kv - n].double(), new[at:at + n]])
        k, v = ((rows[:, :s.kv_rank] @ w.double().t()).view(kv, H, 64) for w in (part.uk, part.uv))
        k = torch.cat([k, rows[:, None, s.kv_rank:].expand(-1, H, -1)], -1)
        pos, key = torch.arange(kv - n, kv, device=DEV)[:, None], torch.arange(kv, device=DEV)[None]
        hidden = (key > pos) | (key <= pos - s.window) if s.window else key > pos
        score = (torch.einsum("thd,khd->thk", q[at:at + n], k) * s.scale).masked_fill(hidden[:, None], float("-inf"))
        if s.sink:
            score = torch.cat([score, part.sink.double()[None, :, None].expand(n, -1, 1)], -1)
        out.append(torch.einsum("thk,khd->thd", torch.softmax(score, -1)[..., :kv], v).flatten(1))
        at += n
    out = torch.cat(out)
    if s.output_gate:
        out = out * torch.sigmoid(proj[:, part.g_off:])
    return out @ part.o.double().t()


@pytest.mark.gpu
@pytest.mark.parametrize("pairing", ["split_half", "interleaved"])
@pytest.mark.parametrize("options", [dict(), dict(q_rank=0, output_gate=True, sink=False), dict(q_rank=0, window=100), dict(q_rank=0, output_gate=True, kv_rank=80)],
                         ids=["query latent", "direct, gated", "direct, window", "direct, gated, short latent"])
def test_mixer_against_64_bits(options, pairing, monkeypatch):
    """The whole mixer in this form: queries rotated in place, which without a query latent are columns of the projection beside the gate's."""
    from sparseengine_b200.config.specs import RotarySpec
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.base import LayerSlot
    monkeypatch.setattr(ops, "latent_takes_heads", lambda *a, **k: True)
    part = _mixer(position=RotarySpec(rotary_dim=64, theta=1e4, pairing=pairing), **options)
    step, row = _mixer_step([257, 1, 70], [0, 64, 500]), part.spec.kv_rank + 64
    g = torch.Generator(device=DEV).manual_seed(8)
    x = torch.randn(328, 256, generator=g, device=DEV).to(torch.bfloat16)
    cache = torch.randn(120, 16, row, generator=g, device=DEV).to(torch.bfloat16)
    table = torch.randperm(120, generator=torch.Generator().manual_seed(9)).to(torch.int32)[:108].view(3, 36).contiguous().to(DEV)
    want = _mixer64(part, x, step, cache.clone(), table)
    before = ops.calls.get("se_latent_gather", 0)
    got = part.forward(x, step, LayerSlot(kv=cache, table=table, page_size=16))
    assert ops.calls.get("se_latent_gather", 0) == before + 1
    ops.error_check(DEV)
    # nine roundings to 16 bits one after another (projection, norm, queries, rotation, keys or values, weights, sums, gate, result), each 2^-9 / sqrt(3)
    # of its vector on average; scores of order one pass theirs on once more: sqrt(2 * 9) * 1.13e-3 = 4.8e-3, three times that
    assert float((got.double() - want).norm()) < 1.5e-2 * float(want.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("pairing", ["split_half", "interleaved"])
@pytest.mark.parametrize("heads,d,rot,rotary,more", [(4, 64, 64, 64, 0), (3, 64, 64, 64, 24), (40, 16, 32, 32, 8), (3, 20, 24, 24, 0), (2, 64, 64, 32, 8), (5, 7, 6, 4, 3)])
def test_queries_rotated_in_place(heads, d, rot, rotary, more, pairing):
    """The same numbers as into another matrix, and nothing else of the rows (views with ``more`` columns behind) touched."""
    from sparseengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(10)
    wide = torch.randn(37, heads * (d + rot) + more, generator=g, device=DEV).to(torch.bfloat16)
    inv, positions = torch.rand(rotary // 2, generator=g, device=DEV), torch.arange(37, dtype=torch.int32, device=DEV) * 13
    sizes = dict(heads=heads, head_dim=d, rank=d, rot=rot, rotary_dim=rotary, pairing=pairing)
    apart, want = torch.zeros(37, heads, d + rot, dtype=torch.bfloat16, device=DEV), wide.clone()
    ops.latent_q_rotate(wide[:, :heads * (d + rot)], inv, positions, apart, **sizes)
    want[:, :heads * (d + rot)].view(37, heads, d + rot)[..., d:] = apart[..., d:]
    assert not torch.equal(want, wide)
    q = wide[:, :heads * (d + rot)]
    ops.latent_q_rotate(q, inv, positions, q, **sizes)
    assert torch.equal(wide, want)


@pytest.mark.gpu
@pytest.mark.parametrize("page", [-1, 64, 10 ** 6])
def test_pages_outside_the_pool(page):
    """A table entry in the gathered range that names no page: reported, its rows zeros, the other entry's outputs as they were."""
    from sparseengine_b200.csrc import ops
    g, i32 = torch.Generator(device=DEV).manual_seed(11), dict(dtype=torch.int32, device=DEV)
    cache = torch.randn(64, 16, 256, generator=g, device=DEV).to(torch.bfloat16)
    uk, uv = ((torch.randn(128, 192, generator=g, device=DEV) * 0.07).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(164, 256, generator=g, device=DEV).to(torch.bfloat16)

    def run(cache, table):
        return ops.latent_attention_heads(q, cache, table, torch.tensor([0, 1], **i32), torch.tensor([0, 64, 164], **i32), torch.tensor([300, 100], **i32),
                                          None, uk, uv, rows=400, most_keys=300, entries=2, max_q_len=100, heads=2, rank=192, page_size=16, scale=0.1)

    table, blank = torch.arange(64, **i32).view(2, 32), cache.clone()
    blank[5] = 0
    want = run(blank, table)
    table[0, 5] = page
    got = run(cache, table)
    with pytest.raises(RuntimeError, match="code 30"):
        ops.error_check(DEV)
    assert torch.equal(got, want)


@pytest.mark.gpu
def test_captured_portion_replayed_with_other_lengths(monkeypatch):
    """A graph of a prompt portion is replayed behind more held keys than it was captured with."""
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.base import LayerSlot
    monkeypatch.setattr(ops, "latent_takes_heads", lambda *a, **k: True)
    part, lens = _mixer(), [70]
    g = torch.Generator(device=DEV).manual_seed(4)
    x = torch.randn(70, 256, generator=g, device=DEV).to(torch.bfloat16)
    cache = torch.randn(80, 16, 256, generator=g, device=DEV).to(torch.bfloat16)
    slot = LayerSlot(kv=cache, table=torch.randperm(80, generator=torch.Generator().manual_seed(5)).to(torch.int32).view(1, 80).to(DEV), page_size=16)
    step, later = _mixer_step(lens, [30]), _mixer_step(lens, [1000])
    before = ops.calls.get("se_latent_gather", 0)
    part.forward(x, step, slot)
    want = part.forward(x, later, slot).clone()
    assert ops.calls.get("se_latent_gather", 0) == before + 2
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        part.forward(x, step, slot)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = part.forward(x, step, slot)
    step.positions.copy_(later.positions)
    step.kv_len.copy_(later.kv_len)
    graph.replay()
    torch.cuda.synchronize()
    ops.error_check(DEV)
    # two forms of the same attention, each with 16-bit weights and intermediate vectors
    assert float((out.double() - want.double()).norm()) < 2e-2 * float(want.double().norm())


@pytest.mark.gpu
@pytest.mark.parametrize("rows_short,keys_short", [(1, 0), (300, 0), (0, 40), (561, 468)])
def test_lengths_beyond_the_planned_ones(rows_short, keys_short):
    """Lengths on the device that go beyond what the workspace and the grid were made for are reported and their rows left alone."""
    from sparseengine_b200.csrc import ops
    heads, rank, lens, kv = 2, 192, [64, 100], [500, 61 + 100]
    g = torch.Generator(device=DEV).manual_seed(6)
    i32 = dict(dtype=torch.int32, device=DEV)
    cache = torch.randn(64, 16, 256, generator=g, device=DEV).to(torch.bfloat16)
    uk, uv = ((torch.randn(heads * 64, rank, generator=g, device=DEV) * 0.07).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(sum(lens), heads * 128, generator=g, device=DEV).to(torch.bfloat16)
    table = torch.arange(64, **i32).view(2, 32)

    def run(rows, most):
        return ops.latent_attention_heads(q, cache, table, torch.tensor([0, 1], **i32), torch.tensor([0, 64, 164], **i32), torch.tensor(kv, **i32), None, uk, uv,
                                          rows=rows, most_keys=most, entries=2, max_q_len=100, heads=heads, rank=rank, page_size=16, scale=0.1)

    want = run(661, 500)
    ops.error_check(DEV)
    got = run(661 - rows_short, 500 - keys_short)
    with pytest.raises(RuntimeError, match="code 31"):
        ops.error_check(DEV)
    if rows_short == 1:                                 # the first entry's rows are all there
        assert torch.equal(got[:64], want[:64])


def test_choice():
    from sparseengine_b200.csrc import ops
    assert ops.latent_seen_keys([5, 1, 8], [5, 90, 20], 10) == [5, 10, 17] and ops.latent_seen_keys([5], [90], None) == [90]
    take = lambda q, kv, window=None, heads=32: ops.latent_takes_heads(max(q), heads, 192, 148, q, kv, window)
    assert take([8192], [8192], 1024) and take([1000], [5000]) and take([500] * 4, [1000] * 4, 1024, 64)
    assert not take([1] * 64, [3000] * 64) and not take([31], [31])            # single tokens: the expansion is never paid back
    assert not take([64], [200000], None, 64)                                 # the keys and values would take more than their bound


def test_choice_compares_with_the_kernel_that_would_run():
    """A latent of 176 is not for the tcgen05 kernel, whose estimate kept steps from the keys per head though the tiled kernel would have run."""
    from sparseengine_b200.csrc import ops
    assert ops.latent_attention_tiled_supported(176, 64) and not ops.latent_attention_tc_supported(176, 64)
    take = lambda q, kv, window=None, heads=16, rank=176: ops.latent_takes_heads(max(q), heads, rank, 148, q, kv, window)
    assert take([64] * 4, [1064] * 4, 1024) and take([100], [100]) and not take([64] * 4, [1064] * 4, 1024, rank=192)
    assert not take([32], [32], heads=2)
