"""The 32-bit path's kernels for prompt portions and routed experts against the general ones (one block per token and head;
tiles of 32 rows) and against 64-bit sums, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _batch(q_lens, kv_lens, page, seed):
    g = torch.Generator().manual_seed(seed)
    most = -(-max(kv_lens) // page)
    n = len(q_lens)
    i32 = dict(dtype=torch.int32, device=DEV)
    cu = [0]
    for t in q_lens:
        cu.append(cu[-1] + t)
    return dict(table=torch.randperm(n * most, generator=g).to(torch.int32).view(n, most).to(DEV), rows=torch.randperm(n, generator=g).to(torch.int32).to(DEV),
                cu=torch.tensor(cu, **i32), kv=torch.tensor(kv_lens, **i32), pages=n * most, tokens=cu[-1],
                seq=torch.tensor([j for j, t in enumerate(q_lens) for _ in range(t)], **i32),
                pos=torch.tensor([k - t + i for t, k in zip(q_lens, kv_lens) for i in range(t)], **i32))


OPTIONS = {"plain": {}, "window": dict(window=37), "wide window": dict(window=129, keep_first=70), "chunk": dict(chunk=50),
           "cap, sink": dict(softcap=3.0, sink=True), "kept, learned sink": dict(window=20, keep_first=5, sink="learned"),
           "slopes": dict(slopes=True, gate="head"), "gate": dict(gate="element", window=64)}


@pytest.mark.parametrize("options", list(OPTIONS))
@pytest.mark.parametrize("d,dv,heads,kv_heads,page", [(128, 128, 6, 1, 16), (64, 64, 4, 2, 8), (20, 12, 5, 5, 4), (100, 68, 3, 1, 16), (32, 128, 64, 1, 5)])
def test_portion_attention(d, dv, heads, kv_heads, page, options):
    """Tiles of 128 rows and 64 keys: entries that end on, before and behind tile edges, single tokens among them, every
    option; and values that are not finite where a row does not see them."""
    from sparseengine_b200.csrc import ops
    b = _batch([64, 1, 130, 2, 63], [64, 129, 209, 17, 191], page, d + heads)
    g = torch.Generator(device=DEV).manual_seed(d)
    cache = torch.randn(b["pages"], page * kv_heads * (d + dv), generator=g, device=DEV) * 0.7
    q = torch.randn(b["tokens"], heads * d, generator=g, device=DEV)
    opt = dict(OPTIONS[options])
    if opt.get("gate"):
        cols = heads * (dv if opt["gate"] == "element" else 1)
        opt["gate"] = torch.randn(b["tokens"], cols + 5, generator=g, device=DEV)[:, 2:2 + cols]
    if opt.get("sink") == "learned":
        opt["sink"] = torch.randn(heads, generator=g, device=DEV)
    if opt.get("slopes"):
        opt["slopes"] = torch.rand(heads, generator=g, device=DEV)
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=d, v_head_dim=dv, page_size=page, scale=d ** -0.5, **opt)

    def both():
        want, got = (torch.full((b["tokens"], heads * dv), float("nan"), device=DEV) for _ in range(2))
        ops.paged_attention_plain(q, cache, b["table"], b["rows"], b["seq"], b["pos"], want, **common)
        ops.attn_prefill_f32(q, cache, b["table"], b["rows"], b["cu"], b["kv"], got, entries=5, max_q_len=130, **common)
        ops.error_check(DEV)
        return want, got

    want, got = both()
    # two orders of the same 32-bit sums over at most 209 keys of products of size one
    assert bool(torch.isfinite(got).all()) and float((got - want).abs().max()) < 4e-6 * max(1.0, float(want.abs().max()))
    # the last token of the first entry has a value of infinity: only rows that see it change
    if page * kv_heads * (d + dv) and options in ("plain", "window", "chunk"):
        where = int(b["table"][int(b["rows"][0]), 63 // page])
        cache[where, page * kv_heads * d + (63 % page) * dv:page * kv_heads * d + (63 % page) * dv + dv] = float("inf")
        want2, got2 = both()
        assert torch.equal(torch.isfinite(got2), torch.isfinite(want2)) and bool(torch.isfinite(got2[:63]).all())
        assert torch.equal(got2[:63], got[:63])


def test_portion_attention_leaves_bad_pages_out():
    from sparseengine_b200.csrc import ops
    b = _batch([40], [200], 16, 1)
    cache = torch.randn(b["pages"], 16 * 2 * 128, device=DEV)
    q = torch.randn(40, 4 * 64, device=DEV)
    b["table"][0, 3] = 10 ** 6
    common = dict(num_heads=4, num_kv_heads=2, head_dim=64, page_size=16, scale=0.2)
    want, got = torch.empty_like(q), torch.empty_like(q)
    for fn in (lambda: ops.paged_attention_plain(q, cache, b["table"], b["rows"], b["seq"], b["pos"], want, **common),
               lambda: ops.attn_prefill_f32(q, cache, b["table"], b["rows"], b["cu"], b["kv"], got, entries=1, max_q_len=40, **common)):
        fn()
        with pytest.raises(Exception):
            ops.error_check(DEV)
    assert float((got - want).abs().max()) < 4e-6


@pytest.mark.parametrize("activation", [None, ("clamped_swiglu", 1.0, 1.7)])
@pytest.mark.parametrize("counts,hidden,inter", [
    ([1, 0, 2, 3, 4, 5, 8, 1, 9, 0, 0, 0, 0, 0, 0, 0], 64, 36),         # streamed: one to eight rows, nine in two tiles
    ([1, 1, 0, 0], 132, 100), ([1], 4, 4),
    ([127, 128, 129, 0, 1, 31, 33, 97], 64, 36), ([300, 5], 132, 100), ([64], 20, 260)])        # tiles of 128 rows
def test_routed_products(counts, hidden, inter, activation):
    """Both products of the experts, tiles of 8 and of 128 rows against the general kernel's, at their edges in rows, features
    and inner dimension."""
    from sparseengine_b200.config.specs import MoESpec
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.moe import SparseMoE
    g = torch.Generator(device=DEV).manual_seed(sum(counts))
    experts, tokens = len(counts), sum(counts)
    spec = MoESpec(hidden_size=hidden, num_experts=experts, top_k=1, intermediate_size=inter,
                   **({} if activation is None else dict(activation=activation[0], activation_limit=activation[1], activation_alpha=activation[2])))
    part = SparseMoE(spec, torch.float32)
    part.bind({"w13": torch.randn(experts, 2 * inter, hidden, generator=g, device=DEV) * hidden ** -0.5,
               "w2": torch.randn(experts, hidden, inter, generator=g, device=DEV) * inter ** -0.5})
    x = torch.randn(tokens, hidden, generator=g, device=DEV)
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[torch.randperm(tokens, generator=torch.Generator().manual_seed(3))]
    ids = ids.view(-1, 1).to(torch.int32).to(DEV)
    weights = torch.rand(tokens, 1, generator=g, device=DEV)
    assert part.plain_tile_rows(x, tokens) == (8 if tokens <= 4 * experts else 128)
    got = part.run_experts(x, ids, weights)
    part.plain_tile_rows = lambda x, a: ops.moe_plain_tile_rows()
    want = part.run_experts(x, ids, weights)
    # sums of at most 260 products of size one in another order
    assert float((got - want).abs().max()) < 4e-6 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("options", [{}, dict(window=37, keep_first=6), dict(softcap=3.0, sink=True)], ids=["plain", "window, kept", "cap, sink"])
@pytest.mark.parametrize("copies", [1, 8, 64])             # few and many blocks: 16, 8 and 4 warps to a token's keys
@pytest.mark.parametrize("d,dv,heads,kv_heads", [(128, 128, 6, 1), (132, 68, 2, 2), (20, 140, 4, 2), (256, 256, 4, 1)])
def test_single_tokens(d, dv, heads, kv_heads, copies, options):
    """Single tokens that see 1 to 200 keys (groups of four keys, partly empty) against 64-bit sums."""
    from sparseengine_b200.csrc import ops
    held, page = [1, 2, 3, 5, 16, 63, 64, 65, 68, 200] * copies, 8
    b = _batch([1] * len(held), held, page, d)
    g = torch.Generator(device=DEV).manual_seed(d)
    cache = torch.randn(b["pages"], page * kv_heads * (d + dv), generator=g, device=DEV)
    q, out = torch.randn(len(held), heads * d, generator=g, device=DEV), torch.empty(len(held), heads * dv, device=DEV)
    ops.paged_attention_plain(q, cache, b["table"], b["rows"], b["seq"], b["pos"], out, num_heads=heads, num_kv_heads=kv_heads, head_dim=d,
                              v_head_dim=dv, page_size=page, scale=d ** -0.5, **options)
    ops.error_check(DEV)
    for e in range(10):
        n = held[e]
        pages = cache[b["table"][b["rows"][e].long()].long()].double()
        k = pages[:, :page * kv_heads * d].view(-1, kv_heads, page, d).transpose(1, 2).reshape(-1, kv_heads, d)[:n]
        v = pages[:, page * kv_heads * d:].view(-1, kv_heads, page, dv).transpose(1, 2).reshape(-1, kv_heads, dv)[:n]
        k, v = (x.repeat_interleave(heads // kv_heads, 1) for x in (k, v))
        s = torch.einsum("hd,nhd->hn", q[e].view(heads, d).double(), k) * d ** -0.5
        if options.get("softcap"):
            s = 3.0 * torch.tanh(s / 3.0)
        if options.get("window"):
            i = torch.arange(n, device=DEV)
            s = s.masked_fill((i < n - 37) & (i >= 6), float("-inf"))
        if options.get("sink"):
            s = torch.cat([s, torch.zeros(heads, 1, dtype=s.dtype, device=DEV)], 1)
        want = torch.einsum("hn,nhd->hd", torch.softmax(s, 1)[:, :n], v)
        # sums over at most 256 products and 200 keys of size one; the scores' error enters through the exponential
        assert float((out[e].view(heads, dv).double() - want).abs().max()) < 4e-6 * max(1.0, float(want.abs().max()))


def _layer(**sizes):
    from sparseengine_b200.config.specs import AttentionSpec
    from sparseengine_b200.parts.base import make_mixer
    return make_mixer(AttentionSpec(hidden_size=64, scale=0.125, position=None, **sizes), torch.float32)


def test_portions_on_odd_addresses_take_the_plain_kernel():
    """A cache, queries or an output that do not lie on 16 bytes are served as aligned ones are."""
    from types import SimpleNamespace

    from sparseengine_b200.csrc import ops
    heads, kv_heads, d, page = 4, 2, 64, 16
    part = _layer(num_heads=heads, num_kv_heads=kv_heads, head_dim=d)
    b = _batch([40, 17], [40, 90], page, 1)
    step = SimpleNamespace(num_tokens=57, num_seqs=2, max_q_len=40, max_kv_len=90, seq_rows=b["rows"], token_seq=b["seq"],
                           positions=b["pos"], cu_q=b["cu"], kv_len=b["kv"], q_lens=[40, 17], kv_lens=[40, 90], max_kv_bound=None, extras={})
    part.f32_tiles_pay = lambda step, device: True
    tensors = {"kv": torch.randn(b["pages"], 2, kv_heads, page, d, device=DEV), "q": torch.randn(57, heads * d, device=DEV),
               "out": torch.empty(57, heads * d, device=DEV)}

    def attend(odd=None):
        t = dict(tensors)
        if odd is not None:
            store = torch.empty(t[odd].numel() + 1, device=DEV)
            store[1:] = t[odd].flatten()
            t[odd] = store[1:].view(t[odd].shape)
        before = ops.calls.get("se_attn_prefill_f32", 0)
        part.attend(t["q"], t["out"], step, SimpleNamespace(kv=t["kv"], table=b["table"], page_size=page))
        ops.error_check(DEV)
        return t["out"].clone(), ops.calls.get("se_attn_prefill_f32", 0) - before

    want, tiled = attend()
    assert tiled == 1
    for odd in tensors:
        got, tiled = attend(odd)
        assert tiled == 0 and float((got - want).abs().max()) < 4e-6


def test_a_seen_key_without_weight_still_shows_what_is_not_finite():
    """A value of infinity under a weight that underflows to zero gives NaN for the rows that see it, as in the plain kernel."""
    from sparseengine_b200.csrc import ops
    b = _batch([150], [150], 16, 1)
    kv_heads, heads, d = 1, 2, 64
    cache = torch.randn(b["pages"], 2, kv_heads, 16, d, device=DEV)
    q = torch.randn(150, heads, d, device=DEV)
    q[:, :, 0] = 10.0
    at, slot = int(b["table"][0, 70 // 16]), 70 % 16
    cache[at, 0, 0, slot] = 0.0
    cache[at, 0, 0, slot, 0] = -1000.0         # scores of -1,250
    cache[at, 1, 0, slot, 5] = float("inf")
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=d, page_size=16, scale=0.125)
    want, got = torch.empty(150, heads * d, device=DEV), torch.empty(150, heads * d, device=DEV)
    ops.paged_attention_plain(q.view(150, -1), cache, b["table"], b["rows"], b["seq"], b["pos"], want, **common)
    ops.attn_prefill_f32(q.view(150, -1), cache, b["table"], b["rows"], b["cu"], b["kv"], got, entries=1, max_q_len=150, **common)
    ops.error_check(DEV)
    bad = ~torch.isfinite(want)
    assert torch.equal(~torch.isfinite(got), bad) and bool(bad.view(150, heads, d)[70:, :, 5].all()) and int(bad.sum()) == 80 * heads
    assert float((got - want)[~bad].abs().max()) < 4e-6
