"""The linear recurrences over prompt portions in chunks (csrc/chunk_walk.cuh) against 64-bit walks token by token, from
non-zero states, with entries that end on, before and behind the chunks' edges."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS = [1, 63, 64, 65, 200, 0, 31, 32, 33, 17]
# two orders of the same 32-bit sums over at most 200 tokens and 128 rows, as a share of the largest value
BOUND = 5e-6


def _step(rows):
    cu = [0]
    for n in LENS:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    return SimpleNamespace(cu_q=torch.tensor(cu, **i32), seq_rows=torch.tensor(rows, **i32), num_seqs=len(LENS), num_tokens=cu[-1],
                           max_q_len=max(LENS), cu=cu, rows=rows,
                           token_seq=torch.tensor([e for e, n in enumerate(LENS) for _ in range(n)], **i32))


def _walk64(q, k, v, keep, S, beta=None):
    """q, k [T, H, d], v [T, H, dv], keep [T, H, 1 or d], S [H, d, dv]; the delta rule with ``beta`` [T, H]."""
    out = []
    for t in range(q.shape[0]):
        S = keep[t][..., None] * S
        u = v[t]
        if beta is not None:
            u = beta[t][:, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], S))
        S = S + k[t][..., None] * u[:, None]
        out.append(torch.einsum("hd,hdv->hv", q[t], S))
    return (torch.stack(out) if out else v), S


def _close(got, want, what):
    worst, most = float((got.double() - want).abs().max()), float(want.abs().max())
    assert worst < BOUND * most, f"{what}: {worst:.3e} of {most:.3e}"


# the last: 32 value columns a block with up to 64 rows
SIZES = [(128, 128, 3, 3), (64, 64, 4, 2), (8, 4, 2, 1), (100, 36, 3, 3), (128, 20, 40, 10), (44, 132, 2, 2), (32, 12, 2, 2), (64, 64, 8, 4)]


@pytest.mark.parametrize("decay", ["slow", "fast"])
@pytest.mark.parametrize("d,dv,heads,kv_heads", SIZES)
@pytest.mark.parametrize("kind", ["retention", "retention, 16-bit values", "state space", "delta, per head", "delta, per channel", "state space, tokens",
                                  "delta, tokens"])
def test_chunks_against_the_walk(kind, d, dv, heads, kv_heads, decay):
    """``fast``: decays down to e^-30 per token, whose products underflow within a chunk.  ``tokens``: the kernels that walk token
    by token, on the same inputs.  ``16-bit values``: as the projection leaves them, whose products need no lower term; with an activation they do."""
    from sparseengine_b200.csrc import ops
    tokens = kind.endswith("tokens")
    step = _step([3, 0, 11, 1, 7, 2, 5, 4, 9, 6])
    T, g = step.num_tokens, torch.Generator(device=DEV).manual_seed(d + heads)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    state = rnd(12, heads * d * dv + 5)
    first = state.double().clone()
    logs = -(torch.rand(T, heads, d, generator=g, device=DEV) * (30.0 if decay == "fast" else 0.2))
    o = torch.full((T, heads, dv), float("nan"), device=DEV)
    rep = heads // kv_heads
    sizes = dict(heads=heads, head_dim=d, v_head_dim=dv)
    column_major = not kind.startswith("retention")          # [head][column][row], retention [head][row][column]
    skip = None
    if not column_major:
        silu = kind == "retention"
        # columns: 4 that nobody reads, k, values, q; rotated where the head size allows the pairs
        wide, rot = heads * (2 * d + dv) + 8, 16 if d >= 16 else 0
        proj, decays = rnd(T, wide + -wide % 4).to(torch.bfloat16), torch.exp(logs[0, :, 0])
        inv, positions = torch.rand(rot // 2, generator=g, device=DEV), torch.arange(T, device=DEV, dtype=torch.int32) * 37 % 101
        v_off = 4 + heads * d
        q_off = v_off + heads * dv
        assert ops.retention_walk_supported(d, dv, rot, proj, q_off, 4, v_off)
        ops.retention_chunk(None, None, proj, v_off, decays, state, step, o.view(T, -1), silu=silu, **sizes,
                            qk=(q_off, 4, d ** -0.5), rotation=(inv, rot, positions) if rot else None)
        x = torch.nn.functional.silu(proj.double()) if silu else proj.double()
        q, k = (x[:, f:f + heads * d].reshape(T, heads, d).clone() for f in (q_off, 4))
        angle = (positions.float()[:, None] * inv).double()[:, None]        # the product in 32-bit, as positions are encoded
        for z in (q, k):
            lo, hi = z[..., :rot // 2].clone(), z[..., rot // 2:rot].clone()
            z[..., :rot // 2], z[..., rot // 2:rot] = lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin()
        k, v = k * d ** -0.5, x[:, v_off:v_off + heads * dv].view(T, heads, dv)
        keep, beta = decays.double().view(1, heads, 1).expand(T, -1, -1), None
    elif kind.startswith("state space"):
        width = heads * dv + 2 * kv_heads * d
        xbc, proj = rnd(T, width), rnd(T, heads + 3)
        bias, a_log, skip = rnd(heads) - 2.0, torch.log(torch.rand(heads, generator=g, device=DEV) * (30 if decay == "fast" else 1) + 0.1), rnd(heads)
        (ops.ssm_scan if tokens else ops.ssm_walk)(xbc, proj, 2, bias, a_log, skip, state, step, o.view(T, -1), heads=heads, head_dim=dv, state_size=d, groups=kv_heads)
        dt = torch.nn.functional.softplus(proj[:, 2:2 + heads].double() + bias.double())
        x = xbc[:, :heads * dv].double().view(T, heads, dv)
        k = xbc[:, heads * dv:heads * dv + kv_heads * d].view(T, kv_heads, d).repeat_interleave(rep, 1)
        q = xbc[:, heads * dv + kv_heads * d:].view(T, kv_heads, d).repeat_interleave(rep, 1)
        v, keep, beta = x * dt[..., None], torch.exp(-torch.exp(a_log.double()) * dt)[..., None], None
    else:
        per_head = kind == "delta, per head"
        qkv, proj, cols = rnd(T, 2 * kv_heads * d + heads * dv), rnd(T, heads + 4), heads * (1 if per_head else d)
        a, bias = rnd(T, cols + (-cols) % 4), rnd(cols) - 1.0
        a_log = torch.log(torch.rand(heads, generator=g, device=DEV) * (20 if decay == "fast" else 0.5) + 0.05)
        delta = dict(heads=heads, kv_heads=kv_heads, head_dim=d, v_head_dim=dv)
        inputs = dict(unit_eps=1e-6, q_scale=d ** -0.5, per_head=per_head)
        if tokens:
            made, dec, b = qkv.clone(), torch.empty(T, heads * d, device=DEV), torch.empty(T, heads, device=DEV)
            ops.delta_prep(made, a[:, :cols].contiguous(), proj, 2, bias, a_log, dec, b, **delta, **inputs)
            ops.delta_scan(made, dec, b, state, step, o.view(T, -1), **delta)
        else:
            ops.delta_walk(qkv, a, proj, 2, bias, a_log, state, step, o.view(T, -1), **delta, **inputs)
        qk = qkv[:, :2 * kv_heads * d].double().view(T, 2 * kv_heads, d)
        qk = qk / torch.sqrt((qk * qk).sum(-1, keepdim=True) + 1e-6)
        q, k = (t.repeat_interleave(rep, 1) for t in (qk[:, :kv_heads] * d ** -0.5, qk[:, kv_heads:]))
        v = qkv[:, 2 * kv_heads * d:].double().view(T, heads, dv)
        steps = torch.nn.functional.softplus(a[:, :cols].double() + bias.double()).view(T, heads, -1)
        keep, beta = torch.exp(-torch.exp(a_log.double())[:, None] * steps), torch.sigmoid(proj[:, 2:2 + heads].double())
    assert bool(torch.isfinite(o).all())
    for e, n in enumerate(LENS):
        a, b, row = step.cu[e], step.cu[e + 1], step.rows[e]
        S = first[row, :heads * d * dv].view(heads, *((dv, d) if column_major else (d, dv)))
        S = S.transpose(1, 2) if column_major else S
        want, S = _walk64(q[a:b].double(), k[a:b].double(), v[a:b], keep[a:b], S, None if beta is None else beta[a:b])
        if n == 0:
            assert torch.equal(state[row].double(), first[row])
            continue
        if skip is not None:
            want = want + skip.double()[:, None] * x[a:b]
        _close(o[a:b], want, f"outputs of {n} tokens")
        got = state[row, :heads * d * dv].view(heads, *((dv, d) if column_major else (d, dv)))
        _close(got.transpose(1, 2) if column_major else got, S, f"state after {n} tokens")
    others = [r for r in range(12) if r not in step.rows]
    assert torch.equal(state[others].double(), first[others]) and torch.equal(state[:, heads * d * dv:].double(), first[:, heads * d * dv:])


@pytest.mark.parametrize("kind", ["per head", "per channel"])
def test_later_tokens_do_not_touch_earlier_ones(kind):
    """A value that is not finite reaches the outputs of its own token and of later ones only."""
    from sparseengine_b200.csrc import ops
    H, d, T = 2, 64, 70
    step = SimpleNamespace(cu_q=torch.tensor([0, T], dtype=torch.int32, device=DEV), seq_rows=torch.zeros(1, dtype=torch.int32, device=DEV), num_seqs=1)
    g = torch.Generator(device=DEV).manual_seed(1)
    qkv, proj = torch.randn(T, 3 * H * d, generator=g, device=DEV), torch.randn(T, H, generator=g, device=DEV)
    cols = H * (1 if kind == "per head" else d)
    decay, bias, a_log = torch.randn(T, cols, generator=g, device=DEV), torch.zeros(cols, device=DEV), torch.zeros(H, device=DEV)
    outs = []
    for bad in (False, True):
        if bad:
            qkv[41, 2 * H * d + 3] = float("inf")
        o = torch.empty(T, H * d, device=DEV)
        ops.delta_walk(qkv, decay, proj, 0, bias, a_log, torch.zeros(1, H * d * d, device=DEV), step, o, heads=H, kv_heads=H, head_dim=d, v_head_dim=d,
                       unit_eps=1e-6, q_scale=0.1, per_head=kind == "per head")
        outs.append(o)
    assert torch.equal(outs[0][:41], outs[1][:41]) and not bool(torch.isfinite(outs[1][41:]).all())


def _one_entry(T):
    i32 = dict(dtype=torch.int32, device=DEV)
    return SimpleNamespace(cu_q=torch.tensor([0, T], **i32), seq_rows=torch.zeros(1, **i32), num_seqs=1, max_q_len=T, num_tokens=T)


def _inputs(kind, T, H, d):
    """What a kind of recurrence reads, and where its q, k, v and decay (or step) inputs of head 0 lie."""
    g = torch.Generator(device=DEV).manual_seed(1)
    cols = H * (d if kind == "delta, per channel" else 1)
    x = {"qkv": torch.randn(T, 3 * H * d, generator=g, device=DEV), "decay": torch.randn(T, cols, generator=g, device=DEV),
         "beta": torch.randn(T, H, generator=g, device=DEV), "bias": torch.zeros(cols, device=DEV), "a_log": torch.zeros(H, device=DEV),
         "skip": torch.ones(H, device=DEV)}
    q, k, v = (2 * H * d, H * d, 0) if kind == "state space" else (0, H * d, 2 * H * d)       # there: values, keys, queries
    return x, {"q": ("qkv", q + 3), "k": ("qkv", k + 3), "v": ("qkv", v + 3), "decay": ("decay", 0)}


def _outputs(kind, x, H, d, tokens=False, one_kernel=False):
    """Outputs and the state after them, from a state of zeros; ``tokens``: by the kernels that walk token by token; ``one_kernel``:
    by the delta rule's other chunked form."""
    from sparseengine_b200.csrc import ops
    T = x["qkv"].shape[0]
    step, o, state = _one_entry(T), torch.empty(T, H * d, device=DEV), torch.zeros(1, H * d * d, device=DEV)
    if kind == "state space":
        (ops.ssm_scan if tokens else ops.ssm_walk)(x["qkv"], x["decay"], 0, x["bias"], x["a_log"], x["skip"], state, step, o, heads=H,
                                                   head_dim=d, state_size=d, groups=H)
    elif kind.startswith("retention"):
        qkv = x["qkv"].to(torch.bfloat16) if kind.endswith("16-bit values") else x["qkv"]
        ops.retention_chunk(None, None, qkv, 2 * H * d, torch.full((H,), 0.9, device=DEV), state, step, o, heads=H, head_dim=d,
                            v_head_dim=d, qk=(0, H * d, 1.0))
    else:
        sizes = dict(heads=H, kv_heads=H, head_dim=d, v_head_dim=d)
        inputs = dict(unit_eps=1e-6, q_scale=0.1, per_head=kind == "delta, per head")
        if tokens or one_kernel:
            log_dec = torch.empty(T, H, device=DEV) if one_kernel else None
            qkv, dec, beta = x["qkv"].clone(), torch.empty(T, H * d, device=DEV), torch.empty(T, H, device=DEV)
            ops.delta_prep(qkv, x["decay"], x["beta"], 0, x["bias"], x["a_log"], dec, beta, **sizes, **inputs, log_dec=log_dec)
            if one_kernel:
                ops.delta_chunk(qkv, log_dec, beta, state, step, o, **sizes)
            else:
                ops.delta_scan(qkv, dec, beta, state, step, o, **sizes)
        else:
            ops.delta_walk(x["qkv"], x["decay"], x["beta"], 0, x["bias"], x["a_log"], state, step, o, **sizes, **inputs)
    return o, state


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("token", [40, 41, 63])         # the first and the second of a pair of tokens, the last of a chunk
@pytest.mark.parametrize("where", ["q", "k", "v", "decay"])
@pytest.mark.parametrize("kind", ["state space", "delta, per head", "delta, per channel", "retention", "retention, 16-bit values"])
def test_inputs_that_are_not_finite_stay_with_their_token_and_later_ones(kind, where, token, value):
    if kind.startswith("retention") and where == "decay":
        pytest.skip("its decays are constants")
    H, d, T = 2, 64, 70
    x, places = _inputs(kind, T, H, d)
    want, _ = _outputs(kind, x, H, d)
    name, column = places[where]
    x[name][token, column] = value
    got, _ = _outputs(kind, x, H, d)
    assert torch.equal(got[:token], want[:token])
    assert torch.equal(got[:, d:], want[:, d:])                  # the other head
    if where == "q":
        assert not bool(torch.isfinite(got[token, :d]).any()) and torch.equal(got[token + 1:], want[token + 1:])
    elif where != "decay" or value != value:                     # an infinite step may be a decay of 0
        assert not bool(torch.isfinite(got[token:, :d]).all(1).any())


@pytest.mark.parametrize("what", ["rate", "some steps", "all but forgotten"])
@pytest.mark.parametrize("kind", ["state space", "delta, per head", "delta, per channel", "delta in one kernel"])
def test_decays_of_zero(kind, what):
    """Decays that are exactly 0 in 32-bit, from an infinite rate, from infinite steps (the delta rules; a state space takes its step
    as a factor too) or from rates of e^80: what the kernels give that walk token by token."""
    H, d, T = 2, 64, 150
    one_kernel = kind == "delta in one kernel"
    kind = "delta, per head" if one_kernel else kind
    x, _ = _inputs(kind, T, H, d)
    if what == "some steps":
        if kind == "state space":
            pytest.skip("outputs are infinite")
        x["decay"][[0, 17, 40, 41, 64, 149]] = float("inf")
    else:
        x["a_log"][1] = 90.0 if what == "rate" else 80.0
    (got, state), (want, last) = (_outputs(kind, x, H, d, tokens=tokens, one_kernel=one_kernel and not tokens) for tokens in (False, True))
    assert bool(torch.isfinite(want).all() and torch.isfinite(last).all())
    _close(got, want.double(), "outputs")
    _close(state, last.double(), "state")


@pytest.mark.parametrize("kind", ["delta", "retention"])
def test_parameters_off_16_bytes(kind):
    """A decay bias or rotation frequencies that are views off 16 bytes: what the same numbers give on 16 bytes."""
    from sparseengine_b200.config.specs import GatedDeltaSpec, RetentionSpec, RotarySpec
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.base import LayerSlot, make_mixer
    from sparseengine_b200.parts.position import as_rotary_args
    T, width, heads, d = 70, 64, 2, 16
    if kind == "delta":
        spec = GatedDeltaSpec(hidden_size=width, num_heads=heads, num_kv_heads=heads, head_dim=d, v_head_dim=d, conv_taps=4, decay_per="channel",
                              gate_activation="sigmoid", decay_rank=8, gate_rank=8)
    else:
        spec = RetentionSpec(hidden_size=width, num_heads=heads, head_dim=d, v_head_dim=d, decays=(0.9, 0.99), position=RotarySpec(rotary_dim=d, theta=1e4))
    step = _one_entry(T)
    step.token_seq, step.positions = torch.zeros(T, dtype=torch.int32, device=DEV), torch.arange(T, dtype=torch.int32, device=DEV)

    def odd(t):
        store = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
        store[1:] = t.flatten()
        return store[1:].view(t.shape)

    outs, walks = [], []
    for off in (False, True):
        part, g = make_mixer(spec, torch.float32), torch.Generator(device=DEV).manual_seed(1)
        tensors = {n: torch.randn(p.shape, generator=g, device=DEV) * 0.3 for n, p in part.parameters().items()}
        x = torch.randn(T, width, generator=g, device=DEV)
        if off and kind == "delta":
            tensors["dt_bias"] = odd(tensors["dt_bias"])
        part.bind(tensors)
        if off and kind == "retention":
            inv = odd(as_rotary_args(part.position.kernel_args(torch.device(DEV))).inv_freq)
            part.position.kernel_args = lambda device: (inv, d, 1.0)
        before = sum(ops.calls.get(n, 0) for n in ("se_delta_walk", "se_retention_prep"))
        outs.append(part.forward(x, step, LayerSlot(state=torch.zeros(1, *part.state_request().shape, device=DEV))))
        walks.append(sum(ops.calls.get(n, 0) for n in ("se_delta_walk", "se_retention_prep")) - before)
    assert walks == ([1, 0] if kind == "delta" else [0, 1])
    _close(outs[1], outs[0].double(), "outputs")


def test_head_sizes_that_the_walk_does_not_take():
    """A delta rule with one decay per head and a head size that is no multiple of four: a prompt goes through the kernel that does
    a chunk at a time, and gives what it gives token by token."""
    from sparseengine_b200.config.specs import GatedDeltaSpec
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.base import LayerSlot, make_mixer
    spec = GatedDeltaSpec(hidden_size=64, num_heads=2, num_kv_heads=1, head_dim=18, v_head_dim=16, conv_taps=3, decay_per="head", gate_activation="silu")
    T = 150
    step = _one_entry(T)
    step.token_seq = torch.zeros(T, dtype=torch.int32, device=DEV)
    outs, chunks = [], []
    for least in (None, 48):
        part, g = make_mixer(spec, torch.float32), torch.Generator(device=DEV).manual_seed(2)
        part.bind({n: torch.randn(p.shape, generator=g, device=DEV) * 0.3 for n, p in part.parameters().items()})
        part.chunk_min_tokens = least
        state, before = torch.zeros(1, *part.state_request().shape, device=DEV), ops.calls.get("se_delta_chunk", 0)
        outs.append((part.forward(torch.randn(T, 64, generator=g, device=DEV), step, LayerSlot(state=state)), state))
        chunks.append(ops.calls.get("se_delta_chunk", 0) - before)
    assert chunks == [0, 1]
    _close(outs[1][0], outs[0][0].double(), "outputs")
    _close(outs[1][1], outs[0][1].double(), "state")
