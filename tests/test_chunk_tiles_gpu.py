"""Linear recurrences by chunks of 128 tokens side by side (csrc/chunk_tiles.cuh) against 64-bit walks token by token, from non-zero states, with entries that
end on, before and behind the chunks' edges."""
from types import SimpleNamespace

import pytest
import torch

from test_chunk_walk_gpu import _close, _walk64

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    rows = [(3 * i + 1) % (len(lens) + 2) for i in range(len(lens))] if len(lens) % 3 != 1 else list(range(len(lens)))
    return SimpleNamespace(cu_q=torch.tensor(cu, **i32), seq_rows=torch.tensor(rows, **i32), num_seqs=len(lens), num_tokens=cu[-1],
                           max_q_len=max(lens), cu=cu, rows=rows)


def _retention(lens, heads, rotary, decay, bad=None, out=False, known=None, positive=False, walk=False):
    """``walk``: by the chunks of 64 tokens one after another (csrc/retention.cu) instead."""
    from sparseengine_b200.csrc import ops
    d, step = 128, _step(lens)
    step.max_q_len = known or step.max_q_len
    T, g = step.num_tokens, torch.Generator(device=DEV).manual_seed(heads)
    proj = torch.randn(T, 8 + 4 * heads * d, generator=g, device=DEV).to(torch.bfloat16)      # v, 8 columns that nobody reads, k, q, gate
    v_off, k_off, q_off, g_off = 0, heads * d + 8, 2 * heads * d + 8, 3 * heads * d + 8
    decays = torch.exp(-torch.rand(heads, generator=g, device=DEV) * (20.0 if decay == "fast" else 0.03))
    state = torch.randn(len(lens) + 2, heads * d * d + 4, generator=g, device=DEV)
    inv, positions = torch.rand(64, generator=g, device=DEV), torch.arange(T, device=DEV, dtype=torch.int32) * 37 % 101
    if positive:
        proj, state = proj.abs(), state.abs()
    if bad is not None:
        proj[bad[0], {"q": q_off, "k": k_off, "v": v_off}[bad[1]] + 5] = bad[2]
    first = state.clone()
    assert ops.retention_tiles_supported(d, d, rotary, proj, state, q_off, k_off, v_off, g_off)
    to = dict(out=torch.empty(T, heads * d, dtype=torch.bfloat16, device=DEV)) if out else dict(o=torch.full((T, heads * d), float("nan"), device=DEV))
    rotation = (inv, rotary, positions) if rotary else None
    if walk:
        got = ops.retention_chunk(None, None, proj, v_off, decays, state, step, to["o"], heads=heads, head_dim=d, v_head_dim=d,
                                  qk=(q_off, k_off, d ** -0.5), rotation=rotation)
    else:
        got = ops.retention_tiles(proj, q_off, k_off, v_off, g_off, d ** -0.5, rotation, decays, state, step, heads=heads, head_dim=d, v_head_dim=d,
                                  eps=1e-6, **to)
    ops.error_check(DEV)
    q, k, v = (proj[:, f:f + heads * d].double().view(T, heads, d) for f in (q_off, k_off, v_off))
    if rotary:
        a = (positions.float()[:, None] * inv).double()[:, None]
        q, k = (torch.cat([x[..., :64] * a.cos() - x[..., 64:] * a.sin(), x[..., 64:] * a.cos() + x[..., :64] * a.sin()], -1) for x in (q, k))
    return step, got, first, state, (q, k * d ** -0.5, v, decays.double().view(1, heads, 1).expand(T, -1, -1)), proj[:, g_off:]


@pytest.mark.parametrize("decay", ["slow", "fast"])
@pytest.mark.parametrize("rotary", [0, 128])
@pytest.mark.parametrize("lens,heads", [([1, 127, 128, 129, 0, 300, 64, 17], 3), ([1500], 2), ([257], 40)])       # the second: several segments of chunks
def test_retention_against_the_walk(lens, heads, rotary, decay):
    step, o, first, state, inputs, _ = _retention(lens, heads, rotary, decay)
    d = 128
    for e, n in enumerate(lens):
        a, b, row = step.cu[e], step.cu[e + 1], step.rows[e]
        if n == 0:
            assert torch.equal(state[row], first[row])
            continue
        want, S = _walk64(*(x[a:b] for x in inputs), first[row, :heads * d * d].double().view(heads, d, d))
        _close(o[a:b].view(n, heads, d), want, f"outputs of {n} tokens")
        _close(state[row, :heads * d * d].view(heads, d, d), S, f"state after {n} tokens")
    others = [r for r in range(len(lens) + 2) if r not in step.rows]
    assert torch.equal(state[others], first[others]) and torch.equal(state[:, heads * d * d:], first[:, heads * d * d:])


def _norm_error(got, want):
    return float((got.double() - want).norm() / want.norm())


# Values of one sign: a step of tensor memory cuts off up to a unit of the 24th bit of the sum so far, always towards zero: half on average, of sums that are
# half of the last one on average.  Four steps in either part of a product, two products behind one another: 8 x 2^-26, and what 32-bit rounding leaves.
ONE_SIGN = 1.5e-7


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("rotary", [0, 128])
@pytest.mark.parametrize("n", [128, 700])
def test_retention_is_as_exact_as_the_walk(n, rotary, positive):
    errors = []
    for walk in (False, True):
        _, o, first, state, inputs, _ = _retention([n], 4, rotary, "slow", positive=positive, walk=walk)
        want, S = _walk64(*inputs, first[0, :4 * 128 * 128].double().view(4, 128, 128))
        errors.append((_norm_error(o.view(n, 4, 128), want), _norm_error(state[0, :4 * 128 * 128].view(4, 128, 128), S)))
    for here, walked in zip(*errors):
        assert here <= (max(walked, ONE_SIGN) if positive else walked), errors


@pytest.mark.parametrize("lens,known", [([1500, 40], 300), ([900], 60)])
def test_retention_of_entries_longer_than_the_host_knows(lens, known):
    """What a captured step meets when it is replayed with the same tokens in other entries."""
    step, o, first, state, inputs, _ = _retention(lens, 2, 128, "slow", known=known)
    for e, n in enumerate(lens):
        a, b, row = step.cu[e], step.cu[e + 1], step.rows[e]
        want, S = _walk64(*(x[a:b] for x in inputs), first[row, :2 * 128 * 128].double().view(2, 128, 128))
        _close(o[a:b].view(n, 2, 128), want, f"outputs of {n} tokens")
        _close(state[row, :2 * 128 * 128].view(2, 128, 128), S, f"state after {n} tokens")


def test_retention_with_norm_and_gate():
    _, o, _, _, _, gate = _retention([200, 5], 2, 128, "slow")
    _, y, _, _, _, _ = _retention([200, 5], 2, 128, "slow", out=True)
    o = o.double().view(-1, 2, 128)
    want = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)).view(-1, 256) * torch.nn.functional.silu(gate.double())
    # rounded to the nearest of 8 bits: half a step is at most 2^-8 of the value; the 32-bit value before it 1e-5 (the gate's fast exponential and quotient)
    assert bool(((y.double() - want).abs() <= want.abs() * (2.0 ** -8 + 1e-5) + 1e-30).all())


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("out", [False, True])
def test_retention_inputs_that_are_not_finite_stay_with_their_token_and_later_ones(where, value, out):
    """Token 150 of 400: the second of four chunks, head 0 of two."""
    lens, t = [400], 150
    _, want, _, s_want, _, _ = _retention(lens, 2, 128, "slow", out=out)
    _, got, _, s_got, _, _ = _retention(lens, 2, 128, "slow", bad=(t, where, value), out=out)
    want, got = want.float(), got.float()
    # its chunk is done again token by token: another order of the same sums, within a step of what is stored
    near = dict(rtol=2.0 ** -7 if out else 1e-4, atol=1e-4)
    assert torch.equal(got[:128], want[:128]) and torch.equal(got[:, 128:], want[:, 128:])
    torch.testing.assert_close(got[128:t], want[128:t], **near)
    if where == "q":
        assert not bool(torch.isfinite(got[t, :128]).any())
        torch.testing.assert_close(got[t + 1:], want[t + 1:], **near)
        assert torch.equal(s_got, s_want)
    else:
        assert not bool(torch.isfinite(got[t:, :128]).all(1).any()) and not bool(torch.isfinite(s_got[0, :128 * 128]).all())
        assert torch.equal(s_got[0, 128 * 128:], s_want[0, 128 * 128:])


# more items (chunks and heads) than two for each SM: a block's loop goes on to other chunks of other heads, past places without a token
MANY = [([2500], 16), ([130, 0, 257, 1, 64] * 5, 16)]


@pytest.mark.parametrize("lens,heads", MANY)
def test_retention_blocks_of_several_items(lens, heads):
    from sparseengine_b200.csrc import ops
    assert (sum(lens) // 128 + len(lens)) * heads > 2 * ops.sm_count(DEV)
    step, o, first, state, inputs, gate = _retention(lens, heads, 128, "slow")
    for e, n in enumerate(lens):
        a, b, row = step.cu[e], step.cu[e + 1], step.rows[e]
        if n == 0:
            assert torch.equal(state[row], first[row])
            continue
        want, S = _walk64(*(x[a:b] for x in inputs), first[row, :heads * 128 * 128].double().view(heads, 128, 128))
        _close(o[a:b].view(n, heads, 128), want, f"outputs of {n} tokens")
        _close(state[row, :heads * 128 * 128].view(heads, 128, 128), S, f"state after {n} tokens")
    _, y, _, state2, _, _ = _retention(lens, heads, 128, "slow", out=True)
    assert torch.equal(state2, state)
    o = o.double().view(-1, heads, 128)
    want = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)).view(len(o), -1) * torch.nn.functional.silu(gate.double())
    assert bool(((y.double() - want).abs() <= want.abs() * (2.0 ** -8 + 1e-5) + 1e-30).all())       # as in the test of norm and gate


@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("out", [False, True])
def test_retention_goes_on_behind_a_chunk_that_is_done_again(where, out):
    """Token 150 of 2,500, head 0 of 16: the block that does its chunk again has fetched another chunk of another head meanwhile, which it fetches again."""
    (lens, heads), t = MANY[0], 150
    _, want, _, s_want, _, _ = _retention(lens, heads, 128, "slow", out=out)
    _, got, _, s_got, _, _ = _retention(lens, heads, 128, "slow", bad=(t, where, float("nan")), out=out)
    assert torch.equal(got[:, 128:], want[:, 128:]) and torch.equal(s_got[:, 128 * 128:], s_want[:, 128 * 128:])
    assert torch.equal(got[:128, :128], want[:128, :128]) and not bool(torch.isfinite(got[t, :128].float()).all())
    if where == "q":
        assert torch.equal(got[256:, :128], want[256:, :128]) and torch.equal(s_got, s_want)
    else:
        assert not bool(torch.isfinite(got[t:, :128].float()).all(1).any())


def test_retention_mixer_keeps_to_the_other_forms_beyond_its_workspace():
    from sparseengine_b200.config.specs import RetentionSpec
    from sparseengine_b200.parts.base import make_mixer
    part = make_mixer(RetentionSpec(hidden_size=64, num_heads=32, head_dim=128, v_head_dim=128, decays=(0.9,) * 32, position=None), torch.bfloat16)
    few, many = (SimpleNamespace(num_seqs=n, max_q_len=20) for n in (64, 512))
    assert part.in_tiles(few, 20 + 63, 0, DEV) and not part.in_tiles(many, 20 + 511, 0, DEV)


@pytest.mark.parametrize("norm", ["per_head", "joint"])
def test_retention_mixer_through_the_chunks(norm):
    """Both output norms against the other forms; and beside what the step needs nothing as large as 32-bit outputs is held where the kernel norms them."""
    from sparseengine_b200.config.specs import RetentionSpec
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.base import LayerSlot, make_mixer
    heads, T, width = 4, 8192, 64
    part = make_mixer(RetentionSpec(hidden_size=width, num_heads=heads, head_dim=128, v_head_dim=128, decays=(0.99,) * heads, position=None, output_norm=norm),
                      torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(1)
    part.bind({name: (torch.randn(*p.shape, generator=g, device=DEV) * 0.05).to(torch.bfloat16) for name, p in part.parameters().items()})
    x, step, ys = torch.randn(T, width, generator=g, device=DEV).to(torch.bfloat16), _step([T]), []
    step.positions = torch.arange(T, dtype=torch.int32, device=DEV)
    for least in (16, None):                         # the chunks side by side; token by token
        part.chunk_min_tokens = least
        slot = LayerSlot(state=torch.zeros(3, heads * 128 * 128, device=DEV))
        for _ in range(2):                           # the second call's memory: what the library keeps is there
            slot.state.zero_()
            before, calls = torch.cuda.memory_allocated(), ops.calls.get("se_retention_tiles", 0)
            torch.cuda.reset_peak_memory_stats()
            y = part.forward(x, step, slot)
            held = torch.cuda.max_memory_allocated() - before
        assert ops.calls.get("se_retention_tiles", 0) - calls == (least is not None)
        if least is not None and norm == "per_head":
            vv = heads * 128
            needed = T * 4 * vv * 2 + T * vv * 2 + 4 * ops.retention_tiles_plan(step, T, heads, 0, DEV)[2] + T * width * 2
            assert held < needed + T * vv * 2, (held, needed)        # columns, outputs after the norm, workspace, result; no 32-bit outputs
        ys.append((y.double(), slot.state[0].double()))
    ops.error_check(DEV)
    # outputs after the norm are 16-bit in both, rounded at different values at times: 2^-8 of a value, in sums over 512 of either sign
    assert float((ys[0][0] - ys[1][0]).norm() / ys[1][0].norm()) < 2.0 ** -8
    assert float((ys[0][1] - ys[1][1]).norm() / ys[1][1].norm()) < 1e-6


def _state_space(lens, heads, groups, decay, bad=None, positive=False, walk=False, per=None):
    from sparseengine_b200.csrc import ops
    P, N, step = 64, 128, _step(lens)
    T, g = step.num_tokens, torch.Generator(device=DEV).manual_seed(heads)
    xbc = torch.randn(T, heads * P + 2 * groups * N, generator=g, device=DEV)
    proj = torch.randn(T, heads + 5, generator=g, device=DEV).to(torch.bfloat16)
    bias, skip = torch.randn(heads, generator=g, device=DEV) - 2.0, torch.randn(heads, generator=g, device=DEV)
    a_log = torch.log(torch.rand(heads, generator=g, device=DEV) * (30 if decay == "fast" else 1) + 0.1)
    state = torch.randn(len(lens) + 2, heads * P * N + 4, generator=g, device=DEV)
    if positive:
        xbc, skip, state = xbc.abs(), skip.abs(), state.abs()
    if bad is not None:
        t, where, value = bad
        if where == "dt":
            proj[t, 3] = value
        else:
            xbc[t, {"v": 5, "k": heads * P + 5, "q": heads * P + groups * N + 5}[where]] = value
    first, y = state.clone(), torch.full((T, heads * P), float("nan"), device=DEV)
    assert ops.ssm_tiles_supported(N, P, proj, state)
    (ops.ssm_walk if walk else ops.ssm_tiles)(xbc, proj, 3, bias, a_log, skip, state, step, y, heads=heads, head_dim=P, state_size=N, groups=groups,
                                                **({} if walk else {"heads_per_block": per}))
    ops.error_check(DEV)
    dt = torch.nn.functional.softplus(proj[:, 3:3 + heads].double() + bias.double())
    x, rep = xbc[:, :heads * P].double().view(T, heads, P), heads // groups
    k, q = (c.double().reshape(T, groups, N).repeat_interleave(rep, 1) for c in xbc[:, heads * P:].split(groups * N, 1))
    return step, y, first, state, (q, k, x * dt[..., None], torch.exp(-torch.exp(a_log.double()) * dt)[..., None]), skip.double()[:, None] * x


# heads a block: one, five of a group of nine, eight and three more
@pytest.mark.parametrize("decay", ["slow", "fast"])
@pytest.mark.parametrize("lens,heads,groups", [([1, 127, 128, 129, 0, 300, 64, 17], 4, 4), ([513], 18, 2), ([130] * 64, 11, 1)])
def test_state_space_against_the_walk(lens, heads, groups, decay):
    step, y, first, state, inputs, add = _state_space(lens, heads, groups, decay)
    P, N = 64, 128
    for e, n in enumerate(lens):
        a, b, row = step.cu[e], step.cu[e + 1], step.rows[e]
        if n == 0:
            assert torch.equal(state[row], first[row])
            continue
        if e > 8:                                    # 64 equal ones: the first few and the last
            if e != len(lens) - 1:
                continue
        want, S = _walk64(*(x[a:b] for x in inputs), first[row, :heads * P * N].double().view(heads, P, N).transpose(1, 2))
        _close(y[a:b].view(n, heads, P), want + add[a:b], f"outputs of {n} tokens")
        _close(state[row, :heads * P * N].view(heads, P, N).transpose(1, 2), S, f"state after {n} tokens")
    others = [r for r in range(len(lens) + 2) if r not in step.rows]
    assert torch.equal(state[others], first[others]) and torch.equal(state[:, heads * P * N:], first[:, heads * P * N:])


@pytest.mark.parametrize("lens,heads,groups", [([130, 1, 0, 300], 11, 1), ([200], 12, 3)])
def test_state_space_is_the_same_with_any_number_of_heads_a_block(lens, heads, groups):
    runs = [_state_space(lens, heads, groups, "slow", per=per) for per in (None, 1, 3, 8)]
    for _, y, _, state, _, _ in runs[1:]:
        assert torch.equal(y, runs[0][1]) and torch.equal(state, runs[0][3])


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("decay", ["slow", "fast"])
@pytest.mark.parametrize("n", [128, 700])
def test_state_space_is_as_exact_as_the_walk(n, decay, positive):
    errors = []
    for walk in (False, True):
        _, y, first, state, inputs, add = _state_space([n], 4, 2, decay, positive=positive, walk=walk)
        want, S = _walk64(*inputs, first[0, :4 * 64 * 128].double().view(4, 64, 128).transpose(1, 2))
        errors.append((_norm_error(y.view(n, 4, 64), want + add), _norm_error(state[0, :4 * 64 * 128].view(4, 64, 128).transpose(1, 2), S)))
    for here, walked in zip(*errors):
        assert here <= (max(walked, ONE_SIGN) if positive else walked), errors


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["q", "k", "v", "dt"])
def test_state_space_inputs_that_are_not_finite_stay_with_their_token_and_later_ones(where, value):
    """Token 150 of 400: the second of four chunks, the first of two groups of two heads (of v and dt its first head)."""
    t, P = 150, 64
    _, want, _, s_want, _, _ = _state_space([400], 4, 2, "slow")
    _, got, _, s_got, _, _ = _state_space([400], 4, 2, "slow", bad=(t, where, value))
    own = P if where in ("v", "dt") else 2 * P       # columns that it may reach
    near = dict(rtol=1e-4, atol=1e-4)                # its chunk is done again token by token: another order of the same sums
    assert torch.equal(got[:128], want[:128]) and torch.equal(got[:, own:], want[:, own:])
    torch.testing.assert_close(got[128:t], want[128:t], **near)
    if where == "q":
        assert not bool(torch.isfinite(got[t, :own]).any())
        torch.testing.assert_close(got[t + 1:], want[t + 1:], **near)
        assert torch.equal(s_got, s_want)
    else:                                            # also of an infinite step, whose decay is 0: what the token adds is not finite
        assert not bool(torch.isfinite(got[t:, :own]).all(1).any()) and not bool(torch.isfinite(s_got[0, :own * 128]).all())
        assert torch.equal(s_got[0, own * 128:], s_want[0, own * 128:])


def test_state_space_mixer_chooses_by_both_estimates():
    from sparseengine_b200.config.specs import StateSpaceSpec
    from sparseengine_b200.parts.base import make_mixer
    part = make_mixer(StateSpaceSpec(hidden_size=64, num_heads=64, head_dim=64, state_size=128, groups=8, conv_taps=4, norm_groups=8), torch.bfloat16)

    def asked(lens):
        return part.in_tiles(SimpleNamespace(num_seqs=len(lens), max_q_len=max(lens), num_tokens=sum(lens), q_lens=lens), DEV)
    assert asked([2048]) and asked([60] * 4) and asked([40] * 64) and not asked([20] * 64) and not asked([90] + [1] * 63)
    assert not asked([17]) and not asked([100] * 200)        # the last: its states would take 419 MB
    part.chunk_min_tokens = None
    assert not asked([2048])
