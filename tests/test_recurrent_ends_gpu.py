"""What stands around the linear recurrences (convolution, rotation, gated norms) against 64-bit equations: sizes that the
kernels which move 8 or 16 bytes at a time take, at their edges, and sizes that they leave to the general ones."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def rnd(*shape, seed=0, dtype=torch.float32):
    return torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed + shape[0]), device=DEV).to(dtype)


def close(got, want, dtype):
    """32-bit: a dozen roundings; 16-bit: one rounding of the result (and a fast exponential)."""
    assert got.dtype == dtype or got.dtype == torch.float32
    bound = 3e-6 if got.dtype == torch.float32 else 4.5e-3
    assert float(((got.double() - want).abs() / want.abs().clamp(min=1.0)).max()) < bound


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("lens", [[1, 1, 1], [40], [3, 1, 17, 2, 9, 8]])
@pytest.mark.parametrize("C,off,taps", [(4, 0, 4), (516, 8, 4), (512, 4, 4), (6, 0, 4), (20, 3, 4), (16, 0, 5)])
def test_convolution(C, off, taps, lens, dtype):
    from sparseengine_b200.csrc import ops
    T = sum(lens)
    pitch = off + C + (-(off + C) % 4)
    x, w, b = rnd(T, pitch, seed=1, dtype=dtype), rnd(C, taps, seed=2), rnd(C, seed=3)
    conv_off = 8
    state = rnd(len(lens) + 1, conv_off + (taps - 1) * C, seed=4)
    held = state.double().clone()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    rows = list(range(len(lens), 0, -1))
    step = SimpleNamespace(token_seq=torch.tensor([e for e, n in enumerate(lens) for _ in range(n)], **i32), cu_q=torch.tensor(cu, **i32),
                           seq_rows=torch.tensor(rows, **i32), num_seqs=len(lens), max_q_len=max(lens))
    out = torch.full((T, C), float("nan"), device=DEV)
    ops.causal_conv(x, off, w, b, state, conv_off, step, out)
    for e, n in enumerate(lens):
        before = held[rows[e], conv_off:].view(taps - 1, C)
        full = torch.cat([before, x[cu[e]:cu[e + 1], off:off + C].double()])
        want = sum(full[j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
        close(out[cu[e]:cu[e + 1]], torch.nn.functional.silu(want), dtype)
        assert torch.equal(state[rows[e], conv_off:].view(taps - 1, C).double(), full[n:])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dv", [(1, 4), (3, 128), (2, 132), (5, 256), (2, 260), (3, 30)])
def test_delta_output(heads, dv, dtype):
    from sparseengine_b200.csrc import ops
    T = 9
    o, w, gate = rnd(T, heads * dv, seed=1), rnd(dv, seed=2), rnd(T, heads * dv + 8, seed=3, dtype=dtype)[:, 4:4 + heads * dv]
    for silu in (False, True):
        out = torch.empty(T, heads * dv, dtype=dtype, device=DEV)
        ops.delta_out(o, gate, w, out, heads=heads, v_head_dim=dv, eps=1e-6, silu=silu)
        v, g = o.double().view(T, heads, dv), gate.double().view(T, heads, dv)
        want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6) * w.double() * torch.sigmoid(g) * (g if silu else 1.0)
        close(out.view(T, heads, dv), want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("parts,n,off", [(3, 4, 0), (1, 128, 4), (2, 132, 4), (2, 1028, 8), (1, 4096, 4), (1, 4100, 0), (2, 30, 2)])
def test_gated_group_norm(parts, n, off, dtype):
    from sparseengine_b200.csrc import ops
    T, inner = 5, parts * n
    y, w, proj = rnd(T, inner, seed=1), rnd(inner, seed=2), rnd(T, inner + 8, seed=3, dtype=dtype)
    out = torch.empty(T, inner, dtype=dtype, device=DEV)
    ops.gated_group_norm(y, proj, off, w, out, parts=parts, eps=1e-6)
    v = (y.double() * torch.nn.functional.silu(proj[:, off:off + inner].double())).view(T, parts, n)
    close(out, (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6)).view(T, inner) * w.double(), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("parts,n,off", [(1, 4, 0), (3, 508, 4), (1, 512, 0), (7, 512, 8), (1, 516, 4)])
def test_gated_group_norm_by_warps(parts, n, off, dtype):
    """Around the 512 columns that a warp takes, with warps of the last block that have no part."""
    test_gated_group_norm(parts, n, off, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,d,rot,off,silu", [(1, 16, 16, 0, False), (3, 24, 16, 8, True), (40, 128, 128, 0, False), (2, 128, 64, 8, True),
                                                  (2, 20, 16, 0, False), (2, 32, 24, 0, True), (2, 32, 32, 4, False)])
def test_retention_preparation_and_output(heads, d, rot, off, silu, dtype):
    from sparseengine_b200.csrc import ops
    T, n = 7, heads * d
    proj = rnd(T, 3 * n + off + (-(3 * n + off)) % 8, seed=1, dtype=dtype)
    inv = torch.rand(rot // 2, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV) * 3
    q32, k32 = torch.empty(T, n, device=DEV), torch.empty(T, n, device=DEV)
    ops.retention_prep(proj, off, off + n, inv, pos, q32, k32, heads=heads, head_dim=d, rotary_dim=rot, k_scale=0.3, silu=silu)
    ang = (pos[:, None].float() * inv).double()
    cs, sn = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    for got, at, f in ((q32, off, 1.0), (k32, off + n, 0.3)):
        x = proj[:, at:at + n].double().view(T, heads, d)
        x = torch.nn.functional.silu(x) if silu else x
        u, v = x[..., :rot // 2], x[..., rot // 2:rot]
        close(got.view(T, heads, d), f * torch.cat([u * cs - v * sn, v * cs + u * sn, x[..., rot:]], -1), dtype)
    o, out = rnd(T, n, seed=4), torch.empty(T, n, dtype=dtype, device=DEV)
    ops.retention_out(o, proj, off + 2 * n, out, heads=heads, v_head_dim=d, eps=1e-6)
    v = o.double().view(T, heads, d)
    want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6) * torch.nn.functional.silu(proj[:, off + 2 * n:off + 3 * n].double()).view(T, heads, d)
    close(out.view(T, heads, d), want, dtype)
