"""Decode attention whose blocks start with the longest contexts, against the plain paged attention of the library."""
import pytest
import torch

from test_kernels_gpu import _cache_setup, rnd

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("lens,hq,hkv,page,options", [
    ([3000, 1, 63, 64, 65, 1700] + [500 + 37 * i for i in range(58)], 48, 8, 16, {}),
    ([1600] * 50 + [20] * 14, 40, 8, 16, {"sink": True, "softcap": 30.0}),       # equals keep their order
    ([1 + 6 * i for i in range(256)], 10, 2, 5, {"window": 300, "keep_first": 40})])       # the most tokens that are sorted
def test_sorted_blocks_against_the_plain_kernel(lens, hq, hkv, page, options):
    from sparseengine_b200.csrc import ops
    d, t, dtype = 128, len(lens), torch.bfloat16
    table, rows, _, _, cache = _cache_setup(lens, hkv, d, page, dtype)
    cache.copy_(torch.randn(cache.shape, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV))
    q = rnd(t, hq, d, dtype=dtype, seed=7)
    positions = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    token_seq = torch.arange(t, dtype=torch.int32, device=DEV)
    args = (q.view(t, hq * d), cache, table, rows, token_seq, positions)
    sizes = dict(num_heads=hq, num_kv_heads=hkv, head_dim=d, page_size=page, scale=d ** -0.5, **options)
    splits, _ = ops.attn_decode_plan(t, hq, hkv, max(lens))
    assert ops.attn_decode_sorted(t, hq, hkv, max(lens), splits, ops.sm_count(DEV))
    out, plain = (torch.empty_like(q).view(t, hq * d) for _ in range(2))
    ops.attn_decode(*args, out, max_keys=max(lens), **sizes)
    ops.paged_attention_plain(*args, plain, **sizes)
    # weights rounded to bfloat16 (2^-9) against unrounded ones, both rounded to bfloat16: values of order one, as the split kernel's bound
    torch.testing.assert_close(out.float(), plain.float(), atol=2e-2, rtol=2e-2)


def test_choice():
    from sparseengine_b200.csrc import ops
    ask = ops.attn_decode_sorted
    assert ask(64, 48, 8, 3001, 1, 148) and not ask(64, 48, 8, 3001, 2, 148) and not ask(64, 48, 8, 1000, 1, 148)
    assert not ask(300, 48, 8, 3001, 1, 148) and not ask(37, 48, 8, 3001, 1, 148) and ask(38, 48, 8, 3001, 1, 148)
