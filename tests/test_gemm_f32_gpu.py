"""32-bit products on the tensor cores in tf32 terms (csrc/gemm_f32_tc.cu) against 64 bits, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bound(x, w):
    """What a result may be off, over the sum of the products' sizes.  The weights' hi is the nearest tf32 value (rest up to 2^-11 of the value),
    the activations' is cut off (2^-10): lo lo, left out, is up to 2^-21; the activations' rest is rounded to 11 bits (2^-22), the weights' cut off
    there (2^-23).  64 products are summed in 8 steps, each cut off below 2^-23 of the sum (2^-20 in all), and every 64 products take one rounded
    addition (2^-24).  2^-21 + 2^-22 + 2^-23 + 2^-20 < 2^-19."""
    return (2.0 ** -19 + x.shape[1] / 64 * 2.0 ** -24) * (x.double().abs() @ w.double().abs().t())


@pytest.mark.parametrize("k", [4, 28, 32, 36, 64, 68, 516, 1100])
@pytest.mark.parametrize("rows,n", [(1, 1), (63, 127), (64, 128), (65, 129), (127, 4), (128, 257), (129, 130), (300, 3000)])
def test_dense(rows, n, k):
    from sparseengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(rows * 7 + n + k)
    wide = torch.randn(rows, k + 12, generator=g, device=DEV)
    w = torch.randn(n, k, generator=g, device=DEV)
    for x in (wide[:, 4:4 + k], wide[:, :k].abs().contiguous()):        # rows apart; sums without cancellation
        out = torch.full((rows, n), float("nan"), device=DEV)
        ops.gemm_f32_dense(x, w, out)
        assert bool(((out.double() - x.double() @ w.double().t()).abs() <= _bound(x, w)).all())
    ops.error_check(DEV)


@pytest.mark.parametrize("sms", [1, 2, 3])
@pytest.mark.parametrize("k", [36, 68, 516, 1100])
@pytest.mark.parametrize("rows,n", [(191, 700), (150, 1100), (64, 520), (300, 260)])
def test_dense_item_after_item(rows, n, k, sms):
    """Few blocks, so that each takes several items in turn: last tiles of 22 to 63 rows after full ones, odd numbers of steps (k 36, 68, 516, 1100: 2, 3,
    17 and 35) and of sums (1, 2, 9 and 18)."""
    from sparseengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(rows + n + k)
    x, w = torch.randn(rows, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV)
    out = torch.full((rows, n), float("nan"), device=DEV)
    ops.gemm_f32_dense(x, w, out, sms=sms)
    assert bool(((out.double() - x.double() @ w.double().t()).abs() <= _bound(x, w)).all())
    whole = torch.empty_like(out)
    ops.gemm_f32_dense(x, w, whole)
    assert torch.equal(out, whole)              # an item's sums do not depend on the items before it
    ops.error_check(DEV)


def test_dense_ends_of_the_range():
    """Infinities, NaN and the largest values come out as multiply-adds leave them."""
    from sparseengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    x, w = torch.randn(70, 256, generator=g, device=DEV), torch.randn(300, 256, generator=g, device=DEV)
    top = torch.finfo(torch.float32).max
    x[3, 5], x[9, 7], w[11, 3], w[12, 200] = float("inf"), float("nan"), -float("inf"), float("nan")
    x[30] = 0.0
    x[31], w[13] = 0.0, 0.0
    x[31, 0], w[13, 1], x[32, :], x[32, 1] = top, -top, 0.0, 0.25     # products of the largest with small values stay finite
    w[:11, 0] = 0.25
    out = torch.empty(70, 300, device=DEV)
    ops.gemm_f32_dense(x, w, out)
    want = x.double() @ w.double().t()
    finite = want.isfinite() & (want.abs() <= top)
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out[want.isinf()], want[want.isinf()].float()) and bool(out[finite].isfinite().all())
    assert bool(((out.double() - want).abs()[finite] <= 1e-4 * want.abs()[finite] + 1e-3).all())
    ops.error_check(DEV)


def test_dense_nan_of_any_bits():
    """A NaN may have its set bits among those that the tensor cores cut off, or be negative, in an activation and in a weight."""
    from sparseengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(2)
    x, w = torch.randn(140, 256, generator=g, device=DEV), torch.randn(300, 256, generator=g, device=DEV)
    bits = torch.tensor([0x7f800001, 0x7f801fff, 0x7fffffff, -0x7fffff], dtype=torch.int32, device=DEV).view(torch.float32)     # the last: 0xff800001
    x[torch.tensor([2, 40, 77, 139]), torch.tensor([0, 31, 32, 255])] = bits
    w[torch.tensor([0, 64, 130, 299]), torch.tensor([255, 3, 64, 31])] = bits
    out = torch.empty(140, 300, device=DEV)
    ops.gemm_f32_dense(x, w, out)
    want = x.double() @ w.double().t()
    assert torch.equal(out.isnan(), want.isnan()) and not bool(out.isinf().any())
    finite = ~want.isnan()
    assert bool(((out.double() - want).abs() <= _bound(x, w))[finite].all())
    ops.error_check(DEV)


@pytest.mark.parametrize("activation", [None, ("clamped_swiglu", 2.0, 1.3), ("gelu_tanh", 0.0, 0.0)], ids=["silu", "clamped", "gelu"])
@pytest.mark.parametrize("counts,hidden,inter", [([127, 128, 129, 0, 1, 31, 33, 97], 512, 516), ([300, 5], 640, 1028), ([64, 63, 65], 1024, 512)])
def test_routed_products(counts, hidden, inter, activation):
    """Both products of the experts against the general kernel's, at the edges of tiles in rows, features and inner dimension."""
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
    before = ops.calls.get("se_gemm_f32_grouped", 0)
    got = part.run_experts(x, ids, weights)
    assert ops.calls.get("se_gemm_f32_grouped", 0) == before + 2
    part.use_tensor_cores = False
    want = part.run_experts(x, ids, weights)
    assert ops.calls.get("se_gemm_f32_grouped", 0) == before + 2
    # two sums of at most 1,028 products of size one each (results of size one), some 1e-6 off in either order
    assert float((got - want).abs().max()) < 2e-5 * max(1.0, float(want.abs().max()))
    ops.error_check(DEV)


@pytest.mark.parametrize("sms", [1, 3])
def test_routed_products_item_after_item(sms, monkeypatch):
    """Few blocks: tiles of 1 to 128 rows of an expert in turn, products issued apart and joined, gate and up rows and routing weights of item
    after item through the same buffers."""
    from sparseengine_b200.csrc import ops
    whole = ops.gemm_f32_grouped
    monkeypatch.setattr(ops, "gemm_f32_grouped", lambda *a, **kw: whole(*a, sms=sms, **kw))
    test_routed_products([1, 128, 5, 65, 0, 64, 200, 17, 66, 3], 516, 548, None)
    test_routed_products([300, 5], 640, 1028, ("gelu_tanh", 0.0, 0.0))


def test_projections_take_it():
    """Float32 projections that fill the device run on it, small ones and those on odd addresses through the library."""
    from sparseengine_b200.csrc import ops
    from sparseengine_b200.parts.linear import linear
    x, w = torch.randn(1024, 2052, device=DEV), torch.randn(2048, 2048, device=DEV)

    def calls(a, b, **options):
        before = ops.calls.get("se_gemm_f32_dense", 0)
        y = linear(a, b, **options)
        assert bool(((y.double() - a.double() @ b.double().t()).abs() <= 4 * _bound(a, b)).all())
        return ops.calls.get("se_gemm_f32_dense", 0) - before

    assert calls(x[:, :2048], w) == 1 and calls(x[:, 4:], w) == 1 and calls(x[:, 4:], w, f32_terms=False) == 0
    assert calls(x[:, 1:2049], w) == 0 and calls(x[:3, :2048], w) == 0 and calls(x[:, :64], w[:, :64].contiguous()) == 0
