"""Which float32 projections this library's kernel takes and which go on to the library product (no GPU: the kernel is a stand-in)."""
import pytest
import torch

from sparseengine_b200.csrc import ops
from sparseengine_b200.parts import linear as module
from sparseengine_b200.parts.linear import linear32


@pytest.fixture
def taken(monkeypatch):
    """The sizes that reached the kernel; every size pays."""
    seen = []

    def dense(x, w, out):
        seen.append((tuple(x.shape), tuple(w.shape)))
        return out.zero_()

    monkeypatch.setattr(ops, "gemm_f32_dense", dense)
    monkeypatch.setattr(ops, "gemm_f32_tc_supported", lambda k: True)
    monkeypatch.setattr(ops, "gemm_f32_dense_pays", lambda *sizes: True)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    return seen


@pytest.fixture
def reached(monkeypatch):
    """The CPU's tensors count as the device's."""
    monkeypatch.setattr(module, "_kernel_reaches", lambda *tensors: True)


def test_sizes_that_do_not_fit_together_are_refused(taken, reached):
    x = torch.randn(16, 32)
    for w in (torch.randn(8, 28), torch.randn(8, 36), torch.randn(4, 8, 32)):
        with pytest.raises(RuntimeError):
            linear32(x, w)
    assert linear32(x, torch.randn(32)).shape == (16,)          # a vector is a product with a vector, not 32 rows of weights
    assert not taken
    assert linear32(x, torch.randn(8, 32)).shape == (16, 8) and taken == [((16, 32), (8, 32))]


def test_binding_refuses_sizes_that_do_not_fit_together():
    x = torch.randn(16, 32)
    for w, out in ((torch.randn(8, 28), torch.empty(16, 8)), (torch.randn(8, 32), torch.empty(16, 4)), (torch.randn(32), torch.empty(16, 32))):
        with pytest.raises(ValueError, match="fit together"):
            ops.gemm_f32_dense(x, w, out)


def test_tensors_elsewhere_go_to_the_library_product(taken, monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    x, w = torch.randn(16, 32), torch.randn(8, 32)
    assert torch.equal(linear32(x, w), x @ w.t())
    assert torch.equal(linear32(x, w.to_sparse()), x @ w.t())
    assert not taken
    cuda, other = (type("T", (), dict(device=torch.device("cuda", i), layout=torch.strided, is_neg=lambda self: False))() for i in (0, 1))
    assert module._kernel_reaches(cuda, cuda) and not module._kernel_reaches(other, other) and not module._kernel_reaches(cuda, other)
    assert not module._kernel_reaches(cuda, w)


def test_what_sees_the_product_sees_it(taken, reached, monkeypatch):
    """Gradients, tangents, vmap, torch.func, tracing, dispatch modes, subclasses and autocast: the library product is one that they know."""
    import torch.autograd.forward_ad as fwd
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode
    x, w = torch.randn(16, 32), torch.randn(8, 32)
    want = x @ w.t()
    with fwd.dual_level():
        y, tangent = fwd.unpack_dual(linear32(fwd.make_dual(x, 2 * x), w))
        assert torch.equal(y, want) and torch.equal(tangent, 2 * want)
    assert torch.allclose(torch.vmap(lambda r: linear32(r, w))(x.expand(3, 16, 32)), want.expand(3, 16, 8))
    assert torch.allclose(torch.func.jvp(lambda r: linear32(r, w), (x,), (x,))[1], want)
    assert torch.equal(torch.func.grad(lambda r: linear32(r, w).sum())(x), torch.autograd.functional.jacobian(lambda r: (r @ w.t()).sum(), x))
    assert torch.equal(make_fx(lambda a, b: linear32(a, b))(x, w)(2 * x, w), 2 * x @ w.t())
    assert torch.equal(torch.jit.trace(linear32, (x, w), check_trace=False)(2 * x, w), 2 * x @ w.t())
    with FlopCounterMode(display=False) as count:
        linear32(x, w)
    assert count.get_total_flops() == 2 * 16 * 8 * 32
    z = x.clone().requires_grad_()
    assert linear32(z, w).requires_grad and linear32(x, torch.nn.Parameter(w)).requires_grad
    with monkeypatch.context() as m:            # (autocast itself is off without a GPU)
        m.setattr(torch, "is_autocast_enabled", lambda kind: kind == "cuda")
        linear32(x, w)
    linear32(x.as_subclass(type("Sub", (torch.Tensor,), {})), w)
    assert not taken
    with torch.no_grad():
        linear32(z, torch.nn.Parameter(w))
    linear32(x, w)
    assert len(taken) == 2


def test_the_caller_may_have_the_library_product(taken, reached):
    x, w = torch.randn(16, 32), torch.randn(8, 32)
    assert torch.equal(linear32(x, w, f32_terms=False), x @ w.t()) and not taken
    linear32(x, w)
    assert len(taken) == 1
