"""The native operator implementations: gradients without a bias, errors raised from C++, attributes."""

import pytest
import torch

import iree_turbine_b200 as tb
from iree_turbine_b200 import _launcher as L
from iree_turbine_b200 import ops
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (77, 264, 136), (515, 72, 320)])
def test_linear_gradients(bias, m, n, k):
    g = torch.Generator().manual_seed(3)
    x, w, dy = (torch.randn(*s, generator=g).half() for s in ((m, k), (n, k), (m, n)))
    b = torch.randn(n, generator=g).half() if bias else None
    leaves = [t.to(DEV).requires_grad_() for t in (x, w) + ((b,) if bias else ())]
    y = ops.linear(leaves[0], leaves[1], leaves[2] if bias else None)
    grads = torch.autograd.grad(y, leaves, dy.to(DEV))
    refs = (dy.float() @ w.float(), dy.float().t() @ x.float(), dy.float().sum(0))
    for got, ref in zip(grads, refs):
        assert got.dtype == torch.float16
        # one rounding to f16 (2^-11) of a sum whose terms are exact in fp32
        oracle.assert_close_half(got, ref)
    # inputs that need no gradient get none
    y = ops.linear(x.to(DEV), leaves[1], None)
    assert torch.equal(torch.autograd.grad(y, leaves[1], dy.to(DEV))[0], grads[1])


def test_errors_keep_their_types():
    a = torch.zeros(136, 300, dtype=torch.float16, device=DEV)
    with pytest.raises(ValueError, match="BAD_ALIGN"):
        torch.ops.b200k.gemm(a, a[:, :200].contiguous(), True, False, None)
    with pytest.raises(RuntimeError, match="do not match"):
        torch.ops.b200k.gemm_nt(a, a[:, :64].contiguous())
    with pytest.raises(RuntimeError, match="one device"):
        torch.ops.b200k.gemm_nt(a, a.cpu())
    assert tb.device_status() == 0


def test_attention_kernel_attribute_reaches_the_ops():
    assert ops.ATTENTION_KERNEL == L.ATTN_AUTO
    q = torch.randn(1, 1, 200, 64, device=DEV).half()
    ops.ATTENTION_KERNEL = 7  # head dim 64 ignores it, head dim 128 passes it on
    try:
        torch.ops.b200k.attention(q, q, q, 0.1, False)
        q = torch.randn(1, 1, 200, 128, device=DEV).half()
        with pytest.raises(ValueError, match="unknown kernel choice 7"):
            torch.ops.b200k.attention(q, q, q, 0.1, False)
    finally:
        ops.ATTENTION_KERNEL = L.ATTN_AUTO


def test_bias_gradient_can_be_differentiated():
    g = torch.Generator().manual_seed(5)
    x, w, b = (torch.randn(*s, generator=g).half().to(DEV) for s in ((40, 64), (24, 64), (24,)))
    dy = torch.randn(40, 24, generator=g).half().to(DEV).requires_grad_()
    b.requires_grad_()
    db, = torch.autograd.grad(ops.linear(x, w, b), b, dy, create_graph=True)
    plain, = torch.autograd.grad(ops.linear(x, w, b), b, dy.detach())
    # one rounding to f16 (2^-11) of the same fp32 sum in two orders
    oracle.assert_close_half(db, plain.float().cpu(), rtol=2.0 ** -10, atol=1e-4)
    weight = torch.randn(24, generator=g).half().to(DEV)
    ddy, = torch.autograd.grad(db, dy, weight)
    assert torch.equal(ddy, weight.expand(40, 24))
