"""float32 products whose operands do not fit together: the tensor-core kernel (csrc/gemm_split.cu) reads what its arguments say, so they
are compared before, and what does not fit is left to torch.mm and its errors."""
from types import SimpleNamespace

import pytest
import torch

from tiny_inference_server_b200.kernels import ops


def _like(rows, cols, device="cuda:0", at=1 << 20, storage=None, dtype=torch.float32, grad=False):
    """What the rule asks of a tensor, without one."""
    return SimpleNamespace(dtype=dtype, shape=(rows, cols), device=device, is_cuda=device.startswith("cuda"), requires_grad=grad,
                           dim=lambda: 2, stride=lambda i=None: (cols, 1) if i is None else (cols, 1)[i], data_ptr=lambda: at,
                           untyped_storage=lambda: SimpleNamespace(data_ptr=lambda: storage or at))


X, W, OUT = (800, 1024), (1024, 512), (800, 512)


@pytest.mark.parametrize("a,w,out,taken", [
    (_like(*X), _like(*W, at=1 << 21), None, True),
    (_like(*X), _like(*W, at=1 << 21), _like(*OUT, at=1 << 22), True),
    (_like(*X), _like(1020, 512, at=1 << 21), None, False),                             # too few rows of W, too many
    (_like(*X), _like(2048, 512, at=1 << 21), None, False),
    (_like(*X), _like(*W, at=1 << 21), _like(799, 512, at=1 << 22), False),             # a result of another shape
    (_like(*X), _like(*W, at=1 << 21), _like(800, 516, at=1 << 22), False),
    (_like(*X), _like(*W, "cpu", at=1 << 21), None, False),                             # tensors of other devices
    (_like(*X), _like(*W, "cuda:1", at=1 << 21), None, False),
    (_like(*X, "cpu"), _like(*W, "cpu", at=1 << 21), None, False),
    (_like(*X), _like(*W, at=1 << 21), _like(*OUT, "cpu", at=1 << 22), False),
    (_like(*X), _like(*W, at=1 << 21), _like(*OUT, at=(1 << 20) + 4096, storage=1 << 20), False),   # a result inside an operand
    (_like(*X), _like(*W, at=1 << 21, grad=True), None, False),                         # a gradient is wanted
])
def test_what_the_kernel_is_given(a, w, out, taken):
    with torch.enable_grad():
        assert ops._split_ok(a, w, out) is taken


def test_without_gradients_parameters_are_taken():
    with torch.no_grad():
        assert ops._split_ok(_like(*X), _like(*W, at=1 << 21, grad=True), None)


@pytest.mark.gpu
def test_errors_stay_errors():
    a, w = torch.randn(X, device="cuda"), torch.randn(W, device="cuda")
    with pytest.raises(RuntimeError):
        ops.gemm(a, w[:1020])
    with pytest.raises(RuntimeError):
        ops.gemm(a, w.cpu())
    out = torch.empty(0, device="cuda")
    assert torch.equal(ops.gemm(a, w, out=out), torch.mm(a, w)) and out.shape == OUT
    p = torch.nn.Parameter(w)
    before = ops.calls["gemm_split"]
    ops.gemm(a, p).sum().backward()
    torch.testing.assert_close(p.grad, a.sum(0)[:, None].expand(W), rtol=1e-4, atol=1e-3)
    assert ops.calls["gemm_split"] == before
    # the same operands without any of this
    ops.gemm(a, w, out=torch.empty(OUT, device="cuda"))
    assert ops.calls["gemm_split"] == before + 1
