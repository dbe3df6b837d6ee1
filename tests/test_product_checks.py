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


def _bf16(rows, cols, ld=None, at=1 << 20):
    t = _like(rows, cols, at=at, dtype=torch.bfloat16)
    t.stride = lambda i=None: (cols if ld is None else ld, 1) if i is None else (cols if ld is None else ld, 1)[i]
    return t


@pytest.mark.parametrize("a,w,taken", [
    (_bf16(128, 256), _bf16(256, 512), True),
    (_bf16(128, 256, ld=512), _bf16(256, 512, ld=1024), True),
    (_bf16(128, 256, ld=0), _bf16(256, 512), False),                        # one row, seen 128 times
    (_bf16(128, 256, ld=8), _bf16(256, 512), False),                        # rows that overlap
    (_bf16(128, 256), _bf16(256, 512, ld=0), False),
    (_bf16(128, 0, ld=8), _bf16(0, 512), False),                            # empty sums
    (_bf16(128, 256), _bf16(248, 512), False),
])
def test_what_the_bfloat16_kernel_of_many_rows_is_given(a, w, taken):
    assert ops._tc_ok(a, w, 65) is taken


def test_the_library_is_given_operands_that_fit(monkeypatch):
    def reached():
        raise AssertionError("the library's product was asked for")
    monkeypatch.setattr(ops, "LIBRARY_GEMM_DIRECT", True)
    monkeypatch.setattr(ops, "_blas_state", None)
    monkeypatch.setattr(ops, "library", reached)
    assert ops._library_gemm(_bf16(128, 256), _bf16(248, 512), None, False) is None
    with pytest.raises(AssertionError):
        ops._library_gemm(_bf16(128, 256), _bf16(256, 512), None, False)


@pytest.mark.gpu
def test_rows_that_are_one_row():
    """Gate/up of a row that is expanded to many, as before the kernel took steps from 65 rows on."""
    row, w = torch.randn(1, 256, device="cuda").to(torch.bfloat16), torch.randn(256, 256, device="cuda").to(torch.bfloat16) * 0.1
    got = ops.gemm_swiglu(row.expand(200, 256), w, 128, 32)
    torch.testing.assert_close(got, ops.gemm_swiglu(row.expand(200, 256).contiguous(), w, 128, 32), rtol=2e-2, atol=2e-3)
    with pytest.raises(RuntimeError):
        ops.gemm(row.expand(200, 256).contiguous(), w[:248])
