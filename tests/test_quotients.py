"""The quotient of csrc/common.cuh, for denominators of at least one, against the division operator: a small program of the header and this
file's kernel, built here and run on the GPU."""
import ctypes
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "common.cuh"
__global__ void both(const float* a, const float* b, float* q, float* w, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        q[i] = quotient(a[i], b[i]);
        w[i] = a[i] / b[i];
    }
}
extern "C" __attribute__((visibility("default"))) int run(const float* a, const float* b, float* q, float* w, int n) {
    both<<<512, 256>>>(a, b, q, w, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from tiny_inference_server_b200.kernels import build
    where = tmp_path_factory.mktemp("quotients")
    (where / "both.cu").write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(where / "both.so"), str(where / "both.cu")], check=True)
    lib = ctypes.CDLL(str(where / "both.so"))

    def call(a, b):
        a, b = a.cuda().contiguous(), b.cuda().contiguous()
        q, w = torch.empty_like(a), torch.empty_like(a)
        torch.cuda.synchronize()
        assert lib.run(*(ctypes.c_void_p(t.data_ptr()) for t in (a, b, q, w)), a.numel()) == 0
        return q, w
    return call


def _same(q, w):
    """The same bits, NaN for NaN; a result below 2^-126 is rounded twice, to a neighbour at most."""
    nan = torch.isnan(w)
    assert torch.equal(torch.isnan(q), nan)
    normal = ~nan & (w.abs() >= 2.0 ** -126)
    assert torch.equal(q[normal].view(torch.int32), w[normal].view(torch.int32))
    small = ~nan & ~normal
    assert bool(((q[small] - w[small]).abs() <= 2.0 ** -149).all()) and torch.equal(torch.signbit(q[small]), torch.signbit(w[small]))


def _floats(bits):
    return bits.to(torch.int32).view(torch.float32)


def test_any_numerator_and_denominator(run):
    g = torch.Generator().manual_seed(1)
    n = 1 << 24
    a = _floats(torch.randint(-2 ** 31, 2 ** 31, (n,), generator=g))                     # all there are: NaN, infinities, subnormal ones
    b = _floats(torch.randint(0x3f800000, 0x7f800002, (n,), generator=g))                # one to infinity
    _same(*run(a, b))
    mantissa = torch.randint(0, 1 << 23, (2, n), generator=g)
    _same(*run(_floats(mantissa[0] + 0x3f800000), _floats(mantissa[1] + 0x3f800000)))


@pytest.mark.parametrize("b", [0x3f800000, 0x3f800001, 0x3fffffff, 0x3ffffffe, 0x40400000, 0x5f7fffff, 0x5f800000, 0x7effffff, 0x7f000000, 0x7f7fffff, 0x7f800000])
def test_every_mantissa_of_the_numerator(run, b):
    a = _floats(torch.arange(1 << 23) + 0x3f800000)
    for x in (a, -a * 2.0 ** 100, a * 2.0 ** -31, a * 2.0 ** -120):
        _same(*run(x, _floats(torch.tensor([b])).expand(len(x))))


def test_quotients_next_to_where_rounding_turns(run):
    """a 2^25 = +-1 modulo b: no quotients of 24-bit numbers are nearer to a number of 25 bits that is none of 24."""
    g = torch.Generator().manual_seed(2)
    a, b = [], []
    for m in (torch.randint(1 << 22, 1 << 23, (40000,), generator=g) * 2 + 1).tolist() + list(range((1 << 24) - 4001, 1 << 24, 2)):
        inverse = pow(1 << 25, -1, m)
        for x in (inverse, m - inverse):
            while x < 1 << 23:
                x *= 2
            a.append(x)
            b.append(m)
    a, b = torch.tensor(a, dtype=torch.float64).float(), torch.tensor(b, dtype=torch.float64).float()
    assert float(a.max()) < 2 ** 24 and float(b.max()) < 2 ** 24
    for x, y in ((1.0, 1.0), (-2.0 ** -60, 1.0), (1.0, 2.0 ** 60), (2.0 ** -100, 1.0)):
        _same(*run(a * x, b * y))
