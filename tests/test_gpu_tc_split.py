"""The tcgen05 product with operands split into two float16 parts of scaled rows, at the edges of its tiles and on rows,
columns and elements that differ by many orders of magnitude."""

import ctypes as C

import pytest

from quabla_b200 import _lib

pytestmark = pytest.mark.gpu


def _ptr(tensor):
    return C.c_void_p(tensor.data_ptr())


@pytest.mark.parametrize("spread", ["even", "rows and columns", "elements", "tiny", "large"])
@pytest.mark.parametrize("M,N,K", [(1, 64, 32), (127, 64, 64), (128, 128, 32), (129, 192, 96), (1000, 256, 512),
                                   (38017, 256, 256), (76033, 64, 64)])
def test_product_against_float64(cuda_device, M, N, K, spread):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(K, N, device="cuda", generator=g) / K ** 0.5

    def powers(n, low, high):
        return torch.exp2(torch.randint(low, high + 1, (n,), device="cuda", generator=g).float())

    if spread == "rows and columns":
        a = a * powers(M, -40, 40)[:, None]
        w = w * powers(N, -20, 20)[None, :]
    elif spread == "elements":
        a = a * powers(M * K, -12, 0).reshape(M, K)
        w = w * powers(K * N, -12, 0).reshape(K, N)
    elif spread == "tiny":
        a = a * 2.0 ** -100
    elif spread == "large":
        a, w = a * 2.0 ** 100, w * 2.0 ** 20
    bias = torch.randn(N, device="cuda", generator=g) * w.abs().amax(0) * a.abs().max()
    out = torch.full((M, N), float("nan"), device="cuda")
    biased = M // 2
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().qb200_matmul_3xtf32(_ptr(a), _ptr(w), _ptr(bias), _ptr(out), M, N, K, biased, stream))
    expected = a.double() @ w.double()
    size = a.double().abs() @ w.double().abs()
    expected[:biased] += bias.double()
    size[:biased] += bias.double().abs()
    # Per entry and relative to the sum of the terms' magnitudes: the parts carry each factor to 2^-23 or, below 2^-16 of
    # its row's largest element, to 2^-39 of that (hence the row term), the dropped lo.lo is 2^-22 at most, a k-tile's six
    # instructions truncate by 2^-23 each and every one of the K / 32 additions rounds by 2^-24.
    row = a.double().abs().amax(1)[:, None] * w.double().abs().amax(0)[None, :]
    bound = size * (2 * 2.0 ** -23 + 2.0 ** -22 + 6 * 2.0 ** -23 + (K / 32 + 2) * 2.0 ** -24) + 2 * K * row * 2.0 ** -39
    assert bool(((out.double() - expected).abs() <= bound + 2.0 ** -148).all())


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_non_finite_rows_stay_non_finite_and_alone(cuda_device, value):
    import torch

    M, N, K = 300, 128, 128
    a = torch.ones(M, K, device="cuda")
    a[131, 77] = value
    w = torch.ones(K, N, device="cuda")
    out = torch.zeros(M, N, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().qb200_matmul_3xtf32(_ptr(a), _ptr(w), None, _ptr(out), M, N, K, 0, stream))
    finite = torch.isfinite(out).all(dim=1)
    assert not torch.isfinite(out[131]).any()
    assert int(finite.sum()) == M - 1
    assert torch.equal(out[finite], torch.full((M - 1, N), float(K), device="cuda"))


def test_truncation_leaves_no_common_factor(cuda_device):
    # <error, exact> / <exact, exact>: the six truncating accumulations of a k-tile lower every product by 5.6e-8 of itself,
    # which the weight operand makes up for; over 2^23 entries of random sign the rest of the error (1e-7 per entry) leaves
    # less than 1e-9 here, and 2e-8 is a third of the uncorrected factor.
    import torch

    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(65536, 256, device="cuda", generator=g)
    w = torch.randn(256, 128, device="cuda", generator=g) / 16
    out = torch.zeros(65536, 128, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().qb200_matmul_3xtf32(_ptr(a), _ptr(w), None, _ptr(out), 65536, 128, 256, 0, stream))
    exact = a.double() @ w.double()
    error = out.double() - exact
    assert abs(float((error * exact).sum() / (exact * exact).sum())) <= 2e-8
    assert float(error.pow(2).mean().sqrt() / exact.pow(2).mean().sqrt()) <= 2e-7
