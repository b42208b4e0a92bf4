"""32-bit activations times a 16-bit matrix on the tensor cores (kernels/ops.py: gemm_split), against 64-bit products."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from transformers_neuronx_b200.kernels import ops as o
    return o


def _operands(M, N, K, dtype, seed, pitch=0, spread=0.0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    a = torch.randn(M, K + pitch, generator=g)
    if spread:                                         # sizes over `spread` powers of two, within a row and between rows
        a = a * torch.exp2((torch.rand(M, K + pitch, generator=g) - 0.5) * spread)
    w = torch.randn(N, K, generator=g) * 0.02
    return a.to(DEV)[:, :K], w.to(dtype).to(DEV), torch.randn(N, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)


def _bound(a, w, K):
    """The accumulators cut off at most 2^-22 of the chunk's largest partial sum an MMA (8 of them a chunk of 128), the chunks
    are added in 32 bits; both against the sum of the products' sizes."""
    return (8 * 2.0 ** -22 + (-(-K // 128) + 3) * 2.0 ** -24) * (a.double().abs() @ w.double().abs().t())


# one token to more than a tile of 64, one and two feature tiles a CTA, K split or not, remainders of every tile, an unaligned pitch
SHAPES = [(1, 128, 256, 0), (1, 2048, 2048, 0), (3, 300, 1032, 4), (16, 768, 3072, 0), (17, 130, 520, 1), (32, 2304, 768, 0),
          (33, 257, 264, 0), (64, 2048, 8192, 0), (65, 5000, 640, 0), (200, 9001, 328, 2), (502, 6144, 2048, 0), (700, 9000, 1096, 0)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K,pitch", SHAPES)
def test_gemm_split(M, N, K, pitch, dtype):
    o = ops()
    a, w, bias, res = _operands(M, N, K, dtype, M + N + K, pitch)
    want, bound = a.double() @ w.double().t(), _bound(a, w, K)
    out = torch.empty(M, N, device=DEV)
    o.gemm_split(a, w, out)
    o.raise_on_device_error()
    assert bool(((out.double() - want).abs() <= bound).all())
    fma = torch.empty(M, N, device=DEV)
    o.gemm_simt(a, w, fma)
    assert float((out.double() - want).norm()) <= 1.02 * float((fma.double() - want).norm())   # no further off than the chain of FMAs
    if M > 1:                                            # a row's bits are its own
        for m in sorted({0, M // 2, M - 1}):
            one = torch.empty(1, N, device=DEV)
            o.gemm_split(a[m:m + 1], w, one)
            assert torch.equal(one[0], out[m]), m
    joined = res.clone()
    o.gemm_split(a, w, joined, bias=bias, residual=joined, activation="relu")
    o.raise_on_device_error()
    assert torch.equal(joined, torch.relu(out + bias) + res)
    half = torch.empty(M, N, dtype=dtype, device=DEV)
    o.gemm_split(a, w, half, bias=bias)
    assert torch.equal(half, (out + bias).to(dtype))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e30])
def test_gemm_split_sizes_far_apart(scale, dtype):
    """Elements that differ by up to 2^40 within a row, rows far from one, keep their bits."""
    M, N, K = 40, 256, 512
    a, w, _, _ = _operands(M, N, K, dtype, 5, spread=40.0)
    a = a * scale
    out, fma = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops().gemm_split(a, w, out)
    ops().gemm_simt(a, w, fma)
    want = a.double() @ w.double().t()
    assert bool(((out.double() - want).abs() <= _bound(a, w, K)).all())
    assert float((out.double() - want).norm()) <= 1.02 * float((fma.double() - want).norm())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gemm_split_elements_that_are_not_finite(dtype):
    M, N, K = 70, 384, 640
    a, w, _, _ = _operands(M, N, K, dtype, 9)
    inf, nan = float("inf"), float("nan")
    a[1, 5], a[2, 300], a[3, 639] = inf, -inf, nan
    a[4, 0], a[4, 1] = inf, -inf
    a[6] = 0.0
    a[7] = 1e-42                                        # a row of denormal numbers
    a[8, 3] = 3.4e38
    w[10, 5] = 0.0                                      # inf * 0
    w[20, 77], w[21, 78], w[22, 400] = inf, -inf, nan
    out, fma = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops().gemm_split(a, w, out)
    ops().gemm_simt(a, w, fma)
    ops().raise_on_device_error()
    keep = torch.ones(M, 1, dtype=torch.bool, device=DEV)
    keep[8] = False                                     # overflows or not by the order of its sum
    same = torch.isnan(out) == torch.isnan(fma)
    assert bool((same | ~keep).all())
    big = torch.isinf(fma) & keep
    assert torch.equal(out[big], fma[big])
    fine = torch.isfinite(fma) & keep
    assert bool(torch.isfinite(out[fine]).all())
    assert float((out[fine] - fma[fine]).abs().max()) <= 1e-4
    if dtype == torch.bfloat16:                         # float16 weights: the scaled row's products are denormal no more
        assert bool(((out[7] - fma[7]).abs()[torch.isfinite(fma[7])] <= K * 2.0 ** -132).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("small", [1e-10, -1e-10, 1e-30, -1e-42])
def test_gemm_split_small_elements_opposite_infinite_weights(small, dtype):
    """An infinite weight times any number but zero is infinite, however small the number is beside the others in its row: in rows
    that are finite, that reach the largest number, and that hold an infinity or a NaN themselves."""
    inf = float("inf")
    a, w, _, _ = _operands(5, 128, 256, dtype, 3)
    a[:, 7], a[:, 9] = small, 0.0
    a[1, 100] = 3e38                                    # scaled down by 2^113 for float16
    a[2, 100], a[3, 100], a[4, 100] = inf, -inf, float("nan")
    w[:, 100] = w[:, 100].abs() + 1e-3
    w[1, 7], w[2, 7], w[3, 9] = inf, -inf, inf          # (the last: infinity times zero has no value)
    out, fma = torch.empty(5, 128, device=DEV), torch.empty(5, 128, device=DEV)
    ops().gemm_split(a, w, out)
    ops().gemm_simt(a, w, fma)
    ops().raise_on_device_error()
    assert bool(torch.isinf(fma[0, 1:3]).all()) and bool(torch.isnan(fma[:, 3]).all())
    assert torch.equal(torch.isnan(out), torch.isnan(fma))
    big = torch.isinf(fma)
    assert torch.equal(out[big], fma[big]) and bool(torch.isfinite(out[torch.isfinite(fma)]).all())


def test_gemm_split_in_slices_of_rows(monkeypatch):
    o = ops()
    a, w, bias, res = _operands(300, 256, 512, torch.float16, 3)
    whole, cut = torch.empty(300, 256, device=DEV), res.clone()
    o.gemm_split(a, w, whole, bias=bias)
    monkeypatch.setattr(o, "SPLIT_TERMS_BYTES", 6 * 512 * 128)
    o.gemm_split(a, w, cut, bias=bias, residual=cut)
    assert torch.equal(cut, whole + res)
