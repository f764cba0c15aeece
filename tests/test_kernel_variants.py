"""Kernels that a rule on sizes, types or alignment chooses, at the sizes where each can go wrong: edges of tiles,
remainders, the smallest and the largest of the rule's range."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _k():
    from ccinfer_b200 import kernels
    return kernels


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rel(got, ref):
    got, ref = got.double(), ref.double()
    assert torch.isfinite(got).all()
    return float((got - ref).abs().max() / ref.abs().max().clamp_min(1e-30))


# rows kernel: 1, 2, 3, 5, 9, 16 rows; tiles of 32, 64, 128 rows; with and without a cluster (K below and from 512); rows
# that start on no 16 bytes; more tiles than two rounds
@pytest.mark.parametrize("M,N,K,pad,batch", [
    (1, 1, 1, 0, 1), (2, 15, 31, 0, 1), (3, 17, 256, 0, 2), (4, 33, 260, 1, 1), (5, 64, 2048, 0, 1), (8, 300, 1001, 3, 1),
    (9, 16, 8192, 0, 1), (16, 2049, 512, 4, 3), (17, 129, 511, 0, 1), (32, 128, 512, 0, 2), (33, 257, 516, 0, 1),
    (64, 100, 4100, 2, 1), (65, 128, 1024, 0, 1), (120, 300, 100, 0, 1), (128, 1000, 2048, 0, 1), (300, 16384, 544, 0, 1),
    (1030, 5000, 72, 0, 1)])
def test_float_product_of_every_shape_is_one_order_of_sums(M, N, K, pad, batch):
    """Against float64: eight chains of K / 8 float multiply-adds and seven sums stay within (K / 8 + 8) roundings of
    the sum of magnitudes; and a row alone gives the bits that it has among others."""
    g = _gen(M + 7 * N + 13 * K)
    a = torch.randn((batch, M, K + pad), generator=g, device="cuda")[:, :, :K]
    w = torch.randn((batch, N, K + pad), generator=g, device="cuda")[:, :, :K]
    c = torch.full((batch, M, N), float("nan"), device="cuda")
    k = _k()
    if batch > 1:
        k.gemm_f32_batched(c, a, w)
    else:
        k.gemm_f32(c[0], a[0], w[0])
    ref = a.double() @ w.double().transpose(1, 2)
    size = a.double().abs() @ w.double().abs().transpose(1, 2)
    assert ((c.double() - ref).abs() <= (K / 8 + 8) * 2.0 ** -24 * size).all()
    for rows in (1, 7, 20):   # a few rows by themselves: other kernels, the same sums
        n = min(rows, M)
        c1 = torch.full((n, N), float("nan"), device="cuda")
        k.gemm_f32(c1, a[0, M - n:], w[0])
        assert torch.equal(c1, c[0, M - n:])
