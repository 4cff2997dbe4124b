"""Rows behind the last whole tile of the float32 product: the same, bit for bit, as those rows alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M", [129, 131, 144, 145, 257, 272])
@pytest.mark.parametrize("N,K", [(38001, 333), (5001, 4100), (40, 600)])
def test_rest_rows(M, N, K):
    from paged_batch_engine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w, b = (torch.randn(*s, device=DEV, generator=g) for s in ((M, K), (N, K), (N,)))
    full = torch.full((M, N), float("nan"), device=DEV)
    ops.sgemm_nt(x, w, b, full)
    whole = M // 128 * 128
    for lo, hi in ((0, whole), (whole, M)):
        part = torch.empty(hi - lo, N, device=DEV)
        ops.sgemm_nt(x[lo:hi].contiguous(), w, b, part)
        assert torch.equal(part, full[lo:hi])
    # 2 K products and sums a value, each rounded by 2^-24 of numbers of about sqrt(K)
    assert (full.double() - (x.double() @ w.double().t() + b)).abs().max() <= 8e-6 * K ** 0.5
