"""The float32 product on tcgen05 at the edges of its row tiles (up to 192 rows, of one size), of the rows of W a tile has, and of the K
blocks that are added in one chain; and matrices that do not start on a 16-byte boundary."""
import pytest
import torch

from tests.test_gpu_sgemm_tc5 import _inputs, _ops, _product

pytestmark = pytest.mark.gpu


def _check(got, x, w, b):
    want, size = x.double() @ w.double().t() + b.double(), x.double().abs() @ w.double().abs().t() + b.double().abs()
    # the bound of test_gpu_sgemm_tc5.py: 24 additions cut off a K block, and the blocks', slices', parts' and bias' roundings
    assert ((got.double() - want).abs() <= size * (2.0 ** -24 + 24 * 2.0 ** -23 + (41 + x.shape[1] / 2048) * 2.0 ** -24)).all()


@pytest.mark.parametrize("M,N,K", [(16, 127, 64), (17, 129, 128), (176, 128, 1792), (177, 64, 1856), (192, 384, 3584), (193, 130, 3648),
                                   (385, 257, 68), (700, 18944, 512), (80, 8, 12000)])
def test_edges(M, N, K):
    x, w, b = _inputs(M, N, K)
    _check(_product(_ops().sgemm_tc5, x, w, b), x, w, b)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_matrices_off_the_boundary(offset):
    x, w, b = _inputs(200, 130, 320)
    off = torch.empty(w.numel() + offset, device=w.device)[offset:].view_as(w).copy_(w)
    got = _product(_ops().sgemm_tc5, x, off, b)
    assert torch.equal(got, _product(_ops().sgemm_tc5, x, w, b))
    _check(got, x, w, b)
