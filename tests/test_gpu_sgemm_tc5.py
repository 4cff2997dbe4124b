"""The float32 product on tcgen05 (three bfloat16 terms an operand) against 64 bits and against the multiply-adds: edges of
its tiles, K blocks and parts of K, rows behind the last whole tile, columns multiplied in several goes, numbers that are
not finite, and which products take it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from paged_batch_engine_b200.csrc import ops
    return ops


def _inputs(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    return rand(M, K), rand(N, K), rand(N)


def _product(fn, x, w, b):
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), device=DEV)
    fn(x, w, b, out)
    return out


@pytest.mark.parametrize("M,N,K", [(65, 64, 256), (128, 256, 320), (129, 257, 333), (144, 130, 1100), (300, 2049, 63),
                                   (513, 128, 8960), (1028, 1536, 2112), (66, 6000, 8200), (1, 1, 1)])
def test_against_64_bits(M, N, K):
    x, w, b = _inputs(M, N, K)
    got, fma = _product(_ops().sgemm_tc5, x, w, b), _product(_ops().sgemm_nt, x, w, b)
    want, size = x.double() @ w.double().t() + b.double(), x.double().abs() @ w.double().abs().t() + b.double().abs()
    # left out: 2^-24 of a product's size.  In a block of 64 k at most 24 additions are cut off at 2^-23 of what they
    # add to; the blocks' sums, the parts and the bias are added with less than 2^-24 each, 32 + K / 2048 + 9 of them in
    # a row at most
    assert ((got.double() - want).abs() <= size * (2.0 ** -24 + 24 * 2.0 ** -23 + (41 + K / 2048) * 2.0 ** -24)).all()
    if K >= 256:                    # and no further off than the multiply-adds
        assert (got.double() - want).norm() <= (fma.double() - want).norm()


@pytest.mark.parametrize("M,N,K", [(2433, 130, 18944), (4700, 3000, 18944), (1000, 64, 50000)])
def test_rows_whose_terms_are_made_in_several_goes(M, N, K):
    x, w, b = _inputs(M, N, K)
    got = _product(_ops().sgemm_tc5, x, w, b)
    want = torch.cat([x[i:i + 500].double() @ w.double().t() + b.double() for i in range(0, M, 500)])
    # sums of K products of normal numbers, off by the roundings' random walk: see the first test for the worst
    assert float((got.double() - want).norm() / want.norm()) <= 4e-7


def test_scratch_memory_is_bounded():
    """However many rows a step brings, and however many columns the matrix has."""
    ops = _ops()
    need = ops._fn("sgemm_tc5", "pbe_sgemm_tc5_scratch", [ops.c_int] * 3)
    need.restype = ops.c_ll
    for M in (65, 1000, 4096, 4097, 100000, 1 << 24):
        for N in (64, 5000, 152064):
            for K in (256, 1536, 18944, 65536):
                assert need(M, N, K) <= (640 << 20) + 4096, (M, N, K)


def test_numbers_that_are_not_finite():
    ops = _ops()
    x, w, b = _inputs(130, 200, 300)
    for value in (float("inf"), float("nan"), 3.4e38):
        x2, w2 = x.clone(), w.clone()
        x2[5, 7] = value
        w2[11, 299] = -value
        for xs, ws in ((x2, w), (x, w2), (x2, w2)):
            got, want = _product(ops.sgemm_tc5, xs, ws, b), _product(ops.sgemm_nt, xs, ws, b)
            assert torch.equal(got.nan_to_num(1.25), want.nan_to_num(1.25)) and torch.equal(got.isnan(), want.isnan())
    assert torch.isfinite(_product(ops.sgemm_tc5, x, w, b)).all()       # nothing is left behind


@pytest.mark.parametrize("x_value,w_value", [(1e-36, 1.0), (-3e-39, 2.0), (1e25, 1e25), (2.0 ** 70, -1.0), (1.0, 1e-33)])
def test_numbers_that_three_terms_do_not_hold(x_value, w_value):
    """Beside ordinary numbers: products that overflow stay the infinity that the multiply-adds make of them, and the last
    bits of tiny numbers are not lost."""
    ops = _ops()
    x, w, b = _inputs(130, 200, 300)
    x[5] = 0.0
    x[5, 7], w[:, 7] = x_value * 1.2345678, w_value * 1.1234567
    got, want = _product(ops.sgemm_tc5, x, w, None), _product(ops.sgemm_nt, x, w, None)
    assert torch.equal(got[5], want[5]) and not want[5].isnan().any()
    assert torch.equal(got, want)


@pytest.mark.parametrize("x_scale,w_scale", [(2.0 ** -60, 2.0 ** -55), (2.0 ** -65, 2.0 ** -60), (2.0 ** 40, 2.0 ** 42), (2.0 ** -85, 2.0 ** 45)])
def test_sizes_of_the_operands(x_scale, w_scale):
    ops = _ops()
    x, w, _ = _inputs(130, 200, 300)
    x, w = x.sign() * x.abs().clamp(min=1e-3) * x_scale, w.sign() * w.abs().clamp(min=1e-3) * w_scale
    got = _product(ops.sgemm_tc5, x, w, None)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    # as above, and the smallest float32 number for each of the sums that may end below 2^-126
    assert ((got.double() - want).abs() <= size * (2.0 ** -24 + 24 * 2.0 ** -23 + 41 * 2.0 ** -24) + 200 * 2.0 ** -149).all()


def test_captured():
    ops = _ops()
    x, w, b = _inputs(150, 256, 512)
    out = torch.empty(150, 256, device=DEV)
    ops.sgemm_tc5(x, w, b, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.sgemm_tc5(x, w, b, out)
    for value in (float("inf"), 1.0):
        x[3, 3] = value
        graph.replay()
        assert torch.equal(out.nan_to_num(1.25), _product(ops.sgemm_tc5, x, w, b).nan_to_num(1.25))


def test_which_products_take_it():
    ops = _ops()
    x, w, b = _inputs(80, 64, 256)
    assert torch.equal(ops.linear(x[:64], w, b), _product(ops.sgemm_nt, x[:64], w, b))
    assert torch.equal(ops.linear(x[:65], w, b), _product(ops.sgemm_tc5, x[:65], w, b))
    assert torch.equal(ops.linear(x, w[:63], b[:63]), _product(ops.sgemm_nt, x, w[:63], b[:63]))
    assert ops.linear(x.bfloat16(), w).dtype == torch.bfloat16          # rows of 16 bits stay with the multiply-adds
