"""Row tiles of every height for the experts' tcgen05 products: runs that lie one behind the other, tiles that share a
run's rows evenly, more tiles than a band, output widths off the eight columns of a store; and one group without a list."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# rows of each expert: the edges of the sixteen rows of a product, of the boxes the rows come in, and of a tile
COUNTS = {"edges": [0, 1, 15, 16, 17, 0, 31, 33, 127, 128, 129, 240, 255, 256, 257, 264, 511, 513, 0],
          "one_row_each": [1] * 9, "one_long_run": [0, 2100, 3]}


def _close(got, want):
    # exact operands, float32 sums (2^-24 sqrt(K) of numbers around 1), a result rounded to bfloat16 (2^-9 of its size)
    return ((got.double() - want).abs() <= 2 ** -8 * (want.abs() + 1.0)).all()


def _runs(counts, K, N, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = torch.randn(sum(counts), K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(len(counts), N, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    return a, w


@pytest.mark.parametrize("counts", list(COUNTS))
def test_even_tiles(counts):
    from paged_batch_engine_b200.csrc import ops
    counts = COUNTS[counts]
    most = ops.most_run_tiles(sum(counts), len(counts), ops.GROUPED_TC5_ROWS)
    start, tiles = ops.run_tiles(torch.tensor(counts, dtype=torch.int32, device=DEV), most, ops.GROUPED_TC5_ROWS, padded=False)
    first, seen = 0, []
    for e, n in enumerate(counts):
        assert start[e] == first
        own = -(-n // ops.GROUPED_TC5_ROWS)
        height = -(-n // (16 * own)) * 16 if own else 0
        seen += [[e, first + j * height, min(height, n - j * height)] for j in range(own)]
        first += n
    seen += [[-1, 0, 0]] * (most - len(seen))
    assert tiles.tolist() == seen


@pytest.mark.parametrize("activation", [None, "silu"])
@pytest.mark.parametrize("counts,K,N", [("edges", 136, 264), ("edges", 64, 250), ("edges", 520, 656), ("one_row_each", 2048, 512),
                                        ("one_long_run", 72, 1040)])
def test_products_of_every_height(counts, K, N, activation):
    from paged_batch_engine_b200.csrc import ops
    counts = COUNTS[counts]
    a, w = _runs(counts, K, N, K + N)
    most = ops.most_run_tiles(sum(counts), len(counts), ops.GROUPED_TC5_ROWS)
    _, tiles = ops.run_tiles(torch.tensor(counts, dtype=torch.int32, device=DEV), most, ops.GROUPED_TC5_ROWS, padded=False)
    got = ops.grouped_runs_tc5(a, w, tiles, activation)
    ops.raise_on_kernel_status(DEV)
    first = 0
    for e, n in enumerate(counts):
        want = a[first:first + n].double() @ w[e].double().t()
        if activation:
            gate, up = want.chunk(2, dim=-1)
            want = torch.nn.functional.silu(gate) * up
        assert _close(got[first:first + n], want), e
        first += n


@pytest.mark.parametrize("rows", [1, 256, 257, 2500])
def test_one_group(rows):
    from paged_batch_engine_b200.csrc import ops
    a, w = _runs([rows], 512, 384, rows)
    got = ops.grouped_runs_tc5(a, w, None)
    ops.raise_on_kernel_status(DEV)
    assert _close(got, a.double() @ w[0].double().t())
