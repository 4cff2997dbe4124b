"""Prompt portions of the window and pooled-block attention on tcgen05, at the edges of its row tiles (128), key tiles (64), window, blocks
and pages, with one and two key/value heads a block, in several goes, and with values that are not finite."""
import pytest
import torch

from tests.test_gpu_gebadra import _attention_part, _plain_attention_rounded_pool, _run_attention

pytestmark = pytest.mark.gpu
D = E = 128


def _case(H, G, window, pool, cuts, seed=0):
    T = sum(cuts)
    g = torch.Generator().manual_seed(H * 100 + window + seed)
    talk = torch.eye(H) + 0.3 * torch.randn(H, H, generator=g)
    part, hidden, _ = _attention_part(H, G, D, E, window, pool, torch.bfloat16, talk)
    part.scale = D ** -0.5
    n_in = (H + G) * D + G * E
    x = torch.zeros(T, hidden)
    x[:, :n_in] = torch.randn(T, n_in, generator=g)
    return part, x.bfloat16().float(), talk, n_in


def _run(part, x, cuts, page, H, tc5=True):
    T = sum(cuts)
    part._takes_tc5 = lambda ctx, seen: tc5
    return _run_attention(part, x, cuts, page, 2 * ((T + page - 1) // page + 1 + len(cuts)), torch.bfloat16)[:, :H * E]


@pytest.mark.parametrize("H,G,window,pool,page,cuts,goes", [
    (16, 4, 64, 16, 16, [97, 1, 128, 16, 129], False),
    (16, 4, 1024, 64, 16, [700, 250], True),
    (16, 2, 1, 1, 8, [130], False),                   # every older token a block of its own
    (8, 8, 100, 4, 64, [255, 65], False),
    (5, 5, 63, 7, 32, [64, 193], True),               # one key/value head a block
    (16, 1, 65, 32, 128, [127, 2, 300], False),
    (4, 2, 500, None, 16, [63, 400], False),          # no blocks
])
def test_portions(H, G, window, pool, page, cuts, goes, monkeypatch):
    from paged_batch_engine_b200.csrc import ops
    if goes:
        monkeypatch.setattr(ops, "POOLED_TC5_SCRATCH", 1)
    part, x, talk, n_in = _case(H, G, window, pool, cuts)
    T = sum(cuts)
    q, k, v = x[:, :H * D].reshape(T, H, D), x[:, H * D:(H + G) * D].reshape(T, G, D), x[:, (H + G) * D:n_in].reshape(T, G, E)
    want = _plain_attention_rounded_pool(q, k, v, talk, D ** -0.5, window, pool or 10 * T).reshape(T, H * E)
    got = _run(part, x, cuts, page, H)
    assert part._tc5
    # weights and mixture hold 24 bits, sums are float32: the bound is the result's own rounding to bfloat16 (2^-9 of it), doubled,
    # and as much of 0.05 for sums that cancel
    assert ((got - want).abs() <= 2 ** -8 * (want.abs() + 0.05)).all()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("place", [3, 70, 128, 290])
def test_values_that_are_not_finite(value, place):
    """They reach the rows that they reached on mma.sync, whose tiles are smaller, and no earlier ones."""
    H, G, window, pool, cuts = 16, 4, 100, 16, [300]
    part, x, _, n_in = _case(H, G, window, pool, cuts)
    x[place, (H + G) * D + 5] = value
    got = _run(part, x, cuts, 16, H)
    assert part._tc5
    want = _run(part, x, cuts, 16, H, tc5=False)
    bad = ~torch.isfinite(want)
    assert bad.any() and torch.equal(bad, ~torch.isfinite(got)) and torch.isfinite(got[:place // 16 * 16]).all()
    assert ((got - want)[~bad].abs() <= 2 ** -7 * (want[~bad].abs() + 0.05)).all()      # either off by its own rounding


def test_which_steps_take_it():
    import numpy as np
    part, _, _, _ = _case(16, 4, 1024, 64, [4])

    def takes(*reqs):
        class Step:
            q_len_host, seq_len_host = np.array([n for _, n in reqs]), np.array([c + n for c, n in reqs])
        longest = int(Step.seq_len_host.max())
        return part._takes_tc5(Step(), min(longest, 1024 + 16) + longest // 64)
    assert takes((0, 2048)) and takes((0, 400)) and takes((1057, 16)) and takes((0, 8192)) and takes((0, 700), (0, 80), (0, 33))
    assert not takes((0, 100)) and not takes((300, 16)) and not takes(*[(1000, 1)] * 30, (0, 64))
