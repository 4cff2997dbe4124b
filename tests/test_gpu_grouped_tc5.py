"""The experts' products on tcgen05 (rows sorted by expert in tiles of 128) against plain float32 products, and the
launches that sort the rows: edges of row tiles, column blocks and K steps, experts without rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _activated(z, activation, limit, alpha):
    if activation is None:
        return z
    if activation == "relu2":
        return torch.relu(z) ** 2
    g, u = z.chunk(2, dim=-1)
    if activation == "silu":
        return torch.nn.functional.silu(g) * u
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(alpha * g) * (u + 1.0)


@pytest.mark.parametrize("activation", [None, "relu2", "silu", "capped_swish"])
@pytest.mark.parametrize("T,K,N,E,top", [(1, 8, 2, 1, 1), (16, 64, 256, 3, 2), (129, 72, 258, 4, 1), (300, 200, 130, 5, 3),
                                         (1000, 136, 528, 300, 2), (700, 2048, 320, 7, 4)])
def test_sorted_rows_through_the_experts(T, K, N, E, top, activation):
    from paged_batch_engine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T * 7 + N)
    x = torch.randn(T, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(E, N, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    # the last expert is chosen by nobody where there is more than enough
    live = E - 1 if E > top else E
    chosen = torch.rand(T, live, device=DEV, generator=g).topk(top, -1).indices.to(torch.int32).contiguous()
    counts, place = ops.expert_places(chosen, E)
    flat = chosen.flatten().long()
    assert torch.equal(counts.long(), torch.bincount(flat, minlength=E))
    for e in range(min(E, 8)):
        mine = place[flat == e]
        assert torch.equal(mine.long(), torch.arange(mine.numel(), device=DEV))        # pair order inside a run
    rows = ops.GROUPED_TC5_ROWS
    max_tiles = (T * top + rows - 1) // rows + E
    start, tiles = ops.run_tiles(counts, max_tiles, rows)
    own = (counts + rows - 1) // rows
    assert torch.equal(start, ((torch.cumsum(own, 0) - own) * rows).to(torch.int32))
    assert int((tiles[:, 0] >= 0).sum()) == int(own.sum()) and int(tiles[tiles[:, 0] >= 0][:, 2].sum()) == T * top
    gathered = ops.expert_gather(x, chosen, place, start, total_rows=max_tiles * rows)
    at = (start[flat] + place).long()
    assert torch.equal(gathered[at], x.repeat_interleave(top, 0))
    got = ops.grouped_runs_tc5(gathered, w, tiles, activation, limit=1.5, alpha=1.702)[at].float()
    ops.raise_on_kernel_status(DEV)
    want = torch.empty_like(got)
    for e in range(E):
        of_e = flat == e
        want[of_e] = _activated(x.repeat_interleave(top, 0)[of_e].double() @ w[e].double().t(), activation, 1.5, 1.702).float()
    # operands are exact, sums float32 (relative 2^-24 sqrt(K) of numbers around 1), the result is rounded to
    # bfloat16 (2^-9 of its size): 2^-8 of the result and as much of 1 covers both
    assert ((got - want).abs() <= 2 ** -8 * (want.abs() + 1.0)).all()
    # the way back: the sum over a token's experts, in float32, rounded once
    if activation is None and T > 1:
        y = torch.randn(max_tiles * rows, N, device=DEV, generator=g).bfloat16()
        weights = torch.rand(T, top, device=DEV, generator=g)
        back = ops.expert_scatter(y, chosen, place, start, weights, T).float()
        plain = (y[at].float().view(T, top, N) * weights[..., None]).sum(1)
        assert ((back - plain).abs() <= 2 ** -8 * (plain.abs() + 1e-3)).all()
