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


@pytest.mark.parametrize("W", [128, 2052, 2048])
def test_what_reads_the_result_next(W):
    """The kernels that read the experts' result start while it is written: over inputs that change from call to call,
    with the same buffers handed out again, each of them sees the call's own result."""
    from paged_batch_engine_b200.csrc import ops
    T, top, E = 257, 3, 5
    g = torch.Generator(device=DEV).manual_seed(W)
    chosen = torch.rand(T, E, device=DEV, generator=g).topk(top, -1).indices.to(torch.int32).contiguous()
    counts, place = ops.expert_places(chosen, E)
    max_tiles = (T * top + 127) // 128 + E
    start, _ = ops.run_tiles(counts, max_tiles, 128)
    weights = torch.rand(T, top, device=DEV, generator=g)
    gain = torch.rand(W, device=DEV, generator=g)
    ys = [torch.randn(max_tiles * 128, W, device=DEV, generator=g).bfloat16() for _ in range(3)]
    xs = [torch.randn(T, W, device=DEV, generator=g) for _ in range(3)]

    def chain(i, wait):
        def scattered():
            y = ops.expert_scatter(ys[i % 3], chosen, place, start, weights, T)
            if wait:
                torch.cuda.synchronize()
            return y
        x1, x2 = xs[i % 3].clone(), xs[(i + 1) % 3].clone()
        out = [*ops.add2_rmsnorm2(x1, scattered(), None, gain, gain, 1e-5, torch.bfloat16), x1]
        out.append(ops.norm_add(x2, scattered(), gain, 1e-5, torch.bfloat16))
        out.append(ops.fold_pair(xs[i % 3], scattered(), None, 0.5, xs[2], torch.bfloat16))
        return out
    want = [chain(i, True) for i in range(3)]
    got = [chain(i, False) for i in range(30)]
    for i, outs in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(outs, want[i % 3])), i
