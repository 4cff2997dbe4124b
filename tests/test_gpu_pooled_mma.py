"""Prompt portions of the window and pooled-block attention on the tensor cores, at the edges of its row tiles (16),
key tiles (32, or 16 with many key/value heads), window and blocks, against the plain function in float32."""
import pytest
import torch

from tests.test_gpu_gebadra import _attention_part, _plain_attention_rounded_pool, _run_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,D,E,window,pool,page,cuts", [
    (16, 4, 128, 128, 64, 16, 16, [97, 1, 33, 16, 2]),
    (16, 4, 128, 128, 33, 32, 16, [31, 32, 65]),
    (8, 8, 128, 128, 20, 4, 8, [48, 17]),             # sixteen keys a tile
    (16, 2, 128, 128, 1, 1, 16, [35]),                # every older token a block of its own
    (5, 1, 32, 32, 40, 7, 8, [50, 3]),
    (1, 1, 64, 16, 16, None, 16, [15, 2, 40]),        # no blocks, no mixture
])
def test_portions(H, G, D, E, window, pool, page, cuts):
    from paged_batch_engine_b200.csrc import ops
    assert ops.pooled_mma_applies(torch.bfloat16, H, D, E) and ops.pooled_mma_fits(H, G, D, E)
    T = sum(cuts)
    g = torch.Generator().manual_seed(H * 100 + window)
    talk = torch.eye(H) + 0.3 * torch.randn(H, H, generator=g) if pool else None
    part, hidden, _ = _attention_part(H, G, D, E, window, pool, torch.bfloat16, talk)
    part.scale = D ** -0.5
    n_in = (H + G) * D + G * E
    x = torch.zeros(T, hidden)
    x[:, :n_in] = torch.randn(T, n_in, generator=g)
    x = x.bfloat16().float()
    q, k, v = x[:, :H * D].reshape(T, H, D), x[:, H * D:(H + G) * D].reshape(T, G, D), x[:, (H + G) * D:n_in].reshape(T, G, E)
    mix = torch.eye(H) if talk is None else talk
    # without blocks: one that is never whole
    want = _plain_attention_rounded_pool(q, k, v, mix, D ** -0.5, window, pool or 10 * T).reshape(T, H * E)
    got = _run_attention(part, x, cuts, page, 2 * ((T + page - 1) // page + 1), torch.bfloat16)[:, :H * E]
    # probabilities and mixture hold seventeen bits, sums are float32: the bound is the result's own rounding to
    # bfloat16 (2^-9 of it), doubled, and as much of 0.05 for sums that cancel
    assert ((got - want).abs() <= 2 ** -8 * (want.abs() + 0.05)).all()


def test_as_close_to_64_bits_as_the_multiply_adds(monkeypatch):
    """A mixture of heads that see nearly the same and takes their mean away, so that the weights' last bits show: both forms
    against float64, whose results they round to bfloat16."""
    from paged_batch_engine_b200.csrc import ops
    from tests.plain import plain_gebadra as pg
    H, G, D, E, window, pool, T = 16, 4, 128, 128, 64, 16, 150
    g = torch.Generator().manual_seed(5)
    talk = torch.eye(H) - 1.0 / H
    part, hidden, _ = _attention_part(H, G, D, E, window, pool, torch.bfloat16, talk)
    part.scale = 0.05 * D ** -0.5
    n_in = (H + G) * D + G * E
    x = torch.zeros(T, hidden)
    x[:, :n_in] = torch.randn(T, n_in, generator=g)
    x = x.bfloat16().float()
    q, k, v = (x[:, a:b].double().reshape(T, n, D) for a, b, n in ((0, H * D, H), (H * D, (H + G) * D, G), ((H + G) * D, n_in, G)))
    kp, vp = (z[:T // pool * pool].reshape(T // pool, pool, G, D).mean(1).bfloat16().double() for z in (k, v))
    want = torch.zeros(T, H, E, dtype=torch.float64)
    for t in range(T):
        seen, first = pg.visible_keys(t, window, pool)
        keys, values = (torch.cat([a[:seen], b[first:t + 1]]).repeat_interleave(H // G, 1) for a, b in ((kp, k), (vp, v)))
        w = torch.softmax(torch.einsum("jhd,hd->hj", keys, q[t]) * part.scale, -1)
        want[t] = torch.einsum("hj,jhe->he", talk.double() @ w, values)
    off = []
    for fits in (True, False):
        monkeypatch.setattr(ops, "pooled_mma_fits", lambda *a: fits)
        part._tile_rows = None
        got = _run_attention(part, x, [T], 16, 40, torch.bfloat16)[:, :H * E].double().reshape(T, H, E)
        off.append(float((got - want).norm() / want.norm()))
    assert off[0] <= (1 + 5e-5) * off[1], off           # two bfloat16 terms a weight: 1 + 5e-4
