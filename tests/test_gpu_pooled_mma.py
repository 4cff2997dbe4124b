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
