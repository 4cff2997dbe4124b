"""The kernels that norm, turn and write heads in pieces of four channels against those for one channel an access, which
the same rows take when they start one element further."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _close(a, b, dtype):
    # a norm's sum of squares is added in another order: at most 4,096 * 2^-24 of it, half of that in the result; rounded
    # to bfloat16 that is at most one step, which for eight significant bits is 2^-8 to 2^-7 of the value
    rel = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -13
    assert ((a.float() - b.float()).abs() <= rel * b.float().abs() + rel * 1e-2).all()


@pytest.mark.parametrize("H,G,D,E", [(16, 4, 128, 128), (3, 2, 64, 32), (1, 1, 4, 8), (7, 1, 100, 24)])
@pytest.mark.parametrize("dims", [0, 8, -1])                   # channels that turn: none, some, the most that are whole eights
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("plain", [False, True])
def test_head_norm_write(H, G, D, E, dims, dtype, plain):
    from paged_batch_engine_b200.csrc import ops
    dims = min(D // 8 * 8, 8 if dims == 8 else D) if dims else 0
    T, page = 37, 4
    g = torch.Generator(device=DEV).manual_seed(D + H)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    wide = (H + G) * D + G * E
    rows, bias, scale = rand(T, wide).to(dtype), rand(wide), rand(H)
    gains = (None, None) if plain else (rand(D), rand(D))
    slots, positions = _i32([i if i % 5 else -1 for i in range(T)]), _i32([37 * i for i in range(T)])
    turn = ops.turn_frequencies(dims // 2, 1e4, DEV) if dims else None
    value_turn = ops.turn_frequencies(E // 2, 1e4, DEV) if dims and not plain else None
    out = []
    for first in (0, 1):
        proj = torch.zeros(T, wide + 8 - wide % 4, dtype=dtype, device=DEV)
        proj[:, first:first + wide] = rows
        b = torch.zeros(proj.shape[1], device=DEV)
        b[first:first + wide] = bias
        k_pages = torch.full((10, G, page, D), 7.0, dtype=dtype, device=DEV)
        v_pages = torch.full((10, G, page, E), 7.0, dtype=dtype, device=DEV)
        q = ops.head_norm_write(proj, first, first + H * D, first + (H + G) * D, None if plain else b, *gains, slots, k_pages, v_pages,
                                H, G, D, E, page, 1e-5, q_head_scale=None if plain else scale,
                                positions=positions if dims else None, rot_freq=turn, value_freq=value_turn)
        q = q if isinstance(q, tuple) else (q,)
        out.append((q[0], k_pages, v_pages) + tuple(x for x in q[1:] if x is not None))
    for i, (a, b) in enumerate(zip(*out)):
        _close(a, b, dtype if i in (1, 2) else torch.float32)


@pytest.mark.parametrize("H,G,D,E,rot", [(16, 4, 128, 128, 128), (12, 4, 256, 64, 100), (3, 1, 36, 20, 34), (2, 2, 4, 4, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("plain", [False, True])
def test_qk_prepare(H, G, D, E, rot, dtype, plain):
    from paged_batch_engine_b200.csrc import ops
    T, page = 37, 4
    g = torch.Generator(device=DEV).manual_seed(D + H)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    wide = (H + G) * D + G * E
    rows = rand(T, wide).to(dtype)
    gains = (None, None) if plain else (rand(H * D), rand(G * D))
    freq = torch.rand(rot // 2, device=DEV, generator=g) if rot else None
    slots, positions = _i32([i if i % 5 else -1 for i in range(T)]), _i32([37 * i for i in range(T)])
    out = []
    for first in (0, 1):
        proj = torch.zeros(T, wide + 8 - wide % 4, dtype=dtype, device=DEV)
        proj[:, first:first + wide] = rows
        parts = proj[:, first:first + wide].split([H * D, G * D, G * E], dim=1)
        k_pages = torch.full((10, G, page, D), 7.0, dtype=dtype, device=DEV)
        v_pages = torch.full((10, G, page, E), 7.0, dtype=dtype, device=DEV)
        q = ops.qk_prepare(*parts, *gains, freq, rot, positions, slots, k_pages, v_pages, H, G, 1e-5, page)
        out.append((q, k_pages, v_pages))
    for a, b in zip(*out):
        _close(a, b, dtype)
