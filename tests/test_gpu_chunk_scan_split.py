"""The delta rule's scan over chunks with two and four warps to sixteen columns (few long requests): against the multiply-adds, at edges
of the warps' key channels and the blocks' columns, and against 64 bits."""
import pytest
import torch

from tests.test_gpu_chunk_scan_mma import DEV, _close, _i32

pytestmark = pytest.mark.gpu


def _case(D, E, H, lens, seed=0):
    T = sum(lens)
    g = torch.Generator(device=DEV).manual_seed(T + D + seed)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    qk = rand(T, H // 2, 2, D)
    qk = (qk / qk.norm(dim=-1, keepdim=True)).contiguous()
    kq = (qk[:, :, 0] * qk[:, :, 1]).sum(-1).contiguous()
    decay = torch.exp(-torch.rand(T, H * D, device=DEV, generator=g) ** 4 * 8)
    return qk, kq, rand(T, H * E), torch.rand(T, H, device=DEV, generator=g), decay, rand(len(lens) + 1, H, E, D) * 0.3


def _run(case, lens, longest, matrix=True):
    from paged_batch_engine_b200.csrc import ops
    qk, kq, v, beta, decay, start = case
    state, R = start.clone(), len(lens)
    o = ops.delta_scan(qk, kq, v.clone(), beta, decay, state, _i32([sum(lens[:i]) for i in range(R)]), _i32(lens),
                       _i32(list(range(R))[::-1]), R, chunked=True, matrix=matrix, longest=longest)
    return o, state


@pytest.mark.parametrize("D,E,H,lens,longest", [
    (128, 128, 4, [200, 1, 33], 200), (64, 64, 4, [31], 31), (100, 72, 2, [16, 15, 17], 17), (34, 200, 2, [65], 65),      # four warps
    (2, 16, 2, [40], 40),
    (128, 128, 16, [90, 7, 80], 90), (64, 72, 32, [50, 60], 60), (100, 40, 46, [33], 33),                                  # two
])
def test_against_the_multiply_adds(D, E, H, lens, longest):
    case = _case(D, E, H, lens)
    one, split, fma = _run(case, lens, 0), _run(case, lens, longest), _run(case, lens, longest, matrix=False)
    for a, b, c in zip(split, fma, one):
        _close(a, b)
        _close(a, c)
    assert torch.equal(split[1][-1], case[-1][-1])


@pytest.mark.parametrize("H,E", [(2, 64), (16, 128)])
def test_as_close_to_64_bits(H, E):
    D, lens = 128, [400, 300]
    case = _case(D, E, H, lens, seed=1)
    qk, kq, v, beta, decay, start = case
    o, states, t0 = torch.empty(700, H, E, dtype=torch.float64, device=DEV), [], 0
    for i, n in enumerate(lens):
        S = start[len(lens) - 1 - i].double().transpose(1, 2)
        for t in range(t0, t0 + n):
            S = S * decay[t].double().view(H, D, 1)
            q, k = (qk[t, :, j].double().repeat_interleave(2, 0) for j in (0, 1))
            u = beta[t].double()[:, None] * (v[t].double().view(H, E) - torch.einsum("hde,hd->he", S, k))
            S = S + k[:, :, None] * u[:, None]
            o[t] = torch.einsum("hde,hd->he", S, q)
        states.insert(0, S.transpose(1, 2))
        t0 += n
    want = torch.stack(states)

    def off(got):
        return [float((a.double() - b).norm() / b.norm()) for a, b in ((got[0].view(o.shape), o), (got[1][:-1], want))]
    split, one, fma = off(_run(case, lens, 400)), off(_run(case, lens, 0)), off(_run(case, lens, 0, matrix=False))
    assert all(a <= 1.4 * max(b, c) for a, b, c in zip(split, one, fma)), (split, one, fma)
    print(split, one, fma)


@pytest.mark.parametrize("D,E,H,lens", [(128, 128, 16, [144, 90, 130, 17]), (128, 128, 16, [33, 144]), (64, 64, 32, [95, 96, 80, 2, 90]),
                                        (100, 72, 16, [70, 64, 66])])
def test_a_request_alone_and_beside_others(D, E, H, lens):
    """One, two or four warps to sixteen columns, as its neighbours in the step let the blocks be cut: a request has the same bits."""
    qk, kq, v, beta, decay, start = case = _case(D, E, H, lens, seed=2)
    together, t0 = _run(case, lens, max(lens)), 0
    for i, n in enumerate(lens):
        slot, rows = len(lens) - 1 - i, slice(t0, t0 + n)
        own = (qk[rows].contiguous(), kq[rows].contiguous(), v[rows].contiguous(), beta[rows].contiguous(), decay[rows].contiguous(),
               start[slot:slot + 1].contiguous())
        alone = _run(own, [n], n)
        assert torch.equal(alone[0], together[0][rows])
        assert torch.equal(alone[1][0], together[1][slot])
        t0 += n
