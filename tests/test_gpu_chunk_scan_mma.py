"""The scans over chunks of sixteen tokens on the tensor cores against the same scans in float32 multiply-adds: requests
of one token to several chunks, segments, heads narrower than a record or a block's columns, states carried on."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _close(got, want):
    # every factor enters the products with its 24 bits: sums in another order, some of whose additions cut off instead of
    # rounding; each form is 1e-7 to 5e-7 off 64 bits (below)
    assert float((got - want).double().norm()) <= 2e-6 * float(want.double().norm()) + 1e-12
    assert ((got - want).abs() <= 1e-5 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("D,E", [(128, 128), (64, 64), (100, 72), (34, 200), (2, 16)])
@pytest.mark.parametrize("lens", [[1], [16, 15, 17], [200, 1, 33]])
@pytest.mark.parametrize("channel", [False, True])
def test_delta_rule(D, E, lens, channel):
    from paged_batch_engine_b200.csrc import ops
    T, H, G, R = sum(lens), 4, 2, len(lens)
    g = torch.Generator(device=DEV).manual_seed(T + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    qk = rand(T, G, 2, D)
    qk = (qk / qk.norm(dim=-1, keepdim=True)).contiguous()
    kq = (qk[:, :, 0] * qk[:, :, 1]).sum(-1).contiguous()
    v, beta = rand(T, H * E), torch.rand(T, H, device=DEV, generator=g)
    decay = torch.exp(-torch.rand(T, H * D if channel else H, device=DEV, generator=g) ** 4 * 8)
    start = rand(R + 1, H, E, D) * 0.3
    starts, slots = [sum(lens[:i]) for i in range(R)], list(range(R))[::-1]
    out = []
    for matrix in (False, True):
        state = start.clone()
        o = ops.delta_scan(qk, kq, v.clone(), beta, decay, state, _i32(starts), _i32(lens), _i32(slots), R, chunked=True,
                           matrix=matrix)
        out.append((o, state))
    _close(out[1][0], out[0][0])
    _close(out[1][1], out[0][1])
    assert torch.equal(out[1][1][R], start[R])


@pytest.mark.parametrize("D,E", [(128, 128), (64, 64), (100, 72), (2, 16)])
@pytest.mark.parametrize("lens,segment", [([1], 0), ([16, 15, 17], 0), ([300, 40, 129], 64), ([513], 128)])
def test_time_mixing(D, E, lens, segment):
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import RecurrencePlan, recurrence_plan_arrays
    T, H, R = sum(lens), 3, len(lens)
    g = torch.Generator(device=DEV).manual_seed(T + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    r, k, v = rand(T, H * D).bfloat16(), rand(T, H * D).bfloat16(), rand(T, H * E).bfloat16()
    decay = torch.exp(-torch.rand(T, H * D, device=DEV, generator=g) ** 4 * 8)
    bonus, start = rand(H * D), rand(R + 1, H, E, D)
    starts, slots = [sum(lens[:i]) for i in range(R)], list(range(R))[::-1]
    plan = None
    if segment:
        first, scan, second, entries = recurrence_plan_arrays(starts, lens, slots, segment)
        plan = RecurrencePlan(entries, _i32(first), len(first), _i32(scan), len(scan), _i32(second), len(second),
                              rows_per_chunk=segment)
    rows = _i32([i for i, n in enumerate(lens) for _ in range(n)])
    out = []
    for matrix in (False, True):
        state = start.clone()
        o = ops.wkv(r, k, v, decay, bonus, state, _i32(starts), _i32(lens), _i32(slots), R, H, chunked=True, plan=plan,
                    request_of_row=rows, matrix=matrix)
        out.append((o, state))
    _close(out[1][0], out[0][0])
    _close(out[1][1], out[0][1])


def _errors(y, state, o, S):
    return float((y.view(o.shape) - o).norm() / o.norm()), float((state[0] - S.transpose(1, 2)).norm() / S.norm())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("strength", [0.01, 1.0, 8.0])
@pytest.mark.parametrize("kind", ["delta", "mixing", "segments"])
def test_as_close_to_64_bits_as_the_multiply_adds(D, strength, kind):
    """Read-outs and the state that is carried on, of both forms, against the recurrence in float64 over hundreds of
    tokens; decays from hardly any to strong ones.  (Two bfloat16 terms a factor were ten to eighty times further off.)"""
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import RecurrencePlan, recurrence_plan_arrays
    T, H, E = 900, 3, 64
    g = torch.Generator(device=DEV).manual_seed(D + int(strength * 100))
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    decay = torch.exp(-torch.rand(T, H * D, device=DEV, generator=g) ** 4 * strength)
    start = rand(1, H, E, D) * 0.3
    S, o = start[0].double().transpose(1, 2), torch.empty(T, H, E, dtype=torch.float64, device=DEV)
    f = decay.double().view(T, H, D, 1)
    if kind == "delta":
        qk = rand(T, H, 2, D)
        qk = (qk / qk.norm(dim=-1, keepdim=True)).contiguous()
        kq = (qk[:, :, 0] * qk[:, :, 1]).sum(-1).contiguous()
        v, beta = rand(T, H * E), torch.rand(T, H, device=DEV, generator=g)
        for t in range(T):
            S, (q, k) = S * f[t], qk[t].double().unbind(1)
            u = beta[t].double()[:, None] * (v[t].double().view(H, E) - torch.einsum("hde,hd->he", S, k))
            S = S + k[:, :, None] * u[:, None]
            o[t] = torch.einsum("hde,hd->he", S, q)
    else:
        r, k, v, bonus = rand(T, H * D).bfloat16(), rand(T, H * D).bfloat16(), rand(T, H * E).bfloat16(), rand(H * D)
        for t in range(T):
            write = k[t].double().view(H, D, 1) * v[t].double().view(H, 1, E)
            o[t] = torch.einsum("hde,hd->he", S + bonus.double().view(H, D, 1) * write, r[t].double().view(H, D))
            S = S * f[t] + write
        plan = None
        if kind == "segments":
            first, scan, second, entries = recurrence_plan_arrays([0], [T], [0], 128)
            plan = RecurrencePlan(entries, _i32(first), len(first), _i32(scan), len(scan), _i32(second), len(second),
                                  rows_per_chunk=128)
    found = []
    for matrix in (True, False):
        state = start.clone()
        if kind == "delta":
            y = ops.delta_scan(qk, kq, v.clone(), beta, decay, state, _i32([0]), _i32([T]), _i32([0]), 1, chunked=True,
                               matrix=matrix)
        else:
            y = ops.wkv(r, k, v, decay, bonus, state, _i32([0]), _i32([T]), _i32([0]), 1, H, chunked=True, plan=plan,
                        request_of_row=_i32([0] * T), matrix=matrix)
        found.append(_errors(y, state, o, S))
    for got, plain in zip(*found):
        assert got <= 1.5 * plain, found
