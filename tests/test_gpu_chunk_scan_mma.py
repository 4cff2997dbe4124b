"""The scans over chunks of sixteen tokens on the tensor cores against the same scans in float32 multiply-adds: requests
of one token to several chunks, segments, heads narrower than a record or a block's columns, states carried on."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _close(got, want):
    # a factor's two terms hold seventeen bits and the product of the lower ones is left out: 2^-16 of an addend, which
    # the sums carry on in both passes; the read-outs and states are sums of many of them
    assert float((got - want).double().norm()) <= 3e-5 * float(want.double().norm()) + 1e-12
    assert ((got - want).abs() <= 2e-3 * want.abs() + 2e-4 * want.abs().max()).all()


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
