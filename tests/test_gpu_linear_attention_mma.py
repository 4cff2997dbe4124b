"""The decayed recurrence as products of matrices (chunks of 64 tokens) against the recurrence in float64: edges of
chunks and work items, strong decays and ones that underflow, states that are carried on; and the gated norm per head."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D,E", [(128, 64), (64, 64), (64, 128)])
@pytest.mark.parametrize("lens,chunk,decays", [([1], None, "mild"), ([63, 64, 65], None, "mild"), ([200, 17], None, "strong"),
                                               ([300, 40, 129], 64, "mild"), ([700], 128, "strong")])
def test_matrix_form(D, E, lens, chunk, decays):
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import RecurrencePlan, recurrence_plan_arrays
    H, share, T = 4, 2, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(T + D)
    q, k = (torch.randn(T, H // share * D, device=DEV, generator=g).bfloat16() / D ** 0.25 for _ in range(2))
    v = torch.randn(T, H * E, device=DEV, generator=g).bfloat16()
    wide = torch.cat([q, k, v], 1).contiguous()
    q, k, v = wide[:, :q.shape[1]], wide[:, q.shape[1]:2 * q.shape[1]], wide[:, 2 * q.shape[1]:]
    dt = torch.rand(T, H, device=DEV, generator=g) * 0.2
    rate = torch.tensor([0.5, 2.0, 8.0, 40.0], device=DEV) * (1.0 if decays == "mild" else 30.0)
    if decays == "strong":       # some tokens keep everything, some nothing at all
        dt = torch.where(torch.rand(T, H, device=DEV, generator=g) < 0.5, dt * 1e-6, dt)
    a = torch.exp(-rate * dt)
    skip = torch.randn(H, device=DEV, generator=g)
    state = torch.randn(len(lens) + 1, H, D, E, device=DEV, generator=g)
    start = state.double().clone()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    slots = list(range(len(lens)))[::-1]
    plan = None
    if chunk:
        first, scan, second, entries = recurrence_plan_arrays(starts, lens, slots, chunk)
        plan = RecurrencePlan(entries, i32(first), len(first), i32(scan), len(scan), i32(second), len(second), rows_per_chunk=chunk)
    out = ops.linear_attention(q, k, v, state, None, i32(starts), i32(lens), i32(slots), len(lens), H, plan=plan,
                               tok_decay=a, tok_scale=dt, skip=skip, kq_share=share, matrix=True)
    qd, kd = (x.double().view(T, H // share, D).repeat_interleave(share, 1) for x in (q, k))
    vd = v.double().view(T, H, E)
    want = torch.empty(T, H, E, dtype=torch.float64, device=DEV)
    size = torch.empty_like(want)         # the same sums over absolute values: what the errors are relative to
    for s0, n, slot in zip(starts, lens, slots):
        S, A = start[slot], start[slot].abs()
        for t in range(s0, s0 + n):
            w = a[t].double()[:, None, None]
            write = kd[t][:, :, None] * (dt[t].double()[:, None] * vd[t])[:, None, :]
            S, A = w * S + write, w * A + write.abs()
            want[t] = torch.einsum("hde,hd->he", S, qd[t]) + skip.double()[:, None] * vd[t]
            size[t] = torch.einsum("hde,hd->he", A, qd[t].abs()) + (skip.double()[:, None] * vd[t]).abs()
        assert ((state[slot].double() - S).abs() <= 2 ** -20 * A + 1e-12).all()
    # every factor enters the products with its 24 bits; exponentials and some forty additions that round or cut off, by
    # 2^-23 of what they add to at most, most of them far less
    assert ((out.double().view(T, H, E) - want).abs() <= 2 ** -19 * size).all()
    assert torch.equal(state[len(lens)].double(), start[len(lens)])


@pytest.mark.parametrize("D,E", [(128, 64), (64, 64), (64, 128)])
@pytest.mark.parametrize("rate", [0.05, 1.0])
@pytest.mark.parametrize("chunk", [None, 128])
def test_as_close_to_64_bits_as_the_recurrence(D, E, rate, chunk):
    """The matrix form against the recurrence token by token, both measured against float64: read-outs and the state that
    is carried on.  (Two bfloat16 terms a factor were ten to thirty times further off.)"""
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import RecurrencePlan, recurrence_plan_arrays
    T, H = 700, 4
    g = torch.Generator(device=DEV).manual_seed(D + E)
    wide = torch.randn(T, H * (2 * D + E), device=DEV, generator=g).bfloat16()
    q, k, v = wide[:, :H * D], wide[:, H * D:2 * H * D], wide[:, 2 * H * D:]
    dt = torch.exp(torch.rand(T, H, device=DEV, generator=g) * 4.6 - 6.9)          # 0.001 to 0.1
    a = torch.exp(-rate * (1 + 15 * torch.rand(H, device=DEV, generator=g)) * dt)
    start = torch.randn(1, H, D, E, device=DEV, generator=g) * 0.1
    S, o = start[0].double(), torch.empty(T, H, E, dtype=torch.float64, device=DEV)
    for t in range(T):
        S = a[t].double()[:, None, None] * S + k[t].double().view(H, D, 1) * (dt[t].double()[:, None] * v[t].double().view(H, E))[:, None]
        o[t] = torch.einsum("hde,hd->he", S, q[t].double().view(H, D))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    plan = None
    if chunk:
        first, scan, second, entries = recurrence_plan_arrays([0], [T], [0], chunk)
        plan = RecurrencePlan(entries, i32(first), len(first), i32(scan), len(scan), i32(second), len(second), rows_per_chunk=chunk)

    def errors(matrix):
        state = start.clone()
        y = ops.linear_attention(q, k, v, state, None, i32([0]), i32([T]), i32([0]), 1, H, plan=plan, tok_decay=a, tok_scale=dt,
                                 matrix=matrix)
        return float((y.view(T, H, E) - o).norm() / o.norm()), float((state[0] - S).norm() / S.norm())
    for got, plain in zip(errors(True), errors(False)):
        assert got <= 1.5 * plain, (got, plain)


@pytest.mark.parametrize("D,E", [(128, 64), (64, 64), (64, 128)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 13, 15, 16, 70, 99])
def test_what_is_not_finite_stays_behind_its_token(D, E, value, at):
    """A token's value reaches its own output and later ones, as in the recurrence token by token, never an earlier one."""
    from paged_batch_engine_b200.csrc import ops
    T, H = 100, 2
    g = torch.Generator(device=DEV).manual_seed(at + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v = (rand(T, H * D).bfloat16(), rand(T, H * D).bfloat16(), rand(T, H * E).bfloat16())
    a, dt = torch.exp(-0.1 * rand(T, H).abs()), rand(T, H).abs()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def run(v, matrix):
        state = torch.zeros(1, H, D, E, device=DEV)
        wide = torch.cat([q, k, v], 1).contiguous()
        parts = wide[:, :H * D], wide[:, H * D:2 * H * D], wide[:, 2 * H * D:]
        o = ops.linear_attention(*parts, state, None, i32([0]), i32([T]), i32([0]), 1, H, tok_decay=a, tok_scale=dt,
                                 matrix=matrix)
        return o.view(T, H, E), state
    clean, _ = run(v, True)
    v2 = v.clone()
    v2.view(T, H, E)[at, 1, 5] = value
    got, state = run(v2, True)
    want, want_state = run(v2, False)
    # the tokens of its tile of sixteen are added one by one, not as terms: another order of sums
    assert ((got[:at] - clean[:at]).abs() <= 2 ** -19 * clean.abs().max()).all()
    assert torch.equal(got.isfinite(), want.isfinite()) and torch.equal(state.isfinite(), want_state.isfinite())
    assert torch.equal(got[:, 0], clean[:, 0])             # nor another head's


@pytest.mark.parametrize("E", [4, 64, 100, 128, 256, 512, 132])
@pytest.mark.parametrize("gate_first", [False, True])
@pytest.mark.parametrize("dtype,gate_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16),
                                              (torch.bfloat16, torch.float32)])
def test_gated_norm_per_head(E, gate_first, dtype, gate_dtype):
    from paged_batch_engine_b200.csrc import ops
    T, H = 13, 3
    g = torch.Generator(device=DEV).manual_seed(E)
    o = torch.randn(T, H * E, device=DEV, generator=g) * 3
    wide = torch.randn(T, 2 * H * E + 4, device=DEV, generator=g).to(gate_dtype)
    gain = torch.randn(H * E, device=DEV, generator=g)
    for off in (0, 4, 1):               # 1: a gate that lies on no boundary
        gate = wide[:, off:off + H * E]
        for act in ("silu", "sigmoid"):
            got = ops.gated_rms(o, gate, gain, H, 1e-6, True, act, dtype, gate_first).double()
            s = torch.sigmoid(gate.double()) * (gate.double() if act == "silu" else 1.0)
            u = o.double() * s if gate_first else o.double()
            n = u.view(T, H, E) / torch.sqrt((u.view(T, H, E) ** 2).mean(-1, keepdim=True) + 1e-6)
            want = n.reshape(T, H * E) * gain.double() * (1.0 if gate_first else s)
            tol = 2 ** -8 if dtype == torch.bfloat16 else 2e-6
            assert ((got - want).abs() <= tol * (want.abs() + 1e-3)).all()


@pytest.mark.parametrize("E", [64, 512])
@pytest.mark.parametrize("gate_dtype", [torch.float32, torch.bfloat16])
def test_gates_that_are_almost_closed(E, gate_dtype):
    """Gates so negative that their sigmoid is close to float32's smallest normal number, with rows that are rounded to
    bfloat16 and bring the result back to an ordinary size."""
    from paged_batch_engine_b200.csrc import ops
    T, H = 5, 2
    g = torch.Generator(device=DEV).manual_seed(E)
    gate = (-80.0 - 8.5 * torch.rand(T, H * E, device=DEV, generator=g)).to(gate_dtype)
    o = torch.rand(T, H * E, device=DEV, generator=g) + 0.5
    gain = torch.full((H * E,), 1e30, device=DEV)
    got = ops.gated_rms(o, gate, gain, H, 1e-6, True, "silu", torch.bfloat16).double()
    n = o.double().view(T, H, E) / torch.sqrt((o.double().view(T, H, E) ** 2).mean(-1, keepdim=True) + 1e-6)
    want = n.reshape(T, H * E) * 1e30 * gate.double() * torch.sigmoid(gate.double())
    # the sigmoid may lie just below 2^-126, where a number holds 22 bits and more; the result is rounded to bfloat16
    assert ((got - want).abs() <= (2 ** -8 + 2 ** -16) * want.abs()).all()
