"""The sampling kernel's three ways to a token (the threads' maxima for the first k, bins, radix descent) give the same one, over row
lengths around the loads' groups and the clusters' slices, equal logits, masks and what is no number; and the draws of many rows
made at once are those made one by one."""
import pytest
import torch

from paged_batch_engine_b200.sampling.params import request_sample_uniform, request_sample_uniforms

DEV = "cuda:0"


def _tokens(logits, k, p, t, u):
    from paged_batch_engine_b200.csrc import ops
    n = logits.shape[0]
    full = lambda x, dt: torch.full((n,), x, dtype=dt, device=DEV)
    out = []
    for mode in (0, 2, 1):
        ops.sample_set_mode(mode)
        try:
            out.append(ops.sample(logits, full(t, torch.float32), full(k, torch.int32), full(p, torch.float32), u).tolist())
        finally:
            ops.sample_set_mode(0)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("V,rows,stride", [(5, 3, 5), (200, 3, 203), (1000, 4, 1000), (1027, 3, 1028), (8191, 5, 8191), (8192, 20, 8192), (9001, 40, 9003),
                                           (32000, 64, 32000), (40001, 100, 40001), (152064, 64, 152064), (151936, 150, 151936)])
@pytest.mark.parametrize("kind", ["normal", "coarse", "equal", "masked"])
def test_three_ways(V, rows, stride, kind):
    g = torch.Generator(device=DEV).manual_seed(V + rows)
    x = torch.empty(rows, stride, device=DEV).normal_(0, 2.5, generator=g)
    if kind == "coarse":
        x = (x * 2).round() / 2
    elif kind == "equal":
        x = x.sign()
    elif kind == "masked":
        x[:, ::3] = float("-inf")
        x[:, 1::7] = float("nan")
        x[0] = float("-inf")
        x[-1, V // 2] = 1e9
    x = x[:, :V]
    u = torch.rand(rows, device=DEV, generator=g)
    for k in {1, 2, 50, 127, 128, 129, 511, 512, 513, V - 1, 0} - ({0} if V > 100000 and kind == "equal" else set()):
        for p, t in ((1.0, 0.8), (0.9, 0.8), (0.0, 1.5), (0.5, 1e-7)):
            top, bins, radix = _tokens(x, k, p, t, u)
            assert top == bins == radix, (k, p, t)


@pytest.mark.gpu
@pytest.mark.parametrize("V,rows", [(200, 3), (9001, 5), (32000, 2), (152064, 64)])
@pytest.mark.parametrize("low", [float("-inf"), -1e9, torch.finfo(torch.float32).min])
@pytest.mark.parametrize("finite,neighbours", [(1, False), (20, False), (127, False), (128, True), (150, True)])
def test_rows_with_few_logits(V, rows, low, finite, neighbours):
    """All but a few logits masked, by an infinity, a large number or the type's lowest."""
    g = torch.Generator(device=DEV).manual_seed(V + finite)
    x = torch.full((rows, V), low, device=DEV)
    at = torch.arange(finite, device=DEV)
    at = at + (V - finite) // 3 if neighbours else at * (V // finite)
    x[:, at] = torch.empty(rows, finite, device=DEV).normal_(0, 2.5, generator=g)
    u = torch.rand(rows, device=DEV, generator=g)
    for k in {1, 50, 128, V - 1}:
        for p, t in ((1.0, 0.8), (0.9, 0.8), (1.0, 100.0)):
            top, bins, radix = _tokens(x, k, p, t, u)
            assert top == bins == radix, (k, p, t)


@pytest.mark.gpu
@pytest.mark.parametrize("V,rows", [(32000, 1), (152064, 1), (152064, 64)])
@pytest.mark.parametrize("finite,neighbours", [(20, False), (200, True)])
def test_masked_rows_take_no_longer(V, rows, finite, neighbours):
    """17 to 19 us either way; with the masked logits in the list it was 100 to 1,900, hence a bound of three times."""
    from paged_batch_engine_b200.csrc import ops
    full = lambda x, dt: torch.full((rows,), x, dtype=dt, device=DEV)
    args = full(0.8, torch.float32), full(50, torch.int32), full(0.9, torch.float32), full(0.5, torch.float32)

    def time(x):
        best = float("inf")
        for _ in range(5):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            for _ in range(10):
                ops.sample(x, *args)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        return best
    x = torch.randn(rows, V, device=DEV)
    whole = time(x)
    keep = torch.arange(finite, device=DEV)
    keep = keep + V // 3 if neighbours else keep * (V // finite)
    masked = torch.full_like(x, float("-inf"))
    masked[:, keep] = x[:, keep]
    assert time(masked) <= 3 * whole


def test_draws_of_many_rows():
    seeds = [0, 1, 0xC0FFEE, 2 ** 63 + 5, 2 ** 64 - 1, 2 ** 64 + 7, -3]
    counters = [0, 5, 2 ** 20, 1, 3, 2, 7]
    assert request_sample_uniforms(seeds, counters).tolist() == [request_sample_uniform(s, c) for s, c in zip(seeds, counters)]
    # pairs as zip makes them: what is left over on either side is not looked at
    want = [request_sample_uniform(s, c) for s, c in zip(seeds, counters)]
    assert request_sample_uniforms(seeds, counters + [9, 10]).tolist() == want
    assert request_sample_uniforms(seeds[:3], iter(counters)).tolist() == want[:3]
    assert request_sample_uniforms(seeds, counters[:1]).tolist() == want[:1]
    assert request_sample_uniforms([], counters).tolist() == []


@pytest.mark.gpu
def test_more_counters_than_rows():
    from paged_batch_engine_b200.sampling import Sampler, SamplingParams
    params = [SamplingParams(temperature=0.8, top_k=20, seed=i) for i in range(3)]
    logits, tokens = torch.randn(3, 1000, device=DEV), []
    for counters in ([4, 5, 6], [4, 5, 6, 7, 8]):
        _, host, event = Sampler(torch.device(DEV)).sample_async(logits, params, counters)
        event.synchronize()
        tokens.append(host[:3].tolist())
    assert tokens[0] == tokens[1]
