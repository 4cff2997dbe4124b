"""Float32 prompt attention on tcgen05 (three bfloat16 terms a factor) against 64 bits and against the multiply-adds: edges of its row
and key tiles, windows, key splits of few-row requests beside long portions, page sizes, and elements whose terms do not hold them."""
import math

import numpy as np
import pytest
import torch

from tests.test_gpu_kernels import AttnCase, ops

pytestmark = pytest.mark.gpu

SHAPES = [
    # H, KV, hd, P, window, [(context, new rows)...]
    (1, 1, 128, 16, None, [(0, 65), (0, 64)]),
    (4, 4, 64, 16, None, [(0, 128), (3, 129), (64, 66)]),
    (6, 2, 128, 24, None, [(0, 21), (0, 22), (0, 43), (127, 43)]),
    (14, 2, 64, 7, 77, [(0, 200), (70, 33), (400, 9)]),
    (28, 4, 128, 16, None, [(300, 1), (0, 70), (1100, 3), (513, 1)]),
    (7, 1, 128, 1, 130, [(600, 1), (0, 300), (259, 2)]),
    (12, 2, 128, 16, None, [(0, 17), (0, 311), (0, 700)]),
    (2, 2, 64, 32, None, [(2000, 33), (1, 190), (0, 1)]),
    (2, 1, 128, 16, 600, [(1700, 5), (100, 100), (0, 1), (900, 2), (513, 1)]),
]


def _both(shape, monkeypatch, change=lambda case: None):
    """(the case, its result by the multiply-adds, on the tensor cores)"""
    H, KV, hd, P, window, reqs = shape
    out = []
    for wide in (False, True):
        case = AttnCase(H, KV, hd, P, window, reqs, torch.float32, seed=3, kind="simple")
        change(case)
        case.write_cache()
        with monkeypatch.context() as m:
            if not wide:
                m.setattr(ops(), "attention_f32_tiles", lambda *a: 0)
            out.append(case.run())
    return case, out[0], out[1]


def _exact(case):
    outs = []
    for q, k, v, c, n, h in case.seqs:
        G = case.H // case.KV
        q, k, v = q[c:].double(), k.double().repeat_interleave(G, 1), v.double().repeat_interleave(G, 1)
        s = torch.einsum("qhd,khd->hqk", q, k) * case.hd ** -0.5
        d = torch.arange(n)[:, None] + c - torch.arange(c + n)[None]
        see = (d >= 0) & (d < (case.window or math.inf))
        outs.append(torch.einsum("hqk,khd->qhd", s.masked_fill(~see, -math.inf).softmax(-1), v))
    return torch.cat(outs)


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"H{s[0]}kv{s[1]}hd{s[2]}P{s[3]}w{s[4]}")
def test_against_64_bits(shape, monkeypatch):
    case, fma, got = _both(shape, monkeypatch)
    assert case.meta.wide_tiles > 0
    want = _exact(case)
    # the bound of the multiply-adds' own test, and no further off than they are
    assert (got.double() - want).abs().max() <= 2e-5 * max(1.0, want.abs().max().item())
    assert (got.double() - want).norm() <= (fma.double() - want).norm()


@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e30, 1e-35])
def test_elements_that_three_terms_do_not_hold(where, value, monkeypatch):
    """The row tiles that meet one are made by the multiply-adds, to the last bit; the others are not."""
    def change(case):
        q, k, v, *_ = case.seqs[0]
        dict(q=q, k=k, v=v)[where][90, 0, 5] = value
    case, fma, got = _both((12, 2, 128, 16, None, [(0, 150), (0, 64), (300, 2)]), monkeypatch, change)
    rows = slice(86, 106 if where == "q" else 150)           # of the tiles of 128 packed rows (six heads) that meet it
    assert torch.equal(got[rows, :6].nan_to_num(3.25), fma[rows, :6].nan_to_num(3.25))
    assert torch.equal(got.isnan(), fma.isnan()) and torch.isfinite(got[150:]).all()
    want = _exact(case)[150:]
    assert (got[150:].double() - want).norm() <= (fma[150:].double() - want).norm()


def test_blocks_are_those_of_the_work_list():
    """The blocks that the host counts are the row tiles and splits that the step's work list has."""
    from paged_batch_engine_b200.engine.batch import attention_work_arrays
    o = ops()
    rng = np.random.default_rng(5)
    for _ in range(200):
        R, G = int(rng.integers(1, 9)), int(rng.integers(1, 9))
        window, split = [None, 1, 77, 600][rng.integers(4)], [256, 512][rng.integers(2)]
        q_len = rng.integers(1, 90, R)
        seq_len = q_len + rng.integers(0, 3000, R)
        work, *_ = attention_work_arrays(q_len, seq_len, np.cumsum(q_len) - q_len, G, o.SIMPLE_TILE_ROWS, window, split)
        wide = q_len * G > o.F32_SMALL_ROWS
        want = sum(-(-int(n) * G // o.F32_TILE_ROWS) if w else int(work[work[:, 0] == r][0, 3])
                   for r, (n, w) in enumerate(zip(q_len, wide)))
        seen = np.minimum(seq_len, q_len + window - 1) if window else seq_len
        takes = wide.any() and seen[wide].max() > o.F32_FEW_KEYS * (1 if q_len.sum() > 64 else 2)
        assert o.attention_f32_tiles(q_len, seq_len, G, window, split) == (want if takes else 0)
