"""Which matrix-product kernel a projection of a step goes to: decided from the step's rows, the
projection and the size of the matrix alone (no GPU needed to check the rule)."""
import itertools
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from paged_batch_engine_b200.csrc import ops


def _bf16(rows, cols):
    return torch.empty((rows, cols), dtype=torch.bfloat16, device="meta")


def test_stream_mask_by_rows():
    assert ops.stream_mask(1) == ops.STREAM_MASK_FEW and ops.stream_mask(ops.SKINNY_MAX_ROWS) == ops.STREAM_MASK_FEW
    assert ops.stream_mask(ops.SKINNY_MAX_ROWS + 1) == ops.STREAM_MASK
    assert ops.stream_mask(ops.STREAM_MID_ROWS) == ops.STREAM_MASK
    assert ops.stream_mask(ops.STREAM_MID_ROWS + 1) == ops.STREAM_MASK_MANY
    assert ops.stream_mask(ops.STREAM_MAX_ROWS) == ops.STREAM_MASK_MANY
    assert ops.stream_mask(ops.STREAM_MAX_ROWS + 1) == 0


def test_stream_applies_to_large_matrices_of_the_masked_projections_only(monkeypatch):
    monkeypatch.setattr(ops, "STREAM_MASK_FEW", 4)
    monkeypatch.setattr(ops, "STREAM_MASK", 12)
    monkeypatch.setattr(ops, "STREAM_MASK_MANY", 4)
    monkeypatch.setattr(ops, "STREAM_MIN_WEIGHT", 48 << 20)
    big_gate_up, big_down = _bf16(37888, 3584), _bf16(3584, 18944)
    small_gate_up = _bf16(17920, 1536)
    for rows in (1, 8, 16, 33, 64):
        assert ops.stream_applies(_bf16(rows, 3584), big_gate_up, 4)
        assert not ops.stream_applies(_bf16(rows, 1536), small_gate_up, 4)      # below the size gate
        assert not ops.stream_applies(_bf16(rows, 3584), _bf16(4608, 3584), 1)  # QKV is in no default mask
    assert ops.stream_applies(_bf16(12, 18944), big_down, 8)                    # down: 9 to 16 rows only
    assert not ops.stream_applies(_bf16(8, 18944), big_down, 8)
    assert not ops.stream_applies(_bf16(40, 18944), big_down, 8)
    assert not ops.stream_applies(_bf16(65, 3584), big_gate_up, 4)              # more rows than the kernel's range
    assert not ops.stream_applies(torch.empty((8, 3584), dtype=torch.float32, device="meta"), big_gate_up, 4)
    assert not ops.stream_applies(_bf16(8, 3580), _bf16(37888, 3580), 4)        # rows not on 16-byte boundaries
    assert ops.stream_wanted(big_gate_up.numel()) and not ops.stream_wanted(small_gate_up.numel())


def test_skinny_and_tc5_rules(monkeypatch):
    w = _bf16(4608, 3584)
    assert ops.skinny_applies(_bf16(ops.SKINNY_MAX_ROWS, 3584), w)
    assert not ops.skinny_applies(_bf16(ops.SKINNY_MAX_ROWS + 1, 3584), w)
    monkeypatch.setattr(ops, "TC5_MASK", 0)
    assert not ops.tc5_applies(_bf16(2048, 3584), w, 1)
    monkeypatch.setattr(ops, "TC5_MASK", 4)
    assert ops.tc5_applies(_bf16(2048, 3584), w, 4) and not ops.tc5_applies(_bf16(2048, 3584), w, 1)
    assert not ops.tc5_applies(_bf16(ops.TC5_MIN_ROWS - 1, 3584), w, 4)


def test_padded_rows_of_the_experts_are_as_many_as_can_be_filled():
    """Few rows of many experts: a tile for every expert that a row can have chosen, not for every expert there is."""
    def tiles(counts, rows):
        return sum((c + rows - 1) // rows for c in counts)
    for rows in (1, 3, 8):
        for groups in (1, 2, 5):
            for pairs in range(1, 30):
                most = 0
                for cut in itertools.combinations(range(pairs + groups - 1), groups - 1):     # all ways to share them out
                    ends = (-1,) + cut + (pairs + groups - 1,)
                    most = max(most, tiles([b - a - 1 for a, b in zip(ends, ends[1:])], rows))
                assert ops.most_run_tiles(pairs, groups, rows) == most
    assert ops.most_run_tiles(16 * 8, 512, 128) == 128                  # 16 rows, 8 of 512 experts
    assert ops.most_run_tiles(2048 * 4, 32, 128) == 32 + (8192 - 32) // 128


def _masked_part(**options):
    from paged_batch_engine_b200.config import PartSpec
    from paged_batch_engine_b200.parts import build_part
    return build_part("mixer", PartSpec("masked_attention", dict(
        hidden_size=256, num_heads=16, num_kv_heads=2, key_dim=128, value_dim=128, scale=128 ** -0.5, eps=1e-6, **options)),
        torch.bfloat16, torch.device("cpu"))


def _lengths(rows, before):
    return SimpleNamespace(q_len_host=np.array(rows), seq_len_host=np.array(rows) + np.array(before))


@pytest.mark.parametrize("options,rows,before,long", [
    (dict(mask="chunk", mask_size=512, out_gate=True), [150], [0], False),
    (dict(mask="chunk", mask_size=512, out_gate=True), [192], [0], True),
    (dict(mask="chunk", mask_size=512, out_gate=True), [16], [300], False),        # one block a head group, 316 keys
    (dict(mask="chunk", mask_size=512, out_gate=True), [17], [2000], True),        # 481 of the chunk
    (dict(mask="chunk", mask_size=512, out_gate=True), [128], [2048], False),      # a chunk of its own
    (dict(mask="chunk", mask_size=512, out_gate=True), [100, 100, 1, 100], [0, 0, 4000, 0], False),
    (dict(mask="window", mask_size=1024), [16], [300], True),
    (dict(mask="window", mask_size=128), [700], [0], False),
    (dict(), [1, 1, 2], [5000, 4000, 3000], False),
    (dict(), [1, 64], [5000, 2048], True),
])
def test_masked_prompts_that_take_the_form_for_long_rows(options, rows, before, long):
    part = _masked_part(**options)
    assert part.tcgen05 and part._long_rows(_lengths(rows, before)) is long


def test_a_steps_lengths_are_looked_at_once_for_all_layers():
    """Not once a layer: a step of few rows waits for the host."""
    class Lengths:
        looks = 0

        def tolist(self):
            Lengths.looks += 1
            return [300]
    ctx = SimpleNamespace(q_len_host=Lengths(), seq_len_host=Lengths())
    layers = [_masked_part() for _ in range(4)]
    assert all(layer._long_rows(ctx) for layer in layers) and Lengths.looks == 2
    assert not _masked_part(mask="window", mask_size=64)._long_rows(ctx) and Lengths.looks == 4     # another mask


@pytest.mark.parametrize("state,head,dtype,matrix", [(128, 64, torch.bfloat16, True), (64, 64, torch.bfloat16, True),
                                                     (64, 128, torch.bfloat16, True), (128, 128, torch.bfloat16, False),
                                                     (128, 64, torch.float32, False), (32, 64, torch.bfloat16, False)])
def test_state_space_form_is_known_from_the_widths(state, head, dtype, matrix):
    """At construction: a step's rows lie on 16-byte boundaries for these widths, and looking was 10 us of a layer's 120."""
    from paged_batch_engine_b200.config import PartSpec
    from paged_batch_engine_b200.parts import build_part
    part = build_part("mixer", PartSpec("selective_state_space", dict(
        hidden_size=256, num_heads=4, head_dim=head, state_dim=state, groups=1, conv_taps=4, norm_groups=4, eps=1e-6)),
        dtype, torch.device("cpu"))
    assert part.matrix is matrix
    assert (("linear_attention_mma", None) in part.kernel_libraries(dtype)) is matrix
    assert not matrix or all(n % 8 == 0 for n in (part.inner, part.groups * state, part.conv_channels))


def _latent_part(heads):
    from paged_batch_engine_b200.config import PartSpec
    from paged_batch_engine_b200.parts import build_part
    return build_part("mixer", PartSpec("latent_attention", dict(
        hidden_size=256, num_heads=heads, head_dim=128, rot_dim=64, value_dim=128, kv_rank=512, q_rank=192, scale=192 ** -0.5,
        eps=1e-6, rotary=dict(base=1e4, dims=64))), torch.bfloat16, torch.device("cpu"))


def test_portions_that_expand_their_latents(monkeypatch):
    """Decided for each request by its own rows and keys, on either side of every threshold."""
    part = _latent_part(16)
    assert [part.expanded(n, k) for n, k in ((7, 500), (8, 500), (8, 4096), (8, 4097), (31, 4097), (32, 4097))] \
        == [0, 500, 4096, 0, 0, 4097]
    assert part.expanded(512, 65536) == 65536 and part.expanded(512, 65537) == 0       # 512 MB of keys and values
    assert _latent_part(128).expanded(512, 8192) == 8192 and _latent_part(128).expanded(512, 8193) == 0
    rows, before = np.array([1, 300, 7, 16, 40, 1]), np.array([9000, 0, 30, 4081, 100, 20])
    step = SimpleNamespace(q_len_host=rows, context_before_host=before)
    assert part.ROWS_A_KEY == 8
    operands = torch.empty(1, 16 * 192, dtype=torch.bfloat16), torch.empty(1, 1, 16, 576, dtype=torch.bfloat16)
    assert part._expanded_keys(step, *operands) is None                                 # no weights yet
    part.w_kv = torch.empty(2 * 16 * 128, 512, dtype=torch.bfloat16)
    assert part._expanded_keys(step, *operands) == [0, 300, 0, 0, 140, 0]
    alone = [SimpleNamespace(q_len_host=rows[i:i + 1], context_before_host=before[i:i + 1]) for i in range(6)]
    assert [(part._expanded_keys(one, *operands) or [0])[0] for one in alone] == [0, 300, 0, 0, 140, 0]
    part.window = 50
    assert part._expanded_keys(step, *operands) == [0, 300, 0, 65, 89, 0]               # the keys that the rows see
    part.window = None
    step.device = torch.device("cpu")
    step2 = SimpleNamespace(q_len_host=np.array([70, 1, 200, 64, 33]), device=torch.device("cpu"))
    monkeypatch.setattr(ops, "LATENT_TC5_BYTES", 400 * 16 * 512)
    goes = part._goes(step2, [70, 0, 300, 71, 283])
    assert [(g[0].tolist(),) + g[1:] for g in goes] == [([0, 2], 370, 300, 1 + 2), ([3, 4], 354, 283, 1 + 1)]
    assert part._goes(step2, [70, 0, 300, 71, 283]) is goes                             # once a step
    assert part._goes(SimpleNamespace(q_len_host=np.array([300, 20]), device=torch.device("cpu")), [310, 50]) \
        == [(None, 360, 310, 3 + 1)]


def test_a_work_list_of_some_requests():
    """The same tiles and key splits that these requests have in a list of all."""
    from paged_batch_engine_b200.engine.batch import attention_work_arrays
    q_len, seq_len = np.array([1, 300, 3, 1, 700]), np.array([2000, 300, 900, 5, 900])
    q_start = np.cumsum(q_len) - q_len
    some = np.array([True, False, True, True, False])
    every = attention_work_arrays(q_len, seq_len, q_start, 16, 16, None)
    part = attention_work_arrays(np.where(some, q_len, 0), seq_len, q_start, 16, 16, None)
    assert sorted(map(tuple, part[0])) == sorted(tuple(w) for w in every[0] if some[w[0]])
    split = [t for t in every[2].tolist() if some[np.searchsorted(q_start, t, side="right") - 1]]
    assert part[2].tolist() == split and (part[1][split] >= 0).all() and part[4] == every[0][np.isin(every[0][:, 0], [0, 2, 3]), 3].max()
    none = attention_work_arrays(np.zeros(5, dtype=np.int64), seq_len, q_start, 16, 16, None)
    assert len(none[0]) == 0 and len(none[2]) == 0
