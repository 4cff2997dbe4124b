"""The kernels that make a mixer's inputs for eight rows a thread against those for one row: requests of one row to many,
portions that begin behind their state, rows behind the last whole group of eight, columns behind the last whole block."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS = [[512], [513, 1, 2], [3, 500, 9, 1], [2, 0, 709]]


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _step(lens, pad):
    """The step's arrays and number of rows: `pad` rows behind the requests' belong to none."""
    rows = [i for i, n in enumerate(lens) for _ in range(n)] + [-1] * pad
    return (_i32(rows), _i32([sum(lens[:i]) for i in range(len(lens))]), _i32(lens),
            _i32(list(range(len(lens)))[::-1])), len(rows)


def _moved(state, x, lens, slots):
    """The convolution state behind the step: the last inputs of each request, those of the state before them."""
    want = state.clone()
    for i, n in enumerate(lens):
        first, s = sum(lens[:i]), int(slots[i])
        want[s] = torch.cat([state[s], x[first:first + n].float()])[-state.shape[1]:] if n else state[s]
    return want


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("C,silu", [(1024, True), (8, False), (1544, True)])
def test_short_conv(lens, C, silu):
    from paged_batch_engine_b200.csrc import ops
    arrays, T = _step(lens, 5)
    g = torch.Generator(device=DEV).manual_seed(C + T)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    u = rand(T, C + 16).bfloat16()[:, 8:8 + C]
    weight, bias, start = rand(C, 4), rand(C), rand(len(lens) + 1, 3, C)
    out = []
    for weight_t in (None, weight.t().contiguous()):
        state = start.clone()
        out.append(ops.short_conv(u, weight, bias, state, *arrays, len(lens), silu=silu, weight_t=weight_t))
        assert torch.equal(state, _moved(start, u, lens, arrays[3]))
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("G,H,D,E", [(2, 4, 128, 128), (3, 3, 36, 20), (1, 5, 4, 128)])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_delta_inputs(lens, G, H, D, E, channel, dtype):
    from paged_batch_engine_b200.csrc import ops
    arrays, T = _step(lens, 3)
    g = torch.Generator(device=DEV).manual_seed(T + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    C = 2 * G * D + H * E
    proj, conv_t, start = rand(T, C + 8).to(dtype), rand(4, C), rand(len(lens) + 1, 3, C)
    small = rand(T, H if channel else 2 * H)
    chan = rand(T, H * D) * 3 if channel else None
    dt_bias, a_log = rand(H * D if channel else H), rand(H)
    out = []
    for single in (True, False):                          # steps said to be of single tokens take a row a warp
        state = start.clone()
        out.append(ops.delta_inputs(proj, conv_t, state, small, chan, dt_bias, a_log, *arrays, len(lens), G, H, D, E,
                                    D ** -0.5, 1e-6, update_state=not single, single_tokens=single))
    assert torch.equal(state, _moved(start, proj[:, :C], lens, arrays[3]))
    for a, b in zip(*out):
        assert torch.equal(a, b)
