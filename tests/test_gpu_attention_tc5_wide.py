"""Prompt portions of the masked attention and of the latent attention on tcgen05, against float64: edges of row tiles
(128), key tiles (64), windows, chunks and pages, portions behind a context, several requests in a step, pages that hold
no numbers beyond the requests; and a latent attention's requests alone and beside others."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(need, lens, before, page):
    """A storage with requests that hold ``before`` tokens each, and the step's entries of ``lens`` tokens."""
    from paged_batch_engine_b200.cache.storage import CacheStorage
    from paged_batch_engine_b200.engine.batch import StepEntry
    pages = sum((b + n + page - 1) // page + 1 for n, b in zip(lens, before))
    st = CacheStorage([need], page, pages, len(lens), torch.bfloat16, torch.device(DEV), poison=True)
    entries = []
    for i, (n, b) in enumerate(zip(lens, before)):
        h = st.manager.add_request(f"r{i}")
        if b:
            assert st.manager.reserve(h, b)
            st.manager.commit(h, b)
        assert st.manager.reserve(h, n)
        entries.append(StepEntry(h, [0] * n))
    return st, entries


def _softmax(s, see, sink):
    s = s.masked_fill(~see, -math.inf)
    top = s.max(-1, keepdim=True).values
    if sink is not None:
        top = top.clamp(min=float(sink))
    e = torch.exp(s - top)
    return e / (e.sum(-1, keepdim=True) + (torch.exp(sink - top) if sink is not None else 0.0))


def _sees(pos, n_keys, mask, size):
    d = pos[:, None] - torch.arange(n_keys, device=DEV)[None, :]
    see = d >= 0
    if mask == "window":
        see &= d < size
    if mask == "chunk":
        see &= (pos // size)[:, None] == (torch.arange(n_keys, device=DEV) // size)[None, :]
    return see


@pytest.mark.parametrize("page", [8, 16, 64, 128])
@pytest.mark.parametrize("H,G,lens,before,mask,size,options", [
    (8, 1, [16, 17], [0, 0], None, None, ()),
    (8, 2, [33, 1, 200], [100, 3, 0], None, None, ("sink", "cap", "turn")),
    (4, 4, [129], [0], "window", 40, ("unit", "gate")),
    (2, 1, [65, 300], [63, 129], "chunk", 48, ("unit", "gate", "turn")),
    (3, 1, [40, 2], [700, 1500], "window", 600, ("sink",)),          # key splits
    (8, 1, [70], [1000], None, None, ("gate", "cap")),
])
def test_masked(page, H, G, lens, before, mask, size, options):
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import StepContext
    from paged_batch_engine_b200.parts.base import CacheTensor, PagedNeed
    D = E = 128
    scale = D ** -0.5
    assert ops.masked_tc5_applies(torch.bfloat16, D, E, page, scale)
    st, entries = _step(PagedNeed((CacheTensor("k", G, D), CacheTensor("v", G, E)), window=size), lens, before, page)
    gen = torch.Generator(device=DEV).manual_seed(sum(lens) + H)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    layer, T = st.layer(0), sum(lens)
    ks, vs = [], []
    rows = ops.masked_tile_rows(torch.bfloat16, D, E)
    ctx = StepContext(st.manager, entries, torch.device(DEV), [(0, H // G, rows, size)])
    for i, (n, b) in enumerate(zip(lens, before)):
        k, v = rand(b + n, G, D).bfloat16(), rand(b + n, G, E).bfloat16()
        table = ctx.group(0).block_table[i].tolist()
        for j, pg in enumerate(table):
            if pg >= 0:
                part = slice(j * page, min((j + 1) * page, b + n))
                m = part.stop - part.start
                if m > 0:
                    layer.k[pg, :, :m] = k[part].transpose(0, 1)
                    layer.v[pg, :, :m] = v[part].transpose(0, 1)
        ks.append(k.double()), vs.append(v.double())
    q = rand(T, H * D) * 1.5
    sink = rand(H) if "sink" in options else None
    cap = 5.0 if "cap" in options else None
    ang = rand(T, E // 2) if "turn" in options else None
    turn = torch.stack([ang.cos(), ang.sin()], -1).contiguous() if ang is not None else None
    wide = rand(T, H * E + 8).bfloat16()
    gate = wide[:, 8:] if "gate" in options else None
    meta = ctx.attention_work(0, H // G, rows, size, H, E)
    assert (meta.num_split_rows > 0) == (size == 600)
    got = ops.masked_attention(q, layer.k, layer.v, meta, H, G, scale, mask, size, page, unit_sink="unit" in options,
                               gate=gate, sink=sink, softcap=cap, turn=turn, tcgen05=True).double().view(T, H, E)
    ops.raise_on_kernel_status(DEV)
    at = 0
    for i, (n, b) in enumerate(zip(lens, before)):
        pos = torch.arange(b, b + n, device=DEV)
        see = _sees(pos, b + n, mask, size)
        for h in range(H):
            s = q[at:at + n].double().view(n, H, D)[:, h] @ ks[i][:, h // (H // G)].t() * scale
            s = cap * torch.tanh(s / cap) if cap else s
            w = _softmax(s, see, sink[h].double() if sink is not None else (torch.zeros((), device=DEV, dtype=torch.float64)
                                                                            if "unit" in options else None))
            v = vs[i][:, h // (H // G)]
            o, size_o = w @ v, w @ v.abs()
            if ang is not None:
                c, sn = ang[at:at + n].double().cos(), ang[at:at + n].double().sin()
                u, x = o[:, :64], o[:, 64:]
                o = torch.cat([u * c + x * sn, x * c - u * sn], -1)
                size_o = torch.cat([size_o[:, :64] + size_o[:, 64:]] * 2, -1)
            if gate is not None:
                o = o * torch.sigmoid(gate[at:at + n].double().view(n, H, E)[:, h])
            # the result is rounded to bfloat16 (2^-9 of it); queries and weights hold seventeen bits, which the
            # scores' size (under 16) turns into 2^-13 of the weighted sum over absolute values
            err = (got[at:at + n, h] - o).abs()
            assert (err <= 2 ** -8 * o.abs() + 2 ** -12 * size_o).all(), (i, h, float(err.max()))
        at += n


def _latent_layer_64(part, tensors, x, old, lens, before):
    """The latent attention's layer over requests that bring ``lens`` rows of x behind ``before`` rows of old, in float64."""
    t = {n: v.double() for n, v in tensors.items()}
    H, rank, R, E = part.num_heads, part.kv_rank, part.rot_dim, part.value_dim
    norm = lambda v, gain: v / torch.sqrt((v * v).mean(-1, keepdim=True) + part.eps) * gain

    def turned(v, pos):
        a = pos[:, None].double() * part.inv_freq.double()
        while a.dim() < v.dim():
            a = a.unsqueeze(1)
        u, w = v[..., 0:part.rot_dims:2], v[..., 1:part.rot_dims:2]
        pair = torch.stack([u * a.cos() - w * a.sin(), w * a.cos() + u * a.sin()], -1).flatten(-2) * part.rot_scale
        return torch.cat([pair, v[..., part.rot_dims:]], -1)
    out, at, at_old = [], 0, 0
    for n, b in zip(lens, before):
        rows = torch.cat([old[at_old:at_old + b], x[at:at + n]]).double()
        at, at_old, pos = at + n, at_old + b, torch.arange(b + n, device=DEV)
        down = rows @ t["dkv"].t()
        c, kr = norm(down[:, :rank], t["dkv.norm"]), turned(down[:, rank:], pos)
        q = (norm(rows[b:] @ t["dq"].t(), t["dq.norm"]) @ t["uq"].t()).view(n, H, -1)
        q = torch.cat([q[..., :part.head_dim], turned(q[..., part.head_dim:], pos[b:])], -1)
        k, v = (c @ t["uk"].t()).view(b + n, H, -1), (c @ t["uv"].t()).view(b + n, H, -1)
        see = _sees(pos[b:], b + n, "window" if part.window else None, part.window)
        heads = []
        for h in range(H):
            s = (q[:, h] @ torch.cat([k[:, h], kr], -1).t()) * part.scale
            heads.append(_softmax(s, see, t["sink"][h] if part.sink else None) @ v[:, h])
        o = torch.stack(heads, 1)
        if part.out_gate:
            o = o * torch.sigmoid(rows[b:] @ t["g"].t()).view(n, H, -1)
        out.append(o.reshape(n, H * E) @ t["o"].t())
    return torch.cat(out)


@pytest.mark.parametrize("H,lens,before,window,options,page", [
    (1, [64], [0], None, (), 16),
    (4, [70, 200], [0, 0], None, ("sink", "head"), 16),
    (3, [129, 130], [40, 0], 50, ("each", "yarn"), 8),
    (2, [300], [100], 128, ("sink", "each"), 64),
])
def test_latent(H, lens, before, window, options, page):
    from paged_batch_engine_b200.config import PartSpec
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import StepContext
    from paged_batch_engine_b200.parts import build_part
    rank, w, qr = 512, 256, 192
    rotary = dict(base=1e4, dims=64)
    if "yarn" in options:
        rotary["scaling"] = dict(factor=4.0, original=64, fast=8.0, slow=1.0)
    part = build_part("mixer", PartSpec("latent_attention", dict(
        hidden_size=w, num_heads=H, head_dim=128, rot_dim=64, value_dim=128, kv_rank=rank, q_rank=qr, scale=192 ** -0.5,
        eps=1e-6, rotary=rotary, sink="sink" in options, window=window,
        out_gate="each" if "each" in options else "head" in options)), torch.bfloat16, torch.device(DEV))
    gen = torch.Generator(device=DEV).manual_seed(sum(lens))
    tensors = {}
    for p in part.param_specs(""):
        t = torch.randn(p.shape, device=DEV, generator=gen) * (p.shape[-1] ** -0.5 if len(p.shape) > 1 else 0.2)
        tensors[p.name] = t.bfloat16() if len(p.shape) > 1 else t + (1.0 if "norm" in p.name else 0.0)
    part.load(dict(tensors), "")
    T = sum(lens)
    x = torch.randn(T, w, device=DEV, generator=gen).bfloat16()
    old = torch.randn(sum(before) + 1, w, device=DEV, generator=gen).bfloat16()

    def run(expand):
        part.ROWS_A_KEY = 0 if expand else 1 << 30
        from paged_batch_engine_b200.cache.storage import CacheStorage
        from paged_batch_engine_b200.engine.batch import StepEntry
        pages = sum((b + n + page - 1) // page + 1 for n, b in zip(lens, before))
        st = CacheStorage([part.cache_need()], page, pages, len(lens), torch.bfloat16, torch.device(DEV), poison=True)
        keys = part.paged_work(st.layer(0))
        handles, o = [st.manager.add_request(f"r{i}") for i in range(len(lens))], 0
        for h, b in zip(handles, before):           # what lies before comes through the part itself
            if b:
                assert st.manager.reserve(h, b)
                part.forward(old[o:o + b].contiguous(), StepContext(st.manager, [StepEntry(h, [0] * b)], torch.device(DEV), keys),
                             st.layer(0))
                st.manager.commit(h, b)
            o += b
        entries = []
        for h, n in zip(handles, lens):
            assert st.manager.reserve(h, n)
            entries.append(StepEntry(h, [0] * n))
        ctx = StepContext(st.manager, entries, torch.device(DEV), keys)
        keys = part._expanded_keys(ctx, torch.empty(T, H * 192, dtype=torch.bfloat16, device=DEV), st.layer(0).tensors["latent"])
        assert (keys is not None) == expand
        y = part.forward(x, ctx, st.layer(0)).double()
        ops.raise_on_kernel_status(DEV)
        return y
    got, want = run(True), run(False)
    # both forms round one factor of the scores and one of the outputs to bfloat16, each another one: two roundings of
    # 2^-9 a side, under sums of hundreds of terms of either sign
    assert float((got - want).norm() / want.norm()) < 8e-3
    assert ((got - want).abs() <= 0.06 * want.square().mean().sqrt() + 0.02 * want.abs()).all()
    # against float64: no further off than the form on the latents, but for what chance gives two sets of roundings
    exact = _latent_layer_64(part, tensors, x, old, lens, before)
    off = [float((y - exact).norm() / exact.norm()) for y in (got, want)]
    assert off[0] <= 1.15 * off[1] and off[1] < 1e-2, off


def _latent_part(H, window=None):
    from paged_batch_engine_b200.config import PartSpec
    from paged_batch_engine_b200.parts import build_part
    rank, w, qr = 512, 256, 192
    part = build_part("mixer", PartSpec("latent_attention", dict(
        hidden_size=w, num_heads=H, head_dim=128, rot_dim=64, value_dim=128, kv_rank=rank, q_rank=qr, scale=192 ** -0.5,
        eps=1e-6, rotary=dict(base=1e4, dims=64), sink=True, window=window, out_gate=True)), torch.bfloat16, torch.device(DEV))
    gen = torch.Generator(device=DEV).manual_seed(H)
    tensors = {}
    for p in part.param_specs(""):
        t = torch.randn(p.shape, device=DEV, generator=gen) * (p.shape[-1] ** -0.5 if len(p.shape) > 1 else 0.2)
        tensors[p.name] = t.bfloat16() if len(p.shape) > 1 else t + (1.0 if "norm" in p.name else 0.0)
    part.load(tensors, "")
    return part


def _latent_steps(part, steps, lens, before, page, seed):
    """The rows' results of requests that hold ``before`` tokens, stepped as ``steps`` say: lists of requests that share a
    step.  A request's inputs are the same whichever step it is in."""
    from paged_batch_engine_b200.cache.storage import CacheStorage
    from paged_batch_engine_b200.csrc import ops
    from paged_batch_engine_b200.engine.batch import StepContext, StepEntry
    gen = torch.Generator(device=DEV).manual_seed(seed)
    x = [torch.randn(n, part.hidden_size, device=DEV, generator=gen).bfloat16() for n in lens]
    old = [torch.randn(b, part.hidden_size, device=DEV, generator=gen).bfloat16() for b in before]
    pages = sum((b + n + page - 1) // page + 1 for n, b in zip(lens, before))
    st = CacheStorage([part.cache_need()], page, pages, len(lens), torch.bfloat16, torch.device(DEV), poison=True)
    layer, device = st.layer(0), torch.device(DEV)
    keys = part.paged_work(layer)
    handles, got = [st.manager.add_request(f"r{i}") for i in range(len(lens))], [None] * len(lens)
    for h, rows in zip(handles, old):
        if len(rows):
            assert st.manager.reserve(h, len(rows))
            part.forward(rows, StepContext(st.manager, [StepEntry(h, [0] * len(rows))], device, keys), layer)
            st.manager.commit(h, len(rows))
    for step in steps:
        for i in step:
            assert st.manager.reserve(handles[i], lens[i])
        ctx = StepContext(st.manager, [StepEntry(handles[i], [0] * lens[i]) for i in step], device, keys)
        y = part.forward(torch.cat([x[i] for i in step]), ctx, layer)
        for i, rows in zip(step, y.split([lens[i] for i in step])):
            got[i] = rows.double()
    ops.raise_on_kernel_status(DEV)
    return got


@pytest.mark.parametrize("H,lens,before,window", [
    (4, [1, 300], [700, 0], None),
    (4, [1, 3, 200, 1, 90, 16], [300, 5, 0, 1200, 40, 33], None),        # short ones between portions
    (3, [1, 40, 15, 129], [90, 200, 31, 60], 64),
    (2, [150, 31, 20], [0, 4200, 10], None),                             # 31 rows behind too many keys
])
def test_latent_alone_and_among_others(H, lens, before, window, monkeypatch):
    """What a request computes does not follow from which others share its step: the sums are taken in another order at
    most, and few results round to the neighbouring bfloat16 number.  (The projections, which run on other kernels for
    other numbers of rows, are taken out of it.)"""
    from paged_batch_engine_b200.csrc import ops
    monkeypatch.setattr(ops, "linear", lambda x, w, bias, out_dtype, kind: (x.double() @ w.double().t()).to(out_dtype))
    part = _latent_part(H, window)
    together = _latent_steps(part, [list(range(len(lens)))], lens, before, 16, 7)
    alone = _latent_steps(part, [[i] for i in range(len(lens))], lens, before, 16, 7)
    for i, (a, b) in enumerate(zip(together, alone)):
        assert float((a - b).norm() / b.norm()) < 8e-4, (i, lens[i])           # 4e-3 between the two forms


def test_latent_keys_in_several_goes(monkeypatch):
    """Portions whose expanded keys do not fit at a time are expanded one group after the other."""
    from paged_batch_engine_b200.csrc import ops
    part, lens, before = _latent_part(2), [70, 1, 200, 64, 33], [0, 60, 100, 7, 250]
    want = _latent_steps(part, [list(range(5))], lens, before, 16, 9)
    monkeypatch.setattr(ops, "LATENT_TC5_BYTES", 400 * 2 * 512)          # 70 + 300 keys, then 71 + 283
    goes = []
    inner = ops.latent_attention_expanded
    monkeypatch.setattr(ops, "latent_attention_expanded", lambda *a: goes.append(a[3]) or inner(*a))
    got = _latent_steps(part, [list(range(5))], lens, before, 16, 9)
    assert goes[-2:] == [370, 354]
    assert all(torch.equal(a, b) for a, b in zip(got, want))
