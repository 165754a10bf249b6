"""The tcgen05 attention kernels for prompt portions (csrc/attention_tc.cu) alone, against attention written out in float64:
portions around the kernels' tile sizes (64 keys; 64, 128 and 256 tokens), cached context that starts inside a tile, heads that do
not fill a CTA, every mask, bias and output form they serve.  Pool and buffer rows that no query may see hold NaN.

Bound: the weights enter the second product as bfloat16 (half a unit: 2^-9 of sum p |v|), the result is rounded once more
(2^-9 of |out|), and both are at most max |v|; products and sums are float.  2^-8 max |v| holds the two, 1.1 times that is asked."""
import ctypes

import pytest
import torch

BF = torch.bfloat16
CTX = [0, 70, 0, 63, 1, 190, 0]
NEW = [300, 150, 17, 64, 65, 257, 128]


def _close(out, want, vmax):
    assert torch.isfinite(out.float()).all()
    err = (out.double().cpu() - want).abs().max().item()
    assert err < 1.1 * 2.0 ** -8 * vmax, err


def _no_wait_ran_out(lib):
    n = ctypes.c_int(-1)
    assert lib.pa_attention_tc_errors(ctypes.byref(n)) == 0 and n.value == 0


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 1, 128, 128), (6, 2, 64, 128), (4, 2, 128, 64), (3, 3, 64, 64), (10, 2, 128, 128)])
@pytest.mark.parametrize("mask,size,keep,form", [("causal", 0, 0, "plain"), ("causal", 0, 0, "sink"), ("window", 37, 0, "bucket"),
                                                 ("window", 100, 9, "turned"), ("chunk", 50, 0, "slope")])
def test_paged_portions(heads, kv_heads, dim, vdim, mask, size, keep, form):
    _paged_portions(heads, kv_heads, dim, vdim, mask, size, keep, form)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,bias_len", [(4, 1, 114), (4, 1, 600), (4, 1, 2560), (2, 1, 227), (2, 1, 600), (2, 1, 5120), (1, 1, 454),
                                                     (1, 1, 10240)])
def test_long_bias_tables(heads, kv_heads, bias_len):
    """Tables beside the largest stages: longer than what two buffers of query rows leave, up to the 40 KB that are taken."""
    _paged_portions(heads, kv_heads, 128, 128, "window", 200, 0, "bucket", bias_len)


# enough portions that a CTA has several work items in turn (at least 444 with two query tiles, 888 with one), of one key tile and of
# many, whole and ragged
MANY_NEW = [[64, 17, 200, 128, 65, 256, 33, 64, 192, 16][i % 10] + (i % 7 == 3) for i in range(90)]
MANY_CTX = [[0, 70, 0, 300, 1, 0, 512, 0, 63, 0, 190][i % 11] for i in range(90)]


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(10, 2, 128, 128), (10, 2, 64, 128), (8, 2, 128, 64), (6, 3, 64, 64), (8, 8, 128, 128)])
@pytest.mark.parametrize("mask,size,keep,form", [("causal", 0, 0, "plain"), ("causal", 0, 0, "sink"), ("window", 70, 9, "gate"), ("chunk", 50, 0, "slope"),
                                                 ("window", 37, 0, "bucket")])
def test_several_work_items_per_cta(heads, kv_heads, dim, vdim, mask, size, keep, form):
    """The walk of a CTA over its items: ring, accumulators and query buffers carried over, queries of whole items (TMA) after ragged ones
    (their threads) and the other way round, a query tile without rows (ten heads over two: the fifth alone) between others."""
    _paged_portions(heads, kv_heads, dim, vdim, mask, size, keep, form, ctx=MANY_CTX, new=MANY_NEW, per_cta=3 if kv_heads == 2 and dim == 128 else 2)


@pytest.mark.gpu
@pytest.mark.parametrize("form,mask,size", [("plain", "causal", 0), ("slope", "window", 90)])
def test_work_items_without_tokens(form, mask, size):
    """Items of no tokens among the others, also first and next to each other: nothing to do, and the walk goes on."""
    def with_empty(tiles):
        out = []
        for i, t in enumerate(tiles):
            if i % 5 == 0:
                out += [[t[0], 0, t[2], t[3]]] * (1 + i % 3)
            out.append(t)
        return out
    _paged_portions(10, 2, 128, 128, mask, size, 0, form, ctx=MANY_CTX, new=MANY_NEW, change=with_empty)


def _paged_portions(heads, kv_heads, dim, vdim, mask, size, keep, form, bias_len=23, ctx=CTX, new=NEW, change=None, per_cta=0):
    """change: the list of work items (first row, tokens, slot, first position) -> the one that is launched.  per_cta: how many of them
    some CTA has at least, with two query tiles (one CTA an SM)."""
    from llm_decoder import _cabi
    from llm_decoder.hybrid import MASK_KIND
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    g = torch.Generator().manual_seed(heads * 7 + dim + size)
    per, scale, n = heads // kv_heads, dim ** -0.5 * 2.0, len(new)
    states = SequenceStateCache(n, 4096 if n == len(NEW) else sum(ctx) + sum(new) + 32 * n, 32, dev)
    kv = states.add_kv_layer(kv_heads, dim, vdim, "bf16")
    kv.key_buffer_.fill_(float("nan"))
    kv.value_buffer_.fill_(float("nan"))
    slots = [states.alloc() for _ in range(n)]
    turns = [2, 0, 3, 1, 6, 5, 4] + list(range(7, n))
    for r in range(max(ctx) // 16 + 1):                     # growth in turns, so that the sequences' pages interleave
        for i in turns:
            if ctx[i] > 16 * r:
                states.extend(slots[i], min(16, ctx[i] - 16 * r))
    K = [torch.randn(c + m, kv_heads * dim, generator=g).to(BF) for c, m in zip(ctx, new)]
    V = [torch.randn(c + m, kv_heads * vdim, generator=g).to(BF) for c, m in zip(ctx, new)]
    Q = [torch.randn(m, heads * dim, generator=g).to(BF) for m in new]
    for i in range(n):
        if ctx[i]:
            kv.append_rows(torch.cat([K[i][:ctx[i]], V[i][:ctx[i]]], 1).to(dev), 0, kv_heads * dim,
                           torch.full((ctx[i],), slots[i], dtype=torch.int32, device=dev), torch.arange(ctx[i], dtype=torch.int32, device=dev))
    batch = states.make_batch([(slots[i], [0] * new[i]) for i in range(n)])
    proj = torch.cat([torch.cat([Q[i], K[i][ctx[i]:], V[i][ctx[i]:]], 1) for i in range(n)], 0).to(dev)
    kv.append_rows(proj, heads * dim, heads * dim + kv_heads * dim, batch.row_slot, batch.row_pos)

    temp = torch.rand(heads, generator=g) * 2 - 0.5 if form == "sink" else None     # one negative factor among them
    sink = torch.randn(heads, generator=g) if form in ("sink", "turned") else None
    cap = 6.0 if form == "bucket" else 0.0
    bias, bias_kind = None, 0
    if form == "bucket":
        bias, bias_kind = torch.randn(bias_len, heads, generator=g), 2
    elif form == "slope":
        bias, bias_kind = torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)]), 1
    rows = batch.rows
    ang = torch.rand(rows, vdim // 2, generator=g) * 6.0
    turn = torch.stack([torch.cos(ang), torch.sin(ang)], -1) if form == "turned" else None
    want, r0 = torch.zeros(rows, heads, vdim, dtype=torch.float64), 0
    for i in range(n):
        pos, j = torch.arange(ctx[i], ctx[i] + new[i])[:, None], torch.arange(ctx[i] + new[i])[None]
        dist = pos - j
        vis = dist >= 0
        if mask == "window":
            vis &= (dist < size) | (j < keep)
        elif mask == "chunk":
            vis &= (pos // size) == (j // size)
        for h in range(heads):
            k, v = K[i].double()[:, h // per * dim:(h // per + 1) * dim], V[i].double()[:, h // per * vdim:(h // per + 1) * vdim]
            s = Q[i].double()[:, h * dim:(h + 1) * dim] @ k.T * scale * (float(temp[h]) if temp is not None else 1.0)
            s = cap * torch.tanh(s / cap) if cap else s
            if bias_kind == 2:
                s = s + bias.double()[dist.clamp(0, bias_len - 1), h]
            elif bias_kind == 1:
                s = s - float(bias[h]) * dist
            s = s.masked_fill(~vis, -float("inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(new[i], 1)], 1)
            want[r0:r0 + new[i], h] = torch.softmax(s, -1)[:, :k.shape[0]] @ v
        r0 += new[i]
    gate = torch.randn(rows, heads * vdim + 8, generator=g).to(BF) if form == "gate" else None
    if gate is not None:
        want *= torch.sigmoid(gate[:, 8:].double()).reshape(rows, heads, vdim)
    if turn is not None:
        u, w = want[..., 0::2].clone(), want[..., 1::2].clone()
        c, s = turn.double()[:, None, :, 0], turn.double()[:, None, :, 1]
        want[..., 0::2], want[..., 1::2] = u * c + w * s, w * c - u * s
    keepalive = [t.to(dev).contiguous() if t is not None else None for t in (bias, temp, sink, turn, gate)]
    pt = kv.page_table_
    table = pt.device_data()
    for q_tiles, kind in ((2, 4), (1, 5)):
        tokens = lib.pa_masked_attention_tc_tile_tokens(heads, kv_heads, dim, vdim, 2, q_tiles)
        tiles, ntiles, _longest = batch.query_tiles(1, tokens, 16)[2]
        if change:
            tiles = torch.tensor(change(tiles.tolist()), dtype=torch.int32, device=dev)
            ntiles = len(tiles)
        if q_tiles == 2 and form != "bucket":       # tables of biases: a CTA each
            assert ntiles * lib.pa_masked_attention_tc_units(heads, kv_heads, 2) > (per_cta - 1) * _cabi.device_info()[0]
        out = torch.full((rows, heads * vdim), float("nan"), dtype=BF, device=dev)
        rc = lib.pa_masked_attention_gated(
            proj.data_ptr(), proj.stride(0), 0, kv.key_buffer_.data_ptr(), kv.value_buffer_.data_ptr(), table.data_ptr(), pt.num_beams_,
            pt.num_heads_, pt.num_tiles_, kv.total_pages_, kv.tile_size_, tiles.data_ptr(), ntiles, heads, dim, vdim, scale, cap,
            MASK_KIND[mask], size, keep, bias_kind, _cabi.ptr(keepalive[0]), bias_len if bias_kind == 2 else 0, _cabi.ptr(keepalive[1]),
            _cabi.ptr(keepalive[2]), _cabi.ptr(keepalive[3]), None, 0, None, _cabi.ptr(keepalive[4]),
            heads * vdim + 8 if gate is not None else 0, 8 if gate is not None else 0, out.data_ptr(), 2, kind, _cabi.stream())
        assert rc == 0, rc
        _close(out, want.reshape(rows, -1), max(v.abs().max().item() for v in V) * (1.42 if turn is not None else 1.0))
    _no_wait_ran_out(lib)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,dim,rot_dim,vdim,kv_rank", [(3, 128, 64, 128, 64), (2, 64, 32, 64, 96), (2, 64, 16, 128, 64), (2, 128, 48, 64, 64)])
@pytest.mark.parametrize("sink", [False, True])
def test_expanded_latent_portions(heads, dim, rot_dim, vdim, kv_rank, sink):
    """Rows of several sequences gathered from a paged latent pool, then attention on keys and values given per head."""
    _expanded_latent_portions(heads, dim, rot_dim, vdim, kv_rank, sink)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,dim,rot_dim,vdim,kv_rank", [(7, 128, 64, 128, 64), (7, 64, 32, 64, 96)])
def test_latent_portions_with_several_work_items_per_cta(heads, dim, rot_dim, vdim, kv_rank):
    _expanded_latent_portions(heads, dim, rot_dim, vdim, kv_rank, True, MANY_CTX, MANY_NEW)


def _expanded_latent_portions(heads, dim, rot_dim, vdim, kv_rank, sink, ctx=CTX, new=NEW):
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    g = torch.Generator().manual_seed(heads + dim + rot_dim)
    kd, n = kv_rank + rot_dim, len(new)
    states = SequenceStateCache(n, 4096 if n == len(NEW) else sum(ctx) + sum(new) + 16 * n, 16, dev)
    kv = states.add_kv_layer(1, kd, 0, "bf16")
    slots = [states.alloc() for _ in range(n)]
    for i in [3, 0, 5, 1, 2, 6, 4] + list(range(7, n)):
        if ctx[i]:
            states.extend(slots[i], ctx[i])
    batch = states.make_batch([(s, [0] * m) for s, m in zip(slots, new)])
    kv.key_buffer_.copy_(torch.randn(kv.key_buffer_.shape, generator=g))
    pt = kv.page_table_
    groups = batch.whole_sequences(16, 128)
    assert len(groups) == 1
    items, nitems, longest, rows, _tiles, _ntiles = groups[0]
    lat = torch.full((rows, kd), float("nan"), dtype=BF, device=dev)
    assert lib.pa_latent_gather(kv.key_buffer_.data_ptr(), pt.device_data().data_ptr(), pt.num_beams_, pt.num_tiles_, kv.total_pages_, 16,
                                kd * 2, items.data_ptr(), nitems, longest, lat.data_ptr(), _cabi.stream()) == 0
    tab, pool = pt.device_data().cpu().reshape(pt.num_beams_, pt.num_tiles_), kv.key_buffer_.cpu()
    first = {int(s): int(r) for s, _t, r in items.cpu()}
    for s, c, m in zip(slots, ctx, new):
        got = lat[first[s]:first[s] + c + m].cpu()
        assert torch.equal(got, torch.stack([pool[int(tab[s, j // 16]), j % 16] for j in range(c + m)]))
    Kn, V = torch.randn(rows, heads * dim, generator=g).to(BF), torch.randn(rows, heads * vdim, generator=g).to(BF)
    Q = torch.randn(batch.rows, heads * (dim + rot_dim), generator=g).to(BF)
    sk = torch.randn(heads, generator=g) if sink else None
    want, r0, scale = torch.zeros(batch.rows, heads, vdim, dtype=torch.float64), 0, 1.5 * (dim + rot_dim) ** -0.5
    for s, c, m in zip(slots, ctx, new):
        rr = slice(first[s], first[s] + c + m)
        hidden = torch.arange(c + m)[None] > torch.arange(c, c + m)[:, None]
        for h in range(heads):
            k = torch.cat([Kn[rr, h * dim:(h + 1) * dim], lat[rr, kv_rank:].cpu()], 1).double()
            sc = (Q[r0:r0 + m, h * (dim + rot_dim):(h + 1) * (dim + rot_dim)].double() @ k.T * scale).masked_fill(hidden, -float("inf"))
            if sink:
                sc = torch.cat([sc, sk[h].double().expand(m, 1)], 1)
            want[r0:r0 + m, h] = torch.softmax(sc, -1)[:, :c + m] @ V[rr, h * vdim:(h + 1) * vdim].double()
        r0 += m
    Kd, Vd, Qd, skd = Kn.to(dev), V.to(dev), Q.to(dev), sk.to(dev) if sink else None
    for q_tiles in (2, 1):
        tokens = lib.pa_masked_attention_tc_tile_tokens(1, 1, dim, vdim, 2, q_tiles)
        tiles, ntiles = batch.whole_sequences(16, tokens)[0][4:]
        assert n == len(NEW) or ntiles * heads > 3 * _cabi.device_info()[0]
        out = torch.full((batch.rows, heads * vdim), float("nan"), dtype=BF, device=dev)
        assert lib.pa_latent_attention_expanded(Qd.data_ptr(), Qd.stride(0), 0, Kd.data_ptr(), Kd.stride(0), lat.data_ptr(), kd, kv_rank,
                                                Vd.data_ptr(), Vd.stride(0), rows, tiles.data_ptr(), ntiles, heads, dim, rot_dim, vdim, scale,
                                                _cabi.ptr(skd), out.data_ptr(), q_tiles, _cabi.stream()) == 0
        _close(out, want.reshape(batch.rows, -1), V.abs().max().item())
    _no_wait_ran_out(lib)
