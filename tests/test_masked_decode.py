"""pa_masked_decode (csrc/masked_decode.cu) alone, against attention written out in float64: tokens whose keys end inside, on and
just past a unit of 16 keys, one worker for everything, many times more workers than pairs, more query heads than the 16 rows of a
product, every mask, bias and output form.  Pool rows that no query may see hold NaN.

Bound: the weights enter the second product as bfloat16 (2^-9 of sum p |v|) and the result is rounded once more (2^-9): 2^-8 max |v|;
1.1 times that is asked, and the square root of two more where neighbouring columns are turned into each other."""
import pytest
import torch

BF = torch.bfloat16
POS = [0, 15, 16, 17, 300, 1, 257, 95, 511]


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 1, 128, 128), (6, 2, 64, 128), (4, 4, 128, 64), (40, 2, 64, 64), (16, 1, 128, 128)])
@pytest.mark.parametrize("mask,size,keep,form", [("causal", 0, 0, "plain"), ("causal", 0, 0, "sink"), ("window", 37, 0, "bucket"),
                                                 ("window", 100, 21, "turned"), ("chunk", 50, 0, "slope")])
def test_shares_of_decoded_tokens(heads, kv_heads, dim, vdim, mask, size, keep, form):
    from llm_decoder import _cabi
    from llm_decoder.hybrid import MASK_KIND
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    g = torch.Generator().manual_seed(heads * 7 + dim + size)
    per, scale, n = heads // kv_heads, dim ** -0.5 * 2.0, len(POS)
    states = SequenceStateCache(n, 4096, 16, dev)
    kv = states.add_kv_layer(kv_heads, dim, vdim, "bf16")
    kv.key_buffer_.fill_(float("nan"))
    kv.value_buffer_.fill_(float("nan"))
    slots = [states.alloc() for _ in range(n)]
    for r in range(32):                                     # growth in turns, so that the sequences' pages interleave
        for i in (2, 0, 3, 1, 6, 5, 4, 8, 7):
            if POS[i] > 16 * r:
                states.extend(slots[i], min(16, POS[i] - 16 * r))
    K = [torch.randn(c + 1, kv_heads * dim, generator=g).to(BF) for c in POS]
    V = [torch.randn(c + 1, kv_heads * vdim, generator=g).to(BF) for c in POS]
    Q = torch.randn(n, heads * dim, generator=g).to(BF)
    for i, c in enumerate(POS):
        if c:
            kv.append_rows(torch.cat([K[i][:c], V[i][:c]], 1).to(dev), 0, kv_heads * dim,
                           torch.full((c,), slots[i], dtype=torch.int32, device=dev), torch.arange(c, dtype=torch.int32, device=dev))
    batch = states.make_batch([(s, [0]) for s in slots])
    proj = torch.cat([Q, torch.stack([torch.cat([K[i][-1], V[i][-1]]) for i in range(n)])], 1).to(dev)
    kv.append_rows(proj, heads * dim, heads * dim + kv_heads * dim, batch.row_slot, batch.row_pos)
    temp = torch.rand(heads, generator=g) * 2 - 0.5 if form == "sink" else None
    sink = torch.randn(heads, generator=g) if form in ("sink", "turned") else None
    cap = 6.0 if form == "bucket" else 0.0
    bias, bias_kind = None, 0
    if form == "bucket":
        bias, bias_kind = torch.randn(23, heads, generator=g), 2
    elif form == "slope":
        bias, bias_kind = torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)]), 1
    ang = torch.rand(n, vdim // 2, generator=g) * 6.0
    turn = torch.stack([torch.cos(ang), torch.sin(ang)], -1) if form == "turned" else None
    gate = torch.randn(n, heads * vdim + 8, generator=g).to(BF) if form == "slope" else None
    want = torch.zeros(n, heads, vdim, dtype=torch.float64)
    for i, c in enumerate(POS):
        j = torch.arange(c + 1)
        dist = c - j
        vis = torch.ones(c + 1, dtype=torch.bool)
        if mask == "window":
            vis = (dist < size) | (j < keep)
        elif mask == "chunk":
            vis = (c // size) == (j // size)
        for h in range(heads):
            k, v = K[i].double()[:, h // per * dim:(h // per + 1) * dim], V[i].double()[:, h // per * vdim:(h // per + 1) * vdim]
            s = k @ Q[i].double()[h * dim:(h + 1) * dim] * scale * (float(temp[h]) if temp is not None else 1.0)
            s = cap * torch.tanh(s / cap) if cap else s
            if bias_kind == 2:
                s = s + bias.double()[dist.clamp(0, 22), h]
            elif bias_kind == 1:
                s = s - float(bias[h]) * dist
            s = s.masked_fill(~vis, -float("inf"))
            if sink is not None:
                s = torch.cat([s, sink[h:h + 1].double()])
            want[i, h] = torch.softmax(s, 0)[:c + 1] @ v
    if turn is not None:
        u, w = want[..., 0::2].clone(), want[..., 1::2].clone()
        c, s = turn.double()[:, None, :, 0], turn.double()[:, None, :, 1]
        want[..., 0::2], want[..., 1::2] = u * c + w * s, w * c - u * s
    if gate is not None:
        want = want * torch.sigmoid(gate[:, 8:].double()).reshape(n, heads, vdim)
    biasd, tempd, sinkd, turnd, gated = (t.to(dev).contiguous() if t is not None else None for t in (bias, temp, sink, turn, gate))
    pt = kv.page_table_
    tiles, ntiles, longest = batch.query_tiles(1)[1]
    assert ntiles == n
    for workers in (1, 5, lib.pa_masked_decode_workers(n, heads, kv_heads, longest), 1000):
        ws = torch.empty(lib.pa_masked_decode_workspace_bytes(n, heads, kv_heads, vdim, workers), dtype=torch.uint8, device=dev)
        out = torch.full((n, heads * vdim), float("nan"), dtype=BF, device=dev)
        rc = lib.pa_masked_decode(
            proj.data_ptr(), proj.stride(0), 0, kv.key_buffer_.data_ptr(), kv.value_buffer_.data_ptr(), pt.device_data().data_ptr(),
            pt.num_beams_, pt.num_heads_, pt.num_tiles_, kv.total_pages_, kv.tile_size_, tiles.data_ptr(), n, heads, dim, vdim, scale, cap,
            MASK_KIND[mask], size, keep, bias_kind, _cabi.ptr(biasd), 23 if bias_kind == 2 else 0, _cabi.ptr(tempd), _cabi.ptr(sinkd),
            _cabi.ptr(turnd), None, _cabi.ptr(gated), gated.stride(0) if gate is not None else 0, 8 if gate is not None else 0, out.data_ptr(),
            workers, ws.data_ptr(), ws.numel(), _cabi.stream())
        assert rc == 0, rc
        assert torch.isfinite(out.float()).all()
        err = (out.double().cpu() - want.reshape(n, -1)).abs().max().item()
        assert err < 1.1 * 2.0 ** -8 * max(v.abs().max().item() for v in V) * (1.42 if turn is not None else 1.0), (workers, err)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(8, 2, 128, 128), (20, 1, 64, 128), (4, 4, 128, 64)])
@pytest.mark.parametrize("stride", [0, 2])
def test_weights_of_small_batches_are_float(heads, kv_heads, dim, vdim, stride):
    """With fewer (token, kv head) pairs than SMs, and for query rows that are not 16-byte aligned, the softmax weights keep the 24 bits of a
    float in the second product, as in the streaming kernel.

    Bound: the result is rounded to bfloat16 once (2^-8 of itself); scores of up to 8 are float sums (error 2^-20, so the weights' too), as
    are the weighted sums: 2^-16 max |v| covers them.  Weights rounded to bfloat16 are off by up to 2^-8 max |v|."""
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    g = torch.Generator().manual_seed(heads + dim + stride)
    pos = [2, 6, 15, 16, 40, 300]
    n, per, scale = len(pos), heads // kv_heads, dim ** -0.5 * 1.5
    if stride:                                  # enough pairs for an SM each, rows of queries at 4-byte places
        pos = (pos * 200)[:max(1, 160 // kv_heads) + 1]
        n = len(pos)
    states = SequenceStateCache(n, sum(c + 17 for c in pos), 16, dev)
    kv = states.add_kv_layer(kv_heads, dim, vdim, "bf16")
    slots = [states.alloc() for _ in range(n)]
    batch = states.make_batch([(s, [0] * (c + 1)) for s, c in zip(slots, pos)])
    KV = torch.randn(batch.rows, kv_heads * (dim + vdim), generator=g).to(BF)
    V = KV[:, kv_heads * dim:].clone()
    KV[1, kv_heads * dim + 3], KV[3, -1] = float("inf"), float("nan")       # of the first and the second token: they stay in their columns
    kv.append_rows(KV.to(dev), 0, kv_heads * dim, batch.row_slot, batch.row_pos)
    Q = torch.randn(n, heads * dim + 8 + stride, generator=g).to(BF)
    want, r0 = torch.zeros(n, heads, vdim, dtype=torch.float64), 0
    for i, c in enumerate(pos):
        x = KV[r0:r0 + c + 1].double()
        k, v = x[:, :kv_heads * dim].reshape(c + 1, kv_heads, dim), x[:, kv_heads * dim:].reshape(c + 1, kv_heads, vdim)
        q = Q[i, stride:stride + heads * dim].double().reshape(kv_heads, per, dim)
        want[i] = torch.einsum("ghj,jgv->ghv", torch.softmax(torch.einsum("ghd,jgd->ghj", q, k) * scale, -1), v).reshape(heads, vdim)
        r0 += c + 1
    tiles = torch.tensor([[i, 1, s, c] for i, (s, c) in enumerate(zip(slots, pos))], dtype=torch.int32, device=dev)
    Qd, pt = Q.to(dev), kv.page_table_
    for workers in (1, lib.pa_masked_decode_workers(n, heads, kv_heads, 301)):
        ws = torch.empty(lib.pa_masked_decode_workspace_bytes(n, heads, kv_heads, vdim, workers), dtype=torch.uint8, device=dev)
        out = torch.full((n, heads * vdim), float("nan"), dtype=BF, device=dev)
        assert lib.pa_masked_decode(
            Qd.data_ptr(), Qd.stride(0), stride, kv.key_buffer_.data_ptr(), kv.value_buffer_.data_ptr(), pt.device_data().data_ptr(),
            pt.num_beams_, pt.num_heads_, pt.num_tiles_, kv.total_pages_, kv.tile_size_, tiles.data_ptr(), n, heads, dim, vdim, scale, 0.0, 0, 0, 0,
            0, None, 0, None, None, None, None, None, 0, 0, out.data_ptr(), workers, ws.data_ptr(), ws.numel(), _cabi.stream()) == 0
        got, fin = out.double().cpu().reshape(want.shape), torch.isfinite(want)
        assert torch.equal(torch.nan_to_num(got[~fin], 7.0), torch.nan_to_num(want[~fin], 7.0)), (workers, got[~fin], want[~fin])
        err = (got - want)[fin].abs() - 2.0 ** -8 * want[fin].abs()
        assert err.max().item() < 2.0 ** -16 * V.abs().max().item(), (workers, err.max().item())
