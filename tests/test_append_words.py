"""The forms of the append kernels that read and write whole 16-byte words, against the forms that go element by element: the same
numbers at a column offset and a row stride that only the latter take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, dtype):
    # one rounding of the result's type, where a sum of squares in another order moved it
    rel = 2.0 ** -7 if dtype == torch.bfloat16 else 2e-5
    got, want = got.double(), want.double()
    assert ((got - want).abs() <= rel * want.abs() + 1e-6).all()


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,rot_dims,norm", [(16, 4, 128, 128, 128, 1), (3, 1, 64, 128, 32, 1), (5, 2, 24, 40, 8, 1),
                                                                   (2, 1, 256, 200, 64, 1), (12, 12, 64, 64, 64, 0), (1, 1, 104, 8, 0, 1)])
@pytest.mark.parametrize("taps", [0, 1, 3, 4, 6])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_convolved_rows(heads, kv_heads, dim, vdim, rot_dims, norm, taps, dtype):
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    g = torch.Generator().manual_seed(dim + taps)
    channels = heads * dim + kv_heads * (dim + vdim)
    wt = (torch.randn(taps, channels, generator=g) * 0.6).to(dev) if taps else None
    out = []
    for off, pad in ((8, 0), (1, 3)):
        states = SequenceStateCache(3, 512, 16, dev)
        kv = states.add_kv_layer(kv_heads, dim, vdim, "f32" if dtype == torch.float32 else "bf16")
        kv.key_buffer_.zero_(), kv.value_buffer_.zero_()
        state = states.add_state((taps - 1) * channels) if taps > 1 else None
        slots = [states.alloc() for _ in range(3)]
        r, res = torch.Generator().manual_seed(7), []
        for step in ([(0, 34), (1, 1), (2, 17)], [(2, 1), (0, 15), (1, 4)]):
            batch = states.make_batch([(slots[i], [0] * n) for i, n in step])
            x = torch.zeros(batch.rows, off + channels + 8 + pad, dtype=dtype, device=dev)
            x[:, off:off + channels] = torch.randn(batch.rows, channels, generator=r).to(dtype)
            rope = torch.randn(batch.rows, max(rot_dims, 1), generator=r).to(dev)
            q = torch.zeros(batch.rows, heads * dim, dtype=dtype, device=dev)
            items, n = batch.portion_items(16)
            pt = kv.page_table_
            assert lib.pa_conv_rope_norm_append(
                x.data_ptr(), x.stride(0), off, heads, kv_heads, dim, vdim, taps, _cabi.ptr(wt), _cabi.ptr(state), rot_dims,
                rope.data_ptr() if rot_dims else None, norm, 1e-5, q.data_ptr(), heads * dim, kv.key_buffer_.data_ptr(), kv.value_buffer_.data_ptr(),
                pt.device_data().data_ptr(), pt.num_beams_, pt.num_tiles_, kv.total_pages_, kv.tile_size_, items.data_ptr(), n, 16,
                4 if dtype == torch.float32 else 2, _cabi.stream()) == 0
            res.append(q)
        out.append(res + [kv.key_buffer_, kv.value_buffer_] + ([state[slots]] if state is not None else []))
    for got, want in zip(*out):
        _close(got, want, dtype)
    if taps > 1:
        assert torch.equal(out[0][-1], out[1][-1])


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,rot_dims,norm", [(16, 4, 128, 128, 128, 1), (12, 2, 64, 128, 32, 1), (16, 4, 64, 64, 64, 0),
                                                                   (8, 4, 104, 104, 104, 1), (5, 3, 40, 64, 8, 1), (7, 1, 72, 40, 0, 1)])
@pytest.mark.parametrize("taps", [0, 1, 2, 3, 4])
def test_convolved_rows_of_many_items(heads, kv_heads, dim, vdim, rot_dims, norm, taps):
    """The form for many long items: portions of one to 64 tokens (whole, ragged and single-token items), two steps of which the second
    starts inside pages, pages that are missing, pages out of range, a portion whose slot is none."""
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    units, columns, channels = heads + 2 * kv_heads, max(dim, vdim), heads * dim + kv_heads * (dim + vdim)
    lens = [48, 16, 31, 15, 32, 17, 64, 2, 16, 29]                     # 19 items of 14.2 tokens on average
    rounds = -(-(20 * _cabi.device_info()[0] * (1 if columns > 64 else 2) // units + 1) // 19)
    n, g = 10 * rounds, torch.Generator().manual_seed(dim + taps)
    wt = (torch.randn(taps, channels, generator=g) * 0.6).to(dev) if taps else None
    steps = [(lens * rounds)[i:] + (lens * rounds)[:i] for i in (0, 3)]
    raw = [torch.randn(sum(s), channels, generator=g).to(torch.bfloat16) for s in steps]
    rope = [torch.randn(sum(s), max(rot_dims, 1), generator=g).to(dev) for s in steps]
    out = []
    for off, pad in ((8, 0), (1, 3)):
        states = SequenceStateCache(n, 144 * n, 16, dev)
        kv = states.add_kv_layer(kv_heads, dim, vdim, "bf16")
        kv.key_buffer_.zero_(), kv.value_buffer_.zero_()
        state = states.add_state((taps - 1) * channels) if taps > 1 else None
        slots, res = [states.alloc() for _ in range(n)], []
        for step, x0, turns in zip(steps, raw, rope):
            batch = states.make_batch([(s, [0] * m) for s, m in zip(slots, step)])
            x = torch.zeros(batch.rows, off + channels + 8 + pad, dtype=torch.bfloat16, device=dev)
            x[:, off:off + channels] = x0.to(dev)
            q = torch.zeros(batch.rows, heads * dim, dtype=torch.bfloat16, device=dev)
            items, count = batch.portion_items(16)
            assert lib.pa_conv_append_in_words(units, columns, count, batch.rows) == 1
            items, lost = items.clone(), batch.portions[4]
            items[(items[:, 0] >= lost[0]) & (items[:, 0] < lost[0] + lost[1]), 2] = n + 3
            pt = kv.page_table_
            table = pt.device_data().clone().reshape(n, kv_heads, -1)
            table[slots[2], :, 0], table[slots[6], 0, 1], table[slots[0], -1, 2] = -1, kv.total_pages_, -1
            assert lib.pa_conv_rope_norm_append_rows(
                x.data_ptr(), x.stride(0), off, heads, kv_heads, dim, vdim, taps, _cabi.ptr(wt), _cabi.ptr(state), rot_dims,
                turns.data_ptr() if rot_dims else None, norm, 1e-5, q.data_ptr(), heads * dim, kv.key_buffer_.data_ptr(), kv.value_buffer_.data_ptr(),
                table.data_ptr(), pt.num_beams_, pt.num_tiles_, kv.total_pages_, kv.tile_size_, items.data_ptr(), count, 16, batch.rows, 2,
                _cabi.stream()) == 0
            q[lost[0]:lost[0] + lost[1]] = 0            # nobody's rows: what they hold is not said
            res.append(q)
        out.append(res + [kv.key_buffer_, kv.value_buffer_] + ([state] if state is not None else []))
    for got, want in zip(*out):
        assert bool((want != 0).any())
        _close(got, want, torch.bfloat16)
    if taps > 1:
        assert torch.equal(out[0][-1], out[1][-1])


def test_form_of_many_items():
    """Where the form for many long items is taken: not for decoded tokens, however many, nor for small heads."""
    from llm_decoder import _cabi
    lib, most = _cabi.lib(), 20 * _cabi.device_info()[0]        # warps that the other form holds at once
    words = lambda units, columns, items, tokens: lib.pa_conv_append_in_words(units, columns, items, int(items * tokens))  # noqa: E731
    for columns, per in ((128, 1), (72, 1), (64, 2), (40, 2)):
        items = most * per // 24
        assert not words(24, columns, items, 16) and words(24, columns, items + per, 16) and words(24, columns, 8 * items, 12)
        assert not any(words(24, columns, 8 * items, m) for m in (1, 2, 8, 11))
    for columns in (8, 32, 136):
        assert not words(24, columns, 100 * most, 16)


@pytest.mark.parametrize("kv_rank,rot_dim,rot_dims", [(512, 64, 64), (256, 32, 32), (8, 16, 16), (264, 24, 16), (1024, 8, 0), (40, 0, 0)])
@pytest.mark.parametrize("pairing", [0, 1])
@pytest.mark.parametrize("queries", ["turn", "norm", None])
def test_latent_rows(kv_rank, rot_dim, rot_dims, pairing, queries):
    from llm_decoder import _cabi
    lib, dev, heads, hs, q_rank = _cabi.lib(), torch.device("cuda"), 5, 16 + rot_dim, 136
    g = torch.Generator().manual_seed(kv_rank)
    rows, tile, ntiles, slots, pages = 21, 16, 3, 2, 5
    table = torch.tensor([[0, 3, -1], [9, 1, 2]], dtype=torch.int32)        # one place without a page, one page out of range
    place = torch.randperm(slots * ntiles * tile, generator=g)[:rows]
    slot, pos = (place // (ntiles * tile)).to(torch.int32), (place % (ntiles * tile)).to(torch.int32)
    pos[3], slot[4], pos[5] = -1, 7, 99                                     # rows that go nowhere
    raw = torch.randn(rows, kv_rank + rot_dim, generator=g).to(torch.bfloat16)
    qraw = torch.randn(rows, max(heads * hs, q_rank), generator=g).to(torch.bfloat16)
    gain, q_gain, rope = (torch.randn(n, generator=g).to(dev) for n in (kv_rank, q_rank, rows * max(rot_dims, 1)))
    out = []
    for off in (8, 1):
        cols = -(-(off + kv_rank + rot_dim + qraw.shape[1]) // 8) * 8 + 16
        x = torch.zeros(rows, cols, dtype=torch.bfloat16, device=dev)
        x[:, off:off + raw.shape[1]] = raw
        qo = off + raw.shape[1]
        x[:, qo:qo + qraw.shape[1]] = qraw
        pool = torch.zeros(pages, tile, kv_rank + rot_dim, dtype=torch.bfloat16, device=dev)
        q = torch.zeros(rows, 160, dtype=torch.bfloat16, device=dev) if queries == "norm" else x
        tabled, slotd, posd = table.to(dev), slot.to(dev), pos.to(dev)
        head = (pool.data_ptr(), tabled.data_ptr(), slots, ntiles, pages, tile, kv_rank, rot_dim, rot_dims, pairing, x.data_ptr(), x.stride(0),
                off, gain.data_ptr(), 1e-5, rope.data_ptr())
        if queries == "turn":
            rc = lib.pa_latent_turn_append(*head, x.data_ptr(), x.stride(0), qo, heads, hs, slotd.data_ptr(), posd.data_ptr(), rows, 2, _cabi.stream())
        else:
            rc = lib.pa_latent_norm_append(*head, qo, q_rank if queries else 0, q_gain.data_ptr() if queries else None,
                                           q.data_ptr() if queries else None, 160, slotd.data_ptr(), posd.data_ptr(), rows, 2, _cabi.stream())
        assert rc == 0
        out.append((pool, q if queries == "norm" else x[:, qo:qo + qraw.shape[1]], x[:, off:off + raw.shape[1]]))
    for got, want in zip(*out):
        _close(got, want, torch.bfloat16)
    assert torch.equal(out[0][2].cpu(), raw) and out[0][0].abs().sum() > 0
