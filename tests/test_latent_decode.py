"""pa_latent_decode (csrc/latent_decode.cu) alone, against attention written out in float64: tokens whose keys end inside, on and just
past a unit of 32 keys and a half of it, one worker for everything, more workers than units, more heads than the 16 rows of a
product, rotated parts that end inside a 16-column step.  Pool rows that no query may see hold NaN.

Bound: the weights enter the second product as bfloat16 (2^-9 of sum p |c|) and the result is rounded once more (2^-9): 2^-8 max |c|;
1.1 times that is asked."""
import pytest
import torch

BF = torch.bfloat16
POS = [0, 15, 16, 31, 32, 300, 1, 257, 47, 511]


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_rank,rot_dim", [(16, 512, 64), (8, 256, 32), (3, 128, 8), (20, 384, 24), (40, 128, 0)])
@pytest.mark.parametrize("sink", [None, 0.0, 30.0])
def test_shares_of_decoded_tokens(heads, kv_rank, rot_dim, sink):
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev = _cabi.lib(), torch.device("cuda")
    g = torch.Generator().manual_seed(heads + kv_rank)
    n, kd, scale = len(POS), kv_rank + rot_dim, 1.5 * (kv_rank + rot_dim) ** -0.5
    states = SequenceStateCache(n, 4096, 16, dev)
    kv = states.add_kv_layer(1, kd, 0, "bf16")
    slots = [states.alloc() for _ in range(n)]
    for r in range(32):                                     # growth in turns, so that the sequences' pages interleave
        for i in (2, 0, 3, 1, 6, 5, 4, 9, 8, 7):
            if POS[i] > 16 * r:
                states.extend(slots[i], min(16, POS[i] - 16 * r))
    batch = states.make_batch([(s, [0]) for s in slots])
    pt = kv.page_table_
    tab = pt.device_data().cpu().reshape(pt.num_beams_, pt.num_tiles_)
    C = [torch.randn(c + 1, kd, generator=g).to(BF) for c in POS]
    pool = torch.full(kv.key_buffer_.shape, float("nan"), dtype=BF)
    for i, c in enumerate(POS):
        for j in range(c + 1):
            pool[int(tab[slots[i], j // 16]), j % 16] = C[i][j]
    kv.key_buffer_.copy_(pool)
    ql = torch.randn(heads, n, kv_rank, generator=g).to(BF)
    qr = torch.randn(n, heads * (rot_dim + 4), generator=g).to(BF)
    sk = None if sink is None else torch.randn(heads, generator=g) + sink
    want = torch.zeros(heads, n, kv_rank, dtype=torch.float64)
    for i in range(n):
        k = C[i].double()
        q = torch.cat([ql[:, i].double(), qr[i].double().reshape(heads, rot_dim + 4)[:, 4:]], 1)
        s = q @ k.T * scale
        if sk is not None:
            s = torch.cat([s, sk.double()[:, None]], 1)
        want[:, i] = torch.softmax(s, -1)[:, :k.shape[0]] @ k[:, :kv_rank]
    qld, qrd, skd = ql.to(dev), qr.to(dev), sk.to(dev) if sk is not None else None
    tiles, ntiles, longest = batch.query_tiles(1)[1]
    for workers in (1, 3, lib.pa_latent_decode_workers(n, heads, longest), 148):
        ws = torch.empty(lib.pa_latent_decode_workspace_bytes(n, heads, kv_rank, workers), dtype=torch.uint8, device=dev)
        out = torch.full((heads, n, kv_rank), float("nan"), dtype=BF, device=dev)
        rc = lib.pa_latent_decode(qld.data_ptr(), kv_rank, n * kv_rank, qrd.data_ptr() + 8, heads * (rot_dim + 4), rot_dim + 4,
                                  kv.key_buffer_.data_ptr(), pt.device_data().data_ptr(), pt.num_beams_, pt.num_tiles_, kv.total_pages_, 16,
                                  tiles.data_ptr(), ntiles, heads, kv_rank, rot_dim, scale, _cabi.ptr(skd), out.data_ptr(), kv_rank,
                                  n * kv_rank, workers, ws.data_ptr(), ws.numel(), _cabi.stream())
        assert rc == 0, rc
        assert torch.isfinite(out.float()).all()
        err = (out.double().cpu() - want).abs().max().item()
        assert err < 1.1 * 2.0 ** -8 * max(c.abs().max().item() for c in C), (workers, err)
