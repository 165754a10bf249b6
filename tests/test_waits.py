"""Kernels whose waits run out (the limit of a wait is an argument; with 0 nothing is requested, so that the first wait runs out): the call
returns, its rows are NaN and never plausible numbers, the count of waits that ran out goes up, and the next call is served.  In processes
of their own, since other tests ask for a count of zero."""
import os
import subprocess
import sys

import pytest
import torch

BF = torch.bfloat16


def _count(fn):
    import ctypes
    n = ctypes.c_int(-1)
    assert fn(ctypes.byref(n)) == 0
    return n.value


def masked_decode():
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev, H, G, D, pos = _cabi.lib(), torch.device("cuda"), 8, 2, 128, [0, 30, 700, 5, 2000]
    for copies in (1, 30):                      # float and bfloat16 weights
        tokens = pos * copies
        n = len(tokens)
        st = SequenceStateCache(n, sum(tokens) + 32 * n, 16, dev)
        kv = st.add_kv_layer(G, D, D, "bf16")
        slots = [st.alloc() for _ in tokens]
        b = st.make_batch([(s, [0] * (c + 1)) for s, c in zip(slots, tokens)])
        kv.append_rows(torch.randn(b.rows, 2 * G * D, device=dev).to(BF), 0, G * D, b.row_slot, b.row_pos)
        tiles = torch.tensor([[i, 1, s, c] for i, (s, c) in enumerate(zip(slots, tokens))], dtype=torch.int32, device=dev)
        q, pt = torch.randn(n, H * D, device=dev).to(BF), kv.page_table_
        workers = lib.pa_masked_decode_workers(n, H, G, 2001)
        ws = torch.empty(lib.pa_masked_decode_workspace_bytes(n, H, G, D, workers), dtype=torch.uint8, device=dev)
        for polls in (0, 1 << 25):
            out, before = torch.zeros(n, H * D, dtype=BF, device=dev), _count(lib.pa_attention_tc_errors)
            assert lib.pa_masked_decode_polls(
                q.data_ptr(), H * D, 0, kv.key_buffer_.data_ptr(), kv.value_buffer_.data_ptr(), pt.device_data().data_ptr(), pt.num_beams_,
                pt.num_heads_, pt.num_tiles_, kv.total_pages_, 16, tiles.data_ptr(), n, H, D, D, 0.1, 0.0, 0, 0, 0, 0, None, 0, None, None, None,
                None, None, 0, 0, out.data_ptr(), workers, ws.data_ptr(), ws.numel(), polls, _cabi.stream()) == 0
            ran_out = _count(lib.pa_attention_tc_errors) - before
            assert torch.isnan(out.float()).all() and ran_out > 0 if polls == 0 else torch.isfinite(out.float()).all() and ran_out == 0


def latent_decode():
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev, H, kvr, rot, pos = _cabi.lib(), torch.device("cuda"), 20, 256, 32, [0, 30, 300, 5, 90, 40]
    n, kd = len(pos), kvr + rot
    st = SequenceStateCache(n, sum(pos) + 32 * n, 16, dev)
    kv = st.add_kv_layer(1, kd, 0, "bf16")
    slots = [st.alloc() for _ in pos]
    st.make_batch([(s, [0] * (c + 1)) for s, c in zip(slots, pos)])
    kv.key_buffer_.normal_()
    tiles = torch.tensor([[i, 1, s, c] for i, (s, c) in enumerate(zip(slots, pos))], dtype=torch.int32, device=dev)
    ql, qr, pt = torch.randn(H, n, kvr, device=dev).to(BF), torch.randn(n, H * rot, device=dev).to(BF), kv.page_table_
    for workers in (lib.pa_latent_decode_workers(n, H, 301), 7):
        ws = torch.empty(lib.pa_latent_decode_workspace_bytes(n, H, kvr, workers), dtype=torch.uint8, device=dev)
        for polls in (0, 1 << 25):
            out, before = torch.zeros(H, n, kvr, dtype=BF, device=dev), _count(lib.pa_attention_tc_errors)
            assert lib.pa_latent_decode_polls(
                ql.data_ptr(), kvr, n * kvr, qr.data_ptr(), H * rot, rot, kv.key_buffer_.data_ptr(), pt.device_data().data_ptr(), pt.num_beams_,
                pt.num_tiles_, kv.total_pages_, 16, tiles.data_ptr(), n, H, kvr, rot, 0.1, None, out.data_ptr(), kvr, n * kvr, workers, ws.data_ptr(),
                ws.numel(), polls, _cabi.stream()) == 0
            ran_out = _count(lib.pa_attention_tc_errors) - before
            assert torch.isnan(out.float()).all() and ran_out > 0 if polls == 0 else torch.isfinite(out.float()).all() and ran_out == 0


def grouped():
    from llm_decoder import _cabi
    lib, dev, rows, experts, top, width, ff = _cabi.lib(), torch.device("cuda"), 700, 3, 2, 192, 264
    g, pairs = torch.Generator().manual_seed(1), 1400
    ids = torch.randint(0, experts, (pairs,), generator=g).to(torch.int32).to(dev)
    order, meta = torch.empty(pairs, dtype=torch.int32, device=dev), torch.empty(lib.pa_moe_meta_ints(pairs, experts), dtype=torch.int32, device=dev)
    assert lib.pa_moe_sort(ids.data_ptr(), pairs, experts, order.data_ptr(), meta.data_ptr(), _cabi.stream()) == 0
    h, mid = torch.randn(rows, width, device=dev).to(BF), torch.randn(pairs, ff, device=dev).to(BF)
    wu, wd = torch.randn(experts, 2 * ff, width, device=dev).to(BF), torch.randn(experts, width, ff, device=dev).to(BF)
    for mode, a, w, K, n_out, t in ((0, h, wu, width, ff, top), (1, mid, wd, ff, width, 1), (2, h, wu[:, :ff].contiguous(), width, ff, top)):
        for act in (0, 1) if mode != 1 else (0,):
            for polls in (0, 1 << 25):
                out = torch.zeros(pairs, n_out, device=dev, dtype=torch.float32 if mode == 1 else BF)
                before = _count(lib.pa_moe_tc_errors)
                assert lib.pa_moe_grouped_polls(mode, a.data_ptr(), K, w.data_ptr(), K, n_out, experts, order.data_ptr(), None, t, meta.data_ptr(),
                                                pairs, act, out.data_ptr(), polls, _cabi.stream()) == 0
                ran_out = _count(lib.pa_moe_tc_errors) - before
                assert torch.isnan(out.float()).all() and ran_out > 0 if polls == 0 else torch.isfinite(out.float()).all() and ran_out == 0


def grouped_pairs():
    """Pairs of CTAs, several tiles for each, with their sorted rows: all waits, or those of one CTA's epilogue alone."""
    from llm_decoder import _cabi
    lib, dev, pairs, experts, K, n_out = _cabi.lib(), torch.device("cuda"), 6400, 2, 2048, 3072
    ids = torch.randint(0, experts, (pairs,), generator=torch.Generator().manual_seed(1)).to(torch.int32).to(dev)
    order, meta = torch.empty(pairs, dtype=torch.int32, device=dev), torch.empty(lib.pa_moe_meta_ints(pairs, experts), dtype=torch.int32, device=dev)
    assert lib.pa_moe_sort(ids.data_ptr(), pairs, experts, order.data_ptr(), meta.data_ptr(), _cabi.stream()) == 0
    a, w = torch.randn(pairs, K, device=dev).to(BF), torch.randn(experts, 2 * n_out, K, device=dev).to(BF)
    nb = lib.pa_moe_sorted_rows_bytes(pairs, experts, K, 2)
    rows, most = torch.empty(nb, dtype=torch.uint8, device=dev), 1 << 25
    for mode in (0, 1, 2):
        wt, whole = w if mode == 0 else w[:, :n_out].contiguous(), None
        for limits in ((most, most, most), (0, 0, 0), (most, 0, most), (most, most, 0), (most, most, most)):
            out = torch.zeros(pairs, n_out, device=dev, dtype=torch.float32 if mode == 1 else BF)
            before = _count(lib.pa_moe_tc_errors)
            assert lib.pa_moe_grouped_waits(mode, a.data_ptr(), K, wt.data_ptr(), K, n_out, experts, order.data_ptr(), None, 1, meta.data_ptr(), pairs,
                                            0, out.data_ptr(), rows.data_ptr(), nb, *limits, _cabi.stream()) == 0
            ran_out, lost = _count(lib.pa_moe_tc_errors) - before, torch.isnan(out.float())
            if min(limits) == most:
                assert ran_out == 0 and not lost.any() and (whole is None or torch.equal(out, whole))
                whole = out
            else:                   # what the other CTA writes is what it should be, or NaN too
                assert ran_out > 0 and lost.any() and (limits[0] or lost.all()), (mode, limits)
                assert bool((lost | (out == whole)).all()), (mode, limits)


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["masked_decode", "latent_decode", "grouped", "grouped_pairs"])
def test_rows_of_waits_that_run_out(case):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), case], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stdout + r.stderr


if __name__ == "__main__":
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    sys.path.insert(0, os.path.join(root, "pagedattention-based-transformer-decoder-inference-framework_b200"))
    globals()[sys.argv[1]]()
    torch.cuda.synchronize()
    print("done")
