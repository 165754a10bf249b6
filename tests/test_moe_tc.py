"""The tcgen05 form of the grouped expert products (csrc/moe_tc.cu) alone, against the same products in float64: experts without
pairs, with less than a row tile and with several, output sizes that end inside a strip of 128 or 256, inner sizes that end
inside a stage of 64, with and without a weight on the input, gate / up pairs and single products with each activation.

Bound of the first product: gate, up and their product are rounded to bfloat16 (half a unit each, 2^-9 relative), relu squared and
gate * up double a relative error: 4 * 2^-9 of the largest result, and as much again for values next to a rounding border.  The second
product is float on bfloat16 operands: 1e-5 of sum |a| |w|."""
import ctypes

import pytest
import torch

BF = torch.bfloat16


@pytest.mark.gpu
@pytest.mark.parametrize("rows,experts,top,width,ff", [(700, 3, 2, 192, 264), (257, 2, 1, 64, 520), (1300, 20, 2, 136, 128), (129, 1, 1, 72, 8),
                                                        # from 6144 pairs and 256 an expert on also by pairs of CTAs, tiles of 256
                                                        (6144, 1, 1, 72, 8), (3300, 3, 2, 136, 264), (3205, 24, 2, 320, 136),
                                                        # several tiles for each pair: up, down
                                                        (3200, 2, 2, 136, 3208), (3200, 2, 2, 3080, 136)])
@pytest.mark.parametrize("act,gated,weighted", [(0, True, False), (1, True, True), (2, False, False)])
def test_grouped_products(rows, experts, top, width, ff, act, gated, weighted):
    from llm_decoder import _cabi
    lib, dev, s = _cabi.lib(), torch.device("cuda"), _cabi.stream
    g = torch.Generator().manual_seed(rows + act)
    pairs = rows * top
    h = torch.randn(rows, width, generator=g).to(BF)
    wu = (torch.randn(experts, (2 if gated else 1) * ff, width, generator=g) / width ** 0.5).to(BF)
    wd = (torch.randn(experts, width, ff, generator=g) / ff ** 0.5).to(BF)
    ids = torch.randint(0, experts, (pairs,), generator=g)
    if experts > 2:
        ids[ids == 1] = 0                       # one expert without pairs
        ids[ids == 2] = 0
        ids[:5] = 2                             # one with five
    sel_w = torch.rand(pairs, generator=g) + 0.1
    idd, swd = ids.to(torch.int32).to(dev), sel_w.to(dev)
    order = torch.empty(pairs, dtype=torch.int32, device=dev)
    meta = torch.empty(lib.pa_moe_meta_ints(pairs, experts), dtype=torch.int32, device=dev)
    _cabi.check(lib.pa_moe_sort(idd.data_ptr(), pairs, experts, order.data_ptr(), meta.data_ptr(), s()), "sort")
    hd, wud, wdd = h.to(dev), wu.to(dev), wd.to(dev)
    mid = torch.full((pairs, ff), float("nan"), device=dev, dtype=BF)
    out = torch.full((pairs, width), float("nan"), device=dev)
    fn = lib.pa_moe_gate_up_act if gated else lib.pa_moe_up
    _cabi.check(fn(hd.data_ptr(), width, wud.data_ptr(), width, ff, experts, order.data_ptr(), swd.data_ptr() if weighted else None, top,
                   meta.data_ptr(), pairs, act, mid.data_ptr(), 2, s()), "up")
    nb = lib.pa_moe_sorted_rows_bytes(pairs, experts, width, 2)
    assert (nb > 0) == (pairs >= 6144)
    if nb:                      # the same through sorted rows, by pairs of CTAs: the same sums
        rows_ws, mid2 = torch.empty(nb, dtype=torch.uint8, device=dev), torch.full_like(mid, float("nan"))
        _cabi.check(lib.pa_moe_up_sorted(hd.data_ptr(), width, wud.data_ptr(), 1 if gated else 0, width, ff, experts, order.data_ptr(),
                                         swd.data_ptr() if weighted else None, top, meta.data_ptr(), pairs, act, mid2.data_ptr(),
                                         rows_ws.data_ptr(), nb, 2, s()), "sorted")
        assert torch.equal(mid, mid2)
    _cabi.check(lib.pa_moe_down(mid.data_ptr(), wdd.data_ptr(), ff, width, experts, order.data_ptr(), meta.data_ptr(), pairs, out.data_ptr(), 2,
                                s()), "down")
    if nb:                      # by pairs of CTAs whether or not they pay at this size
        out2 = torch.full_like(out, float("nan"))
        _cabi.check(lib.pa_moe_grouped_polls(1, mid.data_ptr(), ff, wdd.data_ptr(), ff, width, experts, order.data_ptr(), None, 1, meta.data_ptr(),
                                             pairs, 0, out2.data_ptr(), 1 << 25, s()), "down by pairs")
        assert torch.equal(out, out2)
    o = order.long().cpu()
    assert sorted(o.tolist()) == list(range(pairs)) and bool((ids[o][1:] >= ids[o][:-1]).all())
    a = h[o // top].double() * (sel_w[o].double()[:, None] if weighted else 1.0)
    want_mid, want = torch.empty(pairs, ff, dtype=torch.float64), torch.empty(pairs, width, dtype=torch.float64)
    bound = torch.empty(pairs, width, dtype=torch.float64)
    f = [lambda v: v * torch.sigmoid(v), lambda v: v.clamp(min=0), lambda v: v.clamp(min=0) ** 2][act]
    got_mid = mid.cpu()
    for e in range(experts):
        r = ids[o] == e
        p = a[r] @ wu[e].double().T
        want_mid[r] = f(p[:, :ff]) * p[:, ff:] if gated else f(p)
        want[r], bound[r] = got_mid[r].double() @ wd[e].double().T, got_mid[r].double().abs() @ wd[e].double().abs().T
    assert (got_mid.double() - want_mid).abs().max() < 8 * 2.0 ** -9 * want_mid.abs().max()
    assert ((out.double().cpu()[o] - want).abs() <= 1e-5 * bound + 1e-30).all()
    n = ctypes.c_int(-1)
    assert lib.pa_moe_tc_errors(ctypes.byref(n)) == 0 and n.value == 0


@pytest.mark.gpu
def test_waits_of_a_pair_of_ctas():
    """Pairs of CTAs whose waits run out leave NaN and are counted, and the next launch is whole."""
    from llm_decoder import _cabi
    lib, dev, s = _cabi.lib(), torch.device("cuda"), _cabi.stream
    g = torch.Generator().manual_seed(5)
    pairs, experts, K, n_out = 6200, 2, 136, 264
    a, w = torch.randn(pairs, K, generator=g).to(BF).to(dev), torch.randn(experts, n_out, K, generator=g).to(BF).to(dev)
    ids = torch.randint(0, experts, (pairs,), generator=g, dtype=torch.int32).to(dev)
    order = torch.empty(pairs, dtype=torch.int32, device=dev)
    meta = torch.empty(lib.pa_moe_meta_ints(pairs, experts), dtype=torch.int32, device=dev)
    _cabi.check(lib.pa_moe_sort(ids.data_ptr(), pairs, experts, order.data_ptr(), meta.data_ptr(), s()), "sort")
    out, counts = [], []
    for polls in (1 << 25, 0, 1 << 25):
        o, n = torch.zeros(pairs, n_out, device=dev), ctypes.c_int()
        assert lib.pa_moe_grouped_polls(1, a.data_ptr(), K, w.data_ptr(), K, n_out, experts, order.data_ptr(), None, 1, meta.data_ptr(), pairs, 0,
                                        o.data_ptr(), polls, s()) == 0
        assert lib.pa_moe_tc_errors(ctypes.byref(n)) == 0
        out.append(o)
        counts.append(n.value)
    assert counts[1] > counts[0] and counts[2] == counts[1]
    assert bool(torch.isnan(out[1]).all()) and torch.equal(out[0], out[2]) and not bool(torch.isnan(out[0]).any())


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [True, False])
def test_pairs_without_an_expert(gated):
    """Ids of no expert (a router's identity outputs) have no place in the sorted order: the copy of the rows ends where the sort did."""
    from llm_decoder import _cabi
    lib, dev, s = _cabi.lib(), torch.device("cuda"), _cabi.stream
    g = torch.Generator().manual_seed(9)
    rows, top, experts, width, ff = 3600, 2, 4, 136, 264
    pairs = rows * top
    ids = torch.randint(0, experts + 2, (pairs,), generator=g, dtype=torch.int32).to(dev)
    order = torch.zeros(pairs, dtype=torch.int32, device=dev)           # its end, which the sort leaves alone, names a row that there is
    meta = torch.empty(lib.pa_moe_meta_ints(pairs, experts), dtype=torch.int32, device=dev)
    _cabi.check(lib.pa_moe_sort(ids.data_ptr(), pairs, experts, order.data_ptr(), meta.data_ptr(), s()), "sort")
    count = int((ids < experts).sum())
    assert int(meta[experts]) == count < pairs
    h = torch.randn(rows, width, generator=g).to(BF).to(dev)
    w = (torch.randn(experts, (2 if gated else 1) * ff, width, generator=g) / width ** 0.5).to(BF).to(dev)
    nb = lib.pa_moe_sorted_rows_bytes(pairs, experts, width, 2)
    assert nb == pairs * width * 2
    scratch = torch.full((pairs, width), 7.5, dtype=BF, device=dev)
    out = []
    for ws in (scratch, None):
        o = torch.full((pairs, ff), 3.25, dtype=BF, device=dev)
        _cabi.check(lib.pa_moe_up_sorted(h.data_ptr(), width, w.data_ptr(), 1 if gated else 0, width, ff, experts, order.data_ptr(), None, top,
                                         meta.data_ptr(), pairs, 1, o.data_ptr(), _cabi.ptr(ws), nb if ws is not None else 0, 2, s()), "sorted")
        out.append(o)
    assert bool((scratch[count:] == 7.5).all()) and torch.equal(scratch[:count], h[order[:count].long() // top])
    assert torch.equal(out[0], out[1]) and bool((out[0][count:] == 3.25).all())


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [300, 6200])
def test_silu_of_large_negative_gates(rows):
    """Gates near -88, whose sigmoid's denominator is above 2^126, with an up value that makes the result an ordinary number.  Bound: gate
    and up are exact here, expf and the division are off by a few units of 2^-24, and the result is rounded to bfloat16, whose eight bits
    leave half a unit: up to 2^-8 of the value."""
    from llm_decoder import _cabi
    lib, dev, s = _cabi.lib(), torch.device("cuda"), _cabi.stream
    K, ff = 64, 16
    gates = torch.tensor([-87.5, -88.0, -88.5, -60.0, -87.0, -20.0, -1.0, 4.0]).repeat(2)
    w = torch.zeros(1, 2 * ff, K)
    w[0, :ff, 0], w[0, ff:, 1] = gates, 2.0 ** 100
    h = torch.zeros(rows, K)
    h[:, 0], h[:, 1] = 1.0, 2.0
    hd, wd, ids = h.to(BF).to(dev), w.to(BF).to(dev), torch.zeros(rows, dtype=torch.int32, device=dev)
    order, out = torch.empty(rows, dtype=torch.int32, device=dev), torch.empty(rows, ff, dtype=BF, device=dev)
    meta = torch.empty(lib.pa_moe_meta_ints(rows, 1), dtype=torch.int32, device=dev)
    _cabi.check(lib.pa_moe_sort(ids.data_ptr(), rows, 1, order.data_ptr(), meta.data_ptr(), s()), "sort")
    nb = lib.pa_moe_sorted_rows_bytes(rows, 1, K, 2)
    ws = torch.empty(nb, dtype=torch.uint8, device=dev) if nb else None
    _cabi.check(lib.pa_moe_up_sorted(hd.data_ptr(), K, wd.data_ptr(), 1, K, ff, 1, order.data_ptr(), None, 1, meta.data_ptr(), rows, 0,
                                     out.data_ptr(), _cabi.ptr(ws), nb, 2, s()), "up")
    g = gates.double()
    want = g / (1.0 + torch.exp(-g)) * 2.0 ** 101
    assert ((out.double().cpu() - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs()).all()


@pytest.mark.gpu
def test_where_pairs_of_ctas_pay():
    """The rule asks for full tiles, two rounds of them, and enough columns; what it names is what the scratch is for."""
    from llm_decoder import _cabi
    lib = _cabi.lib()
    worth = lambda *a: lib.pa_moe_sorted_rows_worth(*a, 2)  # noqa: E731
    assert worth(16384, 8, 2048, 2048, 1) == 16384 * 2048 * 2 == worth(16384, 8, 2048, 3072, 0)
    assert worth(16384, 16, 2048, 2048, 1) > 0 and worth(8192, 8, 4096, 1536, 1) > 0
    for few in ((16384, 8, 2048, 1024, 1), (16384, 8, 2048, 2048, 0), (16384, 8, 1024, 4096, 1), (8192, 16, 2048, 2048, 1), (4096, 4, 2048, 4096, 1)):
        assert worth(*few) == 0
    assert lib.pa_moe_sorted_rows_worth(16384, 8, 2048, 2048, 1, 4) == 0
