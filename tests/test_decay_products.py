"""Chunks of a constant-decay scan as matrix products (decay_fold_mma_kernel, decay_replay_mma_kernel) against the recurrence walked
in float64, from a state that is not zero: portions that end inside, on and just past a chunk of 64, queries and keys shared by groups
of heads, every split of the rotation, strong and weak decays.

Bound: every factor keeps 24 bits and sums are float, so the error is that of a float sum of the same terms: the walk on the float
pipe is run on the same operands, and the products may be off by at most twice what it is, plus 2^-22 of the largest output (sums of
64 terms in another order)."""
import pytest
import torch


def _walk(q, k, v, decay, S):
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=torch.float64)
    for t in range(q.shape[0]):
        S = decay[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hd,hdv->hv", q[t], S)
    return out, S


def _turn(x, cs, sn, dims):
    h = dims // 2
    a, b = x[..., :h], x[..., h:dims]
    return torch.cat([a * cs - b * sn, b * cs + a * sn, x[..., dims:]], -1)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,groups,vdim,rot_dims", [(4, 4, 128, 64), (4, 2, 64, 0), (3, 1, 128, 28), (2, 2, 64, 32)])
def test_fold_and_replay(heads, groups, vdim, rot_dims):
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev, dim = _cabi.lib(), torch.device("cuda"), 64
    g = torch.Generator().manual_seed(heads + vdim + rot_dims)
    lens = [300, 64, 65, 1, 129, 63]
    R = sum(lens)
    states = SequenceStateCache(len(lens), 4096, 16, dev)
    st = states.add_state(heads * dim * vdim)
    slots = [states.alloc() for _ in lens]
    batch = states.make_batch([(s, [0] * n) for s, n in zip(slots, lens)])
    start = torch.randn(st.shape, generator=g)
    cols = 2 * groups * dim + heads * vdim
    X = torch.randn(R, cols + 8, generator=g).to(torch.bfloat16)
    decay = torch.tensor([1.0, 0.5, 0.97, 0.999][:heads])
    ang = torch.rand(R, max(rot_dims // 2, 1), generator=g) * 6.0
    rope = torch.stack([torch.cos(ang), torch.sin(ang)], -1)
    k_scale = dim ** -0.5
    want, states64, r0 = torch.empty(R, heads, vdim, dtype=torch.float64), [], 0
    for i, n in enumerate(lens):
        x = X[r0:r0 + n].double()
        q, k = x[:, :groups * dim].reshape(n, groups, dim), x[:, groups * dim:2 * groups * dim].reshape(n, groups, dim)
        if rot_dims:
            cs, sn = rope[r0:r0 + n, None, :, 0].double(), rope[r0:r0 + n, None, :, 1].double()
            q, k = _turn(q, cs, sn, rot_dims), _turn(k, cs, sn, rot_dims)
        rep = heads // groups
        q, k = q.repeat_interleave(rep, 1), (k * torch.tensor(k_scale, dtype=torch.float32).double()).repeat_interleave(rep, 1)
        o, S = _walk(q, k, x[:, 2 * groups * dim:cols].reshape(n, heads, vdim), decay.double(), start[slots[i]].reshape(heads, dim, vdim).double())
        want[r0:r0 + n] = o
        states64.append(S)
        r0 += n
    Xd, decayd, roped = X.to(dev), decay.to(dev), rope.to(dev).contiguous()
    items, n, s0, sn = batch.chunk_items(64)
    ws = torch.empty(lib.pa_decay_scan_workspace_bytes(n, heads, dim, vdim), dtype=torch.uint8, device=dev)
    off = []
    for chunk_tokens in (64, 0):            # as products, and walked
        st.copy_(start)
        out = torch.full((R, heads * vdim), float("nan"), device=dev)
        rc = lib.pa_decay_scan_chunked(Xd.data_ptr(), Xd.stride(0), 0, Xd.data_ptr(), Xd.stride(0), groups * dim, Xd.data_ptr(), Xd.stride(0),
                                       2 * groups * dim, heads, groups, dim, vdim, 0, decayd.data_ptr(), None, 0, 0, None, None, None,
                                       roped.data_ptr() if rot_dims else None, rot_dims, k_scale, st.data_ptr(), out.data_ptr(), out.stride(0),
                                       items.data_ptr(), n, s0.data_ptr(), sn.data_ptr(), batch.seq_slot.data_ptr(), batch.num_seqs, 1,
                                       ws.data_ptr(), ws.numel(), 2, chunk_tokens, _cabi.stream())
        assert rc == 0, rc
        off.append([(out.double().cpu().reshape(R, heads, vdim) - want).abs().max().item()] +
                   [(st[s].double().cpu().reshape(heads, dim, vdim) - S).abs().max().item() for s, S in zip(slots, states64)])
    top = [want.abs().max().item()] + [S.abs().max().item() for S in states64]
    for a, b, t in zip(*off, top):
        assert a <= 2 * b + 2.0 ** -22 * t, off


@pytest.mark.gpu
@pytest.mark.parametrize("vdim,groups", [(64, 2), (128, 1)])
@pytest.mark.parametrize("where", ["value", "nan value", "key", "query", "state", "large"])
def test_values_that_are_not_finite(vdim, groups, where):
    """An infinity or NaN in one token, or in the incoming state, reaches the outputs and states that the walk lets it reach and no others;
    large finite numbers give what the walk gives.

    Bound for what stays finite: both are float sums of up to 128 terms whose magnitudes add up to at most 2^11 here (2^-24 each), or to
    2^6 times the column's largest number where that is large: 2^-13 and 2^-18 of it."""
    from llm_decoder import _cabi
    from llm_decoder.seq_state import SequenceStateCache
    lib, dev, dim, heads, rot_dims = _cabi.lib(), torch.device("cuda"), 64, 2, 32
    g = torch.Generator().manual_seed(vdim + len(where))
    lens = [300, 70, 3]
    R, cols = sum(lens), 2 * groups * dim + heads * vdim
    states = SequenceStateCache(len(lens), 4096, 16, dev)
    st = states.add_state(heads * dim * vdim)
    slots = [states.alloc() for _ in lens]
    batch = states.make_batch([(s, [0] * n) for s, n in zip(slots, lens)])
    start = torch.randn(st.shape, generator=g)
    X = torch.randn(R, cols, generator=g).to(torch.bfloat16)
    v0, inf = 2 * groups * dim, float("inf")
    if where == "value":
        X[70, v0 + 5], X[77, v0 + 5], X[311, v0 + vdim + 3], X[372, v0] = inf, -inf, -inf, inf
    elif where == "nan value":
        X[20, v0 + 9], X[369, v0 + vdim] = float("nan"), float("nan")
    elif where == "key":
        X[130, groups * dim + 7], X[301, groups * dim + 40] = inf, float("nan")
    elif where == "query":
        X[200, 3], X[5, 50] = -inf, float("nan")
    elif where == "state":
        start[slots[0], 17], start[slots[1], dim * vdim + 4], start[slots[2], 2] = inf, float("nan"), -inf
    else:
        X[64:70, v0 + 1], X[305, groups * dim + 2], start[slots[2], 9] = 1e30, -1e25, 3e38
    decay = torch.tensor([0.9, 0.25])
    ang = torch.rand(R, rot_dims // 2, generator=g) * 6.0
    Xd, decayd, roped = X.to(dev), decay.to(dev), torch.stack([torch.cos(ang), torch.sin(ang)], -1).to(dev).contiguous()
    items, n, s0, sn = batch.chunk_items(64)
    ws = torch.empty(lib.pa_decay_scan_workspace_bytes(n, heads, dim, vdim), dtype=torch.uint8, device=dev)
    got = []
    for chunk_tokens in (64, 0):            # as products, and walked
        st.copy_(start)
        out = torch.full((R, heads * vdim), float("nan"), device=dev)
        assert lib.pa_decay_scan_chunked(
            Xd.data_ptr(), Xd.stride(0), 0, Xd.data_ptr(), Xd.stride(0), groups * dim, Xd.data_ptr(), Xd.stride(0), v0, heads, groups, dim, vdim, 0,
            decayd.data_ptr(), None, 0, 0, None, None, None, roped.data_ptr(), rot_dims, 0.125, st.data_ptr(), out.data_ptr(), out.stride(0),
            items.data_ptr(), n, s0.data_ptr(), sn.data_ptr(), batch.seq_slot.data_ptr(), batch.num_seqs, 1, ws.data_ptr(), ws.numel(), 2,
            chunk_tokens, _cabi.stream()) == 0
        got.append((out.cpu().reshape(R, heads, vdim), st.cpu().reshape(len(lens), heads, dim, vdim)[slots].transpose(1, 2)))
    for a, b in zip(*got):                  # outputs [token, head, column], states [sequence, dimension, head, column]
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
        assert torch.equal(a[torch.isinf(a)], b[torch.isinf(b)])
        ok = torch.isfinite(b)
        zero = torch.zeros_like(a)
        a, b = torch.where(ok, a, zero).double(), torch.where(ok, b, zero).double()
        r0 = 0
        for m in (lens if a.shape[0] == R else [1] * len(lens)):
            x, y = a[r0:r0 + m], b[r0:r0 + m]
            top = y.abs().cummax(0).values if m > 1 else y.abs().amax(1, keepdim=True)
            assert ((x - y).abs() <= 2.0 ** -18 * top + 2.0 ** -13).all(), ((x - y).abs() / (top + 1e-30)).max()
            r0 += m
