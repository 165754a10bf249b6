"""Layers of the sizes that the prompt kernels on tcgen05, the shared-out decode kernels and the chunk products serve, inside models and
against their float64 oracles (bfloat16 logits of every position): portions that build keys and values next to short ones and single
tokens, several groups of built rows and a portion past their limit, the three forms of the latent queries and gates, chunks of a constant-decay
scan between decoded tokens.  One error bound for all: that of the other bfloat16 model tests."""
import random

import pytest
import torch

from oracle import domilix_ref, namudra_ref, tiradra_ref

BF16_TOL = 0.06     # relative rms error of bfloat16 logits, median of the positions


def _case(name):
    if name == "tiradra":
        R = tiradra_ref
        c = R.make_config([R.latent_layer(heads=3, dim=128, rot_dim=32, vdim=64, kv_rank=128), R.attention_layer(heads=4, kv_heads=1, dim=64, vdim=128),
                           R.latent_layer(heads=2, dim=64, rot_dim=16, vdim=128, kv_rank=256)])
    elif name == "domilix":
        R = domilix_ref
        c = R.make_config([R.latent_layer(heads=2, dim=64, rot_dim=64, vdim=64, kv_rank=256, q_rank=64, mlp=R.dense_mlp()),
                           R.latent_layer(heads=5, dim=128, rot_dim=64, vdim=64, kv_rank=256, q_rank=40, kv_from=0, mlp=R.dense_mlp())])
    else:
        R = namudra_ref
        c = R.make_config([R.retention_layer(heads=2, dim=64, vdim=128, rot_dims=32), R.latent_layer(heads=2, dim=64, rot_dim=32, vdim=128, kv_rank=128),
                           R.retention_layer(heads=3, dim=64, vdim=64, rot_dims=64)], width=64)
    return R, c, R.random_weights(c, 11)


PLAN = [[("a", 300), ("b", 70)], [("a", 1), ("b", 140), ("c", 20)], [("a", 1), ("b", 1), ("c", 1)], [("a", 64), ("b", 90), ("c", 130)],
        [("a", 1), ("c", 1), ("b", 1)], [("b", 129), ("a", 63), ("c", 260)]]


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["tiradra", "domilix", "namudra"])
@pytest.mark.parametrize("rows", [None, 310])
def test_mixed_steps_against_the_oracle(monkeypatch, name, rows):
    """rows: the most rows of built keys and values at a time, so that a step makes several groups and the longest sequence none."""
    import llm_decoder as ld
    from llm_decoder import hybrid
    if rows is not None:
        monkeypatch.setattr(hybrid.LatentAttentionMixer, "_expand_rows", lambda *_a: rows)
    R, config, W = _case(name)
    rnd = random.Random(4)
    toks = {r: [rnd.randrange(config["vocab"]) for _ in range(sum(n for step in PLAN for q, n in step if q == r))] for r in "abc"}
    model = ld.HybridDecoder(config, W, "bfloat16", max_tokens=2048, max_seqs=4)
    eng, at, got = ld.Engine(model), {r: 0 for r in "abc"}, {r: [] for r in "abc"}
    for step in PLAN:
        logits, r0 = eng.step([(r, toks[r][at[r]:at[r] + n], list(range(n))) for r, n in step]), 0
        for r, n in step:
            got[r].append(logits[r0:r0 + n])
            at[r], r0 = at[r] + n, r0 + n
    for r in "abc":
        y = R.forward(config, W, toks[r])
        x, y = torch.cat(got[r]).double().cpu(), (y[0] if isinstance(y, tuple) else y).double()
        rel = (x - y).pow(2).mean(-1).sqrt() / y.pow(2).mean(-1).sqrt()
        assert torch.isfinite(x).all() and rel.median().item() < BF16_TOL and rel.max().item() < 4 * BF16_TOL, (r, rel.median(), rel.max())


@pytest.mark.gpu
def test_memory_of_built_keys_and_values():
    """A short portion on a long context of many heads takes no more memory than the other form and EXPAND_BYTES; a layer holds its up-projections
    once, and the two forms read the same tensors."""
    import llm_decoder as ld
    from llm_decoder import hybrid
    R, H, kvr = tiradra_ref, 64, 128
    config = R.make_config([R.latent_layer(heads=H, dim=128, rot_dim=64, vdim=128, kv_rank=kvr)])
    model = ld.HybridDecoder(config, R.random_weights(config, 1), "bfloat16", max_tokens=9216, max_seqs=1)
    mixer, eng = model.layers[0].mixer, ld.Engine(model)
    held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for n, t in vars(mixer).items() if n.startswith("w_u")}
    assert sum(held.values()) == 2 * H * 128 * kvr * 2 and mixer.tc_tokens
    for _ in range(8):
        eng.step([(0, [1] * 1024, [])])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    eng.step([(0, [1] * 64, [])])
    most = hybrid.EXPAND_BYTES + 3 * 2 * 64 * H * (kvr + 192 + 128) * 2 + (16 << 20)
    assert torch.cuda.max_memory_allocated() - before < most, (torch.cuda.max_memory_allocated() - before, most)


@pytest.mark.gpu
def test_a_refused_plan_is_not_asked_again():
    """Pages of 8 tokens: the tcgen05 kernel does not serve them.  The portions of later steps run once, on the kernel that does, and give
    what pages of 16 give (2e-2 of the logits' spread: bfloat16 sums in another order)."""
    import llm_decoder as ld
    from oracle import tiradra_ref as R
    config = R.make_config([R.attention_layer(heads=4, kv_heads=2, dim=64, vdim=128)])
    W = R.random_weights(config, 2)
    engines = [ld.Engine(ld.HybridDecoder(config, W, "bfloat16", max_tokens=512, max_seqs=2, tile_size=t)) for t in (8, 16)]
    for step in ([(0, 40)], [(0, 1), (1, 130)], [(0, 30), (1, 1)], [(0, 1), (1, 17)]):
        entries = [(r, [(7 * k + r) % 71 for k in range(n)], [n - 1]) for r, n in step]
        x, y = (e.step(entries) for e in engines)
        assert (x - y).abs().max() < 2e-2 * y.abs().max()
    eight, sixteen = (e.model.layers[0].mixer.core for e in engines)
    assert eight.tc_plans == [] and eight.mma_tokens and len(sixteen.tc_plans) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("kv_rank,tokens", [(64, 256), (128, 128), (256, 64)])
def test_small_ranks_build_keys_for_long_portions_only(monkeypatch, kv_rank, tokens):
    """A portion one token short of the line stays on the other form; both sides agree with the oracle."""
    import llm_decoder as ld
    from llm_decoder import hybrid
    R = tiradra_ref
    config = R.make_config([R.latent_layer(heads=2, dim=64, rot_dim=16, vdim=64, kv_rank=kv_rank)])
    W = R.random_weights(config, 3)
    eng, built, real = ld.Engine(ld.HybridDecoder(config, W, "bfloat16", max_tokens=1024, max_seqs=2)), [], hybrid.LatentAttentionMixer._attend_expanded
    monkeypatch.setattr(hybrid.LatentAttentionMixer, "_attend_expanded", lambda self, *a: (built.append(1), real(self, *a))[1])
    rnd = random.Random(kv_rank)
    for r, n in ((0, tokens - 1), (1, tokens)):
        toks = [rnd.randrange(config["vocab"]) for _ in range(n)]
        x, y = eng.step([(r, toks, list(range(n)))]).double().cpu(), R.forward(config, W, toks)
        assert ((x - y).pow(2).mean(-1).sqrt() / y.pow(2).mean(-1).sqrt()).median().item() < BF16_TOL
        assert len(built) == r
