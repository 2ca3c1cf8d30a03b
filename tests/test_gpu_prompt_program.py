"""The prompt program (all positions of all sequences as rows of dense tensor-core GEMMs) against the
oracle's token-by-token loop: several sequences, a prompt in two parts, and row counts, ranks and widths
on both sides of the tile edges (128 rows, 64 factor rows of a box, 64-wide k-blocks).

Tolerance: the bf16 per-layer bound 2e-2 (rel_linf) over two layers and the head."""
import pytest
import torch

from oracle import lowrank_llama as O

pytestmark = pytest.mark.gpu

RAGGED = O.Shape(d=264, H=4, Hk=2, Dh=64, I=520, Rq=88, Rk=40, Rv=56, Ro=72, Rg=104, Ru=104, Rd=80, vocab=203, n_layers=2)
WIDE_HEADS = O.Shape(d=512, H=8, Hk=1, Dh=128, I=1096, Rq=136, Rk=64, Rv=64, Ro=128, Rg=200, Ru=200, Rd=192, vocab=300, n_layers=2)


def rel_linf(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return float((a - b).abs().max() / b.abs().max().clamp_min(1e-30))


@pytest.mark.parametrize("shape,B,parts", [(RAGGED, 3, (2,)), (RAGGED, 3, (43, 86)), (RAGGED, 1, (128, 1)), (RAGGED, 2, (65, 64)),
                                           (WIDE_HEADS, 5, (26, 3)), (O.TINY, 9, (29,)), (WIDE_HEADS, 1, (257,))])
def test_prompts_in_parts_match_oracle(shape, B, parts):
    from flashsvd_b200 import engine, packing

    dev, dtype, L = torch.device("cuda:0"), torch.bfloat16, sum(parts)
    w = O.make_model_weights(shape, seed=3, dtype=dtype)
    prompt = torch.randint(0, shape.vocab, (B, L), generator=torch.Generator().manual_seed(L))
    toks_ref, logits_ref, st = O.greedy_decode(shape, w, prompt, 1, S_max=L + 4)
    eng = engine.DecodeEngine(layers=[packing.pack_layer(lw, device=dev, dtype=dtype) for lw in w["layers"]],
                              embed=w["embed"].to(dev), final_norm=w["norm"].to(dev), lm_head=w["lm_head"].to(dev),
                              num_heads=shape.H, num_kv_heads=shape.Hk, head_dim=shape.Dh, batch_size=B,
                              max_cache_len=L + 4, rope_theta=shape.theta, eps=shape.eps, max_steps=L + 8)
    t0 = 0
    for n in parts:
        eng.prefill(prompt[:, t0:t0 + n])
        t0 += n
    torch.cuda.synchronize()
    assert eng.status() == 0
    assert eng.seqlens.tolist() == [L] * B
    assert torch.equal(eng.last_tokens(1)[0], eng.tokens)
    assert rel_linf(eng.logits, logits_ref[0]) <= 4e-2
    for li in range(shape.n_layers):
        assert rel_linf(eng.key_cache[li][:, :L], st.k[li][:, :L]) <= 4e-2
        assert rel_linf(eng.value_cache[li][:, :L], st.v[li][:, :L]) <= 4e-2
    with pytest.raises((IndexError, ValueError)):
        eng.prefill(prompt[:, :2].repeat(1, 5))    # past the end of the cache: refused before a launch
    assert eng.status() == 0
    eng.close()
