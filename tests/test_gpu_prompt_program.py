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


def _engine(shape, w, B, S_max, **over):
    from flashsvd_b200 import engine, packing

    dev, dtype = torch.device("cuda:0"), w["embed"].dtype
    return engine.DecodeEngine(layers=[packing.pack_layer(lw, device=dev, dtype=dtype) for lw in w["layers"]],
                               embed=w["embed"].to(dev), final_norm=w["norm"].to(dev), lm_head=w["lm_head"].to(dev),
                               num_heads=shape.H, num_kv_heads=shape.Hk, head_dim=shape.Dh, batch_size=B, max_cache_len=S_max,
                               rope_theta=shape.theta, eps=shape.eps, max_steps=S_max + 4, **over)


def _state(eng):
    return [t.clone() for t in (eng.logits, eng.tokens, eng.seqlens, *eng.key_cache, *eng.value_cache)]


def rel_linf(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return float((a - b).abs().max() / b.abs().max().clamp_min(1e-30))


@pytest.mark.parametrize("shape,B,parts", [(RAGGED, 3, (2,)), (RAGGED, 3, (43, 86)), (RAGGED, 1, (128, 1)), (RAGGED, 2, (65, 64)),
                                           (WIDE_HEADS, 5, (26, 3)), (O.TINY, 9, (29,)), (WIDE_HEADS, 1, (257,))])
def test_prompts_in_parts_match_oracle(shape, B, parts):
    dtype, L = torch.bfloat16, sum(parts)
    w = O.make_model_weights(shape, seed=3, dtype=dtype)
    prompt = torch.randint(0, shape.vocab, (B, L), generator=torch.Generator().manual_seed(L))
    toks_ref, logits_ref, st = O.greedy_decode(shape, w, prompt, 1, S_max=L + 4)
    eng = _engine(shape, w, B, L + 4)
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


@pytest.mark.parametrize("B", [2, 12])
def test_first_prompt_on_a_side_stream(B):
    """The first prompt of an engine (its program and scratch are made by that call, and for 12 sequences the
    decode model just before) on a stream that does not wait for the default stream, which is busy: the same
    values as on an idle device, also after the default stream has run dry."""
    shape, L = RAGGED, 90
    w = O.make_model_weights(shape, seed=5, dtype=torch.bfloat16)
    prompt = torch.randint(0, shape.vocab, (B, L), generator=torch.Generator().manual_seed(B), dtype=torch.int32).cuda()
    ref = _engine(shape, w, B, L + 4)
    ref.prefill(prompt)
    ref.step(2)
    want = _state(ref)
    side = torch.cuda.Stream()
    for busy in (200_000, 2_000_000, 100_000_000):   # clocks
        torch.cuda.synchronize()
        w_dev = dict(w, embed=w["embed"].cuda(), norm=w["norm"].cuda(), lm_head=w["lm_head"].cuda())
        eng = _engine(shape, w_dev, B, L + 4)
        torch.cuda.synchronize()
        torch.cuda._sleep(busy)
        with torch.cuda.stream(side):
            eng.prefill(prompt)
            eng.step(1)
        side.synchronize()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            eng.step(1)
            got = _state(eng)
        side.synchronize()
        assert eng.status() == 0
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        eng.close()
    ref.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_prompt_starts_where_the_device_says(dtype):
    """The caller keeps the view of `seqlens` and writes through it after a prompt: the next prompt of a
    single sequence starts there, and fits or is refused by it."""
    shape, L = O.TINY, 21
    w = O.make_model_weights(shape, seed=6, dtype=dtype)
    first, second = torch.randint(0, shape.vocab, (2, 1, L), generator=torch.Generator().manual_seed(4))
    ref = _engine(shape, w, 1, L + 4)
    ref.prefill(first[:, :13])
    ref.step(2)
    with pytest.raises((IndexError, ValueError)):
        ref.prefill(second)             # 15 + 21 positions, nobody holds a view
    ref.reset()
    for c in (*ref.key_cache, *ref.value_cache):
        c.zero_()
    ref.prefill(second)
    eng = _engine(shape, w, 1, L + 4)
    lens = eng.seqlens
    eng.prefill(first)
    assert lens.tolist() == [L]
    with pytest.raises((IndexError, ValueError)):
        eng.prefill(second)
    lens.zero_()
    eng.prefill(second)                 # the whole cache is free again
    assert lens.tolist() == [L]
    assert all(torch.equal(a, b) for a, b in zip(_state(eng), _state(ref)))
    lens.zero_()
    eng.prefill(second[:, :10])
    lens.fill_(8)
    with pytest.raises((IndexError, ValueError)):
        eng.prefill(first)              # 8 + 21 positions
    assert lens.tolist() == [8] and eng.status() == 0
    eng.close()
    ref.close()


@pytest.mark.parametrize("B", [2, 12])
def test_prompts_in_captured_graphs(B):
    """A prompt captured into a graph replays with the values of a direct call, also after longer prompts have
    gone through the engine in between; an engine's first prompt can be captured too (token by token:
    nothing may be allocated there), where one launch per token can."""
    shape, L = O.TINY_GQA, 40
    w = O.make_model_weights(shape, seed=8, dtype=torch.bfloat16)
    long, prompt = torch.randint(0, shape.vocab, (2, B, 3 * L), generator=torch.Generator().manual_seed(B), dtype=torch.int32).cuda()
    prompt = prompt[:, :L].contiguous()
    ref = _engine(shape, w, B, 3 * L)
    ref.prefill(prompt)
    want = _state(ref)
    eng = _engine(shape, w, B, 3 * L)
    lens = eng.seqlens
    eng.prefill(prompt[:, :5])
    eng.reset()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        eng.prefill(prompt)
    eng.reset()
    eng.prefill(long)
    for c in (*eng.key_cache, *eng.value_cache):
        c.zero_()
    for _ in range(2):
        lens.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert eng.status() == 0
        assert all(torch.equal(a, b) for a, b in zip(_state(eng), want))
    graph.reset()
    eng.close()
    if B == 2:
        first = _engine(shape, w, B, 3 * L)
        tokenwise = _engine(shape, w, B, 3 * L, prefill_chunk=1)
        tokenwise.prefill(prompt)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            first.prefill(prompt)
        graph.replay()
        torch.cuda.synchronize()
        assert first.status() == 0
        assert all(torch.equal(a, b) for a, b in zip(_state(first), _state(tokenwise)))
        graph.reset()
        first.close()
        tokenwise.close()
    ref.close()


@pytest.mark.parametrize("shape,B,L", [(O.TINY, 1, 2049), (O.TINY_GQA, 1, 4100), (O.TINY_GQA, 3, 700), (O.TINY, 128, 17), (O.TINY_GQA, 128, 33)])
def test_prompts_of_several_passes(shape, B, L):
    """More than 2048 rows in one call (a pass that is not the last one, the short last one, keys of an earlier
    pass read by a later one), every sequence at a start of its own with keys and values already there:
    against the same prompt token by token.  Tolerance as above: two orders of addition over two layers and the head."""
    start = [5 + 3 * (b % 4) for b in range(B)]
    S_max = L + 20
    w = O.make_model_weights(shape, seed=9, dtype=torch.bfloat16)
    gen = torch.Generator().manual_seed(L)
    prompt = torch.randint(0, shape.vocab, (B, L), generator=gen, dtype=torch.int32).cuda()
    past = torch.randn(2, shape.n_layers, B, max(start), shape.Hk, shape.Dh, generator=gen).to(torch.bfloat16).cuda()
    engines = []
    for chunk in (None, 1):
        eng = _engine(shape, w, B, S_max, prefill_chunk=chunk)
        for li in range(shape.n_layers):
            eng.key_cache[li][:, :max(start)], eng.value_cache[li][:, :max(start)] = past[0, li], past[1, li]
        eng.seqlens.copy_(torch.tensor(start, dtype=torch.int32))
        before = eng.step_counter.item()
        eng.prefill(prompt)
        torch.cuda.synchronize()
        assert eng.status() == 0
        assert eng.seqlens.tolist() == [s + L for s in start]
        assert eng.step_counter.item() == before + (1 if chunk is None else L)
        assert torch.equal(eng.tokens.long(), eng.logits.argmax(dim=1))
        engines.append(eng)
    one, ref = engines
    assert rel_linf(one.logits, ref.logits) <= 4e-2
    for li in range(shape.n_layers):
        for a, b in ((one.key_cache[li], ref.key_cache[li]), (one.value_cache[li], ref.value_cache[li])):
            assert rel_linf(a, b) <= 4e-2
            for s in range(B):   # nothing outside the prompt's rows is touched
                assert torch.equal(a[s, :start[s]], b[s, :start[s]]) and not bool(a[s, start[s] + L:].any())
    for eng in engines:
        eng.close()


@pytest.mark.parametrize("shape,B,L,at", [(O.TINY, 1, 60, 30), (O.TINY, 1, 60, 55), (O.TINY, 2, 60, 30), (O.TINY_GQA, 6, 60, 30),
                                          (WIDE_HEADS, 3, 20, 9)])
def test_an_infinite_value_stays_at_its_position(shape, B, L, at):
    """One token of sequence 0 has infinite values in the first layer: the rows before it, and the other
    sequences, have the same keys and values in the second layer as without it."""
    dtype = torch.bfloat16
    w = O.make_model_weights(shape, seed=12, dtype=dtype)
    w["embed"][:, 5] = 0.0
    w["embed"][7, 5] = 4.0                      # token 7 alone has this dimension ...
    first = w["layers"][0]
    first["v_v"][0] = 0.0
    first["v_v"][0, 5] = 1.0                    # ... which is rank 0 of the values
    first["v_u"][:, 0] = 3e38
    prompt = torch.randint(8, shape.vocab, (B, L), generator=torch.Generator().manual_seed(B), dtype=torch.int32).cuda()
    bad = prompt.clone()
    bad[0, at] = 7
    states = []
    for ids in (prompt, bad):
        eng = _engine(shape, w, B, L + 4)
        eng.prefill(ids)
        torch.cuda.synchronize()
        assert eng.status() == 0
        states.append([t.clone() for t in (eng.value_cache[0], eng.key_cache[1], eng.value_cache[1])])
        eng.close()
    (v0, *clean), (v0_bad, *got) = states
    assert bool(v0.isfinite().all()) and bool(v0_bad[0, at].isinf().all())
    for a, b in zip(got, clean):
        assert rel_linf(a[0, :at], b[0, :at]) <= 2e-2
        assert torch.equal(a[1:], b[1:])
        assert not bool(a[0, at].isfinite().any())
