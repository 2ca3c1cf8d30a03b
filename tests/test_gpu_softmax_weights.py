"""Softmax weights keep their 24 bits where they meet the value rows (in a long prompt of one sequence: the
last 16 rows').

Three keys have weight, p = exp(-x), 1 and 1, and their value rows cancel to 16 bits: v2 = bf16(-p v1),
v3 = bf16(-p v1 - v2), so that the output (p v1 + v2 + v3) / (2 + p) is about 2^-17 p v1, with |v1| in [256, 512).
Tolerance: half a unit in the last place of the bf16 output, plus 2^-21 |p v1| for p itself (expf / exp2f within 2 units
of 2^-24, two roundings of a score below 1), plus 4 2^-15 for the sum (the accumulator and three products below 512,
each cut at 24 bits of the largest).  x is chosen so that two bf16 numbers miss p by more than 2^-18.5."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _two_terms(p):
    hi = p.to(torch.bfloat16).float()
    return hi.double() + (p - hi).to(torch.bfloat16).double()


def _case(qn, Dh, seed):
    """Dimension 0 of the first key (the query's is qn), and the three value rows [3, Dh] with the output in 64
    bits and its tolerance."""
    keys = -torch.arange(3, 30, dtype=torch.float64) / 64
    p = torch.exp(keys * qn / math.sqrt(Dh))
    miss = ((_two_terms(p.float()) - p) / p).abs()
    i = int(miss.argmax())
    assert float(miss[i]) > 2.0 ** -18.5
    key, p = float(keys[i]), float(p[i])
    gen = torch.Generator().manual_seed(seed)
    v1 = (256 * (1 + torch.rand(Dh, generator=gen)) * (1 - 2 * torch.randint(0, 2, (Dh,), generator=gen))).to(torch.bfloat16)
    v2 = (-p * v1.double()).to(torch.bfloat16)
    v3 = (-(p * v1.double() + v2.double())).to(torch.bfloat16)
    ref = (p * v1.double() + v2.double() + v3.double()) / (2 + p)
    half_ulp = 2.0 ** (torch.floor(torch.log2(ref.abs())) - 8)
    return key, torch.stack([v1, v2, v3]), ref, half_ulp + 2.0 ** -21 * p * v1.double().abs() + 4 * 2.0 ** -15


@pytest.mark.parametrize("B", [5, 9, 70])
@pytest.mark.parametrize("H,Hk,Dh", [(4, 4, 64), (4, 2, 64), (8, 2, 128), (8, 1, 128)])
def test_prompt_rows(H, Hk, Dh, B):
    """`decode_layer` over B consecutive positions of one sequence (its attention is the prompt pass's).  Factors of
    zeros and ones make the layer's output the attention itself: the query is 16 or 32 in dimension 0, the rows' own keys score
    below -1000, their values and the MLP are 0."""
    from flashsvd_b200 import ops

    dev, dtype = torch.device("cuda:0"), torch.bfloat16
    HD, KD, ctx, S_max = H * Dh, Hk * Dh, 3, 80
    d, qn = HD, math.isqrt(HD)               # qn: the normalised one-hot row, 16 or 32
    key, values, ref, tol = _case(qn, Dh, H + B)
    zeros = lambda *s: torch.zeros(*s, dtype=dtype, device=dev)
    qkv_v, q_u, k_u = zeros(24, d), zeros(HD, 8), zeros(KD, 8)
    qkv_v[0, d - 1] = qkv_v[8, d - 1] = 1.0
    q_u[::Dh, 0] = 1.0
    k_u[::Dh, 0] = -64.0
    ones, eye = torch.ones(d, dtype=dtype, device=dev), torch.eye(HD, dtype=dtype, device=dev)
    pk = {"ln1_w": ones, "qkv_v": qkv_v, "q_u": q_u, "k_u": k_u, "v_u": zeros(KD, 8), "o_v": eye, "o_u": eye.clone(), "ln2_w": ones,
          "upgate_v": zeros(16, d), "gate_u": zeros(64, 8), "up_u": zeros(64, 8), "down_v": zeros(8, 64), "down_u": zeros(d, 8),
          "k_cache": zeros(1, S_max, Hk, Dh), "v_cache": zeros(1, S_max, Hk, Dh)}
    pk["k_cache"][0, 0, :, 0] = key
    pk["v_cache"][0, :3] = values.to(dev)[:, None]
    dims = ops.make_dims(dtype=dtype, B=B, d=d, H=H, Hk=Hk, Dh=Dh, I=64, Rq=8, Rk=8, Rv=8, Ro=HD, Rg=8, Ru=8, Rd=8, S_max=S_max,
                         eps=1e-30, rows_are_positions=1)
    ws = ops.make_workspace(dims, dev)
    xin = zeros(B, d)
    xin[:, d - 1] = 2.0 ** -20
    out = zeros(B, d)
    seq = torch.arange(ctx, ctx + B, dtype=torch.int32, device=dev)
    cos, sin = torch.ones(S_max, Dh // 2, dtype=dtype, device=dev), zeros(S_max, Dh // 2)
    run = lambda: ops.decode_layer(dims, ops.make_layer_struct(pk), cos, sin, seq, xin, out, ws)
    run()
    assert ws.status() == 0
    assert bool((pk["k_cache"][0, ctx:ctx + B, :, 0] == -64.0 * qn).all())
    got = out.double().cpu()[-16:].view(-1, H, Dh)
    n = Dh - 1                               # (the last dimension of the last head holds the residual)
    assert bool(((got - ref).abs() <= tol)[..., :n].all())
    # An infinite value at a later position (in dimensions 7 and 8) is nothing to the rows before it, whatever tile they
    # share.  Their values: tolerance as above where the weights have 24 bits, else 2^-8 of |p v1| more.
    qkv_v[16, d - 2] = 1.0
    pk["v_u"][7::Dh, 0], pk["v_u"][8::Dh, 0] = 3e38, -3e38
    for bad in (B - 2, B // 2):
        xin[:] = 0.0
        xin[:, d - 1] = 2.0 ** -20
        xin[bad, d - 1], xin[bad, d - 2] = 0.0, 2.0 ** -20
        run()
        assert bool(pk["v_cache"][0, ctx + bad, :, 7:9].isinf().all())
        got = out.double().cpu()[:bad].view(-1, H, Dh)
        wide = torch.full((bad, 1, 1), 2.0 ** -8).double()
        wide[max(0, B - 16):] = 0.0
        assert bool(((got - ref).abs() <= tol + wide * 512)[..., :n].all())
        assert not bool(out[bad:].view(-1, H, Dh)[..., 7].isfinite().any())


@pytest.mark.parametrize("n", [3, 70, 1200])
@pytest.mark.parametrize("H,Hk,Dh", [(4, 4, 64), (4, 2, 64), (4, 1, 64), (8, 2, 128), (8, 1, 128)])
def test_flash_decode(H, Hk, Dh, n):
    """The op, in one split and in several: the three keys are the last ones, all others score below -1000."""
    from flashsvd_b200 import ops

    dev, dtype, qn = torch.device("cuda:0"), torch.bfloat16, 16
    key, values, ref, tol = _case(qn, Dh, H + n)
    q = torch.zeros(1, H, Dh, dtype=dtype, device=dev)
    q[..., 0] = qn
    k, v = (torch.zeros(1, n, Hk, Dh, dtype=dtype, device=dev) for _ in range(2))
    k[:, :-3, :, 0] = -64.0 * qn
    k[:, -3, :, 0] = key
    v[:, :-3] = 1.0
    v[0, -3:] = values.to(dev)[:, None]
    ws = ops.make_workspace(ops.make_dims(dtype=dtype, B=1, H=H, Hk=Hk, Dh=Dh, S_max=n), dev)
    out = ops.flash_decode(q, k, v, torch.tensor([n], dtype=torch.int32, device=dev), ws)
    assert bool(((out[0].double().cpu() - ref).abs() <= tol).all())
