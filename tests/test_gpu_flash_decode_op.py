"""`flash_decode` on its own against softmax attention in 64 bits.

Tolerance: the output is one bf16 rounding (8 significant bits: 2^-8 of the value) of sums whose weights are kept to 32 bits,
so 2^-8 |ref| plus 5e-5 of the largest value; weights rounded to bf16 miss it (test_gpu_softmax_weights.py
tells 24 bits from 16).  A cache that does not start on a 16-byte boundary takes the interpreter's stage and must agree too."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, n, scale):
    B, H, Dh = q.shape
    G = H // k.shape[2]
    out = torch.zeros(B, H, Dh, dtype=torch.float64)
    for b in range(B):
        if n[b] == 0:
            continue
        kk = k[b, :n[b]].double().repeat_interleave(G, dim=1)
        vv = v[b, :n[b]].double().repeat_interleave(G, dim=1)
        s = torch.einsum("hd,nhd->hn", q[b].double(), kk) * scale
        out[b] = torch.einsum("hn,nhd->hd", torch.softmax(s, dim=1), vv)
    return out


@pytest.mark.parametrize("B,H,Hk,Dh,S,lens", [
    (1, 1, 1, 64, 1, [1]), (1, 4, 4, 128, 40, [33]), (2, 8, 4, 64, 300, [300, 0]), (3, 8, 4, 128, 517, [1, 516, 257]),
    (2, 8, 2, 64, 1030, [1030, 31]), (1, 16, 2, 128, 4100, [4099]), (8, 8, 1, 128, 129, [129, 128, 127, 65, 64, 33, 32, 1]),
    (8, 32, 32, 128, 260, [260] * 8)])
@pytest.mark.parametrize("offset", [0, 4])
def test_flash_decode_keeps_the_weights_in_32_bits(B, H, Hk, Dh, S, lens, offset):
    from flashsvd_b200 import ops

    dev = torch.device("cuda:0")
    gen = torch.Generator().manual_seed(B * 1000 + S)
    q = (2 * torch.randn(B, H, Dh, generator=gen)).to(torch.bfloat16)
    k, v = (torch.randn(B, S, Hk, Dh, generator=gen).to(torch.bfloat16) for _ in range(2))
    dims = ops.make_dims(dtype=torch.bfloat16, B=B, d=64, H=H, Hk=Hk, Dh=Dh, I=64, Rq=8, Rk=8, Rv=8, Ro=8, Rg=8, Ru=8, Rd=8,
                         S_max=S)
    ws = ops.make_workspace(dims, dev)

    def place(t):   # `offset` elements past an aligned address
        buf = torch.empty(t.numel() + offset, dtype=t.dtype, device=dev)
        out = buf[offset:].view(t.shape)
        out.copy_(t)
        return out

    n = torch.tensor(lens, dtype=torch.int32)
    ref = _reference(q, k, v, lens, Dh ** -0.5)
    bound = ref.abs() * 2.0 ** -8 + 5e-5 * float(v.abs().max())
    for _ in range(2):   # the second call finds the arrival counters as the first one left them
        out = ops.flash_decode(q.to(dev), place(k), place(v), n.to(dev), ws)
        assert bool(((out.double().cpu() - ref).abs() <= bound).all())
    again = ops.flash_decode(q.to(dev), place(k), place(v), (n - 1).to(dev), ws, seqlen_add=1)
    assert torch.equal(again, out)


@pytest.mark.parametrize("H,Hk,Dh", [(4, 4, 64), (4, 2, 128), (4, 1, 64), (8, 1, 128)])
@pytest.mark.parametrize("n", [1, 9, 33, 61, 700])
def test_infinity_in_the_last_value_row(H, Hk, Dh, n):
    """An infinity among the values of the last visible position gives an infinity in that dimension (its weight
    is positive), and nothing else: rows past the end of a split take no part."""
    from flashsvd_b200 import ops

    dev = torch.device("cuda:0")
    gen = torch.Generator().manual_seed(n)
    q = torch.randn(1, H, Dh, generator=gen).to(torch.bfloat16)
    k, v = (torch.randn(1, n, Hk, Dh, generator=gen).to(torch.bfloat16) for _ in range(2))
    v[0, -1, :, 5], v[0, -1, :, Dh - 1] = float("inf"), float("-inf")
    ref = _reference(q, k, v, [n], Dh ** -0.5)
    ws = ops.make_workspace(ops.make_dims(dtype=torch.bfloat16, B=1, H=H, Hk=Hk, Dh=Dh, S_max=n), dev)
    out = ops.flash_decode(q.to(dev), k.to(dev), v.to(dev), torch.tensor([n], dtype=torch.int32, device=dev), ws).double().cpu()
    assert bool((out[..., 5] == float("inf")).all()) and bool((out[..., Dh - 1] == float("-inf")).all())
    rest = [i for i in range(Dh) if i not in (5, Dh - 1)]
    assert bool(((out - ref).abs() <= ref.abs() * 2.0 ** -8 + 5e-5 * 5.0)[..., rest].all())
