"""The argmax of a step rides on the lm_head stage of the single-launch kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,factors,B", [(torch.bfloat16, "dense", 1), (torch.bfloat16, "dense", 3), (torch.float32, "dense", 4),
                                             (torch.bfloat16, "int4", 7)])
def test_the_step_takes_the_first_of_equal_maxima(dtype, factors, B):
    """Every logit row has its maximum twice (the head's rows repeat, in tiles of 16 of several CTAs), the
    vocabulary is no multiple of 16, a NaN never wins."""
    from flashsvd_b200 import synthetic

    shape = synthetic.ModelShape(d=256, H=4, Hk=2, Dh=64, I=256, Rq=64, Rk=32, Rv=32, Ro=64, Rg=64, Ru=64, Rd=64, vocab=4003,
                                 n_layers=1)
    eng = synthetic.make_engine(shape, device=torch.device("cuda:0"), dtype=dtype, batch=B, ctx=9, max_new=8, factors=factors)
    eng.lm_head[2000:4000] = eng.lm_head[:2000]
    for poison in (False, True):
        if poison:
            eng.lm_head[5] = float("nan")
        for _ in range(2):
            eng.step(1)
        torch.cuda.synchronize()
        logits = eng.logits.cpu()
        assert bool(logits[:, 5].isnan().all()) == poison
        assert eng.tokens.cpu().tolist() == torch.nan_to_num(logits, nan=-1e30).numpy().argmax(axis=1).tolist()
