"""GPU: the forward at head dims above 128 with a soft cap or a bias, where two threads share a row of scores, against the CPU oracle."""
import pytest
import torch

from tests._cases import FWD_TOL, alibi_slopes, make_qkv

pytestmark = pytest.mark.gpu

# (seqlen_q, seqlen_k): keys for the first thread of a row only, for both, one past a tile of 64; rows that see no key.
SIZES = [(70, 1), (65, 32), (70, 33), (129, 64), (200, 97), (130, 257), (300, 100)]
OPTIONS = {"softcap": dict(softcap=20.0), "alibi": dict(alibi=True), "both": dict(softcap=20.0, alibi=True), "negative": dict(softmax_scale=-0.07)}


@pytest.mark.parametrize("option", OPTIONS)
@pytest.mark.parametrize("head_dim,causal,window,dtype", [(136, True, -1, torch.bfloat16), (192, False, 40, torch.float16),
                                                          (256, True, -1, torch.float16), (256, False, -1, torch.bfloat16)])
def test_shared_rows(head_dim, causal, window, dtype, option):
    from flash_attn2_b200 import cabi_ops as ops
    from oracle.attention_oracle import attention_forward

    for n, (sq, sk) in enumerate(SIZES):
        opt = dict(OPTIONS[option], causal=causal, window_left=window)
        if opt.pop("alibi", False):
            opt["alibi_slopes"] = alibi_slopes(4)
        q, k, v = make_qkv(20 + n, 2, 4, 2, sq, sk, head_dim, dtype)
        # later keys are longer, so the row maximum grows by more than the threshold of the rescale, now in one half, now in the other
        k *= torch.linspace(0.2, 4.0, sk).to(dtype)[None, :, None, None]
        want, want_lse = attention_forward(q.float(), k.float(), v.float(), **opt)
        if "alibi_slopes" in opt:
            opt["alibi_slopes"] = opt["alibi_slopes"].cuda()
        out, lse = ops.fwd(q.cuda(), k.cuda(), v.cuda(), **opt)
        tol = FWD_TOL[dtype]
        # the hardware's tanh is good to 2^-11, so a capped score, and the logarithm of its weight, to 20 * 2^-11 = 0.01: two of them make
        # a relative 0.02 of a weight, of values that are below 5
        extra = 0.1 if "softcap" in opt else 0.0
        out, lse = out.float().cpu(), lse.cpu()
        empty = torch.isposinf(want_lse)
        assert (torch.isposinf(lse) == empty).all() and (out.transpose(1, 2)[empty] == 0).all()
        torch.testing.assert_close(out, want, atol=tol["atol"] + extra, rtol=tol["rtol"])
        torch.testing.assert_close(lse[~empty], want_lse[~empty], atol=tol["lse"], rtol=0)
    assert ops.device_status() == 0
