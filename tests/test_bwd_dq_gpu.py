"""GPU parity of the dQ-only backward call (dense, head dims up to 128) against the CPU oracle: tile edges, ragged
lengths, masks, score transforms, head groups, rows without keys; and the same bits from every run."""
import pytest
import torch

from tests._cases import BWD_TOL, alibi_slopes, make_qkv

pytestmark = pytest.mark.gpu

# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim), options
CASES = [
    ((1, 1, 1, 1, 1, 8), {}),
    ((2, 4, 2, 128, 128, 128), dict(causal=True)),
    ((1, 4, 1, 129, 127, 64), {}),
    ((1, 4, 4, 777, 777, 128), dict(causal=True)),
    ((1, 2, 2, 100, 1409, 96), dict(causal=True)),
    ((1, 2, 2, 640, 200, 128), dict(causal=True)),                      # rows without keys
    ((1, 4, 2, 500, 900, 64), dict(window_left=130, window_right=70)),
    ((1, 2, 1, 300, 300, 128), dict(causal=True, softcap=15.0)),
    ((1, 4, 2, 300, 420, 64), dict(causal=True, alibi=True)),
    ((1, 4, 2, 300, 420, 128), dict(alibi=True)),
    ((1, 2, 2, 260, 260, 128), dict(causal=True, softcap=20.0, alibi=True)),
]


@pytest.mark.parametrize("shape,opt", CASES, ids=[str(c[0]) for c in CASES])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
def test_dq_alone(shape, opt, dtype):
    from flash_attn2_b200 import cabi_ops as ops
    from oracle.attention_oracle import attention_backward

    b, h, hk, sq, sk, d = shape
    opt = dict(opt)
    q, k, v, do = make_qkv(11, b, h, hk, sq, sk, d, dtype, with_do=True)
    slopes = alibi_slopes(h) if opt.pop("alibi", False) else None
    gpu = dict(alibi_slopes=None if slopes is None else slopes.cuda(), **opt)
    qc, kc, vc, doc = q.cuda(), k.cuda(), v.cuda(), do.cuda()
    out, lse = ops.fwd(qc, kc, vc, **gpu)
    delta = ops.bwd_preprocess(doc, out)
    dq = ops.bwd(qc, kc, vc, doc, lse, delta, which=1, **gpu)[0]
    assert ops.device_status() == 0
    ref = attention_backward(q, k, v, do, out=out.float().cpu(), lse=lse.cpu(), alibi_slopes=slopes, **opt)[0]
    torch.testing.assert_close(dq.float().cpu(), ref, **BWD_TOL[dtype])
    for _ in range(2):
        assert torch.equal(ops.bwd(qc, kc, vc, doc, lse, delta, which=1, **gpu)[0], dq)


# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim), options: key blocks whose walk several CTAs share
SPLIT_CASES = [
    ((1, 4, 1, 777, 777, 128), dict(causal=True)),
    ((1, 1, 1, 2000, 130, 64), {}),
    ((2, 8, 2, 513, 513, 96), dict(causal=True, window_left=200)),
    ((1, 2, 2, 1025, 1000, 128), {}),
    ((1, 8, 1, 300, 1100, 64), dict(causal=True, softcap=20.0)),
]


@pytest.mark.parametrize("shape,opt", SPLIT_CASES, ids=[str(c[0]) for c in SPLIT_CASES])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("deterministic", [False, True], ids=["all", "pair"])
def test_split_key_blocks(shape, opt, dtype, deterministic):
    """Through `bwd`, whose first launch computes delta and clears the accumulator as well."""
    import flash_attn2_b200 as fa2
    from oracle.attention_oracle import attention_backward

    b, h, hk, sq, sk, d = shape
    q, k, v, do = make_qkv(12, b, h, hk, sq, sk, d, dtype, with_do=True)
    qc, kc, vc, doc = q.cuda(), k.cuda(), v.cuda(), do.cuda()
    args = dict(is_causal=opt.get("causal", False), window_size_left=opt.get("window_left", -1), softcap=opt.get("softcap", 0.0))
    out, lse = fa2.fwd(qc, kc, vc, **args)[:2]
    got = fa2.bwd(doc, qc, kc, vc, out, lse, deterministic=deterministic, **args)
    ref = attention_backward(q, k, v, do, out=out.float().cpu(), lse=lse.cpu(), **opt)
    for name, g, r in zip(("dq", "dk", "dv"), got, ref):
        torch.testing.assert_close(g.float().cpu(), r, msg=lambda m, n=name: f"{n}: {m}", **BWD_TOL[dtype])
    torch.testing.assert_close(got[3].cpu(), ref[3], atol=2e-5, rtol=1e-5)
    again = fa2.bwd(doc, qc, kc, vc, out, lse, deterministic=deterministic, **args)
    assert torch.equal(again[1], got[1]) and torch.equal(again[2], got[2])
    assert fa2.cabi_ops.device_status() == 0


@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_packed_dq_alone_is_ordered(causal, head_dim):
    """A packed dQ-only call adds the key blocks' contributions in a fixed order when the workspace holds the turn counters:
    the same bits from every run, empty and ragged sequences and head groups included."""
    from flash_attn2_b200 import cabi_ops as ops
    from oracle.attention_oracle import varlen_backward

    lengths = [300, 1, 0, 641, 128, 77]
    g = torch.Generator().manual_seed(13)
    total, cu = sum(lengths), torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32)
    q, do = (torch.randn(total, 4, head_dim, generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(total, 2, head_dim, generator=g).bfloat16() for _ in range(2))
    qc, kc, vc, doc, cc = (t.cuda() for t in (q, k, v, do, cu))
    out, lse = ops.varlen_fwd(qc, kc, vc, cc, cc, 641, 641, causal=causal)
    delta = ops.bwd_preprocess(doc, out, cu_seqlens_q=cc, max_seqlen_q=641)
    runs = [ops.bwd(qc, kc, vc, doc, lse, delta, which=1, causal=causal, cu_seqlens_q=cc, cu_seqlens_k=cc, max_seqlen_q=641,
                    max_seqlen_k=641)[0] for _ in range(4)]
    assert ops.device_status() == 0
    ref = varlen_backward(q, k, v, do, cu, cu, out=out.float().cpu(), lse=lse.cpu(), causal=causal)[0]
    torch.testing.assert_close(runs[0].float().cpu(), ref, **BWD_TOL[torch.bfloat16])
    for again in runs[1:]:
        assert torch.equal(again, runs[0])
