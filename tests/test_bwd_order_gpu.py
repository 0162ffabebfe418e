"""GPU: the order of the backward's CTAs (heads listed in groups, the last one smaller) does not change what a head gets."""
import pytest
import torch

from tests._cases import make_qkv

pytestmark = pytest.mark.gpu

# (heads, heads_k, seqlen, head_dim), causal: enough CTAs and data for several groups, a prime number of (batch, kv head) pairs
CASES = [((43, 43, 4096, 64), True), ((43, 43, 1024, 64), False), ((26, 13, 4000, 128), True), ((14, 7, 4096, 192), True)]


@pytest.mark.parametrize("shape,causal", CASES, ids=[str(c[0]) for c in CASES])
def test_a_head_gets_the_same_in_any_group(shape, causal):
    from flash_attn2_b200 import cabi_ops as ops

    h, hk, s, d = shape
    q, k, v, do = [t.cuda() for t in make_qkv(5, 1, h, hk, s, s, d, torch.bfloat16, with_do=True)]
    out, lse = ops.fwd(q, k, v, causal=causal)
    delta = ops.bwd_preprocess(do, out)
    _, dk, dv = ops.bwd(q, k, v, do, lse, delta, causal=causal)
    dq = ops.bwd(q, k, v, do, lse, delta, causal=causal, which=1)[0] if d <= 128 else None
    g = h // hk
    for head in {0, hk // 2, hk - 2, hk - 1}:
        mine, own = slice(head * g, head * g + g), slice(head, head + 1)
        args = (q[:, :, mine], k[:, :, own], v[:, :, own], do[:, :, mine], lse[:, mine].contiguous(), delta[:, mine].contiguous())
        alone = ops.bwd(*args, causal=causal)
        assert torch.equal(alone[1], dk[:, :, own]) and torch.equal(alone[2], dv[:, :, own])
        if dq is not None:
            assert torch.equal(ops.bwd(*args, causal=causal, which=1)[0], dq[:, :, mine])
    assert ops.device_status() == 0


@pytest.mark.parametrize("shape", [(2, 16, 4, 777, 128), (1, 8, 2, 1500, 64), (3, 4, 4, 130, 96)], ids=str)
def test_dkdv_beside_dq(shape):
    """The second call of a bit-reproducible backward runs beside the first one's last CTAs; what follows on the stream
    (here the next pair, into the same memory, and a copy) waits for both."""
    import flash_attn2_b200 as fa2
    from flash_attn2_b200 import cabi_ops as ops

    b, h, hk, s, d = shape
    q, k, v, do = [t.cuda() for t in make_qkv(6, b, h, hk, s, s, d, torch.bfloat16, with_do=True)]
    out, lse = fa2.fwd(q, k, v, is_causal=True)[:2]
    delta = ops.bwd_preprocess(do, out)
    dq = ops.bwd(q, k, v, do, lse, delta, causal=True, which=1)[0]
    _, dk, dv = ops.bwd(q, k, v, do, lse, delta, causal=True, which=2, share_key_blocks=True)
    for _ in range(20):
        copies = [t.clone() for t in fa2.bwd(do, q, k, v, out, lse, is_causal=True, deterministic=True)[:3]]
    assert all(torch.equal(a, r) for a, r in zip(copies, (dq, dk, dv)))
    assert ops.device_status() == 0
