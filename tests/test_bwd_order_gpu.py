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


# (heads, heads_k, seqlen_q, seqlen_k, head_dim), options: more than two CTAs per SM, so that CTAs take over tiles of others
TAKE_OVER = [((60, 60, 100, 1000, 64), dict(causal=True, window_left=300)),   # key blocks that no row sees, among the others
             ((60, 60, 100, 1000, 40), dict(causal=True, window_left=300)),   # rows of 80 bytes
             ((240, 240, 130, 200, 56), {}), ((700, 350, 5, 3, 64), {}), ((300, 75, 129, 129, 64), dict(causal=True, softcap=15.0))]


@pytest.mark.parametrize("shape,opt", TAKE_OVER, ids=[str(c[0]) for c in TAKE_OVER])
def test_tiles_taken_over_from_other_ctas(shape, opt):
    from flash_attn2_b200 import cabi_ops as ops

    h, hk, sq, sk, d = shape
    q, k, v, do = [t.cuda() for t in make_qkv(7, 1, h, hk, sq, sk, d, torch.bfloat16, with_do=True)]
    out, lse = ops.fwd(q, k, v, **opt)
    delta = ops.bwd_preprocess(do, out)
    dq, dk, dv = ops.bwd(q, k, v, do, lse, delta, **opt)
    assert ops.device_status() == 0
    torch.testing.assert_close(dq, ops.bwd(q, k, v, do, lse, delta, which=1, **opt)[0], atol=2e-2, rtol=2e-2)
    g, few = h // hk, 5
    for first in range(0, hk - few, max(1, hk // 7)):   # a few heads at a time: one wave
        mine, own = slice(first * g, (first + few) * g), slice(first, first + few)
        alone = ops.bwd(q[:, :, mine], k[:, :, own], v[:, :, own], do[:, :, mine], lse[:, mine].contiguous(),
                        delta[:, mine].contiguous(), **opt)
        assert torch.equal(alone[1], dk[:, :, own]) and torch.equal(alone[2], dv[:, :, own])
    assert ops.device_status() == 0
