"""GPU: the order of the backward's CTAs (heads listed in groups, the last one smaller) does not change what a head gets."""
import pytest
import torch

from tests._cases import alibi_slopes, make_qkv

pytestmark = pytest.mark.gpu

# (heads, heads_k, seqlen, head_dim), causal: several groups of several heads and a smaller last one in the kernel for head dim 64,
# 128 and 192 and (the last shape) in the one for dQ alone; all heads in one group. test_plans_cpu.py states which is which.
SEVERAL = [((43, 43, 4096, 64), True), ((43, 43, 1024, 64), False), ((13, 13, 1024, 128), False), ((43, 43, 1024, 192), True),
           ((105, 35, 4096, 128), True)]
CASES = SEVERAL + [((26, 13, 4000, 128), True), ((14, 7, 4096, 192), True)]


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
def test_bit_reproducible_pair_on_changing_inputs(shape):
    """Calls without a pause, into the same memory: every one sees the delta and the inputs of its own pass."""
    import flash_attn2_b200 as fa2
    from flash_attn2_b200 import cabi_ops as ops

    b, h, hk, s, d = shape
    sets, want = [], []
    for seed in (6, 7, 8):
        q, k, v, do = [t.cuda() for t in make_qkv(seed, b, h, hk, s, s, d, torch.bfloat16, with_do=True)]
        do *= 2.0 ** (seed - 7)
        out, lse = fa2.fwd(q, k, v, is_causal=True)[:2]
        delta = ops.bwd_preprocess(do, out)
        torch.cuda.synchronize()
        dq = ops.bwd(q, k, v, do, lse, delta, causal=True, which=1)[0]
        torch.cuda.synchronize()
        sets.append((do, q, k, v, out, lse))
        want.append((dq, *ops.bwd(q, k, v, do, lse, delta, causal=True, which=2, share_key_blocks=True)[1:]))
        torch.cuda.synchronize()
    args = [torch.empty_like(t) for t in sets[0]]
    got = []
    for i in range(30):
        for a, t in zip(args, sets[i % 3]):
            a.copy_(t)
        got.append([t.clone() for t in fa2.bwd(*args, is_causal=True, deterministic=True)[:3]])
    for i, grads in enumerate(got):
        assert all(torch.equal(g, w) for g, w in zip(grads, want[i % 3])), i
    assert ops.device_status() == 0


def test_threads_that_share_a_stream():
    """Bit-reproducible backward calls of one thread among forward calls of another, all on the default stream: what a call
    frees on its return, the other thread's next call gets, scratch memory included."""
    import threading

    import flash_attn2_b200 as fa2
    from flash_attn2_b200 import cabi_ops as ops

    q, k, v, do = [t.cuda() for t in make_qkv(9, 2, 16, 4, 777, 777, 128, torch.bfloat16, with_do=True)]
    out, lse = fa2.fwd(q, k, v, is_causal=True)[:2]
    token = [t.cuda() for t in make_qkv(10, 1, 32, 8, 1, 8192, 128, torch.bfloat16)]
    few = [t.cuda() for t in make_qkv(11, 1, 8, 8, 500, 4096, 128, torch.bfloat16)]   # both forwards take scratch memory
    calls = {"backward": lambda: fa2.bwd(do, q, k, v, out, lse, is_causal=True, deterministic=True)[:3],
             "decode": lambda: fa2.fwd(*token)[:2], "shared tiles": lambda: fa2.fwd(*few, is_causal=True)[:2]}
    want = {}
    for name, call in calls.items():
        want[name] = [t.clone() for t in call()]
        torch.cuda.synchronize()
    wrong, errors = {name: torch.zeros((), dtype=torch.int64, device="cuda") for name in calls}, []
    torch.cuda.synchronize()
    start = threading.Barrier(3)

    def work(name):
        try:
            start.wait(30)
            for _ in range(100):
                for g, w in zip(calls[name](), want[name]):
                    wrong[name] += (g != w).sum()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(name,)) for name in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert {name: int(n) for name, n in wrong.items()} == dict.fromkeys(calls, 0)
    assert ops.device_status() == 0


# (heads, heads_k, seqlen_q, seqlen_k, head_dim), options: more than two CTAs per SM, so that CTAs take over tiles of others, but
# for the last one, which is just below that
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


# More iterations a tile (5, 8, 15), so that stages and phases carry on from one tile to the next in every position; each score
# transform; both types. (heads, heads_k, seqlen_q, seqlen_k, head_dim), type, ALiBi, options
FORMS = [((180, 60, 600, 600, 64), torch.bfloat16, False, dict(causal=True)), ((800, 200, 129, 129, 64), torch.bfloat16, False, dict(causal=True, softcap=15.0)),
         ((62, 62, 600, 600, 64), torch.float16, True, dict(causal=True)), ((62, 62, 600, 600, 64), torch.bfloat16, True, {}),
         ((130, 65, 520, 600, 48), torch.float16, True, dict(causal=True, softcap=20.0))]


@pytest.mark.parametrize("shape,dtype,alibi,opt", FORMS, ids=[f"{c[0]}-{c[1]}" for c in FORMS])
def test_every_form_of_tiles_taken_over(shape, dtype, alibi, opt):
    import flash_attn2_b200 as fa2
    from flash_attn2_b200 import cabi_ops as ops

    h, hk, sq, sk, d = shape
    assert hk * -(-sk // 128) > 2 * torch.cuda.get_device_properties(0).multi_processor_count
    q, k, v, do = [t.cuda() for t in make_qkv(8, 1, h, hk, sq, sk, d, dtype, with_do=True)]
    slopes = alibi_slopes(h).cuda() if alibi else None
    out, lse = ops.fwd(q, k, v, alibi_slopes=slopes, **opt)
    delta = ops.bwd_preprocess(do, out)
    dq, dk, dv = ops.bwd(q, k, v, do, lse, delta, alibi_slopes=slopes, **opt)
    g, few = h // hk, 5
    for first in range(0, hk - few, max(1, hk // 5)):   # a few heads at a time: one wave
        mine, own = slice(first * g, (first + few) * g), slice(first, first + few)
        alone = ops.bwd(q[:, :, mine], k[:, :, own], v[:, :, own], do[:, :, mine], lse[:, mine].contiguous(),
                        delta[:, mine].contiguous(), alibi_slopes=None if slopes is None else slopes[mine].contiguous(), **opt)
        assert torch.equal(alone[1], dk[:, :, own]) and torch.equal(alone[2], dv[:, :, own])
    # dK and dV without dQ, and the bit-reproducible pair
    only = ops.bwd(q, k, v, do, lse, delta, which=2, alibi_slopes=slopes, **opt)
    assert torch.equal(only[1], dk) and torch.equal(only[2], dv)
    dq_alone = ops.bwd(q, k, v, do, lse, delta, which=1, alibi_slopes=slopes, **opt)[0]
    pair = fa2.bwd(do, q, k, v, out, lse, alibi_slopes=slopes, is_causal=opt.get("causal", False), softcap=opt.get("softcap", 0.0),
                   deterministic=True)
    assert all(torch.equal(a, b) for a, b in zip(pair, (dq_alone, dk, dv)))
    torch.testing.assert_close(dq, dq_alone, atol=2e-2, rtol=2e-2)
    assert ops.device_status() == 0
