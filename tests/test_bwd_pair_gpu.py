"""GPU: the backward on pairs of CTAs against the kernels with one CTA per key block, which other tests check against the oracle."""
import pytest
import torch

from tests._cases import make_qkv

pytestmark = pytest.mark.gpu

# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim, causal, window): calls that run on pairs (test_plans_cpu.py states that they
# do). Whole tiles; a last pair of one key block, of one key, with nothing for its second CTA; bottom-right masks with more
# keys than queries and with rows that see no key; windows; grouped heads; head dims below the kernel's; pairs whose keys no query sees
# (EMPTY).
CASES = [(1, 28, 28, 2048, 2048, 128, False, (-1, -1)), (4, 32, 8, 2000, 1000, 128, False, (-1, -1)), (2, 16, 8, 2048, 1810, 120, False, (-1, -1)),
         (2, 16, 8, 1921, 1793, 104, False, (-1, -1)), (2, 16, 8, 4200, 4200, 128, True, (-1, -1)), (2, 8, 8, 4100, 5000, 128, True, (-1, -1)),
         (2, 8, 8, 5000, 4100, 112, True, (-1, -1)), (2, 8, 4, 5000, 5000, 128, False, (3000, 500)),
         (1, 8, 8, 4100, 4900, 128, False, (500, -1))]


# Head dims 192 and 256: one query, one key block and a bit, a last pair with keys for one CTA only or too few for its first; masks as
# above; score transforms.
WIDE = [(1, 2, 2, 128, 128, 256, False, (-1, -1)), (2, 4, 2, 1, 300, 256, False, (-1, -1)), (3, 4, 4, 193, 65, 256, False, (-1, -1)),
        (2, 4, 2, 577, 385, 256, False, (-1, -1)), (2, 8, 2, 777, 777, 256, True, (-1, -1)), (2, 4, 4, 300, 1021, 256, True, (-1, -1)),
        (2, 4, 4, 700, 200, 256, True, (-1, -1)), (2, 4, 4, 1000, 1100, 256, False, (100, 50)), (1, 4, 4, 1024, 1024, 256, True, (127, 0)),
        (1, 2, 2, 128, 128, 192, False, (-1, -1)), (3, 4, 4, 200, 65, 192, False, (-1, -1)), (2, 8, 2, 777, 777, 192, True, (-1, -1)),
        (2, 4, 4, 333, 1021, 192, True, (-1, -1)), (2, 4, 4, 1000, 1100, 192, False, (100, 50)),
        (2, 4, 2, 128, 2000, 256, True, (127, 0)), (2, 4, 4, 200, 1021, 192, False, (100, 50))]
# The cases with pairs that walk no query block: their dK and dV are zeros, and no MMA is issued.
EMPTY = [c for c in CASES + WIDE if c[7][0] >= 0 and c[4] > c[3] + c[7][0]]


def _check(args, causal, window, dtype, **opt):
    from flash_attn2_b200 import cabi_ops as ops

    q, k, v, do = args
    opt.update(causal=causal, window_left=window[0], window_right=window[1])
    out, lse = ops.fwd(q, k, v, **opt)
    delta = ops.bwd_preprocess(do, out)
    dq, dk, dv = ops.bwd(q, k, v, do, lse, delta, **opt)
    want_dq = ops.bwd(q, k, v, do, lse, delta, which=1, **opt)[0]
    _, want_dk, want_dv = ops.bwd(q, k, v, do, lse, delta, which=2, **opt)
    # Every value of dK and dV is the same sum in the same order; keys and rows that see nothing add exact zeros.
    assert torch.equal(dk, want_dk) and torch.equal(dv, want_dv)
    # dQ is summed in fp32 in another order: what lies within a few 1e-6 of a rounding boundary moves by a unit of the type (2^-8,
    # 2^-11). That is at most one value in a hundred, so a 2-norm of at most a tenth of the unit.
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert (dq.double() - want_dq.double()).norm() <= 0.1 * unit * want_dq.double().norm()
    assert ops.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(i) for i in c[:6]))
def test_pairs_give_what_single_ctas_give(case, dtype):
    b, h, hk, sq, sk, d, causal, window = case
    _check([t.cuda() for t in make_qkv(11, b, h, hk, sq, sk, d, dtype, with_do=True)], causal, window, dtype)


def test_pairs_on_views_of_one_projection():
    b, h, s, d = 2, 16, 2048, 128
    gen = torch.Generator().manual_seed(12)
    qkv = torch.randn(b, s, 3, h, d, generator=gen).to(torch.bfloat16).cuda()
    do = torch.randn(b, s, h, d, generator=gen).to(torch.bfloat16).cuda()
    _check([*qkv.unbind(2), do], False, (-1, -1), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("case", WIDE, ids=lambda c: "x".join(str(i) for i in c[:6]))
def test_wide_pairs_give_what_single_ctas_give(case, dtype):
    b, h, hk, sq, sk, d, causal, window = case
    _check([t.cuda() for t in make_qkv(13, b, h, hk, sq, sk, d, dtype, with_do=True)], causal, window, dtype)


@pytest.mark.parametrize("opt", [dict(softcap=20.0), dict(alibi=True), dict(softcap=20.0, alibi=True)], ids=lambda o: "-".join(o))
@pytest.mark.parametrize("head_dim,causal", [(192, True), (256, False), (256, True)])
def test_wide_pairs_with_score_transforms(head_dim, causal, opt):
    from tests._cases import alibi_slopes

    opt = dict(opt)
    if opt.pop("alibi", False):
        opt["alibi_slopes"] = alibi_slopes(8).cuda()
    _check([t.cuda() for t in make_qkv(14, 2, 8, 4, 500, 450, head_dim, torch.bfloat16, with_do=True)], causal, (-1, -1), torch.bfloat16, **opt)


def test_wide_pairs_on_views_of_one_projection():
    gen = torch.Generator().manual_seed(15)
    qkv = torch.randn(2, 300, 3, 4, 256, generator=gen).to(torch.bfloat16).cuda()
    do = torch.randn(2, 300, 4, 256, generator=gen).to(torch.bfloat16).cuda()
    _check([*qkv.unbind(2), do], True, (-1, -1), torch.bfloat16)


# One call on each kernel, many pairs of unequal walks.
REPEATED = [(1, 28, 28, 2048, 2048, 128, False, (-1, -1)), (2, 16, 16, 4200, 4200, 128, True, (-1, -1)), (4, 8, 4, 777, 777, 192, True, (-1, -1)),
            (4, 8, 4, 777, 777, 256, True, (-1, -1))]


@pytest.mark.parametrize("case", REPEATED, ids=lambda c: "x".join(str(i) for i in c[:6]))
def test_pairs_give_the_same_bits_every_time(case):
    """What one CTA tells the other by an arrival alone is there when it is read: three inputs in turn, so that what an earlier call left
    in shared or tensor memory is not what belongs there, several hundred times without a pause."""
    from flash_attn2_b200 import cabi_ops as ops

    b, h, hk, sq, sk, d, causal, _ = case
    calls, want = [], []
    for seed in (31, 32, 33):
        q, k, v, do = [t.cuda() for t in make_qkv(seed, b, h, hk, sq, sk, d, torch.bfloat16, with_do=True)]
        out, lse = ops.fwd(q, k, v, causal=causal)
        calls.append((q, k, v, do, lse, ops.bwd_preprocess(do, out)))
        want.append(ops.bwd(*calls[-1], causal=causal, which=2)[1:])
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(300):
        for g, w in zip(ops.bwd(*calls[i % 3], causal=causal)[1:], want[i % 3]):
            wrong += (g != w).any()
    assert wrong.item() == 0
    assert ops.device_status() == 0


@pytest.mark.parametrize("case", [(8, 16, 16, 2048, 250, 128), (2, 4, 4, 400, 380, 192), (2, 4, 4, 300, 200, 256)], ids=lambda c: "x".join(map(str, c)))
def test_pairs_take_any_layout(case):
    """Transposed, padded, strided and expanded tensors against copies of them."""
    from flash_attn2_b200 import cabi_ops as ops

    b, h, hk, sq, sk, d = case
    gen = torch.Generator(device="cuda").manual_seed(16)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)

    def rows(s, how):
        return {"bhsd": lambda: rand(b, h, s, d).transpose(1, 2), "sbhd": lambda: rand(s, b, h, d).transpose(0, 1),
                "padded": lambda: rand(b, s, h, d + 24)[..., 8:8 + d], "strided": lambda: rand(b, 2 * s, 2 * h, d)[:, ::2, 1::2],
                "one head": lambda: rand(b, s, 1, d).expand(b, s, h, d), "one batch": lambda: rand(1, s, h, d).expand(b, s, h, d)}[how]()

    for how in (("bhsd", "sbhd", "padded", "strided"), ("strided", "one head", "one head", "bhsd"), ("sbhd", "one batch", "padded", "one head"),
                ("one batch", "bhsd", "one batch", "padded")):
        q, k, v, do = [rows(s, x) for s, x in zip((sq, sk, sk, sq), how)]
        out, lse = ops.fwd(q, k, v)
        delta = ops.bwd_preprocess(do, out)
        got = ops.bwd(q, k, v, do, lse, delta)
        want = ops.bwd(*[t.contiguous() for t in (q, k, v, do)], lse, delta)
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
        # dQ: as in _check
        assert (got[0].double() - want[0].double()).norm() <= 0.1 * 2.0 ** -8 * want[0].double().norm()
    assert ops.device_status() == 0


@pytest.mark.parametrize("case,key,first_row", [((2, 16, 16, 4200, 4200, 128), 2300, 2048), ((1, 2, 2, 700, 700, 192), 300, 256),
                                                ((1, 2, 2, 700, 700, 256), 300, 256)], ids=str)
def test_how_far_a_key_that_is_not_finite_reaches(case, key, first_row):
    """Into dQ of the query blocks that its pair walks, which under a causal mask start at the pair's first key; no further."""
    from flash_attn2_b200 import cabi_ops as ops

    q, k, v, do = [t.cuda() for t in make_qkv(17, *case, torch.bfloat16, with_do=True)]
    k[:, key] = float("inf")
    out, lse = ops.fwd(q, k, v, causal=True)
    assert out[:, :key].isfinite().all()
    dq = ops.bwd(q, k, v, do, lse, ops.bwd_preprocess(do, out), causal=True)[0]
    assert dq[:, :first_row].isfinite().all() and not dq[:, key:].isfinite().any()
    assert ops.device_status() == 0
