"""GPU parity of the forward for few query rows (at most 64 per kv head) against the CPU oracle: edges of the 16-row
and 128-key tiles, shares that end inside a unit, masks, score transforms, every head-dim bucket, cache views."""
import ctypes

import pytest
import torch

from tests._cases import alibi_slopes, make_qkv
from tests.test_fwd_gpu import _check
from tests.test_plans_cpu import SMS, _fwd_args, plans  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu

# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim), options
CASES = [
    ((1, 32, 8, 1, 8192, 128), dict(causal=True)),          # 4 rows, every unit split over many CTAs
    ((3, 8, 1, 2, 1000, 128), dict(causal=True)),           # exactly 16 rows
    ((1, 8, 1, 3, 129, 64), dict(causal=True)),             # 24 rows, one key past a tile
    ((2, 16, 1, 2, 2049, 96), {}),                          # exactly 32 rows
    ((1, 12, 4, 11, 640, 192), dict(causal=True)),          # 33 rows
    ((1, 2, 2, 64, 4100, 256), dict(causal=True)),          # 64 rows, the widest head dim
    ((40, 8, 8, 1, 300, 72), {}),                           # more units than CTAs
    ((2, 4, 2, 5, 5000, 128), dict(causal=True, window_left=700)),
    ((2, 4, 2, 5, 500, 128), dict(window_left=0, window_right=3)),
    ((1, 4, 4, 9, 4, 128), dict(causal=True)),              # rows without keys
    ((1, 4, 4, 1, 1, 8), {}),                               # the smallest
    ((2, 8, 2, 4, 3000, 128), dict(causal=True, softcap=20.0, alibi=True)),
    ((1, 4, 4, 7, 3000, 64), dict(alibi=True, softmax_scale=-0.1)),
]


@pytest.mark.parametrize("shape,opt", CASES, ids=[str(c[0]) for c in CASES])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
def test_few_query_rows(shape, opt, dtype):
    from flash_attn2_b200 import cabi_ops as ops
    from oracle.attention_oracle import attention_forward

    b, h, hk, sq, sk, d = shape
    opt = dict(opt)
    q, k, v = make_qkv(5, b, h, hk, sq, sk, d, dtype)
    slopes = alibi_slopes(h) if opt.pop("alibi", False) else None
    o_ref, lse_ref = attention_forward(q, k, v, alibi_slopes=slopes, **opt)
    # k and v as the filled part of a larger cache whose unused rows must not be read
    cache = [torch.full((b, sk + 77, hk, d), float("nan"), dtype=dtype, device="cuda") for _ in range(2)]
    for c, t in zip(cache, (k, v)):
        c[:, :sk] = t.cuda()
    kc, vc = (c[:, :sk] for c in cache)
    gpu = dict(alibi_slopes=None if slopes is None else slopes.cuda(), **opt)
    out, lse = ops.fwd(q.cuda(), kc, vc, **gpu)
    assert ops.device_status() == 0
    _check(out, lse, o_ref, lse_ref, dtype)
    # The parts of a unit are summed in a fixed order, whichever CTA ends last.
    for _ in range(3):
        again = ops.fwd(q.cuda(), kc, vc, **gpu)
        assert torch.equal(again[0], out) and torch.equal(again[1], lse)


def test_workspace_contents_do_not_matter_and_graph_replays():
    """Flags left over from anything else count as clear, and a captured call can be replayed."""
    import flash_attn2_b200 as fa2

    q, k, v = (t.cuda() for t in make_qkv(6, 1, 16, 4, 1, 5000, 128, torch.bfloat16))
    want = fa2.fwd(q, k, v)[:2]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fa2.fwd(q, k, v)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = fa2.fwd(q, k, v)[:2]
    for _ in range(3):
        got[0].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


# Shapes that the few-row kernel takes, and whether parts of units are shared (units = batch x kv heads).
ROUTED = [
    ((40, 8, 4, 1, 3000, 64), {}, True),                                  # more units than SMs: equal shares of the whole list,
    ((19, 16, 8, 4, 2500, 128), dict(causal=True), True),                 # each ending one unit and starting another
    ((21, 16, 8, 2, 3300, 192), dict(causal=True), True),
    ((20, 8, 8, 1, 2600, 256), dict(softcap=15.0), True),
    ((19, 16, 8, 4, 4000, 128), dict(causal=True, window_left=3000, alibi=True), True),
    ((1, 24, 1, 1, 3000, 128), {}, True),                                 # 17 to 32 rows
    ((1, 4, 4, 17, 5000, 256), dict(causal=True), True),
    ((1, 64, 1, 1, 5000, 64), {}, True),                                  # 33 to 64 rows, every head-dim bucket
    ((2, 64, 8, 8, 4096, 128), dict(causal=True), True),
    ((1, 8, 8, 33, 6000, 192), dict(causal=True, window_left=5000), True),
    ((4, 128, 16, 8, 1030, 256), dict(causal=True), True),
    ((3, 64, 2, 2, 260, 64), dict(causal=True), False),                   # whole units
]


@pytest.mark.parametrize("shape,opt,shared", ROUTED, ids=[str(c[0]) for c in ROUTED])
def test_routed_shapes(shape, opt, shared, plans):
    """The plan is the one that the case is about; then the comparison above."""
    args = ctypes.byref(_fwd_args(*shape, **{k: int(v) for k, v in opt.items() if k in ("causal", "window_left")}))
    assert plans.few_rows(args, SMS) == shape[1] // shape[2] * shape[3]
    assert (plans.few_rows_workspace(args, SMS) > 0) == shared
    test_few_query_rows(shape, opt, torch.bfloat16)


def test_workspace_contents_are_irrelevant():
    """One buffer for calls of different shapes, and after it was filled with anything: the same bits as from a buffer of
    their own."""
    import ctypes as C

    from flash_attn2_b200 import _cabi

    lib = _cabi.load()
    buf = torch.zeros(16 << 20, dtype=torch.uint8, device="cuda")

    def call(shape, prepare):
        b, h, hk, sq, sk, d = shape
        q, k, v = (t.cuda() for t in make_qkv(9, b, h, hk, sq, sk, d, torch.bfloat16))
        out, lse = torch.empty_like(q), torch.empty(b, h, sq, device="cuda")
        a = _fwd_args(*shape, causal=1, q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), lse=lse.data_ptr(),
                      dtype=_cabi.FA2_BF16, softmax_scale=d ** -0.5)
        for name, t in (("q", q), ("k", k), ("v", v), ("o", out)):
            setattr(a, name + "_stride", (C.c_int64 * 3)(*t.stride()[:3]))
        need = lib.fa2_fwd_workspace_bytes(C.byref(a))
        assert 0 < need <= buf.numel()
        prepare(need)
        _cabi.check(lib.fa2_fwd_with_workspace(C.byref(a), buf.data_ptr(), need, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        return out, lse

    shapes = [(1, 16, 4, 1, 5000, 128), (19, 16, 8, 1, 2500, 64), (1, 16, 4, 1, 3000, 128), (1, 2, 2, 200, 3000, 64)]
    want = [call(s, lambda n: buf.zero_()) for s in shapes]
    for prepare in (lambda n: None, lambda n: buf.fill_(0xFF), lambda n: buf[:n].random_(0, 256), lambda n: buf.fill_(1)):
        for s, (out, lse) in zip(shapes, want):
            o, l = call(s, prepare)
            assert torch.equal(o, out) and torch.equal(l, lse)
