"""GPU parity of the forward whose work tiles are shared between CTAs (few 256-row tiles for the GPU) against the CPU
oracle: shares that end inside a tile, tiles in many parts, ragged ends, stages without keys, masks, score transforms."""
import ctypes

import pytest
import torch

from tests._cases import alibi_slopes, make_qkv
from tests.test_fwd_gpu import _check
from tests.test_plans_cpu import SMS, _fwd_args, plans  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu

# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim), options
CASES = [
    ((1, 2, 2, 65, 4001, 128), dict(causal=True)),          # one stage only, a tile in many parts
    ((1, 2, 2, 300, 2000, 128), dict(causal=True)),         # the second tile has one stage
    ((1, 4, 1, 257, 1111, 64), {}),                         # one row in the second tile, GQA
    ((2, 2, 2, 1000, 1000, 128), dict(causal=True)),        # tiles of different lengths
    ((2, 2, 2, 130, 3000, 72), dict(causal=True, window_left=700)),
    ((1, 3, 3, 900, 2100, 128), dict(window_left=300, window_right=250)),
    ((1, 2, 2, 300, 1200, 128), dict(window_left=600, window_right=0)),
    ((1, 2, 2, 1100, 1024, 64), dict(causal=True)),         # rows without keys
    ((1, 4, 2, 100, 3000, 128), dict(causal=True, softcap=20.0)),
    ((1, 4, 2, 100, 3000, 64), dict(alibi=True)),
    ((1, 4, 2, 100, 3000, 96), dict(causal=True, softcap=15.0, alibi=True)),
    ((1, 2, 2, 200, 3000, 128), dict(softmax_scale=-0.1)),
    ((3, 37, 37, 70, 1300, 64), {}),                        # 111 tiles: nearly every CTA owns parts of two
]


@pytest.mark.parametrize("shape,opt", CASES, ids=[str(c[0]) for c in CASES])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
def test_shared_tiles(shape, opt, dtype):
    from flash_attn2_b200 import cabi_ops as ops
    from oracle.attention_oracle import attention_forward

    b, h, hk, sq, sk, d = shape
    opt = dict(opt)
    q, k, v = make_qkv(7, b, h, hk, sq, sk, d, dtype)
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
    # Parts are summed in the order of the keys.
    again = ops.fwd(q.cuda(), kc, vc, **gpu)
    assert torch.equal(again[0], out) and torch.equal(again[1], lse)


# Shapes whose tiles are shared: windows, causal tiles of different lengths, a stage without keys beside one with keys, and
# a grid in which nearly every CTA owns parts of two tiles.
ROUTED = [
    ((2, 2, 2, 1000, 3000, 128), dict(causal=True)),
    ((2, 2, 2, 130, 6000, 72), dict(causal=True, window_left=3000)),
    ((1, 3, 3, 900, 4200, 128), dict(window_left=1500, window_right=1250)),
    ((1, 2, 2, 300, 4000, 128), dict(window_left=2200, window_right=0)),
    ((1, 1, 1, 2300, 2124, 128), dict(causal=True)),
    ((1, 2, 2, 1300, 1124, 64), dict(causal=True)),
    ((2, 40, 40, 150, 3000, 64), dict(causal=True, softcap=20.0)),
]


@pytest.mark.parametrize("shape,opt", ROUTED, ids=[str(c[0]) for c in ROUTED])
def test_routed_shapes(shape, opt, plans):
    """The plan shares the tiles; then the comparison above."""
    args = _fwd_args(*shape, **{k: int(v) for k, v in opt.items() if k in ("causal", "window_left", "window_right")})
    assert plans.shared_tiles(ctypes.byref(args), SMS) > 0
    test_shared_tiles(shape, opt, torch.bfloat16)


def test_captured_call_replays():
    """The merge is launched while the forward runs, in a captured graph as well."""
    import flash_attn2_b200 as fa2

    q, k, v = (t.cuda() for t in make_qkv(8, 1, 4, 4, 300, 3000, 128, torch.bfloat16))
    want = fa2.fwd(q, k, v, is_causal=True)[:2]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = fa2.fwd(q, k, v, is_causal=True)[:2]
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
