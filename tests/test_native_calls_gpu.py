"""GPU: calls of `flash_attn_func` that the native front (csrc/torch_calls.cc) has to leave to the autograd function in
Python, or has to take as it does."""
import threading
import time

import pytest
import torch

from tests._cases import BWD_TOL, FWD_TOL, alibi_slopes, make_qkv

pytestmark = pytest.mark.gpu


def _qkv(seed=31, grad=False, seqlen=200, dtype=torch.bfloat16):
    return [t.cuda().requires_grad_(grad) for t in make_qkv(seed, 2, 4, 2, seqlen, seqlen, 64, dtype)]


@pytest.mark.parametrize("grad", [False, True], ids=["plain", "grad"])
def test_traced_call_follows_its_inputs(grad):
    """A traced call is recorded; its output is not a constant of the trace."""
    import flash_attn2_b200 as fa2

    def layer(q, k, v):
        return fa2.flash_attn_func(q, k, v, causal=True) + q

    traced = torch.jit.trace(layer, _qkv(grad=grad), check_trace=False)
    other = _qkv(seed=32, grad=grad)
    assert torch.equal(traced(*other), layer(*other))


@pytest.mark.parametrize("which", ["q", "k", "v", "alibi_slopes"])
@pytest.mark.parametrize("grad", [False, True], ids=["plain", "grad"])
def test_forward_mode_derivatives_are_refused(which, grad):
    """There is no forward-mode formula: an error, not an output without a tangent."""
    import torch.autograd.forward_ad as fwd_ad

    import flash_attn2_b200 as fa2

    args = dict(zip("qkv", _qkv(grad=grad)), alibi_slopes=torch.full((4,), 0.1, device="cuda"))
    with fwd_ad.dual_level():
        args[which] = fwd_ad.make_dual(args[which], torch.ones_like(args[which]))
        with pytest.raises(NotImplementedError, match="jvp"):
            fa2.flash_attn_func(**args, causal=True)


def test_functorch_transforms_are_refused():
    """The autograd function has no rules for them, whichever tensor of the call is transformed."""
    import flash_attn2_b200 as fa2

    q, k, v = _qkv()
    weight = torch.randn(3, device="cuda")
    calls = [lambda: torch.func.vmap(lambda w: fa2.flash_attn_func(q, k, v) * w)(weight),
             lambda: torch.func.vmap(lambda x: fa2.flash_attn_func(x, k, v))(torch.stack([q, q])),
             lambda: torch.func.grad(lambda w: (fa2.flash_attn_func(q, k, v).float() * w).sum())(weight[0]),
             lambda: torch.func.jvp(lambda x: fa2.flash_attn_func(x, k, v), (q,), (q,))]
    for call in calls:
        with pytest.raises(RuntimeError, match="setup_context"):
            call()


def test_slopes_that_require_grad_keep_the_graph():
    """The slopes get no gradient, but the output belongs to the graph as for any other differentiable input."""
    import flash_attn2_b200 as fa2

    q, k, v = _qkv()
    slopes = torch.full((4,), 0.1, device="cuda", requires_grad=True)
    out = fa2.flash_attn_func(q, k, v, causal=True, alibi_slopes=slopes)
    assert out.requires_grad
    out.sum().backward()
    assert slopes.grad is None


def _through_hooks(unpack):
    """Gradients of a call whose saved tensors come back through `unpack`, and of the call without hooks."""
    import flash_attn2_b200 as fa2

    q, k, v = _qkv(grad=True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().clone(), unpack):
        out = fa2.flash_attn_func(q, k, v, causal=True, deterministic=True)
    want = torch.autograd.grad(fa2.flash_attn_func(q, k, v, causal=True, deterministic=True), (q, k, v), torch.ones_like(out))
    return torch.autograd.grad(out, (q, k, v), torch.ones_like(out)), want


def _odd_offset(t):
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return buf[1:].view(t.shape).copy_(t)


def _odd_stride(t):
    buf = torch.empty(*t.shape[:-1], t.shape[-1] + 1, dtype=t.dtype, device=t.device)
    return buf[..., :t.shape[-1]].copy_(t)


@pytest.mark.parametrize("layout", [_odd_offset, _odd_stride], ids=["offset", "stride"])
def test_saved_tensors_may_come_back_in_another_layout(layout):
    got, want = _through_hooks(lambda t: layout(t) if t.dim() == 4 else t)
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.mark.parametrize("rank,change", [(4, torch.Tensor.cpu), (4, torch.Tensor.float), (4, lambda t: t[:, 1:]),
                                         (3, torch.Tensor.cpu), (3, torch.Tensor.half), (3, lambda t: t[:, 1:])],
                         ids=["cpu", "type", "shape", "lse-cpu", "lse-type", "lse-shape"])
def test_saved_tensors_that_do_not_match_are_refused(rank, change):
    """An error before any launch."""
    with pytest.raises(RuntimeError):
        _through_hooks(lambda t: change(t) if t.dim() == rank else t)


@pytest.mark.parametrize("window", [[5, 3], (5, 3, 9)], ids=["list", "longer"])
def test_window_forms(window):
    """Any sequence: its first two elements count. An iterator serves a call that falls back to Python as well."""
    import flash_attn2_b200 as fa2

    q, k, v = _qkv()
    want = fa2.flash_attn_func(q, k, v, window_size=(5, 3))
    assert torch.equal(fa2.flash_attn_func(q, k, v, window_size=window), want)
    assert torch.equal(fa2.flash_attn_func(_odd_offset(q), k, v, window_size=iter(window)), want)


@pytest.mark.parametrize("call", ["fwd", "bwd", "attention", "attention-grad"])
def test_other_threads_run_while_a_call_waits(call):
    """The GPU is busy and the launch queue full, so the calls block; a thread that wants to run every millisecond can."""
    import flash_attn2_b200 as fa2

    q, k, v = _qkv(seqlen=64, grad=call == "attention-grad")
    out, lse = (t.detach() for t in fa2.fwd(q, k, v)[:2])
    calls = {"fwd": lambda: fa2.fwd(q, k, v), "bwd": lambda: fa2.bwd(out, q, k, v, out, lse)}
    once = calls.get(call, lambda: fa2.flash_attn_func(q, k, v))
    once()
    torch.cuda.synchronize()
    gaps, done = [], threading.Event()

    def ticks():
        last = time.perf_counter()
        while not done.wait(0.001):
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    ticker = threading.Thread(target=ticks)
    ticker.start()
    torch.cuda._sleep(1_000_000_000)  # half a second
    start = time.perf_counter()
    for _ in range(1500):
        once()
    blocked = time.perf_counter() - start
    done.set()
    ticker.join()
    torch.cuda.synchronize()
    assert blocked > 0.2, "the queue never filled: nothing was tested"
    assert max(gaps) < 0.1


# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim), options of flash_attn_func
GRADIENTS = [
    ((2, 4, 2, 150, 150, 64), dict()),
    ((2, 4, 2, 150, 220, 64), dict(causal=True, softmax_scale=0.2)),
    ((1, 4, 4, 300, 300, 128), dict(causal=True, softcap=15.0)),
    ((1, 4, 2, 260, 300, 96), dict(window_size=(70, 30))),
    ((2, 4, 4, 200, 200, 64), dict(causal=True, window_size=(50, 0), deterministic=True)),
    ((2, 4, 2, 130, 190, 128), dict(causal=True, alibi="heads")),
    ((2, 4, 2, 130, 190, 64), dict(alibi="batch", softcap=20.0)),
    ((2, 4, 2, 130, 190, 64), dict(causal=True, alibi="batch", deterministic=True)),
    ((1, 4, 2, 200, 200, 192), dict(causal=True, softcap=30.0, softmax_scale=0.1)),
    ((1, 4, 2, 150, 200, 256), dict(alibi="heads", window_size=(100, -1))),
    ((1, 4, 1, 1, 300, 128), dict(causal=True)),                      # one query sees every key
    ((1, 4, 1, 1, 300, 128), dict(causal=True, alibi="heads")),       # ... and with slopes its position matters
]


@pytest.mark.parametrize("shape,opt", GRADIENTS, ids=[f"{s}-{'-'.join(o)}" for s, o in GRADIENTS])
@pytest.mark.parametrize("upstream", ["plain", "strided", "expanded"])
def test_gradients_follow_every_option(shape, opt, upstream):
    """Output and gradients of `flash_attn_func` against the CPU oracle; q, k and v may be views of one projection, the
    gradient that arrives may be laid out in any way."""
    import flash_attn2_b200 as fa2
    from oracle.attention_oracle import attention_backward, attention_forward

    b, h, hk, sq, sk, d = shape
    opt, dtype = dict(opt), torch.bfloat16
    q, k, v, do = make_qkv(35, b, h, hk, sq, sk, d, dtype, with_do=True)
    if h == hk and sq == sk:
        fused = torch.stack([q, k, v], 2).cuda()
        qc, kc, vc = (t.detach().requires_grad_() for t in fused.unbind(2))
        assert not qc.is_contiguous()
    else:
        qc, kc, vc = (t.cuda().requires_grad_() for t in (q, k, v))
    slopes, which = None, opt.pop("alibi", None)
    if which:
        slopes = alibi_slopes(h) if which == "heads" else torch.stack([alibi_slopes(h) * (1 + i) for i in range(b)])
    if upstream == "expanded":
        do = do[:, :1, :, :1].expand(b, sq, h, d)
        arrives = do[:, :1, :, :1].cuda().expand(b, sq, h, d)
    else:
        arrives = do.cuda() if upstream == "plain" else do.transpose(1, 2).contiguous().cuda().transpose(1, 2)
    out = fa2.flash_attn_func(qc, kc, vc, alibi_slopes=None if slopes is None else slopes.cuda(), **opt)
    grads = torch.autograd.grad(out, (qc, kc, vc), arrives)
    left, right = opt.pop("window_size", (-1, -1))
    opt.pop("deterministic", None)
    if sq == 1 and slopes is None:
        opt["causal"] = False
    ref = dict(opt, alibi_slopes=slopes, window_left=left, window_right=right)
    o_ref, lse_ref = attention_forward(q, k, v, **ref)
    torch.testing.assert_close(out.detach().float().cpu(), o_ref, atol=FWD_TOL[dtype]["atol"], rtol=FWD_TOL[dtype]["rtol"])
    want = attention_backward(q, k, v, do.contiguous(), out=out.detach().float().cpu(), lse=lse_ref, **ref)
    for name, g, r in zip(("dq", "dk", "dv"), grads, want):
        torch.testing.assert_close(g.float().cpu(), r, msg=lambda m, n=name: f"{n}: {m}", **BWD_TOL[dtype])
    assert fa2.cabi_ops.device_status() == 0


@pytest.mark.parametrize("opt", [dict(), dict(is_causal=True, softcap=15.0), dict(window_size_left=60, window_size_right=10, softmax_scale=0.2)],
                         ids=["plain", "softcap", "window"])
def test_native_and_operator_route_agree(opt):
    """A supplied output takes the operator library: the same bits, on a side stream and from another thread as well."""
    import flash_attn2_b200 as fa2

    q, k, v = _qkv()
    dout = torch.ones_like(q)
    out = torch.empty_like(q)
    want = fa2.fwd(q, k, v, out=out, **opt)
    want_grads = fa2.bwd(dout, q, k, v, want[0], want[1], dk=torch.empty_like(k), **opt)
    got = []

    def call():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            o, l = fa2.fwd(q, k, v, **opt)[:2]
            got.append((o, l, fa2.bwd(dout, q, k, v, o, l, **opt)))
        stream.synchronize()

    torch.cuda.synchronize()
    call()
    threads = [threading.Thread(target=call) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 3
    for o, l, grads in got:
        assert torch.equal(o, want[0]) and torch.equal(l, want[1])
        assert torch.equal(grads[1], want_grads[1]) and torch.equal(grads[2], want_grads[2]) and torch.equal(grads[3], want_grads[3])
        torch.testing.assert_close(grads[0], want_grads[0], atol=2e-2, rtol=2e-2)  # fp32 adds land in arrival order


class _LittleMemory:
    """Within it the allocator has nothing left but pieces of these sizes."""

    def __init__(self, *spare):
        self.spare = spare

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
        keep, self.held = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in self.spare], []
        for size in (1 << 21, 1 << 18, 1 << 12, 1 << 9):
            try:
                while True:
                    self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        del keep

    def __exit__(self, *exc):
        self.held.clear()
        torch.cuda.set_per_process_memory_fraction(1.0)


@pytest.mark.parametrize("shape", [(1, 32, 8, 1, 8192), (1, 4, 4, 200, 8192)], ids=["few-rows", "shared-tiles"])
@pytest.mark.parametrize("route", ["native", "operator"])
def test_forward_without_room_for_scratch(shape, route):
    """A call whose outputs fit runs; the scratch memory is for speed."""
    import flash_attn2_b200 as fa2

    b, h, hk, sq, sk = shape
    q, k, v = [t.cuda() for t in make_qkv(33, b, h, hk, sq, sk, 128, torch.bfloat16)]
    out = torch.empty_like(q)
    call = (lambda: fa2.fwd(q, k, v)) if route == "native" else (lambda: fa2.fwd(q, k, v, out=out))
    want = [t.clone() for t in call()[:2]]
    with _LittleMemory(1 << 20):
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(3 << 20, dtype=torch.uint8, device="cuda")
        got = call()[:2]
        torch.cuda.synchronize()
    torch.testing.assert_close(got[0], want[0], atol=1e-2, rtol=1e-2)
    torch.testing.assert_close(got[1], want[1], atol=1e-4, rtol=1e-4)


def test_backward_without_room_for_parts():
    """The accumulator of dQ fits, the parts of shared key blocks do not."""
    import flash_attn2_b200 as fa2

    q, k, v, do = [t.cuda() for t in make_qkv(34, 1, 1, 1, 4200, 2048, 128, torch.bfloat16, with_do=True)]
    out, lse = fa2.fwd(q, k, v)[:2]
    want = [t.clone() for t in fa2.bwd(do, q, k, v, out, lse)]
    # dK, dV and delta take the small pieces, dQ 1.1 MB, the accumulator 2.2 MB; the parts would take 16 MB.
    with _LittleMemory(1 << 19, 1 << 19, 1 << 19, 2 << 20, 5 << 20):
        got = fa2.bwd(do, q, k, v, out, lse)
        torch.cuda.synchronize()
    for g, w in zip(got, want):
        torch.testing.assert_close(g, w, atol=2e-2, rtol=2e-2)
