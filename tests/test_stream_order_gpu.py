"""GPU: kernels that start beside the end of the one before them see what it wrote: chains of calls without a pause, each on what
the one before returned, against the same chain with a synchronisation after every call; and training steps in a graph."""
import pytest
import torch

from tests._cases import make_qkv

pytestmark = pytest.mark.gpu


def _inputs(seed, b, h, hk, sq, sk, d, dtype=torch.bfloat16):
    return [t.cuda() for t in make_qkv(seed, b, h, hk, sq, sk, d, dtype, with_do=True)]


def _forwards(seed, shape, causal):
    """The output of a call is the query of the next one."""
    import flash_attn2_b200 as fa2

    x, k, v, _ = _inputs(seed, *shape)
    caches = [(k, v), (v, k), (k.flip(1), v)]

    def chain(pause):
        q, got = x, []
        for i in range(9):
            q, lse = fa2.fwd(q, *caches[i % 3], is_causal=causal)[:2]
            got += [q, lse]
            pause()
        return got

    return chain


def _steps(seed, shape, causal, deterministic):
    """dK and dV of a step are K and V of the next one, its output the next dO."""
    import flash_attn2_b200 as fa2

    q, k0, v0, do0 = _inputs(seed, *shape)

    def chain(pause):
        k, v, do, got = k0, v0, do0, []
        for _ in range(5):
            out, lse = fa2.fwd(q, k, v, is_causal=causal)[:2]
            pause()
            dq, k, v = fa2.bwd(do, q, k, v, out, lse, is_causal=causal, deterministic=deterministic)[:3]
            pause()
            do = out
            got += [out, lse, k, v] + ([dq] if deterministic else [])
        return got

    return chain


# (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim): few rows with parts, in whole units, and with more units than SMs; one tile;
# shared tiles and their merge; many tiles; the wide kernel
FORWARDS = [((1, 32, 8, 1, 8192, 128), True), ((10, 32, 8, 1, 1500, 64), True), ((40, 8, 4, 2, 700, 192), False),
            ((1, 4, 4, 128, 128, 64), False), ((1, 8, 8, 500, 4096, 128), True), ((4, 16, 8, 700, 700, 128), True),
            ((2, 8, 4, 500, 900, 256), True)]
# Steps on pairs of CTAs (test_plans_cpu.py states that they are).
PAIRS = [((1, 28, 28, 2048, 2048, 128), False, False), ((2, 8, 4, 400, 400, 192), True, False), ((2, 8, 4, 300, 300, 256), True, False)]
# shared key blocks; few CTAs; tiles taken over; the wide kernel with one CTA per key block and half of the head dim; bit-reproducible pairs
STEPS = PAIRS + [((1, 8, 2, 777, 777, 128), True, False), ((4, 16, 16, 400, 400, 128), False, False), ((8, 16, 16, 509, 509, 64), True, False),
         ((2, 8, 4, 300, 300, 192), True, False), ((2, 16, 4, 777, 777, 128), True, True), ((10, 16, 16, 300, 300, 64), False, True)]
CHAINS = [(_forwards, c) for c in FORWARDS] + [(_steps, c) for c in STEPS]


@pytest.mark.parametrize("make,case", CHAINS, ids=[f"{m.__name__[1:]}-{c[0]}" for m, c in CHAINS])
def test_a_call_sees_what_the_one_before_it_wrote(make, case):
    from flash_attn2_b200 import cabi_ops as ops

    chains = [make(seed, *case) for seed in (21, 22, 23)]
    want = []
    for chain in chains:
        torch.cuda.synchronize()
        want.append(chain(torch.cuda.synchronize))
    # Other data in the same memory each time: what a chain returns is freed before the one after it.
    for i in range(9):
        got = chains[i % 3](lambda: None)
        assert all(torch.equal(g, w) for g, w in zip(got, want[i % 3])), i
        del got
    assert ops.device_status() == 0


# (shape, causal, deterministic)
GRAPHS = PAIRS[:2] + [((2, 16, 4, 777, 777, 128), True, True), ((8, 16, 16, 509, 509, 64), False, False), ((2, 16, 16, 1000, 1000, 128), True, False),
          ((2, 8, 4, 600, 600, 256), True, False)]


@pytest.mark.parametrize("shape,causal,deterministic", GRAPHS, ids=str)
def test_captured_training_step(shape, causal, deterministic):
    """In a graph the early launches are programmatic edges: replays on changing inputs give what the calls gave."""
    import flash_attn2_b200 as fa2
    from flash_attn2_b200 import cabi_ops as ops

    sets = [_inputs(seed, *shape) for seed in (31, 32, 33)]
    q, k, v = [t.clone().requires_grad_() for t in sets[0][:3]]
    do = sets[0][3].clone()

    def step():
        out = fa2.flash_attn_func(q, k, v, causal=causal, deterministic=deterministic)
        return [out.detach(), *torch.autograd.grad(out, (q, k, v), do)]

    def load(s):
        with torch.no_grad():
            for t, x in zip((q, k, v, do), s):
                t.copy_(x)

    want, side = [], torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for s in sets:
            load(s)
            want.append(step())
            side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = step()
        results = []
        for i in range(9):
            load(sets[i % 3])
            graph.replay()
            results.append([t.clone() for t in got])
        side.synchronize()
    for i, r in enumerate(results):
        out, dq, dk, dv = want[i % 3]
        assert torch.equal(r[0], out) and torch.equal(r[2], dk) and torch.equal(r[3], dv), i
        if deterministic:
            assert torch.equal(r[1], dq), i
        else:  # summed in fp32 in the order of arrival: good to 1e-5 for a few blocks of magnitude 1, which can move the bf16
            # result by one unit in the last place, at most 2^-7 of the value
            torch.testing.assert_close(r[1].float(), dq.float(), rtol=2.0 ** -7, atol=1e-4)
    assert ops.device_status() == 0
