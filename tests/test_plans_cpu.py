"""CPU: how a dense call is divided over the GPU (csrc/fa2_plan.h), through a small library around that header."""
import ctypes
import subprocess
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent
SMS = 148

SHIM = r'''
#include <cuda_runtime.h>
#include "fa2_plan.h"
extern "C" {
// 1: a backward call shares key blocks in a workspace at this address; -1: the plan does not share any
int bwd_shares(const fa2_bwd_args* a, int sms, uint64_t address, int64_t short_by) {
  fa2::BwdSplit s;
  fa2::plan_bwd_split(a, true, sms, &s);
  if (s.items_per_head == 0) return -1;
  return s.fits(reinterpret_cast<const void*>(address), 512 + s.bytes() - short_by, 512);
}
// query rows that the few-row kernel takes at a time (0: it does not take the call)
int few_rows(const fa2_fwd_args* a, int sms) { return fa2::decode_plan(a, sms).rows; }
int shared_tiles(const fa2_fwd_args* a, int sms) {  // CTAs that share the call's work tiles, 0: none are shared
  fa2::StreamPlan p;
  fa2::plan_stream(a, sms, &p);
  return p.grid;
}
int few_rows_ctas(const fa2_fwd_args* a, int sms) { return fa2::decode_plan(a, sms).grid; }
// heads whose key blocks (dq_alone: query blocks) a backward call lists together
int head_group(const fa2_bwd_args* a, int dq_alone, int sms) {
  const fa2::Windows w = fa2::normalise_windows(a->window_left, a->window_right, a->causal != 0, a->seqlen_k, false);
  return dq_alone ? fa2::bwd_dq_head_group(a, w) : fa2::bwd_head_group(a, w, sms);
}
int takes_pairs(const fa2_bwd_args* a, int sms) {
  return fa2::bwd_wide_takes_pairs(a) || fa2::bwd_takes_pairs(a, fa2::normalise_windows(a->window_left, a->window_right, a->causal != 0, a->seqlen_k, false), sms);
}
int few_rows_start_early(const fa2_fwd_args* a, int sms) {
  const fa2::DecodePlan d = fa2::decode_plan(a, sms);
  return fa2::decode_starts_early(a, d.tiles, d.grid, sms);
}
int64_t few_rows_workspace(const fa2_fwd_args* a, int sms) { return fa2::decode_plan(a, sms).workspace_bytes; }
}
'''


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("plans")
    (d / "shim.cc").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{ROOT / 'kernels-community-rs_b200' / 'csrc'}",
                    "-I/usr/local/cuda/include", str(d / "shim.cc"), "-o", str(d / "shim.so")], check=True)
    lib = ctypes.CDLL(str(d / "shim.so"))
    lib.few_rows_workspace.restype = ctypes.c_int64
    return lib


def _fwd_args(b, h, hk, sq, sk, d, **kw):
    from flash_attn2_b200 import _cabi

    return _cabi.FwdArgs(**{**dict(batch=b, heads=h, heads_k=hk, seqlen_q=sq, seqlen_k=sk, head_dim=d, window_left=-1,
                                   window_right=-1), **kw})


def _bwd_args(b, h, hk, sq, sk, d, which=3):
    from flash_attn2_b200 import _cabi

    return _cabi.BwdArgs(batch=b, heads=h, heads_k=hk, seqlen_q=sq, seqlen_k=sk, head_dim=d, which=which,
                         window_left=-1, window_right=-1)


@pytest.mark.parametrize("which", [2, 3])
@pytest.mark.parametrize("offset,shares", [(0, 1), (256, 1), (16, 0), (32, 0), (128, 0), (4, 0)])
def test_key_blocks_are_shared_in_an_aligned_workspace_only(plans, which, offset, shares):
    """Their parts are stored 32 bytes at a time; the workspace's other contents need 16-byte alignment."""
    args = _bwd_args(1, 4, 1, 777, 777, 128, which)
    assert plans.bwd_shares(ctypes.byref(args), SMS, ctypes.c_uint64((1 << 40) + offset), ctypes.c_int64(0)) == shares
    assert plans.bwd_shares(ctypes.byref(args), SMS, ctypes.c_uint64((1 << 40) + offset), ctypes.c_int64(1)) == 0
    assert plans.bwd_shares(ctypes.byref(args), SMS, ctypes.c_uint64(0), ctypes.c_int64(0)) == 0


# Shapes (batch, heads, heads_k, seqlen_q, seqlen_k, head_dim) timed both ways; us general, few-row kernel.
SLOWER = [((64, 8, 8, 64, 64, 128), (17, 35)), ((64, 8, 8, 33, 384, 128), (29, 56)), ((64, 8, 8, 64, 1024, 256), (103, 176)),
          ((5, 8, 8, 64, 384, 256), (13, 25)), ((1, 74, 74, 48, 384, 192), (13, 21)), ((64, 8, 8, 24, 64, 128), (17, 25)),
          ((64, 8, 8, 33, 384, 64), (25, 33))]
FASTER = [((1, 32, 8, 1, 8192, 128), (86, 16)), ((32, 32, 8, 1, 4093, 128), (316, 91)), ((5, 8, 8, 1, 4096, 128), (33, 19)),
          ((2, 64, 8, 8, 4096, 128), (49, 34)), ((64, 8, 8, 1, 2048, 64), (87, 68)), ((5, 64, 8, 8, 1024, 256), (58, 43)),
          ((2, 8, 8, 32, 4096, 192), (62, 29))]


@pytest.mark.parametrize("shape,us", SLOWER + FASTER, ids=[str(s) for s, _ in SLOWER + FASTER])
def test_the_few_row_kernel_takes_what_it_is_faster_for(plans, shape, us):
    b, h, hk, sq, sk, d = shape
    taken = plans.few_rows(ctypes.byref(_fwd_args(*shape)), SMS)
    assert taken == (sq * h // hk if us[1] < us[0] else 0)
    # a window leaves fewer key tiles; a mask that hides every key is not for it
    assert plans.few_rows(ctypes.byref(_fwd_args(b, h, hk, sq, 128, d, causal=1, window_left=3)), SMS) in (0, sq * h // hk)
    assert plans.few_rows(ctypes.byref(_fwd_args(b, h, hk, 65, sk, d)), SMS) == 0


@pytest.mark.parametrize("head_dim", [257, 264, 1024, 0, -8])
def test_head_dims_outside_the_range_have_no_plan(plans, head_dim):
    """Scratch memory is asked for before a call is checked."""
    for sq in (1, 300):
        args = _fwd_args(1, 8, 2, sq, 4000, head_dim)
        assert plans.few_rows(ctypes.byref(args), SMS) == 0 and plans.few_rows_workspace(ctypes.byref(args), SMS) == 0
        if head_dim > 0:
            assert plans.shared_tiles(ctypes.byref(args), SMS) == 0


# Shapes (heads, seqlen_q, seqlen_k, head_dim, causal) timed with and without sharing.
NOT_SHARED = [(12, 2000, 2048, 128, 1), (12, 2000, 4096, 128, 0), (50, 512, 4096, 128, 1), (18, 1000, 2048, 128, 1),
              (6, 4000, 4096, 128, 0), (9, 4000, 4096, 128, 1), (100, 65, 9000, 128, 0), (100, 128, 9000, 128, 0)]
SHARED = [(4, 128, 9000, 64, 0), (4, 256, 9000, 128, 0), (20, 512, 4096, 128, 0), (40, 128, 9000, 128, 1), (74, 128, 2048, 64, 0)]


@pytest.mark.parametrize("shape", NOT_SHARED + SHARED, ids=str)
def test_tiles_are_shared_where_that_is_faster(plans, shape):
    h, sq, sk, d, causal = shape
    got = plans.shared_tiles(ctypes.byref(_fwd_args(1, h, h, sq, sk, d, causal=causal)), SMS)
    assert (got > 0) == (shape in SHARED)


# Which keys share a part's running maximum decides how P is rounded to 16 bits, so the number of parts is part of a call's
# result: 18 parts in place of 16 change the output of 8192 keys by 2e-3 of its 2-norm.
@pytest.mark.parametrize("sk,parts", [(384, 1), (385, 1), (768, 2), (2049, 5), (4093, 10), (6145, 16), (8192, 18), (9000, 18), (30000, 18)])
def test_parts_of_a_few_row_unit(plans, sk, parts):
    """As many equal parts as the SMs allow and leave three key tiles, at most 24."""
    assert plans.few_rows_ctas(ctypes.byref(_fwd_args(1, 32, 8, 1, sk, 128, causal=1)), SMS) == 8 * parts
    assert plans.few_rows_ctas(ctypes.byref(_fwd_args(1, 4, 1, 1, 16384, 128, causal=1)), SMS) == 24


# (batch, heads, heads_k, seqlen_k, head_dim): timed with and without the early start.
LATE = [(10, 32, 8, 4000, 128), (10, 32, 8, 8000, 128), (12, 32, 8, 8192, 128), (16, 64, 8, 16384, 128), (8, 64, 8, 16384, 128),
        (76, 4, 1, 16384, 128), (16, 32, 8, 8192, 192), (10, 32, 8, 4000, 256), (16, 32, 8, 8192, 256)]
EARLY = [(1, 32, 8, 8192, 128), (32, 32, 8, 4093, 128), (10, 32, 8, 1000, 128), (16, 64, 8, 1024, 128), (9, 32, 8, 16000, 128),
         (17, 32, 8, 16000, 128), (10, 32, 8, 4000, 64), (37, 32, 8, 2048, 256)]


@pytest.mark.parametrize("shape", LATE + EARLY, ids=str)
def test_few_row_calls_start_early_where_that_is_faster(plans, shape):
    b, h, hk, sk, d = shape
    assert plans.few_rows_start_early(ctypes.byref(_fwd_args(b, h, hk, 1, sk, d, causal=1)), SMS) == (shape in EARLY)


# (batch, heads, heads_k, seqlen, head_dim), causal, heads in a group: all of them in a call of few CTAs; else about 96 MB in as
# even groups as whole heads allow (25 MB a head: 9 groups of 32 heads; 3 MB: 9 of 256; 96 KB: 1024 heads; 71 MB: pairs), without a
# mask 16 MB (391 KB a head).
GROUPS = [((4, 16, 4, 2048, 128), 1, 16), ((1, 32, 32, 16384, 128), 1, 4), ((16, 16, 16, 2048, 128), 1, 29),
          ((32, 12, 12, 509, 64), 0, 43), ((1, 1, 1, 1, 8), 0, 1), ((65535, 64, 64, 128, 64), 1, 1024), ((2, 64, 8, 8192, 128), 1, 2)]


@pytest.mark.parametrize("shape,causal,want", GROUPS, ids=str)
def test_heads_in_a_group(plans, shape, causal, want):
    b, h, hk, s, d = shape
    args = _bwd_args(b, h, hk, s, s, d)
    args.causal = causal
    assert plans.head_group(ctypes.byref(args), 0, SMS) == want
    assert 1 <= plans.head_group(ctypes.byref(args), 1, SMS) <= b * h
    args.cu_seqlens_q = 8  # packed sequences differ in length: one after the other
    assert plans.head_group(ctypes.byref(args), 0, SMS) == 1


def test_the_gpu_test_of_the_order_has_several_groups(plans):
    from tests.test_bwd_order_gpu import CASES, SEVERAL

    def groups(shape, causal, dq_alone):
        h, hk, s, d = shape
        args = _bwd_args(1, h, hk, s, s, d)
        args.causal = causal
        n, heads = plans.head_group(ctypes.byref(args), dq_alone, SMS), h if dq_alone else hk
        return n, heads

    for shape, causal in CASES:
        n, heads = groups(shape, causal, 0)
        assert 1 < n < heads and heads % n if (shape, causal) in SEVERAL else n == heads
    n, heads = groups(*SEVERAL[-1], 1)
    assert 1 < n < heads and heads % n


def _takes_pairs(plans, case, **kw):
    from flash_attn2_b200 import _cabi

    b, h, hk, sq, sk, d, causal, (left, right) = case
    a = _cabi.BwdArgs(**{**dict(batch=b, heads=h, heads_k=hk, seqlen_q=sq, seqlen_k=sk, head_dim=d, causal=causal, window_left=left,
                                window_right=right, which=3), **kw})
    return bool(plans.takes_pairs(ctypes.byref(a), SMS))


def _empty_pairs(case):
    """Pairs of a head (256 keys, 128 at head dims above 128) none of whose keys a query sees, from the mask itself."""
    _, _, _, sq, sk, d, causal, (left, right) = case
    right = 0 if causal else right
    i, j = torch.arange(sq)[:, None] + (sk - sq), torch.arange(sk)[None, :]
    seen = torch.ones(sq, sk, dtype=torch.bool)
    if right >= 0:
        seen &= j <= i + right
    if left >= 0:
        seen &= j >= i - left
    return sum(not keys.any() for keys in seen.any(0).split(256 if d <= 128 else 128))


def test_backward_calls_that_run_on_pairs(plans):
    from tests import test_canaries_gpu, test_stream_order_gpu, test_zz_no_alloc
    from tests.test_bwd_pair_gpu import CASES, EMPTY, REPEATED, WIDE

    assert all(_takes_pairs(plans, c) for c in CASES + WIDE + REPEATED)
    none = (-1, -1)
    assert all(_takes_pairs(plans, (*c[:6], c[6], none)) for c in test_canaries_gpu.PAIRS)
    assert all(_takes_pairs(plans, (*shape, causal, none)) for shape, causal, _ in test_stream_order_gpu.PAIRS)
    assert all(_takes_pairs(plans, (*shape, False, none)) for shape in test_zz_no_alloc.PAIRS)
    assert {c[5] for c in EMPTY} == {128, 192, 256} and all((_empty_pairs(c) > 0) == (c in EMPTY) for c in CASES + WIDE)
    assert not any(_takes_pairs(plans, WIDE[0], **other) for other in (dict(which=1), dict(which=2), dict(head_dim=248), dict(head_dim=184),
                                                               dict(cu_seqlens_q=256), dict(head_dim=192, seqlen_q=300)))
    # Head dim 256: rows padded by a fifth more than in blocks of 64, and a third of the keys' blocks empty.
    for rows, keys, taken in ((60, 60, False), (64, 170, False), (130, 130, False), (170, 170, False), (171, 171, True), (192, 85, False), (192, 86, True),
                              (65, 65, True), (193, 60, True), (320, 60, False), (60, 2000, True)):
        assert _takes_pairs(plans, WIDE[0], seqlen_q=rows, seqlen_k=keys) == taken, (rows, keys)
    full = (4, 16, 16, 2048, 2048, 128, False, (-1, -1))
    assert _takes_pairs(plans, full)
    # An odd number of key blocks leaves one CTA of a head without keys, which 15 blocks and more make up for, and a causal mask.
    assert [n for n in range(1, 24) if _takes_pairs(plans, full, batch=16, seqlen_k=128 * n - 60)] == [*range(2, 14, 2), *range(14, 24)]
    assert _takes_pairs(plans, full, causal=True, seqlen_q=4200, seqlen_k=4200)
    for other in (dict(which=1), dict(which=2), dict(head_dim=96), dict(head_dim=136), dict(softcap=30.0), dict(alibi_slopes=256),
                  dict(cu_seqlens_q=256), dict(causal=True), dict(window_left=1023), dict(batch=1, heads=8, heads_k=8), dict(seqlen_k=1600)):
        assert not _takes_pairs(plans, full, **other), other
