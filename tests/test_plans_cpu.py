"""CPU: how a dense call is divided over the GPU (csrc/fa2_plan.h), through a small library around that header."""
import ctypes
import subprocess
from pathlib import Path

import pytest

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
}
'''


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("plans")
    (d / "shim.cc").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{ROOT / 'kernels-community-rs_b200' / 'csrc'}",
                    "-I/usr/local/cuda/include", str(d / "shim.cc"), "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


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
