"""CPU: the native libraries load and export every symbol the headers / the reference name.
No compute call is made here (there is no GPU)."""
import ctypes
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def test_cabi_exports_every_declared_symbol(built_libs):
    header = (ROOT / "include" / "fa2_b200.h").read_text()
    declared = re.findall(r"FA2_API\s+[\w\s\*]+?\b(fa2_\w+)\s*\(", header)
    assert len(declared) >= 8
    lib = ctypes.CDLL(str(built_libs / "libfa2_b200.so"))
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in include/fa2_b200.h but not exported"
    from flash_attn2_b200 import _cabi

    assert set(_cabi.EXPORTS) == set(declared)


def test_cabi_struct_layout_matches_header(built_libs):
    """The ctypes mirrors must have the C structs' sizes (checked with a tiny compiled probe)."""
    import subprocess
    import tempfile

    src = '#include <stdio.h>\n#include "fa2_b200.h"\nint main(){printf("%zu %zu %zu", sizeof(fa2_fwd_args), ' \
          'sizeof(fa2_bwd_preprocess_args), sizeof(fa2_bwd_args));return 0;}'
    with tempfile.TemporaryDirectory() as d:
        (Path(d) / "p.c").write_text(src)
        subprocess.run(["gcc", f"-I{ROOT / 'include'}", str(Path(d) / "p.c"), "-o", str(Path(d) / "p")], check=True)
        sizes = [int(x) for x in subprocess.run([str(Path(d) / "p")], capture_output=True, text=True).stdout.split()]
    from flash_attn2_b200 import _cabi

    assert sizes == [ctypes.sizeof(_cabi.FwdArgs), ctypes.sizeof(_cabi.BwdPreprocessArgs), ctypes.sizeof(_cabi.BwdArgs)]


@pytest.mark.parametrize("limit,ok", [("(1ll << 31)", True), ("(1ll << 32)", False), ("(3ll << 32)", False), ("0", False)])
def test_wait_limits_that_32_bits_cannot_hold_do_not_build(limit, ok, tmp_path):
    """The waits compare 32 bits of the clock: 2^32 cycles would be a limit of none."""
    import subprocess

    (tmp_path / "w.cu").write_text('#include "sm100_ptx.cuh"\n')
    run = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", f"-DFA2_WAIT_LIMIT_CYCLES={limit}",
                          f"-I{ROOT / 'kernels-community-rs_b200' / 'csrc'}", "-c", str(tmp_path / "w.cu"), "-o", str(tmp_path / "w.o")],
                         capture_output=True, text=True)
    assert (run.returncode == 0) == ok and ("32 bits of the clock" in run.stderr) != ok, run.stderr


def test_tvm_ffi_library_exports_reference_operator_names(built_libs):
    from flash_attn2_b200 import _ops

    lib = ctypes.CDLL(str(built_libs / "libflash_attn2_b200.so"))
    for name in _ops.OP_NAMES:
        assert hasattr(lib, f"__tvm_ffi_{name}")
        assert hasattr(_ops.ops, name)
    assert _ops.torch_add_op_namespace_prefix("x").endswith("::x")


def test_argument_contract_without_gpu(built_libs):
    """Bad calls fail before any launch with the reference's error kinds."""
    import flash_attn2_b200 as fa

    z = torch.zeros(1, 8, 2, 64, dtype=torch.float16)
    with pytest.raises(NotImplementedError):  # CPU tensors: no CPU implementation
        fa.fwd(z, z, z)
    with pytest.raises(NotImplementedError):
        fa.cabi_ops.fwd(z, z, z)
    with pytest.raises(ValueError):  # wrong positional count
        fa.ops.fwd(z, z)
    with pytest.raises(ValueError):  # CUDA tensors required by the operator itself
        fa.ops.fwd(z, z, z, None, None, False, -1, -1, 0.0)
    with pytest.raises(TypeError):  # scalar of the wrong type
        fa.ops.fwd(z, z, z, None, None, "yes", -1, -1, 0.0)
    with pytest.raises(RuntimeError):  # exports outside the built path fail loudly
        fa.ops.rng_state()
    with pytest.raises(RuntimeError):
        fa.fwd(z.cuda() if torch.cuda.is_available() else z, z, z, p_dropout="0.1")


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from flash_attn2_b200 import _cabi

    monkeypatch.setattr(_cabi, "_lib", None)
    monkeypatch.setattr(_cabi, "LIB_PATH", tmp_path / "libfa2_b200.so")
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        _cabi.load()


def _header_fields(struct):
    """(name, array length) of a struct's fields, from the header."""
    header = re.sub(r"/\*.*?\*/", "", (ROOT / "include" / "fa2_b200.h").read_text(), flags=re.S)
    body = re.search(r"typedef struct %s \{(.*?)\} %s;" % (struct, struct), header, flags=re.S).group(1)
    names = [n for decl in body.split(";") if decl.strip() for n in decl.rsplit("*", 1)[-1].split(",")]
    return [(re.search(r"(\w+)\s*(?:\[\d+\])?\s*$", n).group(1), re.findall(r"\[(\d+)\]", n)) for n in names]


def test_argument_structs_do_not_change_size(built_libs):
    """A host binds these by layout: a field more would be read behind what an older host passes. What a call can do
    besides goes into calls of its own and into fa2_bwd_options, which says its size."""
    from flash_attn2_b200 import _cabi

    assert ctypes.sizeof(_cabi.FwdArgs) == 232
    assert ctypes.sizeof(_cabi.BwdPreprocessArgs) == 112
    assert ctypes.sizeof(_cabi.BwdArgs) == 296
    assert _header_fields("fa2_fwd_args")[-1][0] == "zero_tensors" and _header_fields("fa2_bwd_args")[-1][0] == "softcap"


@pytest.mark.parametrize("struct,mirror", [("fa2_fwd_args", "FwdArgs"), ("fa2_bwd_preprocess_args", "BwdPreprocessArgs"),
                                           ("fa2_bwd_args", "BwdArgs"), ("fa2_bwd_options", "BwdOptions")])
def test_ctypes_mirrors_have_the_fields_of_the_header(struct, mirror):
    from flash_attn2_b200 import _cabi

    got = [(n, [str(t._length_)] if hasattr(t, "_length_") else []) for n, t in getattr(_cabi, mirror)._fields_]
    assert got == _header_fields(struct)


def test_integration_guide_shows_the_header():
    """The guide's Rust mirror has the header's fields in the header's order, and names only functions that exist."""
    guide = (ROOT / "INTEGRATION.md").read_text()
    body = re.search(r"pub struct Fa2FwdArgs \{(.*?)\n\}", guide, flags=re.S).group(1)
    assert [(n, re.findall(r"\[i64; (\d+)\]", t)) for n, t in re.findall(r"pub (\w+): ([^,]*(?:\[[^\]]*\])?)", body)] == \
        _header_fields("fa2_fwd_args")
    header = (ROOT / "include" / "fa2_b200.h").read_text()
    bound = re.findall(r"\bfn (fa2_\w+)\(", guide)
    assert {"fa2_fwd", "fa2_fwd_with_workspace", "fa2_fwd_workspace_bytes", "fa2_bwd", "fa2_bwd_with_options"} <= set(bound)
    for name in set(re.findall(r"\bfa2_(?:fwd|bwd|varlen)\w*", guide)) - {"fa2_fwd_args", "fa2_bwd_args", "fa2_bwd_preprocess_args", "fa2_bwd_options"}:
        assert re.search(r"\b%s\s*\(" % name, header), name


def test_backward_options_of_an_unknown_size_are_refused(built_libs):
    from flash_attn2_b200 import _cabi

    lib = _cabi.load()
    opt = _cabi.BwdOptions(size=ctypes.sizeof(_cabi.BwdOptions) + 8)
    assert lib.fa2_bwd_with_options(ctypes.byref(_cabi.BwdArgs()), ctypes.byref(opt), None) == -1
    assert b"size" in lib.fa2_last_error()


def test_workspace_holds_turn_counters_only_where_they_are_used(built_libs):
    """Behind the fp32 accumulator of dQ, for packed dQ-only calls up to head dim 128."""
    from flash_attn2_b200 import _cabi

    lib = _cabi.load()
    shape = dict(batch=2, seqlen_q=256, seqlen_k=256, heads=4, heads_k=2, window_left=-1, window_right=-1)

    def need(which, d, packed):
        args = _cabi.BwdArgs(which=which, head_dim=d, **shape, **(dict(cu_seqlens_q=8, cu_seqlens_k=8, total_q=512, total_k=512)
                                                                  if packed else {}))
        return lib.fa2_bwd_workspace_bytes(ctypes.byref(args))

    for d in (64, 128, 256):
        accum = 2 * 256 * 4 * d * 4
        assert need(3, d, False) == need(3, d, True) == accum and need(2, d, False) == need(2, d, True) == 0
        assert need(1, d, False) == (0 if d <= 128 else accum)
        assert need(1, d, True) == accum + (2 * 4 * 2 * 4 * 4 if d <= 128 else 0)


def test_kernels_that_start_early_wait_before_they_let_the_next_one_in():
    """Of a kernel launched as a programmatic dependent every CTA waits for what is before it in the stream, whatever the call's
    arguments, and only then lets the next grid start: no grid runs beside another one than the one right before it."""
    sources = {f.name: f.read_text() for f in (ROOT / "kernels-community-rs_b200" / "csrc").glob("*.cu")}
    launches = {(f, when, k) for f, s in sources.items() for when, k in re.findall(r"launch_grid\(([^,]*), (\w+)", s)}
    assert len(launches) >= 7
    for f, when, kernel in launches:
        start = re.search(rf"(template <[^;{{}}]*>\s*)__global__[^;{{]*\b{kernel}\(", sources[f])
        body = sources[f][start.end():]
        assert re.search(r"^  early_wait\(\);$", body[: body.index("early_trigger();")], re.M), (f, kernel)
        # Packed batches are launched the usual way and let the next grid in at their end.
        packed = "bool PACKED" in start.group(1)
        assert when == ("!PACKED" if packed else "early" if kernel == "fwd_decode_kernel" else "true"), (f, kernel)
        assert ("if (!PACKED) early_trigger();" in body) == packed, (f, kernel)


@pytest.mark.parametrize("kernel", ["fwd_sm100.cu", "fwd_wide_sm100.cu"])
def test_the_forward_refills_no_slot_that_the_fixer_has_not_seen(kernel):
    """The fixer warp of packed batches waits for every tile by the parity of its barrier's phase. A stage that came back to the
    loader without it could be filled again meanwhile, and the warp would wait for a phase that has gone by."""
    body = (ROOT / "kernels-community-rs_b200" / "csrc" / kernel).read_text()
    packed, dense = re.search(r"mbar_init\(&kv_empty\[i\], PACKED \? (\d) : (\d)\);", body).groups()
    assert int(packed) == int(dense) + 1
    fixer = body[body.index("- fixer (packed batches)"):body.index("- mma issuer")]
    assert re.search(r"mbar_wait\(&kv_full\[slot\]", fixer) and re.search(r"mbar_arrive\(&kv_empty\[slot\]\)", fixer)


def test_the_backward_refills_no_stage_that_the_fixer_has_not_seen():
    """The same for its Q and dO stages."""
    body = (ROOT / "kernels-community-rs_b200" / "csrc" / "bwd_sm100.cu").read_text()
    counted = re.search(r"if \(PACKED && \(([^;]*)\)\) count = 2;", body).group(1)
    fixer = body[body.index("- fixer (packed batches)"):body.index("- -LSE (log2 domain)")]
    waited = set(re.findall(r"mbar_wait\(&(\w+)_full\[", fixer))
    assert waited == {"q", "do"}
    for name in waited:
        assert f"bar == {name}_empty" in counted and f"bar == {name}_empty + 1" in counted, name
        assert re.search(rf"mbar_arrive\(&{name}_empty\[", fixer), name
