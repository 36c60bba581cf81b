"""CPU-side checks of the boundary: the C-ABI library loads, exports every symbol the
header declares, and the ops refuse to run without CUDA tensors (no CPU fallback)."""
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as ge

    ge.build()
    from flaggems_sglang_b200 import _C

    return _C.lib()


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "fmoe_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(fmoe_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound(lib):
    from flaggems_sglang_b200 import _C

    names = _declared_symbols()
    assert len(names) >= 12
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/fmoe_b200.h but not exported"
        assert n in _C.SIGNATURES, f"{n} has no ctypes signature"
    assert sorted(_C.SIGNATURES) == names


def test_struct_layout_matches_header():
    import ctypes

    from flaggems_sglang_b200 import _C

    # struct_size + w_layout, 8 int32, 6 int64, 10 pointers, bias pointer + 2 floats, out_rows, split_ws + its size, scale_mode + a_scale_gather
    assert ctypes.sizeof(_C.GemmArgs) == 8 + 8 * 4 + 6 * 8 + 10 * 8 + (8 + 4 + 4) + 8 + 16 + 8
    assert _C.GemmArgs.struct_size.offset == 0 and _C.GemmArgs.numel.offset == 40 and _C.GemmArgs.a.offset == 88
    # struct_size + w_layout, 8 int32, 3 int64, 2 float, 9 pointers, 1 int64, 2 pointers + 2 floats, out_rows
    assert ctypes.sizeof(_C.FusedArgs) == 8 + 144 + (8 + 8 + 4 + 4) + 8 and _C.FusedArgs.hidden.offset == 72
    assert _C.GemmArgs().struct_size == ctypes.sizeof(_C.GemmArgs)
    assert _C.FusedArgs(T=3).struct_size == ctypes.sizeof(_C.FusedArgs)


@pytest.mark.parametrize("T", [1024, 4096, 16384])
def test_block_scale_workspace_has_no_row_per_position_in_fp32(lib, T):
    """DeepSeek-V3 with both e4m3 kernels at work: fp32 rows only for experts of up to 64 rows, the rest of the workspace is
    the quantised rows, the per-slot results and tables."""
    from flaggems_sglang_b200 import _C

    E, H, I, k = 256, 7168, 2048, 8
    a = _C.FusedArgs(dtype=_C.E4M3, num_experts=E, top_k=k, T=T, H=H, I=I)
    numel = T * k
    cap = numel + E * 127
    rest = cap * (H + I + I // 128 * 4) + numel * H * 2 + T * H // 128 * 4
    assert lib.fmoe_fused_experts_workspace_bytes(a) <= rest + E * 64 * I * 4 + (4 << 20)


@pytest.mark.parametrize("dtype,T,E,H,I,k,want", [
    ("BF16", 1, 128, 2048, 768, 8, "decode"), ("BF16", 9, 128, 2048, 768, 8, "stream"), ("BF16", 16, 8, 4096, 14336, 2, "tcgen05"),
    # fewer than 3 rows per expert: long rows, short rows, little weight; 3 rows
    ("BF16", 10, 8, 4096, 7168, 2, "tcgen05"), ("BF16", 16, 64, 3072, 2304, 8, "stream"), ("BF16", 10, 8, 4096, 3584, 2, "stream"),
    ("BF16", 24, 64, 3072, 2304, 8, "tcgen05"),
    ("E4M3", 8, 256, 7168, 2048, 8, "decode"), ("E4M3", 64, 256, 7168, 2048, 8, "tcgen05"), ("F32", 3, 8, 256, 512, 2, "simt")])
def test_layer_variant_is_what_the_one_call_layer_takes(lib, dtype, T, E, H, I, k, want):
    """Stage names come from here: the choice of the one-call layer, which is not that of GEMMs launched one by one
    (fmoe_pick_variant says "stream" for the Mixtral, DeepSeek-V3 and decode-sized calls of this list)."""
    from flaggems_sglang_b200 import _C
    from flaggems_sglang_b200.ops.fused_moe import layer_variant

    fa = _C.FusedArgs(dtype=getattr(_C, dtype), num_experts=E, top_k=k, T=T, H=H, I=I)
    route = _C.RouteArgs(logits=16, grouped=0, renormalize=1, n_group=1, topk_group=1)
    for r in (None, route):
        name, block = layer_variant(fa, r)
        assert name == want and block == {"decode": 0, "stream": 8, "tcgen05": 128, "simt": 16}[want]


@pytest.mark.parametrize("dtype,T,E,H,I,k,want", [
    # 3 rows per expert from 0.3 GB of weights on
    ("BF16", 48, 128, 2048, 384, 8, "tcgen05"), ("BF16", 47, 128, 2048, 384, 8, "stream"), ("BF16", 24, 64, 1280, 768, 8, "tcgen05"),
    ("BF16", 24, 16, 2048, 1024, 2, "stream"),
    # e4m3 tokens times row length, by the length of the down rows
    ("E4M3", 3, 256, 7168, 1024, 8, "decode"), ("E4M3", 4, 256, 7168, 1024, 8, "tcgen05"), ("E4M3", 3, 256, 7168, 512, 8, "decode"),
    ("E4M3", 4, 256, 7168, 512, 8, "tcgen05"), ("E4M3", 2, 256, 7168, 256, 8, "decode"), ("E4M3", 3, 256, 7168, 256, 8, "tcgen05"),
    ("E4M3", 6, 64, 4096, 1536, 6, "decode"), ("E4M3", 7, 64, 4096, 1536, 6, "tcgen05"), ("E4M3", 8, 128, 2048, 384, 8, "decode")])
def test_layer_variant_on_both_sides_of_its_lines(lib, dtype, T, E, H, I, k, want):
    test_layer_variant_is_what_the_one_call_layer_takes(lib, dtype, T, E, H, I, k, want)


@pytest.mark.parametrize("T,E,H,I,k,want", [
    (4, 8, 7168, 256, 2, "decode"), (5, 8, 7168, 256, 2, "tcgen05"),                                            # channels of the rows
    (5, 16, 7168, 1024, 1, "decode"), (6, 16, 7168, 1024, 1, "tcgen05"), (8, 16, 7168, 1792, 1, "decode"), (6, 8, 5120, 1792, 2, "decode"),
    (7, 8, 5120, 1536, 2, "decode"), (8, 8, 5120, 1536, 2, "tcgen05"),
    (6, 8, 7168, 128, 2, "decode"), (7, 8, 7168, 128, 2, "tcgen05"), (8, 16, 4096, 128, 2, "decode"),           # bytes of the weights
    (5, 32, 4096, 128, 4, "tcgen05"), (5, 64, 4096, 128, 4, "tcgen05"), (8, 8, 4096, 256, 2, "decode")])
def test_small_e4m3_layers_keep_the_decode_kernels(lib, T, E, H, I, k, want):
    """Few slots or few bytes of weights: the CTA-pair kernels' launches and prologues would be most of the call."""
    test_layer_variant_is_what_the_one_call_layer_takes(lib, "E4M3", T, E, H, I, k, want)


@pytest.mark.parametrize("dtype,T,E,H,I,k,small", [
    ("E4M3", 3, 256, 7168, 256, 8, "decode"), ("E4M3", 64, 256, 7168, 2048, 8, "stream"), ("BF16", 48, 128, 2048, 384, 8, "stream"),
    ("BF16", 300, 128, 2048, 384, 8, None), ("E4M3", 4096, 256, 7168, 2048, 8, None), ("BF16", 65, 128, 2048, 384, 8, None)])
def test_workspace_of_the_smaller_kernels_is_taken(lib, dtype, T, E, H, I, k, small):
    """A caller that brings less than the fastest kernels need keeps the ones that need less, down to what those need (found here
    by halving; without pointers a call whose workspace is large enough ends at the check of its pointers).  With many rows per
    expert the streaming kernels would take many times as long: a workspace that is a byte short is refused."""
    from flaggems_sglang_b200 import _C

    a = _C.FusedArgs(dtype=getattr(_C, dtype), num_experts=E, top_k=k, T=T, H=H, I=I, workspace=256)
    need = lib.fmoe_fused_experts_workspace_bytes(a)

    def taken(size):
        a.workspace_bytes = size
        assert lib.fmoe_fused_experts(a, None) == _C.ERR_INVALID_ARG
        msg = lib.fmoe_last_error()
        assert (b"too small" in msg) != (b"null pointer" in msg), msg
        return b"null pointer" in msg

    if small is None:
        assert taken(need) and not taken(need - 1)
        return
    lo, hi = 0, need
    assert taken(hi) and not taken(lo)
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if taken(mid) else (mid, hi)
    # what holds the per-slot results and the activation; the streaming kernels' blocks hold up to 32 rows
    rows = T * k * 8 if small == "decode" else T * k + min(E, T * k) * 31
    eb = 2 if dtype == "BF16" else 1 + 4 / 128 + 4
    assert hi <= min(need - 1, T * k * H * 2 + rows * I * eb + T * H * 2 + (1 << 20))
    a.variant = _C.VARIANTS["tcgen05"]
    assert not taken(need - 1)


@pytest.mark.parametrize("stray", ["logits", "bias"])
def test_one_call_moe_refuses_a_router_input_on_another_device(monkeypatch, stray):
    """The router's inputs go into the library call as plain pointers: they have to be on the layer's device (devices are
    played by the CPU and the meta device here)."""
    import importlib

    FM = importlib.import_module("flaggems_sglang_b200.ops.fused_moe")

    def require(*tensors):
        devs = {t.device for t in tensors if t is not None}
        if len(devs) > 1:
            raise RuntimeError("tensors on different devices")
        return devs.pop()

    monkeypatch.setattr(FM._C, "require_cuda", require)  # (one module: the router's ops call the same)
    h, w1, w2 = torch.zeros(3, 64), torch.zeros(4, 256, 64), torch.zeros(4, 64, 128)
    logits = torch.zeros(3, 4, device="meta" if stray == "logits" else "cpu")
    bias = torch.zeros(4, device="meta" if stray == "bias" else "cpu")
    with pytest.raises(RuntimeError, match="different devices"):
        FM.fused_moe(h, w1, w2, logits, 2, use_grouped_topk=True, num_expert_group=2, topk_group=1, correction_bias=bias)


def test_calls_run_on_the_device_of_their_tensors(monkeypatch):
    """With another device current, a call switches to the tensors' device and back (two devices are played here)."""
    import importlib

    FM = importlib.import_module("flaggems_sglang_b200.ops.fused_moe")
    now, seen = [0], []
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: now[0], raising=False)
    monkeypatch.setattr(torch._C, "_cuda_setDevice", lambda d: (seen.append(d), now.__setitem__(0, d)), raising=False)
    monkeypatch.setattr(FM._C, "require_cuda", lambda *t: torch.device("cuda", 1))
    x, w1, w2 = torch.zeros(0, 64), torch.zeros(4, 256, 64), torch.zeros(4, 64, 128)
    out = FM.fused_experts(x, w1, w2, torch.zeros(0, 2), torch.zeros(0, 2, dtype=torch.int32), no_combine=True)
    assert out.shape == (0, 2, 64) and seen == [1, 0]
    with pytest.raises(ZeroDivisionError):
        with FM._C.on_device(torch.device("cuda", 1)):
            assert now == [1]
            1 / 0
    assert now == [0]
    with FM._C.on_device(torch.device("cuda", 0)):
        pass
    assert seen == [1, 0, 1, 0]


def test_unknown_struct_size_is_refused(lib):
    """A binding compiled against another version of the header is caught before any field is trusted."""
    import ctypes

    from flaggems_sglang_b200 import _C

    g = _C.GemmArgs(dtype=_C.BF16, num_experts=4, top_k=2, block_size=16, numel=8, n=128, k=128)
    g.struct_size -= 8  # the size of a struct that ends before scale_mode / a_scale_gather (ABI version 3)
    assert lib.fmoe_gemm2(ctypes.byref(g), None) == _C.ERR_INVALID_ARG and b"struct_size" in lib.fmoe_last_error()
    assert lib.fmoe_gemm1_silu(ctypes.byref(g), None) == _C.ERR_INVALID_ARG
    f = _C.FusedArgs(dtype=_C.BF16, num_experts=4, top_k=2, T=4, H=128, I=128)
    f.struct_size = 0
    assert lib.fmoe_fused_experts_workspace_bytes(ctypes.byref(f)) < 0 and b"struct_size" in lib.fmoe_last_error()
    assert lib.fmoe_fused_experts(ctypes.byref(f), None) == _C.ERR_INVALID_ARG
    assert lib.fmoe_fused_experts_static(ctypes.byref(f), None) == _C.ERR_INVALID_ARG


def _integration_snippet():
    """The ctypes stub INTEGRATION.md shows to a maintainer of the reference, as source text."""
    text = open(os.path.join(ROOT, "INTEGRATION.md")).read()
    blocks = re.findall(r"```python\n(.*?)```", text, flags=re.S)
    stub = [b for b in blocks if "class GemmArgs" in b]
    assert len(stub) == 1, "INTEGRATION.md must hold exactly one ctypes stub with a GemmArgs mirror"
    return stub[0]


def test_integration_stub_struct_matches_binding(lib):
    """The struct mirror printed in INTEGRATION.md has the layout of the real one (a stale copy there would make
    the library read past the caller's struct)."""
    import ctypes

    from flaggems_sglang_b200 import _C

    ns = {"LIBFMOE_PATH": _C.LIB_PATH}
    exec(compile(_integration_snippet(), "INTEGRATION.md", "exec"), ns)
    G = ns["GemmArgs"]
    assert ctypes.sizeof(G) == ctypes.sizeof(_C.GemmArgs)
    assert [(n, getattr(G, n).offset) for n, _ in G._fields_] == \
        [(n, getattr(_C.GemmArgs, n).offset) for n, _ in _C.GemmArgs._fields_]
    assert G(n=1).struct_size == ctypes.sizeof(_C.GemmArgs)


def test_version_and_error_buffer(lib):
    assert lib.fmoe_version() == 4
    # an invalid call reports through the status code and the message buffer, without touching a device
    rc = lib.fmoe_topk_softmax(None, 4, 0, 1, 1, None, None, None)
    assert rc == 1
    assert b"E" in lib.fmoe_last_error()
    rc = lib.fmoe_moe_align_block_size(None, 8, 4, 0, None, 0, None, 0, None, None)
    assert rc == 1 and b"block" in lib.fmoe_last_error()


def test_ops_refuse_cpu_tensors():
    import flaggems_sglang_b200 as fg

    x = torch.randn(4, 256)
    with pytest.raises(RuntimeError, match="no CPU path"):
        fg.fused_topk(x, torch.randn(4, 8), 2)
    with pytest.raises(RuntimeError, match="no CPU path"):
        fg.moe_align_block_size(torch.zeros(4, 2, dtype=torch.int32), 16, 8)
    with pytest.raises(RuntimeError, match="no CPU path"):
        fg.fused_experts(x, torch.randn(8, 64, 256), torch.randn(8, 256, 32), torch.rand(4, 2),
                         torch.zeros(4, 2, dtype=torch.int32))


def test_namespace_mirrors_reference_exports():
    import flaggems_sglang_b200 as fg

    for name in ("triton_kernel_fused_experts", "fused_moe_flagos", "fused_moe", "fused_experts",
                 "moe_align_block_size", "topk", "grouped_topk", "fused_topk", "moe_sum"):
        assert callable(getattr(fg, name))
        assert name in fg.all_registered_ops()


def test_reference_entry_point_keeps_its_assertions():
    """Argument checks of the reference op fire before any device work (ref fused_moe.py:170-195)."""
    import flaggems_sglang_b200 as fg

    x = torch.randn(4, 128, dtype=torch.bfloat16)
    w1 = torch.randn(8, 128, 512, dtype=torch.bfloat16)
    w2 = torch.randn(8, 256, 128, dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="use_fp8_w8a8 is not supported"):
        fg.triton_kernel_fused_experts(x, w1, w2, None, None, None, use_fp8_w8a8=True)
    with pytest.raises(AssertionError, match="Inplace is not supported"):
        fg.triton_kernel_fused_experts(x, w1, w2, None, None, None, inplace=True)
    with pytest.raises(AssertionError, match="hidden_states must be bfloat16"):
        fg.triton_kernel_fused_experts(x.float(), w1, w2, None, None, None)
    with pytest.raises(AssertionError, match="hidden size mismatch"):
        fg.triton_kernel_fused_experts(x[:, :64], w1, w2, None, None, None)
    with pytest.raises(ValueError, match="Unsupported FusedMoe activation"):
        fg.triton_kernel_fused_experts(x, w1, w2, None, None, None, activation="relu")


def test_variant_selection_is_shape_only():
    from flaggems_sglang_b200.ops.fused_moe import _pick_variant

    bf = torch.bfloat16
    assert _pick_variant(torch.float32, 32, 8, 512, 256, None) == ("simt", 16)
    assert _pick_variant(bf, 2, 8, 14336, 4096, None) == ("stream", 8)        # Mixtral T=1
    assert _pick_variant(bf, 32, 8, 14336, 4096, None)[0] == "stream"         # Mixtral T=16
    assert _pick_variant(bf, 128, 8, 14336, 4096, None)[0] == "tcgen05"       # Mixtral T=64 (HBM-bound, 128-row tiles)
    assert _pick_variant(bf, 8192, 8, 14336, 4096, None) == ("tcgen05", 128)  # Mixtral T=4096
    assert _pick_variant(bf, 65536, 128, 768, 2048, None) == ("tcgen05", 128)
    assert _pick_variant(torch.float8_e4m3fn, 512, 256, 2048, 7168, None) == ("stream", 8)   # DSV3 T=64
    assert _pick_variant(torch.float8_e4m3fn, 2048, 256, 2048, 7168, None)[0] == "tcgen05"   # DSV3 T=256
    assert _pick_variant(torch.float8_e4m3fn, 131072, 256, 2048, 7168, None) == ("tcgen05", 128)


@pytest.mark.parametrize("src,kernel,count", [
    ("gemm_pair_fold.cu", r"fold_wide_kernelILb[01]ELb0ELb1ELb[01]E", 4), ("gemm_pair_fold.cu", r"fold_kernelILb[01]ELb0ELb1E", 2),
    ("gemm_pair.cu", r"pair_kernelI", 10)])
def test_tensor_core_kernels_keep_their_registers(lib, src, kernel, count):
    """No kernel of the tensor-core GEMMs spills (the e4m3 ones: as they are launched, with the register move and without the
    profile): their warps run at 64, 96 or 104 registers, and a spill is a local-memory access per K block."""
    from flaggems_sglang_b200.build import ptxas_report

    found = re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads",
                       open(ptxas_report(src)).read(), flags=re.S)
    mine = [f for f in found if re.search(kernel, f[0])]
    assert len(mine) == count and all(f[1:] == ("0", "0") for f in mine), mine


def test_header_compiles_as_plain_c_and_cpp(tmp_path):
    """The boundary is a C ABI: the public header must be self-contained C99 (and valid C++), and a C translation unit
    that fills both argument structs must agree with the ctypes mirrors on their sizes."""
    import ctypes
    import shutil
    import subprocess

    from flaggems_sglang_b200 import _C

    gcc = shutil.which("gcc")
    if not gcc:
        pytest.skip("no gcc")
    header = os.path.join(ROOT, "include", "fmoe_b200.h")
    subprocess.run([gcc, "-std=c99", "-Wall", "-Werror", "-fsyntax-only", "-x", "c", header], check=True)
    gxx = shutil.which("g++")
    if gxx:
        subprocess.run([gxx, "-std=c++11", "-Wall", "-Werror", "-fsyntax-only", "-x", "c++", header], check=True)
    src = tmp_path / "sizes.c"
    src.write_text('#include <stdio.h>\n#include "fmoe_b200.h"\nint main(void) {\n'
                   '  fmoe_gemm_args g = {0}; fmoe_fused_args f = {0};\n'
                   '  g.struct_size = (uint32_t)sizeof g; f.struct_size = (uint32_t)sizeof f;\n'
                   '  printf("%u %u %d %d\\n", g.struct_size, f.struct_size, FMOE_W_N_MAJOR, FMOE_SCALE_CHANNEL);\n'
                   '  return 0;\n}\n')
    exe = tmp_path / "sizes"
    subprocess.run([gcc, "-std=c99", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in out] == [ctypes.sizeof(_C.GemmArgs), ctypes.sizeof(_C.FusedArgs), _C.W_N_MAJOR, _C.SCALE_CHANNEL]


def test_hook_output_type_follows_the_serving_stack(monkeypatch):
    """Without sglang the import path is searched once; a serving stack that is loaded later is found all the same."""
    import importlib
    import sys
    import types

    fm = importlib.import_module("flaggems_sglang_b200.ops.fused_moe")
    searched = []

    class Finder:
        def find_spec(self, name, path=None, target=None):
            searched.append(name)

    for name in [m for m in sys.modules if m.split(".")[0] == "sglang"]:
        monkeypatch.delitem(sys.modules, name)
    monkeypatch.setattr(sys, "meta_path", [Finder()])
    monkeypatch.setattr(fm, "_sglang_missing", False)
    for _ in range(3):
        assert fm._standard_output_type() is fm.StandardCombineInput
    assert searched == ["sglang"]
    path = "sglang.srt.layers.moe.token_dispatcher.standard".split(".")
    for i in range(len(path)):
        monkeypatch.setitem(sys.modules, ".".join(path[:i + 1]), types.ModuleType(path[i]))
    sys.modules[".".join(path)].StandardCombineInput = dict
    assert fm._standard_output_type() is dict


@pytest.mark.parametrize("how", ["path", "files"])
def test_hook_output_type_finds_a_serving_stack_that_comes_later(monkeypatch, tmp_path, how):
    """sglang becomes importable after a search has failed, and nobody else imports it: by a new entry of the import path, at
    once; by files in a directory that was on it, at the next search."""
    import importlib
    import sys
    import time

    fm = importlib.import_module("flaggems_sglang_b200.ops.fused_moe")
    for name in [m for m in sys.modules if m.split(".")[0] == "sglang"]:
        monkeypatch.delitem(sys.modules, name)
    monkeypatch.setattr(sys, "path", ([str(tmp_path)] if how == "files" else []) + [p for p in sys.path if p])
    monkeypatch.setattr(fm, "_sglang_missing", False)
    if fm._standard_output_type() is not fm.StandardCombineInput:
        pytest.skip("sglang is installed")
    d = tmp_path / "sglang" / "srt" / "layers" / "moe" / "token_dispatcher"
    d.mkdir(parents=True)
    (d / "standard.py").write_text("class StandardCombineInput:\n    pass\n")
    if how == "path":
        sys.path.insert(0, str(tmp_path))
    else:
        importlib.invalidate_caches()
        monkeypatch.setattr(time, "monotonic", lambda: 1e12)
    try:
        assert fm._standard_output_type().__module__ == "sglang.srt.layers.moe.token_dispatcher.standard"
    finally:
        for name in [m for m in sys.modules if m.split(".")[0] == "sglang"]:
            del sys.modules[name]
