"""The C-ABI library loads on a machine without a GPU and exports every symbol the header declares."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build_module():
    import importlib.util
    spec = importlib.util.spec_from_file_location("st_build", os.path.join(ROOT, "statetree-representation_b200", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def _built():
    from statetree_b200 import ops
    if not os.path.exists(ops.LIB_PATH):
        _build_module().build_library()
    return ops


def test_library_exports_header_symbols():
    ops = _built()
    with open(os.path.join(ROOT, "include", "statetree_b200.h")) as f:
        text = f.read()
    declared = set(re.findall(r"\b(st_[a-z0-9_]+)\s*\(", text))
    assert declared == set(ops.exported_symbols()), declared ^ set(ops.exported_symbols())
    L = ops.lib()                                       # resolves every symbol, checks the ABI version
    assert L.st_abi_version() == ops.ABI
    assert L.st_kv_page_bytes(1) == 6400 and L.st_kv_page_bytes(8) == 51200


def test_argument_errors_are_reported_without_a_gpu():
    ops = _built()
    L = ops.lib()
    assert L.st_dec(None, None, None, 17, 64, None, None) != 0
    assert b"M % 16" in L.st_last_error()
    assert L.st_gemv(None, None, None, None, None, None, None, 33, 16, 64, None, 0, None, None) != 0
    assert b"batch" in L.st_last_error()
    assert L.st_gemm(None, None, None, None, None, None, 64, 64, 64, None, 0, None, None) != 0
    assert L.st_gemv_workspace_bytes(100, 64, 1) == -1
    # the exchange entry points check rank / world and sizes before anything touches a GPU
    assert L.st_comm_bytes() == 8 * 64 * 4 + 64 * 4 + 256 + 2 * 8 * 64 * 16384 + 2 * 8 * (128 << 10) * 4
    assert L.st_gemv_allreduce(None, 0, 9, None, None, None, None, None, None, None, 1, 64, 64, None, 0, None) != 0
    assert b"ranks" in L.st_last_error()
    assert L.st_gemm_list(0, None, None, None, None, None, None, 1, None, 64, None, None) != 0
    assert L.st_gemv_list(5, None, None, None, None, None, None, None, 1, None, 64, None, 0, None) != 0
    assert b"1 to 4" in L.st_last_error()
    assert L.st_comm_set_timeout_ms(0) != 0
    assert L.st_allreduce(None, 0, 1, None, None, 8, None) != 0
    assert b"ranks" in L.st_last_error()
    assert L.st_allreduce_add_rmsnorm(None, 3, 2, None, None, None, None, 1, 4096, 1e-6, None) != 0
    assert L.st_moe_align(None, 1, 0, 8, 8, 8, None, None, None, 4, None) != 0
    assert L.st_moe_align(None, 1, 8, 2048, 2048, 8, None, None, None, 16, None) != 0 and b"experts" in L.st_last_error()
    assert L.st_moe_group_gemm(None, None, None, 4, None, None, None, None, 4, 32, None, None, 8, 128, 64, None) != 0
    assert b"block size" in L.st_last_error()


@pytest.mark.parametrize("M,N,B,slots", [(1024, 4096, 1, 5), (1024, 4096, 8, 5), (512, 2048, 1, 3), (256, 8192, 4, 9)])
def test_row_parallel_plan_cuts_tiles_down_to_two_units(M, N, B, slots):
    """the row-parallel GEMV keeps the grid it was measured with on several GPUs (no CTA below two units): without a workspace
    the call is refused before anything is launched, and names the exchange slots of that grid (slots per tile, of 16 x 8
    words each); st_gemv_workspace_bytes covers them"""
    import ctypes
    ops = _built()
    L = ops.lib()
    p = ctypes.c_void_p(4096)
    need = M // 16 * slots * 16 * 8 * 4
    assert L.st_gemv_allreduce((ctypes.c_void_p * 2)(4096, 4096), 0, 2, p, p, p, p, p, p, None, B, M, N, None, 0, None) != 0
    assert f"workspace of {need} bytes needed".encode() in L.st_last_error(), L.st_last_error()
    assert L.st_gemv_workspace_bytes(M, N, B) >= need


def test_cpu_tensors_are_rejected():
    import torch
    ops = _built()
    with pytest.raises(RuntimeError):
        ops.ext().dec(torch.zeros(1, 1, 1552, dtype=torch.uint8), torch.zeros(2, dtype=torch.int32),
                      torch.zeros(1, dtype=torch.int32), torch.zeros(16, 64, dtype=torch.bfloat16))


def test_package_exports_the_reference_names():
    """`import statetree_b200 as statetree` keeps a caller's lines: the names statetree/__init__.py:10-17 exports"""
    import statetree_b200 as S
    names = ["TreeLinear", "TreeSlice", "TreeEmbedding", "TreeExperts", "DEFAULT_FUSE", "convert", "prepare",
             "save_pretrained", "load_pretrained", "size_report", "tree_modules", "encode", "decode_reference"]
    assert sorted(S.__all__) == sorted(names)
    for n in names:
        assert hasattr(S, n), n
    assert S.DEFAULT_FUSE["qkv_proj"] == ("q_proj", "k_proj", "v_proj")


def test_install_as_makes_the_reference_imports_resolve_here():
    import importlib
    import sys
    import statetree_b200 as S
    try:
        S.install_as("statetree_alias_for_test")
        import statetree_alias_for_test as A                      # noqa: F401
        from statetree_alias_for_test.linear import TreeLinear
        assert A is S and TreeLinear is S.TreeLinear
        assert importlib.import_module("statetree_alias_for_test.ops").ext is S.ops.ext
        assert importlib.import_module("statetree_alias_for_test._vllm").StateTreeLinearMethod is not None
        sys.modules["taken_name_for_test"] = sys
        with pytest.raises(RuntimeError, match="already imported"):
            S.install_as("taken_name_for_test")
    finally:
        for k in [k for k in sys.modules if k.startswith("statetree_alias_for_test") or k == "taken_name_for_test"]:
            del sys.modules[k]


def test_library_alone_is_enough(monkeypatch):
    """a tree with the kernel library and without the native host path of module calls: no error, the calls go out from Python"""
    ops = _built()
    monkeypatch.setattr(ops, "CALLS_PATH", "/nonexistent/_calls.so")
    monkeypatch.setattr(ops, "_CALLS", None)
    assert ops.calls() is None and ops.built()
    assert ops.calls() is None                          # (and when asked again)


def test_native_calls_are_compiled_again(monkeypatch, tmp_path):
    """_calls.so is up to date only for the sources, the C header, the torch and the Python that it was compiled with"""
    import torch
    mod, compiled = _build_module(), []
    src, header = tmp_path / "pkg" / "csrc" / "py_calls.cpp", tmp_path / "include" / "statetree_b200.h"
    for f in (src, header):
        f.parent.mkdir(parents=True)
        f.write_text("")
        os.utime(f, (1000, 1000))
    for name, path in (("HERE", tmp_path / "pkg"), ("CSRC", src.parent), ("OBJ", tmp_path), ("CALLS", tmp_path / "_calls.so"),
                       ("CALLS_FOR", tmp_path / "_calls.txt")):
        monkeypatch.setattr(mod, name, str(path), raising=False)

    def run(cmd, **kw):
        compiled.append(cmd)
        (tmp_path / "_calls.so").write_bytes(b"")
        os.utime(mod.CALLS, (2000 + len(compiled),) * 2)
        return type("Result", (), {"returncode": 0})

    monkeypatch.setattr(mod.subprocess, "run", run)

    def builds():
        before = len(compiled)
        mod.build_calls()
        return len(compiled) - before

    assert (builds(), builds()) == (1, 0)
    for i, f in enumerate((src, header)):
        os.utime(f, (2001.5 + i,) * 2)
        assert (builds(), builds()) == (1, 0), f
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert (builds(), builds()) == (1, 0)


def test_native_calls_of_another_abi_are_not_used(monkeypatch):
    ops = _built()
    if not os.path.exists(os.path.join(os.path.dirname(ops.LIB_PATH), "_calls.so")):
        _build_module().build_calls()
    ops.lib()
    monkeypatch.setattr(ops, "_CALLS", None)
    assert ops.calls() is not None
    monkeypatch.setattr(ops, "_CALLS", None)
    monkeypatch.setattr(ops, "ABI", ops.ABI + 1)
    with pytest.warns(UserWarning, match="another torch or C ABI"):
        assert ops.calls() is None
