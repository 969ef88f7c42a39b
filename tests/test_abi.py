"""The C-ABI library builds, loads, and exports exactly what include/b200decode.h declares (no GPU needed:
nothing here launches a kernel)."""
import ctypes
import re
from pathlib import Path

import pytest

from llm_decode_kernels_b200 import ext

HEADER = Path(__file__).resolve().parents[1] / "include" / "b200decode.h"


def declared_functions():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return re.findall(r"\b(b200_\w+)\s*\(", text)


def test_header_declares_the_six_reference_ops():
    names = set(declared_functions())
    for op in ("gemv_w4a16", "bw_read", "paged_attention", "add_rmsnorm", "swiglu", "rope_append"):
        assert f"b200_{op}" in names


def test_library_exports_every_declared_symbol():
    lib = ext.load_library()
    for name in declared_functions():
        assert hasattr(lib, name), f"{name} is declared in b200decode.h but not exported"
    assert lib.b200_version() >= 100
    assert lib.b200_strerror(-1).decode().startswith("bad argument")


def test_python_signatures_cover_the_header():
    names = set(declared_functions()) - {"b200_version", "b200_strerror", "b200_last_cuda_error", "b200_decode_step",
                                         "b200_decode_step_xchg_bytes", "b200_tp_gemv_slot_bytes",
                                         "b200_gemv_w4a16_tiled_bytes"}   # declared on their own
    assert names == set(ext.SIGNATURES), names ^ set(ext.SIGNATURES)
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    for name, argtypes in ext.SIGNATURES.items():
        m = re.search(name + r"\s*\((.*?)\)\s*;", text, flags=re.S)
        assert m, name
        assert len([a for a in m.group(1).split(",") if a.strip() not in ("", "void")]) == len(argtypes), name


def test_exchange_sizes_are_host_arithmetic():
    """Sizes a caller allocates from: the persistent step's exchange area (per layer qkv, J partial attention outputs
    and their log-sum-exp words, o, act, down; J = min(4, grid / n_q) context slices per query head) and the
    tensor-parallel GEMV region (control, reserved flag rows, W x N tagged words)."""
    lib = ext.load_library()
    L, H, I, n_q, n_kv, D, grid = 22, 2048, 5632, 32, 4, 64, 148           # TinyLlama shape on a B200: J = 4
    per_layer = (n_q + 2 * n_kv) * D + 4 * n_q * D + n_q * 8 + H + I + H
    assert lib.b200_decode_step_xchg_bytes(L, H, I, n_q, n_kv, D, grid) == (L * per_layer + grid * 4) * 4
    per_layer_1 = (64 + 2 * 8) * 128 + 2 * 64 * 128 + 64 * 4 + 8192 + 28672 + 8192      # 64 heads on 148 CTAs: J = 2
    assert lib.b200_decode_step_xchg_bytes(1, 8192, 28672, 64, 8, 128, grid) == (per_layer_1 + grid * 4) * 4
    assert lib.b200_decode_step_xchg_bytes(L, H, I, n_q, n_kv, D, 0) == 0
    assert lib.b200_tp_gemv_slot_bytes(8192, 8) == 256 + 1024 * 16 * 4 + 8 * 8192 * 4


def test_bad_arguments_are_refused_on_the_host():
    """Argument checks run before any CUDA call, so they can be exercised without a device."""
    lib = ext.load_library()
    assert lib.b200_gemv_w4a16(2, 0, 0, 0, None, None, None, None, 4, 128, 7, None) == -1       # null pointers
    buf = ctypes.create_string_buffer(64)
    p = ctypes.addressof(buf)
    p16 = (p + 15) & ~15
    assert lib.b200_gemv_w4a16(2, 0, 0, 0, p16, p16, p16, p16, 4, 100, 7, None) == -3           # K % 32 != 0
    assert lib.b200_gemv_w4a16(2, 0, 0, 0, p16, p16, p16, p16, 4, 128, 4, None) == -3           # group 16 < 32
    assert lib.b200_gemv_w4a16(2, 0, 0, 0, p16 + 4, p16, p16, p16, 4, 128, 7, None) == -2       # misaligned weights
    assert lib.b200_add_rmsnorm(p16, None, p16, p16, 12, 1e-5, None) == -3                      # H % 8 != 0
    peers = (ctypes.c_void_p * 2)(p16, p16)
    assert lib.b200_tp_allreduce_add_rmsnorm(peers, 2, 2, 256, p16, p16, p16, 64, 1e-5, None) == -1   # rank >= W
    assert lib.b200_tp_allreduce_add_rmsnorm(peers, 0, 2, 64, p16, p16, p16, 64, 1e-5, None) == -2    # inside header
    assert lib.b200_tp_allreduce_add_rmsnorm(peers, 0, 2, 256, p16, p16, p16, 60, 1e-5, None) == -3   # H % 8 != 0
    assert lib.b200_tp_allgather(peers, 0, 17, 256, p16, 64, None) == -1                              # too many ranks
    assert lib.b200_comm_alloc(16, ctypes.byref(ctypes.c_void_p())) == -1                             # below the header
    assert lib.b200_comm_header_bytes() == 256
    assert lib.b200_add_rmsnorm(p16, None, p16, p16, 65536, 1e-5, None) == -5                   # H over capacity
    assert lib.b200_swiglu(p16, p16, 0, None) == -1
    assert lib.b200_embed_row(p16, p16, p16, 64, 0, None) == -1                                 # empty table
    assert lib.b200_gemv_w4a16_tune(1, 5632, 2048, 3, 148) == -1                                # ksplit not 1/2/4/8
    assert lib.b200_gemv_w4a16_tune(1, 5632, 2048, 4, 176) == 0 and lib.b200_gemv_w4a16_tune(1, 5632, 2048, 0, 0) == 0
    assert lib.b200_paged_attention(7, p16, p16, p16, p16, p16, 32, 4, 4, 64, 1, p16, p16, p16, p16, None) == -1
    assert lib.b200_paged_attention(2, p16, p16, p16, p16, p16, 12, 4, 4, 64, 1, p16, p16, p16, p16, None) == -3
    assert lib.b200_paged_attention_batched(p16, p16, p16, p16, 8, p16, 1, 32, 4, 96, 4, 64, 1, p16, p16, p16, p16,
                                            None) == -3                                         # head_dim 96


def test_python_face_refuses_cpu_tensors():
    import torch
    K = ext.load()
    x = torch.zeros(128, dtype=torch.float16)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        K.swiglu(torch.zeros(256, dtype=torch.float16), x)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        K.add_rmsnorm(x, None, x, x, 1e-5)


def test_native_call_path_mirrors_the_methods():
    """Every operator of the native call path takes the arguments of the method it stands in for, and hands what it does not
    accept to that method."""
    import inspect
    ops = ext.Ops(ext.load_library())
    from llm_decode_kernels_b200 import _host
    for name, (args, required) in _host.names()[1].items():
        params = list(inspect.signature(getattr(ext.Ops, name)).parameters.values())[1:]
        assert [p.name for p in params] == list(args), name
        assert sum(p.default is p.empty for p in params) == required, name
        assert getattr(ops, name).__doc__ == getattr(ext.Ops, name).__doc__
    with pytest.raises(RuntimeError, match="gu must be a contiguous CUDA tensor"):
        ops.swiglu(None, out=None)
    with pytest.raises(TypeError):
        ops.swiglu(1, 2, 3)
    with pytest.raises(TypeError):
        ops.swiglu(gu=1, nonsense=2)


def test_descriptors_have_the_fields_of_the_header():
    """Same fields in the same order; and b200_step_desc ends where callers built against the first headers have it end."""
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    for cls, name in ((ext.StepLayer, "b200_step_layer"), (ext.StepDesc, "b200_step_desc"), (ext.PrefillDesc, "b200_prefill_desc")):
        body = next(b for b, n in re.findall(r"typedef struct\s*\w*\s*\{([^{}]*)\}\s*(\w+);", text) if n == name)
        fields = [re.sub(r"\[.*?\]", "", f).split()[-1].lstrip("*") for line in body.split(";") for f in line.split(",") if f.strip()]
        assert fields == [f[0] for f in cls._fields_], name
    assert ext.StepDesc._fields_[-1][0] == "trace" and ctypes.sizeof(ext.StepDesc) == 168


def test_native_call_path_leaves_overrides_and_stand_ins_alone():
    """A subclass's method, and whatever stands in for the library, are what a call reaches."""
    import torch
    real = ext.load_library()
    calls = []

    class Counting(ext.Ops):
        def swiglu(self, gu, out):
            calls.append("swiglu")
    Counting(real).swiglu(1, 2)
    assert calls == ["swiglu"]

    class StandIn:
        def __getattr__(self, name):
            return lambda *a: calls.append(name) or 0
    ops = ext.Ops(real)
    native = type(ops.swiglu)
    assert native.__name__ == "operator" and isinstance(ops.add_rmsnorm, native)
    ops.lib = StandIn()
    assert not isinstance(ops.swiglu, native) and ops.lib.b200_swiglu() == 0 and calls[-1] == "b200_swiglu"
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        ops.swiglu(torch.zeros(16), torch.zeros(8))
    ops.lib = real
    assert isinstance(ops.swiglu, native)
    assert not isinstance(ext.Ops(StandIn()).swiglu, native)
    other = ext.Ops(real)                 # one object's binding is not another's
    ops.lib = StandIn()
    assert isinstance(other.swiglu, native)


def test_operators_do_without_the_native_call_path(monkeypatch):
    """No compiler, no headers: one warning, and every operator in its ctypes form."""
    import warnings
    from llm_decode_kernels_b200 import build as B
    real = ext.load_library()

    def no_compiler(*a, **k):
        raise RuntimeError("no compiler")
    monkeypatch.setattr(ext, "_HOST", None)
    monkeypatch.setattr(B, "build_host", no_compiler)
    with pytest.warns(RuntimeWarning, match="no compiler"):
        ops = ext.Ops(real)
    assert ops.swiglu.__func__ is ext.Ops.swiglu
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        ext.Ops(real)


def test_native_call_path_is_made_for_what_loads_it(monkeypatch, tmp_path):
    """Another torch, source or header has another file; the build puts a whole file in place and leaves nothing else behind."""
    import torch
    from llm_decode_kernels_b200 import build as B
    here = B.host_path()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert B.host_path() != here
    monkeypatch.undo()
    src = tmp_path / "host_ops.cpp"
    src.write_bytes(B.HOST_SRC.read_bytes() + b"\n")
    monkeypatch.setattr(B, "HOST_SRC", src)
    assert B.host_path() != here
    monkeypatch.undo()
    monkeypatch.setattr(B, "PKG", tmp_path)
    (tmp_path / "_host_0123456789abcdef.so").write_bytes(b"made for something else")
    out = B.build_host()
    assert out.parent == tmp_path and [p.name for p in tmp_path.glob("*host*.so")] == [out.name] and not list(tmp_path.glob(".*"))
