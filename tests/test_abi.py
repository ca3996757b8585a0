"""The C-ABI library loads on a machine without a GPU and exports every declared symbol."""
import ctypes
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def library():
    from texelator_b200.cuda.build import build
    from texelator_b200 import runtime
    return runtime.load_library(build())


def test_every_declared_symbol_is_exported(library):
    from texelator_b200 import runtime
    header = (ROOT / "include" / "texelator_b200.h").read_text()
    declared = set(re.findall(r"\b(tx_[a-z_0-9]+)\s*\(", header))
    assert declared, "header declares no entry points"
    assert declared == set(runtime.C_API), (declared ^ set(runtime.C_API))
    for name in declared:
        assert getattr(library, name) is not None


def test_header_cites_the_reference_interface():
    header = (ROOT / "include" / "texelator_b200.h").read_text()
    for needle in ("extension.cpp", "texelator_cuda.cu:1260-1327", "texelator_cuda.cu:1329-1469",
                   "texelator_cuda.cu:1471-1478", "texelator_cuda.cu:1540-1595"):
        assert needle in header


def test_calls_without_a_gpu_fail_with_a_message(library):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    assert library.tx_set_lookahead(0, 2) != 0
    assert b"null Texelator handle" in library.tx_last_error()
    out = ctypes.c_uint64(0)
    blocks = (ctypes.c_uint8 * 64)()
    scales = (ctypes.c_float * 1)(1.0)
    status = library.tx_pack_encoded(blocks, 64, scales, 1, None, 1, 0, ctypes.byref(out))
    assert status != 0 and library.tx_last_error()      # no device: a CUDA error, never a CPU fallback
    assert library.tx_launch_count() == 0


@pytest.mark.parametrize("shifted", [0, 1, 2, 6, 7])
def test_prompt_append_refuses_pointers_off_a_16_byte_boundary(library, shifted):
    """Its loads and stores are 16 bytes wide; the check comes before any launch, so no device is needed."""
    pointers = [4096 + (4 if index == shifted else 0) for index in range(8)]
    qkv, cos, sin, k_cache, v_cache = pointers[0], pointers[1], pointers[2], pointers[6], pointers[7]
    assert library.tx_aux_rope_append_prompt(qkv, cos, sin, 0, 0, k_cache, v_cache, 1, 1, 16, 1, None) == -1
    assert b"16-byte aligned" in library.tx_last_error()


def test_operator_refuses_cpu_tensors():
    import torch
    from texelator_b200 import runtime
    ext = runtime.extension()
    with pytest.raises(RuntimeError, match="null Texelator handle"):
        ext.linear(1234, torch.zeros(1, 16, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="at least one texture handle"):
        runtime.TexelatorLinear([])


@pytest.mark.parametrize("number", ["np.int64(5)", "np.uint64(5)", "None", "1.5", "-3", "2 ** 70", "'a'"])
def test_unknown_handle_numbers_are_null_handles(number):
    """An integer of any kind is a handle number; what names no handle is refused as the null handle is."""
    import numpy as np
    import torch
    from texelator_b200 import runtime
    with pytest.raises(RuntimeError, match="null Texelator handle"):
        runtime.extension().linear(eval(number, {"np": np}), torch.zeros(1, 16, dtype=torch.bfloat16))


def test_handle_numbers_of_numpy_are_known():
    import numpy as np
    import torch
    from texelator_b200 import runtime
    ext = runtime.extension()
    ext._remember(1 << 40, 32, 64, 0)
    try:
        with pytest.raises(RuntimeError, match="contiguous CUDA"):      # the handle is found, the CPU tensor refused
            ext.linear(np.int64(1 << 40), torch.zeros(1, 64, dtype=torch.bfloat16))
    finally:
        ext._forget(1 << 40)


def test_operator_refuses_tensors_without_memory():
    """Fake tensors pass for CUDA tensors; a view of one even has a nonzero address (its offset)."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from texelator_b200 import runtime
    ext = runtime.extension()
    handle = 1 << 40                                        # never dereferenced: the call is refused before
    ext._remember(handle, 32, 64, 0)
    try:
        with FakeTensorMode():
            x = torch.empty(4, 64, device="cuda", dtype=torch.bfloat16)
            y = torch.empty(4, 32, device="cuda", dtype=torch.bfloat16)
        for rows in (slice(0, 4), slice(1, 4)):
            with pytest.raises(RuntimeError, match="contiguous CUDA FP16 or BF16"):
                ext.linear(handle, x[rows])
            with pytest.raises(RuntimeError, match="contiguous CUDA FP16 or BF16"):
                ext.linear_out(handle, x[rows], y[rows])
    finally:
        ext._forget(handle)


def test_output_form_refuses_zero_tokens():
    """``linear`` returns an empty tensor for no tokens; with an output of its own the caller must have some."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from texelator_b200 import runtime
    ext = runtime.extension()
    ext._remember(1 << 40, 32, 64, 0)
    try:
        with FakeTensorMode():
            x = torch.empty(0, 64, device="cuda", dtype=torch.bfloat16)
            y = torch.empty(0, 32, device="cuda", dtype=torch.bfloat16)
        with pytest.raises(RuntimeError, match="contiguous CUDA FP16 or BF16"):
            ext.linear_out(1 << 40, x, y)
    finally:
        ext._forget(1 << 40)


def test_binding_for_another_torch_is_refused(monkeypatch):
    import torch
    from texelator_b200 import runtime
    assert runtime.load_binding().built_for.startswith(f"torch {torch.__version__}, Python 3.")
    monkeypatch.setattr(torch, "__version__", "1.0")
    with pytest.raises(ImportError, match="was built for torch"):
        runtime.load_binding()


@pytest.mark.parametrize("reason", ["absent", "another torch"])
def test_library_without_a_usable_binding_still_loads(monkeypatch, tmp_path, reason):
    """A prebuilt library alone, or beside a binding for another torch, serves the operator through ctypes."""
    import torch
    from texelator_b200 import runtime
    runtime.extension()                                     # both files exist from here on
    monkeypatch.setenv("TEXELATOR_DISABLE_JIT", "1")
    monkeypatch.setattr(runtime, "_EXTENSION", None)
    if reason == "absent":
        monkeypatch.setattr(runtime, "BINDING_PATH", tmp_path / "_tx_torch.so")
    else:
        monkeypatch.setattr(torch, "__version__", "1.0")
    with pytest.warns(RuntimeWarning, match="through ctypes"):
        ext = runtime.extension()
    x = torch.zeros(1, 64, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="null Texelator handle"):
        ext.linear(1 << 40, x)
    ext._remember(1 << 40, 32, 64, 0)
    with pytest.raises(RuntimeError, match="contiguous CUDA FP16 or BF16"):
        ext.linear(1 << 40, x)
    ext._forget(1 << 40)


def test_no_product_code_imports_the_oracle():
    for path in list((ROOT / "texelator_b200").rglob("*.py")) + list((ROOT / "texelator_b200").rglob("*.cu")):
        text = path.read_text()
        assert "oracle" not in text.replace("oracle/bc4_oracle.py", ""), path


def test_unknown_handles_take_no_staged_activations():
    """The library reads what a handle number points to, so a number that names none must not reach it."""
    from texelator_b200 import runtime
    assert runtime.extension().takes_staged(1234, 16) is False


def test_staged_calls_refuse_what_they_cannot_read():
    """Buffers of another device or type, short ones and unknown handles are refused before anything is launched."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from texelator_b200 import runtime
    ext = runtime.extension()
    handle = 1 << 40                                        # never dereferenced
    ext._remember(handle, 32, 64, 0)
    try:
        with FakeTensorMode():
            cuda = dict(device="cuda")
            y, rows, gate_up = (torch.empty(4, n, dtype=torch.bfloat16, **cuda) for n in (32, 64, 128))
            staged, weight = torch.empty(ext.staged_bytes(64, 4), dtype=torch.uint8, **cuda), torch.empty(64, dtype=torch.bfloat16, **cuda)
            short, words, strided = staged[:-4], torch.empty(1 << 20, dtype=torch.int32, **cuda), torch.empty(1 << 20, dtype=torch.uint8, **cuda)[::2]
        with pytest.raises(RuntimeError, match="null Texelator handle"):
            ext.linear_staged(1234, staged, y)
        with pytest.raises(RuntimeError, match="input shape/device mismatch"):
            ext.linear_staged(handle, staged, torch.empty(4, 32, dtype=torch.bfloat16))
        calls = (lambda s: ext.linear_staged(handle, s, y), lambda s: ext.add_rmsnorm_staged(rows, None, weight, s, 1e-6),
                 lambda s: ext.silu_mul_pairs_staged(gate_up, s))
        for call in calls:
            with pytest.raises(RuntimeError, match="too small"):
                call(short)
            for wrong in (torch.empty(1 << 20, dtype=torch.uint8), words, strided):
                with pytest.raises(RuntimeError, match="contiguous uint8 tensor on the CUDA device"):
                    call(wrong)
    finally:
        ext._forget(handle)


def test_embedding_norm_refuses_what_it_cannot_read():
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from texelator_b200 import runtime
    ext = runtime.extension()
    with FakeTensorMode():
        cuda, bf = dict(device="cuda"), dict(device="cuda", dtype=torch.bfloat16)
        table, ids, h, weight, y = torch.empty(50, 64, **bf), torch.empty(3, dtype=torch.int64, **cuda), torch.empty(3, 64, **bf), torch.empty(64, **bf), torch.empty(3, 64, **bf)
        short, narrow, few, wrong, flipped = ids[:2], torch.empty(3, dtype=torch.int32, **cuda), torch.empty(50, 32, **bf), table.float(), torch.empty(64, 50, **bf).t()
    for tokens in (short, narrow):
        with pytest.raises(RuntimeError, match="one int64 token a row"):
            ext.embed_rmsnorm(table, tokens, h, weight, y, 1e-6)
    for other in (few, wrong, flipped):
        with pytest.raises(RuntimeError, match="the table is contiguous BF16"):
            ext.embed_rmsnorm(other, ids, h, weight, y, 1e-6)
    for other in ((table, torch.zeros(3, dtype=torch.int64), h), (torch.zeros(50, 64, dtype=torch.bfloat16), ids, h)):
        with pytest.raises(RuntimeError, match="on one CUDA device"):
            ext.embed_rmsnorm(other[0], other[1], other[2], weight, y, 1e-6)
