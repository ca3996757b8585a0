"""The native operator call, the tile that a handle without a tuned backend takes, prompt rows through the library's
kernels, and encoder rows whose block count is not a multiple of the lanes that share a row."""
import numpy as np
import pytest
import torch

from oracle import bc4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    from texelator_b200 import runtime
    return runtime.extension()


def _encoded(m, k, seed, lut):
    gen = torch.Generator().manual_seed(seed)
    w = torch.randn(m, k, generator=gen) * 0.05
    blocks, scales = O.encode_linear(w, torch.ones(k), lut)
    return blocks, scales, gen


def test_native_call_checks_and_keywords(ext, lut):
    blocks, scales, gen = _encoded(48, 64, 1, lut)
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales))
    x = torch.randn(3, 2, 64, generator=gen).cuda().bfloat16()
    y = ext.linear(handle=h, x=x)
    assert y.shape == (3, 2, 48) and y.dtype == x.dtype
    out = torch.empty_like(y)
    assert ext.linear_out(h, x, y=out) is out and torch.equal(out, y)
    assert ext.linear(h, x[:0]).shape == (0, 2, 48)
    for bad, message in ((x.float(), "contiguous CUDA FP16 or BF16"), (x.transpose(0, 1), "contiguous CUDA FP16 or BF16"),
                         (x.cpu(), "contiguous CUDA FP16 or BF16"), (x[..., :32].contiguous(), "shape/device mismatch")):
        with pytest.raises(RuntimeError, match=message):
            ext.linear(h, bad)
    with pytest.raises(RuntimeError, match="shape/device mismatch"):
        ext.linear_out(h, x, out[:2])
    with pytest.raises(TypeError):
        ext.linear(h)
    ext.free(h)
    with pytest.raises(RuntimeError, match="null Texelator handle"):
        ext.linear(h, x)
