"""The native operator call, the tile that a handle without a tuned backend takes, prompt rows through the library's
kernels, and encoder rows whose block count is not a multiple of the lanes that share a row."""
import numpy as np
import pytest
import torch

from graph_kernels import launched
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


def test_native_call_goes_to_the_library_that_packed_the_handle(ext, lut):
    """Two loaded libraries (the second one a stand-in that launches nothing) serve their own handles."""
    import ctypes
    from types import SimpleNamespace
    from texelator_b200 import runtime
    blocks, scales, gen = _encoded(48, 64, 1, lut)
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales))
    x = torch.randn(3, 64, generator=gen).cuda().bfloat16()
    before, calls = ext.linear(h, x), []
    entry = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p)
    stand_in = SimpleNamespace(tx_linear=entry(lambda *arguments: calls.append(arguments) or 0),
                               tx_last_error=ctypes.CFUNCTYPE(ctypes.c_char_p)(lambda: b"stand-in"))
    other = runtime._Extension(stand_in, runtime.load_binding())
    other._remember(1 << 40, 32, 64, x.get_device())
    assert other.linear(1 << 40, x).shape == (3, 32)
    assert len(calls) == 1 and calls[0][:2] == (1 << 40, x.data_ptr()) and calls[0][3:5] == (3, 1)
    assert torch.equal(ext.linear(h, x), before) and len(calls) == 1
    other._forget(1 << 40)
    ext.free(h)


def test_call_without_the_binding_gives_the_same_outputs(ext, lut):
    import numpy as np
    from texelator_b200 import runtime
    blocks, scales, gen = _encoded(48, 64, 1, lut)
    plain = runtime._Extension(ext._lib)
    h = plain.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales))
    ext._remember(h, *plain._shapes[h])
    for tokens in (1, 3, 40):
        for dtype in (torch.bfloat16, torch.float16):
            x = torch.randn(tokens, 64, generator=gen).cuda().to(dtype)
            out = torch.empty(tokens, 48, device="cuda", dtype=dtype)
            assert torch.equal(plain.linear(h, x), ext.linear(h, x))
            assert plain.linear_out(np.uint64(h), x, out) is out and torch.equal(out, ext.linear(np.uint64(h), x))
    for one in (plain, ext):
        assert one.linear(h, x[:0]).shape == (0, 48)
        with pytest.raises(RuntimeError, match="contiguous CUDA FP16 or BF16"):
            one.linear_out(h, x[:0], out[:0])
    ext._forget(h)
    plain.free(h)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [16, 64, 65, 128, 129, 400])
def test_untuned_handle_matches_oracle(ext, lut, tokens, dtype):
    m, k = 200, 656
    blocks, scales, gen = _encoded(m, k, tokens, lut)
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales))
    x = torch.randn(tokens, k, generator=gen).cuda().to(dtype)
    y = ext.linear(h, x).float().cpu().numpy()
    xs = x.float().cpu().numpy()
    ref = O.linear_bf16(xs, blocks, scales, lut) if dtype == torch.bfloat16 else O.linear_f16(xs, blocks, scales, lut)
    # weights are not rounded to the activations' type here: 2^-9 (2^-12) per weight and output at most, in quadrature
    assert O.rel_rms(y, ref) <= (1e-2 if dtype == torch.bfloat16 else 2e-3)
    assert ext.handle_info(h)[4] == 0
    ext.free(h)


@pytest.mark.parametrize("tokens,first,q_heads,kv_heads,head_dim", [(1, 0, 4, 2, 128), (37, 5, 5, 1, 64), (130, 0, 16, 2, 128), (3, 61, 2, 2, 16)])
def test_rope_append_prompt(ext, tokens, first, q_heads, kv_heads, head_dim):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    max_len, half = first + tokens + 3, head_dim // 2
    qkv = torch.randn(tokens, (q_heads + 2 * kv_heads) * head_dim, device="cuda", generator=gen).bfloat16()
    angle = torch.rand(max_len, half, device="cuda", generator=gen) * 6.28
    cos, sin = angle.cos(), angle.sin()
    k_cache = torch.full((kv_heads, max_len, head_dim), 7.0, device="cuda", dtype=torch.bfloat16)
    v_cache = k_cache.clone()
    rows = qkv.float().view(tokens, -1, head_dim)
    c, s = cos[first:first + tokens, None], sin[first:first + tokens, None]
    x1, x2 = rows[..., :half], rows[..., half:]
    rotated = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).bfloat16()
    expected_v = qkv.view(tokens, -1, head_dim)[:, q_heads + kv_heads:].clone()
    ext.rope_append_prompt(qkv, cos, sin, first, k_cache, v_cache, q_heads, kv_heads, head_dim)
    got = qkv.view(tokens, -1, head_dim)
    # one bf16 rounding (2^-8 of the value at most between neighbours) of fp32 sums that may be contracted
    close = lambda a, b: torch.allclose(a.float(), b.float(), rtol=2 ** -7, atol=1e-5)
    assert close(got[:, :q_heads + kv_heads], rotated[:, :q_heads + kv_heads])
    assert torch.equal(got[:, q_heads + kv_heads:], expected_v)
    assert torch.equal(k_cache[:, first:first + tokens], got[:, q_heads:q_heads + kv_heads].transpose(0, 1))
    assert torch.equal(v_cache[:, first:first + tokens], expected_v.transpose(0, 1))
    assert bool((k_cache[:, :first] == 7).all()) and bool((v_cache[:, first + tokens:] == 7).all())
    with pytest.raises(RuntimeError, match="inside the cache"):
        ext.rope_append_prompt(qkv, cos, sin, max_len, k_cache, v_cache, q_heads, kv_heads, head_dim)


@pytest.mark.parametrize("m,k", [(1, 16), (5, 528), (3, 1040), (130, 3168), (9, 2064), (1, 17408), (8, 11200), (7, 2064 * 4), (300, 5136), (593, 4096)])
def test_encoder_ragged_rows_match_restatement(ext, lut, m, k):
    gen = torch.Generator().manual_seed(m + k)
    w = torch.randn(m, k, generator=gen) * torch.exp(4 * torch.randn(m, 1, generator=gen))
    w[w.abs() < 0.3 * w.abs().mean()] = 0
    hdiag = torch.exp(torch.randn(k, generator=gen))
    blocks, scales = ext.encode(w.cuda(), hdiag.cuda(), torch.from_numpy(lut).cuda())
    want_blocks, want_scales = O.encode_linear(w, hdiag, lut)
    assert np.array_equal(scales.cpu().numpy(), want_scales)
    assert np.array_equal(blocks.cpu().numpy(), want_blocks.reshape(-1))


@pytest.mark.parametrize("hardware", [False, True])
@pytest.mark.parametrize("tokens", [1, 9, 128])
def test_low_mode_entries_one_by_one(ext, lut, tokens, hardware):
    """Random endpoints, most blocks in the low mode, every selector; unit activations read single weights back."""
    rng = np.random.default_rng(tokens)
    m, k = 512, 128
    ends = rng.integers(-127, 128, (2, m, k // 16))
    low = rng.random((m, k // 16)) < 0.8
    e0, e1 = np.where(low, ends.min(0), ends.max(0)).astype(np.int8), np.where(low, ends.max(0), ends.min(0)).astype(np.int8)
    e1[:8] = e0[:8]
    blocks = O.pack_blocks(e0, e1, rng.integers(0, 8, (m, k // 16, 16)).astype(np.uint8))
    table = O.hardware_palette() if hardware else lut
    want = O.dequant_palette(blocks, m, table).reshape(m, k).astype(np.float64)
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.ones(m))
    ext.set_palette(h, 1 if hardware else 0)
    got = np.empty((m, k))
    for first in range(0, k, tokens):
        x = torch.zeros(tokens, k, dtype=torch.float16)
        columns = [c % k for c in range(first, first + tokens)]
        x[torch.arange(tokens), torch.tensor(columns)] = 1
        got[:, columns] = ext.linear(h, x.cuda()).float().cpu().numpy().T
    ext.free(h)
    # a low-mode weight: fp16 numerator (2^-11 of it, or half a subnormal step 2^-25 * 65536 / 889), then the fp16 output (2^-11);
    # under the texture palette the high mode rounds its two step sizes to fp16 as well (2^-10 of the steps' sum, at most 2, and
    # 3e-5 of the endpoints' widening)
    bound = np.abs(want) * 2.0 ** -10 + 3e-6 + (0 if not hardware else 2.0 ** -9 + 6e-5) * ~np.repeat(e0 <= e1, 16, 1)
    assert (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,k,backend", [(1, 16, 8), (33, 144, 9), (31, 400, 6), (300, 1680, 6), (450, 80, 7), (600, 912, 5), (18, 102416, 8)])
def test_staging_and_stage_ring_remainders(ext, lut, tokens, k, backend, dtype):
    """Token counts around every number of tokens a staging block takes, rows that fit its shared memory and one that does
    not, K of fewer units than the ring has stages and one past it, an odd number of 128-row blocks for the pair."""
    m = 300
    rng = np.random.default_rng(k)
    ends = np.sort(rng.integers(-127, 128, (2, m, k // 16)), 0)[::-1].astype(np.int8)
    blocks = O.pack_blocks(ends[0], ends[1], rng.integers(0, 8, (m, k // 16, 16)).astype(np.uint8))
    scales = (rng.random(m) + 0.5).astype(np.float32)
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales))
    ext.set_prefill(h, 1, 1024)
    ext.set_prefill_backend(h, backend)
    x = (torch.randn(tokens, k, generator=torch.Generator().manual_seed(tokens)) / k ** 0.5).cuda().to(dtype)
    y = ext.linear(h, x).double().cpu()
    assert ext.kernel_status() == 0
    w = torch.from_numpy(O.dequant_palette(blocks, m, lut).reshape(m, k)).double() * torch.from_numpy(scales).double()[:, None]
    want = x.double().cpu() @ w.T
    # exact products, fp32 sums, one rounding of the output (half a unit in its last place)
    assert float((y - want).norm() / want.norm()) <= (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12) + 1e-5
    ext.free(h)


@pytest.mark.parametrize("variant", ["bias", "fp16 bias", "texture palette", "low mode"])
@pytest.mark.parametrize("tokens,m,k", [(257, 300, 912), (600, 300, 912), (300, 130, 400)])
@pytest.mark.parametrize("backend", [5, 6])
def test_wide_tiles_with_remainders(ext, lut, backend, tokens, m, k, variant):
    """The 256-token tiles with partial token, row and column tiles: bias in both types, both palettes, low-mode blocks."""
    rng = np.random.default_rng(tokens + m)
    ends = np.sort(rng.integers(-127, 128, (2, m, k // 16)), 0)[::-1].astype(np.int8)
    ends[0] = np.maximum(ends[0], ends[1] + 1) if variant != "low mode" else ends[0]
    if variant == "low mode":
        swap = rng.random((m, k // 16)) < 0.3
        ends = np.where(swap, ends[::-1], ends).astype(np.int8)
    blocks = O.pack_blocks(ends[0], ends[1], rng.integers(0, 8, (m, k // 16, 16)).astype(np.uint8))
    scales = (rng.random(m) + 0.5).astype(np.float32)
    dtype = torch.float16 if variant == "fp16 bias" else torch.bfloat16
    bias = torch.from_numpy(rng.standard_normal(m)).to(dtype).cuda() if "bias" in variant else None
    table = O.hardware_palette() if variant == "texture palette" else lut
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales), bias)
    ext.set_palette(h, 1 if variant == "texture palette" else 0)
    ext.set_prefill_backend(h, backend)
    x = (torch.randn(tokens, k, generator=torch.Generator().manual_seed(tokens)) / k ** 0.5).cuda().to(dtype)
    y = ext.linear(h, x).double().cpu()
    ext.free(h)
    assert ext.kernel_status() == 0
    w = torch.from_numpy(O.dequant_palette(blocks, m, table).reshape(m, k)).double() * torch.from_numpy(scales).double()[:, None]
    want = x.double().cpu() @ w.T + (bias.double().cpu() if bias is not None else 0)
    # one rounding of the output (half a unit in its last place); the texture palette's step sizes and the low mode's entries
    # are fp16 (2^-10 and 2^-11 of a weight at most)
    weights = {"texture palette": 2.0 ** -10, "low mode": 2.0 ** -11}.get(variant, 0)
    assert float((y - want).norm() / want.norm()) <= (2.0 ** -12 if dtype == torch.float16 else 2.0 ** -9) + weights + 1e-5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [33, 40, 100])
def test_prompts_kept_on_the_decode_kernel(ext, lut, tokens, dtype):
    """More tokens than one of its passes takes, with the threshold above them."""
    blocks, scales, gen = _encoded(200, 656, tokens, lut)
    h = ext.pack_encoded(torch.from_numpy(blocks).reshape(-1), torch.from_numpy(scales))
    ext.set_prefill(h, tokens + 1, 1024)
    x = torch.randn(tokens, 656, generator=gen).cuda().to(dtype)
    y, out = ext.linear(h, x), torch.empty(tokens, 200, dtype=dtype, device="cuda")
    names = [name for name, _ in launched(lambda: ext.linear_out(h, x, out))]
    assert len(names) > 1 and all("cluster_gemv_tile_kernel" in name for name in names)
    w = ext.dequant(h, 1).double()
    ext.free(h)
    want = x.double() @ w.T
    assert float((y.double() - want).norm() / want.norm()) <= (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12) + 1e-5
