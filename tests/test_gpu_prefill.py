"""GPU parity of the tensor-core prefill tiles and of the tuners (run with ``-m gpu``)."""
import re

import numpy as np
import pytest
import torch

from graph_kernels import launched
from oracle import bc4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200 import runtime
    return runtime.extension()


def _case(seed, m, k, tokens, lut, sparse=0.0, x_scale=1.0):
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((m, k)) * 0.02).astype(np.float32)
    if sparse:
        w[rng.random((m, k)) < sparse] = 0
    blocks, scales = O.encode_minmax(w, lut)
    x = torch.from_numpy((rng.standard_normal((tokens, k)) * x_scale).astype(np.float32)).bfloat16()
    return blocks, scales, x


def _pack(ext, blocks, scales, bias=None):
    return ext.pack_encoded(torch.from_numpy(blocks), torch.from_numpy(scales), bias)


@pytest.mark.parametrize("backend", [5, 6, 7, 8, 9])
@pytest.mark.parametrize("m,k,tokens", [(128, 128, 32), (256, 512, 40), (200, 48, 17), (1024, 1024, 128),
                                        (136, 2064, 300), (5120, 640, 512)])
def test_prefill_tiles_match_oracle(ext, lut, backend, m, k, tokens):
    blocks, scales, x = _case(m + k + tokens, m, k, tokens, lut)
    bias = torch.from_numpy(np.random.default_rng(2).standard_normal(m).astype(np.float32)).bfloat16().cuda()
    h = _pack(ext, blocks, scales, bias)
    try:
        ext.set_prefill(h, 16, 1024)
        ext.set_prefill_backend(h, backend)
        y = ext.linear(h, x.cuda())
        torch.cuda.synchronize()
        assert ext.kernel_status() == 0
        ref = O.linear_bf16(x.float().numpy(), blocks, scales, lut, bias=bias.float().cpu().numpy())
        err = O.rel_rms(y.float().cpu().numpy(), ref)
        assert err <= 1e-2, (backend, m, k, tokens, err)       # stated tolerance vs dequantise-then-matmul
    finally:
        ext.free(h)


def test_prefill_tiles_are_bitwise_identical(ext, lut):
    """The reference's admission rule (texelator/autotune.py:160-168)."""
    blocks, scales, x = _case(9, 384, 1024, 200, lut, x_scale=0.125)
    h = _pack(ext, blocks, scales)
    try:
        ext.set_prefill(h, 1, 32768)
        outs = []
        for backend in (5, 6, 7, 8, 9):
            ext.set_prefill_backend(h, backend)
            outs.append(ext.linear(h, x.cuda()))
        for other in outs[1:]:
            assert torch.equal(outs[0], other)
    finally:
        ext.free(h)


TILES = {5: (1, 256), 6: (2, 256), 7: (1, 128), 8: (1, 64), 9: (1, 192)}      # id -> CTAs per tile, tokens


def _tile_of(call):
    """(CTAs, tokens) of the one tile kernel a call launches, or None."""
    names = [re.search(r"prefill_umma_kernelILi(\d)ELi(\d+)E", name) for name, _ in launched(call)]
    found = [(int(match[1]), int(match[2])) for match in names if match]
    assert len(found) <= 1
    return found[0] if found else None


@pytest.mark.parametrize("tokens", [17, 600])
@pytest.mark.parametrize("backend", sorted(TILES))
def test_a_backend_id_launches_the_tile_it_names(ext, lut, backend, tokens):
    blocks, scales, x = _case(3, 300, 912, tokens, lut)
    h = _pack(ext, blocks, scales)
    try:
        ext.set_prefill_backend(h, backend)
        x, y = x.cuda(), torch.empty(tokens, 300, dtype=torch.bfloat16, device="cuda")
        assert _tile_of(lambda: ext.linear_out(h, x, y)) == TILES[backend]
        info = ext.kernel_info(backend)
        assert (info[5] // 128, info[6]) == TILES[backend]
    finally:
        ext.free(h)


def test_untuned_handle_takes_every_single_tile_somewhere(ext, lut):
    """Id 0 leaves the tile to the library; whichever it is, the output is the named tile's bit for bit."""
    rng = np.random.default_rng(8)
    m, k = 4250, 912
    ends = np.sort(rng.integers(-127, 128, (2, m, k // 16)), 0)[::-1].astype(np.int8)
    blocks = O.pack_blocks(ends[0], ends[1], rng.integers(0, 8, (m, k // 16, 16)).astype(np.uint8)).reshape(-1)
    h = _pack(ext, blocks, (rng.random(m) + 0.5).astype(np.float32))
    taken = set()
    try:
        for tokens in (16, 64, 160, 257, 600, 1000):
            x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens)).bfloat16()
            y = torch.empty(tokens, m, dtype=torch.bfloat16, device="cuda")
            ext.set_prefill_backend(h, 0)
            taken.add(_tile_of(lambda: ext.linear_out(h, x, y)))
            ext.linear_out(h, x, y)
            for backend in TILES:
                ext.set_prefill_backend(h, backend)
                assert torch.equal(ext.linear(h, x), y), (tokens, backend)
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert taken == {(1, 64), (1, 128), (1, 192), (1, 256)}
        assert taken <= set(TILES.values())
    finally:
        ext.free(h)


@pytest.mark.parametrize("m,k", [(512, 5120), (2048, 2048)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_untuned_prompt_is_as_close_to_64_bits_as_the_decode_kernel(ext, dtype, m, k):
    """The tile adds a K range in one fp32 accumulator where the decode kernel has sixteen: on Gaussian rows both end at
    the output's rounding (measured within 1e-4 of each other's distance; 1e-3 allowed)."""
    from texelator_b200 import runtime
    from texelator_b200.modeling import encode_minmax_cuda, software_palette_table
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    h = ext.pack_encoded_device(*encode_minmax_cuda(torch.randn(m, k, device="cuda", generator=gen) * 0.02, software_palette_table("cuda")))
    try:
        w = ext.dequant(h, runtime.DEQUANT_SCALED_F32).double()
        x = torch.randn(160, k, device="cuda", generator=gen).to(dtype)
        want = x.double() @ w.T
        distance = lambda y: float((y.double() - want).norm() / want.norm())
        tile = distance(ext.linear(h, x))
        ext.set_prefill(h, 1 << 30, 1024)
        streamed = distance(ext.linear(h, x))
        assert tile <= streamed * 1.001
        assert tile <= (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)        # half a unit in the last place
    finally:
        ext.free(h)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [1, 2, 8, 9, 15])
def test_untuned_handle_with_a_low_threshold(ext, lut, tokens, dtype):
    """Up to eight tokens the decode kernel serves the call as below a threshold, to the bit; from nine on a tile does."""
    blocks, scales, x = _case(5, 300, 912, tokens, lut)
    h = _pack(ext, blocks, scales)
    try:
        x, y = x.cuda().to(dtype), torch.empty(tokens, 300, dtype=dtype, device="cuda")
        streamed = ext.linear(h, x)
        ext.set_prefill(h, 1, 1024)
        assert (_tile_of(lambda: ext.linear_out(h, x, y)) is None) == (tokens <= 8)
        ext.linear_out(h, x, y)
        if tokens <= 8:
            assert torch.equal(y, streamed)
        # otherwise the same products in another order, then one rounding: neighbours (2^-8, 2^-11 of the value) at most
        assert float((y.double() - streamed.double()).norm() / streamed.double().norm()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
    finally:
        ext.free(h)


def test_prefill_low_mode_blocks(ext, lut):
    blocks, scales, x = _case(4, 256, 512, 64, lut, sparse=0.9)
    h = _pack(ext, blocks, scales)
    try:
        ext.set_prefill_backend(h, 6)
        y = ext.linear(h, x.cuda()).float().cpu().numpy()
        assert O.rel_rms(y, O.linear_bf16(x.float().numpy(), blocks, scales, lut)) <= 1e-2
    finally:
        ext.free(h)


def test_threshold_split_and_hybrid_agreement(ext, lut):
    """tokens < threshold streams through the decode GEMV, tokens >= threshold through the tile;
    both sides of the dispatcher agree within the reference's hybrid gate (rel-RMS <= 0.02,
    texelator/prefill.py:107)."""
    blocks, scales, x = _case(6, 512, 1024, 32, lut)
    h = _pack(ext, blocks, scales)
    try:
        ext.set_prefill_backend(h, 5)
        ext.set_prefill(h, 1 << 30, 1024)
        before = ext.launch_count()
        scalar = ext.linear(h, x.cuda()).float().cpu().numpy()
        ext.set_prefill(h, 1, 1024)
        hybrid = ext.linear(h, x.cuda()).float().cpu().numpy()
        assert ext.launch_count() > before
        assert O.rel_rms(hybrid, scalar) <= 0.02
    finally:
        ext.free(h)


def test_kernel_info_and_autotune_protocol(ext, lut, tmp_path, monkeypatch):
    from texelator_b200 import artifacts, autotune
    monkeypatch.setenv("TEXELATOR_HOME", str(tmp_path / "state"))
    for backend in (0, 5, 6, 7, 8, 9):
        info = ext.kernel_info(backend)
        assert len(info) == 9 and info[0] > 0 and info[8] >= 1
    entries = []
    for index, (m, k) in enumerate([(256, 512), (512, 256)]):
        blocks, scales, _ = _case(index, m, k, 1, lut)
        entries.append(artifacts.write_encoded_entry(tmp_path / "art" / "weights", f"model.layers.{index}.mlp.up_proj", index, blocks, scales))
    artifacts.write_artifact(tmp_path / "art", entries, O.palette_sha256(lut))
    profile = autotune.tune_artifact(tmp_path / "art", tmp_path / "profile.json", [32, 128], warmup=3, measured=10)
    assert profile["status"] == "complete" and len(profile["selections"]) == 4
    for record in profile["selections"].values():
        assert record["correctness_vs_baseline"][autotune.BASELINE]["bitwise_equal"]
        assert not record["rejected"]                          # every tile is bitwise identical to the baseline
    handles = []
    try:
        from texelator_b200 import runtime
        for entry in entries:
            handles.extend(runtime.pack_entry_handles(tmp_path / "art" / "weights", entry))
        assert autotune.apply_profile(handles, 100, profile) is True
        assert autotune.apply_profile(handles, 4000, profile) is False     # unknown bucket -> baseline tile
        assert ext.handle_info(handles[0])[2] == runtime.PREFILL_THRESHOLD  # threshold untouched
    finally:
        from texelator_b200 import runtime
        runtime.free(handles)


def test_lookahead_tuner_protocol(ext, lut, tmp_path, monkeypatch):
    from texelator_b200 import artifacts, tuning
    monkeypatch.setenv("TEXELATOR_HOME", str(tmp_path / "state"))
    entries = []
    for index, (m, k) in enumerate([(256, 512), (512, 256), (1024, 1024)]):
        blocks, scales, _ = _case(index, m, k, 1, lut)
        entries.append(artifacts.write_encoded_entry(tmp_path / "art" / "weights", f"model.layers.{index}.self_attn.q_proj", index, blocks, scales))
    artifacts.write_artifact(tmp_path / "art", entries, O.palette_sha256(lut))
    profile = tuning.tune_artifact(tmp_path / "art", warmup=2, measured=5, runs=2)
    assert profile["selected_lookahead"] in tuning.CANDIDATES
    assert [row["lookahead"] for row in profile["candidates"]] == list(tuning.CANDIDATES)
    assert all(row["max_abs_vs_k1"] <= 1e-3 for row in profile["candidates"])
    assert tuning.selected_lookahead(tmp_path / "art")[0] == profile["selected_lookahead"]
    # palette gate: an artefact encoded against an unknown palette is refused (texelator/tuning.py:38-41)
    artifacts.write_artifact(tmp_path / "art", entries, "0" * 64)
    with pytest.raises(RuntimeError, match="palette does not match"):
        tuning.tune_artifact(tmp_path / "art", warmup=1, measured=1, runs=1)
    # ... while the texture-unit palette the reference publishes is accepted where this GPU's texture
    # unit reproduces it, and such artefacts are packed in hardware-palette mode
    if ext.texture_supported() and O.palette_sha256(ext.palette_probe().numpy()) == O.REFERENCE_TEXTURE_PALETTE_SHA256:
        from texelator_b200 import runtime
        artifacts.write_artifact(tmp_path / "art", entries, O.REFERENCE_TEXTURE_PALETTE_SHA256)
        assert runtime.palette_of(tmp_path / "art" / "weights") == runtime.PALETTE_HARDWARE
        assert tuning.tune_artifact(tmp_path / "art", warmup=1, measured=2, runs=1)["palette_sha256"] == O.REFERENCE_TEXTURE_PALETTE_SHA256


def test_hardware_palettes_and_texture_gate(ext, lut, tmp_path, monkeypatch):
    from texelator_b200 import hardware
    monkeypatch.setenv("TEXELATOR_HOME", str(tmp_path / "state"))
    payload = hardware.doctor_payload(force=True)
    assert payload["palette_sha256"] == O.palette_sha256(lut)
    blocks, scales, x = _case(1, 64, 128, 1, lut)
    h = _pack(ext, blocks, scales)
    try:
        if payload["texture_views"] and not payload["texture_path_allowed"]:
            # texture unit palette differs from the encoder's palette -> ALU path stays in force
            with pytest.raises(RuntimeError, match="palette does not match"):
                ext.set_decode_path(h, 2)
            assert ext.handle_info(h)[5] == 0
    finally:
        ext.free(h)


@pytest.mark.parametrize("tokens,k,m", [(16, 256, 200), (17, 1168, 300), (33, 2048, 128), (700, 5120, 640), (1, 144, 64), (40, 16384, 128),
                                        (303, 2064, 64), (595, 4096, 64), (601, 8192, 64), (593, 8208, 64)])     # two rows a CTA, and one
def test_staged_activations_give_the_linear_of_their_rows(ext, lut, tokens, k, m):
    """A norm or a SwiGLU that writes the tile's form, then the tile: the bits of the rows' own linear, at edges of 128-column units and 32
    tokens, whichever tile; and refused where the linear would not take one."""
    blocks, scales, x = _case(k, m, k, tokens, lut)
    bias = torch.from_numpy(np.random.default_rng(2).standard_normal(m).astype(np.float32)).bfloat16().cuda()
    h = _pack(ext, blocks, scales, bias)
    try:
        gen = torch.Generator(device="cuda").manual_seed(k)
        weight, delta = torch.randn(k, device="cuda", generator=gen).bfloat16(), torch.randn(tokens, k, device="cuda", generator=gen).bfloat16()
        gate_up = (torch.randn(tokens, 2 * k, device="cuda", generator=gen) * 3).bfloat16()
        x[0] = 0
        x = x.cuda()
        ext.set_prefill(h, 1, 1024)
        staged = ext.staged_buffer(k, tokens, "cuda").fill_(0x7e)
        y = torch.empty(tokens, m, dtype=torch.bfloat16, device="cuda")
        for backend in (5, 6, 7, 8, 9):
            ext.set_prefill_backend(h, backend)
            assert ext.takes_staged(h, tokens)
            rows, residual, residual_staged = torch.empty_like(x), x.clone(), x.clone()
            ext.add_rmsnorm(residual, delta, weight, rows, 1e-6)
            ext.add_rmsnorm_staged(residual_staged, delta, weight, staged, 1e-6)
            assert torch.equal(residual, residual_staged)
            assert torch.equal(ext.linear_staged(h, staged, y), ext.linear(h, rows))
            for accurate in (False, True):
                ext.silu_mul_pairs(gate_up, rows, accurate)
                ext.silu_mul_pairs_staged(gate_up, staged, accurate)
                assert torch.equal(ext.linear_staged(h, staged, y), ext.linear(h, rows))
        ext.set_prefill(h, tokens + 1, 1024)
        assert not ext.takes_staged(h, tokens)
        with pytest.raises(RuntimeError, match="does not take staged"):
            ext.linear_staged(h, staged, y)
        assert ext.kernel_status() == 0
    finally:
        ext.free(h)


@pytest.mark.parametrize("tokens", [3073, 3112, 6200])
def test_staged_prompts_beyond_the_scratch_give_the_linear_of_their_rows(ext, lut, tokens):
    """The scratch holds 3072 tokens of 16384 columns, and rows beyond them are a chunk of their own, summed in other K ranges; a staged prompt,
    which needs no scratch, takes the same chunks."""
    m, k = 200, 16384
    blocks, scales, _ = _case(5, m, k, 1, lut)
    h = _pack(ext, blocks, scales)
    try:
        gen = torch.Generator(device="cuda").manual_seed(tokens)
        x, weight = torch.randn(tokens, k, device="cuda", generator=gen).bfloat16(), torch.randn(k, device="cuda", generator=gen).bfloat16()
        ext.set_prefill(h, 1, 1024)
        staged, rows = ext.staged_buffer(k, tokens, "cuda").fill_(0x7e), torch.empty_like(x)
        ext.add_rmsnorm(x.clone(), None, weight, rows, 1e-6)
        ext.add_rmsnorm_staged(x.clone(), None, weight, staged, 1e-6)
        y = torch.empty(tokens, m, dtype=torch.bfloat16, device="cuda")
        for backend in (5, 6, 7, 8, 9, 0):
            ext.set_prefill_backend(h, backend)
            assert torch.equal(ext.linear_staged(h, staged, y), ext.linear(h, rows)), backend
        assert ext.kernel_status() == 0
    finally:
        ext.free(h)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,k,tokens", [(128, 1024, 16), (132, 1024, 33), (130, 1040, 64), (257, 2064, 65), (1024, 4096, 127), (3000, 1536, 1),
                                        (4250, 2896, 29), (5120, 1024, 17), (2304, 8192, 40), (9216, 1024, 31), (9344, 1024, 31)])
def test_k_ranges_add_to_the_sums_of_their_columns(ext, lut, m, k, tokens, dtype):
    """K in two to eight ranges, added by a cluster where all clusters fit and by a second launch elsewhere (the pair tile): the same bits from
    every tile, and the 64-bit sums within the output's rounding and the fp32 adds."""
    blocks, scales, x = _case(m + k, m, k, tokens, lut)
    bias = torch.from_numpy(np.random.default_rng(2).standard_normal(m).astype(np.float32)).to(dtype).cuda()
    h = _pack(ext, blocks, scales, bias)
    try:
        from texelator_b200 import runtime
        x = x.cuda().to(dtype)
        ext.set_prefill(h, 1, 1024)
        outs = []
        for backend in (6, 5, 7, 8, 9):                       # the pair tile always adds by the second launch
            ext.set_prefill_backend(h, backend)
            outs.append(ext.linear(h, x))
        assert all(torch.equal(y, outs[0]) for y in outs[1:])
        want = x.double() @ ext.dequant(h, runtime.DEQUANT_SCALED_F32).double().T + bias.double()
        size = x.double().abs() @ ext.dequant(h, runtime.DEQUANT_SCALED_F32).double().abs().T + bias.double().abs()
        # half a unit of the output (2^-8 or 2^-11 of a value's power of two), and fp32 chains of k / 16 adds that may truncate (2^-23 of the
        # absolute sum each); 2^-24 is under fp16's smallest step
        half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        assert bool(((outs[0].double() - want).abs() <= half * want.abs() + k / 16 * 2.0 ** -23 * size + 2.0 ** -24).all())
        assert ext.kernel_status() == 0
    finally:
        ext.free(h)


@pytest.mark.parametrize("m,k,tokens", [(19072, 16, 17), (18945, 144, 64), (22016, 400, 65), (37889, 128, 33), (9600, 272, 200), (7000, 2080, 900)])
def test_two_tiles_an_sm_are_bitwise_the_tile_of_one(ext, lut, m, k, tokens):
    """Grids of more CTAs than SMs run the 64- and 128-token tiles as two small CTAs an SM (three and two stages): the bits of the wide tiles,
    with one unit, fewer units than stages, ragged rows and tokens."""
    rng = np.random.default_rng(m)
    ends = np.sort(rng.integers(-127, 128, (2, m, k // 16)), 0)[::-1].astype(np.int8)
    blocks = O.pack_blocks(ends[0], ends[1], rng.integers(0, 8, (m, k // 16, 16)).astype(np.uint8)).reshape(-1)
    h = _pack(ext, blocks, (rng.random(m) + 0.5).astype(np.float32))
    try:
        x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(k)).bfloat16()
        ext.set_prefill(h, 1, 1024)
        outs = []
        for backend in (5, 7, 8):
            ext.set_prefill_backend(h, backend)
            outs.append(ext.linear(h, x))
        assert torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])
        assert ext.kernel_status() == 0
    finally:
        ext.free(h)


@pytest.mark.parametrize("hardware,m,k,tokens,backend,groups", [
    (False, 19072, 4224, 64, 8, 1),        # 149 CTAs: two an SM fill one wave instead of two
    (True, 19072, 4224, 64, 8, 2),         # ... but not where a unit takes longer to decode
    (True, 19072, 2048, 64, 8, 1), (True, 19072, 2176, 64, 8, 2),
    (True, 18560, 2176, 385, 7, 1),        # four waves of one, two of two
    (True, 18560, 4224, 385, 7, 2),
    (False, 38400, 2176, 64, 8, 2),        # three waves of one, two of two
    (False, 18944, 2048, 64, 8, 2),        # 148 CTAs: one wave
])
def test_two_tiles_an_sm_where_they_fill_waves(ext, hardware, m, k, tokens, backend, groups):
    """Which instance serves grids of more CTAs than the 148 SMs, and that both give the bits of the wide tile."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the waves are those of 148 SMs")
    from texelator_b200 import modeling, runtime
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    weight = torch.randn(m, k, device="cuda", generator=gen) * 0.02
    h = ext.pack_encoded_device(*modeling.encode_minmax_cuda(weight, modeling.software_palette_table("cuda")), None)
    try:
        if hardware:
            ext.set_palette(h, runtime.PALETTE_HARDWARE)
        ext.set_prefill(h, 1, 1024)
        x = torch.randn(tokens, k, device="cuda", generator=gen).bfloat16()
        ext.set_prefill_backend(h, 5)
        want = ext.linear(h, x)
        ext.set_prefill_backend(h, backend)
        out = []
        names = [name for name, _ in launched(lambda: out.append(ext.linear(h, x)))]
        expected = f"prefill_umma_kernelILi1ELi{ {8: 64, 7: 128}[backend] }ELb{int(hardware)}ELi{groups}E"
        assert any(expected in name for name in names), names
        assert torch.equal(out[0], want) and ext.kernel_status() == 0
    finally:
        ext.free(h)


@pytest.mark.parametrize("m,k,tokens,backend,inside", [
    (256, 2048, 16, 5, True), (256, 2048, 16, 7, True), (256, 2048, 16, 8, True), (256, 2048, 16, 9, True), (256, 2048, 16, 6, False),
    (3968, 2896, 29, 8, True), (1024, 4096, 127, 7, True),
    (4250, 2896, 29, 8, False), (2304, 8192, 40, 8, False),      # 34 clusters of four and 18 of eight: more than are resident at once
])
def test_k_ranges_are_added_by_clusters_where_all_are_resident(ext, m, k, tokens, backend, inside):
    """One launch behind the staging where the clusters fit, else a second one that adds."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the cluster counts are those of 148 SMs")
    from texelator_b200 import modeling
    weight = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)) * 0.02
    h = ext.pack_encoded_device(*modeling.encode_minmax_cuda(weight, modeling.software_palette_table("cuda")), None)
    try:
        ext.set_prefill(h, 1, 1024)
        ext.set_prefill_backend(h, backend)
        x = torch.randn(tokens, k, device="cuda").bfloat16()
        kernels = [(name, grid) for name, grid in launched(lambda: ext.linear(h, x)) if "N2tx" in name]
        tiles = [grid for name, grid in kernels if "prefill_umma" in name]
        assert len(tiles) == 1 and tiles[0][2] > 1, kernels                       # K is cut
        assert any("combine" in name for name, _ in kernels) != inside, kernels
    finally:
        ext.free(h)


def test_staged_calls_without_the_binding_give_the_same_outputs(ext, lut):
    """The methods in Python serve where the native calls cannot be had: the same answers, outputs and refusals."""
    from texelator_b200 import runtime
    blocks, scales, x = _case(3, 300, 528, 40, lut)
    h = _pack(ext, blocks, scales)
    plain = runtime._Extension(ext._lib)
    plain._shapes[h] = ext._shapes[h]
    try:
        x, weight = x.cuda(), torch.ones(528, device="cuda", dtype=torch.bfloat16)
        outs = []
        for one in (plain, ext):
            assert [one.takes_staged(h, tokens) for tokens in (15, 16, 40)] == [False, True, True] and one.takes_staged(1234, 40) is False
            staged, y = one.staged_buffer(528, 40, "cuda"), torch.empty(40, 300, device="cuda", dtype=torch.bfloat16)
            one.add_rmsnorm_staged(x.clone(), None, weight, staged, 1e-6)
            assert one.linear_staged(handle=h, staged=staged, y=y) is y
            outs.append(y)
            with pytest.raises(RuntimeError, match="too small"):
                one.linear_staged(h, staged[:-4], y)
            with pytest.raises(RuntimeError, match="does not take staged"):
                one.linear_staged(h, staged, y[:8])
        assert torch.equal(outs[0], outs[1])
    finally:
        ext.free(h)
