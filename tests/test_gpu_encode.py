"""The GPU encoder against the reference encoder's recorded output (run with ``-m gpu``)."""
import hashlib
import json

import numpy as np
import pytest
import torch

from graph_kernels import recorded
from oracle import bc4_oracle as O

pytestmark = pytest.mark.gpu

GOLDEN = ["small_48x256", "odd_24x48", "edge_32x128", "tall_130x64"]


@pytest.fixture(scope="module")
def ext():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200 import runtime
    return runtime.extension()


@pytest.mark.parametrize("name", GOLDEN)
def test_gpu_encoder_reproduces_the_reference_bytes(ext, lut, golden_dir, name):
    """The fixtures hold what the unmodified reference encoder wrote for these weights and moments."""
    z = np.load(golden_dir / f"{name}.npz")
    blocks, scales = ext.encode(torch.from_numpy(z["weight"]).cuda(), torch.from_numpy(z["hdiag"]).cuda(), torch.from_numpy(lut).cuda())
    assert np.array_equal(scales.cpu().numpy(), z["scales"])
    assert np.array_equal(blocks.cpu().numpy(), z["blocks"])


def test_gpu_encoder_configuration_1_hash(ext, lut, golden_dir):
    """4096 x 4096 from the pinned seed: 1 048 576 blocks, hashes recorded from the reference encoder."""
    manifest = json.loads((golden_dir / "manifest.json").read_text())["cases"]["cfg1_4096x4096"]
    g = torch.Generator().manual_seed(manifest["seed"])
    w = torch.randn(4096, 4096, generator=g) * 0.02
    xc = torch.randn(64, 4096, generator=g)
    blocks, scales = ext.encode(w.cuda(), (xc * xc).mean(0).cuda(), torch.from_numpy(lut).cuda())
    assert hashlib.sha256(blocks.cpu().numpy().tobytes()).hexdigest() == manifest["blocks_sha256"]
    assert hashlib.sha256(scales.cpu().numpy().astype("<f4").tobytes()).hexdigest() == manifest["scales_sha256"]


@pytest.mark.parametrize("palette", ["software", "hardware"])
def test_gpu_encoder_equals_restated_encoder_on_hard_inputs(ext, lut, palette):
    """Sparse rows (low-mode blocks, degenerate normal equations), constant and zero rows, +-max entries, a wide
    range of activation weights -- against the CPU restatement, under both palettes."""
    table = lut if palette == "software" else O.hardware_palette()
    rng = np.random.default_rng(5)
    m, k = 96, 512
    w = (rng.standard_normal((m, k)) * 0.02).astype(np.float32)
    w[rng.random((m, k)) < 0.7] = 0
    w[3] = 0
    w[4] = 0.125
    w[5, ::2] = w[5].max()
    w[6, 1::2] = -np.abs(w[6]).max()
    hdiag = np.exp(rng.standard_normal(k) * 3).astype(np.float32)
    want_blocks, want_scales = O.encode_linear(w, hdiag, table)
    blocks, scales = ext.encode(torch.from_numpy(w).cuda(), torch.from_numpy(hdiag).cuda(), torch.from_numpy(table).cuda())
    assert np.array_equal(scales.cpu().numpy(), want_scales)
    got = blocks.cpu().numpy()
    differing = np.flatnonzero((got.reshape(-1, 8) != want_blocks.reshape(-1, 8)).any(1))
    assert differing.size == 0, differing[:10]


def test_gpu_encoder_feeds_the_operator(ext, lut):
    """Encode on the GPU, pack without a host round trip, multiply: the whole path against the oracle."""
    rng = np.random.default_rng(8)
    m, k = 256, 1024
    w = (rng.standard_normal((m, k)) * 0.02).astype(np.float32)
    hdiag = (rng.standard_normal((64, k)) ** 2).mean(0).astype(np.float32)
    blocks, scales = ext.encode(torch.from_numpy(w).cuda(), torch.from_numpy(hdiag).cuda(), torch.from_numpy(lut).cuda())
    handle = ext.pack_encoded_device(blocks, scales)
    try:
        x = torch.from_numpy(rng.standard_normal((2, k)).astype(np.float32)).bfloat16()
        y = ext.linear(handle, x.cuda()).float().cpu().numpy()
        ref = O.linear_bf16(x.float().numpy(), blocks.cpu().numpy(), scales.cpu().numpy(), lut)
        assert O.rel_rms(y, ref) <= 1e-2
        # the encoder's point: the weighted error is no worse than the min/max start's
        start_blocks, start_scales = O.encode_minmax(w, lut)
        def weighted_error(b, s):
            return float(((O.dequant_weights(b, s, lut, round_bf16=False) - w) ** 2 * hdiag[None, :]).sum())
        assert weighted_error(blocks.cpu().numpy(), scales.cpu().numpy()) <= weighted_error(start_blocks, start_scales)
    finally:
        ext.free(handle)


def test_directory_written_by_the_reference_loads_and_runs(ext, lut, golden_dir):
    """The fixture directory written by the reference's encode_linear_e3 goes through ``pack_entry_handles``
    unchanged (bias attached like ``runtime.install`` does), multiplies like the oracle says, unpacks to the
    file's bytes, and the GPU encoder reproduces the files from the recorded fp32 inputs."""
    import json
    from texelator_b200 import runtime
    root = golden_dir / "reference_artifact"
    metadata = json.loads((root / "weights" / "metadata.json").read_text())
    inputs = np.load(root / "inputs.npz")
    rng = np.random.default_rng(11)
    for entry in metadata["entries"]:
        key = entry["artifact_key"]
        blocks = np.fromfile(root / "weights" / entry["blocks_file"], dtype=np.uint8)
        scales = np.fromfile(root / "weights" / entry["scales_file"], dtype="<f4")
        bias = torch.from_numpy(inputs[f"{key}/bias"]).bfloat16().cuda() if entry["bias"] else None
        handles = runtime.pack_entry_handles(root / "weights", entry, bias=bias, lookahead=2)
        try:
            assert len(handles) == 1 and ext.handle_info(handles[0])[:2] == [entry["M"], entry["K"]]
            assert np.array_equal(ext.unpack_blocks(handles[0]).numpy(), blocks)
            x = torch.from_numpy(rng.standard_normal((3, entry["K"])).astype(np.float32)).bfloat16()
            y = ext.linear(handles[0], x.cuda()).float().cpu().numpy()
            ref = O.linear_bf16(x.float().numpy(), blocks, scales, lut, None if bias is None else bias.float().cpu().numpy())
            assert O.rel_rms(y, ref) <= 1e-2
        finally:
            runtime.free(handles)
        got_blocks, got_scales = ext.encode(torch.from_numpy(inputs[f"{key}/weight"]).cuda(), torch.from_numpy(inputs[f"{key}/hdiag"]).cuda(),
                                            torch.from_numpy(lut).cuda())
        assert np.array_equal(got_blocks.cpu().numpy(), blocks) and np.array_equal(got_scales.cpu().numpy(), scales)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_palette_at_any_float(ext, lut, shift):
    """A palette that is a slice of a larger buffer need not lie on a 16-byte boundary."""
    gen = torch.Generator().manual_seed(shift)
    w, hdiag = torch.randn(37, 592, generator=gen) * 0.05, torch.exp(torch.randn(592, generator=gen))
    buffer = torch.zeros(lut.size + 8, device="cuda")
    table = buffer[shift:shift + lut.size].view(255, 255, 8)
    table.copy_(torch.from_numpy(lut))
    assert buffer.data_ptr() % 16 == 0 and table.data_ptr() % 16 == 4 * shift
    blocks, scales = ext.encode(w.cuda(), hdiag.cuda(), table)
    want_blocks, want_scales = O.encode_linear(w, hdiag, lut)
    assert np.array_equal(scales.cpu().numpy(), want_scales)
    assert np.array_equal(blocks.cpu().numpy(), want_blocks.reshape(-1))


def _rows(kind, m, k, gen):
    w = torch.randn(m, k, device="cuda", generator=gen)
    if kind == "uniform":                    # endpoints at their limit
        w = torch.rand(m, k, device="cuda", generator=gen) - 0.5
    elif kind == "cubed":                    # blocks far below the row's largest weight: endpoints close together
        w = w ** 3
    elif kind == "pruned":
        w = w * (torch.rand(m, k, device="cuda", generator=gen) < 0.1)
    elif kind == "ties":                     # weights on and half way between palette entries
        w = torch.randint(-14 * 127, 14 * 127 + 1, (m, k), device="cuda", generator=gen).float() / (14 * 127)
    elif kind == "numbers":                  # not numbers, infinities, weights far below the scale
        w[::3, 5], w[::5, 9], w[1::5, 17] = float("nan"), float("inf"), -float("inf")
        w[::4, ::3] *= 1e-25
    return w


@pytest.mark.parametrize("kind,m,k,palette", [
    ("normal", 2051, 2048, "software"), ("uniform", 4096, 1040, "software"), ("cubed", 1200, 4096, "software"),
    ("pruned", 1024, 4160, "software"), ("ties", 1024, 4096, "software"), ("numbers", 1024, 4096, "software"),
    ("normal", 90000, 48, "software"), ("normal", 593, 8208, "software"), ("normal", 300, 17408, "software"),
    ("normal", 1024, 4096, "hardware"), ("normal", 1024, 4096, "one entry off"), ("moments", 1024, 4096, "software")])
def test_large_matrices_get_the_bytes_of_their_slabs(ext, lut, kind, m, k, palette):
    """Matrices of 2^21 weights and more have blocks that are searched by a quadratic form; slabs of fewer rows are searched
    neighbour by neighbour.  A row's bytes do not depend on the rows beside it, so both have to agree."""
    gen = torch.Generator(device="cuda").manual_seed(k)
    table = (ext.hardware_palette().reshape(255, 255, 8) if palette == "hardware" else torch.from_numpy(lut)).cuda().clone()
    if palette == "one entry off":
        table[60, 190, 4] += 1e-3            # high mode, endpoints apart
    w = _rows(kind, m, k, gen)
    hdiag = torch.exp(torch.randn(k, device="cuda", generator=gen))
    if kind == "moments":
        hdiag[::7], hdiag[5], hdiag[100], hdiag[200] = 0, -1, float("nan"), float("inf")
    assert m * k >= 1 << 21
    blocks, scales = ext.encode(w, hdiag, table)
    rows = ((1 << 21) - 1) // k
    slabs = [ext.encode(w[i:i + rows], hdiag, table) for i in range(0, m, rows)]
    assert torch.equal(blocks, torch.cat([b for b, _ in slabs]))
    assert torch.equal(scales.view(torch.int32), torch.cat([s for _, s in slabs]).view(torch.int32))


@pytest.mark.parametrize("m,k", [(2048, 1024), (9500, 1024), (10000, 2048), (44000, 48), (40000, 64)])
@pytest.mark.parametrize("offset", [0, 1])
def test_the_search_for_magnitudes_runs_beside_the_verdict(ext, lut, m, k, offset):
    """The kernel behind the verdict on the palette starts with it, the verdict itself behind everything in front; with few and many rows, rows
    shorter than a verdict's bytes, and a palette off the boundary of wide loads.  The bytes are those of the slabs."""
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    w, hdiag = torch.randn(m, k, device="cuda", generator=gen) * 0.02, torch.exp(torch.randn(k, device="cuda", generator=gen))
    table = torch.zeros(255 * 255 * 8 + offset, device="cuda")[offset:].copy_(torch.from_numpy(lut).reshape(-1)).view(255, 255, 8)
    rows, out = ((1 << 21) - 1) // k, []
    kernels = [(name, early) for name, _, early in recorded(lambda: out.append(ext.encode(w, hdiag, table))) if "N2tx" in name]
    assert ["verdict" in name for name, _ in kernels] == [True, False] and [early for _, early in kernels] == [False, True], kernels
    slabs = torch.cat([ext.encode(w[i:i + rows], hdiag, table)[0] for i in range(0, m, rows)])
    assert torch.equal(out[0][0], slabs)


def test_blocks_of_tiny_moments_in_a_large_matrix_get_the_bytes_of_their_slabs(ext, lut):
    """Sixteen moments so small that the reference's products underflow: which neighbour wins is then its rounding's choice."""
    m, k = 1024, 4096
    gen = torch.Generator(device="cuda").manual_seed(11)
    w = torch.randn(m, k, device="cuda", generator=gen) * 0.02
    levels = torch.tensor([1e-28, 1e-30, 1e-32, 1e-36, 1e-38, 1e-40, 1e-41, 1e-42, 1e-44, 0.0, 1.0], device="cuda")
    hdiag = levels[torch.arange(k, device="cuda") // 16 % len(levels)].contiguous()
    table = torch.from_numpy(lut).cuda()
    blocks, _ = ext.encode(w, hdiag, table)
    rows = ((1 << 21) - 1) // k
    slabs = torch.cat([ext.encode(w[i:i + rows], hdiag, table)[0] for i in range(0, m, rows)])
    assert torch.equal(blocks, slabs)


def test_the_software_palette_takes_the_quadratic_form(ext, lut):
    """Both ways through a block give the same bytes, so what shows which one ran is its time: half of the other's (75 and 157 us)."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    w, hdiag = torch.randn(4096, 4096, device="cuda", generator=gen) * 0.02, torch.exp(torch.randn(4096, device="cuda", generator=gen))
    software = torch.from_numpy(lut).cuda()
    other = software.clone()
    other[60, 190, 4] += 1e-3
    times = []
    for table in (software, other):
        call = lambda: ext.encode(w, hdiag, table)
        assert [name for name, _, _ in recorded(call) if "encode_kernel" in name and "ELb1ELb1E" in name]
        best = float("inf")
        for _ in range(5):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(10):
                call()
            end.record()
            end.synchronize()
            best = min(best, begin.elapsed_time(end))
        times.append(best)
    assert times[0] < 0.75 * times[1], times
