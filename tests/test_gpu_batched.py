"""Batched decode: the multi-token decode kernel with K ranges, the batched glue kernels and the batched model
(run with ``-m gpu``)."""
import numpy as np
import pytest
import torch

from graph_kernels import recorded
from oracle import bc4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200 import runtime
    return runtime.extension()


def _cosine(a, b):
    return float(torch.nn.functional.cosine_similarity(a.float().reshape(1, -1), b.float().reshape(1, -1)))


@pytest.mark.parametrize("m,k,tokens,bias", [
    (5120, 17408, 8, False),      # 8 rows of K = 17408 do not fit one CTA's shared memory: K ranges
    (1280, 8192, 32, True),       # few row tiles: ranges also spread the work over the SMs
    (8192, 1024, 32, False),      # short K: one range
    (272, 3584, 24, True),        # ragged rows (M % 16 != 0), three token tiles
    (512, 4112, 17, False),       # K not a multiple of 128, odd token count
    (64, 28672, 32, False),       # the longest rows of the 70B-class shapes
])
def test_multi_token_decode_matches_oracle(ext, lut, m, k, tokens, bias):
    """Reference semantics: every token count below the threshold is the decode operator, one row of x at a time
    (texelator_cuda.cu:1438-1468)."""
    rng = np.random.default_rng(m + k + tokens)
    w = (rng.standard_normal((m, k)) * 0.02).astype(np.float32)
    blocks, scales = O.encode_minmax(w, lut)
    x = torch.from_numpy(rng.standard_normal((tokens, k)).astype(np.float32)).bfloat16()
    b = torch.from_numpy((rng.standard_normal(m) * 0.3).astype(np.float32)).bfloat16() if bias else None
    h = ext.pack_encoded(torch.from_numpy(blocks), torch.from_numpy(scales), None if b is None else b.cuda())
    try:
        ext.set_prefill(h, 64, 1024)
        y = ext.linear(h, x.cuda())
        ref = O.linear_bf16(x.float().numpy(), blocks, scales, lut, None if b is None else b.float().numpy())
        assert O.rel_rms(y.float().cpu().numpy(), ref) <= 1e-2
        # the same rows one at a time: the K ranges change the order of the fp32 sums, nothing else
        single = torch.cat([ext.linear(h, x[i:i + 1].cuda()) for i in range(tokens)])
        assert O.rel_rms(y.float().cpu().numpy(), single.float().cpu().numpy()) <= 4e-3
        again = ext.linear(h, x.cuda())
        assert torch.equal(y, again)                       # deterministic: fixed ranges, fixed order
    finally:
        ext.free(h)


def test_silu_mul_pairs(ext):
    from texelator_b200.modeling import interleave_gate_up
    gen = torch.Generator(device="cuda").manual_seed(1)
    tokens, inter = 5, 264
    gate = torch.randn(tokens, inter, device="cuda", generator=gen).bfloat16()
    up = torch.randn(tokens, inter, device="cuda", generator=gen).bfloat16()
    paired = interleave_gate_up(gate.T.contiguous(), up.T.contiguous()).T.contiguous()       # [tokens, 2 * inter]
    out = torch.empty(tokens, inter, device="cuda", dtype=torch.bfloat16)
    ext.silu_mul_pairs(paired, out)
    want = torch.empty_like(out)
    ext.silu_mul(torch.cat([gate, up], 1).contiguous(), want)
    assert torch.equal(out, want)


def test_attention_step_batch_equals_per_sequence_steps(ext):
    """Sequences at different positions (one of them past the single-chunk length) in one launch."""
    from texelator_b200.modeling import CONFIGS, _rope_tables
    c = CONFIGS["toy128"]
    gen = torch.Generator(device="cuda").manual_seed(2)
    batch, q_heads, kv_heads, max_len = 5, c.q_heads, c.kv_heads, 320
    cos, sin = _rope_tables(c, max_len, torch.device("cuda"))
    k_cache = torch.randn(batch, kv_heads, max_len, 128, device="cuda", generator=gen).bfloat16()
    v_cache = torch.randn(batch, kv_heads, max_len, 128, device="cuda", generator=gen).bfloat16()
    qkv = torch.randn(batch, (q_heads + 2 * kv_heads) * 128, device="cuda", generator=gen).bfloat16()
    positions = torch.tensor([0, 7, 63, 64, 300], device="cuda", dtype=torch.int64)
    want = torch.empty(batch, q_heads * 128, device="cuda", dtype=torch.bfloat16)
    k_ref, v_ref = k_cache.clone(), v_cache.clone()
    scratch = torch.zeros(batch * ext.attention_step_scratch_floats(q_heads, max_len), dtype=torch.float32, device="cuda")
    for b in range(batch):
        ext.attention_step(qkv[b:b + 1], cos, sin, positions[b:b + 1], k_ref[b], v_ref[b], scratch, want[b:b + 1], q_heads, kv_heads, 128)
    got = torch.empty_like(want)
    ext.attention_step_batch(qkv, cos, sin, positions, k_cache, v_cache, scratch, got, q_heads, kv_heads, 128)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert torch.equal(k_cache, k_ref) and torch.equal(v_cache, v_ref)
    for _ in range(3):                                   # the arrival counters were left at zero: launch again
        ext.attention_step_batch(qkv, cos, sin, positions, k_cache, v_cache, scratch, got, q_heads, kv_heads, 128)
    assert torch.equal(got, want)


@pytest.mark.parametrize("batch", [8, 3])
def test_batch_of_sequences_equals_the_sequences_one_by_one(batch):
    """toy128: B sequences with different prompts decode together (library kernels, eagerly and from a CUDA graph)
    and one by one through PyTorch glue with the same handles; the hidden states agree at every step (the one-by-one
    run's tokens are fed to both, so a near-tie in one argmax cannot send the two runs down different sequences)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.batched import BatchedBC4Decoder
    from texelator_b200.modeling import CONFIGS
    config = CONFIGS["toy128"]
    model = BatchedBC4Decoder(config, "cuda:0", max_len=160, batch=batch, seed=5)
    try:
        for sequence in range(batch):
            ids = torch.randint(0, config.vocab, (20 + 9 * sequence,), generator=torch.Generator().manual_seed(sequence))
            model.prefill_sequence(sequence, ids)
            model.tok[sequence] = int(ids[-1])
        state = (model.tok.clone(), model.pos.clone(), model.k_cache.clone(), model.v_cache.clone())

        def rewind():
            model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.k_cache.copy_(state[2]); model.v_cache.copy_(state[3])

        want_hidden, want_tokens = [], []
        for _ in range(6):
            model.decode_step_reference()
            want_hidden.append(model.last_hidden.clone()); want_tokens.append(model.next_tok.clone())
        rewind()
        for step in range(6):
            model.tok.copy_(state[0] if step == 0 else want_tokens[step - 1])
            model.decode_step()
            assert _cosine(model.last_hidden, want_hidden[step]) >= 0.9995, step
        rewind()
        model.capture()
        assert model.launches_per_step > 0
        for step in range(6):
            model.tok.copy_(state[0] if step == 0 else want_tokens[step - 1])
            torch.cuda.synchronize()
            model.decode_graph()
            model.stream.synchronize()
            assert _cosine(model.last_hidden, want_hidden[step]) >= 0.9995, ("graph", step)
        assert torch.equal(model.pos, state[1] + 6)
        model.check_status()
    finally:
        model.free()


@pytest.mark.parametrize("kernel", ["gemv", "umma_128x64x128"])
def test_replays_of_sixteen_sequences_equal_eager_steps(kernel):
    """Forty replays of the captured step leave the bits of forty eager steps: tokens, hidden states and every cache row.
    Both runs start where ``capture`` left the decoder."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.autotune import CANDIDATES
    from texelator_b200.batched import BatchedBC4Decoder
    from texelator_b200.modeling import CONFIGS
    config = CONFIGS["toy128"]
    model = BatchedBC4Decoder(config, "cuda:0", max_len=120, batch=16, seed=9)
    try:
        for handle in model.handles:
            model.ext.set_prefill(handle, 17 if kernel == "gemv" else 16, 1024)
            model.ext.set_prefill_backend(handle, CANDIDATES["umma_128x64x128"])
        for sequence in range(16):
            model.fill_context(sequence, 0, 5 + 4 * sequence, seed=3)
        model.tok.copy_(torch.arange(16, device="cuda") * 100)
        model.capture()
        state = [t.clone() for t in (model.tok, model.pos, model.k_cache, model.v_cache)]
        runs = []
        for step in (model.decode_step, model.decode_graph):
            for tensor, saved in zip((model.tok, model.pos, model.k_cache, model.v_cache), state):
                tensor.copy_(saved)
            torch.cuda.synchronize()
            seen = []
            for _ in range(40):
                step()
                seen.append((model.next_tok.clone(), model.last_hidden.clone()))
            runs.append((seen, model.k_cache.clone(), model.v_cache.clone()))
        torch.cuda.synchronize()
        (eager, *eager_cache), (replayed, *replayed_cache) = runs
        assert all(torch.equal(a, b) for e, r in zip(eager, replayed) for a, b in zip(e, r))
        assert all(torch.equal(a, b) for a, b in zip(eager_cache, replayed_cache))
        model.check_status()
    finally:
        model.free()


@pytest.mark.parametrize("batch", [1, 3])
def test_capture_on_the_last_cache_row(batch):
    """A sequence with room for one more token: ``capture`` touches no row but those of the next positions."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.batched import BatchedBC4Decoder
    from texelator_b200.modeling import BC4Decoder, CONFIGS
    config, max_len = CONFIGS["toy128"], 40
    if batch == 1:
        model, positions = BC4Decoder(config, "cuda:0", max_len=max_len, seed=2), [max_len - 1]
    else:
        model, positions = BatchedBC4Decoder(config, "cuda:0", max_len=max_len, batch=batch, seed=2), [max_len - 1, 5, 20]
    try:
        gen = torch.Generator(device="cuda").manual_seed(1)
        for cache in (model.k_cache, model.v_cache):
            cache.copy_(torch.randn(cache.shape, device="cuda", generator=gen))
        model.pos.copy_(torch.tensor(positions, device="cuda"))
        if batch == 1:
            model.mask[..., :max_len - 1] = True
        before = (model.tok.clone(), model.pos.clone(), model.k_cache.clone(), model.v_cache.clone())
        model.capture()
        torch.cuda.synchronize()
        assert torch.equal(model.tok, before[0]) and torch.equal(model.pos, before[1])
        for cache, saved in ((model.k_cache, before[2]), (model.v_cache, before[3])):
            changed = (cache != saved).any(-1)                               # [layers, (sequences,) heads, rows]
            changed = changed.unsqueeze(1) if batch == 1 else changed
            for sequence, position in enumerate(positions):
                rows = changed[:, sequence].any(0).any(0).nonzero().reshape(-1).tolist()
                assert rows == [position]
        model.decode_graph()
        model.check_status()
        assert model.pos.tolist() == [p + 1 for p in positions]
    finally:
        model.free()


@pytest.mark.parametrize("batch", [1, 3, 16])
def test_a_step_starts_behind_the_whole_step_before(batch):
    """The attention kernel reads the position, which ends a step, before it waits for the launches in front of it; these may all start early,
    so the first launch of a step must not: eager steps behind one another read a finished position."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.batched import BatchedBC4Decoder
    from texelator_b200.modeling import BC4Decoder, CONFIGS
    config = CONFIGS["toy128"]
    model = BC4Decoder(config, "cuda:0", max_len=40, seed=2) if batch == 1 else BatchedBC4Decoder(config, "cuda:0", max_len=40, batch=batch, seed=2)
    step = model._decode_step_fused if batch == 1 else model.decode_step
    try:
        with torch.no_grad():
            kernels = recorded(lambda: (step(), step()))
        attention = [i for i, (name, _, _) in enumerate(kernels) if "attention_step" in name]
        assert len(attention) == 2 * config.layers and any(early for _, _, early in kernels)
        first = attention[config.layers]                     # of the second step
        between = [early for _, _, early in kernels[attention[config.layers - 1] + 1:first + 1]]
        writer = max(i for i, (name, _, _) in enumerate(kernels[:first]) if "N2tx" not in name)    # the step before ends with the position
        assert not all(early for _, _, early in kernels[writer + 1:first + 1]), (between, writer, first)
        model.check_status()
    finally:
        model.free()


@pytest.mark.parametrize("batch", [1, 3, 16])
def test_a_token_outside_the_vocabulary_ends_the_decoder_s_next_call(batch):
    """Steps are asynchronous: the step itself leaves a hidden state that is not a number, and the call behind it refuses; the other
    sequences' states are those of a step without the token, and the decoder is usable again once the token is mended."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.batched import BatchedBC4Decoder
    from texelator_b200.modeling import BC4Decoder, CONFIGS
    config = CONFIGS["toy128"]
    model = BC4Decoder(config, "cuda:0", max_len=40, seed=2) if batch == 1 else BatchedBC4Decoder(config, "cuda:0", max_len=40, batch=batch, seed=2)
    eager = (lambda: model.decode_eager(fused=True)) if batch == 1 else model.decode_step
    try:
        model.capture()
        for step in (eager, model.decode_graph):
            start = (model.tok.clone(), model.pos.clone())
            step()
            want = model.last_hidden.clone()
            model.tok.copy_(start[0]); model.pos.copy_(start[1])
            model.tok[-1] = config.vocab
            step()
            torch.cuda.synchronize()
            assert bool(model.last_hidden[-1].isnan().all()) and torch.equal(model.last_hidden[:-1], want[:-1])
            with pytest.raises(RuntimeError, match="outside the vocabulary"):
                step()
            model.tok.copy_(start[0]); model.pos.copy_(start[1])
            step()
            assert torch.equal(model.last_hidden, want)
            model.check_status()
        model.tok[-1] = -1
        with pytest.raises(RuntimeError, match="outside the vocabulary"):
            model.capture()
        assert model.ext.kernel_status() == 0
    finally:
        model.free()
