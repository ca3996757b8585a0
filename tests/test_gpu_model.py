"""Model-level parity on a GPU: BC4 decoder vs the same model with dequantised dense weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def toy():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.modeling import CONFIGS, BC4Decoder
    model = BC4Decoder(CONFIGS["toy"], "cuda:0", max_len=96, seed=3, keep_dense=True)
    yield model
    model.free()


def _cosine(a, b):
    return float(torch.nn.functional.cosine_similarity(a.float().reshape(1, -1), b.float().reshape(1, -1)).item())


def test_prefill_hidden_state_cosine(toy):
    ids = torch.randint(0, toy.config.vocab, (40,), generator=torch.Generator().manual_seed(0))
    for backend in (0, 5):
        for h in toy.handles:
            toy.ext.set_prefill_backend(h, backend)
        got = toy.prefill(ids)
        ref = toy.prefill(ids, dense=True)
        assert _cosine(got, ref) >= 0.999, backend      # final hidden-state gate of the operator


def test_prefill_through_the_decode_kernel(toy):
    """The same gate with the prompt kept off the tiles."""
    ids = torch.randint(0, toy.config.vocab, (40,), generator=torch.Generator().manual_seed(0))
    before = [toy.ext.handle_info(h)[2:4] for h in toy.handles]
    for h in toy.handles:
        toy.ext.set_prefill(h, 1 << 30, 1024)
    try:
        assert _cosine(toy.prefill(ids), toy.prefill(ids, dense=True)) >= 0.999
    finally:
        for h, (threshold, rows) in zip(toy.handles, before):
            toy.ext.set_prefill(h, threshold, rows)


def test_decode_graph_matches_eager_and_dense(toy):
    ids = torch.randint(0, toy.config.vocab, (24,), generator=torch.Generator().manual_seed(1))
    toy.prefill(ids)
    toy.tok.fill_(int(ids[-1]))
    state = (toy.tok.clone(), toy.pos.clone(), toy.mask.clone())
    toy.decode_eager()
    eager_hidden, eager_tok = toy.last_hidden.clone(), toy.next_tok.clone()
    toy.tok.copy_(state[0]); toy.pos.copy_(state[1]); toy.mask.copy_(state[2])
    toy.decode_eager(dense=True)
    dense_hidden = toy.last_hidden.clone()
    assert _cosine(eager_hidden, dense_hidden) >= 0.999
    toy.tok.copy_(state[0]); toy.pos.copy_(state[1]); toy.mask.copy_(state[2])
    toy.capture()
    assert toy.launches_per_step == 4 * toy.config.layers
    toy.decode_graph()
    torch.cuda.synchronize()
    assert torch.equal(toy.last_hidden, eager_hidden) and torch.equal(toy.next_tok, eager_tok)
    assert int(toy.pos.item()) == 25


def test_fused_decode_step_matches_pytorch_glue():
    """The library's glue kernels (norm, RoPE + cache append, attention, SwiGLU) against the PyTorch
    formulation of the same step, on a model with 128-wide heads."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.modeling import CONFIGS, BC4Decoder
    model = BC4Decoder(CONFIGS["toy128"], "cuda:0", max_len=600, seed=5)
    try:
        assert model.fused
        ids = torch.randint(0, model.config.vocab, (300,), generator=torch.Generator().manual_seed(2))
        model.prefill(ids)
        model.tok.fill_(int(ids[-1]))
        state = (model.tok.clone(), model.pos.clone(), model.mask.clone(), model.k_cache.clone(), model.v_cache.clone())
        hidden, tokens = [], []
        for _ in range(3):
            model.decode_eager()
            hidden.append(model.last_hidden.clone()); tokens.append(int(model.next_tok))
        model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
        model.k_cache.copy_(state[3]); model.v_cache.copy_(state[4])
        for step in range(3):
            model.decode_eager(fused=True)
            assert _cosine(model.last_hidden, hidden[step]) >= 0.9995, step
        assert model.single                      # staged activations + K-split partials (tx_linear_single)
        model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
        model.k_cache.copy_(state[3]); model.v_cache.copy_(state[4])
        for step in range(3):
            model.decode_eager(single=True)
            assert _cosine(model.last_hidden, hidden[step]) >= 0.9995, step
        model.prefer_single = lambda: True                                   # the same path under graph replay
        model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
        model.capture()
        assert model.launches_per_step == model.config.layers * 8 + 1
        for step in range(3):
            model.decode_graph()
            torch.cuda.synchronize()
            assert _cosine(model.last_hidden, hidden[step]) >= 0.9995, step
        del model.prefer_single
        model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
        for fuse_norm, per_layer in ((False, 8), (True, 6)):
            model.fuse_norm = fuse_norm
            model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
            model.capture()
            assert model.launches_per_step == model.config.layers * per_layer + 1
            for step in range(3):      # graph replays overlap kernels (programmatic dependent launch): same results
                model.decode_graph()
                torch.cuda.synchronize()
                assert _cosine(model.last_hidden, hidden[step]) >= 0.9995, (fuse_norm, step)
    finally:
        model.free()


def _relative_rms(a, b):
    return float((a.float() - b.float()).square().mean().sqrt() / b.float().square().mean().sqrt())


def test_configuration_2_model_gate():
    """BASELINE configuration 2 at its real shape (hidden 2048, 36 layers, 16 q / 2 kv heads, intermediate 11008,
    q/k/v bias): final hidden states of a 64-token prompt and of eight decoded tokens against the same model with
    dense ``bf16(pal*scale)`` weights multiplied in fp32.  A random-init stack of 36 layers amplifies rounding: the
    same dense weights through the library's bf16 GEMM already end 5 % (rel-RMS) away from the fp32 run, so the
    gate is relative to that distance -- the BC4 operator may not sit further from the fp32 run than 1.5 times what
    a bf16 GEMM does -- plus cosine >= 0.995 as an absolute backstop.  (The reference's whole-model gate,
    texelator/prefill.py:88-108, is rel-RMS <= 0.02 between its own two paths on a trained model.)
    Eager PyTorch glue, the fused kernels and the CUDA graph are all held to it."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200 import prefill as prefill_check
    from texelator_b200.modeling import CONFIGS, BC4Decoder
    config = CONFIGS["qwen2.5-3b-shaped"]
    model = BC4Decoder(config, "cuda:0", max_len=128, seed=11, keep_dense=True)
    try:
        assert len(model.handles) == 4 * config.layers and model.fused
        ids = torch.randint(0, config.vocab, (64,), generator=torch.Generator().manual_seed(12))
        ref = model.prefill(ids, dense=True)
        floor = _relative_rms(model.prefill(ids, dense="bf16"), ref)
        for threshold in (prefill_check.TILES, prefill_check.STREAMED):      # tensor-core tiles, then the decode kernel
            prefill_check._force(model.handles, threshold)
            got = model.prefill(ids)
            assert _relative_rms(got, ref) <= 1.5 * floor + 1e-3, (threshold, floor)
            assert _cosine(got, ref) >= 0.995
        from texelator_b200.runtime import PREFILL_THRESHOLD, PREFILL_TILE_ROWS
        prefill_check._force(model.handles, PREFILL_THRESHOLD)
        model.prefill(ids)
        model.tok.fill_(int(ids[-1]))
        state = (model.tok.clone(), model.pos.clone(), model.mask.clone(), model.k_cache.clone(), model.v_cache.clone())

        def rewind():
            model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
            model.k_cache.copy_(state[3]); model.v_cache.copy_(state[4])

        fed = []                                     # the fp32 run's tokens, fed to every other run: a different
                                                     # greedy pick at one step would compare two different sequences
        def decode(steps=8, **mode):
            rewind()
            out = []
            for step in range(steps):
                if len(fed) > step:
                    model.tok.copy_(fed[step])
                else:
                    fed.append(model.tok.clone())
                model.decode_eager(**mode)
                out.append(model.last_hidden.clone())
            return out

        dense_hidden = decode(dense=True)
        floors = [_relative_rms(a, b) for a, b in zip(decode(dense="bf16"), dense_hidden)]
        for mode in (dict(), dict(fused=True)):
            for step, hidden in enumerate(decode(**mode)):
                # later steps attend to cache rows written by the model under test itself: the gate is on every step
                assert _relative_rms(hidden, dense_hidden[step]) <= 1.5 * max(floors) + 1e-3, (mode, step, floors)
                assert _cosine(hidden, dense_hidden[step]) >= 0.995, (mode, step)
        rewind()
        model.capture()
        for step in range(8):
            model.tok.copy_(fed[step])
            torch.cuda.synchronize()
            model.decode_graph()
            model.stream.synchronize()
            assert _relative_rms(model.last_hidden, dense_hidden[step]) <= 1.5 * max(floors) + 1e-3, ("graph", step, floors)
        model.check_status()
    finally:
        model.free()


def test_model_with_weights_from_the_gpu_encoder():
    """The harness with its projections encoded by the reference's endpoint search on the GPU (`encoder="e3"`):
    same gates as with the min/max encoding -- the operator against dense dequantised weights, eager and graph."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.modeling import CONFIGS, BC4Decoder
    model = BC4Decoder(CONFIGS["toy128"], "cuda:0", max_len=96, seed=21, keep_dense=True, encoder="e3")
    try:
        ids = torch.randint(0, model.config.vocab, (40,), generator=torch.Generator().manual_seed(22))
        assert _cosine(model.prefill(ids), model.prefill(ids, dense=True)) >= 0.999
        model.prefill(ids)
        model.tok.fill_(int(ids[-1]))
        state = (model.tok.clone(), model.pos.clone(), model.mask.clone())
        model.decode_eager(dense=True)
        want = model.last_hidden.clone()
        model.tok.copy_(state[0]); model.pos.copy_(state[1]); model.mask.copy_(state[2])
        model.capture()
        model.decode_graph()
        model.stream.synchronize()
        assert _cosine(model.last_hidden, want) >= 0.999
        model.check_status()
    finally:
        model.free()


@pytest.mark.parametrize("tokens", [40, 3000])
def test_a_prompt_takes_no_memory_for_its_hand_over(tokens):
    """What the norms hand over staged lies where SwiGLU's rows do: beyond the rows of the layer's steps, a prompt takes no memory
    (but for 32 tokens' padding of the staged form and soft-max statistics)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from texelator_b200.modeling import CONFIGS, BC4Decoder
    c = CONFIGS["toy128"]
    model = BC4Decoder(c, "cuda:0", max_len=tokens, seed=3)
    try:
        ids = torch.randint(0, c.vocab, (tokens,), device="cuda")
        for handle in model.handles:
            model.ext.set_prefill_backend(handle, 8)
        assert all(model.ext.takes_staged(handle, tokens) for handle in model.handles)
        model.prefill(ids)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_stats()["requested_bytes.all.current"]
        model.prefill(ids)
        torch.cuda.synchronize()
        taken = torch.cuda.memory_stats()["requested_bytes.all.peak"] - before
        # residual, x, out; qkv; gate and up; SwiGLU; attention's output twice (as the kernel leaves it, and in rows)
        rows = 2 * tokens * (3 * c.hidden + c.q_rows + 2 * c.kv_rows + 3 * c.intermediate + 2 * c.q_rows)
        slack = 32 * 2 * max(c.hidden, c.intermediate) + 4 * tokens * c.q_heads + (64 << 10)
        assert taken <= rows + slack, (taken, rows, slack)
    finally:
        model.free()
