"""GPU parity of the whole decoder against the oracle's Llama forward (random weights)."""
import numpy as np
import pytest

import fixtures as F
import kalosm_b200 as kb
from gpu_util import dev  # noqa: F401
from llama_util import build_models, llama3_8b_cfg, tiny_cfg, write_checkpoint
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _margin(logits):
    s = np.sort(logits, axis=-1)
    return s[..., -1] - s[..., -2]


@pytest.mark.parametrize("batch", [1, 3])
def test_prefill_and_decode_logits(dev, batch):
    cfg = tiny_cfg()
    gpu, cpu = build_models(dev, cfg, batch=batch, seed=1)
    rng = np.random.default_rng(2)
    prompt = rng.integers(0, cfg["vocab"], size=(batch, 9), dtype=np.uint32)
    lg, nxt = gpu.forward(prompt)
    lo = cpu.forward(prompt)
    assert F.rel_l2(lg, lo) < 2e-3, F.rel_l2(lg, lo)
    tok = nxt.copy()
    for step in range(6):
        lo = cpu.forward(tok[:, None])
        lg, nxt = gpu.forward(tok[:, None])
        err = np.max(np.abs(lg - lo))
        assert F.rel_l2(lg, lo) < 2e-3, (step, F.rel_l2(lg, lo))
        want = np.array([O.top_k(lo[b], 1)[0][0] for b in range(batch)])
        decided = _margin(lo) > 4 * err
        assert np.array_equal(nxt[decided], want[decided])
        tok = want.astype(np.uint32)
    assert gpu.position == 9 + 6


@pytest.mark.parametrize("batch", [1, 3])
def test_decoder_with_five_bit_weights(dev, batch):
    # a Q5_K_M-style mix: Q5_K body, Q6_K for attn_v / ffn_down / output, Q5_0 embeddings. Q5_K matrices
    # stay in file order (their own product kernel, no fused decode step), Q5_0 ones become Q8_0 tiles.
    cfg = tiny_cfg()
    types = {"token_embd": O.Q5_0, "attn_q": O.Q5K, "attn_k": O.Q5K, "attn_output": O.Q5K, "ffn_gate": O.Q5K,
             "ffn_up": O.Q5K}
    gpu, cpu = build_models(dev, cfg, batch=batch, seed=41, types=types)
    prompt = np.random.default_rng(42).integers(0, cfg["vocab"], size=(batch, 40), dtype=np.uint32)
    lg, nxt = gpu.forward(prompt)
    lo = cpu.forward(prompt)
    assert F.rel_l2(lg, lo) < 4e-3, F.rel_l2(lg, lo)  # 40 rows: fp16 operands in every product of the chain
    tok = np.array([O.top_k(lo[b], 1)[0][0] for b in range(batch)], dtype=np.uint32)
    for step in range(6):
        lo = cpu.forward(tok[:, None])
        lg, nxt = gpu.forward(tok[:, None])
        err = np.max(np.abs(lg - lo))
        assert F.rel_l2(lg, lo) < 4e-3, (step, F.rel_l2(lg, lo))
        want = np.array([O.top_k(lo[b], 1)[0][0] for b in range(batch)])
        decided = _margin(lo) > 4 * err
        assert np.array_equal(nxt[decided], want[decided])
        tok = want.astype(np.uint32)
    assert dev.status() == 0


@pytest.mark.parametrize("flagged_rows", [False, True], ids=["grid-barriers", "flagged-rows"])
def test_greedy_tokens_match_for_32_steps(dev, flagged_rows, monkeypatch):
    monkeypatch.setenv("FB200_FUSED_LL", "1" if flagged_rows else "0")
    # first 32 greedy tokens identical on a random-weight model; a step whose oracle top-1/top-2
    # margin is below the measured logit error is indeterminate and re-synchronised
    cfg = tiny_cfg()
    gpu, cpu = build_models(dev, cfg, batch=1, seed=3)
    rng = np.random.default_rng(4)
    prompt = rng.integers(0, cfg["vocab"], size=(1, 5), dtype=np.uint32)
    _, first = gpu.forward(prompt)
    lo = cpu.forward(prompt)
    assert first[0] == O.top_k(lo[0], 1)[0][0]
    # device-side loop: 32 steps without reading logits back
    gpu_tokens = gpu.generate_greedy(first, 32)[0]
    tok = first.copy()
    indeterminate = 0
    for step in range(32):
        lo = cpu.forward(tok[:, None])
        want = O.top_k(lo[0], 1)[0][0]
        if gpu_tokens[step] != want:
            assert _margin(lo)[0] < 1e-3, (step, _margin(lo)[0])
            indeterminate += 1
            break  # sequences diverge legitimately after an undecidable step
        tok = np.array([want], dtype=np.uint32)
    assert indeterminate == 0 or step > 8
    assert gpu.position == 5 + 32


def test_graph_step_equals_eager_prefill(dev):
    # decoding token by token (captured graph) and prefilling the same tokens give the same logits
    cfg = tiny_cfg()
    gpu, _ = build_models(dev, cfg, batch=1, seed=5, want_cpu=False)
    rng = np.random.default_rng(6)
    toks = rng.integers(0, cfg["vocab"], size=(1, 12), dtype=np.uint32)
    lg_prefill, _ = gpu.forward(toks)
    gpu.reset()
    for i in range(12):
        lg_step, _ = gpu.forward(toks[:, i:i + 1])
    assert F.rel_l2(lg_step, lg_prefill) < 2e-3
    with pytest.raises(kb.FusorError) as e:
        gpu.forward(rng.integers(0, cfg["vocab"], size=(1, cfg["ctx"]), dtype=np.uint32))
    assert e.value.code == kb.ERR_CAPACITY


@pytest.mark.parametrize("flagged_rows", [False, True], ids=["grid-barriers", "flagged-rows"])
@pytest.mark.parametrize("head_dim,n_head,n_kv_head", [(64, 4, 2), (128, 8, 2), (128, 8, 1)])
def test_decode_over_a_long_context(dev, head_dim, n_head, n_kv_head, flagged_rows, monkeypatch):
    monkeypatch.setenv("FB200_FUSED_LL", "1" if flagged_rows else "0")
    # several attention splits per KV head (one per 128 cached keys), 4 or 8 query rows per KV
    # head, a prompt whose length is not a multiple of the split size
    cfg = dict(tiny_cfg(), ctx=448, head_dim=head_dim, n_head=n_head, n_kv_head=n_kv_head)
    gpu, cpu = build_models(dev, cfg, batch=1, seed=11)
    rng = np.random.default_rng(12)
    prompt = rng.integers(0, cfg["vocab"], size=(1, 291), dtype=np.uint32)
    lg, nxt = gpu.forward(prompt)
    lo = cpu.forward(prompt)
    assert F.rel_l2(lg, lo) < 2e-3, F.rel_l2(lg, lo)
    tok = np.array([O.top_k(lo[0], 1)[0][0]], dtype=np.uint32)
    for step in range(5):
        lo = cpu.forward(tok[:, None])
        lg, _ = gpu.forward(tok[:, None])
        assert F.rel_l2(lg, lo) < 2e-3, (step, F.rel_l2(lg, lo))
        tok = np.array([O.top_k(lo[0], 1)[0][0]], dtype=np.uint32)
    # the device-side loop gives the same tokens as stepping through forward()
    first = tok.copy()
    toks = gpu.generate_greedy(first, 6)[0]
    t = first.copy()
    for step in range(6):
        lo = cpu.forward(t[:, None])
        want = O.top_k(lo[0], 1)[0][0]
        if toks[step] != want:
            assert _margin(lo)[0] < 1e-3, (step, _margin(lo)[0])
            break
        t = np.array([want], dtype=np.uint32)
    assert gpu.position == 291 + 5 + 6


@pytest.mark.parametrize("flagged_rows", [False, True], ids=["grid-barriers", "flagged-rows"])
@pytest.mark.parametrize("n_head,n_kv_head,prompt", [(48, 8, 30), (6, 2, 62)])
def test_decode_across_split_counts(dev, n_head, n_kv_head, prompt, flagged_rows, monkeypatch):
    # The merge of an attention phase: from one split to two and on (a split per 32 keys), more 32-element blocks of the row
    # than CTAs (48 heads of 128) and fewer, launches of one step and of several, whose partial rows carry growing
    # epochs in the same memory. Tolerance of the other decode tests: 2e-3 of the oracle's logits (fp16 cache).
    monkeypatch.setenv("FB200_FUSED_LL", "1" if flagged_rows else "0")
    cfg = dict(tiny_cfg(), ctx=128, head_dim=128, n_head=n_head, n_kv_head=n_kv_head)
    gpu, cpu = build_models(dev, cfg, batch=1, seed=21)
    rng = np.random.default_rng(prompt)
    toks = rng.integers(0, cfg["vocab"], size=(1, prompt + 6), dtype=np.uint32)
    gpu.forward(toks[:, :prompt])
    cpu.forward(toks[:, :prompt])
    for i in range(prompt, prompt + 6):
        lg, _ = gpu.forward(toks[:, i:i + 1])
        lo = cpu.forward(toks[:, i:i + 1])
        assert F.rel_l2(lg, lo) < 2e-3, (i, F.rel_l2(lg, lo))
    first = np.array([O.top_k(lo[0], 1)[0][0]], dtype=np.uint32)
    run = gpu.generate_greedy(first, 34)[0]
    t = first
    for step in range(34):
        lo = cpu.forward(t[:, None])
        if run[step] != O.top_k(lo[0], 1)[0][0]:
            assert _margin(lo)[0] < 1e-3, (step, _margin(lo)[0])
            break
        t = run[step:step + 1].astype(np.uint32)


def test_decode_across_the_wrap_of_the_epochs(dev, monkeypatch):
    # The granules of q, k, v and of the partial rows carry a 32-bit epoch that grows from launch to launch. 0 is what cleared rows carry:
    # a count that would run over it, in a launch of one step or of several, starts again at 1.
    cfg = dict(tiny_cfg(), ctx=128, head_dim=128, n_head=6, n_kv_head=2)
    toks = np.random.default_rng(9).integers(0, cfg["vocab"], size=(1, 46), dtype=np.uint32)
    want = None
    for first in (1, 2**32 - 1, 2**32 - 2, 2**32 - 7, 2**32 - 40, 2**32 - 100, 0):
        monkeypatch.setenv("FB200_FUSED_EPOCH", str(first))
        gpu, _ = build_models(dev, cfg, batch=1, seed=22)
        gpu.forward(toks[:, :40])
        logits = [gpu.forward(toks[:, i:i + 1])[0] for i in range(40, 46)]
        ids = gpu.generate_greedy(toks[0, :1], 30)
        logits.append(gpu.forward(toks[:, :1])[0])
        got = np.stack(logits).view(np.uint32)
        want = want or (got, ids)
        assert np.array_equal(got, want[0]) and np.array_equal(ids, want[1]), first
        gpu.free()
    assert dev.status() == 0


def test_model_loaded_from_a_gguf_file_equals_the_directly_built_one(dev, tmp_path):
    # checkpoint -> GGUF file -> kalosm_b200.gguf.load_llama: same bytes on the device as setting
    # the tensors one by one, so logits and greedy ids agree bit for bit
    from kalosm_b200 import gguf
    cfg = tiny_cfg()
    path = tmp_path / "tiny.gguf"
    write_checkpoint(path, cfg, seed=9)
    direct, cpu = build_models(dev, cfg, batch=1, seed=9)
    loaded = gguf.load_llama(dev, path, max_batch=1)
    prompt = np.random.default_rng(10).integers(0, cfg["vocab"], size=(1, 7), dtype=np.uint32)
    lg_a, nxt_a = direct.forward(prompt)
    lg_b, nxt_b = loaded.forward(prompt)
    assert np.array_equal(lg_a, lg_b) and np.array_equal(nxt_a, nxt_b)
    assert F.rel_l2(lg_b, cpu.forward(prompt)) < 2e-3
    assert np.array_equal(direct.generate_greedy(nxt_a, 8), loaded.generate_greedy(nxt_b, 8))


@pytest.mark.parametrize("flagged_rows", [False, True], ids=["grid-barriers", "flagged-rows"])
def test_decoder_at_llama3_8b_widths(dev, flagged_rows, monkeypatch):
    # both forms of the persistent decode kernel: phases separated by grid barriers (the default) and
    # the barrier-free variant whose phases exchange flagged rows (two-limb activations)
    monkeypatch.setenv("FB200_FUSED_LL", "1" if flagged_rows else "0")
    # the program the benchmark times, two layers deep: hidden 4096, FFN 14336, 32/8 heads of 128,
    # vocabulary 128256, Q4_K body with Q6_K attn_v / ffn_down / output head.
    cfg = dict(llama3_8b_cfg(ctx=256), n_layer=2)
    gpu, cpu = build_models(dev, cfg, batch=1, seed=7)
    rng = np.random.default_rng(8)
    prompt = rng.integers(0, cfg["vocab"], size=(1, 64), dtype=np.uint32)
    lo = cpu.forward(prompt)
    want = O.top_k(lo[0], 1)[0][0]
    # (1) The prompt pass runs the products and the attention on fp16 tensor-core operands. Each
    # of its 15 operations is held to 2e-3 relative L2 on its own (test_gpu_quant, test_gpu_ops);
    # chained through two layers and the head the rounding compounds (about sqrt(15) x 5e-4 per
    # operation, amplified by the norms), so the end-to-end bound for the logits is 8e-3, and the
    # greedy id must agree unless the oracle's own margin is inside the logit error.
    lg, nxt = gpu.forward(prompt)
    assert lg.shape == (1, cfg["vocab"])
    err = F.rel_l2(lg, lo)
    print(f"8B-width prefill (tensor cores): rel-L2 of the logits {err:.2e}")
    assert err < 8e-3, err
    assert nxt[0] == want or _margin(lo)[0] < 4 * np.max(np.abs(lg - lo))
    # (2) The decode path (the fused persistent kernel: integer-limb products, exact to ~1e-6) is
    # held to 2e-3 on the logits of every step. To keep the prompt pass's fp16 rounding out of its
    # KV cache, the same prompt is fed again position by position through that path.
    gpu.reset()
    for i in range(prompt.shape[1]):
        lg, nxt = gpu.forward(prompt[:, i:i + 1])
    err = F.rel_l2(lg, lo)
    print(f"8B-width prompt through the decode path: rel-L2 of the logits {err:.2e}")
    assert err < 2e-3, err
    assert nxt[0] == want or _margin(lo)[0] < 4 * np.max(np.abs(lg - lo))
    tok = np.array([want], dtype=np.uint32)
    worst = 0.0
    for step in range(6):
        lo = cpu.forward(tok[:, None])
        lg, nxt = gpu.forward(tok[:, None])
        worst = max(worst, F.rel_l2(lg, lo))
        assert F.rel_l2(lg, lo) < 2e-3, (step, F.rel_l2(lg, lo))
        want = O.top_k(lo[0], 1)[0][0]
        assert nxt[0] == want or _margin(lo)[0] < 4 * np.max(np.abs(lg - lo)), (step, nxt[0], want)
        tok = np.array([want], dtype=np.uint32)
    print(f"8B-width decode steps: worst rel-L2 of the logits {worst:.2e}")
    # (3) 32 greedy ids out of ONE generate_greedy launch (the persistent kernel running 32 steps)
    first = tok.copy()
    gpu_tokens = gpu.generate_greedy(first, 32)[0]
    assert dev.status() == 0
    t = first.copy()
    for step in range(32):
        lo = cpu.forward(t[:, None])
        want = O.top_k(lo[0], 1)[0][0]
        if gpu_tokens[step] != want:
            # an undecidable step (top-1 / top-2 closer than the logit error) ends the comparison
            assert _margin(lo)[0] < 2e-3 * np.abs(lo).max(), (step, _margin(lo)[0])
            assert step > 8, step
            break
        t = np.array([want], dtype=np.uint32)
    assert gpu.position == 64 + 6 + 32


@pytest.mark.parametrize("hidden", [2048, 2304, 4352, 8448, 14592, 20480])
def test_prompt_norm_of_row_lengths(dev, hidden):
    # more than 32 rows are normalised as they are packed (the second norm with a residual): one to seven pieces of a row per
    # thread, values behind the 14336 that the packing kernel holds in registers are read, and normalised, again. Weights as small
    # as it takes for projections with the spread that they have at a width of 256 (0.3): at 0.02 and 20480 they spread by 2.9 and
    # the scores by 2.9^2 sqrt(64) = 67, so that 2^-11 of a score is 3 % of a softmax weight
    cfg = dict(n_layer=1, hidden=hidden, ffn=256, n_head=4, n_kv_head=2, head_dim=64, vocab=256, ctx=64)
    gpu, cpu = build_models(dev, cfg, batch=1, seed=3, sigma=0.02 * (256 / hidden) ** 0.5)
    prompt = np.random.default_rng(5).integers(0, cfg["vocab"], size=(1, 41), dtype=np.uint32)
    err = F.rel_l2(gpu.forward(prompt)[0], cpu.forward(prompt))
    assert err < 8e-3, err
    assert dev.status() == 0
    gpu.free()


def test_tied_embeddings(dev):
    # no output tensor: the head falls back to token_embd (models/kalosm-llama/src/raw/mod.rs:480-486)
    cfg = tiny_cfg()
    gpu, cpu = build_models(dev, cfg, batch=1, seed=21, tied=True)
    prompt = np.random.default_rng(22).integers(0, cfg["vocab"], size=(1, 7), dtype=np.uint32)
    lg, nxt = gpu.forward(prompt)
    lo = cpu.forward(prompt)
    assert F.rel_l2(lg, lo) < 2e-3
    tok = np.array([O.top_k(lo[0], 1)[0][0]], dtype=np.uint32)
    for _ in range(3):
        lo = cpu.forward(tok[:, None])
        lg, _ = gpu.forward(tok[:, None])
        assert F.rel_l2(lg, lo) < 2e-3
        tok = np.array([O.top_k(lo[0], 1)[0][0]], dtype=np.uint32)


def test_captured_step_survives_scratch_growth(dev):
    # a multi-sequence decode step is a captured CUDA graph that recorded the address of the
    # handle's packed-activation scratch; a larger product on the same handle moves that scratch.
    # The next step must notice and run on the new buffer (compared with the oracle).
    own = kb.Device(0)
    cfg = tiny_cfg()
    gpu, cpu = build_models(own, cfg, batch=2, seed=31)
    rng = np.random.default_rng(32)
    prompt = rng.integers(0, cfg["vocab"], size=(2, 5), dtype=np.uint32)
    gpu.forward(prompt)
    lo = cpu.forward(prompt)
    tok = np.array([O.top_k(lo[b], 1)[0][0] for b in range(2)], dtype=np.uint32)
    lg, _ = gpu.forward(tok[:, None])          # captures the graph
    lo = cpu.forward(tok[:, None])
    assert F.rel_l2(lg, lo) < 2e-3
    # 32 rows of K = 16384: far more packed activations than the tiny model ever needed
    ty, n, k = O.Q4K, 32, 16384
    raw = O.random_qweights(5, 0.02, n * k, ty)
    w = kb.QMatrix.from_raw_bytes(own, (n, k), raw, ty)
    x = rng.standard_normal((32, k)).astype(np.float32)
    y = own.tensor(x).q_mat_mul(w).as_slice()
    assert F.rel_l2(y, O.q_mat_mul(x, raw, ty, n, k)) < 2e-3
    for _ in range(2):
        tok = np.array([O.top_k(lo[b], 1)[0][0] for b in range(2)], dtype=np.uint32)
        lg, _ = gpu.forward(tok[:, None])
        lo = cpu.forward(tok[:, None])
        assert F.rel_l2(lg, lo) < 2e-3
    assert own.status() == 0
    gpu.free()
    w.free()
    own.close()
