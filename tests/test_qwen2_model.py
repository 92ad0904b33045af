"""Qwen2 model on the C model API against Hugging Face's Qwen2ForCausalLM with the same random-init weights
(reference: test/test_infer.py:83-148 compares generated tokens with the Hugging Face model under greedy settings).

No checkpoint is read: a small configuration with the real model's head geometry (head_dim 128, GQA, q/k/v biases,
untied output embedding) is initialised from a seed. f32 on CPU must reproduce Hugging Face's greedy tokens exactly;
16-bit runs compare logits within a tolerance and tokens wherever the top-2 margin exceeds it.
"""
import numpy as np
import pytest
import torch

import llaisys_b200 as llaisys

transformers = pytest.importorskip("transformers")

CFG = dict(hidden_size=256, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1, intermediate_size=512,
           vocab_size=320, max_position_embeddings=512, rms_norm_eps=1e-6, rope_theta=10000.0, eos_token_id=319,
           tie_word_embeddings=False)


def hf_model(seed=0, dtype=torch.float32, std=0.08, **overrides):
    cfg = dict(CFG, **overrides)
    torch.manual_seed(seed)
    config = transformers.Qwen2Config(**cfg, attn_implementation="eager")
    model = transformers.Qwen2ForCausalLM(config).eval()
    with torch.no_grad():
        for name, p in model.named_parameters():  # default init leaves biases zero and norms one: make them matter
            if name.endswith("bias"):
                p.normal_(0, 0.1)
            elif "norm" in name:
                p.uniform_(0.5, 1.5)
            else:
                p.normal_(0, std)
    return cfg, model.to(dtype)


def hf_greedy(model, prompt, n_new):
    ids = torch.tensor([prompt])
    with torch.no_grad():
        out = model.generate(ids, attention_mask=torch.ones_like(ids), max_new_tokens=n_new, do_sample=False, top_k=None, top_p=None, temperature=None,
                             eos_token_id=None, pad_token_id=0)
    return out[0].tolist()


def hf_logits(model, tokens):
    with torch.no_grad():
        return model(torch.tensor([tokens])).logits[0].float()


def test_oracle_model_is_pinned_to_hugging_face():
    """The oracle's composition of the per-operator definitions must be Hugging Face's Qwen2: same greedy tokens and
    logits in f32 (this is the comparison the reference's own end-to-end test makes)."""
    from oracle.qwen2 import Qwen2Oracle
    cfg, hf = hf_model(seed=7, num_attention_heads=4, num_key_value_heads=2, hidden_size=512)
    oracle = Qwen2Oracle(cfg, hf.state_dict())
    rng = np.random.default_rng(5)
    for plen, n_new in [(1, 4), (23, 8)]:
        prompt = rng.integers(0, 318, plen).tolist()
        assert oracle.generate(prompt, n_new) == hf_greedy(hf, prompt, n_new)
    oracle.reset()
    prompt = rng.integers(0, 318, 37).tolist()
    assert (oracle.forward(prompt) - hf_logits(hf, prompt)[-1]).abs().max().item() < 2e-4


def make(cfg, model, device=llaisys.DeviceType.CPU, dtype=llaisys.DataType.F32):
    return llaisys.models.Qwen2(config=cfg, state_dict=model.state_dict(), device=device, dtype=dtype)


def test_generate_matches_hugging_face_greedy_f32_cpu():
    cfg, hf = hf_model(seed=1)
    ours = make(cfg, hf)
    rng = np.random.default_rng(0)
    for plen, n_new in [(1, 6), (7, 12), (33, 9)]:  # 33 crosses two pages of the cache
        prompt = rng.integers(0, 318, plen).tolist()
        assert ours.generate(prompt, max_new_tokens=n_new, top_k=1) == hf_greedy(hf, prompt, n_new)


def test_prefill_logits_match_hugging_face_f32_cpu():
    cfg, hf = hf_model(seed=2, num_attention_heads=4, num_key_value_heads=2, hidden_size=512)
    ours = make(cfg, hf)
    prompt = np.random.default_rng(1).integers(0, 318, 21).tolist()
    ours.generate(prompt, max_new_tokens=1)
    got = torch.from_numpy(ours.last_logits())[0]
    want = hf_logits(hf, prompt)[-1]
    assert (got - want).abs().max().item() < 2e-4


def test_tied_embedding_checkpoint_loads():
    cfg, hf = hf_model(seed=3)
    state = {k: v for k, v in hf.state_dict().items() if k != "lm_head.weight"}
    ours = llaisys.models.Qwen2(config=cfg, state_dict=state)
    with torch.no_grad():
        hf.lm_head.weight.copy_(hf.model.embed_tokens.weight)
    prompt = [5, 9, 200]
    assert ours.generate(prompt, max_new_tokens=4) == hf_greedy(hf, prompt, 4)


def test_missing_weight_is_an_error():
    cfg, hf = hf_model(seed=3)
    state = {k: v for k, v in hf.state_dict().items() if "layers.1.mlp.up_proj" not in k}
    with pytest.raises(ValueError, match="lacks"):
        llaisys.models.Qwen2(config=cfg, state_dict=state)


def test_batched_steps_and_decode_loop_equal_single_sequence_runs_cpu():
    """Chunked prefill mixed with decode steps in one batch, then the device-side decode loop: every sequence must get
    the tokens it gets when generated alone."""
    cfg, hf = hf_model(seed=4)
    ours = make(cfg, hf)
    rng = np.random.default_rng(2)
    prompts = [rng.integers(0, 318, n).tolist() for n in (19, 5, 40)]
    n_new = 8
    want = [hf_greedy(hf, p, n_new)[len(p):] for p in prompts]

    ours.configure_cache(4, 64)
    seqs = [ours.add_seq() for _ in prompts]
    # step 1: seq0 first 10 tokens, seq1 whole prompt, seq2 first 16
    nxt = ours.step(seqs, [prompts[0][:10], prompts[1], prompts[2][:16]])
    got = [[], [nxt[1]], []]
    # step 2: seq0 rest of the prompt, seq1 one decode token, seq2 rest
    nxt = ours.step(seqs, [prompts[0][10:], [got[1][-1]], prompts[2][16:]])
    got[0].append(nxt[0]); got[1].append(nxt[1]); got[2].append(nxt[2])
    # seq1 is one token ahead: give the others one plain decode step, then loop all three together
    nxt = ours.step([seqs[0], seqs[2]], [[got[0][-1]], [got[2][-1]]])
    got[0].append(nxt[0]); got[2].append(nxt[1])
    loop = ours.decode_loop(seqs, [g[-1] for g in got], n_new - 2)
    for i in range(3):
        got[i] += loop[:, i].tolist()
        assert got[i] == want[i], f"sequence {i}"
    assert ours.last_loop_ms > 0
    for s in seqs:
        ours.free_seq(s)


def test_model_argument_errors():
    cfg, hf = hf_model(seed=4)
    ours = make(cfg, hf)
    with pytest.raises(llaisys.LlaisysError):
        ours.add_seq()  # cache not configured
    ours.configure_cache(2, 32)
    s = ours.add_seq()
    with pytest.raises(llaisys.LlaisysError):
        ours.step([s], [[400]])  # token out of range
    with pytest.raises(llaisys.LlaisysError):
        ours.step([s], [list(range(40))])  # longer than the configured maximum
    with pytest.raises(llaisys.LlaisysError):
        ours.step([s, s], [[1], [2]])  # same sequence twice
    with pytest.raises(llaisys.LlaisysError):
        ours.step([7], [[1]])  # unknown sequence
    assert ours.step([s], [[1, 2, 3]])[0] in range(320)


def test_sampling_is_seeded_and_respects_top_k():
    cfg, hf = hf_model(seed=5)
    ours = make(cfg, hf)
    a = ours.generate([3, 4, 5], max_new_tokens=6, top_k=5, top_p=0.9, temperature=0.7, seed=11)
    b = ours.generate([3, 4, 5], max_new_tokens=6, top_k=5, top_p=0.9, temperature=0.7, seed=11)
    assert a == b and len(a) <= 9
    logits = np.array([0.0, 5.0, 4.0, -1.0])
    rng = np.random.default_rng(0)
    picks = {llaisys.models.Qwen2._sample(logits, 2, 1.0, 1.0, rng) for _ in range(50)}
    assert picks <= {1, 2}
    assert {llaisys.models.Qwen2._sample(logits, 0, 0.5, 1.0, rng) for _ in range(20)} == {1}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype_name", ["f32", "bf16", "f16"])
def test_model_on_gpu_matches_hugging_face(dtype_name):
    tdt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype_name]
    ldt = {"f32": llaisys.DataType.F32, "bf16": llaisys.DataType.BF16, "f16": llaisys.DataType.F16}[dtype_name]
    # std 0.02 as in a real checkpoint: with larger weights a 1536-wide network saturates its softmaxes and 16-bit
    # rounding (Hugging Face's own bf16 run included) moves logits by 10 % and more
    cfg, hf32 = hf_model(seed=6, std=0.02, num_attention_heads=12, num_key_value_heads=2, hidden_size=1536, intermediate_size=1024)
    hf = hf32.to(tdt).float()  # the rounded weights, evaluated in f32: what a 16-bit run approximates
    ours = llaisys.models.Qwen2(config=cfg, state_dict=hf.state_dict(), device=llaisys.DeviceType.NVIDIA, dtype=ldt)
    rng = np.random.default_rng(3)
    prompts = [rng.integers(0, 318, n).tolist() for n in (150, 33, 64, 1)]
    tol = 2e-3 if dtype_name == "f32" else 0.05
    ours.configure_cache(4, 256)
    seqs = [ours.add_seq() for _ in prompts]
    nxt = ours.step(seqs, prompts)
    logits = torch.from_numpy(ours.last_logits(len(seqs)))
    history = [list(p) for p in prompts]
    for i, p in enumerate(prompts):
        want = hf_logits(hf, p)[-1]
        assert (logits[i] - want).abs().max().item() < tol * max(1.0, want.abs().max().item())
        top2 = want.topk(2).values
        if (top2[0] - top2[1]).item() > 2 * tol * max(1.0, want.abs().max().item()):
            assert nxt[i] == int(want.argmax())
        history[i].append(nxt[i])
    # graph-replayed decode loop: teacher-force Hugging Face with our tokens and compare the last step's logits
    n_steps = 12
    loop = ours.decode_loop(seqs, nxt, n_steps)
    assert loop.shape == (n_steps, len(seqs)) and ours.last_loop_ms > 0
    logits = torch.from_numpy(ours.last_logits(len(seqs)))
    for i in range(len(seqs)):
        fed = history[i] + loop[:-1, i].tolist()
        want_all = hf_logits(hf, fed)
        want = want_all[-1]
        assert (logits[i] - want).abs().max().item() < tol * max(1.0, want.abs().max().item())
        # every looped token must be (near-)optimal under the reference's logits at its position
        for s in range(n_steps):
            row = want_all[len(history[i]) - 1 + s]
            assert (row.max() - row[loop[s, i]]).item() <= 2 * tol * max(1.0, row.abs().max().item())
    # the eager single-step path must agree with the replayed loop on a fresh copy of the sequences
    ours.configure_cache(4, 256)
    seqs = [ours.add_seq() for _ in prompts]
    cur = ours.step(seqs, prompts)
    assert cur == nxt
    for s in range(n_steps):
        cur = ours.step(seqs, [[t] for t in cur])
        assert cur == loop[s].tolist(), f"step {s}"


@pytest.mark.gpu
def test_cached_step_graph_survives_a_first_prefill_nvidia():
    """Eight sequences decode from one-token prompts until their step is replayed from its cached CUDA graph; then the
    cache serves its FIRST prompt chunk (another sequence, fewer rows than the workspace holds) and a decode step of
    another batch size, and the eight are stepped again through the old graph. Everything the captured kernels point at --
    the attention workspace of the cache included -- must still be where it was: every token of every step has to be
    (near-)optimal under Hugging Face's logits for the tokens fed so far."""
    tol = 0.05
    cfg, hf32 = hf_model(seed=8, std=0.02, num_attention_heads=12, num_key_value_heads=2, hidden_size=1536, intermediate_size=1024)
    hf = hf32.to(torch.bfloat16).float()
    ours = llaisys.models.Qwen2(config=cfg, state_dict=hf.state_dict(), device=llaisys.DeviceType.NVIDIA,
                                dtype=llaisys.DataType.BF16)
    ours.configure_cache(10, 64)
    rng = np.random.default_rng(4)
    seqs = [ours.add_seq() for _ in range(8)]
    history = [[int(t)] for t in rng.integers(0, 318, 8)]

    def step_eight():
        nxt = ours.step(seqs, [[h[-1]] for h in history])
        for h, t in zip(history, nxt):
            h.append(t)

    for _ in range(4):  # step 1 eager, step 2 captures the graph, steps 3-4 replay it
        step_eight()
    other = ours.add_seq()
    prompt = rng.integers(0, 318, 5).tolist()
    first = ours.step([other], [prompt])[0]  # the cache's first chunk call
    more = ours.add_seq()
    ours.step([other, more], [[first], [7]])  # a decode step of another batch size
    for _ in range(3):  # the eight again, through the graph captured before all that
        step_eight()
    for h in history:
        rows = hf_logits(hf, h[:-1])
        for pos in range(len(h) - 1):
            row = rows[pos]
            assert (row.max() - row[h[pos + 1]]).item() <= 2 * tol * max(1.0, row.abs().max().item()), (h, pos)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("hidden,inter,vocab", [(256, 512, 321), (264, 6400, 320), (1536, 200, 1001), (512, 12008, 64), (256, 36, 320)])
def test_single_rows_take_one_launch_per_projection_nvidia(cuda_device, dtype, hidden, inter, vocab):
    """One token of one sequence runs norm + projection + what follows in single launches: depths that one warp and that eight warps share,
    odd output counts, a depth past the kernel's bound and one that is not made of 16-byte pieces (general path). The logits after several
    steps lie no further from the f32 model than those of the general path, give or take the two paths' rounding."""
    kind, t = (llaisys.DataType.BF16, torch.bfloat16) if dtype == "bf16" else (llaisys.DataType.F16, torch.float16)
    cfg, hf = hf_model(seed=3, std=0.03, hidden_size=hidden, intermediate_size=inter, vocab_size=vocab, head_dim=128)
    hf = hf.to(t).float()  # the rounded weights, in f32
    prompt = np.random.default_rng(hidden).integers(0, min(vocab, 300), 21).tolist()
    want = hf_logits(hf, prompt)[-1]
    off = {}
    for policy in (0, 2):
        llaisys.Ops.set_linear_policy(policy)
        try:
            model = make(cfg, hf.to(t), llaisys.DeviceType.NVIDIA, kind)
            seq = model.add_seq() if model.configure_cache(1, 64) is None else -1
            for token in prompt:  # (the first steps run eagerly, the later ones as a graph)
                model.step([seq], [[token]])
            off[policy] = (torch.from_numpy(model.last_logits()[0]) - want).norm().item() / want.norm().item()
            hf = hf.float()
        finally:
            llaisys.Ops.set_linear_policy(0)
    assert off[0] <= 1.5 * off[2] + {"bf16": 2 ** -8, "f16": 2 ** -11}[dtype], off
