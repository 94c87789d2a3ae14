"""GPU engine tests: native executor, CUDA graphs and the overlap scheduler against the
fp32 eager reference of the same model."""

import numpy as np
import pytest
import torch

from modular_b200 import ops
from modular_b200.entrypoints.llm import LLM
from modular_b200.models.llama3 import Llama3Config, Llama3Weights
from modular_b200.pipelines.context import SamplingParams

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    cfg = Llama3Config(hidden_size=512, intermediate_size=1408, num_hidden_layers=3,
                       num_attention_heads=8, num_key_value_heads=2, head_dim=64, vocab_size=2048,
                       max_position_embeddings=2048, rope_theta=500000.0)
    w = Llama3Weights.random_init(cfg, "cuda", torch.bfloat16, seed=0, std=0.05)
    return cfg, w


def _cpu_copy(cfg, w):
    from modular_b200.models.llama3 import LayerWeights

    f = lambda t: t.float().cpu()
    layers = [LayerWeights(*(f(getattr(l, n)) for n in ("attn_norm", "wqkv", "wo", "mlp_norm", "wgu", "wd")))
              for l in w.layers]
    return Llama3Weights(f(w.embed), layers, f(w.final_norm), f(w.lm_head))


def _mk(cfg, w, **kw):
    args = dict(device="cuda", dtype=torch.bfloat16, max_length=1024, max_batch_size=8,
                max_batch_input_tokens=512, page_size=16, num_kv_pages=400)
    args.update(kw)
    return LLM(cfg, w, **args)


def test_executor_logits_match_fp32_reference(small):
    from tests.test_engine_cpu import eager_logits

    cfg, w = small
    rng = np.random.default_rng(0)
    prompt = rng.integers(0, cfg.vocab_size, size=150).tolist()
    llm = _mk(cfg, w, enable_overlap_scheduler=False, device_graph_capture=False)
    llm.generate([prompt], SamplingParams(temperature=0.0, max_new_tokens=1, ignore_eos=True))
    got = llm.model.logits_buf[0].float().cpu()
    ref = eager_logits(cfg, _cpu_copy(cfg, w), prompt)[-1]
    torch.cuda.synchronize()
    ops.check_device_error()
    err = (got - ref).abs().max().item()
    assert err < 0.06 * ref.abs().max().item() + 0.02, err
    assert int(got.argmax()) == int(ref.argmax()) or ref.topk(2).values.diff().abs().item() < 0.05


@pytest.mark.parametrize("T", [1, 17, 33, 64, 65, 128, 129])
def test_small_steps_with_norms_in_their_reductions(small, T):
    """Steps of up to 128 rows hand the norm's factor from layer to layer; a prompt of T tokens and the decode steps after it are as near to
    the fp32 model as steps that run op by op, up to half as much again (single rows, rounded in other places)."""
    from tests.test_engine_cpu import eager_logits

    cfg, w = small
    wc, errs = _cpu_copy(cfg, w), []
    prompt = np.random.default_rng(T).integers(0, cfg.vocab_size, size=T).tolist()
    for native in (True, False):
        llm = _mk(cfg, w, enable_overlap_scheduler=False, device_graph_capture=False, enable_prefix_caching=False)
        if native:
            assert llm.model.executor.lean_usable(T) == (T <= 128)
        llm.model.use_executor = native
        seen, step = [], llm.model.forward_tensors
        llm.model.forward_tensors = lambda *a, **kw: seen.append(step(*a, **kw)) or seen[-1]
        per_step = []
        for new in (1, 2, 5):
            rec = llm.generate([prompt], SamplingParams(temperature=0.0, max_new_tokens=new, ignore_eos=True))[0]
            logits = (llm.model.logits_buf if native else seen[-1])[0].float().cpu()
            ref = eager_logits(cfg, wc, prompt + list(rec.tokens[: new - 1]))[-1]
            per_step.append((logits - ref).norm().item() / ref.norm().item())
        errs.append(per_step)
    ops.check_device_error()
    assert max(errs[0]) <= 1.5 * max(errs[1]) and max(errs[0]) < 0.06, errs


def test_executor_matches_op_by_op(small):
    cfg, w = small
    rng = np.random.default_rng(1)
    prompts = [rng.integers(0, cfg.vocab_size, size=n).tolist() for n in (90, 33, 200)]
    sp = SamplingParams(temperature=0.0, max_new_tokens=6, ignore_eos=True)
    a = _mk(cfg, w, enable_overlap_scheduler=False, device_graph_capture=False).generate(prompts, sp)
    llm_b = _mk(cfg, w, enable_overlap_scheduler=False, device_graph_capture=False)
    llm_b.model.use_executor = False     # same kernels, launched op by op from Python
    b = llm_b.generate(prompts, sp)
    assert [r.tokens for r in a] == [r.tokens for r in b]


def test_qwen2_projection_bias_on_the_executor():
    """Qwen2 layers (bias on the fused q / k / v projection): the native executor adds it after the GEMM on the
    prefill path, the decode-step path and under CUDA graphs, like the op-by-op path does; the bias matters (the
    tokens change without it)."""
    from modular_b200.models.llama3 import Qwen2Config

    cfg = Qwen2Config(hidden_size=512, intermediate_size=1408, num_hidden_layers=3, num_attention_heads=8,
                      num_key_value_heads=2, vocab_size=2048, max_position_embeddings=2048)
    w = Llama3Weights.random_init(cfg, "cuda", torch.bfloat16, seed=2, std=0.05)
    assert w.layers[0].qkv_bias is not None
    for l in w.layers:
        l.qkv_bias.mul_(20.0)          # std 0.05 would drown in the projections
    rng = np.random.default_rng(8)
    prompts = [rng.integers(0, cfg.vocab_size, size=n).tolist() for n in (90, 33, 600)]
    sp = SamplingParams(temperature=0.0, max_new_tokens=6, ignore_eos=True)
    kw = dict(enable_overlap_scheduler=False, device_graph_capture=False, max_batch_input_tokens=1024)
    a = _mk(cfg, w, **kw).generate(prompts, sp)
    llm_b = _mk(cfg, w, **kw)
    llm_b.model.use_executor = False
    b = llm_b.generate(prompts, sp)
    assert [r.tokens for r in a] == [r.tokens for r in b]
    g = _mk(cfg, w, enable_overlap_scheduler=True, device_graph_capture=True, graph_batch_sizes=[4],
            max_batch_input_tokens=1024).generate(prompts, sp)
    assert sum(x.tokens[:3] == y.tokens[:3] for x, y in zip(a, g)) >= 2
    import copy

    w0 = copy.copy(w)
    w0.layers = [copy.copy(l) for l in w.layers]
    for l in w0.layers:
        l.qkv_bias = torch.zeros_like(l.qkv_bias)
    z = _mk(cfg, w0, **kw).generate(prompts, sp)
    assert [r.tokens for r in a] != [r.tokens for r in z]
    torch.cuda.synchronize()
    ops.check_device_error()


def test_qwen3_query_key_norm_on_the_executor():
    """Qwen3 layers (RMSNorm over head_dim on every query and key head before the rotation): the kernel equals the
    fp32 reference, and the native executor (prefill path, decode-step path) gives the tokens of the op-by-op path."""
    from modular_b200.models.llama3 import Qwen3Config
    from modular_b200.ops import reference as ref

    torch.manual_seed(3)
    T, n_q, n_kv, hd = 37, 8, 2, 128
    qkv = torch.randn(T, (n_q + 2 * n_kv) * hd, device="cuda", dtype=torch.bfloat16)
    qw = (1 + 0.2 * torch.randn(hd, device="cuda")).to(torch.bfloat16)
    kw_ = (1 + 0.2 * torch.randn(hd, device="cuda")).to(torch.bfloat16)
    want = qkv.clone()
    for w_, lo, n in ((qw, 0, n_q), (kw_, n_q * hd, n_kv)):
        part = want[:, lo: lo + n * hd].reshape(T * n, hd)
        want[:, lo: lo + n * hd] = ref.rms_norm(part, w_, 1e-6).reshape(T, n * hd)
    got = ops.qk_norm(qkv.clone(), qw, kw_, n_q, n_kv, hd, 1e-6)
    assert torch.equal(got[:, (n_q + n_kv) * hd:], qkv[:, (n_q + n_kv) * hd:])          # values untouched
    assert (got.float() - want.float()).abs().max() <= 0.02 * want.float().abs().max()

    cfg = Qwen3Config(hidden_size=512, intermediate_size=1408, num_hidden_layers=3, num_attention_heads=8,
                      num_key_value_heads=2, head_dim=128, vocab_size=2048, max_position_embeddings=2048)
    w = Llama3Weights.random_init(cfg, "cuda", torch.bfloat16, seed=4, std=0.05)
    for l in w.layers:
        l.q_norm.copy_((1 + 0.3 * torch.randn(128, device="cuda")).to(torch.bfloat16))
        l.k_norm.copy_((1 + 0.3 * torch.randn(128, device="cuda")).to(torch.bfloat16))
    rng = np.random.default_rng(9)
    prompts = [rng.integers(0, cfg.vocab_size, size=n).tolist() for n in (90, 33, 600)]
    sp = SamplingParams(temperature=0.0, max_new_tokens=6, ignore_eos=True)
    kw = dict(enable_overlap_scheduler=False, device_graph_capture=False, max_batch_input_tokens=1024)
    a = _mk(cfg, w, **kw).generate(prompts, sp)
    llm_b = _mk(cfg, w, **kw)
    llm_b.model.use_executor = False
    b = llm_b.generate(prompts, sp)
    assert [r.tokens for r in a] == [r.tokens for r in b]
    torch.cuda.synchronize()
    ops.check_device_error()


@pytest.mark.parametrize("family", ["mixtral", "qwen3_moe"])
def test_llama_family_moe_layers_on_gpu(family):
    """Mixtral / Qwen3-MoE layers on the GPU (router kernel, grouped GEMMs; op-by-op, no native executor): logits
    agree with the fp32 CPU reference of the same weights, and the engine serves several requests."""
    from modular_b200.models.llama3 import MixtralConfig, Qwen3MoeConfig
    from modular_b200.pipelines.speculative import _SeqCache

    cfg = (MixtralConfig.tiny(num_experts=8) if family == "mixtral"
           else Qwen3MoeConfig.tiny(mlp_only_layers=(0,), num_experts=64, num_experts_per_tok=4))
    w = Llama3Weights.random_init(cfg, "cuda", torch.bfloat16, seed=6, std=0.05)
    wc = Llama3Weights.random_init(cfg, "cpu", torch.float32, seed=6, std=0.05)
    assert w.layers[-1].moe is not None
    llm = _mk(cfg, w, enable_overlap_scheduler=False, device_graph_capture=False)
    assert llm.model.use_executor is False
    rng = np.random.default_rng(12)
    prompt = rng.integers(0, cfg.vocab_size, size=70).tolist()
    got = _SeqCache(llm.model, 128).step(prompt, all_logits=True).float().cpu()
    ref_llm = LLM(cfg, wc, device="cpu", dtype=torch.float32, max_length=256, max_batch_size=2,
                  max_batch_input_tokens=128, page_size=16, num_kv_pages=40)
    want = _SeqCache(ref_llm.model, 128).step(prompt, all_logits=True).float()
    # bf16 rounding moves a token across a routing boundary now and then, and that token's logits then differ for
    # a legitimate reason: most rows must agree closely, and on the whole the two must correlate
    row_err = (got - want).abs().amax(dim=1)
    tol = 0.08 * want.abs().max().item() + 0.03
    assert (row_err < tol).float().mean().item() >= 0.7, (row_err.tolist(), tol)
    assert torch.corrcoef(torch.stack([got.flatten(), want.flatten()]))[0, 1].item() > 0.97
    prompts = [rng.integers(0, cfg.vocab_size, size=n).tolist() for n in (90, 33, 200)]
    out = llm.generate(prompts, SamplingParams(temperature=0.0, max_new_tokens=6, ignore_eos=True))
    assert all(len(r.tokens) == 6 for r in out)
    torch.cuda.synchronize()
    ops.check_device_error()


@pytest.mark.parametrize("inflight", [False, True])
def test_overlap_and_graphs_match_sync(small, inflight):
    cfg, w = small
    rng = np.random.default_rng(2)
    prompts = [rng.integers(0, cfg.vocab_size, size=n).tolist() for n in (64, 64, 64, 64, 30, 100, 7)]
    sp = SamplingParams(temperature=0.0, max_new_tokens=12, ignore_eos=True)
    sync = _mk(cfg, w, enable_overlap_scheduler=False, device_graph_capture=False,
               enable_in_flight_batching=inflight, max_batch_input_tokens=96)
    ref = sync.generate(prompts, sp, max_concurrency=4)
    ov = _mk(cfg, w, enable_overlap_scheduler=True, device_graph_capture=True, graph_batch_sizes=[4, 8],
             enable_in_flight_batching=inflight, max_batch_input_tokens=96)
    got = ov.generate(prompts, sp, max_concurrency=4)
    torch.cuda.synchronize()
    ops.check_device_error()
    assert ov.pipeline.stats.graph_replays > 0
    same = sum(r.tokens == g.tokens for r, g in zip(ref, got))
    # batch composition differs between the two schedules, which changes GEMM tile shapes and
    # so the last bits of the logits; require agreement of the first tokens everywhere and of
    # full sequences for most requests
    assert all(r.tokens[:2] == g.tokens[:2] for r, g in zip(ref, got))
    assert same >= len(prompts) - 2
    assert ov.kv.pool.used_blocks == 0


def test_sampling_and_penalties_on_gpu(small):
    cfg, w = small
    rng = np.random.default_rng(3)
    prompts = [rng.integers(0, cfg.vocab_size, size=40).tolist() for _ in range(3)]
    sps = [SamplingParams(temperature=0.8, top_k=40, top_p=0.9, max_new_tokens=10, ignore_eos=True, seed=i)
           for i in range(2)] + [SamplingParams(temperature=0.0, repetition_penalty=1.3, frequency_penalty=0.2,
                                                max_new_tokens=10, ignore_eos=True)]
    llm = _mk(cfg, w)
    recs = llm.generate(prompts, sps)
    torch.cuda.synchronize()
    ops.check_device_error()
    assert all(len(r.tokens) == 10 and all(0 <= t < cfg.vocab_size for t in r.tokens) for r in recs)


# ---------------------------------------------------------------------------- block-scaled fp8 weights
@pytest.fixture(scope="module")
def fp8_model():
    cfg = Llama3Config(hidden_size=1024, intermediate_size=2816, num_hidden_layers=4, num_attention_heads=8,
                       num_key_value_heads=2, head_dim=128, vocab_size=4096, max_position_embeddings=2048)
    w = Llama3Weights.random_init(cfg, "cuda", torch.bfloat16, seed=0, std=0.05).quantize_fp8()
    return cfg, w


def test_fp8_executor_matches_op_by_op_and_dequantised_model(fp8_model):
    """fp8 layers through the native executor (activation quantiser + block-scaled fp8 GEMM per projection):
    same tokens as the same kernels launched op by op, and agreement with the model whose fp8 weights were
    expanded to bf16 (what differs is only the 1 x 128 activation quantisation)."""
    cfg, w = fp8_model
    assert w.layers[0].is_fp8 and w.layers[0].wqkv.dtype == torch.float8_e4m3fn
    rng = np.random.default_rng(5)
    prompts = [rng.integers(0, cfg.vocab_size, size=n).tolist() for n in (150, 40, 300, 17)]
    sp = SamplingParams(temperature=0.0, max_new_tokens=8, ignore_eos=True)
    # 16-token pages: the executor and the op-by-op path then run the same attention kernel, so the two must
    # agree bit for bit
    kw = dict(enable_overlap_scheduler=False, device_graph_capture=False)
    a = _mk(cfg, w, **kw).generate(prompts, sp)
    llm_b = _mk(cfg, w, **kw)
    llm_b.model.use_executor = False
    b = llm_b.generate(prompts, sp)
    torch.cuda.synchronize()
    ops.check_device_error()
    assert [r.tokens for r in a] == [r.tokens for r in b]
    # against the model whose weights were expanded to bf16: random weights give flat logits, so argmax ties
    # flip under the activation quantisation noise; compare the logits themselves
    one = SamplingParams(temperature=0.0, max_new_tokens=1, ignore_eos=True)
    q8 = _mk(cfg, w, **kw)
    q8.generate([prompts[0]], one)
    got = q8.model.logits_buf[0].float().clone()
    bf = _mk(cfg, w.dequantize(), **kw)
    bf.generate([prompts[0]], one)
    want = bf.model.logits_buf[0].float()
    cos = torch.nn.functional.cosine_similarity(got, want, dim=0).item()
    assert cos > 0.9, cos       # e4m3 activations add a few percent of noise per projection
    # and against the fp32 emulation of the very same fp8 arithmetic (PyTorch ops on CPU, same quantisers)
    from modular_b200.models.llama3 import LayerWeights
    cpu = lambda t: None if t is None else t.cpu()
    w_cpu = Llama3Weights(w.embed.cpu(), [LayerWeights(*(cpu(getattr(l, f)) for f in (
        "attn_norm", "wqkv", "wo", "mlp_norm", "wgu", "wd", "wqkv_s", "wo_s", "wgu_s", "wd_s"))) for l in w.layers],
        w.final_norm.cpu(), w.lm_head.cpu())
    emu = LLM(cfg, w_cpu, device="cpu", dtype=torch.bfloat16, max_length=1024, max_batch_size=8,
              max_batch_input_tokens=512, page_size=16, num_kv_pages=400)
    emu.generate([prompts[0]], one)
    want_emu = emu.pipeline.last_logits[0].float()
    # not bit-comparable: a last-bit difference in a bf16 activation can move an e4m3 value to its neighbour
    # (a 6 % step), and four layers of random weights amplify that
    cos = torch.nn.functional.cosine_similarity(got.cpu(), want_emu, dim=0).item()
    assert cos > 0.98, cos
    # with graphs and the overlap scheduler
    c = _mk(cfg, w, graph_batch_sizes=[4]).generate(prompts, sp)
    assert all(x.tokens[:2] == y.tokens[:2] for x, y in zip(a, c))


def test_fp8_checkpoint_roundtrip_keeps_fp8(fp8_model, tmp_path):
    from safetensors.torch import load_file, save_file

    cfg, w = fp8_model
    sd = {k: v.cpu() for k, v in w.to_hf_state_dict(cfg).items()}
    save_file(sd, str(tmp_path / "m.safetensors"))
    w2 = Llama3Weights.from_state_dict(cfg, load_file(str(tmp_path / "m.safetensors")), "cuda", torch.bfloat16)
    assert all(l.is_fp8 for l in w2.layers)
    assert torch.equal(w2.layers[1].wgu.view(torch.uint8), w.layers[1].wgu.view(torch.uint8))
    assert torch.equal(w2.layers[1].wo_s, w.layers[1].wo_s)
    w3 = Llama3Weights.from_state_dict(cfg, load_file(str(tmp_path / "m.safetensors")), "cuda", torch.bfloat16,
                                       keep_fp8=False)
    assert not w3.layers[0].is_fp8 and w3.layers[0].wqkv.dtype == torch.bfloat16
