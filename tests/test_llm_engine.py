"""End-to-end numerics of the CUDA LLM program against the PyTorch fp32 reference model."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["bf16", "int4", "moe", "moe-gather", "bf16-u8kv"])
def test_tiny_llama_generate_matches_reference(fmt, monkeypatch):
    from openvino_b200.genai.pipeline import ContinuousBatchingPipeline, GenerationConfig
    from openvino_b200.genai.scheduler import SchedulerConfig
    from openvino_b200.models import llama
    from openvino_b200.models.llm_config import TINY_LLAMA, TINY_MOE
    from openvino_b200.ops import cuda as K
    from openvino_b200.runtime.cuda_llm import CudaLlmExecutor, LlmWeights, StepShape

    if fmt == "moe-gather":
        # prefill batches take the path that runs every expert on its own (gathered) tokens only
        from openvino_b200.runtime import cuda_llm
        monkeypatch.setattr(cuda_llm, "MOE_GATHER_MIN_TOKENS", 8)
    cfg = TINY_MOE if fmt.startswith("moe") else TINY_LLAMA.with_(weight_format=fmt.split("-")[0])
    state = llama.random_float_state(cfg, seed=3, std=0.05)
    eff = {k: v.cuda() for k, v in llama.effective_state(cfg, state).items()}
    w = LlmWeights.from_float(cfg, state, "cuda")
    # "-u8kv": KV_CACHE_PRECISION = u8 (rows quantised per token and head by the cache-write kernel)
    ex = CudaLlmExecutor(cfg, w, num_kv_blocks=64, max_batch_tokens=256, max_seqs=4, kv_cache_precision="u8" if fmt.endswith("u8kv") else "bf16")
    sc = SchedulerConfig(max_num_batched_tokens=48, max_num_seqs=4, num_kv_blocks=64)   # forces chunked prefill
    pipe = ContinuousBatchingPipeline(ex, sc)
    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (5, 37, 70, 16)]
    res = pipe.generate(prompts, GenerationConfig(max_new_tokens=6), lookahead=1 if fmt == "int4" else 0)
    K.check_status("llm")
    assert pipe.metrics.prefill_steps >= 3 and pipe.metrics.decode_steps >= 5
    for p, r in zip(prompts, res):
        # teacher-forced check: at every generated position the engine's token must be the reference
        # argmax, or a near-tie of it (bf16 activations vs fp32 reference)
        seq = p + r.tokens
        logits = llama.reference_logits(cfg, eff, torch.tensor(seq[:-1], device="cuda"))
        for i, tok in enumerate(r.tokens):
            row = logits[len(p) - 1 + i]
            assert row[tok] >= row.max() - 0.05 * row.abs().max(), (i, tok, int(row.argmax()))


def test_logits_close_to_reference():
    from openvino_b200.models import llama
    from openvino_b200.models.llm_config import TINY_LLAMA
    from openvino_b200.runtime.cuda_llm import CudaLlmExecutor, LlmWeights, StepShape
    import numpy as np

    cfg = TINY_LLAMA.with_(weight_format="int4")
    state = llama.random_float_state(cfg, seed=5, std=0.05)
    eff = {k: v.cuda() for k, v in llama.effective_state(cfg, state).items()}
    ex = CudaLlmExecutor(cfg, LlmWeights.from_float(cfg, state, "cuda"), num_kv_blocks=16, max_batch_tokens=128, max_seqs=2,
                         use_cuda_graphs=False)
    ids = torch.randint(0, cfg.vocab_size, (50,))
    sb = ex.prefill
    v = {n: sb.view(n, host=0).numpy() for n in sb.offsets}
    v["ids"][:50] = ids.numpy()
    v["positions"][:50] = np.arange(50)
    v["slot_map"][:50] = np.arange(50) + 16 * 3          # blocks 3,4,5,6
    v["tok_src"][:50] = -1
    v["tok_dst"][0] = -1
    v["logit_idx"][0] = 49
    v["past_lens"][0] = 0
    v["subsequence_begins"][:2] = [0, 50]
    v["block_indices_begins"][:2] = [0, 4]
    v["block_indices"][:4] = [3, 4, 5, 6]
    ex.upload(sb)
    ex.run(sb, StepShape(50, 1, 50, 50))
    torch.cuda.synchronize()
    ref = llama.reference_logits(cfg, eff, ids.cuda())[-1]
    got = sb.logits[0].float()
    rel = ((got - ref).norm() / ref.norm()).item()
    assert rel < 3e-2, rel


@pytest.mark.parametrize("native", [True, False])
def test_python_and_native_scheduler_generate_the_same_tokens(native):
    from openvino_b200.genai.pipeline import ContinuousBatchingPipeline, GenerationConfig
    from openvino_b200.genai.scheduler import SchedulerConfig
    from openvino_b200.models import llama
    from openvino_b200.models.llm_config import TINY_LLAMA
    from openvino_b200.ops import cuda as K
    from openvino_b200.runtime.cuda_llm import CudaLlmExecutor, LlmWeights

    cfg = TINY_LLAMA
    state = llama.random_float_state(cfg, seed=9, std=0.05)
    g = torch.Generator().manual_seed(2)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (40, 9, 25)]
    out = []
    for use_native in (native, not native):
        ex = CudaLlmExecutor(cfg, LlmWeights.from_float(cfg, state, "cuda"), num_kv_blocks=64, max_batch_tokens=128, max_seqs=4)
        sc = SchedulerConfig(max_num_batched_tokens=32, max_num_seqs=4, num_kv_blocks=64, use_native=use_native)
        out.append([r.tokens for r in ContinuousBatchingPipeline(ex, sc).generate(prompts, GenerationConfig(max_new_tokens=6), lookahead=1)])
        K.check_status("generate")
    assert out[0] == out[1]


def test_prefix_caching_reuses_kv_blocks_and_keeps_the_tokens():
    from openvino_b200.genai.pipeline import ContinuousBatchingPipeline, GenerationConfig
    from openvino_b200.genai.scheduler import SchedulerConfig
    from openvino_b200.models import llama
    from openvino_b200.models.llm_config import TINY_LLAMA
    from openvino_b200.ops import cuda as K
    from openvino_b200.runtime.cuda_llm import CudaLlmExecutor, LlmWeights

    cfg = TINY_LLAMA
    state = llama.random_float_state(cfg, seed=11, std=0.05)
    g = torch.Generator().manual_seed(4)
    system = torch.randint(0, cfg.vocab_size, (70,), generator=g).tolist()          # shared "system prompt": four full blocks
    prompts = [system + torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (5, 11, 3)]
    gen = GenerationConfig(max_new_tokens=5)
    results = {}
    for caching in (False, True):
        ex = CudaLlmExecutor(cfg, LlmWeights.from_float(cfg, state, "cuda"), num_kv_blocks=64, max_batch_tokens=128, max_seqs=4)
        sc = SchedulerConfig(max_num_batched_tokens=128, max_num_seqs=4, num_kv_blocks=64, enable_prefix_caching=caching)
        pipe = ContinuousBatchingPipeline(ex, sc)
        first = pipe.generate(prompts[:1], gen, lookahead=0)          # fills the cache
        rest = pipe.generate(prompts[1:], gen, lookahead=0)           # later requests with the same prefix
        K.check_status("prefix caching")
        results[caching] = ([r.tokens for r in first + rest], pipe.metrics.scheduled_tokens,
                            getattr(pipe.scheduler, "prefix_hit_tokens", 0))
    assert results[True][0] == results[False][0]
    assert results[True][2] == 2 * 64                                  # two later requests x four cached blocks of 16 tokens
    assert results[True][1] == results[False][1] - 2 * 64


def _fill_step(ex, spans, blocks, vocab, seed):
    """A step of ``spans`` (earlier tokens, new tokens) whose blocks are handed out in turn."""
    import numpy as np
    from openvino_b200.genai.pipeline import step_shape
    from openvino_b200.genai.scheduler import Scheduler, SchedulerConfig, Sequence
    rng = np.random.RandomState(seed)
    T = sum(n for _, n in spans)
    sched = Scheduler(SchedulerConfig(max_num_batched_tokens=max(T, 64), max_num_seqs=len(spans), num_kv_blocks=blocks, block_size=16))
    free, seqs = list(rng.permutation(blocks)), []
    for i, (past, n) in enumerate(spans):
        s = Sequence(i, rng.randint(0, vocab, past + n).astype(np.int32), 0)
        s.num_computed, s.blocks = past, [int(free.pop()) for _ in range((past + n + 15) // 16)]
        sched.admit(s)
        seqs.append(s)
    step = sched.place(seqs, [n for _, n in spans])
    sb = ex.decode if step.max_q_len == 1 and len(seqs) <= ex.decode.Bcap else ex.prefill
    sched.fill(step, {name: sb.view(name, host=0).numpy() for name in sb.offsets})
    return sb, step_shape(step)


STEPS = [
    [(33, 1)],                                              # norms inside the products, the rotation inside the attention
    [(700, 1), (3, 1), (15, 1), (16, 1)],
    [(5 * i, 1) for i in range(5)],                         # the gathered norm as a launch of its own
    [(1100 + i, 1) for i in range(65)],                     # rotation, attention and sum as launches of their own
    [(40, 1), (0, 37), (100, 20), (7, 1)],                  # decoding beside portions of prompts
    [(0, 1023)], [(0, 1025)],
]


@pytest.mark.parametrize("fmt,kv,gate,bias,window", [("int4", "bf16", True, False, 0), ("bf16", "bf16", True, False, 100), ("int8", "u8", True, False, 0),
                                                     ("fp8", "bf16", False, False, 0), ("bf16", "u8", False, True, 0), ("int4", "bf16", False, True, 0)])
def test_native_step_against_the_launches_one_by_one(fmt, kv, gate, bias, window, monkeypatch):
    """One call into the kernel library against `_forward`'s own launches: logits, tokens and all cache rows. Where they differ, 32-bit sums were added in
    another order, so that a 16-bit value between two kernels is a neighbour now and then: far less than the 2^-8 of rounding all of them once. A
    wrong pointer, size, flag or stride shows as a difference of the order of one."""
    from openvino_b200.models.llm_config import TINY_LLAMA
    from openvino_b200.ops import cuda as K
    from openvino_b200.runtime.cuda_llm import CudaLlmExecutor, LlmWeights

    cfg = TINY_LLAMA.with_(weight_format=fmt, sliding_window=window)
    w = LlmWeights.random(cfg, "cuda", seed=4)
    g = torch.Generator(device="cuda").manual_seed(1)
    for lw in w.layers:
        lw.gate_up.swiglu = gate
        lw.norm1.normal_(1.0, 0.1, generator=g)
        lw.norm2.normal_(1.0, 0.1, generator=g)
        for p in (lw.qkv, lw.o, lw.gate_up, lw.down) if bias else ():
            p.bias = torch.randn(p.N, device="cuda", generator=g).bfloat16()
    w.final_norm.normal_(1.0, 0.1, generator=g)
    blocks = 65 * 73
    ex = CudaLlmExecutor(cfg, w, blocks, max_batch_tokens=1100, max_seqs=65, max_blocks_per_seq=80, use_cuda_graphs=False, kv_cache_precision=kv)
    caches = [t for t in ex.k_cache + ex.v_cache + ex.k_meta + ex.v_meta if t is not None]
    for t in caches:
        t.copy_(torch.randint(100, 156, t.shape, device="cuda", generator=g).to(t.dtype) if t.dtype == torch.uint8 else
                torch.rand(t.shape, device="cuda", generator=g) * 0.01 + 0.01 if t.dtype == torch.float16 else torch.randn(t.shape, device="cuda", generator=g))
    before = [t.clone() for t in caches]

    def rel(a, b):
        a, b = a.double(), b.double()
        return float((a - b).norm() / b.norm())
    for n, spans in enumerate(STEPS):
        sb, shape = _fill_step(ex, spans, blocks, cfg.vocab_size, n)
        got = []
        for native in (True, False):
            for t, v in zip(caches, before):
                t.copy_(v)
            sb.logits.zero_()
            ex.last_token.fill_(-7)
            monkeypatch.setattr(CudaLlmExecutor, "_is_native", lambda self, native=native: native)
            ex.upload(sb)
            tokens = ex.run(sb, shape)
            got.append((sb.logits[:shape.B].clone(), tokens.clone(), ex.last_token.clone(), [t.clone() for t in caches]))
        K.check_status("native step")
        (la, ta, fa, ca), (lb, tb, fb, cb) = got
        assert rel(la, lb) < 2.0 ** -8, (n, rel(la, lb))
        best = lb.float().gather(1, ta.long()[:, None])[:, 0]
        assert (best >= lb.float().max(1).values - 0.02 * lb.float().abs().max()).all(), n        # the same token, or one as good
        assert torch.equal(fa == -7, fb == -7)
        slots = sb.view("slot_map")[:shape.T].long()
        new = torch.zeros(blocks * 16, dtype=torch.bool, device="cuda")
        new[slots] = True
        new = new.reshape(blocks, 1, 16, 1)
        for a, b, v in zip(ca, cb, before):
            assert torch.equal(a.masked_fill(new, 0), v.masked_fill(new, 0)), n                   # nothing but the step's rows was written
            a, b = (t.permute(0, 2, 1, 3).reshape(blocks * 16, -1)[slots] for t in (a, b))
            if a.dtype == torch.uint8:
                assert (a.int() - b.int()).abs().max() <= 2, n
            else:
                assert rel(a, b) < 2.0 ** -8, n


def test_native_step_shares_the_memory_for_expanded_weights(monkeypatch):
    """Quantised products of many tokens expand their weights: one piece of memory for the four products of a layer, sized for the largest."""
    from openvino_b200.models.llm_config import LLAMA3_8B
    from openvino_b200.ops import cuda as K
    from openvino_b200.runtime.cuda_llm import CudaLlmExecutor, LlmWeights

    cfg = LLAMA3_8B.with_(num_layers=1, vocab_size=512)
    ex = CudaLlmExecutor(cfg, LlmWeights.random(cfg, "cuda", seed=2), 80, max_batch_tokens=1100, max_seqs=1, max_blocks_per_seq=80, use_cuda_graphs=False)
    asked, plain = [], K._gemm_scratch
    monkeypatch.setattr(K, "_gemm_scratch", lambda n, d: asked.append(n) or plain(n, d))
    for T in (1023, 1024, 1100):
        sb, shape = _fill_step(ex, [(0, T)], 80, cfg.vocab_size, T)
        out = []
        for native in (True, False):
            monkeypatch.setattr(CudaLlmExecutor, "_is_native", lambda self, native=native: native)
            del asked[:]
            ex.upload(sb)
            ex.run(sb, shape)
            out.append((sb.logits[:1].clone(), ex.k_cache[0].clone(), ex.v_cache[0].clone(), max(asked, default=0)))
        K.check_status("native step")
        assert (out[0][3] > 0) == (T >= 1024) and out[0][3] == out[1][3]
        assert all(torch.equal(a, b) for a, b in zip(out[0][:3], out[1][:3])), T                  # the same kernels in the same order
