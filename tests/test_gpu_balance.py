"""Decode steps whose attention deals its blocks out by the requests' lengths, through the engine: layers of different kv heads in
one model, steps launched, recorded and replayed while lengths grow, a batch that becomes even and uneven again. Against the
model written out in float64."""
import math

import pytest
import torch

from tests.util import TOL, max_rel_diff, random_tokens

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAME = "ToyUnevenHeads"
HIDDEN, HEADS, HD, INTER, VOCAB, EPS = 256, 16, 64, 256, 97, 1e-5


def _register():
    from dataclasses import dataclass
    from vllm_oxide_b200.config import Architecture, register_architecture
    from vllm_oxide_b200.parts import Attention, Block, Embedding, LayerCall, LMHead, ModelSpec, RMSNorm, SwiGLU
    from vllm_oxide_b200.weights import TensorSpec

    @dataclass(frozen=True)
    class ToyConfig:
        kv_heads: tuple

    def manifest(c):
        m = {"emb": TensorSpec((VOCAB, HIDDEN)), "final": TensorSpec((HIDDEN,))}
        for i, kv in enumerate(c.kv_heads):
            m |= {f"l{i}.q": TensorSpec((HEADS * HD, HIDDEN)), f"l{i}.k": TensorSpec((kv * HD, HIDDEN)), f"l{i}.v": TensorSpec((kv * HD, HIDDEN)),
                  f"l{i}.o": TensorSpec((HIDDEN, HEADS * HD)), f"l{i}.n1": TensorSpec((HIDDEN,)), f"l{i}.n2": TensorSpec((HIDDEN,)),
                  f"l{i}.gate": TensorSpec((INTER, HIDDEN)), f"l{i}.up": TensorSpec((INTER, HIDDEN)), f"l{i}.down": TensorSpec((HIDDEN, INTER))}
        return m

    def build(c, w, ctx):
        emb = Embedding(w.take("emb"), ctx.dtype, ctx.device)
        blocks = [Block(RMSNorm(w.take(f"l{i}.n1"), EPS, ctx.device),
                        Attention(*(w.take(f"l{i}.{x}") for x in "qkvo"), HEADS, kv, HD, dtype=ctx.dtype, device=ctx.device),
                        RMSNorm(w.take(f"l{i}.n2"), EPS, ctx.device),
                        SwiGLU(w.take(f"l{i}.gate"), w.take(f"l{i}.up"), w.take(f"l{i}.down"), ctx.dtype, ctx.device))
                  for i, kv in enumerate(c.kv_heads)]
        spec = ModelSpec(embedding=emb, blocks=blocks, schedule=[LayerCall(i, i) for i in range(len(blocks))],
                         final_norm=RMSNorm(w.take("final"), EPS, ctx.device), lm_head=LMHead(emb.table), hidden_size=HIDDEN, vocab_size=VOCAB)
        w.finish()
        return spec
    arch = Architecture(NAME, ToyConfig, manifest, build)
    register_architecture(arch, replace=True)
    return arch, ToyConfig


def _tensors(arch, cfg):
    """An output head that prefers the token it was given: the tokens are then the same whatever the rounding."""
    g = torch.Generator().manual_seed(9)
    std = {"emb": (1.0, 0.0), "final": (0.0, 0.05), "n1": (0.0, 1.0), "n2": (0.0, 1.0), "q": (0.06, 0.0), "k": (0.06, 0.0), "v": (0.2, 0.0),
           "o": (0.01, 0.0), "gate": (0.05, 0.0), "up": (0.05, 0.0), "down": (0.02, 0.0)}
    got = {}
    for name, spec in arch.manifest(cfg).items():
        s, m = std[name.split(".")[-1]]
        got[name] = (torch.randn(spec.shape, generator=g) * s + m).to(torch.bfloat16)
    return got


def _plain_logits(cfg, tensors, tokens):
    """The logits behind the last token, in float64."""
    t = {k: v.to(DEV).double() for k, v in tensors.items()}
    T = len(tokens)
    norm = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)  # noqa: E731
    x = t["emb"][torch.tensor(tokens, device=DEV)]
    mask = torch.full((T, T), -math.inf, device=DEV, dtype=torch.float64).triu(1)
    for i, kv in enumerate(cfg.kv_heads):
        n = norm(x) * t[f"l{i}.n1"]
        q, k, v = (n @ t[f"l{i}.{c}"].T for c in "qkv")
        heads = [torch.softmax(q[:, h * HD:(h + 1) * HD] @ k[:, (s := h // (HEADS // kv)) * HD:(s + 1) * HD].T / 8 + mask, -1)
                 @ v[:, s * HD:(s + 1) * HD] for h in range(HEADS)]
        x = x + torch.cat(heads, 1) @ t[f"l{i}.o"].T
        n = norm(x) * t[f"l{i}.n2"]
        x = x + (torch.nn.functional.silu(n @ t[f"l{i}.gate"].T) * (n @ t[f"l{i}.up"].T)) @ t[f"l{i}.down"].T
    return ((norm(x[-1:]) * t["final"]) @ t["emb"].T)[0].cpu()


def _engine(kv_heads):
    from vllm_oxide_b200.config import EngineConfig
    from vllm_oxide_b200.engine import LLM, ModelRunner
    arch, ToyConfig = _register()
    cfg = ToyConfig(kv_heads)
    tensors = _tensors(arch, cfg)
    runner = ModelRunner(cfg, dict(tensors), EngineConfig(max_batch_tokens=1024, max_seqs=8, max_model_len=4096, block_size=16, num_pages=300,
                                                          dtype="bfloat16"), arch)
    return LLM(runner), cfg, tensors


def _generate(llm, cfg, tensors, prompts, new, wanted):
    from vllm_oxide_b200.sampling import SamplingParams
    outs = llm.generate(prompts, [SamplingParams(max_new_tokens=n, stop_token_ids=(), capture_logits=w) for n, w in zip(new, wanted)])
    for p, o, n, w in zip(prompts, outs, new, wanted):
        assert len(o.token_ids) == n and sorted(o.logits) == list(w)
        for i in w:
            assert max_rel_diff(o.logits[i], _plain_logits(cfg, tensors, p + o.token_ids[:i])) <= TOL[torch.bfloat16], (len(p), i)
    return outs


LENGTHS = (31, 2600, 50, 20, 44, 76, 33, 60)


def test_layers_of_different_kv_heads_are_balanced_each_by_its_own(monkeypatch):
    from vllm_oxide_b200.config import unregister_architecture
    from vllm_oxide_b200.tuning import TUNING
    monkeypatch.setattr(TUNING, "balance_tiles", 2)
    try:
        llm, cfg, tensors = _engine((8, 16))
        prompts = [random_tokens(n, VOCAB, 40 + n) for n in LENGTHS]
        for _ in range(2):
            _generate(llm, cfg, tensors, prompts, [6] * 8, [(2, 5)] * 8)
        sms = torch.cuda.get_device_properties(DEV).multi_processor_count
        assert (((8, HD), min(64, 3 * sms // 8)), ((16, HD), min(64, 3 * sms // 16))) in {key[4] for key in llm.runner._graphs}
    finally:
        unregister_architecture(NAME)


def test_batches_that_become_even_and_uneven_again(monkeypatch):
    """The long request ends first: its steps are balanced, those behind are not, and the next call begins balanced again. Launched
    one by one, recorded and replayed at other lengths; a call whose steps are all replayed gives the bits of the one before."""
    from vllm_oxide_b200.config import unregister_architecture
    from vllm_oxide_b200.tuning import TUNING
    monkeypatch.setattr(TUNING, "balance_tiles", 2)
    try:
        llm, cfg, tensors = _engine((8, 8))
        prompts = [random_tokens(n, VOCAB, 40 + n) for n in LENGTHS]
        new = [9 if n > 2000 else 20 for n in LENGTHS]
        wanted = [(3, n - 1) for n in new]
        got = [_generate(llm, cfg, tensors, prompts, new, wanted) for _ in range(4)]
        balances = {key[4] for key in llm.runner._graphs}
        assert () in balances and len(balances) == 2 and llm.stats["ahead_steps"] > 0
        for a, b in zip(got[2], got[3]):
            assert a.token_ids == b.token_ids and all(torch.equal(a.logits[i], b.logits[i]) for i in a.logits)
        # other lengths on the same recordings
        _generate(llm, cfg, tensors, [random_tokens(n, VOCAB, 90 + n) for n in (3000, 70, 20, 90, 33, 45, 28, 61)], [9, 20, 20, 20, 20, 20, 20, 20], [(8,)] + [(19,)] * 7)
    finally:
        unregister_architecture(NAME)
