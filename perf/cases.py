"""The work this framework is used for, as timed cases: training steps, scoring and text generation through
``MerakTrainer`` and its engine, from one short prompt to a pre-training step of BERT-large.

Every case builds a model of one family at the widths of this repository's own configurations
(``models.{bert,gpt2,llama,moe}`` presets, ``bench.py``, ``bench_configs.py``), hands it to a trainer, and then makes
the call a training or serving loop makes once per batch.  Deep models are cut to a few layers of their real width,
as ``bench_configs.py --layers`` does.  Data are synthetic, weights random-init.

``mode``
    ``train``     one ``engine.train_batch``: forward, backward, clip and AdamW over ``accum`` micro-batches
    ``score``     one ``engine.eval_batch`` that returns the logits (evaluation, scoring, a prompt's first pass)
    ``generate``  ``text_generation_pipeline.generate`` greedily, and the logits of what came out
"""
from __future__ import annotations

import math
import os

os.environ.setdefault("MERAK_QUIET", "1")

import torch  # noqa: E402

import merak_b200 as Merak  # noqa: E402
from merak_b200.inference import text_generation_pipeline  # noqa: E402
from merak_b200.models.bert import BertForMaskedLM, bert_config  # noqa: E402
from merak_b200.models.gpt2 import GPT2LMHeadModel, gpt2_config  # noqa: E402
from merak_b200.models.llama import LlamaForCausalLM, llama_config  # noqa: E402
from merak_b200.models.moe import DeepseekV2ForCausalLM, deepseek_v2_config  # noqa: E402
from merak_b200.parallel import mpu  # noqa: E402

# Widths by preset: hidden, layers, heads, ffn, vocab.  kv heads equal heads unless a case says otherwise.
_WIDTHS = {
    "bert-base": dict(family="bert", hidden=768, layers=12, heads=12, ffn=3072, vocab=30522),
    "bert-large": dict(family="bert", hidden=1024, layers=24, heads=16, ffn=4096, vocab=30522),
    "gpt2": dict(family="gpt2", hidden=768, layers=12, heads=12, ffn=3072, vocab=50257),
    "gpt2-medium": dict(family="gpt2", hidden=1024, layers=24, heads=16, ffn=4096, vocab=50257),
    "gpt2-xl": dict(family="gpt2", hidden=1600, layers=48, heads=25, ffn=6400, vocab=50257),
    "llama-7b": dict(family="llama", hidden=4096, layers=32, heads=32, ffn=11008, vocab=32000),
    "deepseek-v2-lite": dict(family="moe", hidden=2048, layers=27, heads=16, ffn=10944, vocab=102400),
}
_KV_LORA, _QK_DIM, _ROPE_DIM, _V_DIM, _EXPERT_FFN, _TOP_K, _SHARED = 512, 192, 64, 128, 1408, 6, 2


def _case(model, mode, batch, seq, name=None, **more):
    w = _WIDTHS[model]
    c = dict(model=model, mode=mode, layers=w["layers"], heads=w["heads"], kv_heads=w["heads"], hidden=w["hidden"],
             ffn=w["ffn"], vocab=w["vocab"], experts=0, batch=batch, seq=seq, accum=1, new_tokens=0, dropout=0.0,
             attn_dropout=0.0, padded=False, graph=False, recompute=False)
    c.update(more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # bench.py's default workload: BERT-large masked-LM pre-training, captured step, hidden dropout as published
        _case("bert-large", "train", 32, 512, "bert-large-pretrain", dropout=0.1, graph=True),
        # fine-tuning BERT-base on short padded sentences, eager: many launches on little data
        _case("bert-base", "train", 6, 77, "bert-base-short", dropout=0.1, attn_dropout=0.1, padded=True),
        # GPT-2 training with the trainer's default recomputation, the model's default dropouts (attention
        # probabilities too) and gradient accumulation
        _case("gpt2", "train", 8, 1024, "gpt2-accum", dropout=0.1, attn_dropout=0.1, accum=2, recompute=True),
        # the GPT-2 1.5B workload of bench_configs.py (25 heads, width 1600, vocabulary 50257), six layers of it
        _case("gpt2-xl", "train", 4, 1024, "gpt2-xl-layers", layers=6, recompute=True),
        # the Llama-7B workload of bench_configs.py, two layers of it: long causal rows, head dim 128, SwiGLU, RoPE
        _case("llama-7b", "train", 1, 4096, "llama-7b-layers", layers=2),
        # grouped-query Llama on ragged lengths (no tile divides 1001 tokens), captured step
        _case("llama-7b", "train", 3, 1001, "llama-gqa-ragged", layers=4, hidden=2048, heads=16, kv_heads=4, ffn=5504,
              graph=True),
        # the DeepSeek-V2-Lite shape of bench_configs.py: a dense and a mixture-of-experts layer with the experts
        # one rank holds there (8) doubled, top-6 routing, latent attention
        _case("deepseek-v2-lite", "train", 1, 2048, "moe-layers", layers=2, experts=16),
        # scoring full documents with GPT-2-medium: forward only, whole logits
        _case("gpt2-medium", "score", 4, 1000, "gpt2-medium-score"),
        # encoding padded texts with BERT-large: forward only
        _case("bert-large", "score", 16, 333, "bert-large-encode", padded=True),
        # one short prompt: the smallest call, latency only
        _case("gpt2", "score", 1, 37, "gpt2-prompt"),
        # greedy continuation of two prompts
        _case("gpt2", "generate", 2, 48, "gpt2-generate", new_tokens=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above; tokens per call up to those of the pre-training step's share of depth."""
    kind = rng.choice(["bert-train", "gpt2-train", "llama-train", "moe-train", "score", "score", "generate"])
    if kind == "bert-train":
        model = rng.choice(["bert-base", "bert-large"])
        seq = _log_int(rng, 17, 512)
        batch = max(1, min(64, _log_int(rng, 64, 12000) // seq))
        return _case(model, "train", batch, seq, dropout=rng.choice([0.0, 0.1]), attn_dropout=rng.choice([0.0, 0.1]),
                     padded=rng.random() < 0.5, graph=rng.random() < 0.5, layers=rng.choice([4, 12]))
    if kind == "gpt2-train":
        model = rng.choice(["gpt2", "gpt2-medium", "gpt2-xl"])
        seq = _log_int(rng, 33, 1024)
        batch = max(1, min(64, _log_int(rng, 64, 8192) // seq))
        p = rng.choice([0.0, 0.1])
        return _case(model, "train", batch, seq, dropout=p, attn_dropout=p, layers=rng.choice([3, 6]),
                     accum=rng.choice([1, 2]), recompute=rng.random() < 0.5, graph=rng.random() < 0.3)
    if kind == "llama-train":
        seq = _log_int(rng, 65, 4096)
        batch = max(1, min(16, _log_int(rng, 128, 6144) // seq))
        hidden, heads, ffn = rng.choice([(1024, 16, 2816), (2048, 16, 5504), (4096, 32, 11008)])
        return _case("llama-7b", "train", batch, seq, layers=rng.choice([1, 2]), hidden=hidden, heads=heads, ffn=ffn,
                     kv_heads=heads // rng.choice([1, 2, 4]), graph=rng.random() < 0.5, recompute=rng.random() < 0.3)
    if kind == "moe-train":
        seq = _log_int(rng, 129, 3000)
        return _case("deepseek-v2-lite", "train", 1, seq, layers=2, experts=rng.choice([8, 16]))
    if kind == "generate":
        return _case("gpt2", "generate", rng.choice([1, 2, 3, 4]), _log_int(rng, 9, 200), new_tokens=rng.randint(4, 24))
    model = rng.choice(["bert-base", "bert-large", "gpt2", "gpt2-medium"])
    seq = _log_int(rng, 5, 512 if model.startswith("bert") else 1024)
    batch = max(1, min(32, _log_int(rng, 32, 6000) // seq))
    return _case(model, "score", batch, seq, padded=model.startswith("bert") and rng.random() < 0.5,
                 layers=rng.choice([6, 12]))


def _build(c):
    """The model, with its large parameters on the meta device: the engine allocates and initialises them on the GPU."""
    family = _WIDTHS[c["model"]]["family"]
    with Merak.init_empty_weights():
        if family == "bert":
            return BertForMaskedLM(bert_config(
                c["model"], num_hidden_layers=c["layers"], hidden_dropout_prob=c["dropout"],
                attention_probs_dropout_prob=c["attn_dropout"]))
        if family == "gpt2":
            return GPT2LMHeadModel(gpt2_config(
                c["model"], n_layer=c["layers"], resid_pdrop=c["dropout"], embd_pdrop=c["dropout"],
                attn_pdrop=c["attn_dropout"], tie_word_embeddings=c["mode"] != "generate"))
        if family == "llama":
            return LlamaForCausalLM(llama_config(
                "llama-7b", num_hidden_layers=c["layers"], hidden_size=c["hidden"], num_attention_heads=c["heads"],
                num_key_value_heads=c["kv_heads"], intermediate_size=c["ffn"], max_position_embeddings=4096))
    cfg = deepseek_v2_config("deepseek-v2-lite", num_hidden_layers=c["layers"], n_routed_experts=c["experts"])
    with torch.device("meta"):       # the stacked expert weights are plain parameters: all of it on meta
        return DeepseekV2ForCausalLM(cfg)


def _batches(c, gen, device):
    """``accum`` micro-batches on the device: uniform token ids; masked-LM or next-token labels; padding lengths
    between half a row and a whole one."""
    bert = c["model"].startswith("bert")
    out = []
    for _ in range(c["accum"]):
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=gen, device=device)
        b = {"input_ids": ids}
        if c["padded"]:
            low = (c["seq"] + 1) // 2
            lengths = torch.randint(low, c["seq"] + 1, (c["batch"], 1), generator=gen, device=device)
            b["attention_mask"] = (torch.arange(c["seq"], device=device)[None, :] < lengths).to(torch.int64)
        if c["mode"] == "train":
            labels = ids.clone()
            if bert:
                keep = torch.rand(ids.shape, generator=gen, device=device) < 0.15
                keep[:, 0] = True
                labels = torch.where(keep, labels, torch.full_like(labels, -100))
                b["input_ids"] = torch.where(keep, torch.full_like(ids, 103), ids)
            b["labels"] = labels
        out.append(b)
    return out


def _confident_head(engine, c, gen):
    """Next-token distributions as peaked as a trained model's: every token's output row points at the embedding of
    the token it follows, so that the most likely token stands clear of the others at any rounding."""
    named = dict(engine.module.named_parameters())
    head = next(p for n, p in named.items() if n.endswith("lm_head.weight"))
    wte = next(p for n, p in named.items() if n.endswith("wte.weight"))
    follows = torch.randperm(c["vocab"], generator=gen, device=head.device)
    with torch.no_grad():
        wte.mul_(50.0)
        head.copy_(wte[follows] * 0.03)


def prepare(case, seed):
    if not mpu.is_initialized():
        Merak.init(1, 1, 1)
    device = torch.device("cuda", torch.cuda.current_device())
    c = dict(case)
    torch.manual_seed(seed)
    args = Merak.MerakArguments(
        output_dir="/tmp/merak_b200_cases", bf16=True, per_device_train_batch_size=c["batch"],
        per_device_eval_batch_size=c["batch"], gradient_accumulation_steps=c["accum"], max_steps=10 ** 9,
        learning_rate=1e-4, weight_decay=0.01, max_grad_norm=1.0, lr_scheduler_type="constant", logging_steps=0,
        wall_clock_breakdown=False, report_to="none", activation_checkpointing=c["recompute"],
        split_method="layer_split", cuda_graph=c["graph"], seed=1 + seed % 1000003, out_seq_length=1024,
        input_names=["input_ids", "attention_mask"] if c["padded"] else ["input_ids"])
    trainer = Merak.MerakTrainer(_build(c), args)
    engine = trainer.init_engine()
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    state = {"case": c, "engine": engine, "batches": _batches(c, gen, device)}
    if c["mode"] == "generate":
        _confident_head(engine, c, gen)
        state["pipe"] = text_generation_pipeline(engine, args)
        state["prompts"] = state["batches"][0]["input_ids"].tolist()
    return state


def run(state):
    c, engine = state["case"], state["engine"]
    if c["mode"] == "train":
        loss = engine.train_batch(iter(state["batches"]))
        return {"loss": loss, "weights": engine.flat.model, "master": engine.optimizer.master}
    if c["mode"] == "score":
        return engine.eval_batch(iter(state["batches"]), compute_loss=False, num_micro_batches=1)
    ids = state["pipe"].generate(state["prompts"], max_new_tokens=c["new_tokens"], greedy=True)
    tokens = torch.tensor(ids, device=engine.device)
    logits = engine.eval_batch(iter([{"input_ids": tokens}]), compute_loss=False, num_micro_batches=1)
    return {"tokens": tokens, "logits": logits}


def _counts(c):
    """(weights, weights a token multiplies with, attention operations per token pair and layer)."""
    h, L = c["hidden"], c["layers"]
    family = _WIDTHS[c["model"]]["family"]
    emb = c["vocab"] * h
    if family == "moe":
        attn = h * c["heads"] * _QK_DIM + h * (_KV_LORA + _ROPE_DIM) + _KV_LORA * c["heads"] * (128 + _V_DIM) \
            + c["heads"] * _V_DIM * h
        dense, expert, shared = 3 * h * c["ffn"], 3 * h * _EXPERT_FFN, 3 * h * _EXPERT_FFN * _SHARED
        total = 2 * emb + L * attn + dense + (L - 1) * (c["experts"] * (expert + h) + shared)
        used = emb + L * attn + dense + (L - 1) * (_TOP_K * expert + c["experts"] * h + shared)
        return total, used, 2 * c["heads"] * (_QK_DIM + _V_DIM)
    d = h // c["heads"]
    if family == "llama":
        per = h * (c["heads"] + 2 * c["kv_heads"]) * d + h * h + 3 * h * c["ffn"]
        return 2 * emb + L * per, emb + L * per, 4 * h
    per = 4 * h * h + 2 * h * c["ffn"]
    extra = h * h if family == "bert" else 0
    tied = 1 if c["mode"] != "generate" else 2
    return tied * emb + L * per + extra, emb + L * per + extra, 4 * h


def work(case):
    c = dict(case)
    total, used, pair = _counts(c)
    causal = not c["model"].startswith("bert")
    tokens = c["batch"] * c["seq"] * c["accum"]
    pairs = tokens * c["seq"] // (2 if causal else 1)
    forward = 2.0 * used * tokens + float(pair) * pairs * c["layers"]
    if c["mode"] == "train":
        # weights, master weights and two moments read and written once, the token ids and labels read
        return {"bytes": 28.0 * total + 16.0 * tokens, "flops": 3.0 * forward}
    if c["mode"] == "score":
        return {"bytes": 2.0 * total + 8.0 * tokens + 2.0 * tokens * c["vocab"], "flops": forward}
    # generation: the prompt once, then every new token reads the weights it multiplies with; the final logits
    new, out = c["new_tokens"], c["batch"] * (c["seq"] + c["new_tokens"])
    return {"bytes": 2.0 * used * (1 + new) + 2.0 * out * c["vocab"],
            "flops": forward + 2.0 * used * (c["batch"] * new + out)}


def tolerance(case):
    """bf16 activations, fp32 sums.  Measured against the same call in fp32 throughout (dropout off): logits are off by
    0.009 to 0.014 of their norm (largest single value 0.08 of the root mean square); updated weights by 0.0016 to
    0.0018 (largest 0.011), mostly their own rounding to bf16, and those of the mixture of experts, whose weights are
    smaller beside the same step, by 0.0020 (largest 0.029).  One step moves the weights by 0.004 of their norm, so a
    wrong direction shows."""
    if case["mode"] != "train":
        return {"rel": 3e-2, "max": 0.3, "differ": 0.005}
    if case["experts"]:
        return {"rel": 5e-3, "max": 0.1}
    return {"rel": 3.5e-3, "max": 0.04}
