"""The workloads this framework is measured on, through the entry points its users call.

Five kinds of work, on the model configurations shipped under ``configs/``:

* ``train``: one optimizer step (``TrainEngine.train_step``): pinned host batches in, forward,
  backward, gradient norm, clip and update.
* ``eval``: the loss of held-out text and the carried EFLA states (``EflaLM.forward`` with
  targets, no gradients), from one short document to one long context.
* ``prefill``: the logits and states of a prompt (``EflaLM.forward`` without targets).
* ``decode``: one token for every running sequence (``EflaLM.decode_step``).
* ``generate``: a prompt and the tokens sampled after it (``Generator.generate_ids``).

``listed()`` names one point of each range that is in everyday use and its ends; ``draw()``
samples the same ranges.  Weights are random (``_condition``), tokens are the Zipf(1.1) stream
of the benchmark; both come from the seed alone.
"""
from __future__ import annotations

import math

import torch

from ceo_b200.data.synthetic import SyntheticTokens
from ceo_b200.models.model import EflaLM, model_flops_per_token
from ceo_b200.runtime.engine import TrainEngine
from ceo_b200.runtime.evaluator import Generator
from ceo_b200.utils.config import Config

CONFIG = {"smoke": "configs/smoke.yaml", "340m": "configs/efla_340m.yaml",
          "1p3b": "configs/efla_1p3b.yaml", "7b": "configs/efla_7b.yaml"}
CHUNK = 64  # the GPU path takes sequence lengths that are multiples of the EFLA chunk


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smoke run a user starts with: GELU MLP, PRISM branch, q = k, one scalar beta,
        # Lion + Muon; two layers, so launches and host work are all there is
        _train("train_smoke", "smoke", 1, 128, 1, "lion_muon", "none"),
        # the 340M configuration's own micro-batch
        _train("train_340m", "340m", 8, 2048, 1, "adamw", "none"),
        # a fine-tuning step on short ragged sequences, two micro-batches, with the optimizer
        # mix the reference trains with
        _train("train_340m_muon", "340m", 2, 1088, 2, "lion_muon", "none"),
        # FP8 training with 8-bit gradients
        _train("train_340m_fp8", "340m", 4, 2048, 1, "adamw", "all"),
        # the headline configuration's micro-batch (8 x 4096 tokens)
        _train("train_1p3b", "1p3b", 8, 4096, 1, "adamw", "none"),
        # perplexity of one sequence at the training length (the evaluator's default batch)
        _forward("eval_1p3b", "eval", "1p3b", 1, 4096),
        # long-context evaluation: one sequence, so few (batch, head) chains
        _forward("eval_340m_long", "eval", "340m", 1, 65536),
        # a prompt of odd length
        _forward("prefill_1p3b", "prefill", "1p3b", 1, 576),
        # interactive decoding, a small server batch, the largest model on one GPU
        _forward("decode_1p3b", "decode", "1p3b", 1, 1),
        _forward("decode_340m_b40", "decode", "340m", 40, 1),
        _forward("decode_7b_b7", "decode", "7b", 7, 1),
        # the generate command with its default sampling
        {"name": "generate_1p3b", "kind": "generate", "model": "1p3b", "prompt": 90, "new": 30},
    ]


def draw(rng):
    kind = rng.choice(("train", "train", "eval", "prefill", "decode", "decode", "generate"))
    if kind == "train":
        model = rng.choice(("smoke", "340m", "340m", "1p3b"))
        if model == "smoke":
            seq = CHUNK * rng.randint(1, 16)
            return _train(None, model, rng.randint(1, 8), seq, rng.randint(1, 2), "lion_muon",
                          "none")
        most = 32768
        tokens = _log_int(rng, 256, most)
        seq = CHUNK * max(1, min(64, _log_int(rng, 128, min(tokens, 4096)) // CHUNK))
        batch = max(1, min(16, tokens // seq))
        micro = 2 if rng.random() < 0.3 and 2 * batch * seq <= most else 1
        opt = "adamw" if model == "1p3b" else rng.choice(("adamw", "adamw", "lion", "lion_muon"))
        fp8 = rng.choice(("none", "none", "none", "forward", "all"))
        return _train(None, model, batch, seq, micro, opt, fp8)
    if kind in ("eval", "prefill"):
        model = rng.choice(("340m", "1p3b", "7b") if kind == "eval" else ("340m", "1p3b"))
        most = {"340m": 65536, "1p3b": 32768, "7b": 8192}[model] if kind == "eval" else 8192
        tokens = _log_int(rng, CHUNK, most)
        batch = _log_int(rng, 1, 8)
        seq = CHUNK * max(1, tokens // batch // CHUNK)
        return _forward(None, kind, model, batch, seq)
    if kind == "decode":
        return _forward(None, kind, rng.choice(("340m", "1p3b", "7b")), _log_int(rng, 1, 128), 1)
    return {"kind": "generate", "model": rng.choice(("340m", "1p3b")),
            "prompt": _log_int(rng, 1, 90), "new": rng.randint(2, 30)}


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def _train(name, model, batch, seq, micro, optimizer, fp8):
    c = {"kind": "train", "model": model, "batch": batch, "seq": seq, "micro": micro,
         "optimizer": optimizer, "fp8": fp8}
    return c if name is None else {"name": name, **c}


def _forward(name, kind, model, batch, seq):
    c = {"kind": kind, "model": model, "batch": batch, "seq": seq}
    return c if name is None else {"name": name, **c}


# ------------------------------------------------------------- what a program has in hand
def _config(case):
    cfg = Config.parse_from_file(CONFIG[case["model"]])
    r = cfg.runtime
    r.world_size = r.tensor_parallel_size = r.pipeline_parallel_size = 1
    return cfg


@torch.no_grad()
def _condition(model, gen):
    """Weights that behave as those of a run in progress: embeddings of unit variance and block
    outputs that add up to the same order whatever the depth and width, instead of the fresh
    N(0, 0.02) model, whose residual stream is all block output and turns bf16 rounding into
    several per cent at the logits."""
    model.embed_tokens.normal_(0.0, 1.0, generator=gen)
    scale = (512.0 / (len(model.blocks) * model.cfg.hidden_dim)) ** 0.5
    for b in model.blocks:
        b.efla.w_o.mul_(scale)
        b.mlp.w_down.mul_(scale)


def prepare(case, seed):
    cfg = _config(case)
    dev = torch.device("cuda", torch.cuda.current_device())
    data = SyntheticTokens(cfg.model.vocab_size, "zipf", 1.1, seed)
    kind = case["kind"]
    if kind == "train":
        t = cfg.training
        t.optimizer = case["optimizer"]
        t.fp8_training, t.fp8_gradients = case["fp8"] != "none", case["fp8"] == "all"
        engine = TrainEngine(cfg, dev, seed=seed)
        _condition(engine.model, torch.Generator(device=dev).manual_seed(seed + 1))
        engine.flat.refresh_master()
        batches = [data.batch(case["batch"], case["seq"], pin=True) for _ in range(case["micro"])]
        # an orthogonalised update has entries far below one: Muon runs at a larger rate
        lr = 2e-3 if t.optimizer == "lion_muon" else t.learning_rate
        return {"kind": kind, "engine": engine, "batches": batches, "lr": lr}
    model = EflaLM(cfg.model, dev, seed=seed).eval()
    gen = torch.Generator(device=dev).manual_seed(seed + 1)
    _condition(model, gen)
    if kind == "generate":
        # a trained model's next-token distribution is peaked, a random one's is flat and its
        # samples say nothing: a head that maps each token to one successor gives a distribution
        # whose top token holds the nucleus, so that the ids can be compared
        with torch.no_grad():
            nxt = torch.randperm(cfg.model.vocab_size, generator=gen, device=dev)
            model.head_weight().copy_(model.embed_tokens[nxt])
        prompt = [int(v) for v in data.sample(case["prompt"])]
        return {"kind": kind, "generator": Generator(model, seed=seed), "prompt": prompt,
                "new": case["new"]}
    state = {"kind": kind, "model": model}
    if kind == "decode":
        tokens = torch.from_numpy(data.sample(case["batch"])).to(dev)
        states = model.new_states(case["batch"])
        for s in states:  # as after a prompt: sums of unit keys times values
            s.normal_(0.0, 0.5, generator=gen)
        return {**state, "tokens": tokens, "states": states}
    tok, tgt = data.batch(case["batch"], case["seq"])
    return {**state, "tokens": tok.to(dev), "targets": tgt.to(dev)}


# ------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "train":
        # the updated weights stand for every gradient: the first moments are heavy-tailed (rows
        # of frequent tokens), which makes single entries incomparable between summation orders
        engine = state["engine"]
        loss, norm = engine.train_step(state["batches"], state["lr"])
        return {"loss": loss, "norm": norm, "params": engine.flat.params,
                "master": engine.flat.master}
    if kind == "generate":
        ids = state["generator"].generate_ids(state["prompt"], state["new"], temperature=1.0,
                                              top_p=0.9)
        return torch.tensor(ids)
    model = state["model"]
    with torch.no_grad():
        if kind == "decode":
            return model.decode_step(state["tokens"], state["states"]), list(state["states"])
        return model(state["tokens"], state["targets"] if kind == "eval" else None,
                     return_states=True)


# ------------------------------------------------------------------ what it cannot do without
def _parameters(m):
    """(parameters in all, those of the embedding table's lookup)."""
    P = 3 if m.efla.use_query else 2
    hd = m.num_heads * m.head_dim
    block = (P * hd + (m.num_heads if m.efla.per_token_beta else 0)) * m.hidden_dim
    block += hd * m.hidden_dim + 2 * m.hidden_dim
    block += (3 if m.activation == "swiglu" else 2) * m.hidden_dim * m.intermediate_dim
    if m.prism.enabled:
        block += 3 * m.prism.num_iterations * m.head_dim * m.hidden_dim
        block += m.hidden_dim * m.prism.shortconv_window
    table = m.vocab_size * m.hidden_dim
    n = m.num_layers * block + m.hidden_dim + table
    return (n, 0) if m.tie_embeddings else (n + table, table)


def work(case):
    cfg = _config(case)
    m = cfg.model
    n, table = _parameters(m)
    per_token = model_flops_per_token(m)  # forward + backward
    kind = case["kind"]
    state_bytes = 4 * m.num_layers * m.num_heads * m.head_dim ** 2
    if kind == "train":
        tokens = case["batch"] * case["seq"] * case["micro"]
        flops = per_token * tokens
        if case["optimizer"] == "lion_muon":
            # Newton-Schulz: a symmetric product and a full one, each iteration
            hd, D, F = m.num_heads * m.head_dim, m.hidden_dim, m.intermediate_dim
            up = (2 if m.activation == "swiglu" else 1) * F
            P = 3 if m.efla.use_query else 2
            mats = [(P * hd, D), (D, hd), (up, D), (D, F)] * m.num_layers
            mats += [(m.vocab_size, D)] * (1 if m.tie_embeddings else 2)
            flops += sum(3.0 * min(a, b) * a * b for a, b in mats) * cfg.training.muon_iterations
        # bf16 weight, fp32 master and moments: read once, written once
        moments = 2 if case["optimizer"] == "adamw" else 1
        return {"bytes": n * 2.0 * (2 + 4 + 4 * moments) + 16 * tokens, "flops": flops}
    weights = 2.0 * (n - table)
    if kind == "generate":
        # the prompt in one pass over the weights, then one pass for each new token but the last
        steps = case["new"]
        return {"bytes": steps * weights + 2.0 * steps * state_bytes,
                "flops": per_token / 3 * (case["prompt"] + case["new"] - 1)}
    tokens = case["batch"] * case["seq"]
    rows = 2.0 * m.hidden_dim * min(tokens, m.vocab_size)
    states = case["batch"] * state_bytes * (2.0 if kind == "decode" else 1.0)
    logits = 0.0 if kind == "eval" else 4.0 * tokens * m.vocab_size
    return {"bytes": weights + rows + states + logits + 8.0 * tokens,
            "flops": per_token / 3 * tokens}


def tolerance(case):
    """About four times the largest relative error seen between this framework's kernels and the
    same model on library GEMMs, with one rounding in a thousand of the normed activations moved
    by a bit (forward paths are held to at most 0.03)."""
    if case["kind"] == "generate":
        return "exact"
    if case["kind"] == "train":
        rel = 1e-4 if case["optimizer"] == "lion_muon" else 4e-4
        return {"rel": rel, "max": 0.05} if case["fp8"] == "none" else {"rel": 8 * rel, "max": 0.05}
    return {"rel": 0.03, "max": 0.5}
