"""What a user of this framework has it do, as timed cases: training steps, validation passes, move
predictions and tree search, each through the public classes a program calls.

Every case names a kind of work and the sizes of one pass; ``prepare`` builds what the program holds
before the pass (the model with random weights, the trainer or evaluator, the inputs), ``run`` is one
pass.  Weights are random-init as in the benchmarks, tokens are uniform random moves with ratings,
think times and outcomes packed like training data.
"""
from __future__ import annotations

import logging
import math
import os
import random
import tempfile

import numpy as np
import torch

os.environ.setdefault("ALLIE_NO_WANDB", "1")

N_MOVES = 1968          # ids below this are chess moves
VOCAB = 2048            # the tokenizer's vocabulary padded to a multiple of 128
ELO_LO, ELO_HI = 800, 2600

MEDIUM = dict(n_layer=24, n_embd=1024, n_head=16, n_inner=4096)


def listed() -> list[dict]:
    return [
        # One optimizer step of the tiny model (the CPU-sized shape of the smoke run and the tests):
        # a few dozen small kernels, so launches and latencies are what a user waits for.
        _train("train_tiny", 8, 256, n_layer=4, n_embd=256, n_head=4, n_inner=1024),
        # The small ablation with a batch and context that fill no tile evenly (37 windows of 328
        # words): sequence lengths are a tokenizer option.
        _train("train_small_ragged", 37, 328, n_layer=12, n_embd=768, n_head=12, n_inner=3072),
        # The headline: one micro-batch of 64 windows and an optimizer step of the medium model.
        _train("train_medium", 64, 512, **MEDIUM),
        # The large ablation (GPT-2-large shape) at half the medium micro-batch.
        _train("train_large", 32, 512, n_layer=36, n_embd=1280, n_head=20, n_inner=5120),
        # The mixture-of-experts configuration with its depth and expert count reduced to one GPU:
        # heads of 128, every third block routes top-2 over 16 experts of FFN 4096.
        _train("train_moe", 32, 512, n_layer=6, n_embd=2048, n_head=16, n_inner=4096, experts=16),
        # A validation batch of the medium model: forward pass with labels, logits kept.
        dict(name="validate_medium", kind="validate", batch=32, seq=512, **MEDIUM),
        # A move server answering one request: one game, one position, batch 1.
        dict(name="policy_one_game", kind="policy", games=1, longest=90, **MEDIUM),
        # A move server answering everyone in its backlog: 64 games of all lengths share a pass.
        dict(name="policy_64_games", kind="policy", games=64, longest=300, **MEDIUM),
        # The start of a batched search: the prompts of 256 games go into the key/value cache.
        dict(name="search_prefill_256", kind="prefill", trees=256, longest=300, **MEDIUM),
        # Leaf evaluations of a search, the inner loop of move selection: 256 trees (the
        # benchmark), and the 4 trees of a small server at a quiet hour.
        dict(name="search_leaves_256", kind="leaves", trees=256, longest=300, steps=8, **MEDIUM),
        dict(name="search_leaves_4", kind="leaves", trees=4, longest=120, steps=8, **MEDIUM),
    ]


def _train(name: str, batch: int, seq: int, *, n_layer: int, n_embd: int, n_head: int, n_inner: int,
           experts: int = 0, dropout: float = 0.1, norm: str = "layernorm") -> dict:
    case = dict(kind="train", batch=batch, seq=seq, n_layer=n_layer, n_embd=n_embd, n_head=n_head, n_inner=n_inner,
                experts=experts, dropout=dropout, norm=norm)
    return dict(case, name=name) if name else case


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    """A case of the same kinds: model shapes between the tiny and the large one, batches and lengths
    over their whole range, odd ones included."""
    kind = rng.choice(["train", "train", "train_moe", "validate", "policy", "prefill", "leaves"])
    head = 64
    heads = 2 * _log(rng, 2, 10)        # the residual width is a multiple of 128
    layers = _log(rng, 2, 24)
    if kind == "train_moe":
        heads, head, layers = rng.choice([4, 8, 12, 16]), 128, rng.choice([3, 4, 6])
    shape = dict(n_layer=layers, n_embd=heads * head, n_head=heads)
    shape["n_inner"] = shape["n_embd"] * (2 if kind == "train_moe" else 4)
    if kind in ("train", "train_moe"):
        dropout = rng.choice([0.1, 0.1, 0.0]) if kind == "train" else 0.1
        seq = _log(rng, 48, 1000)
        if dropout:
            seq = -(-seq // 8) * 8      # attention dropout draws its mask in groups of eight keys
        batch = max(1, min(_log(rng, 1, 96), 32768 // seq))
        if kind == "train_moe":
            return _train("", max(batch, -(-512 // seq)), seq, experts=rng.choice([4, 8, 16]), **shape)
        return _train("", batch, seq, dropout=dropout,
                      norm=rng.choice(["layernorm", "layernorm", "rmsnorm"]), **shape)
    if kind == "validate":
        seq = _log(rng, 48, 1000)
        return dict(kind=kind, batch=max(1, min(_log(rng, 1, 64), 32768 // seq)), seq=seq, **shape)
    if kind == "policy":
        return dict(kind=kind, games=_log(rng, 1, 128), longest=_log(rng, 8, 400), **shape)
    if kind == "prefill":
        return dict(kind=kind, trees=_log(rng, 1, 256), longest=_log(rng, 8, 300), **shape)
    return dict(kind=kind, trees=_log(rng, 1, 256), longest=_log(rng, 8, 300), steps=rng.choice([4, 8]), **shape)


# ------------------------------------------------------------------------------------- inputs ---
def _words(rng: np.random.Generator, batch: int, seq: int) -> np.ndarray:
    """Training words: move id, think time (+1) in the upper half, outcome in bits 14-15; a game
    starts with two ratings and a time control, ends with an end-of-game token and is followed by
    the next, and the windows cut the stream anywhere."""
    shape = (batch, seq)
    ids = rng.integers(0, N_MOVES, size=shape, dtype=np.uint32)
    secs = np.minimum(rng.lognormal(1.0, 1.0, size=shape), 600.0).astype(np.uint32)
    words = ids | ((secs + 1) << 16)
    start = rng.integers(0, seq, size=batch)
    for b in range(batch):
        for k, word in ((0, VOCAB + rng.integers(ELO_LO, ELO_HI)), (1, VOCAB + rng.integers(ELO_LO, ELO_HI)),
                        (2, rng.integers(N_MOVES, N_MOVES + 24) | (4 << 16))):
            if start[b] + k < seq:
                words[b, start[b] + k] = word
    outcome = rng.integers(0, 3, size=(batch, 2)).astype(np.uint32) << 14
    words |= np.where(np.arange(seq)[None, :] < start[:, None], outcome[:, :1], outcome[:, 1:])
    return words


def _games(rng: np.random.Generator, n: int, longest: int):
    """Games whose prompts are 4 to ``longest`` tokens (one of them exactly that long)."""
    from allie_b200.data import Game
    from allie_b200.moves import CHESS_MOVES

    games = []
    for i in range(n):
        tokens = longest if i == n // 2 else int(rng.integers(4, longest + 1))
        plies = max(0, tokens - 3)
        moves = [CHESS_MOVES[j] for j in rng.integers(0, N_MOVES, size=plies)]
        games.append(Game("180+0", int(rng.integers(ELO_LO, ELO_HI)), int(rng.integers(ELO_LO, ELO_HI)), None, False,
                          moves, [int(s) for s in rng.integers(0, 30, size=plies)]))
    return games


def _leaf_requests(rng: np.random.Generator, prefix: list[int], steps: int, anc_max: int, legal_max: int) -> list[dict]:
    """One request block per step: every tree grows by one node below a random earlier one (or the
    root); about one tree in fifteen has reached a finished game and asks for nothing."""
    n = len(prefix)
    chains: list[list[list[int]]] = [[[]] for _ in range(n)]     # slots on the path to each node
    out = []
    for s in range(steps):
        req = dict(need_eval=np.zeros(n, np.int32), tok=np.zeros(n, np.int32), pos=np.zeros(n, np.int32),
                   slot=np.zeros(n, np.int32), n_anc=np.zeros(n, np.int32), n_legal=np.zeros(n, np.int32),
                   anc=np.zeros((n, anc_max), np.int32), legal=np.zeros((n, legal_max), np.int32))
        for t in range(n):
            if n > 1 and rng.random() < 1 / 15:
                continue
            slot = prefix[t] + len(chains[t]) - 1
            chain = chains[t][int(rng.integers(0, len(chains[t])))] + [slot]
            chains[t].append(chain)
            nl = int(rng.integers(20, 45))
            req["need_eval"][t], req["tok"][t] = 1, rng.integers(0, N_MOVES)
            req["slot"][t], req["pos"][t] = slot, prefix[t] + len(chain) - 1
            req["n_anc"][t], req["anc"][t, :len(chain)] = len(chain), chain
            req["n_legal"][t], req["legal"][t, :nl] = nl, rng.choice(N_MOVES, size=nl, replace=False)
        out.append(req)
    return out


# ------------------------------------------------------------------------------------ prepare ---
def _model(case: dict, seed: int, tok):
    """A random-init model, built on the GPU (the weights of a user's checkpoint are there, too)."""
    from allie_b200.models import initialize_model

    p = case.get("dropout", 0.1)
    extra = {}
    if case.get("experts"):
        # capacity for any load: rows beyond an expert's capacity would be dropped in arrival order
        extra = dict(num_experts=case["experts"], moe_top_k=2, moe_ffn=case["n_inner"], moe_layer_freq=3,
                     aux_loss_coef=0.01, capacity_factor=case["experts"] / 2)
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = initialize_model(tok, "gpt2-medium", use_control_token=True, use_regression_head=True,
                                 n_layer=case["n_layer"], n_embd=case["n_embd"], n_head=case["n_head"],
                                 n_inner=case["n_inner"], n_positions=1024, norm_type=case.get("norm", "layernorm"),
                                 embd_pdrop=p, resid_pdrop=p, attn_pdrop=p, **extra)
    if case.get("experts"):
        _specialise_routers(model, case)
    return model


@torch.no_grad()
def _specialise_routers(model, case: dict) -> None:
    """Routers as training leaves them: moves fall into groups that share a direction of the
    embedding space, and each group has a first and a second expert.  (A fresh router decides between
    experts that are nearly tied, so a token's route hangs on the last bits of its activation.)"""
    E, d, groups = case["experts"], case["n_embd"], 24
    params = dict(model.named_parameters())
    wte = next(p for n, p in params.items() if n.endswith("wte.weight"))
    dirs = torch.randn(groups, d, device=wte.device) * 0.04
    wte += dirs[torch.arange(wte.shape[0], device=wte.device) % groups]
    next(p for n, p in params.items() if "control_embeds" in n).add_(dirs[0])
    for layer, w in enumerate(p for n, p in params.items() if "router" in n):
        want = torch.zeros(E, groups, device=wte.device)
        g = torch.arange(groups, device=wte.device)
        want[(5 * g + layer) % E, g] = 1.0
        want[(5 * g + layer + 1 + g % (E - 1)) % E, g] = 0.9
        w.copy_(0.25 * want @ (dirs / dirs.norm(dim=1, keepdim=True)))


def prepare(case: dict, seed: int) -> dict:
    from allie_b200.data import UCITokenizer
    from allie_b200.models.engine import B200Engine

    logging.disable(logging.INFO)
    rng = np.random.default_rng(seed)
    tok = UCITokenizer(max_length=case.get("seq", 512), vocab_size_multiple_of=128)
    assert len(tok) == VOCAB
    model = _model(case, seed, tok)
    state = dict(kind=case["kind"])
    if case["kind"] == "train":
        from allie_b200.config import Config
        from allie_b200.train.trainer import Trainer

        trainer = Trainer(Config({}), output_dir=tempfile.mkdtemp(prefix="allie_perf_"), batch_size=case["batch"],
                          gradient_accumulation_steps=1, lr=6e-4, min_lr=1e-5, weight_decay=1e-2, grad_clip=1.0,
                          warmup_iters=2000, decay_iters=2_000_000, max_iters=2_000_000, eval_interval=0,
                          log_interval=-1, save_interval=0, use_wandb=False)
        trainer.setup_model(model)
        trainer.iter_num = 10           # the learning rate of the first warm-up iterations
        words = torch.from_numpy(_words(rng, case["batch"], case["seq"]).view(np.int32))
        state.update(trainer=trainer, windows=[words.pin_memory()])   # as the trainer's sampler hands them out
    elif case["kind"] == "validate":
        words = _words(rng, case["batch"], case["seq"])
        state.update(engine=B200Engine(model, "cuda"), batch=tok.pad_and_collate(list(words)))
    elif case["kind"] == "policy":
        from allie_b200.search.runner import EngineRunner, attach_engine

        state.update(runner=EngineRunner(model, tok), games=_games(rng, case["games"], case["longest"]))
        attach_engine(model, None)      # this program looks the engine up nowhere else
    else:
        from allie_b200.search.batched import KVStepEvaluator

        games = _games(rng, case["trees"], case["longest"])
        steps = case.get("steps", 0)
        ev = KVStepEvaluator(B200Engine(model, "cuda"), tok, case["trees"], anc_max=128, legal_max=224,
                             max_prefix=320, max_nodes=408)
        state.update(evaluator=ev, games=games)
        if case["kind"] == "leaves":
            ev.prefill(games)
            prefix = [len(tok.tokenize(g)) for g in games]
            state["requests"] = _leaf_requests(rng, prefix, steps, 128, 224)
            state["asked"] = [(r["need_eval"] != 0, np.arange(224)[None, :] < r["n_legal"][:, None])
                              for r in state["requests"]]
    return state


def run(state: dict):
    kind = state["kind"]
    if kind == "train":
        trainer = state["trainer"]
        loss = trainer.train_step(state["windows"])
        arena = trainer.engine.arena
        return {"loss": loss, "weights": arena.master, "exp_avg": arena.exp_avg, "exp_avg_sq": arena.exp_avg_sq}
    if kind == "validate":
        out = state["engine"].evaluate_batch(state["batch"])
        keys = ("loss", "lm_loss", "value_loss", "time_loss", "logits", "value_logits", "time_logits")
        return {k: out[k] for k in keys}
    if kind == "policy":
        ev = state["runner"].evaluate(state["games"])
        return {"logits": ev.logits, "value": ev.value, "time": ev.time}
    if kind == "prefill":
        logits, value, time = state["evaluator"].prefill(state["games"])
        return {"logits": logits, "value": value, "time": time}
    priors, values = [], []
    for req, (active, legal) in zip(state["requests"], state["asked"]):
        p, v = state["evaluator"].step(req)
        priors.append(np.where(legal, p, np.float32(0)))       # what the search reads: the legal moves' priors
        values.append(np.where(active, v, np.float32(0)))      # and the values of the leaves it asked for
    return {"priors": np.stack(priors), "values": np.stack(values)}


# ------------------------------------------------------------------------------ work, tolerance ---
def _mean_tokens(case: dict) -> float:
    return 0.5 * (4 + case["longest"])


def work(case: dict) -> dict:
    d, f, layers = case["n_embd"], case["n_inner"], case["n_layer"]
    moe_layers = layers // 3 if case.get("experts") else 0
    dense = layers * 4 * d * d + (layers - moe_layers) * 2 * d * f          # matrix weights every token meets
    expert = moe_layers * 2 * d * f                                         # weights of one expert per MoE layer
    n_params = dense + expert * case.get("experts", 0) + VOCAB * d + 1024 * d
    active = dense + 2 * expert + VOCAB * d                                  # multiplied with each token (top-2)
    kind = case["kind"]
    if kind == "train":
        tokens = case["batch"] * case["seq"]
        flops = tokens * (6 * active + 6 * layers * d * case["seq"])         # causal: half of 12 L d T
        # activations: per token and layer the residual stream in and out (fp32), the packed
        # projections, the MLP activation and its derivative, written forward and read backward;
        # weights, gradient and moments once in, weights and moments once out (fp32)
        bytes_ = 7 * 4 * n_params + 2 * tokens * layers * (2 * 4 * d + 2 * 6 * d + 2 * 2 * f)
        return {"bytes": bytes_, "flops": flops}
    if kind == "validate":
        tokens = case["batch"] * case["seq"]
        return {"bytes": 2 * n_params + 2 * tokens * VOCAB + 8 * tokens * d,
                "flops": tokens * (2 * active + 2 * layers * d * case["seq"])}
    if kind in ("policy", "prefill"):
        n = case["games"] if kind == "policy" else case["trees"]
        tokens = n * _mean_tokens(case)
        square = n * (case["longest"] ** 2) / 3                              # mean of the squared lengths
        return {"bytes": 2 * n_params + n * VOCAB * 4 + (4 * layers * d * tokens if kind == "prefill" else 0),
                "flops": tokens * 2 * dense + n * 2 * VOCAB * d + 2 * layers * d * square}
    tokens = case["trees"] * case["steps"]
    keys = tokens * (_mean_tokens(case) + 3)
    return {"bytes": case["steps"] * 2 * active + keys * layers * 4 * d, "flops": tokens * 2 * active + 4 * keys * layers * d}


def tolerance(case: dict) -> dict:
    """bf16 operands with fp32 sums, measured against the plain PyTorch model in 64 bits: logits,
    values and priors are off by 0.4 to 1.0 % (largest element 0.04 of the rms or of itself), the
    gradients of 12 to 36 blocks by 0.7 to 1.6 % and their squares by 1 to 2.5 % (single elements by
    more than the rms of all)."""
    return {"rel": 0.03, "max": 0.99} if case["kind"] == "train" else {"rel": 0.03, "max": 0.15}
