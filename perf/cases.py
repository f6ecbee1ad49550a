"""The work that users of this framework give it, as timed cases.

Every case goes through a public entry point: ``Trainer.train_step`` (forward, losses,
backward, clip + AdamW on a pinned host batch), a deterministic forward with the loss
(validation), ``inference.prefill`` and ``inference.DecodeSession.step``.  Models are the named
presets and example configurations of this repository, in the
state of a run under way (see ``_model``).
"""
import math

import torch

from dawn_srw_b200.config import preset
from dawn_srw_b200.models.inference import DecodeSession, prefill
from dawn_srw_b200.models.registry import build_model_from_config
from dawn_srw_b200.train.optimizer import DawnAdamW
from dawn_srw_b200.train.trainer import Trainer

VOCAB, MAX_SEQ = 30522, 512

# preset and what the example configurations change of it
MODELS = {
    "40M": ("40M", dict(model_version="spatial-r1-v4.0.1")),          # dawn_v4_0_1_40M.yaml
    "40M-d512": ("40M", dict(model_version="spatial-r1-v4.0.1", d_model=512, n_heads=8,
                             n_qk=976, n_v=1606, n_know=15563)),      # dawn_v4_0_1_40M_d512.yaml
    "400M": ("400M", {}),                                             # dawn_v4_0_1_400M.yaml
    "1B": ("1B", {}),                                                 # dawn_v3_9_4_1B.yaml
    "dense-40M": ("40M", dict(model_version="baseline", d_ff=1536)),  # baseline_40M.yaml
    "dense-400M": ("400M", dict(model_version="baseline", d_ff=5120)),   # baseline_400M.yaml
}


def listed():
    return [
        # one user's reply, token by token, on the smallest and on the flagship model: latency
        dict(name="decode_40M_1", op="decode", model="40M", batch=1, seq=290),
        dict(name="decode_400M_1", op="decode", model="400M", batch=1, seq=333),
        # a handful of users, and a full serving batch, on the largest model
        dict(name="decode_1B_6", op="decode", model="1B", batch=6, seq=129),
        dict(name="decode_1B_32", op="decode", model="1B", batch=32, seq=440),
        # prompts: a few short ragged ones, one full-length one, several on the largest model
        dict(name="prefill_40M_3x109", op="prefill", model="40M", batch=3, seq=109),
        dict(name="prefill_400M_1x512", op="prefill", model="400M", batch=1, seq=512),
        dict(name="prefill_1B_4x301", op="prefill", model="1B", batch=4, seq=301),
        # a validation batch of the 40M configuration
        dict(name="eval_40M_16x512", op="eval", model="40M", batch=16, seq=512),
        # training: a small run on short sequences, one GPU's share of the 40M configuration and of
        # its dense counterpart (128 sequences over 8 GPUs), one GPU's share of the flagship
        dict(name="train_40M_4x128", op="train", model="40M", batch=4, seq=128),
        dict(name="train_40M_16x512", op="train", model="40M", batch=16, seq=512),
        dict(name="train_dense_40M_16x512", op="train", model="dense-40M", batch=16, seq=512),
        dict(name="train_400M_32x512", op="train", model="400M", batch=32, seq=512),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["decode", "decode", "prefill", "prefill", "eval", "train", "train"])
    seq = _log_int(rng, 16, MAX_SEQ)             # ragged, many short sequences or few long ones
    if op == "decode":
        model = rng.choice(["40M", "400M", "1B", "1B"])
        batch = _log_int(rng, 1, 32 if model == "1B" else 4)
        return dict(op=op, model=model, batch=batch, seq=_log_int(rng, 272, MAX_SEQ - 1))
    if op == "prefill":
        model = rng.choice(["40M", "400M", "1B", "dense-400M"])
        tokens = _log_int(rng, 272, 8192 if model != "1B" else 2048)
    elif op == "eval":
        model = rng.choice(["40M", "400M"])
        tokens = _log_int(rng, 256, 16384)
    else:
        model = rng.choice(["40M", "40M-d512", "400M", "dense-40M"])
        tokens = _log_int(rng, 256, 12288)
    seq = min(seq, tokens)
    return dict(op=op, model=model, batch=-(-tokens // seq), seq=seq)


# ---------------------------------------------------------------------------
def _config(case, seed):
    base, changes = MODELS[case["model"]]
    cfg = preset(base, **changes)
    cfg.seed = seed
    cfg.model.vocab_size, cfg.model.max_seq_len = VOCAB, MAX_SEQ
    cfg.model.gradient_checkpointing = False
    t = cfg.training
    t.batch_size, t.log_interval = case["batch"], 0
    t.lr = 3e-4 if base == "400M" else 6.5e-4
    if cfg.model.is_spatial:
        t.load_balance_weight, t.diversity_weight = 0.1, 0.1
    return cfg


def _model(cfg, seed):
    """The configured model with weights drawn on the GPU, at the scales of a run under way:
    logits with a standard deviation of about two, thresholds where about 28 % of a token's units
    are active (what training settles at with unit-norm pools)."""
    with torch.device("meta"):
        model = build_model_from_config(cfg)
    model = model.to_empty(device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for name, p in model.named_parameters():
            leaf = name.split(".")[-1]
            if leaf.endswith("_scale"):
                p.fill_(math.sqrt(cfg.model.d_model))
            elif "norm" in name and leaf == "weight":
                p.fill_(1.0)
            elif "tau_" in name:
                p.normal_(std=0.002, generator=gen) if leaf == "weight" else p.fill_(0.6)
            elif leaf == "bias":
                p.normal_(std=0.02, generator=gen)
            elif "neuron_pool" in name:
                p.normal_(generator=gen)
                p.div_(torch.linalg.vector_norm(p, dim=-1, keepdim=True))
            else:
                std = 1.0 / math.sqrt(p.shape[1])
                p.normal_(std=2 * std if "emb" in name else 0.02 if "expand_O" in name else std,
                          generator=gen)
    return model


def _trainer(cfg, seed):
    """A trainer around the model: it is built on a one-layer stand-in, whose host-side
    initialisation takes no time, and then handed the model and its optimizer."""
    model = _model(cfg, seed)
    m = cfg.model
    full = dict(vars(m))
    m.vocab_size, m.n_layers, m.n_qk, m.n_v, m.n_know = 64, 1, 64, 64, 64
    tr = Trainer(cfg, device=torch.device("cuda"), total_steps=1000, build_data=False)
    vars(m).update(full)
    model.backend = tr.backend
    t = cfg.training
    tr.model = model
    tr.optimizer = DawnAdamW(model.named_parameters(), lr=t.lr, weight_decay=t.weight_decay,
                             pool_weight_decay=t.pool_weight_decay, schedule=tr.schedule)
    # a run past its warm-up: the gradients of earlier steps were clipped to a norm of one
    tr.optimizer.count = 100
    n = sum(p.numel() for p in model.parameters())
    for v in tr.optimizer.exp_avg_sq:
        v.fill_(1.0 / n)
    return tr


def prepare(case, seed):
    cfg = _config(case, seed)
    B, S = case["batch"], case["seq"]
    gen = torch.Generator().manual_seed(seed + 1)
    ids = torch.randint(1, VOCAB, (B, S), generator=gen)
    state = {"op": case["op"], "seed": seed}
    if case["op"] == "train":
        mask = torch.ones(B, S, dtype=torch.int32)
        state.update(trainer=_trainer(cfg, seed), ids=ids.int().pin_memory(), mask=mask.pin_memory())
        return state
    model = _model(cfg, seed)
    model.eval()
    state.update(model=model, ids=ids.cuda())
    if case["op"] == "decode":
        # the prompt is in the cache; the session has been opened by its first token
        logits, ck, cv, n = prefill(model, state["ids"])
        state.update(session=DecodeSession(model, ck, cv, n), length=n,
                     token=logits[:, -1].argmax(-1))
        state["session"].step(state["token"])
    return state


def _grouped(named):
    """Few tensors for many parameters: embeddings and pools by themselves, the matrices of the
    layers stacked by kind, and all that is small (router, biases, LayerNorm, scales) in one."""
    out, layers, small = {}, {}, []
    for name, t in named:
        if t.ndim == 1 or name.startswith("router."):
            small.append(t.reshape(-1))
        elif name.startswith("layers."):
            layers.setdefault(name.split(".", 2)[2], []).append(t)
        else:
            out[name] = t
    out.update({k: torch.stack(v) for k, v in layers.items()})
    out["small"] = torch.cat(small)
    return out


def run(state):
    op = state["op"]
    if op == "train":
        tr = state["trainer"]
        torch.manual_seed(state["seed"])                      # dropout
        m = tr.train_step(state["ids"], state["mask"])
        return {"loss": m["total_loss"], "ce": m["ce_loss"],
                "weights": _grouped((n, p.detach()) for n, p in tr.optimizer.named)}
    if op == "prefill":
        logits, ck, cv, _ = prefill(state["model"], state["ids"])
        return {"logits": logits, "cache_k": ck, "cache_v": cv}
    if op == "eval":
        with torch.no_grad():
            r = state["model"](state["ids"], labels=state["ids"], want_diag=False)
        return {"loss": r["loss"], "per_token_ce": r["per_token_ce"]}
    s = state["session"]
    s.length = state["length"]                                # the same position in every pass
    logits = s.step(state["token"])
    return {"logits": logits, "cache_k": s.cache_k, "cache_v": s.cache_v}


# ---------------------------------------------------------------------------
L2_BYTES = 126e6


def work(case):
    """FLOPs of the matrix products (pools dense: with rows of many tokens in a tile some token
    uses nearly every unit; a decoding step counts the units that one of its rows uses) and bytes
    of weights, caches, inputs and results.  A pool that fits the L2 cache is read once for all
    layers, a larger one once per layer."""
    m = _config(case, 0).model
    B, S, D, L = case["batch"], case["seq"], m.d_model, m.n_layers
    op, new = case["op"], (1 if case["op"] == "decode" else case["seq"])
    T = B * new
    attn = 4.0 * B * L * D * (S + 1 if op == "decode" else S * (S + 1) / 2)      # QK^T and PV
    head = 2.0 * D * VOCAB * T
    weights = float(VOCAB * D + L * D * D)                                       # embedding, O
    used = 1.0
    if m.is_spatial:
        r, nq, nv, nk = m.d_route, m.n_qk, m.n_v, m.n_know
        units = nq + nv + nk
        active = 0.28 if op == "decode" else 1.0
        used = 1.0 - (1.0 - active) ** T
        per_tok = 2.0 * r * (units + nq) + active * 2.0 * D * (units + units + nq)
        per_tok += 2.0 * D * (4 * r + 4) + 2.0 * D * D                           # router, O
        pool = 2.0 * units * (r + 2 * D * used)                                  # bf16
        pools = pool * (L if 2.0 * units * (r + 2 * D) > L2_BYTES else 1)
        weights += D * (4 * r + 4)
        params = weights + units * (r + 2.0 * D)
    else:
        per_tok = 2.0 * (4 * D * D + 2 * D * m.d_ff)
        weights += L * (3.0 * D * D + 2.0 * D * m.d_ff)
        pools, params = 0.0, weights
    flops = L * per_tok * T + attn + head
    cache = 2.0 * 4 * L * D * B                                                  # fp32 K and V, one position
    if op == "train":
        # parameters and both moments are read and written in fp32; three times the forward's products
        return {"bytes": 24.0 * params + 8.0 * T, "flops": 3.0 * flops}
    moved = 2.0 * weights + pools
    if op == "eval":
        return {"bytes": moved + 8.0 * T, "flops": flops}
    if op == "prefill":
        return {"bytes": moved + 4.0 * T * VOCAB + cache * MAX_SEQ, "flops": flops}
    return {"bytes": moved + 4.0 * T * VOCAB + cache * (S + 1), "flops": flops}


def tolerance(case):
    """About four times what the framework shows against its fp32 and its bf16 library backends
    (bf16 operands through 12 to 18 layers).  A training step moves a weight by about 1e-3 of its
    size, of which the bf16 gradient is a few per cent off."""
    if case["op"] == "train":
        return {"rel": 3e-4, "max": 0.03}
    return {"rel": 0.01} if case["op"] == "eval" else {"rel": 0.03}
