"""The work this framework is measured on: training steps, optimizer steps, Newton-Schulz calls, the decoder with
grouped-query attention and logits for sampling, each through the entry points a user's program calls.

``listed()`` names the fixed cases, ``draw(rng)`` gives one more of the same ranges; ``prepare`` makes what the
program has in hand before the call, ``run`` is one pass, ``work`` what the pass cannot do without, ``tolerance`` what
two correct implementations of the same precision may differ by.
"""

from __future__ import annotations

import math

import torch

from dion_b200 import Dion, DionMixedPrecisionConfig, Muon
from dion_b200.models import GPT, GPTConfig
from dion_b200.models.llama import Llama, LlamaConfig
from dion_b200.optim.newton_schulz import newton_schulz
from dion_b200.training import Hyperparameters, TrainStep, build_model, init_optimizer

VOCAB = 50304  # the GPT-2 vocabulary padded to a multiple of 128, as in the trainer


# ----------------------------------------------------------------------------------------------- the cases

def _train(layers, heads, head_dim, seq, batch, vocab, optimizer, rank_fraction, mixed, scalar):
    return dict(kind="train", layers=layers, heads=heads, head_dim=head_dim, seq=seq, batch=batch, vocab=vocab,
                optimizer=optimizer, rank_fraction=rank_fraction, mixed=mixed, scalar=scalar)


def _logits(layers, heads, head_dim, seq, batch, vocab=VOCAB):
    return dict(kind="logits", layers=layers, heads=heads, head_dim=head_dim, seq=seq, batch=batch, vocab=vocab)


def _opt(optimizer, matrices, rank_fraction, mixed, scalar, scalar_rows, scalar_cols):
    return dict(kind="optimizer", optimizer=optimizer, matrices=matrices, rank_fraction=rank_fraction, mixed=mixed,
                scalar=scalar, scalar_rows=scalar_rows, scalar_cols=scalar_cols)


def _ns(batch, m, n):
    return dict(kind="newton_schulz", batch=batch, m=m, n=n)


def _llama(layers, heads, kv_heads, head_dim, ffn, vocab, seq, batch):
    return dict(kind="llama", layers=layers, heads=heads, kv_heads=kv_heads, head_dim=head_dim, ffn=ffn, vocab=vocab,
                seq=seq, batch=batch)


def listed():
    return [
        # the benchmark recipe: GPT-160M, Dion with full rank, states in bf16, 64 sequences of 1024 tokens per GPU
        dict(_train(12, 12, 64, 1024, 64, VOCAB, "dion", 1.0, True, "lion"), name="train_160m_dion"),
        # the shipped Muon recipe: GPT-160M with 6 heads of 128, 32 sequences per GPU
        dict(_train(12, 6, 128, 1024, 32, VOCAB, "muon", 1.0, False, "lion"), name="train_160m_muon"),
        # a small model as used for plumbing runs and ablations: every kernel is short, launches count
        dict(_train(4, 4, 64, 256, 8, VOCAB, "dion", 0.25, False, "adamw"), name="train_small_dion"),
        # two layers of the 8B-shaped decoder on one 4096-token sequence: forward and backward, gradients in hand
        dict(_llama(2, 32, 8, 128, 14336, 128256, 4096, 1), name="llama_8b_shape_grads"),
        # prompts of a length nobody rounded, several at once: the logits that sampling starts from
        dict(_logits(12, 12, 64, 777, 8), name="logits_ragged"),
        # one short prompt: what every sampled token costs at the start of a text
        dict(_logits(12, 6, 128, 24, 1), name="logits_short"),
        # the optimizer step of the low-rank recipe (rank fraction 1/8) on the GPT-160M parameters
        dict(_opt("dion", "48x768x768,12x3072x768,12x768x3072", 0.125, True, "lion", 2 * VOCAB, 768),
             name="dion_step_160m_low_rank"),
        # the optimizer step on the matrices of two layers of the 8B shape, fp32 states, gains on AdamW
        dict(_opt("dion", "4x4096x4096,4x1024x4096,4x14336x4096,2x4096x14336", 0.125, False, "adamw", 5, 4096),
             name="dion_step_8b_shape"),
        # Muon on matrices whose sides fit no tile, and some whose rows are not even 16-byte aligned
        dict(_opt("muon", "6x1000x2504,8x520x1000,2x333x1001", 1.0, False, "adamw", 1000, 520), name="muon_step_ragged"),
        # Newton-Schulz called by itself: the smallest matrix, the square class of GPT-160M, the largest of the 8B shape
        dict(_ns(1, 256, 256), name="newton_schulz_256"),
        dict(_ns(48, 768, 768), name="newton_schulz_48x768"),
        dict(_ns(1, 4096, 14336), name="newton_schulz_4096x14336"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _seq(rng, hi):
    """Training and sampling lengths: mostly whole tiles of 128, one in three of any length."""
    return _log(rng, 16, hi) if rng.random() < 1 / 3 else 128 * rng.randint(1, hi // 128)


def _side(rng, hi):
    """A matrix side: multiples of 64, of 8, or any number, spread over the logarithm."""
    s = _log(rng, 64, hi)
    step = rng.choice((64, 64, 8, 1))
    return max(step, s // step * step)


def draw(rng):
    kind = rng.choice(("train", "train", "optimizer", "optimizer", "newton_schulz", "logits", "llama"))
    vocab = 8 * _log(rng, 500, VOCAB // 8)
    if kind == "train":
        head_dim = rng.choice((64, 128))
        heads = rng.randint(2, 768 // head_dim)
        seq = _seq(rng, 1024)
        return _train(rng.randint(2, 12), heads, head_dim, seq, min(64, _log(rng, 1, max(2, 65536 // seq))), vocab,
                      rng.choice(("dion", "dion", "muon")), rng.choice((0.125, 0.25, 0.5, 1.0)),
                      rng.random() < 0.5, rng.choice(("lion", "adamw")))
    if kind == "logits":
        head_dim = rng.choice((64, 128))
        return _logits(rng.randint(2, 12), rng.randint(2, 768 // head_dim), head_dim, _seq(rng, 1024), _log(rng, 1, 32), vocab)
    if kind == "llama":
        kv = rng.choice((1, 2, 4, 8))
        head_dim = rng.choice((64, 128))
        return _llama(rng.randint(1, 2), kv * rng.choice((1, 2, 4)), kv, head_dim, 256 * rng.randint(2, 56), vocab,
                      128 * rng.randint(2, 32), 1)
    if kind == "newton_schulz":
        m, n = _side(rng, 4096), _side(rng, 14336)
        m, n = (n, m) if rng.random() < 0.3 and n <= 4096 else (m, n)
        return _ns(max(1, min(48, int(48 * (768 / max(m, 768)) ** 2 * (768 / max(n, 768)) * rng.random()))), m, n)
    optimizer = rng.choice(("dion", "dion", "muon"))
    classes = []
    for _ in range(rng.randint(1, 3)):
        m, n = _side(rng, 4096), _side(rng, 4096)
        if optimizer == "dion":  # low-rank factors are kept for matrices with whole 16-byte rows
            m, n = max(8, m // 8 * 8), max(8, n // 8 * 8)
        classes.append("%dx%dx%d" % (min(48, _log(rng, 1, max(2, (1 << 26) // (m * n)))), m, n))
    return _opt(optimizer, ",".join(classes), rng.choice((0.125, 0.25, 0.5)), rng.random() < 0.5,
                rng.choice(("lion", "adamw")), _log(rng, 1, VOCAB), rng.choice((256, 520, 768)))


# ----------------------------------------------------------------------------------------------- states

def _classes(text):
    return [tuple(int(v) for v in c.split("x")) for c in text.split(",")]


def _stack(params):
    """Lays parameters of one shape out in one buffer (each stays a contiguous, aligned tensor of its own) and
    returns the buffers, so that all updated weights of a model come back as a handful of tensors."""
    by_shape = {}
    for p in params:
        by_shape.setdefault(tuple(p.shape), []).append(p)
    out = []
    for shape, members in by_shape.items():
        per = (math.prod(shape) + 15) // 16 * 16
        buf = torch.zeros(len(members), per, dtype=members[0].dtype, device=members[0].device)
        for row, p in zip(buf, members):
            view = row[:p.numel()].view(shape)
            view.copy_(p.data)
            p.data = view
        out.append(buf)
    return out


def _tokens(batch, seq, vocab):
    t = torch.randint(0, vocab, (batch, seq + 1), device="cuda")
    return t[:, :-1].contiguous(), t[:, 1:].contiguous()


def _gradient(count, m, n):
    """Gradients as they come out of a backward pass: a decaying spectrum, up to eight times as high as the largest
    singular value of the flat floor of noise under it."""
    k = min(64, m, n)
    scale = torch.logspace(0, -1.5, k, device="cuda") * (8 * (m ** 0.5 + n ** 0.5) / (m * n) ** 0.5)
    left = torch.randn(count, m, k, device="cuda") * scale
    g = torch.bmm(left, torch.randn(count, k, n, device="cuda"))
    return g.add_(torch.randn(count, m, n, device="cuda")).mul_(1e-3)


def _resume(case, optimizer, sigma):
    """Gives the optimizer the state of a run under way, as a checkpoint does: momentum of `sigma` per entry, the
    right factors Q of the last step, second moments."""
    saved = optimizer.state_dict()
    states, index = {}, 0
    for group in optimizer.param_groups:
        for p in group["params"]:
            state = dict(momentum=torch.randn_like(p) * sigma)
            if group["algorithm"] == "dion":
                m, n = p.shape
                r = _rank(case, m, n)
                state["Q"] = torch.nn.functional.normalize(torch.randn(n if m >= n else m, r, device="cuda"), dim=0)
            elif group["algorithm"] == "adamw":
                state["variance"] = torch.full_like(p, sigma * sigma)
            states[index] = state
            index += 1
    optimizer.load_state_dict(dict(state=states, param_groups=saved["param_groups"]))


def prepare(case, seed):
    torch.manual_seed(seed)
    kind = case["kind"]
    if kind == "train":
        hp = Hyperparameters(model_dim=case["heads"] * case["head_dim"], n_layer=case["layers"], n_head=case["heads"],
                             sequence_length=case["seq"], device_batch_size=case["batch"], batch_size=case["batch"],
                             optimizer=case["optimizer"], scalar_opt=case["scalar"], lr=0.02, mu=0.95, weight_decay=0.01,
                             rank_fraction=case["rank_fraction"], mixed_precision=case["mixed"], num_iterations=10 ** 6)
        model, raw = build_model(hp, None, False, vocab_size=case["vocab"])
        weights = _stack(raw.parameters())
        optimizer = init_optimizer(raw, None, None, hp)
        # gradient entries of this model are 1e-5 to 2e-4 at 65536 tokens and grow as the batch gets smaller
        _resume(case, optimizer, 1e-4 * math.sqrt(65536 / (case["batch"] * case["seq"])))
        return dict(kind=kind, step=TrainStep(model, raw, optimizer), weights=weights,
                    batch=_tokens(case["batch"], case["seq"], case["vocab"]))
    if kind == "logits":
        with torch.device("cuda"):
            model = GPT(GPTConfig(sequence_len=case["seq"], vocab_size=case["vocab"], n_layer=case["layers"],
                                  n_head=case["heads"], n_embd=case["heads"] * case["head_dim"]))
        model.init_weights()
        model.eval()
        return dict(kind=kind, model=model, idx=_tokens(case["batch"], case["seq"], case["vocab"])[0])
    if kind == "llama":
        with torch.device("cuda"):
            model = Llama(LlamaConfig(sequence_len=case["seq"], vocab_size=case["vocab"], n_layer=case["layers"],
                                      n_head=case["heads"], n_kv_head=case["kv_heads"],
                                      n_embd=case["heads"] * case["head_dim"], ffn_dim=case["ffn"]))
        model.init_weights()
        return dict(kind=kind, model=model, params=list(model.parameters()),
                    batch=_tokens(case["batch"], case["seq"], case["vocab"]))
    if kind == "newton_schulz":
        g = _gradient(case["batch"], case["m"], case["n"]).bfloat16()
        return dict(kind=kind, g=g if case["batch"] > 1 else g[0])
    matrices, grads, weights = [], [], []
    for count, m, n in _classes(case["matrices"]):
        members = [torch.nn.Parameter(torch.randn(m, n, device="cuda") / math.sqrt(n)) for _ in range(count)]
        weights += _stack(members)
        matrices += members
        grads += [g.clone() for g in _gradient(count, m, n)]
    scalar = torch.nn.Parameter(torch.randn(case["scalar_rows"], case["scalar_cols"], device="cuda"))
    weights.append(scalar.data)
    groups = [dict(params=matrices), dict(params=[scalar], algorithm=case["scalar"], lr=0.002, weight_decay=0)]
    bf16 = torch.bfloat16
    if case["optimizer"] == "dion":
        mp = DionMixedPrecisionConfig(momentum_dtype=bf16, Q_dtype=bf16, variance_dtype=bf16) if case["mixed"] else None
        optimizer = Dion(groups, rank_fraction=case["rank_fraction"], rank_multiple_of=8, lr=0.02, mu=0.95,
                         weight_decay=0.01, mixed_precision_config=mp)
    else:
        optimizer = Muon(groups, lr=0.02, mu=0.95, weight_decay=0.01, nesterov=True)
    _resume(case, optimizer, 1e-3)
    grads.append(torch.randn_like(scalar) * 1e-3)
    return dict(kind=kind, optimizer=optimizer, params=matrices + [scalar], grads=grads, weights=weights,
                matrices=matrices)


# ----------------------------------------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "train":
        loss = state["step"]([state["batch"]])
        return [loss] + state["weights"]
    if kind == "logits":
        with torch.no_grad():
            return state["model"](state["idx"], return_logits=True)
    if kind == "llama":
        for p in state["params"]:
            p.grad = None
        loss = state["model"](*state["batch"])
        loss.backward()
        return [loss.detach()] + [p.grad for p in state["params"]]
    if kind == "newton_schulz":
        return newton_schulz(state["g"])
    for p, g in zip(state["params"], state["grads"]):
        p.grad = g
    optimizer = state["optimizer"]
    optimizer.step()
    out = list(state["weights"])
    if len(state["matrices"]) <= 16:  # few enough to hand the state back too
        out += [v for p in state["matrices"] for v in optimizer.state[p].values()]
    return out


# ----------------------------------------------------------------------------------------------- work, tolerance

def _rank(case, m, n):
    r = case["rank_fraction"] * min(m, n)
    return min(8 * math.ceil(r / 8), m, n)


def _update_work(case, matrices):
    """Operations and bytes of one optimizer step over `matrices` (count, m, n), without the gradients' producer."""
    flops = nbytes = 0.0
    state = 2 if case["mixed"] else 4
    for count, m, n in matrices:
        k, l = min(m, n), max(m, n)
        if case["optimizer"] == "muon":
            flops += count * 5 * (3.0 * k * k * l + k ** 3)       # the symmetric products counted once
            nbytes += count * m * n * (8 + 8 + 4)                 # weights and momentum in and out, gradient in
        else:
            r = _rank(case, m, n)
            # P = M Q, R = M^T P, error feedback, update; Gram matrix, triangular factor and its application
            flops += count * (8.0 * m * n * r + 3.0 * l * r * r + 2.0 / 3.0 * r ** 3)
            nbytes += count * (m * n * (8 + 4 + 2 * state) + 2 * state * r * k)
    return flops, nbytes


def _scalar_bytes(case, numel):
    return numel * (8 + 4 + (2 if case["mixed"] else 4) * (4 if case["scalar"] == "adamw" else 2))


def work(case):
    kind = case["kind"]
    if kind == "newton_schulz":
        k, l = sorted((case["m"], case["n"]))
        return dict(flops=case["batch"] * 5 * (3.0 * k * k * l + k ** 3), bytes=4.0 * case["batch"] * k * l)
    if kind == "optimizer":
        flops, nbytes = _update_work(case, _classes(case["matrices"]))
        return dict(flops=flops, bytes=nbytes + _scalar_bytes(case, case["scalar_rows"] * case["scalar_cols"]))
    d, tokens, v = case["heads"] * case["head_dim"], case["batch"] * case["seq"], case["vocab"]
    attention = 2.0 * case["layers"] * case["batch"] * case["heads"] * case["seq"] ** 2 * case["head_dim"]  # causal half
    if kind == "llama":
        kv = case["kv_heads"] * case["head_dim"]
        params = case["layers"] * (2 * d * d + 2 * kv * d + 3 * d * case["ffn"])
        flops = 6.0 * tokens * (params + v * d) + 3.5 * attention
        return dict(flops=flops, bytes=4.0 * (2 * (params + v * d) + v * d + min(v, tokens) * d))
    params = case["layers"] * 12 * d * d
    if kind == "logits":
        flops = 2.0 * tokens * params + attention + 2.0 * case["batch"] * v * d
        return dict(flops=flops, bytes=4.0 * (params + v * d + min(v, tokens) * d + case["batch"] * v))
    flops = 6.0 * tokens * (params + v * d) + 3.5 * attention
    matrices = [(4 * case["layers"], d, d), (2 * case["layers"], 4 * d, d)]
    update_flops, nbytes = _update_work(case, matrices)
    # weights and states in and out; gradients need not exist in memory
    nbytes += _scalar_bytes(case, 2 * v * d) - 4.0 * (params + 2 * v * d) + 16.0 * tokens
    return dict(flops=flops + update_flops, bytes=nbytes)


def tolerance(case):
    """About four times what the path differs by when it runs with another attention, another split of its sums, in
    fp32, or with the plain statement of the same iteration."""
    kind = case["kind"]
    if kind == "newton_schulz":      # bf16 iterates; small singular values are amplified in every step: 0.02 / 0.18 seen
        return dict(rel=0.03, max=0.7)
    if kind == "logits":             # bf16 activations against fp32 ones: 0.011 / 0.05 seen
        return dict(rel=0.03, max=0.2)
    if kind == "llama":              # gradients through bf16 activations, another attention: 0.010 / 0.26 seen
        return dict(rel=0.03, max=0.9)
    if kind == "train":
        # updated weights: the update is 2 % of them; single Lion updates change sign (0.07 of an entry).  With high
        # rank the smallest directions of the momentum are below the gradients' own rounding: 0.013 / 0.19 seen
        if case["optimizer"] == "dion" and case["rank_fraction"] > 0.25:
            return dict(rel=0.03, max=0.8)
        return dict(rel=4e-3, max=0.3)               # 8e-4 / 0.06 seen
    if case["optimizer"] == "muon":  # the same bf16 iteration, of which the weights take a part: 5e-4 / 6e-3 seen
        return dict(rel=2e-3, max=0.025)
    # products in tf32 or bf16, orthonormalisation close to fp32; after two steps 3e-4 / 1.6e-3 seen (the columns of the
    # smallest directions move).  bf16 states: an entry may round the other way
    return dict(rel=1e-3, max=0.03 if case["mixed"] else 8e-3)
