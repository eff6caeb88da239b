"""The work that a user of this framework has it do, as measurable cases.

Five kinds, each through the entry points that a program calls:

  train     Trainer.train_sequence: the chunks of a sequence in order with hidden-state carry, forward + backward, a
            Schedule-Free AdamW step every ``accum`` chunks (what train.py runs)
  autograd  the module API: loss = model(chunk, return_loss=True), loss.backward(), gradients left in ``.grad``
            (a program with an optimizer or gradient clipping of its own)
  evaluate  model(chunk, return_loss=True) without gradients: validation loss
  prefill   Decoder.prefill: a prompt through the parallel kernels, last logits and recurrent state
  generate  runtime.generation.generate: prompt, then token by token with sampling (what generate.py runs)
  scan      the minGRU recurrence on its own, forward and backward, with a carried state

Shapes are minLM's: ``dim``, ``depth``, ``expansion``, ``ff_mult``; vocabulary 256.
"""
from __future__ import annotations

import gc
import io
import math

import torch

from gruboros_b200.models.minlm import minLM
from gruboros_b200.ops import kernels as K
from gruboros_b200.optim.schedulefree import AdamWScheduleFree
from gruboros_b200.runtime import generation
from gruboros_b200.runtime.trainer import Trainer

VOCAB = 256


def _case(name, kind, dim=0, depth=0, expansion=1.5, ff_mult=4.0, **kw):
    if kind == "scan":
        return dict(name=name, kind=kind, **kw)
    return dict(name=name, kind=kind, dim=dim, depth=depth, expansion=expansion, ff_mult=ff_mult, **kw)


def listed():
    return [
        # the smallest configuration of the benchmark file: a sequence of 512 bytes as two chunks of 256, batch 2;
        # short kernels, so launches and the host path count
        _case("train_small", "train", 512, 6, batch=2, chunk=256, chunks=2, accum=1),
        # train.py's defaults: --params 100m (512 x 32), --chunk_size 2k, --batch_size 4, a step per chunk
        _case("train_default", "train", 512, 32, batch=4, chunk=2048, chunks=1, accum=1),
        # the launch script's production recipe: 1g parameters at dim 1024, expansion 3, ff_mult 1.5, batch 1,
        # 8 chunks of 2048 with carry and one optimizer step for the eight
        _case("train_recipe", "train", 1024, 85, expansion=3.0, ff_mult=1.5, batch=1, chunk=2048, chunks=8, accum=8),
        # the headline benchmark: ~1B parameters, sequences of 4096 as two chunks, batch 8, a step per chunk; the largest
        _case("train_headline", "train", 2048, 20, batch=8, chunk=2048, chunks=2, accum=1),
        # --params 15m with odd sizes (rows that fill no tile) through loss.backward()
        _case("autograd_ragged", "autograd", 320, 12, batch=3, chunk=778),
        # validation of the 1B model on ragged sequences
        _case("evaluate_1b", "evaluate", 2048, 20, batch=3, chunk=1000),
        # a long document as the prompt of one sequence: large GEMMs, few channels for the scan to spread
        _case("prefill_long", "prefill", 2048, 20, batch=1, prompt=4096),
        # short prompts for a full batch of sequences: few rows, so reading the weights counts
        _case("prefill_short", "prefill", 2048, 20, batch=8, prompt=37),
        # generate.py as it comes: the default model, the default primer "The ", text streamed as it appears
        _case("generate_default", "generate", 512, 32, batch=1, prompt=4, tokens=64, stream=True),
        # the 1B model, one sequence and a full batch: every step reads every weight
        _case("generate_1b", "generate", 2048, 20, batch=1, prompt=128, tokens=48, stream=False),
        _case("generate_1b_batch", "generate", 2048, 20, batch=8, prompt=61, tokens=48, stream=False),
        # the operator benchmark of the benchmark file: batch 8, 8192 steps, 3072 channels
        _case("scan_op", "scan", batch=8, steps=8192, channels=3072),
    ]


# ---------------------------------------------------------------------- sizes
def _dims(c):
    return int(c["dim"] * c["expansion"]), int(c["dim"] * c["ff_mult"])


def _matrix_params(c):
    """Elements of the matrices that a token is multiplied with (the embedding is looked up)."""
    d, (di, f) = c["dim"], _dims(c)
    return c["depth"] * (3 * di * d + 2 * f * d) + VOCAB * d


def _params(c):
    return _matrix_params(c) + VOCAB * c["dim"] + c["depth"] * (3 * c["dim"] + _dims(c)[1]) + c["dim"]


def _activation_bytes(c, rows):
    d, (di, f) = c["dim"], _dims(c)
    return rows * c["depth"] * (12 * d + 6 * di + 4 * f)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "scan":
        n = c["batch"] * c["steps"] * c["channels"]
        return {"bytes": 6 * 2 * n, "flops": 30 * n}            # k, u, g read; h, dk, du written
    p, d = _matrix_params(c), c["dim"]
    if kind == "train":
        rows = c["batch"] * (c["chunk"] - 1) * c["chunks"]
        steps = c["chunks"] // c["accum"]
        # a step reads and writes the parameters and the two optimizer states in fp32
        return {"bytes": 24 * _params(c) * steps + c["batch"] * c["chunk"] * c["chunks"], "flops": 6 * p * rows}
    if kind == "autograd":
        rows = c["batch"] * (c["chunk"] - 1)
        return {"bytes": (2 + 4) * _params(c) + c["batch"] * c["chunk"], "flops": 6 * p * rows}      # bf16 weights, fp32 gradients
    if kind == "evaluate":
        rows = c["batch"] * (c["chunk"] - 1)
        return {"bytes": 2 * p + 4 * VOCAB * d + c["batch"] * c["chunk"], "flops": 2 * p * rows}
    rows = c["batch"] * c["prompt"]
    state = 4 * c["depth"] * c["batch"] * _dims(c)[0]
    if kind == "prefill":
        return {"bytes": 2 * p + rows + state, "flops": 2 * (p - VOCAB * d) * rows + 2 * VOCAB * d * c["batch"]}
    # every token reads every weight once (bf16); the prompt reads them once more
    return {"bytes": 2 * p * (1 + c["tokens"]) + 2 * state * c["tokens"],
            "flops": 2 * p * (rows + c["batch"] * c["tokens"])}


def tolerance(case):
    if case["kind"] == "generate":
        # tokens are whole numbers of a distribution with one likely entry; logits and state come from bf16 products
        return {"rel": 1e-2, "differ": 0.005}
    return {"rel": 1e-2}            # bf16 operands and saved activations, fp32 accumulation


# ----------------------------------------------------------------- drawn cases
def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng):
    expansion, ff_mult = rng.choice([(1.5, 4.0), (1.5, 4.0), (3.0, 1.5)])
    return dict(dim=64 * max(2, _size(rng, 128, 2048) // 64), depth=_size(rng, 2, 85), expansion=expansion, ff_mult=ff_mult)


def draw(rng):
    kind = rng.choice(["train", "train", "autograd", "evaluate", "prefill", "generate", "generate", "scan"])
    full = [c for c in listed() if c["name"] == "train_headline"][0]
    most = work(full)["flops"]
    memory = _activation_bytes(full, full["batch"] * (full["chunk"] - 1))
    while True:
        if kind == "scan":
            c = dict(kind=kind, batch=rng.randint(1, 8), steps=_size(rng, 64, 8192), channels=8 * _size(rng, 16, 384))
            return c
        c = dict(kind=kind, **_shape(rng), batch=rng.randint(1, 8))
        if _params(c) > 1.1e9:
            continue
        if kind == "train":
            chunks = rng.choice([1, 2, 4])
            c.update(chunk=_size(rng, 33, 2048), chunks=chunks, accum=rng.choice([1, chunks]))
        elif kind in ("autograd", "evaluate"):
            c.update(chunk=_size(rng, 33, 2048))
        elif kind == "prefill":
            c.update(prompt=_size(rng, 2, 4096))
        else:
            c.update(prompt=_size(rng, 2, 512), tokens=rng.randint(12, 64), stream=rng.random() < 0.5)
        rows = c["batch"] * max(c.get("chunk", 0), c.get("prompt", 0))
        if work(c)["flops"] <= most and _activation_bytes(c, rows) <= memory:
            return c


# ---------------------------------------------------------------------- inputs
def _model(c, gen, predictable):
    """A minLM with weights of a trained model's magnitudes.  ``predictable``: the head expects one byte after each byte,
    as text does in the middle of a word; otherwise the head is drawn like the other matrices."""
    with torch.device("meta"):
        model = minLM(num_tokens=VOCAB, dim=c["dim"], depth=c["depth"], expansion=c["expansion"], ff_mult=c["ff_mult"])
    model = model.to_empty(device="cuda")
    normal = lambda t, std: t.normal_(0.0, std, generator=gen)
    branch = 1.0 / math.sqrt(2 * c["depth"])          # the residual branches add up to about the embedding's size
    with torch.no_grad():
        normal(model.token_emb.weight, 1.0)
        normal(model.norm.weight, 0.1).add_(1.0)
        if predictable:
            follows = torch.randperm(VOCAB, generator=gen, device="cuda")
            model.to_logits.weight[follows] = model.token_emb.weight * (20.0 / c["dim"])
        else:
            normal(model.to_logits.weight, 1.0 / math.sqrt(c["dim"]))
        for _, norm, rnn, ff_norm, ff, _ in model.layers:
            normal(norm.weight, 0.1).add_(1.0)
            normal(ff_norm.weight, 0.1).add_(1.0)
            for lin, gain in ((rnn.to_hidden_and_gate, 1.0), (rnn.to_out, branch), (ff[0], 1.0), (ff[2], branch)):
                normal(lin.weight, gain / math.sqrt(lin.in_features))
            normal(ff[0].bias, 0.02)
            normal(ff[2].bias, 0.02)
    return model


def _bytes(gen, *shape):
    """Zipf(1.1) bytes, the synthetic corpus of the benchmark."""
    w = 1.0 / torch.arange(1, VOCAB + 1, dtype=torch.float64, device="cuda") ** 1.1
    n = math.prod(shape)
    return torch.multinomial(w / w.sum(), n, replacement=True, generator=gen).to(torch.uint8).view(*shape)


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["kind"] == "scan":
        B, T, C = c["batch"], c["steps"], c["channels"]
        ku = torch.randn(B, T, 2 * C, device="cuda", generator=gen, dtype=torch.bfloat16)      # u | k, as the gate GEMM leaves them
        h0 = torch.randn(B, C, device="cuda", generator=gen)
        h0 = torch.where(h0 >= 0, h0 + 0.5, torch.sigmoid(h0))
        g = torch.randn(B, T, C, device="cuda", generator=gen, dtype=torch.bfloat16)
        return dict(kind="scan", ku=ku, h0=h0, g=g, h=torch.empty_like(g), dku=torch.empty_like(ku),
                    h_last=torch.empty_like(h0), dh0=torch.empty_like(h0))
    gc.collect()            # a model and its engine refer to one another: give an earlier, dropped one's memory back now
    model = _model(c, gen, predictable=c["kind"] == "generate")
    s = dict(kind=c["kind"], model=model)
    if c["kind"] == "train":
        # in the middle of a run: the averaged state has a history, the second moments are of the gradients' size
        opt = AdamWScheduleFree(model.parameters(), lr=1e-3, betas=(0.9, 0.995), weight_decay=1e-4)
        flat = model.fused_engine().ensure_flat(model.token_emb.weight.device)
        opt.train()
        opt.ensure_state()
        flat.sf_v.uniform_(0.5e-7, 2e-7, generator=gen)
        opt.param_groups[0].update(k=1000, lr_max=1e-3, weight_sum=1000 * 1e-3 ** 2)
        s.update(opt=opt, flat=flat, tokens=_bytes(gen, c["batch"], c["chunk"] * c["chunks"]),
                 trainer=Trainer(model, opt, chunk_size=c["chunk"], grad_accum=c["accum"]))
    elif c["kind"] in ("autograd", "evaluate"):
        if c["kind"] == "evaluate":
            model.eval()
        s.update(flat=model.fused_engine().ensure_flat(model.token_emb.weight.device), tokens=_bytes(gen, c["batch"], c["chunk"]))
    else:
        model.eval()
        s.update(decoder=model.fused_engine().decoder(c["batch"]), tokens=_bytes(gen, c["batch"], c["prompt"]),
                 n=c.get("tokens", 0), stream=c.get("stream", False))
    return s


# -------------------------------------------------------------------- one pass
def run(state):
    s = state
    kind = s["kind"]
    if kind == "scan":
        C = s["g"].shape[2]
        k, u, dk, du = s["ku"][..., C:], s["ku"][..., :C], s["dku"][..., C:], s["dku"][..., :C]
        K.scan_fwd(k, u, s["h"], h0=s["h0"], h_last=s["h_last"])
        K.scan_bwd(k, u, s["h"], s["g"], dk, du, h0=s["h0"], dh0=s["dh0"])
        return s["h"], s["h_last"], s["dku"], s["dh0"]
    if kind == "train":
        losses = s["trainer"].train_sequence(s["tokens"])
        flat = s["flat"]
        return losses, torch.stack(s["trainer"].hidden), flat.data, flat.sf_z, flat.sf_v
    model = s["model"]
    if kind == "autograd":
        model.zero_grad()
        loss, hidden = model(s["tokens"], return_loss=True, return_prev_hiddens=True)
        loss.backward()
        return loss.detach(), torch.stack(hidden), s["flat"].grad
    if kind == "evaluate":
        with torch.no_grad():
            loss, hidden = model(s["tokens"], return_loss=True, return_prev_hiddens=True)
        return loss, torch.stack(hidden)
    dec = s["decoder"]
    if kind == "prefill":
        dec.reset()
        return dec.prefill(s["tokens"]), dec.h
    tokens = generation.generate(model, s["tokens"], s["n"], 0.85, 0, 0.9, device="cuda", stream=s["stream"], out=io.StringIO())
    return tokens, dec.logits, dec.h
