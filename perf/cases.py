"""The work that a user of this library has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes its inputs on the GPU from a seed,
``run`` is one pass through the public entry points.  The sizes are those of the
library's tests and benchmark (the recursion on 32 lattices, the unpruned loss, the
pruned pipeline at 500 and 5000 symbols) and generic ones around them.

Kinds of work:

  simple    rnnt_loss_simple / rnnt_loss_smoothed, forward and backward
  mi        mutual_information_recursion with occupancies, forward and backward
  unpruned  rnnt_loss on full joiner logits, forward and backward
  step      the pruned pipeline of one training step: smoothed simple loss -> prune
            ranges -> fused joiner and pruned loss, forward and backward
  eval      the same losses without gradients of the pruned branch (validation)
  joiner    the documented composition with the caller's own network between
            do_rnnt_pruning and rnnt_loss_pruned, forward and backward
"""
import math
import random

import torch

import fast_rnnt_b200 as fr

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16,
           "f64": torch.float64}

_BASE = dict(kind="step", B=64, T=500, S=100, C=500, D=512, R=5, dtype="f32",
             rnnt_type="regular", lm_scale=0.25, am_scale=0.0, delay=0.0, ragged=True)


def _case(**kw):
    c = dict(_BASE)
    c.update(kw)
    if c["kind"] in ("simple", "mi", "unpruned"):
        c["D"] = c["R"] = 0
    if c["kind"] == "mi":
        c["C"] = 0
    return c


def listed():
    return [
        # a handful of short utterances with a character vocabulary: launches and host time
        _case(name="simple small", kind="simple", B=4, T=100, S=20, C=50, lm_scale=0.0),
        # fine-tuning on single short utterances, the whole pipeline: latency of a step
        _case(name="step tiny", B=2, T=61, S=13, C=72, D=128, R=4),
        # the recursion alone on padded lattices, as other alignment losses use it
        _case(name="recursion", kind="mi", B=32, T=512, S=128, ragged=False),
        # long-form audio: few utterances, tall and wide lattices, the modified topology
        _case(name="recursion long", kind="mi", B=6, T=2211, S=423, rnnt_type="modified"),
        # the unpruned loss, small vocabulary and short utterances (the classic transducer)
        _case(name="unpruned", kind="unpruned", B=8, T=200, S=50, C=500),
        # odd vocabulary (characters of a large script), default smoothing, both branches on
        _case(name="smoothed odd vocabulary", kind="simple", B=16, T=293, S=59, C=4233,
              lm_scale=0.1, am_scale=0.1),
        # validation of a 500-symbol model between epochs
        _case(name="evaluation", kind="eval", B=24, T=500, S=100, C=500),
        # the training step of the benchmark: 64 utterances, 500 symbols
        _case(name="step 500 symbols", B=64, T=500, S=100, C=500),
        # mixed-precision training: 16-bit activations, modified topology, a delay penalty,
        # sizes that are no multiple of anything
        _case(name="step mixed precision", B=23, T=411, S=77, C=500, D=512, dtype="bf16",
              rnnt_type="modified", delay=0.01),
        # the caller keeps a joiner of its own between pruning and loss
        _case(name="step own joiner", kind="joiner", B=32, T=400, S=80, C=500, D=512),
        # one GPU's share of a large batch with 5000 symbols
        _case(name="step 5000 symbols", B=64, T=400, S=60, C=5000, D=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above; batches shrink until a case costs no more than
    the largest listed one."""
    kind = rng.choice(["step", "step", "step", "simple", "simple", "mi", "mi", "unpruned",
                       "eval", "joiner"])
    rnnt_type = rng.choice(["regular", "regular", "modified", "constrained"])
    if kind == "mi":
        rnnt_type = rng.choice(["regular", "modified"])
        S = _log_int(rng, 16, 440)
        T = S + _log_int(rng, 40, 1800)
        c = _case(kind=kind, B=_log_int(rng, 4, 64), T=T, S=S, rnnt_type=rnnt_type,
                  ragged=rng.random() < 0.5)
    elif kind == "unpruned":
        S = rng.randint(8, 60)
        c = _case(kind=kind, B=_log_int(rng, 2, 16), T=S + rng.randint(40, 240), S=S,
                  C=_log_int(rng, 28, 1000), rnnt_type=rnnt_type,
                  dtype=rng.choice(["f32", "f32", "bf16"]))
    elif kind == "simple":
        S = rng.randint(10, 110)
        c = _case(kind=kind, B=_log_int(rng, 2, 64), T=S + _log_int(rng, 60, 500), S=S,
                  C=_log_int(rng, 28, 5000), rnnt_type=rnnt_type,
                  lm_scale=rng.choice([0.0, 0.1, 0.25]), am_scale=rng.choice([0.0, 0.1]))
    else:
        S = rng.randint(10, 110)
        c = _case(kind=kind, B=_log_int(rng, 2, 64), T=S + _log_int(rng, 40, 450), S=S,
                  C=4 * _log_int(rng, 8, 1250), D=8 * rng.randint(16, 80), R=rng.randint(4, 6),
                  rnnt_type=rnnt_type, delay=rng.choice([0.0, 0.0, 0.01]),
                  dtype=("f32" if kind == "joiner" else rng.choice(["f32", "f32", "bf16", "f16"])))
    top = work(listed()[-1])
    while c["B"] > 1 and (work(c)["bytes"] > top["bytes"] or work(c)["flops"] > top["flops"]):
        c["B"] -= max(1, c["B"] // 8)
    return c


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    r = random.Random(seed)
    B, T, S, C, D = case["B"], case["T"], case["S"], case["C"], case["D"]
    dt = _DTYPES[case["dtype"]]

    def normal(scale, *shape):
        t = torch.randn(*shape, generator=g, device=dev)
        return t.mul_(scale).to(dt).requires_grad_(True)

    rows = None
    if case["ragged"]:
        # lengths of a padded batch: the first utterance fills it
        rows = [[0, 0, S, T]]
        for _ in range(B - 1):
            s = r.randint((S + 1) // 2, S)
            rows.append([0, 0, s, max(s, r.randint(7 * T // 10, T))])
    state = dict(case=case, boundary=None)
    if rows is not None:
        state["boundary"] = torch.tensor(rows, dtype=torch.int64).to(dev)
        if case["kind"] in ("step", "eval", "joiner"):
            # a training program's loader has the lengths on the host
            fr.provide_boundary_rows(state["boundary"], rows)
    if case["kind"] == "mi":
        t1 = T if case["rnnt_type"] == "modified" else T + 1
        for name, shape in (("px", (B, S, t1)), ("py", (B, S + 1, T))):
            x = torch.rand(*shape, generator=g, device=dev).mul_(-6.0)
            state[name] = x.to(dt).requires_grad_(True)
        return state
    state["symbols"] = torch.randint(1, C, (B, S), generator=g, device=dev)
    if case["kind"] == "unpruned":
        state["logits"] = normal(1.0, B, T, S + 1, C)
        return state
    state["am"] = normal(0.5, B, T, C)
    state["lm"] = normal(0.5, B, S + 1, C)
    if case["kind"] == "simple":
        return state
    state["enc"] = normal(1.0, B, T, D)
    state["dec"] = normal(1.0, B, S + 1, D)
    # the joiner's last layer, initialised as torch.nn.Linear does, kept in float32
    k = 1.0 / math.sqrt(D)
    for name, shape in (("weight", (C, D)), ("bias", (C,))):
        w = torch.rand(*shape, generator=g, device=dev).mul_(2 * k).sub_(k)
        state[name] = w.requires_grad_(True)
    return state


def _simple(st, return_grad):
    c = st["case"]
    common = dict(boundary=st["boundary"], rnnt_type=c["rnnt_type"], delay_penalty=c["delay"],
                  reduction="sum", return_grad=return_grad)
    if c["lm_scale"] == 0.0 and c["am_scale"] == 0.0:
        return fr.rnnt_loss_simple(st["lm"], st["am"], st["symbols"], 0, **common)
    return fr.rnnt_loss_smoothed(st["lm"], st["am"], st["symbols"], 0, c["lm_scale"],
                                 c["am_scale"], **common)


def _pruned(st, ranges):
    c = st["case"]
    common = dict(boundary=st["boundary"], rnnt_type=c["rnnt_type"], delay_penalty=c["delay"],
                  reduction="sum")
    if c["kind"] != "joiner":
        return fr.rnnt_loss_pruned_joiner(st["enc"], st["dec"], ranges, st["weight"], st["bias"],
                                          st["symbols"], 0, **common)
    am_p, lm_p = fr.do_rnnt_pruning(st["enc"], st["dec"], ranges)
    logits = fr.linear(torch.tanh(am_p + lm_p), st["weight"], st["bias"])
    return fr.rnnt_loss_pruned(logits, st["symbols"], ranges, 0, **common)


def run(state):
    st, c = state, state["case"]
    if c["kind"] == "mi":
        scores, occ = fr.mutual_information_recursion(st["px"], st["py"], st["boundary"],
                                                      return_grad=True)
        return [scores.detach(), torch.autograd.grad(scores.sum(), [st["px"], st["py"]])]
    if c["kind"] == "unpruned":
        loss = fr.rnnt_loss(st["logits"], st["symbols"], 0, boundary=st["boundary"],
                            rnnt_type=c["rnnt_type"], delay_penalty=c["delay"], reduction="sum")
        return [loss.detach(), torch.autograd.grad(loss, [st["logits"]])]
    if c["kind"] == "simple":
        loss = _simple(st, False)
        return [loss.detach(), torch.autograd.grad(loss, [st["lm"], st["am"]])]
    if c["kind"] == "eval":
        with torch.no_grad():
            loss, occ = _simple(st, True)
            ranges = fr.get_rnnt_prune_ranges(occ[0], occ[1], st["boundary"], c["R"])
            return [loss, occ, ranges, _pruned(st, ranges)]
    loss, occ = _simple(st, True)
    ranges = fr.get_rnnt_prune_ranges(occ[0], occ[1], st["boundary"], c["R"])
    pruned = _pruned(st, ranges)
    leaves = [st[k] for k in ("am", "lm", "enc", "dec", "weight", "bias")]
    return [loss.detach(), pruned.detach(), ranges, torch.autograd.grad(loss + pruned, leaves)]


def work(case):
    """Inputs read once, outputs written once, and the multiply-adds of the products (the
    recursion's 20 or so operations per lattice cell are left out beside them)."""
    B, T, S, C, D, R = (case[k] for k in "BTSCDR")
    eb = {"f64": 8, "f32": 4}.get(case["dtype"], 2)
    lattice = B * (S * (T + 1) + (S + 1) * T)
    if case["kind"] == "mi":
        return {"bytes": 2 * eb * lattice, "flops": 20 * lattice}
    if case["kind"] == "unpruned":
        n = B * T * (S + 1) * C
        return {"bytes": 2 * eb * n, "flops": 6 * n}
    vocab = B * (T + S + 1) * C              # am and lm
    simple = 2 * B * (S + 1) * T * C         # one product between them
    if case["kind"] == "simple":
        return {"bytes": 2 * eb * vocab, "flops": 3 * simple}
    width = B * (T + S + 1) * D              # enc and dec
    rows = B * T * R
    join = 2 * rows * D * C
    if case["kind"] == "eval":
        return {"bytes": eb * (vocab + width) + 4 * (lattice + C * (D + 1)) + 8 * rows,
                "flops": simple + join}
    w = {"bytes": 2 * eb * (vocab + width) + 8 * C * (D + 1) + 8 * rows,
         "flops": 3 * simple + 3 * join}
    if case["kind"] == "joiner":
        # the pruned tensor, the logits and their gradients exist in the caller's program
        w["bytes"] += 4 * 2 * rows * (2 * D + 2 * C)
    return w


def tolerance(case):
    # float32 scores reach a few thousand, so a cell of the recursion carries 1e-4 of
    # rounding and a chain of several hundred cells 1e-4 to 1e-3 in the occupancies
    rel = 3e-4 if case["T"] + case["S"] < 800 else 1e-3
    if case["dtype"] in ("bf16", "f16"):
        rel = 5e-3                           # gradients come back in 16 bits
    if case["kind"] in ("step", "eval", "joiner"):
        # the ranges are an argmax over window sums of float32 occupancies: where two windows
        # tie within rounding, a frame's band may move, and its gradients with it
        return {"rel": max(rel, 1e-2), "max": 0.99, "differ": 2e-3}
    return {"rel": rel}
