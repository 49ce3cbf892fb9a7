"""The optimizer steps that users of this package run, as cases that can be timed and compared.

A case names an optimizer class, a family of parameter shapes with its sizes, and the options of the run.  One pass is
one ``step()`` of that optimizer over all parameters, in the middle of a training run: the state tensors exist, the
gradients of the step are in device memory.  The shapes are those of the models these optimizers train: small
multi-layer perceptrons (the learned optimizers' own meta-training tasks, where a step is all latency), convolutional
networks (four-dimensional weights), and the transformer shapes of ``pylo_b200.workloads`` from a few million to a few
hundred million parameters.  Everything is fp32, as the optimizers require.

All parameters of a model are views into one flat buffer, and so are their gradients and every kind of state tensor,
each view on a 512-byte boundary as if it had been allocated by itself.  Sharded training lays parameters out this way,
and the whole result of a step can then be handed back as a few tensors.
"""

import random

import torch

from pylo_b200 import models, optim

ALIGN = 128  # floats: every tensor starts on a 512-byte boundary, as a separate allocation would

# ---------------------------------------------------------------------------------------------------------------------
# parameter shapes
# ---------------------------------------------------------------------------------------------------------------------


def shapes_of(case):
    """The parameter shapes of a case, in the order in which the optimizer gets them."""
    net, d, ff, layers = case["net"], case["width"], case.get("ff", 0), case["layers"]
    if net == "mlp":  # inputs -> width -> ... -> width -> outputs
        s, fan_in = [], case["inputs"]
        for out in [d] * layers + [case["outputs"]]:
            s += [(out, fan_in), (out,)]
            fan_in = out
        return s
    if net == "conv":  # 3x3 convolutions with batch-norm vectors, channels doubling at every stage, a linear classifier
        s, fan_in, out = [(d, 3, 7, 7), (d,), (d,)], d, d
        for stage in range(layers):
            for k in range(2):
                s += [(out, fan_in, 3, 3), (out,), (out,)]
                fan_in = out
            out *= 2
        return s + [(case["outputs"], fan_in), (case["outputs"],)]
    if net == "vit":
        s = [(d, 3, 16, 16), (d,), (case["context"], d), (d,)]
        for _ in range(layers):
            s += [(d,), (d,), (d, 3 * d), (3 * d,), (d, d), (d,), (d,), (d,), (d, ff), (ff,), (ff, d), (d,)]
        return s + [(d,), (d,), (d, case["outputs"]), (case["outputs"],)]
    if net == "gpt":
        s = [(case["outputs"], d), (case["context"], d)]
        for _ in range(layers):
            s += [(d,), (d,), (d, 3 * d), (3 * d,), (d, d), (d,), (d,), (d,), (d, ff), (ff,), (ff, d), (d,)]
        return s + [(d,), (d,)]
    s = [(case["outputs"], d)] if case["outputs"] else []  # "llama": gated feed-forward, grouped keys and values, no biases
    for _ in range(layers):
        s += [(d, d), (d // 4, d), (d // 4, d), (d, d), (ff, d), (ff, d), (d, ff), (d,), (d,)]
    return s + [(d,)] + ([(case["outputs"], d)] if case["outputs"] else [])


def numel(shape):
    n = 1
    for x in shape:
        n *= x
    return n


def is_embedding(case, shape):
    """Token embeddings and output heads, which the CELO2 family leaves to AdamW (an ``is_embedding`` group)."""
    return case["opt"].endswith("celo2") and case["net"] in ("gpt", "llama") and len(shape) == 2 and shape[0] == case["outputs"]


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------


def listed():
    return [
        # the 784-128-128-10 perceptron of the learned optimizers' own tasks (118 K parameters): the step is launches
        # and host work, and thousands of steps are run one after the other
        dict(name="adafaclo mlp", opt="adafaclo", net="mlp", inputs=784, width=128, layers=2, outputs=10),
        dict(name="celo2 mlp", opt="celo2", net="mlp", inputs=784, width=128, layers=2, outputs=10, orthogonalize=True),
        dict(name="velo mlp", opt="velo", net="mlp", inputs=784, width=128, layers=2, outputs=10),
        # tabular data with sizes that are multiples of nothing: no row starts on a 16-byte boundary
        dict(name="velo ragged mlp", opt="velo", net="mlp", inputs=1433, width=1001, layers=3, outputs=7),
        # an image classifier of four stages: most of the parameters sit in four-dimensional weights
        dict(name="adafaclo conv", opt="adafaclo", net="conv", width=64, layers=4, outputs=1000),
        # ViT-B/16 with weight decay on the matrices only, i.e. two param groups, as such models are trained
        dict(name="adafaclo vit", opt="adafaclo", net="vit", width=768, ff=3072, layers=12, context=197, outputs=1000,
             wd=0.01, groups=2),
        dict(name="elo_celo2 vit", opt="elo_celo2", net="vit", width=768, ff=3072, layers=12, context=197, outputs=1000,
             wd=0.1, clip=True, orthogonalize=True),
        # a small language model (odd vocabulary), gradient clipping by the global norm
        dict(name="elo gpt", opt="elo", net="gpt", width=768, ff=3072, layers=6, context=1024, outputs=50257, wd=0.1, clip=True),
        # GPT-2-medium shapes, gradients with outliers
        dict(name="velo gpt", opt="velo", net="gpt", width=1024, ff=4096, layers=24, context=1024, outputs=50257, wd=0.01),
        # one 4096 x 4096 matrix and its bias: Newton-Schulz decides
        dict(name="celo2 square", opt="celo2", net="mlp", inputs=4096, width=4096, layers=0, outputs=4096, wd=0.1,
             orthogonalize=True),
        # one Llama-3-8B block with an embedding and a head that go to AdamW, steps not orthogonalised
        dict(name="celo2 llama", opt="celo2", net="llama", width=4096, ff=14336, layers=1, outputs=32000, wd=0.1,
             orthogonalize=False),
        # two Llama-3-8B blocks (436 M parameters), what one of many ranks owns of the whole model
        dict(name="adafaclo llama", opt="adafaclo", net="llama", width=4096, ff=14336, layers=2, outputs=0),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _round(rng, x):
    """Most models have widths that are multiples of 64 or 8; some do not care."""
    m = rng.choice((64, 64, 8, 4, 1))
    return max(m, x // m * m)


def draw(rng: random.Random):
    """One more case: any optimizer over any of the shape families, sizes spread over their logarithm."""
    most = max(work(c)["bytes"] for c in listed())
    most_flops = {o: max(work(c)["flops"] for c in listed() if bool(c.get("orthogonalize")) == o) for o in (False, True)}
    while True:
        opt = rng.choice(("adafaclo", "elo", "celo2", "elo_celo2", "velo"))
        net = rng.choice(("mlp", "mlp", "conv", "vit", "gpt", "llama"))
        if net == "conv" and opt.endswith("celo2"):
            continue  # CELO2 normalises per 3x3 kernel there, which is not how it is used
        c = dict(opt=opt, net=net)
        if net == "mlp":
            c.update(inputs=_log(rng, 16, 8192), width=_round(rng, _log(rng, 32, 4096)), layers=rng.randint(1, 6),
                     outputs=_log(rng, 2, 4096))
        elif net == "conv":
            c.update(width=_log(rng, 8, 72), layers=rng.randint(2, 4), outputs=rng.choice((10, 100, 1000)))
        else:
            d = {"vit": _log(rng, 128, 1280), "gpt": _log(rng, 128, 1600), "llama": _log(rng, 512, 4096)}[net]
            d = max(64, d // 64 * 64) if rng.random() < 0.8 else max(16, d // 4 * 4)
            c.update(width=d, ff=int(d * rng.choice((2, 2.5, 3.5, 4))) // 4 * 4, layers=_log(rng, 1, 24))
            if net == "vit":
                c.update(context=rng.choice((50, 197, 257)), outputs=rng.choice((10, 1000)))
            elif net == "gpt":
                c.update(context=rng.choice((256, 1024)), outputs=rng.choice((256, 5000, 32768, 50257)))
            else:
                c.update(outputs=rng.choice((0, 4096, 32000)))
        c["wd"] = rng.choice((0.0, 0.01, 0.1))
        if opt in ("adafaclo", "elo") and rng.random() < 0.5:
            c["groups"] = 2
        if opt != "adafaclo" and opt != "velo":
            c["clip"] = rng.random() < 0.5
        if opt.endswith("celo2"):
            c["orthogonalize"] = rng.random() < 0.6
        w = work(c)
        n = sum(numel(s) for s in shapes_of(c))
        ragged = net == "conv" or any(len(s) == 2 and s[1] % 4 for s in shapes_of(c))
        if n >= 20000 and w["bytes"] <= most and w["flops"] <= most_flops[bool(c.get("orthogonalize"))] / (8 if ragged else 1) and not (ragged and n > 6e7):
            return c


def work(case):
    """Every input read once, every output written once; the network of each element with everything folded into the first
    layer that does not depend on the element, and the products of Newton-Schulz (symmetric ones counted half)."""
    opt = case["opt"]
    nbytes = flops = 0
    hidden = {"adafaclo": 2 * (16 * 32 + 32 * 32 + 32 * 2), "elo": 2 * (16 * 32 + 32 * 32 + 32 * 2),
              "celo2": 2 * (18 * 8 + 8 * 8 + 8 * 2), "elo_celo2": 2 * (18 * 8 + 8 * 8 + 8 * 2),
              "velo": 2 * (18 * 4 + 4 * 4 + 4 * 2)}[opt]
    shapes = shapes_of(case)
    for s in shapes:
        n = numel(s)
        if opt.endswith("celo2") and (len(s) < 2 or is_embedding(case, s)):
            nbytes += (28 if opt == "celo2" else 44) * n  # AdamW: own two moments, or the shared four
            flops += 20 * n
            continue
        nbytes += 44 * n  # reads gradient, parameter, three momenta, second moment; writes all but the gradient
        flops += (hidden + 60) * n
        if len(s) < 2:
            nbytes += (24 if opt == "velo" else 48) * n  # three (six) full-size accumulators
            continue
        big, small = sorted(s)[-1], sorted(s)[-2]
        nbytes += 24 * (n // big + n // small)
        if case.get("orthogonalize"):
            r, c = sorted(s[-2:])
            flops += 5 * (3 * r * r * c + r * r * r) * (n // (r * c))
    if opt == "velo":
        h, bank, t = 512, 256, len(shapes)
        nbytes += 4 * (8 * h * h + bank * (h + 159) + 60 * h) + 16 * t * h
        flops += 2 * t * (8 * h * h + bank * (h + 159) + 60 * h)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """fp32 throughout: sums over a tensor (or a row) in another order, and a network of fp32 products."""
    return {"rel": 1e-5, "max": 1e-4}


# ---------------------------------------------------------------------------------------------------------------------
# one user's program
# ---------------------------------------------------------------------------------------------------------------------


class Flat:
    """Tensors of the given shapes as views into one buffer."""

    def __init__(self, shapes, device):
        self.at, end = [], 0
        for s in shapes:
            self.at.append((end, s))
            end += -(-numel(s) // ALIGN) * ALIGN
        self.buffer = torch.zeros(end, device=device)

    def views(self):
        return [self.buffer[o:o + numel(s)].view(s) for o, s in self.at]


def gradients(case, shapes, gen, device):
    """iid entries; with outliers for VeLO; for CELO2 every row with a log-normal scale of its own."""
    flat = Flat(shapes, device)
    flat.buffer.normal_(generator=gen)
    if case["opt"] == "velo":
        flat.buffer.mul_(1e-3)
        flat.buffer[torch.rand(flat.buffer.shape, generator=gen, device=device) < 0.01] *= 100.0
    elif case["opt"] == "celo2":
        for g in flat.views():
            if g.dim() >= 2:
                g.mul_(torch.exp(torch.randn((g.shape[0],) + (1,) * (g.dim() - 1), generator=gen, device=device) - 7.0))
            else:
                g.mul_(1e-3)
    else:
        flat.buffer.mul_(1e-3)
    return flat


def optimizer(case, params, seed):
    opt, wd = case["opt"], case.get("wd", 0.0)
    groups = params
    if case.get("groups") == 2:
        groups = [{"params": [p for p in params if p.dim() >= 2], "weight_decay": wd},
                  {"params": [p for p in params if p.dim() < 2], "weight_decay": 0.0}]
    elif any(is_embedding(case, tuple(p.shape)) for p in params):
        groups = [{"params": [p for p in params if not is_embedding(case, tuple(p.shape))]},
                  {"params": [p for p in params if is_embedding(case, tuple(p.shape))], "is_embedding": True}]
    with torch.random.fork_rng(devices=[]):  # trained meta-weights come from a hub; here they are seeded draws
        torch.manual_seed(seed)
        if opt == "velo":
            rnn, mlp = models.VeLORNN(), models.VeLOMLP()
            with torch.no_grad():
                for name, w in mlp.named_parameters():
                    if "weights_" in name:
                        w.mul_(0.05)  # the bank is N(0, 1) by default and is multiplied by 100 when it is mixed
            return optim.VeLO_CUDA(groups, lr=1e-1, num_steps=100000, weight_decay=wd, rnn=rnn, mlp=mlp)
        net = models.CELO2MLP() if opt.endswith("celo2") else models.MetaMLP(39, 32, 1)
    if opt == "adafaclo":
        return optim.AdafacLO_CUDA(groups, lr=1.0, weight_decay=wd, network=net)
    if opt == "elo":
        return optim.ELO_CUDA(groups, lr=1e-3, weight_decay=wd, clip_grad=case.get("clip", False), network=net)
    cls = optim.CELO2_CUDA if opt == "celo2" else optim.ELO_CELO2_CUDA
    return cls(groups, lr=1e-3, weight_decay=wd, clip_grad=case.get("clip", False), orthogonalize=case["orthogonalize"], network=net)


def prepare(case, seed):
    device = torch.device("cuda")
    gen = torch.Generator(device=device).manual_seed(seed)
    shapes = shapes_of(case)
    flat = Flat(shapes, device)
    flat.buffer.normal_(generator=gen).mul_(0.02)
    params = [torch.nn.Parameter(v) for v in flat.views()]
    opt = optimizer(case, params, seed)
    loss = torch.full((), 2.5, device=device) if case["opt"] == "velo" else None
    for _ in range(2):  # the first steps of the run; the gradients of the second are also those of the passes below
        grads = gradients(case, shapes, gen, device)
        for p, g in zip(params, grads.views()):
            p.grad = g
        opt.step(loss)
    # the state moves into flat buffers, one per kind of tensor, through the checkpoint interface
    saved = opt.state_dict()
    kinds = {}
    for st in saved["state"].values():
        for key, x in st.items():
            if torch.is_tensor(x) and x.is_cuda and x.numel() and key != "rank_onehot":
                kinds.setdefault(key, []).append((st, tuple(x.shape)))
    out = {"params": flat.buffer}
    for key, owners in kinds.items():
        store = Flat([s for _, s in owners], device)
        for (st, _), view in zip(owners, store.views()):
            st[key] = view.copy_(st[key])
        out[key] = store.buffer
    opt.load_state_dict(saved)
    return {"opt": opt, "loss": loss, "out": out, "grads": grads}


def run(state):
    opt = state["opt"]
    opt.step(state["loss"])
    out = dict(state["out"])
    if state["loss"] is not None:
        out["lstm_h"], out["lstm_c"] = opt.lstm_hidden_state
        out["loss_means"], out["loss_min"] = opt.loss_buffer["means"], opt.loss_buffer["running_min"]
        out["loss_iteration"] = opt.loss_buffer["iteration"]
    return out
