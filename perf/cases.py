"""The work a user has this package do, as a list of timed cases.

A DLR-Net replaces the MLP of every layer of a locked decoder, so its forward runs once per layer for every decode
step (a few rows) and for every prompt (thousands of rows), over the widths, ranks and depths of
``registry.MODEL_CONFIGS``.  It is reached through the module (``DLRNet.forward``), through packed weights
(``PackedNet``, what a serving process holds) and, when weights come in, through ``pack_state_dict``.

Weights follow the initialisation of the module (V ~ N(0, 1/d), U ~ N(0, 1/(r L))) with gains around 1 and layer scales
around 0.3, so that a forward moves the activations by a good part of themselves; inputs are N(0, 1) rows.  Everything
is made on the GPU from the seed.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "ml-dlr-lock_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import dlr_lock_b200 as D  # noqa: E402

MODELS = {name: (c["d"], c["d_ff"], c["r"]) for name, c in D.registry.MODEL_CONFIGS.items()}
SMALL, MEDIUM, LARGE, WIDEST = MODELS          # widths 1024, 2048, 4096, 5120 with ranks 32, 64, 128, 256


def _case(name, model, call, batch, seq, nets=1, multiplier=1.0):
    return {"name": name, "model": model, "call": call, "batch": batch, "seq": seq, "nets": nets, "multiplier": multiplier}


def listed():
    return [
        # One user, one token: a single net of the small model on one row, through the module.  The smallest call.
        _case("module d1024 1 row", SMALL, "module", 1, 1),
        # A decode step of the whole small model at batch 8: its 28 nets one after the other (517 MB of weights).
        _case("28 modules d1024 8 rows", SMALL, "module", 8, 1, nets=28),
        # The prompt of that batch: 8 sequences of 512 tokens through one net.
        _case("module d1024 8x512 rows", SMALL, "module", 8, 512),
        # Decode of the medium model for a few users.
        _case("packed d2048 4 rows", MEDIUM, "packed", 4, 1),
        # A prompt of an ordinary, ragged length on the medium model.
        _case("packed d2048 333 rows", MEDIUM, "packed", 1, 333),
        # Decode of the large model: one user, a small batch, a full batch.
        _case("packed d4096 1 row", LARGE, "packed", 1, 1),
        _case("packed d4096 16 rows", LARGE, "packed", 16, 1),
        _case("packed d4096 64 rows", LARGE, "packed", 64, 1),
        # Prompts of the large model: a ragged one, and the largest batch (the benchmark's headline).
        _case("packed d4096 1000 rows", LARGE, "packed", 1, 1000),
        _case("packed d4096 8192 rows", LARGE, "packed", 4, 2048),
        # The widest model with the highest rank: a prompt batch.
        _case("packed d5120 4096 rows", WIDEST, "packed", 2, 2048),
        # Weights coming in: the state dict of a net into folded stacks.
        _case("pack d2048", MEDIUM, "pack", 1, 1),
    ]


def _depth(case):
    d, d_ff, r = MODELS[case["model"]]
    return D.compute_depth(d, d_ff, r, case["multiplier"])


def _flops(case):
    d, _, r = MODELS[case["model"]]
    return 4.0 * case["nets"] * _depth(case) * case["batch"] * case["seq"] * d * r


def draw(rng):
    """Any model, rows from 1 to 8192 spread over their logarithm (decode batches and prompts of any length), the three
    ways in, and nets of half the depth (the ``multiplier`` of ``build_locked_model``)."""
    largest = max(_flops(c) for c in listed())
    while True:
        model = rng.choice(list(MODELS))
        call = rng.choice(["packed"] * 5 + ["module"] * 2 + ["pack"])
        rows = 1 if call == "pack" else int(round(2.0 ** rng.uniform(0.0, 13.0)))
        batch, seq = (rows, 1) if rows <= 64 else (1, rows)
        multiplier = rng.choice([1.0, 1.0, 1.0, 0.5]) if call != "pack" else round(rng.uniform(0.3, 1.0), 2)
        c = _case("", model, call, batch, seq, multiplier=multiplier)
        del c["name"]
        if _flops(c) <= largest:
            return c


def _module(d, r, depth, gen, device):
    with torch.device(device):
        net = D.DLRNet(d, r, depth)
        for p in net.parameters():
            p.requires_grad_(False)
        u_scale = 1.0 / math.sqrt(r * depth)
        for i in range(depth):
            net.Vs[i].normal_(0.0, 1.0 / math.sqrt(d), generator=gen)
            net.Us[i].normal_(0.0, u_scale, generator=gen)
            net.rms_w[i].normal_(1.0, 0.1, generator=gen)
            net.alphas[i].uniform_(0.2, 0.4, generator=gen)
    return net.to(torch.bfloat16).eval()


def _packed(d, r, depth, gen, device):
    kw = dict(device=device, dtype=torch.bfloat16)
    V = torch.empty(depth, r, d, **kw).normal_(0.0, 1.0 / math.sqrt(d), generator=gen)
    U = torch.empty(depth, d, r, **kw).normal_(0.0, 1.0 / math.sqrt(r * depth), generator=gen)
    gain = torch.empty(depth, d, **kw).normal_(1.0, 0.1, generator=gen)
    alpha = torch.empty(depth, **kw).uniform_(0.2, 0.4, generator=gen)
    return D.PackedNet(*D.ops.fold_weights(V, U, gain, alpha))


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    d, _, r = MODELS[case["model"]]
    depth = _depth(case)
    make = _packed if case["call"] == "packed" else _module
    nets = [make(d, r, depth, gen, device) for _ in range(case["nets"])]
    x = torch.empty(case["batch"], case["seq"], d, device=device, dtype=torch.bfloat16).normal_(generator=gen)
    if case["call"] == "pack":
        return {"call": "pack", "weights": {k: v.clone() for k, v in nets[0].state_dict().items()}, "device": device}
    return {"call": case["call"], "nets": nets, "x": x}


@torch.no_grad()
def run(state):
    if state["call"] == "pack":
        net = D.pack_state_dict(state["weights"], state["device"])
        return net.Vp, net.Up
    h = state["x"]
    for net in state["nets"]:
        h = net(h)
    return h


def work(case):
    d, _, r = MODELS[case["model"]]
    depth = _depth(case)
    weights = 4 * depth * d * r                                    # V and U in bf16
    if case["call"] == "pack":
        return {"bytes": 2 * weights + 2 * depth * (d + 1), "flops": 2 * depth * d * r}
    rows = case["batch"] * case["seq"]
    return {"bytes": case["nets"] * weights + 4 * rows * d, "flops": _flops(case)}


def tolerance(case):
    # bf16 in and out, sums in fp32; each of the ~140 layers rounds its matrix operands to bf16.  Beyond 64 rows an
    # implementation may also carry the activations between layers in bf16, as the torch module does, or in fp32: those
    # two differ by the ~140 roundings of the activations (2e-2 of the result, as measured between the two kinds)
    if case["call"] == "pack":
        return "exact"
    return {"rel": 1e-2 if case["batch"] * case["seq"] <= 64 else 2.5e-2}
