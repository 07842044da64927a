"""Performance cases: what users of haste_b200 have it do, through `haste_b200`'s layer classes.

A case is one call of a layer (or of a `Stack` of layers):
  task "step"   one time step in evaluation mode, the state handed from call to call;
  task "infer"  whole sequences in evaluation mode, without gradients;
  task "train"  forward and backward, all gradients.
Zoneout and DropConnect masks are given explicitly (the layers' `zoneout_mask=` and
`dropconnect_mask=`), so that a pass is a function of the seed alone.
"""
import math

import torch

import haste_b200

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
GATES = {"LSTM": 4, "GRU": 3, "IndRNN": 1, "LayerNormLSTM": 4, "LayerNormGRU": 3,
         "LayerNormIndRNN": 1}


def _case(cell, task, dtype, T, N, C, H, layers=1, bidirectional=False, zoneout=0.0, dropout=0.0,
          batch_first=False, lengths=False, **name):
    return dict(cell=cell, task=task, dtype=dtype, T=T, N=N, C=C, H=H, layers=layers,
                bidirectional=bidirectional, zoneout=zoneout, dropout=dropout,
                batch_first=batch_first, lengths=lengths, **name)


def listed():
    return [
        # A recogniser or synthesiser that runs frame by frame: one stream, the lowest latency.
        _case("LSTM", "step", "fp32", 1, 1, 512, 512, name="step-lstm-n1"),
        # The same for a server that batches its streams, in reduced precision.
        _case("GRU", "step", "bf16", 1, 32, 256, 1024, name="step-gru-bf16-n32"),
        # One recording at a time (a corner of the benchmark grid, forward only).
        _case("GRU", "infer", "fp32", 1000, 1, 256, 256, name="infer-gru-n1"),
        # A batch of utterances of unequal length as a data loader hands it over: batch first,
        # final states taken at each row's own length, sizes that fit no tile.
        _case("LSTM", "infer", "fp32", 237, 19, 83, 320, batch_first=True, lengths=True,
              name="infer-lstm-ragged"),
        # The small training configuration (T=100, N=32, C=128, H=256).
        _case("LSTM", "train", "fp32", 100, 32, 128, 256, name="train-lstm-small"),
        # The headline benchmark: LSTM N=64, C=H=512, T=1000, forward and backward.
        _case("LSTM", "train", "fp32", 1000, 64, 512, 512, name="train-lstm-headline"),
        # Training on sizes that nobody rounded, with zoneout.
        _case("GRU", "train", "fp32", 333, 37, 161, 250, zoneout=0.1, name="train-gru-odd"),
        # A wide layer with DropConnect (the width of the 1024-unit configurations, one layer).
        _case("LSTM", "train", "fp32", 200, 32, 1024, 1024, dropout=0.05, name="train-lstm-wide"),
        # Layer-normalised LSTM, three bidirectional levels with both regularisers.
        _case("LayerNormLSTM", "train", "fp32", 100, 64, 80, 512, layers=3, bidirectional=True,
              zoneout=0.1, dropout=0.05, name="train-lnlstm-stack"),
        # Layer-normalised GRU in bfloat16.
        _case("LayerNormGRU", "train", "bf16", 200, 32, 256, 256, name="train-lngru-bf16"),
        # Six IndRNN layers over long sequences: time-parallel work and a memory-bound scan.
        _case("IndRNN", "train", "fp32", 2000, 128, 1024, 1024, layers=6, zoneout=0.1,
              name="train-indrnn-stack"),
        # Four bidirectional bfloat16 GRU levels, one GPU's share of the data-parallel workload.
        _case("GRU", "train", "bf16", 500, 128, 512, 1024, layers=4, bidirectional=True,
              name="train-gru-bf16-stack"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _width(rng, lo, hi):
    """A layer or input width: a multiple of 8 three times out of four, else as it falls."""
    w = _log_int(rng, lo, hi)
    return w if rng.random() < 0.25 else max(lo, w // 8 * 8)


def _draw_once(rng):
    kind = rng.choice(["step", "infer", "train", "train", "layer_norm", "indrnn", "stack"])
    if kind == "step":
        return _case(rng.choice(["LSTM", "GRU"]), "step", rng.choice(["fp32", "bf16"]), 1,
                     _log_int(rng, 1, 64), _width(rng, 64, 1024), _width(rng, 64, 1024))
    if kind == "infer":
        return _case(rng.choice(["LSTM", "GRU"]), "infer", rng.choice(["fp32", "fp32", "bf16"]),
                     _log_int(rng, 50, 1000), _log_int(rng, 1, 64), _width(rng, 64, 1024),
                     _width(rng, 64, 1024), batch_first=rng.random() < 0.5,
                     lengths=rng.random() < 0.5)
    if kind == "train":
        return _case(rng.choice(["LSTM", "GRU"]), "train", rng.choice(["fp32", "fp32", "bf16"]),
                     _log_int(rng, 50, 1000), _log_int(rng, 8, 128), _width(rng, 64, 1024),
                     _width(rng, 64, 1024), zoneout=rng.choice([0.0, 0.1]),
                     dropout=rng.choice([0.0, 0.05]))
    if kind == "layer_norm":
        cell, dtype = rng.choice(["LayerNormLSTM", "LayerNormGRU"]), rng.choice(["fp32", "bf16"])
        return _case(cell, "train", dtype, _log_int(rng, 50, 200), _log_int(rng, 8, 64),
                     _width(rng, 64, 512), _width(rng, 64, 512),
                     layers=rng.randint(1, 3) if dtype == "fp32" else 1,
                     bidirectional=rng.random() < 0.5, zoneout=rng.choice([0.0, 0.1]),
                     dropout=rng.choice([0.0, 0.05]))
    if kind == "indrnn":
        return _case(rng.choice(["IndRNN", "LayerNormIndRNN"]), "train", "fp32",
                     _log_int(rng, 200, 2000), _log_int(rng, 8, 128), _width(rng, 128, 1024),
                     _width(rng, 128, 1024), layers=rng.randint(1, 6),
                     zoneout=rng.choice([0.0, 0.1]))
    return _case(rng.choice(["LSTM", "GRU"]), "train", "bf16", _log_int(rng, 50, 500),
                 _log_int(rng, 16, 256), _width(rng, 128, 1024), _width(rng, 256, 1024),
                 layers=rng.randint(2, 4), bidirectional=True)


def draw(rng):
    # no more arithmetic than the largest listed case, and no more dependent steps than it
    # would take at the pace of the slowest cell
    most = max(work(c)["flops"] for c in listed())
    while True:
        case = _draw_once(rng)
        stack_steps = case["T"] * case["layers"] if case["bidirectional"] else 0
        if work(case)["flops"] <= most and stack_steps <= 800:
            return case


def _layers_of(net):
    return [l for level in net.layers for l in level] if isinstance(net, haste_b200.Stack) else [net]


def _fill(layer, gen):
    """Weights as an initialised or lightly trained layer has them, from `gen`."""
    H = layer.hidden_size
    for name, p in layer.named_parameters():
        if name == "kernel":
            p.normal_(0.0, math.sqrt(2.0 / (p.shape[0] + H)), generator=gen)
        elif name == "recurrent_kernel":
            p.normal_(0.0, 1.0 / math.sqrt(H), generator=gen)
        elif name == "recurrent_scale":
            p.uniform_(0.0, 1.0, generator=gen)
        elif name == "gamma":
            p.uniform_(0.8, 1.2, generator=gen)
            p[1].mul_(0.25)  # the recurrent gain below the input's, where training keeps it
        elif name == "gamma_h":
            p.uniform_(0.8, 1.2, generator=gen)
        else:  # biases, beta_h
            p.uniform_(-0.1, 0.1, generator=gen)
            if name == "bias" and hasattr(layer, "forget_bias"):
                p[2 * H:3 * H].add_(layer.forget_bias)


def prepare(case, seed):
    dtype, dev = DTYPES[case["dtype"]], torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    T, N, C, H = case["T"], case["N"], case["C"], case["H"]
    cell = getattr(haste_b200, case["cell"])
    opts = {}
    if case["zoneout"]:
        opts["zoneout"] = case["zoneout"]
    if case["dropout"]:
        opts["dropout"] = case["dropout"]
    dirs = 2 if case["bidirectional"] else 1
    stacked = case["layers"] > 1 or dirs > 1
    with torch.device("meta"):  # the constructor's own initialisation is replaced by _fill
        if stacked:
            net = haste_b200.Stack(cell, C, H, num_layers=case["layers"],
                                   bidirectional=case["bidirectional"], **opts)
        else:
            net = cell(C, H, batch_first=case["batch_first"], **opts)
    net = net.to_empty(device=dev).to(dtype)

    def normal(*shape):
        return torch.randn(*shape, device=dev, generator=gen).to(dtype)

    with torch.no_grad():
        for layer in _layers_of(net):
            _fill(layer, gen)
    net.train(case["task"] == "train")
    s = {"net": net, "task": case["task"], "stacked": stacked, "kw": {}}
    s["x"] = normal(N, T, C) if case["batch_first"] else normal(T, N, C)
    if case["task"] == "step":
        s["state"] = normal(1, N, H).tanh()
        if case["cell"].endswith("LSTM"):
            s["state"] = (s["state"], normal(1, N, H))
        s["kw"]["state"] = s["state"]
    if case["lengths"]:
        s["kw"]["lengths"] = torch.randint(max(1, T // 2), T + 1, (N,), device=dev, generator=gen)
    if case["task"] != "train":
        return s

    s["x"].requires_grad_(True)
    s["dy"] = normal(T, N, dirs * H)
    s["params"] = list(net.parameters())
    masks = []
    for layer in _layers_of(net):
        m = {}
        if case["zoneout"]:
            m["zoneout_mask"] = torch.empty(T, N, H, device=dev, dtype=dtype).bernoulli_(
                1.0 - case["zoneout"], generator=gen)
        if case["dropout"]:
            m["dropconnect_mask"] = torch.empty(
                H, layer.recurrent_kernel.shape[1], device=dev, dtype=dtype).bernoulli_(
                    1.0 - case["dropout"], generator=gen)
        masks.append(m)
    if stacked:
        s["kw"]["masks"] = [masks[i:i + dirs] for i in range(0, len(masks), dirs)]
    else:
        s["kw"] = masks[0]
    return s


def run(s):
    net, x = s["net"], s["x"]
    if s["task"] != "train":
        with torch.no_grad():
            return net(x, **s["kw"])  # output and final state
    y = net(x, **s["kw"])
    out = [y]
    if not s["stacked"]:
        y, state = y
        out = [y, state]
    return out + list(torch.autograd.grad(y, [x] + s["params"], s["dy"]))


def work(case):
    T, N, H, G = case["T"], case["N"], case["H"], GATES[case["cell"]]
    size = 4 if case["dtype"] == "fp32" else 2
    dirs = 2 if case["bidirectional"] else 1
    train = case["task"] == "train"
    values = macs = 0.0
    C = case["C"]
    for level in range(case["layers"]):
        for _ in range(dirs):
            recurrent = H * G * H if G > 1 else H
            weights = C * G * H + recurrent + G * H
            values += weights * (2 if train else 1)  # read; their gradients written
            macs += T * N * (C * G * H + recurrent)
            if train and case["zoneout"]:
                values += T * N * H
            if train and case["dropout"] and G > 1:
                values += recurrent
        C = dirs * H
    # the network's input and output, and in training the gradients of both
    values += (T * N * case["C"] + T * N * dirs * H) * (2 if train else 1)
    if case["task"] == "step":
        values += N * H * (4 if case["cell"].endswith("LSTM") else 2)
    return {"bytes": values * size, "flops": 2.0 * macs * (3 if train else 1)}


def tolerance(case):
    # fp32: sums of 16-bit plane products and fast gate functions, carried through the whole
    # sequence; bf16: every state and activation is rounded to 8 bits on the way.
    return {"rel": 1e-4} if case["dtype"] == "fp32" else {"rel": 1e-2}
