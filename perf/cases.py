"""Performance cases of bats_gb300: what its users run, through its public entry points.

A case is a dict of plain values. prepare() makes its inputs on the GPU from the seed alone and builds what a
program keeps between calls (the network, the train step with its CUDA graph, the server); run() is one call;
exact() restates the call in 64 bits with torch, without this package.

Training cases use a small learning rate (late in a schedule), so that a step repeated on the same state keeps
doing the same work. The train steps run with their default plan: the optional autotuner picks from timings,
which differ between runs and, through the order of the gradient's partial sums, in the last bits of the results.
"""
import math

import numpy as np
import torch

TAU_S = 0.13
LR = 1e-5
TARGETS = (15.0, 3.0)
MAX_SIM = 0.2


# -- cases ------------------------------------------------------------------------------------------------------------

def _fc(name, kind, batch, sizes, k_in, events, spread, window, weights, theta, k):
    """A fully-connected case. events: mean (spread 0) or median input events of a sample, spread: sigma of their
    logarithm over the batch; weights: "uniform" U(-1, 1) (the reference's MNIST training, every layer spikes),
    "normal" N(0, 1/sqrt(fan_in)) (hidden layers nearly silent) or "positive" N(1.5, 1)/sqrt(fan_in) (the serving
    network's: strongly driven neurons); theta: of the hidden layers (the last one: 1.3)."""
    return {"name": name, "kind": kind, "batch": batch, "sizes": sizes, "k_in": k_in, "events": events,
            "spread": spread, "window": window, "weights": weights, "theta": theta, "k": k}


def _conv(name, kind, batch, shape, events, c1, f1, c2, f2, fc, k):
    """A convolutional case: (X, Y, C) input, conv f1 x f1 x c1 -> 2x2 pool -> conv f2 x f2 x c2, then (kind
    "conv_train") pool -> fc -> 10."""
    return {"name": name, "kind": kind, "batch": batch, "shape": shape, "events": events, "c1": c1, "f1": f1,
            "c2": c2, "f2": f2, "fc": fc, "k": k}


def _serve(name, requests, sizes, lo, hi):
    return {"name": name, "kind": "serve", "requests": requests, "sizes": sizes, "lo": lo, "hi": hi, "k": 30}


def listed():
    return [
        # The benchmark's train step: MNIST-shaped single-spike input, every layer spikes.
        _fc("train_mnist", "train", 256, "784-800-800-10", 1, 149, 0.0, 0.01, "uniform", 0.2, 30),
        # The same step on the configuration's literal constants: silent hidden layers, launches and screens.
        _fc("train_quiet", "train", 256, "784-800-800-10", 1, 149, 0.0, 0.01, "normal", 1.0, 30),
        # Uneven event streams (20 to 4000 events a sample) in one large batch: the largest case.
        _fc("train_uneven", "train", 4096, "1024-1024-20", 16, 200, 1.0, 0.1, "uniform", 0.2, 30),
        # A small batch of a small network: launches and latency.
        _fc("train_small", "train", 8, "784-800-10", 1, 149, 0.0, 0.01, "uniform", 0.2, 30),
        # Odd sizes, several spikes per input, K 20.
        _fc("train_ragged", "train", 77, "333-517-131-11", 3, 190, 0.5, 0.05, "uniform", 0.2, 20),
        # The reference's MNIST training iteration through the layer classes: host input, per-sample gradients.
        _fc("api_mnist", "api", 50, "784-800-10", 1, 149, 0.0, 0.01, "uniform", 0.2, 30),
        # One wide layer behind torch.autograd: times, gradients of weights and of input times.
        _fc("grad_wide", "grad", 256, "800-800", 6, 650, 0.3, 0.1, "positive", 1.0, 30),
        # A narrow output layer fed by a hidden layer's many spikes, K at its default.
        _fc("grad_narrow", "grad", 256, "800-32", 30, 2400, 0.3, 0.2, "positive", 1.3, 32),
        # The reference's MNIST convolutional network.
        _conv("conv_train", "conv_train", 128, "28-28-1", 149, 15, 5, 40, 5, 300, 10),
        # Conv layers alone through the layer classes, odd sizes.
        _conv("conv_block", "conv_block", 21, "23-17-2", 150, 9, 5, 24, 3, 0, 10),
        # One inference request, and a burst of them.
        _serve("serve_one", 1, "700-512-512-20", 500, 500),
        _serve("serve_burst", 256, "700-512-512-20", 50, 5000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "api", "grad", "grad", "conv_train", "conv_block", "serve"])
    if kind == "serve":
        lo = _log(rng, 30, 800)
        c = _serve("", _log(rng, 1, 256), "700-%d-%d" % (_log(rng, 64, 600), rng.randint(2, 40)), lo,
                   min(5000, lo * rng.randint(1, 20)))
    elif kind.startswith("conv"):
        x, y, ch = rng.randint(12, 28), rng.randint(12, 28), rng.randint(1, 3)
        c = _conv("", kind, _log(rng, 4, 128), "%d-%d-%d" % (x, y, ch), rng.randint(40, 160), rng.randint(4, 15),
                  rng.choice([3, 5]), rng.randint(8, 40), 3, _log(rng, 32, 300) if kind == "conv_train" else 0,
                  rng.choice([5, 10]))
    else:
        n_in, k_in = _log(rng, 60, 1100), rng.choice([1, 1, 2, 4, 8])
        sizes = [n_in] + [_log(rng, 48, 1100) for _ in range(1 if kind == "grad" else rng.choice([0, 1, 1, 2]))]
        if kind != "grad":
            sizes.append(rng.randint(2, 40))
        most = {"train": 1024, "api": 100, "grad": 512}[kind]
        batch = max(1, min(_log(rng, 4, most), int(2.0e8 / max(a * b for a, b in zip(sizes[:-1], sizes[1:])))))
        events = _log(rng, 20, max(21, min(700, int(0.4 * n_in * k_in))))
        weights = rng.choice(["uniform", "positive"] if kind == "grad" else ["uniform", "uniform", "normal"])
        c = _fc("", kind, batch, "-".join(map(str, sizes)), k_in, events, 0.0 if k_in == 1 else rng.choice([0.3, 0.8]),
                0.01 if k_in == 1 else rng.choice([0.05, 0.1, 0.2]), weights, 0.2 if weights == "uniform" else 1.0,
                rng.choice([10, 20, 30, 32]))
    del c["name"]
    return c


# -- inputs, from the seed alone --------------------------------------------------------------------------------------

def _ints(text):
    return [int(v) for v in text.split("-")]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _trains(case, n_in, k_in, g):
    """Spike trains (batch, n_in, k_in), +inf past a neuron's spikes, and their counts. k_in 1: every input fires
    once with the same probability; else events on uniform channels, lognormal numbers of them, capped at k_in."""
    B, win = case["batch"], case.get("window", 0.01)
    if k_in == 1:
        fire = torch.rand((B, n_in), generator=g, device="cuda") < case["events"] / n_in
        t = torch.rand((B, n_in), generator=g, device="cuda") * win
        t = torch.where(fire, t, torch.full_like(t, math.inf))[:, :, None].contiguous()
        return t, fire.to(torch.int32)
    e = torch.randn(B, generator=g, device="cuda") * case["spread"]
    m = (case["events"] * e.exp()).round().clamp(max(1, case["events"] // 10), 20 * case["events"]).long()
    total = int(m.sum())
    b = torch.repeat_interleave(torch.arange(B, device="cuda"), m, output_size=total)
    ch = torch.randint(0, n_in, (total,), generator=g, device="cuda")
    t = torch.rand(total, generator=g, device="cuda") * win
    o = torch.argsort(t)
    key = (b * n_in + ch)[o]
    o2 = torch.argsort(key, stable=True)
    key, t = key[o2], t[o][o2]
    first = torch.searchsorted(key, key)
    slot = torch.arange(total, device="cuda") - first
    keep = slot < k_in
    out = torch.full((B * n_in, k_in), math.inf, device="cuda")
    out[key[keep], slot[keep]] = t[keep]
    out = out.reshape(B, n_in, k_in)
    return out, torch.isfinite(out).sum(2).to(torch.int32)


def _fc_data(case, seed):
    g = _gen(seed)
    sizes = _ints(case["sizes"])
    ws = []
    for i, o in zip(sizes[:-1], sizes[1:]):
        if case["weights"] == "uniform":
            ws.append(torch.rand((o, i), generator=g, device="cuda") * 2 - 1)
        else:
            mean = 1.5 if case["weights"] == "positive" else 0.0
            ws.append((torch.randn((o, i), generator=g, device="cuda") + mean) / math.sqrt(i))
    t, n = _trains(case, sizes[0], case["k_in"], g)
    labels = torch.randint(0, sizes[-1], (case["batch"],), generator=g, device="cuda", dtype=torch.int32)
    thetas = [case["theta"]] * (len(ws) - 1) + [1.3 if len(ws) > 1 else case["theta"]]
    return ws, thetas, t, n, labels, g


def _conv_data(case, seed):
    g = _gen(seed)
    X, Y, C = _ints(case["shape"])
    u = lambda *s: torch.rand(s, generator=g, device="cuda") * 2 - 1  # noqa: E731
    w1, w2 = u(case["c1"], case["f1"], case["f1"], C), u(case["c2"], case["f2"], case["f2"], case["c1"])
    x, y = ((v - case["f1"] + 1) // 2 - case["f2"] + 1 for v in (X, Y))
    fcs = [u(case["fc"], (x // 2) * (y // 2) * case["c2"]), u(10, case["fc"])] if case["fc"] else []
    t, n = _trains(case, X * Y * C, 1, g)
    labels = torch.randint(0, 10, (case["batch"],), generator=g, device="cuda", dtype=torch.int32)
    err = torch.randn((case["batch"], x * y * case["c2"], case["k"]), generator=g, device="cuda")
    return w1, w2, fcs, t, n, labels, err


CONV_THETAS = (0.04, 0.8, 0.6, 0.3)


def _serve_data(case, seed):
    rng = np.random.default_rng(seed)
    sizes = _ints(case["sizes"])
    ws = [((rng.standard_normal((o, i)) + 1.5) / math.sqrt(i)).astype(np.float32) for i, o in zip(sizes[:-1], sizes[1:])]
    reqs = []
    for _ in range(case["requests"]):
        m = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 1e-9)))))
        reqs.append((rng.integers(0, sizes[0], m).astype(np.int32), np.sort(rng.uniform(0, 0.2, m)).astype(np.float32)))
    return ws, [1.0] * (len(ws) - 1) + [1.3], reqs


# -- what a program keeps, and one call -------------------------------------------------------------------------------

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_train(case, seed):
    from bats_gb300.train import FCLayerSpec, FCTrainStep
    ws, thetas, t, _, labels, _ = _fc_data(case, seed)
    specs = [FCLayerSpec(w.shape[0], TAU_S, th, th, case["k"]) for w, th in zip(ws, thetas)]
    ts = FCTrainStep(case["batch"], t.shape[1], t.shape[2], specs, ws, *TARGETS, learning_rate=LR,
                     max_simulation=MAX_SIM)
    if not ts.try_capture():  # on empty inputs: no spike, no gradient, the weights stay as they are
        raise RuntimeError("capture failed: %s" % ts.capture_error)
    ts.set_inputs(t, labels)
    return {"run": _run_train, "ts": ts}


def _run_train(state):
    ts = state["ts"]
    ts.run()
    return {"loss": ts.loss, "counts": [o[0] for o in ts.out], "times": ts.out[-1][3], "grad": ts.grad, "w": ts.W,
            "m": ts.m, "v": ts.v}


def _prepare_api(case, seed):
    from bats_gb300 import Network, SpikeCountClassLoss
    from bats_gb300.Layers import InputLayer, LIFLayer
    from bats_gb300.Optimizers import AdamOptimizer
    ws, thetas, t, n, labels, _ = _fc_data(case, seed)
    net = Network()
    prev = InputLayer(n_neurons=t.shape[1], name="in")
    net.add_layer(prev, input=True)
    for i, (w, th) in enumerate(zip(ws, thetas)):
        prev = LIFLayer(prev, n_neurons=w.shape[0], tau_s=TAU_S, theta=th, delta_theta=th,
                        weight_initializer=lambda a, b, w=w: w.clone(), max_n_spike=case["k"], name="l%d" % i)
        net.add_layer(prev)
    return {"run": _run_api, "net": net, "loss": SpikeCountClassLoss(*TARGETS), "opt": AdamOptimizer(learning_rate=LR),
            "t": t.cpu().numpy(), "n": n.cpu().numpy(), "labels": labels}


def _run_api(state):
    net = state["net"]
    net.reset()
    net.forward(state["t"], state["n"], max_simulation=MAX_SIM, training=True)
    times, counts = net.output_spike_trains
    loss, errors = state["loss"].compute_loss_and_errors(times, counts, state["labels"])
    grads = [None if g is None else g.mean(0) for g in net.backward(errors)]
    net.apply_deltas(state["opt"].step(grads))
    return {"loss": loss, "counts": [x.spike_trains[1] for x in net.layers[1:]], "times": times, "grad": grads[1:],
            "w": [x.weights for x in net.layers[1:]]}


def _prepare_grad(case, seed):
    ws, thetas, t, _, _, g = _fc_data(case, seed)
    coef = torch.randn((case["batch"], ws[0].shape[0], case["k"]), generator=g, device="cuda")
    return {"run": _run_grad, "x": t.requires_grad_(), "w": ws[0].requires_grad_(), "theta": thetas[0], "coef": coef,
            "k": case["k"]}


def _run_grad(state):
    from bats_gb300.autograd import lif_fc
    times, counts = lif_fc(state["x"], state["w"], TAU_S, state["theta"], state["theta"], state["k"], MAX_SIM)
    loss = (torch.where(torch.isfinite(times), times, torch.zeros_like(times)) * state["coef"]).sum()
    gw, gx = torch.autograd.grad(loss, [state["w"], state["x"]])
    return {"counts": counts, "times": times.detach(), "gw": gw, "gx": gx}


def _prepare_conv_train(case, seed):
    from bats_gb300.conv_train import ConvLayerSpec, ConvTrainStep, PoolLayerSpec
    from bats_gb300.train import FCLayerSpec
    w1, w2, fcs, t, _, labels, _ = _conv_data(case, seed)
    k, th = case["k"], CONV_THETAS
    specs = [ConvLayerSpec((case["f1"], case["f1"], case["c1"]), TAU_S, th[0], th[0], k), PoolLayerSpec(),
             ConvLayerSpec((case["f2"], case["f2"], case["c2"]), TAU_S, th[1], th[1], k), PoolLayerSpec(),
             FCLayerSpec(case["fc"], TAU_S, th[2], th[2], k), FCLayerSpec(10, TAU_S, th[3], th[3], k)]
    ts = ConvTrainStep(case["batch"], _ints(case["shape"]), 1, specs, [w1, None, w2, None, *fcs], *TARGETS,
                       learning_rate=LR, max_simulation=MAX_SIM)
    if not ts.try_capture():
        raise RuntimeError("capture failed: %s" % ts.capture_error)
    ts.set_inputs(t, labels)
    return {"run": _run_conv_train, "ts": ts}


def _run_conv_train(state):
    ts = state["ts"]
    ts.replay()
    held = [d for d in ts.L if d["kind"] != "pool"]
    return {"loss": ts.loss, "counts": [d["out"][0] for d in ts.L], "times": ts.L[-1]["out"][3],
            "grad": [d["grad"] for d in held], "w": [d["W"] for d in held], "m": [d["m"] for d in held],
            "v": [d["v"] for d in held]}


def _prepare_conv_block(case, seed):
    from bats_gb300 import Network
    from bats_gb300.Layers import ConvInputLayer, ConvLIFLayer, PoolingLayer
    w1, w2, _, t, n, _, err = _conv_data(case, seed)
    net = Network()
    inp = ConvInputLayer(neurons_shape=np.array(_ints(case["shape"])), name="in")
    net.add_layer(inp, input=True)
    c1 = ConvLIFLayer(inp, filters_shape=np.array([case["f1"], case["f1"], case["c1"]]), tau_s=TAU_S,
                      theta=CONV_THETAS[0], delta_theta=CONV_THETAS[0], weight_initializer=lambda *a: w1,
                      max_n_spike=case["k"], name="conv1")
    pool = PoolingLayer(c1, name="pool1")
    c2 = ConvLIFLayer(pool, filters_shape=np.array([case["f2"], case["f2"], case["c2"]]), tau_s=TAU_S,
                      theta=CONV_THETAS[1], delta_theta=CONV_THETAS[1], weight_initializer=lambda *a: w2,
                      max_n_spike=case["k"], name="conv2")
    for layer in (c1, pool, c2):
        net.add_layer(layer)
    return {"run": _run_conv_block, "net": net, "t": t, "n": n, "err": err}


def _run_conv_block(state):
    net = state["net"]
    net.reset()
    net.forward(state["t"], state["n"], max_simulation=MAX_SIM, training=True)
    times, counts = net.output_spike_trains
    grads = net.backward(state["err"].clone())  # the reset errors are added to a loss's errors in place
    return {"counts": [x.spike_trains[1] for x in net.layers[1:]], "times": times, "grad1": grads[1], "grad2": grads[3]}


def _prepare_serve(case, seed):
    from bats_gb300.serving import InferenceServer, LayerSpec, Request
    ws, thetas, reqs = _serve_data(case, seed)
    specs = [LayerSpec(w.shape[0], TAU_S, th, th, case["k"]) for w, th in zip(ws, thetas)]
    server = InferenceServer(ws, specs, ws[0].shape[1], max_events=5001)
    return {"run": _run_serve, "server": server, "reqs": [Request(i, c, t) for i, (c, t) in enumerate(reqs)]}


def _run_serve(state):
    results = state["server"].infer(state["reqs"])
    return {"counts": np.stack([r.counts for r in results]), "times": np.stack([r.spike_times for r in results])}


_PREPARE = {"train": _prepare_train, "api": _prepare_api, "grad": _prepare_grad, "conv_train": _prepare_conv_train,
            "conv_block": _prepare_conv_block, "serve": _prepare_serve}


# -- the least work ---------------------------------------------------------------------------------------------------

def work(case):
    """Bytes: inputs, weights (for a training step with its optimizer state, read and written) and the arrays that
    come back; operations: two multiply-adds per (input event, first-layer neuron), again for each gradient. The
    spikes of the hidden layers, which only the run gives, are left out."""
    if case["kind"] == "serve":
        sizes = _ints(case["sizes"])
        events = case["requests"] * math.sqrt(case["lo"] * case["hi"])
        return {"bytes": 8 * events + 4 * sum(a * b for a, b in zip(sizes[:-1], sizes[1:]))
                + 4 * case["requests"] * sizes[-1] * (1 + case["k"]), "flops": 4 * events * sizes[1]}
    B, k = case["batch"], case["k"]
    if case["kind"].startswith("conv"):
        X, Y, C = _ints(case["shape"])
        f1, f2, c1, c2 = case["f1"], case["f2"], case["c1"], case["c2"]
        taps = f1 * f1 * c1
        x2, y2 = (X - f1 + 1) // 2 - f2 + 1, (Y - f1 + 1) // 2 - f2 + 1
        filters = taps * C + f2 * f2 * c1 * c2
        fc = case["fc"] * ((x2 // 2) * (y2 // 2) * c2 + 10)
        size = 4 * B * (X * Y * C + 3 * k * x2 * y2 * c2)
        size += 4 * (1 + B) * filters if case["kind"] == "conv_block" else 28 * (filters + fc)
        return {"bytes": size, "flops": 8 * B * case["events"] * taps}
    sizes = _ints(case["sizes"])
    weights = sum(a * b for a, b in zip(sizes[:-1], sizes[1:]))
    events = case["events"] * math.exp(case["spread"] ** 2 / 2)
    size = 4 * B * sizes[0] * case["k_in"] * (2 if case["kind"] == "grad" else 1) + 4 * B * sizes[-1] * (1 + k)
    size += (8 if case["kind"] == "grad" else 28) * weights
    return {"bytes": size, "flops": (12 if case["kind"] == "grad" else 8) * B * events * sizes[1]}


# -- the same calls in 64 bits ----------------------------------------------------------------------------------------

def _sorted(times):
    """Events of every sample in time order: times (+inf past the last), source slots, counts."""
    flat = times.double().reshape(times.shape[0], -1)
    t, idx = torch.sort(flat, dim=1, stable=True)
    n = torch.isfinite(t).sum(1)
    most = int(n.max()) if n.numel() else 0
    return t[:, :most].contiguous(), idx[:, :most].contiguous(), n


def _forward64(times, W, theta, K, max_sim):
    """One LIF layer: counts (B, M), and a, x, t, z (B, M, K) of its spikes, +inf past the counts."""
    tau_s, tau = TAU_S, 2 * TAU_S
    c = dtt = theta / tau
    t, idx, E = _sorted(times)
    j = idx // times.shape[2]
    Wt = W.double().t().contiguous()
    B, M, T = times.shape[0], W.shape[0], t.shape[1]
    a, b = torch.zeros((2, B, M), dtype=torch.float64, device=W.device)
    n = torch.zeros((B, M), dtype=torch.int64, device=W.device)
    out = torch.full((4, B, M, K), math.inf, dtype=torch.float64, device=W.device)
    tf = torch.where(torch.isfinite(t), t, torch.zeros_like(t))
    es, ee = (tf / tau_s).exp(), (tf / tau).exp()
    end = torch.cat([t, torch.full((B, 1), math.inf, dtype=torch.float64, device=W.device)], 1).clamp(max=max_sim)
    for m in range(T):
        act = (m < E)[:, None]
        w = Wt[j[:, m]] * act
        a = a + w * es[:, m, None]
        b = b + w * ee[:, m, None]
        live, last, stop = act & (n < K), t[:, m, None].expand(B, M), end[:, m + 1, None]
        while True:
            d = b * b - 4 * a * c
            x = d.sqrt()  # NaN where negative: every comparison below is false
            z = 2 * a / (x + b)
            s = tau * z.log()
            ok = live & (s > last) & (s <= stop)
            hit = ok.nonzero(as_tuple=True)
            if hit[0].numel() == 0:
                break
            for q, v in enumerate((a, x, s, z)):
                out[q][hit[0], hit[1], n[hit]] = v[hit]
            b = torch.where(ok, b - dtt * z, b)
            last = torch.where(ok, s, last)
            n = n + ok
            live = ok & (n < K)
    return n, out


def _backward64(times, W, theta, n, out, err, per_sample=False):
    """Sum over the batch (or each sample's) of the weight gradient, and the errors of the input spikes."""
    tau_s, tau = TAU_S, 2 * TAU_S
    c = dtt = theta / tau
    a, x, t, z = out
    B, M, K = t.shape
    valid = torch.arange(K, device=t.device) < n[:, :, None]
    one = torch.ones_like(t)
    a, x, z = (torch.where(valid, v, one) for v in (a, x, z))
    e = torch.where(valid, err.double(), 0 * one)
    cum = torch.zeros((B, M), dtype=torch.float64, device=t.device)
    for k in reversed(range(K)):
        e[:, :, k] = torch.where(valid[:, :, k], e[:, :, k] + cum * z[:, :, k], e[:, :, k])
        cum = cum + torch.where(valid[:, :, k], e[:, :, k] * dtt / x[:, :, k], 0 * cum)
    tabs = []
    for f in (tau / a * (1 + z * c / x), tau / x):
        s = torch.flip(torch.cumsum(torch.flip(e * f * valid, [2]), 2), [2])
        tabs.append(torch.cat([s, torch.zeros((B, M, 1), dtype=torch.float64, device=t.device)], 2))
    te, idx, E = _sorted(times)
    Kp, W = times.shape[2], W.double()
    G = torch.zeros((B if per_sample else 1, M, W.shape[1]), dtype=torch.float64, device=t.device)
    pre = torch.zeros((B, times.shape[1] * Kp), dtype=torch.float64, device=t.device)
    for s, m in enumerate(E.tolist()):
        tm, j = te[s, :m], idx[s, :m] // Kp
        p = torch.searchsorted(t[s].contiguous(), tm.expand(M, m).contiguous(), right=True)
        SA, SB = tabs[0][s].gather(1, p) * (tm / tau_s).exp(), tabs[1][s].gather(1, p) * (tm / tau).exp()
        G[s if per_sample else 0].index_add_(1, j, SA - SB)
        pre[s, idx[s, :m]] = (W[:, j] * (SA / tau_s - SB / tau)).sum(0)
    return (G if per_sample else G[0]), pre.reshape(times.shape)


def _dense(W, shape):
    """The (outputs, inputs) matrix of a valid convolution with filters (C_out, fx, fy, C), and the index that
    takes every filter entry's places out of it."""
    Co, fx, fy, C = W.shape
    X, Y = shape[:2]
    Xo, Yo = X - fx + 1, Y - fy + 1
    ar = [torch.arange(v, device=W.device) for v in (Xo, Yo, Co, fx, fy, C)]
    xo, yo, co, dx, dy, c = torch.meshgrid(*ar, indexing="ij")
    row, col = (xo * Yo + yo) * Co + co, ((xo + dx) * Y + yo + dy) * C + c
    D = torch.zeros((Xo * Yo * Co, X * Y * C), dtype=torch.float64, device=W.device)
    D[row, col] = W.double()[co, dx, dy, c]
    return D, (row, col, (Xo, Yo, Co))


def _filters(G, at):
    row, col, _ = at
    return torch.stack([g[row, col].sum((0, 1)) for g in G])


def _pool64(n, t, shape):
    X, Y, C = shape
    B, _, K = t.shape
    ix = torch.arange(X * Y * C, device=t.device).reshape(X, Y, C)[: X // 2 * 2, : Y // 2 * 2]
    ix = ix.reshape(X // 2, 2, Y // 2, 2, C).permute(0, 2, 4, 1, 3).reshape(-1, 4)
    src = (ix[:, :, None] * K + torch.arange(K, device=t.device)).reshape(ix.shape[0], 4 * K)
    ts, o = torch.sort(t.reshape(B, -1)[:, src], dim=2, stable=True)
    return n[:, ix].sum(2), ts, src.expand(B, -1, -1).gather(2, o)


def _unpool64(err, src, shape):
    pre = torch.zeros((err.shape[0], shape[1] * shape[2]), dtype=torch.float64, device=err.device)
    return pre.scatter_(1, src.reshape(err.shape[0], -1), err.reshape(err.shape[0], -1)).reshape(shape)


def _loss64(n, labels):
    goal = torch.full(n.shape, TARGETS[1], dtype=torch.float64, device=n.device)
    goal[torch.arange(n.shape[0], device=n.device), labels.long()] = TARGETS[0]
    return 0.5 * (goal - n).square().sum(1), goal - n


def _adam64(w, g, t):
    """Adam's step number t after steps on zero gradients: the new weights, m and v."""
    b1, b2 = 0.9, 0.999
    m, v = (1 - b1) * g, (1 - b2) * g * g
    return w.double() - LR * (m / (1 - b1 ** t)) / ((v / (1 - b2 ** t)).sqrt() + 1e-8), m, v


def _layers64(t, ws, thetas, K, max_sim):
    outs, trains = [], [t]
    for w, th in zip(ws, thetas):
        outs.append(_forward64(trains[-1], w, th, K, max_sim))
        trains.append(outs[-1][1][2])
    return outs, trains


def exact(case, seed):
    """No value for the gradients of deep networks and of layers with U(-1, 1) weights and many events: a potential
    that only grazes the threshold spikes in one precision and not in the other, and its gradient can be of any size."""
    kind, K = case["kind"], case["k"]
    if kind == "serve":
        ws, thetas, reqs = _serve_data(case, seed)
        t = np.full((len(reqs), ws[0].shape[1], max(int(np.bincount(r[0]).max()) for r in reqs)), np.inf, np.float32)
        for q, (ch, tm) in enumerate(reqs):
            o = np.argsort(ch, kind="stable")
            t[q, ch[o], np.arange(len(o)) - np.searchsorted(ch[o], ch[o])] = tm[o]
        outs, _ = _layers64(torch.from_numpy(t).cuda(), [torch.from_numpy(w).cuda() for w in ws], thetas, K, math.inf)
        return {"counts": outs[-1][0], "times": outs[-1][1][2]}
    if kind == "conv_train" or kind == "conv_block":
        return _exact_conv(case, seed)
    ws, thetas, t, _, labels, g = _fc_data(case, seed)
    outs, trains = _layers64(t, ws, thetas, K, MAX_SIM)
    counts = [o[0] for o in outs]
    if kind == "grad":
        n, out = outs[0]
        coef = torch.randn(out[2].shape, generator=g, device="cuda")
        gw, gx = (None, None) if case["weights"] == "uniform" else _backward64(t, ws[0], thetas[0], n, out, coef)
        return {"counts": n, "times": out[2], "gw": gw, "gx": gx}
    loss, err = _loss64(counts[-1], labels)
    err = err[:, :, None].expand(-1, -1, K)
    grads = [None] * len(ws)
    for li in reversed(range(len(ws))):
        G, err = _backward64(trains[li], ws[li], thetas[li], *outs[li], err)
        grads[li] = G / case["batch"]
    new = [_adam64(w, x, 2 if kind == "train" else 1) for w, x in zip(ws, grads)]
    res = {"loss": loss, "counts": counts, "times": outs[-1][1][2], "grad": grads, "w": [v[0] for v in new]}
    if kind == "train":
        res.update(m=[v[1] for v in new], v=[v[2] for v in new])
    if case["weights"] == "uniform" and (len(ws) > 2 or case["k_in"] > 1):
        res.update({key: None for key in ("grad", "m", "v") if key in res})
    return res


def _exact_conv(case, seed):
    w1, w2, fcs, t, _, labels, err = _conv_data(case, seed)
    K, th, shape = case["k"], CONV_THETAS, _ints(case["shape"])
    D1, at1 = _dense(w1, shape)
    o1 = _forward64(t, D1, th[0], K, MAX_SIM)
    p1 = _pool64(o1[0], o1[1][2], at1[2])
    s1 = (at1[2][0] // 2, at1[2][1] // 2, at1[2][2])
    D2, at2 = _dense(w2, s1)
    o2 = _forward64(p1[1], D2, th[1], K, MAX_SIM)
    counts, block, grads = [o1[0], p1[0], o2[0]], case["kind"] == "conv_block", []
    if not block:
        p2 = _pool64(o2[0], o2[1][2], at2[2])
        outs, trains = _layers64(p2[1], fcs, th[2:], K, MAX_SIM)
        counts += [p2[0]] + [o[0] for o in outs]
        loss, e = _loss64(outs[-1][0], labels)
        e = e[:, :, None].expand(-1, -1, K)
        for li in (1, 0):
            G, e = _backward64(trains[li], fcs[li], th[2 + li], *outs[li], e)
            grads.insert(0, G / case["batch"])
        err = _unpool64(e, p2[2], o2[1][2].shape)
    # The filters' gradients, sample by sample (the dense matrices are large).
    fold = [], []
    for s in range(case["batch"]):
        one = slice(s, s + 1)
        G2, e = _backward64(p1[1][one], D2, th[1], o2[0][one], o2[1][:, one], err[one])
        e = _unpool64(e, p1[2][one], o1[1][2][one].shape)
        G1, _ = _backward64(t[one], D1, th[0], o1[0][one], o1[1][:, one], e)
        fold[0].append(_filters(G1[None], at1)[0])
        fold[1].append(_filters(G2[None], at2)[0])
    g1, g2 = (torch.stack(f) for f in fold)
    if block:
        return {"counts": counts, "times": o2[1][2], "grad1": g1, "grad2": g2}
    grads = [g1.mean(0), g2.mean(0)] + grads
    w = [_adam64(w, g, 2)[0] for w, g in zip([w1, w2, *fcs], grads)]
    return {"loss": loss, "counts": counts, "times": outs[-1][1][2], "grad": None, "w": w, "m": None, "v": None}
