"""What the forward pipe is timed on: the calls an engine, an analysis front end
or a self-play server makes, from one position on a small network to a full
batch on the largest one.

A case names a call, an arithmetic mode, a network (blocks x filters) and a
batch.  The calls are the public ones of the package:

  planes         Context.forward: fp32 planes in host memory -> raw head planes
                 (what an engine's search thread asks of its pipe)
  planes_packed  Context.forward_packed: the same with bit-packed positions
  heads          Context.forward_heads: fp32 planes in host memory -> policy and
                 winrate
  heads_packed   Context.forward_heads_packed: bit-packed positions -> policy
                 and winrate (what a self-play or analysis server asks)
  heads_device   Context.forward_heads_device: positions and results stay on the
                 GPU (a server that keeps its queue there; enqueued, not waited for)
  scheduler      Scheduler.forward: a block of positions through the batching
                 queue (many games sharing one GPU)

Networks are random, He-normal, with batch-norm statistics measured on a few
positions, as a trained file has them; positions are random 0/1 planes.
"""
import importlib
import math

import numpy as np
import torch

lzb = importlib.import_module("leela-zero_b200")

BOARD, SQ, PLANES, MOVES, HIDDEN = 19, 361, 18, 362, 256


def _case(call, precision, blocks, filters, batch, name=None):
    c = {"call": call, "precision": precision, "blocks": blocks, "filters": filters, "batch": batch}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small network in single precision, one position: an engine on its first games
        _case("planes", "fp32", 6, 64, 1, "planes fp32 6x64 n1"),
        # one position on a large network: a lone search thread, analysis of a game
        _case("planes", "fp16x2", 20, 256, 1, "planes fp16x2 20x256 n1"),
        # a handful of search threads on one GPU, the engine's usual batch of 8
        _case("planes_packed", "fp16x2", 15, 192, 8, "packed fp16x2 15x192 n8"),
        # a narrow network answering a small server, fast mode
        _case("heads_packed", "fp16", 10, 128, 8, "heads fp16 10x128 n8"),
        # an odd small batch on the large network, planes from the caller
        _case("heads", "fp16", 20, 256, 5, "heads fp16 20x256 n5"),
        # a server with a few dozen games in flight
        _case("heads_packed", "fp16x2", 20, 256, 32, "heads fp16x2 20x256 n32"),
        # a block of games through the batching queue
        _case("scheduler", "fp16x2", 15, 192, 64, "queue fp16x2 15x192 n64"),
        # a ragged batch in the bf16 mode that holds the half-precision bounds
        _case("heads_packed", "bf16x3", 20, 256, 21, "heads bf16x3 20x256 n21"),
        # a wide batch kept on the GPU, fast mode
        _case("heads_device", "fp16", 20, 256, 128, "device fp16 20x256 n128"),
        # single precision where an engine asks for it: a few search threads
        _case("planes", "fp32", 20, 256, 8, "planes fp32 20x256 n8"),
        # single precision over a ragged batch: checking and rating positions in bulk
        _case("heads_packed", "fp32", 10, 128, 77, "heads fp32 10x128 n77"),
        # the largest network with a full batch: self-play at scale
        _case("heads_device", "fp16x2", 40, 256, 256, "device fp16x2 40x256 n256"),
    ]


#: networks that are trained: filters in steps of 32, deeper ones wider
_NETS = ((5, 64), (6, 64), (6, 96), (6, 128), (8, 96), (10, 128), (10, 160), (12, 128), (15, 192), (15, 256),
         (20, 192), (20, 224), (20, 256), (24, 256), (30, 256), (40, 256))


def draw(rng):
    """A network, a mode, a call and a batch; batches spread over their logarithm."""
    blocks, filters = rng.choice(_NETS)
    precision = rng.choice(("fp16x2", "fp16x2", "fp16x2", "fp16", "fp16", "fp32", "fp32", "bf16x3"))
    # relative cost of a position: no drawn case above 40x256, 256 positions, fp16x2
    cost = {"fp16x2": 1.0, "fp16": 1.0, "bf16x3": 3.0, "fp32": 8.0}[precision]
    most = int(256 * 40.0 / (blocks * cost))
    batch = max(1, min(256, most, int(round(math.exp(rng.uniform(0.0, math.log(257.0)))))))
    calls = ["planes", "planes_packed", "heads", "heads_packed", "heads_packed"]
    if batch >= 16:
        calls.append("scheduler")
    if batch >= 64:
        calls += ["heads_device", "heads_device"]
    return _case(rng.choice(calls), precision, blocks, filters, batch)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _network(blocks, filters, gen):
    """Random-init network in the form of a weights file, made on the GPU:
    He-normal filters, batch-norm statistics = those of the layer's own outputs
    on four positions, perturbed by m ~ N(0, 0.1) and v ~ U(0.5, 1.5)."""
    dev = torch.device("cuda")

    def normal(shape, sigma):
        return torch.randn(shape, generator=gen, device=dev) * sigma

    def stats(y):
        y = y.double().transpose(0, 1).reshape(y.shape[1], -1)
        return y.mean(1).float(), y.var(1, unbiased=False).clamp_min(1e-6).float()

    def perturbed(mu, var):
        m = normal(mu.shape, 0.1)
        v = torch.rand(var.shape, generator=gen, device=dev) + 0.5
        return mu + m * var.sqrt(), var * v

    x = torch.from_numpy(lzb.weights.synthetic_positions(4, 977)).to(dev)
    raw = {"blocks": blocks, "channels": filters, "conv_w": [], "conv_b": [], "bn_mean": [], "bn_var": []}
    res = None
    with torch.backends.cudnn.flags(enabled=True, benchmark=False, deterministic=True, allow_tf32=False):
        for l in range(1 + 2 * blocks):
            cin = PLANES if l == 0 else filters
            w = normal((filters, cin, 3, 3), math.sqrt(2.0 / (9 * cin)))
            y = torch.nn.functional.conv2d(x, w, padding=1)
            mean, var = perturbed(*stats(y))
            z = (y - mean[None, :, None, None]) / (var + 1e-5).sqrt()[None, :, None, None]
            if l > 0 and l % 2 == 0:
                z = z + res
            x = z.clamp_min(0)
            if l % 2 == 0:
                res = x
            raw["conv_w"].append(w)
            raw["bn_mean"].append(mean)
            raw["bn_var"].append(var)
    zero = torch.zeros(filters)
    raw["conv_b"] = [zero.numpy()] * (1 + 2 * blocks)
    flat = x.reshape(4, filters, SQ).double()
    for head, planes in (("pol", 2), ("val", 1)):
        w = normal((planes, filters), math.sqrt(2.0 / filters))
        mean, var = perturbed(*stats(torch.einsum("kc,ncs->nks", w.double(), flat)))
        raw[head + "_w"], raw["bn_%s_mean" % head], raw["bn_%s_var" % head] = w, mean, var
        raw[head + "_b"] = np.zeros(planes, np.float32)
    raw["ip_pol_w"] = normal((MOVES, 2 * SQ), math.sqrt(1.0 / SQ))
    raw["ip1_val_w"] = normal((HIDDEN, SQ), math.sqrt(2.0 / SQ))
    raw["ip2_val_w"] = normal((1, HIDDEN), math.sqrt(2.0 / HIDDEN))
    raw["ip_pol_b"], raw["ip1_val_b"] = np.zeros(MOVES, np.float32), np.zeros(HIDDEN, np.float32)
    raw["ip2_val_b"] = np.zeros(1, np.float32)

    def host(v):
        return v.cpu().numpy() if isinstance(v, torch.Tensor) else v

    return {k: [host(a) for a in v] if isinstance(v, list) else host(v) for k, v in raw.items()}


def _winograd_filters(w):
    """[K][C][3][3] -> [36][C][K], the transformed filters a scheduler is given."""
    s = math.sqrt(2.0)
    g = torch.tensor([[1, 0, 0], [-2 / 3, -s / 3, -1 / 3], [-2 / 3, s / 3, -1 / 3], [1 / 6, s / 6, 1 / 3],
                      [1 / 6, -s / 6, 1 / 3], [0, 0, 1]], dtype=torch.float64, device="cuda")
    f = torch.from_numpy(w).cuda().double()
    u = torch.einsum("ik,ockl,jl->ijco", g, f, g).float()
    return np.ascontiguousarray(u.reshape(36, w.shape[1], w.shape[0]).cpu().numpy())


def prepare(case, seed):
    """A network on the GPU, a context (or a scheduler) for batches of this
    size, and the positions: host arrays, or device tensors for heads_device."""
    n, call = case["batch"], case["call"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    raw = _network(case["blocks"], case["filters"], gen)
    net = lzb.weights.prepare(raw, transform=False)
    x = lzb.weights.synthetic_positions(n, seed)
    state = {"call": call, "n": n}
    if call == "scheduler":
        net["U"] = [_winograd_filters(w) for w in net["filters"]]
        state["scheduler"] = lzb.Scheduler(net, case["precision"], batch_size=max(64, n), num_threads=64)
        state["x"] = x
        return state
    state["context"] = lzb.Pipe(net, case["precision"], from_filters=True).context(n)
    if call == "heads_device":
        state["x"] = torch.from_numpy(x).cuda()
        state["policy"] = torch.empty((n, MOVES), device="cuda")
        state["winrate"] = torch.empty((n,), device="cuda")
    else:
        state["x"] = lzb.pack_positions(x) if call.endswith("_packed") else x
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    call, x = state["call"], state["x"]
    if call == "planes":
        return state["context"].forward(x)
    if call == "planes_packed":
        return state["context"].forward_packed(x)
    if call == "heads":
        return state["context"].forward_heads(x)
    if call == "heads_packed":
        return state["context"].forward_heads_packed(x)
    if call == "scheduler":
        return state["scheduler"].forward(x)
    policy, winrate = state["policy"], state["winrate"]
    state["context"].forward_heads_device(x.data_ptr(), state["n"], 1.0, policy.data_ptr(), winrate.data_ptr())
    return policy, winrate


def work(case):
    """Positions in, results out and every weight once; multiply-adds of the
    3x3 layers as direct convolutions (fp32: as Winograd F(4x4,3x3), which needs
    fewer), one product for each weight, plus the heads."""
    n, c, layers = case["batch"], case["filters"], 2 * case["blocks"]
    call = case["call"]
    packed = call.endswith("_packed")
    heads = call.startswith("heads")
    fp32 = case["precision"] == "fp32"
    weight_bytes = {"fp32": 4, "bf16x3": 4}.get(case["precision"], 2)
    filters = 9 * c * (PLANES + layers * c)
    data = n * ((PLANES * 12 * 4 if packed else PLANES * SQ * 4) + ((MOVES + 1) * 4 if heads else 3 * SQ * 4))
    data += filters * weight_bytes + 3 * c * 4 + (1 + layers) * 2 * c * 4
    per_filter = 2 * 36 * 25 / 9 if fp32 else 2 * SQ
    flops = n * (filters * per_filter + 2 * 3 * c * SQ)
    if heads:
        fc = MOVES * 2 * SQ + HIDDEN * SQ + HIDDEN
        data += fc * 4
        flops += n * 2 * fc
    return {"bytes": data, "flops": flops}


def tolerance(case):
    """Rounding of the operands grows with depth: 16-bit planes are rounded once
    per layer, and a softmax turns an error of its logits into a relative one.
    fp16 carries 11 bits, fp16x2 and bf16x3 some 14 and 16; in fp32 only the order
    of summation differs."""
    depth = math.sqrt(case["blocks"] / 40.0)
    rel = {"fp16": 2e-2, "fp16x2": 1e-2, "bf16x3": 2e-3, "fp32": 6e-5}[case["precision"]] * depth
    return {"rel": max(rel, 1e-5)}
