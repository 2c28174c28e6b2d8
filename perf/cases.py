"""Performance cases: the work that users of spiral_b200 have it do, through its public entry points.

Every kind of case below is one way in which the package is called: a bare GEMM, a hidden layer of a
training forward pass, narrow-net inference, a training step, inference from compact game states, the
per-decision call, a layer graph.  ``listed`` names the sizes that the benchmark and the tests run;
``draw`` takes others from the same ranges.  Inputs are made from a seed on the device; ``exact``
computes the same outputs in float64 with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spiral-s-ml-library_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import spiral_b200 as sb  # noqa: E402

TORCH = {"bf16": torch.bfloat16, "f16": torch.float16, "tf32": torch.float32, "f32": torch.float32}
ITEM = {"bf16": 2, "f16": 2, "tf32": 4, "f32": 4}

# Compact game states: one byte per one-hot field, the value `width` meaning "none".
LEDUC_WIDTHS = (3, 4, 14, 3) + (1,) * 8
HOLDEM_WIDTHS = (4, 13) * 7
NETS = {
    "leduc": [32, 256, 256, 256, 3],
    "holdem": [512, 1024, 1024, 1024, 1024, 10],
    "leduc_ensemble": [32, 64, 64],
    "holdem_ensemble": [512, 64],
}


def listed():
    return [
        # A large product as the layout sweep of the benchmark runs it: A [M, K] times B [K, N], fp32 out.
        {"name": "gemm_bf16_nn_4096", "kind": "gemm", "a_trans": False, "b_trans": False, "m": 4096, "n": 4096, "k": 4096, "dtype": "bf16"},
        # The reference's own arithmetic on sizes that fit no tile.
        {"name": "gemm_tf32_tn_ragged", "kind": "gemm", "a_trans": True, "b_trans": False, "m": 4000, "n": 3000, "k": 1000, "dtype": "tf32"},
        # The 1e-5 class, at the reference's test size (a latency-bound call) and at a size that fills the GPU.
        {"name": "gemm_f32_nt_512", "kind": "gemm", "a_trans": False, "b_trans": True, "m": 512, "n": 512, "k": 512, "dtype": "f32"},
        {"name": "gemm_f32_nt_2048", "kind": "gemm", "a_trans": False, "b_trans": True, "m": 2048, "n": 2048, "k": 2048, "dtype": "f32"},
        # A hidden layer of a training forward pass on one GPU's share of the batch: bias, ReLU, sign words.
        {"name": "layer_holdem_hidden", "kind": "layer", "rows": 32768, "fan_in": 1024, "fan_out": 1024, "dtype": "bf16"},
        # Policy evaluation with the Leduc net: the benchmark's batch, and one that fills the GPU many times.
        {"name": "infer_leduc_16384", "kind": "infer", "rows": 16384, "dtype": "f16"},
        {"name": "infer_leduc_262144", "kind": "infer", "rows": 262144, "dtype": "f16"},
        # One training step (forward, backward, SGD) of either net at the benchmark's batch.
        {"name": "train_leduc_65536", "kind": "train", "net": "leduc", "rows": 65536, "dtype": "bf16"},
        {"name": "train_holdem_262144", "kind": "train", "net": "holdem", "rows": 262144, "dtype": "bf16"},
        # Policy evaluation from compact records: the states are serialised on the device, then the wide net.
        {"name": "records_holdem_65536", "kind": "records", "rows": 65536, "dtype": "bf16"},
        # Decisions of an ensemble for the games in flight: few states, all members, one action each.
        {"name": "decide_leduc_256", "kind": "decide", "net": "leduc_ensemble", "members": 16, "rows": 256, "dtype": "f16"},
        # The reference's test graph: dense layers with row normalisation, a sampling head over a prefix.
        {"name": "graph_8192", "kind": "graph", "rows": 8192, "width": 128},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _mult(x, step):
    return max(step, x // step * step)


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "layer", "infer", "train", "train", "records", "decide", "graph"])
    if kind == "gemm":
        dtype = rng.choice(["bf16", "f16", "tf32", "f32"])
        top = 2048 if dtype == "f32" else 4096
        a_trans, b_trans = rng.choice([(False, True), (False, False), (True, False)])
        m, n, k = (_log(rng, 128, top) for _ in range(3))
        step = 16 // ITEM[dtype]                # contiguous dimensions are whole 16-byte pieces
        m = _mult(m, step) if a_trans else m
        n = _mult(n, 4 if b_trans else step)
        k = k if a_trans else _mult(k, step)
        if not a_trans and not b_trans:
            k = _mult(k, step)
        return {"kind": "gemm", "a_trans": a_trans, "b_trans": b_trans, "m": m, "n": n, "k": k, "dtype": dtype}
    if kind == "layer":
        return {"kind": "layer", "rows": _log(rng, 256, 65536), "fan_in": 64 * rng.randint(1, 16),
                "fan_out": 64 * rng.randint(1, 16), "dtype": rng.choice(["bf16", "f16"])}
    if kind == "infer":
        return {"kind": "infer", "rows": _log(rng, 64, 1 << 18), "dtype": rng.choice(["bf16", "f16"])}
    if kind == "train":
        net = rng.choice(["leduc", "holdem"])
        return {"kind": "train", "net": net, "rows": _log(rng, 256, 131072), "dtype": "bf16"}
    if kind == "records":
        return {"kind": "records", "rows": _log(rng, 128, 131072), "dtype": "bf16"}
    if kind == "decide":
        net = rng.choice(["leduc_ensemble", "holdem_ensemble"])
        return {"kind": "decide", "net": net, "members": rng.choice([4, 16, 32]), "rows": _log(rng, 64, 8192),
                "dtype": rng.choice(["bf16", "f16"])}
    return {"kind": "graph", "rows": _log(rng, 64, 65536), "width": 64 * rng.randint(1, 4)}


# -- inputs ----------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, shape, dtype, std=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def _states(g, rows, widths, none_share):
    """Compact records: a uniform value per field, some fields empty."""
    cols = []
    for w in widths:
        v = torch.randint(0, w, (rows,), generator=g, device="cuda")
        empty = torch.rand(rows, generator=g, device="cuda") < none_share
        cols.append(torch.where(empty, torch.full_like(v, w), v))
    return torch.stack(cols, 1).to(torch.uint8)


def _encoded(fields, widths, dense=None):
    cols = [(fields[:, j:j + 1] == torch.arange(w, device="cuda", dtype=torch.uint8)).float() for j, w in enumerate(widths)]
    return torch.cat(cols + ([] if dense is None else [dense.float()]), 1)


def _legal(g, rows, n):
    """Legal-action masks: the first two actions always, the others with probability 0.6."""
    mask = (torch.rand((rows, n), generator=g, device="cuda") < 0.6).to(torch.uint8)
    mask[:, :2] = 1
    return mask


def _weights(g, sizes):
    """Kaiming-uniform weights and small biases, fp32 on the host."""
    ws, bs = [], []
    for i in range(len(sizes) - 1):
        bound = math.sqrt(6.0 / sizes[i])
        ws.append(((torch.rand((sizes[i + 1], sizes[i]), generator=g, device="cuda") * 2 - 1) * bound).cpu().numpy())
        bs.append(((torch.rand(sizes[i + 1], generator=g, device="cuda") * 2 - 1) * 0.1).cpu().numpy())
    return ws, bs


def _inputs(case, seed):
    """Everything a pass reads, as torch tensors (weights as host arrays), from the seed alone."""
    g, kind = _gen(seed), case["kind"]
    if kind == "gemm":
        m, n, k, dt = case["m"], case["n"], case["k"], TORCH[case["dtype"]]
        return {"a": _normal(g, (k, m) if case["a_trans"] else (m, k), dt), "b": _normal(g, (n, k) if case["b_trans"] else (k, n), dt)}
    rows = case["rows"]
    if kind == "layer":
        dt = TORCH[case["dtype"]]
        return {"x": torch.relu(_normal(g, (rows, case["fan_in"]), dt)), "bias": _normal(g, (case["fan_out"],), torch.float32, 0.1),
                "w": _normal(g, (case["fan_out"], case["fan_in"]), dt, math.sqrt(2.0 / case["fan_in"]))}
    if kind == "graph":
        w = case["width"]
        return {"x": _normal(g, (rows, w), torch.float32), "w": [_normal(g, (w, w), torch.float32, 0.1) for _ in range(3)]}
    if kind == "decide":
        sizes, dt = NETS[case["net"]], TORCH[case["dtype"]]
        if case["net"] == "leduc_ensemble":
            d = {"fields": _states(g, rows, LEDUC_WIDTHS, 0.2)}
        else:
            d = {"x": (torch.rand((rows, sizes[0]), generator=g, device="cuda") < 0.1).to(dt)}
        return dict(d, w=[_weights(g, sizes)[0] for _ in range(case["members"])])
    net = {"infer": "leduc", "records": "holdem"}.get(kind) or case["net"]
    sizes, dt = NETS[net], TORCH[case["dtype"]]
    if net == "leduc":
        fields, dense = _states(g, rows, LEDUC_WIDTHS, 0.2), None
    else:
        fields = _states(g, rows, HOLDEM_WIDTHS, 0.3)
        dense = torch.rand((rows, sizes[0] - sum(HOLDEM_WIDTHS)), generator=g, device="cuda").to(dt)
    mask = _legal(g, rows, sizes[-1])
    d = {"mask": mask}
    if kind == "records":
        d.update(fields=fields, dense=dense)
    else:
        d["x"] = _encoded(fields, LEDUC_WIDTHS if net == "leduc" else HOLDEM_WIDTHS, dense).to(dt)
    if kind == "train":
        t = torch.rand((rows, sizes[-1]), generator=g, device="cuda") * mask
        d["target"] = t / t.sum(1, keepdim=True)
    d["w"], d["bias"] = _weights(g, sizes)
    return d


# -- the calls -------------------------------------------------------------------------------------------
class _Buffer:
    """The package's device buffer under the array interface that torch reads."""

    TYPES = {"f32": "<f4", "i32": "<i4"}

    def __init__(self, a):
        self.array = a
        self.__cuda_array_interface__ = {"shape": a.shape, "typestr": self.TYPES[a.dtype], "data": (a.ptr, False), "version": 3}


def _torch(a):
    return torch.as_tensor(_Buffer(a), device="cuda")


def _array(t, dtype):
    return sb.DeviceArray(tuple(t.shape), dtype, ptr=t.data_ptr(), owner=t)


def prepare(case, seed):
    s, kind, d = {"case": case}, case["kind"], _inputs(case, seed)
    if kind == "gemm":
        return dict(s, a=d["a"], b=d["b"], c=torch.empty((case["m"], case["n"]), device="cuda"))
    rows = case["rows"]
    if kind == "layer":
        n = case["fan_out"]
        return dict(s, x=d["x"], w=d["w"], bias=d["bias"], y=torch.empty((rows, n), dtype=TORCH[case["dtype"]], device="cuda"),
                    bits=torch.empty((n // 32, rows), dtype=torch.int32, device="cuda"))
    if kind == "graph":
        L, w = sb.layers, case["width"]
        h = L.relu(L.ln_l2(L.matmul((w, w), L.input("x", (1, rows, w)))))
        h = L.relu(L.ln_l2(L.matmul((w, w), h)))
        sample = L.masked_softmax_and_discrete_sample(3, L.matmul((w, w), h))
        model = L.create_model(sample)
        L.key_extract(model, "x").upload(d["x"].cpu().numpy())
        for node, v in zip([n for n in model.nodes if n.op == "matmul"], d["w"]):
            model.weight(node).upload(v.cpu().numpy())
        return dict(s, model=model, seed=seed, out={"probs": _torch(model.tensor(sample.src)), "indices": _torch(model.tensor(sample))})
    if kind == "decide":
        sizes = NETS[case["net"]]
        ens = sb.EnsemblePolicyMLP(sizes, rows, case["members"], in_dtype=case["dtype"], with_bias=False)
        ens.load_weights(d["w"])
        return dict(s, ens=ens, fields=d.get("fields"), x=d.get("x"), seed=seed, action=None, out=None)
    if kind == "infer":
        net = sb.PolicyMLP(NETS["leduc"], rows, in_dtype=case["dtype"], head=("masked_softmax", "regret_matching", "argmax"))
        net.load_weights(d["w"], d["bias"])
        return dict(s, net=net, x=d["x"], mask=d["mask"], out={"probs": _torch(net.probs), "actions": _torch(net.actions)})
    if kind == "records":
        sizes = NETS["holdem"]
        net = sb.PolicyMLP(sizes, rows, in_dtype=case["dtype"], head=("masked_softmax", "argmax"))
        net.load_weights(d["w"], d["bias"])
        return dict(s, net=net, fields=d["fields"], dense=_array(d["dense"], case["dtype"]), x=sb.DeviceArray((rows, sizes[0]), case["dtype"]),
                    mask=d["mask"], out={"probs": _torch(net.probs), "actions": _torch(net.actions)})
    net = sb.PolicyMLP(NETS[case["net"]], rows, in_dtype=case["dtype"], training=True)
    net.load_weights(d["w"], d["bias"])
    return dict(s, net=net, x=d["x"], mask=d["mask"], target=d["target"],
                out={"grads": _torch(net.grads), "params": _torch(net.params), "probs": _torch(net.probs), "loss": _torch(net.loss)})


LEARNING_RATE = 1e-3


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "gemm":
        if case["dtype"] == "tf32":
            return sb.matmul_tf32(case["a_trans"], case["b_trans"], 1.0, s["a"], s["b"], 0.0, s["c"])
        return sb.matmul(case["a_trans"], case["b_trans"], 1.0, s["a"], s["b"], 0.0, s["c"], in_dtype=case["dtype"])
    if kind == "layer":
        sb.matmul(False, True, 1.0, s["x"], s["w"], 0.0, s["y"], epilogue=("bias", "relu", "relu_mask_out"), bias=s["bias"], aux_out=s["bits"])
        return {"y": s["y"], "bits": s["bits"]}
    if kind == "infer":
        s["net"].forward_fused(s["x"], mask=s["mask"])
    elif kind == "train":
        s["net"].loss.fill_zero()
        s["net"].train_step(s["x"], s["mask"], s["target"], LEARNING_RATE)
    elif kind == "records":
        sb.primitives.encode_states(s["fields"], HOLDEM_WIDTHS, s["dense"], s["x"])
        s["net"].forward(s["x"], mask=s["mask"])
    elif kind == "graph":
        sb.layers.graph_run_host(s["model"], seed=s["seed"])
    else:
        if s["fields"] is not None:
            r = s["ens"].decide(s["seed"], fields=s["fields"], widths=LEDUC_WIDTHS, head=("masked_softmax",), prefix=3)
        else:
            r = s["ens"].decide(s["seed"], x=s["x"], head=("regret_matching",), prefix=3)
        if s["out"] is None or s["action"] is not r["action"]:      # the buffers are made by the first call
            s["action"], s["out"] = r["action"], {k: _torch(v) for k, v in r.items()}
    return s["out"]


# -- what a pass cannot do without -----------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "gemm":
        m, n, k, es = case["m"], case["n"], case["k"], ITEM[case["dtype"]]
        return {"bytes": (m * k + n * k) * es + m * n * 4, "flops": 2.0 * m * n * k}
    rows = case["rows"]
    if kind == "layer":
        i, o = case["fan_in"], case["fan_out"]
        return {"bytes": (rows * i + i * o + rows * o) * 2 + o * 4 + rows * o // 8, "flops": 2.0 * rows * i * o}
    if kind == "graph":
        w = case["width"]
        return {"bytes": rows * w * 8 + 3 * w * w * 4 + rows * 4, "flops": 6.0 * rows * w * w}
    if kind == "decide":
        sizes, e = NETS[case["net"]], case["members"]
        dense = sum(sizes[i] * sizes[i + 1] for i in range(len(sizes) - 1))
        state = len(LEDUC_WIDTHS) if case["net"] == "leduc_ensemble" else 2 * sizes[0]
        return {"bytes": rows * (state + e * (sizes[-1] * 4 + 8) + 12) + e * dense * 2, "flops": 2.0 * rows * e * dense}
    sizes = NETS[{"infer": "leduc", "records": "holdem"}.get(kind) or case["net"]]
    dense = sum(sizes[i] * sizes[i + 1] for i in range(len(sizes) - 1))
    n = sizes[-1]
    if kind == "train":
        # Input, mask and target in, probabilities out; parameters read and written; the activations of a
        # step that does not fit on the chip written and read once.
        acts = 4 * sum(sizes[1:-1])
        return {"bytes": rows * (2 * sizes[0] + 9 * n + acts) + dense * 14, "flops": 2.0 * rows * (3 * dense - sizes[0] * sizes[1])}
    state = 2 * sizes[0] if kind == "infer" else len(HOLDEM_WIDTHS) + 2 * (sizes[0] - sum(HOLDEM_WIDTHS))
    return {"bytes": rows * (state + 5 * n + 4) + dense * 2, "flops": 2.0 * rows * dense}


def tolerance(case):
    # About four times what the path is off from float64 (measured: GEMM 4e-6 bf16, 8e-4 tf32, 2e-6 f32; a layer
    # and whole nets 1.4e-3 to 2.1e-3 in bf16, 1e-4 to 2e-4 in f16; the graph 2.7e-4).  `differ`: sign words with
    # a value next to zero, indices whose two best values are next to each other.
    kind = case["kind"]
    if kind == "gemm":
        return {"rel": {"f32": 1e-5, "tf32": 3e-3}.get(case["dtype"], 2e-5)}
    rel = 1.2e-3 if kind == "graph" or case["dtype"] == "f16" else 8e-3
    if kind == "train":
        return {"rel": rel, "max": 0.3}
    return {"rel": rel, "max": 0.3, "differ": 1e-3 if kind == "layer" else 5e-3}


# -- the same outputs in float64 -------------------------------------------------------------------------
def _round_tf32(t):
    u = t.contiguous().view(torch.int32)
    u = (u + 0x0FFF + ((u >> 13) & 1)) & ~0x1FFF
    return u.view(torch.float32)


def _softmax(x, legal):
    x = torch.where(legal, x, torch.full_like(x, -1e300))
    e = torch.where(legal, torch.exp(x - x.max(-1, keepdim=True).values), torch.zeros_like(x))
    return e / e.sum(-1, keepdim=True)


def _regret(x, legal):
    q = torch.where(legal, x.clamp(min=0), torch.zeros_like(x))
    s = q.sum(-1, keepdim=True)
    return torch.where(s != 0, q / s, legal / legal.sum(-1, keepdim=True))


def _dense64(x, ws, bs, dt):
    """Hidden activations and the last layer's output; weights as the storage type holds them."""
    hs = [x.double()]
    for i, w in enumerate(ws):
        y = hs[-1] @ torch.from_numpy(w).cuda().to(dt).double().T
        if bs is not None:
            y += torch.from_numpy(bs[i]).cuda().double()
        hs.append(torch.relu(y) if i + 1 < len(ws) else y)
    return hs


def exact(case, seed):
    kind, d = case["kind"], _inputs(case, seed)
    if kind == "gemm":
        a, b = d["a"].double(), d["b"].double()
        return (a.T if case["a_trans"] else a) @ (b.T if case["b_trans"] else b)
    if kind == "layer":
        return {"y": torch.relu(d["x"].double() @ d["w"].double().T + d["bias"].double()), "bits": None}
    if kind == "graph":
        h = d["x"].double()
        for i, w in enumerate(d["w"]):
            h = h @ _round_tf32(w).double().T
            if i < 2:
                h = torch.relu(h / (h * h).sum(-1, keepdim=True))
        legal = (torch.arange(case["width"], device="cuda") < 3).expand_as(h)
        return {"probs": _softmax(h, legal), "indices": None}
    dt = TORCH[case["dtype"]]
    if kind == "decide":
        x = (_encoded(d["fields"], LEDUC_WIDTHS) if "fields" in d else d["x"]).to(dt)
        y = torch.stack([_dense64(x, ws, None, dt)[-1] for ws in d["w"]])
        legal = (torch.arange(y.shape[-1], device="cuda") < 3).expand_as(y)
        probs = _softmax(y, legal) if "fields" in d else _regret(y, legal)
        return {"action": None, "ensemble_id": None, "sampling_prob_selected": None, "sampling_prob_ensemble": None, "output_indices": None,
                "output_probs": probs}
    x = _encoded(d["fields"], HOLDEM_WIDTHS, d["dense"]).to(dt) if kind == "records" else d["x"]
    legal = d["mask"] != 0
    hs = _dense64(x, d["w"], d["bias"], dt)
    probs = _softmax(hs[-1], legal)
    if kind == "infer":
        return {"probs": _regret(probs, legal), "actions": None}
    if kind == "records":
        return {"probs": probs, "actions": None}
    # Cross-entropy of the masked softmax, mean over the batch; gradients and parameters in the flat layout
    # [W0 | b0 | W1 | b1 | ...]: weight rows padded to a multiple of 8, segments to 64 elements.
    sizes, rows = NETS[case["net"]], case["rows"]
    t = torch.where(legal, d["target"].double(), torch.zeros_like(probs))
    loss = -(t * torch.log(probs.clamp(min=1e-38))).sum() / rows
    dy = torch.where(legal, (probs * t.sum(-1, keepdim=True) - t) / rows, torch.zeros_like(probs))
    gw, gb = [None] * (len(sizes) - 1), [None] * (len(sizes) - 1)
    for i in range(len(sizes) - 2, -1, -1):
        gw[i], gb[i] = dy.T @ hs[i], dy.sum(0)
        if i:
            dy = (dy @ torch.from_numpy(d["w"][i]).cuda().to(dt).double()) * (hs[i] > 0)
    grads, params = [], []
    for i in range(len(sizes) - 1):
        pad = (-sizes[i + 1]) % 8 * sizes[i]
        for g, p, extra in ((gw[i], d["w"][i], pad), (gb[i], d["bias"][i], 0)):
            zeros = torch.zeros(extra + (-(g.numel() + extra)) % 64, dtype=torch.float64, device="cuda")
            grads += [g.reshape(-1), zeros]
            params += [torch.from_numpy(np.ascontiguousarray(p)).cuda().double().reshape(-1), zeros]
    grads, params = torch.cat(grads), torch.cat(params)
    return {"grads": grads, "params": params - LEARNING_RATE * grads, "probs": probs, "loss": loss.reshape(1)}
