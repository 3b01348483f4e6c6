"""What a program does with this library, as cases that can be timed: MoE layers driven through the public Python
binding (q36_b200.moe) at every size between one decoded token and a 32,768-token prompt, from device and from host
buffers, on a whole layer and on an expert shard, plus loading a layer's weights.

The layer shapes are the model's (hidden 2048, expert intermediate 512) with the expert counts the router supports.
Steps run through a stack of distinct layers, as decoding and prompt processing do, so that weights come from HBM and
not from a cache that an earlier pass filled; the layers' inputs are independent of one another.

  kind     the call a pass makes for every layer of the stack
  -------  ---------------------------------------------------------------------------------------------
  layer    MoELayer.forward: normalised activations and router logits in, layer output out
  decode   MoELayer.decode, the engine's one-token entry by name
  prefill  MoELayer.prefill, its batched entry by name
  graph    MoELayer.forward over the stack, captured once into a CUDA graph and replayed, as a serving loop does
  block    MoELayer.block: residual stream in and out (add, norm, router, experts, combine, add, next norm)
  host     HostStack.step: the whole stack from pinned host buffers, results back on the host
  load     MoELayer.load_gguf_blocks: a layer's GGUF MXFP4 blocks from host memory onto the device
"""
import math

import numpy as np
import torch

from q36_b200 import moe

D, FF = 2048, 512
EXPERT_BYTES = 3 * D * FF * 17 // 32     # gate + up + down of one expert, 17 bytes per 32 weights
ASSIGNMENT_FLOPS = 2 * 3 * D * FF        # one (token, expert) evaluation


def _case(name, kind, T, layers, E=256, k=8, x="bf16", zipf=False, se0=0, se1=None, shared=True):
    c = {"kind": kind, "T": T, "layers": layers, "E": E, "k": k, "x": x, "zipf": zipf, "se0": se0,
         "se1": E if se1 is None else se1, "shared": shared}
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # one user's token through the 40-layer stack, launched call by call: latency and launches are everything
        _case("decode_1", "decode", 1, 40, x="f32"),
        # the serving loop's usual step: a small batch, one CUDA graph of the 40-layer stack
        _case("decode_8_graph", "graph", 8, 40),
        # the same step for a program that keeps activations on the host
        _case("decode_8_host", "host", 8, 40),
        # decoding from the residual stream, an odd batch
        _case("decode_block_5", "block", 5, 16, x="f32"),
        # a smaller model: 32 experts, 4 used, 3 tokens
        _case("decode_3_small", "layer", 3, 40, E=32, k=4),
        # more users than one token tile holds
        _case("batch_33", "layer", 33, 16),
        # one rank of four that keeps its quarter of the experts and leaves the shared expert to rank 0
        _case("batch_96_shard", "layer", 96, 16, se0=64, se1=128, shared=False),
        # a short prompt, or a large batch of users, from the residual stream
        _case("block_300", "block", 300, 8, x="f32"),
        # prompts: the bucket of 1000 words with skewed experts, and the usual chunk of 4096 with skewed experts
        _case("prefill_1001_zipf", "prefill", 1001, 8, zipf=True),
        _case("prefill_4096_zipf", "layer", 4096, 4, zipf=True),
        # a long prompt in one call
        _case("prefill_32768", "prefill", 32768, 2),
        # loading a layer of a 64-expert model
        _case("load_64", "load", 0, 1, E=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    group = rng.choice(["decode", "decode", "batch", "batch", "prefill", "prefill", "host", "load"])
    E = rng.choice([256, 256, 256, 128, 64, 32])
    k = rng.choice([8, 8, 8, 6, 4, 2])
    x = rng.choice(["bf16", "bf16", "f32"])
    zipf = rng.random() < 0.4
    if group == "load":
        e = rng.choice([16, 32, 48, 64])
        se0 = rng.randrange(0, 65 - e)
        return _case("", "load", 0, 1, E=64, se0=se0, se1=se0 + e, shared=rng.random() < 0.7)
    if group == "host":
        return _case("", "host", _log_int(rng, 1, 128), rng.randint(8, 24), E=E, k=k, x=x, zipf=zipf)
    if group == "decode":
        kind = rng.choice(["decode", "graph", "block", "layer"])
        T, layers = rng.randint(1, 16), rng.randint(8, 16)
    elif group == "batch":
        kind = rng.choice(["layer", "graph", "block", "layer"])
        T, layers = _log_int(rng, 17, 600), rng.randint(6, 12)
    else:
        kind = rng.choice(["prefill", "layer", "block", "prefill"])
        T, layers = _log_int(rng, 600, 12000), rng.randint(1, 3)
    se0, se1, shared = 0, E, True
    if kind != "block" and rng.random() < 0.25:      # an expert shard of 2 or 4 ranks
        world = rng.choice([2, 4])
        r = rng.randrange(world)
        se0, se1, shared = r * E // world, (r + 1) * E // world, r == 0
    return _case("", kind, T, layers, E=E, k=k, x="f32" if kind == "block" else x, zipf=zipf, se0=se0, se1=se1, shared=shared)


# ------------------------------------------------------------------------------------------------- inputs
def _zipf_bias(E, device=None):
    return 1.1 * torch.log(1.0 / torch.arange(1, E + 1, dtype=torch.float32, device=device))


def _host_blocks(g, n, M, K):
    """GGUF MXFP4 blocks as a file reader hands them over: uniform codes, scale bytes in [118, 130]."""
    b = torch.randint(0, 256, (n, M, K // 32, 17), dtype=torch.uint8, device="cuda", generator=g)
    b[..., 0] = torch.randint(118, 131, (n, M, K // 32), dtype=torch.uint8, device="cuda", generator=g)
    return b.cpu().numpy()


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind, T, NL, E = case["kind"], case["T"], case["layers"], case["E"]
    if kind == "load":
        shared = [_host_blocks(g, 1, M, K) for M, K in ((FF, D), (FF, D), (D, FF))] if case["shared"] else [None] * 3
        return {"case": case, "blocks": [_host_blocks(g, E, M, K) for M, K in ((FF, D), (FF, D), (D, FF))] + shared}
    layers = [moe.MoELayer(n_expert=E, k=case["k"], D=D, FF=FF, se0=case["se0"], se1=case["se1"])
              .random_planes(seed * 1009 + l, shared=case["shared"]) for l in range(NL)]
    dtype = torch.bfloat16 if case["x"] == "bf16" else torch.float32
    s = {"case": case, "layers": layers}
    if kind == "block":
        # residual stream, attention output to add, norm weights around 1, router rows that give logits of unit variance
        s["h"] = torch.randn((NL, T, D), device="cuda", generator=g)
        s["a"] = torch.randn((NL, T, D), device="cuda", generator=g) * 0.5
        s["post_norm"] = 1 + 0.1 * torch.randn((NL, D), device="cuda", generator=g)
        s["next_norm"] = 1 + 0.1 * torch.randn((NL, D), device="cuda", generator=g)
        s["router"] = torch.randn((NL, E + 1, D), device="cuda", generator=g) / math.sqrt(D)
        if case["zipf"]:     # some experts are liked more: a common direction in the stream, weighed by popularity
            v = torch.randn(D, device="cuda", generator=g)
            v /= v.norm()
            s["h"] += math.sqrt(D) * v
            s["router"][:, :E] += (0.7 * _zipf_bias(E, "cuda") / math.sqrt(D))[None, :, None] * v
        return s
    X = torch.randn((NL, T, D), device="cuda", generator=g).to(torch.bfloat16).to(dtype)
    L = torch.randn((NL, T, E + 1), device="cuda", generator=g)     # the last column is the shared expert's gate
    if case["zipf"]:
        L[:, :, :E] += _zipf_bias(E, "cuda")
    if kind == "host":
        s["X"], s["L"] = X.cpu().pin_memory(), L.cpu().pin_memory()
        s["out"] = torch.empty((NL, T, D), dtype=torch.float32).pin_memory()
        s["stack"] = moe.HostStack(layers, T, x_is_bf16=dtype == torch.bfloat16)
        return s
    s["X"], s["L"] = [X[l] for l in range(NL)], [L[l] for l in range(NL)]
    s["out"] = torch.empty((NL, T, D), dtype=torch.float32, device="cuda")
    s["outs"] = [s["out"][l] for l in range(NL)]
    if kind == "prefill" or kind == "decode":
        return s
    s["ws"] = layers[0].workspace(T)         # the layers of a step run one after another and share the scratch
    if kind == "graph":
        _forward(s)
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                _forward(s)
        s["graph"] = graph
    return s


# ------------------------------------------------------------------------------------------------- one pass
def _forward(s):
    inc = s["case"]["shared"]
    for layer, X, L, out in zip(s["layers"], s["X"], s["L"], s["outs"]):
        layer.forward(X, L, out=out, inc_shared=inc, ws=s["ws"])


def run(s):
    case = s["case"]
    kind, inc = case["kind"], case["shared"]
    if kind == "layer":
        _forward(s)
        return s["out"]
    if kind == "decode":
        for layer, X, L, out in zip(s["layers"], s["X"], s["L"], s["outs"]):
            layer.decode(X, L, out=out, inc_shared=inc)
        return s["out"]
    if kind == "prefill":
        for layer, X, L, out in zip(s["layers"], s["X"], s["L"], s["outs"]):
            layer.prefill(X, L, out=out, inc_shared=inc)
        return s["out"]
    if kind == "graph":
        s["graph"].replay()
        return s["out"]
    if kind == "host":
        return s["stack"].step(s["X"], s["L"], s["out"])
    if kind == "block":
        h = s["h"].clone()          # the step's residual stream; the call updates it in place
        res = [layer.block(h[l], s["a"][l], s["post_norm"][l], s["router"][l], s["next_norm"][l])
               for l, layer in enumerate(s["layers"])]
        return [h, [r[0] for r in res], [r[1] for r in res]]
    layer = moe.MoELayer(n_expert=case["E"], k=case["k"], D=D, FF=FF, se0=case["se0"], se1=case["se1"])
    layer.load_gguf_blocks(*s["blocks"])
    return [layer.Wg, layer.Wu, layer.Wd] + ([layer.Sg, layer.Su, layer.Sd] if case["shared"] else [])


# ------------------------------------------------------------------------------------------------- bounds
def _load(case):
    """(distinct resident routed experts, resident assignments) of one layer, from a sample of the routing."""
    T, E, k = case["T"], case["E"], case["k"]
    rng = np.random.default_rng(0)
    n = min(T, 4096)
    L = rng.standard_normal((n, E), dtype=np.float32)
    if case["zipf"]:
        L += _zipf_bias(E).numpy()
    idx = np.argpartition(-L, k - 1, axis=1)[:, :k]
    mine = idx[(idx >= case["se0"]) & (idx < case["se1"])]
    return np.unique(mine).size, mine.size * T / n


def work(case):
    E, T, NL = case["E"], case["T"], case["layers"]
    if case["kind"] == "load":       # blocks read, planes written
        return {"bytes": 2 * (case["se1"] - case["se0"] + case["shared"]) * EXPERT_BYTES, "flops": 0}
    experts, rows = _load(case)
    if case["shared"]:
        experts, rows = experts + 1, rows + T
    nbytes = experts * EXPERT_BYTES + T * D * 4                                  # weights touched, the output
    flops = rows * ASSIGNMENT_FLOPS
    if case["kind"] == "block":      # h in and out, a, x_next, the router matrix
        nbytes += 4 * T * D * 4 + (E + 1) * D * 4
        flops += 2 * T * D * (E + 1)
    else:
        nbytes += T * D * (2 if case["x"] == "bf16" else 4) + T * (E + 1) * 4
    return {"bytes": nbytes * NL, "flops": flops * NL}


def tolerance(case):
    if case["kind"] == "load":
        return "exact"
    if case["kind"] == "block":
        # on top of the below: the router's logits are sums of 2048 products in f32, so two experts that tie to the last
        # bits may change places for a token, which then sees another eighth expert
        return {"rel": 5e-3, "max": 0.9}
    # f32 sums, but the intermediate passes through E4M3 (3 mantissa bits): a SwiGLU value that sits on a rounding
    # boundary may land on either side, which moves its row by about 1e-3
    return {"rel": 1e-3}
