"""The work whose speed counts: what users of ruquant_b200 have it do, as cases that can be prepared and run.

Two kinds of work go through the public entry points.  "node" is the ggml MUL_MAT node -- `mul_mat` on one to three
prepared weights that share an activation -- alone, or as the nodes of decoder layers of the 27B shape (q, k, v / o /
gate, up / down), called one by one or replayed from a CUDA graph as ggml-cuda does when it decodes.  "convert" is the
weight quantizer, `quantize_weights`, that turns fp32 rows into the blocks such a node multiplies by.

Fields of a node case
    layers   0: one node of the given K, N; else this many decoder layers of the 27B shape (K = N = 0)
    K, N     input width and weight rows per weight;  n_w: weights of the node, 1 to 3
    M        tokens
    had      W4A4H (online Hadamard rotation) or plain W4A4;  rot_blocks: blocks of a block-diagonal rotation
    wgroup   weight multipliers: 0 none, 256 per block, 64 per 64 inputs;  group: inputs per activation group
    clip     activation clip in the weights' headers, 0: unset
    x        distribution of the activations
    graph    the nodes are replayed from a CUDA graph
    kept     outputs and workspaces are kept by the caller; else every call makes its own (the call's defaults)
"""
import math

import numpy as np
import torch

import ruquant_b200 as rq
from ruquant_b200 import synth

# the nodes of a decoder layer: matmuls that share an activation are one node
LAYER = [(5120, (6144, 1024, 1024)), (6144, (5120,)), (5120, (17408, 17408)), (17408, (5120,))]

NODE = {"do": "node", "layers": 0, "K": 0, "N": 0, "n_w": 1, "M": 1, "had": True, "rot_blocks": 1, "wgroup": 0, "group": 64,
        "clip": 0.0, "x": "normal", "graph": False, "kept": True}
CONVERT = {"do": "convert", "K": 0, "N": 0, "had": True, "rot_blocks": 1, "wgroup": 0}


def node(name, **over):
    return dict(NODE, name=name, **over)


def listed():
    return [
        # the smallest call there is, with every default: one token, a small unrotated weight
        node("call_m1_4096x1024", K=4096, N=1024, had=False, kept=False),
        # one token through a decoder layer, node by node from the host: no graph, as while a graph is not yet captured
        node("decode_layer_m1", layers=1),
        # single-stream decoding: the captured graph of a few layers
        node("decode_graph_m1", layers=4, graph=True),
        # decoding for a handful of sequences, or verifying a draft of a few tokens
        node("decode_graph_m8", layers=2, M=8, x="outliers", clip=0.9, graph=True),
        # a batch of sequences at the widest decode pass
        node("decode_graph_m16", layers=2, M=16, x="outliers", clip=0.9, graph=True),
        # a ragged batch between decode and prefill: many sequences, or the end of a prompt
        node("batch_m47_layer", layers=1, M=47, x="outliers", clip=0.9),
        # the square projection at 64 tokens
        node("batch_m64_5120x5120", K=5120, N=5120, M=64, x="outliers", clip=0.9),
        # a prompt in llama.cpp's default micro-batches of 512 tokens
        node("prefill_m512_layer", layers=1, M=512),
        # an odd number of tokens and rows, weights with a multiplier per 64 inputs, another Hadamard order (44 x 256)
        node("ragged_m777_11264x3001", K=11264, N=3001, M=777, wgroup=64, clip=0.95),
        # long prompts: the gate / up and the down projection
        node("prefill_m4096_5120x17408", K=5120, N=17408, M=4096, x="heavy"),
        node("prefill_m4096_17408x5120", K=17408, N=5120, M=4096, x="spikes", clip=0.9),
        # converting one tensor of a model
        dict(CONVERT, name="convert_5120x17408", K=5120, N=17408),
    ]


# input widths of the tests and the benchmark, with the blocks their rotation needs when the whole width has no
# factorisation (p * 2^k with p in 1, 12, 20, 44, 60, 68, 72, 84, 104, 108)
WIDTHS = [256, 512, 1024, 2048, 3072, 4096, 5120, 6144, 8192, 11008, 11264, 15360, 17408, 18432, 21504, 26624, 27648, 32768]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.12:
        K = rng.choice([w for w in WIDTHS if w != 11008])
        return dict(CONVERT, K=K, N=max(1, min(log_uniform(rng, 64, 17408), 5120 * 17408 // K)), had=rng.random() < 0.7,
                    wgroup=rng.choice([0, 0, 256, 64]))
    c = dict(NODE)
    if rng.random() < 0.3:
        c["layers"] = rng.choice([1, 2])
        c["M"] = log_uniform(rng, 1, 890 // c["layers"])
        c["graph"] = c["M"] <= 64 and rng.random() < 0.6
    else:
        c["K"] = rng.choice(WIDTHS)
        c["N"] = log_uniform(rng, 16, 17408)
        if rng.random() < 0.5:
            c["N"] = (c["N"] + 63) // 64 * 64
        c["n_w"] = rng.choice([1, 1, 1, 2, 3])
        # the largest listed node is 4096 tokens of 5120 x 17408
        c["M"] = max(1, min(log_uniform(rng, 1, 4096), 4096 * 5120 * 17408 // (c["K"] * c["N"] * c["n_w"])))
        c["had"] = c["K"] != 11008 and rng.random() < 0.75
        if c["had"] and c["K"] % 1024 == 0 and rng.random() < 0.15:
            c["rot_blocks"] = 2
        c["graph"] = c["M"] <= 64 and rng.random() < 0.3
        c["kept"] = c["graph"] or rng.random() < 0.8
    c["wgroup"] = rng.choice([0, 0, 0, 256, 64])
    c["group"] = 64 if c["wgroup"] == 64 else rng.choice([64, 64, 64, 128, 256])
    c["clip"] = rng.choice([0.0, 0.0, 0.9, round(rng.uniform(0.8, 1.0), 3)])
    c["x"] = rng.choice(["normal", "outliers", "heavy", "spikes"])
    return c


def activations(kind, M, K, gen):
    x = torch.randn((M, K), generator=gen, device="cuda", dtype=torch.float32)
    if kind == "outliers":          # a few channels carry large values for every token
        cols = torch.randint(0, K, (8,), generator=gen, device="cuda")
        x[:, cols] *= 40.0
    elif kind == "heavy":           # Student's t with three degrees of freedom, and outlier channels
        chi2 = sum(torch.randn((M, K), generator=gen, device="cuda", dtype=torch.float32) ** 2 for _ in range(3))
        x /= (chi2 / 3.0).clamp_min_(1e-6).sqrt_()
        cols = torch.randint(0, K, (16,), generator=gen, device="cuda")
        x[:, cols] *= 50.0
    elif kind == "spikes":          # one entry in a hundred is +-30
        at = torch.rand((M, K), generator=gen, device="cuda") < 0.01
        x = torch.where(at, torch.sign(x) * 30.0, x)
    return x.contiguous()


def make_weight(case, K, N, seed):
    type_ = rq.TYPE_W4A4H if case["had"] else rq.TYPE_W4A4
    blocks = synth.random_weights(N, K, type_, seed=seed, wgroup=case["wgroup"], rot_blocks=case["rot_blocks"])
    if case["clip"] > 0:            # the second padding word of a block's 16-byte header
        word = np.array([case["clip"]], dtype=np.float32).view(np.uint8)
        blocks.view(N, K // 256, 144)[:, :, 12:16] = torch.from_numpy(word.copy()).cuda()
    w = rq.Weight(blocks.view(-1), type_, K, N=N)
    w.blocks = None                 # the kernels read only the prepared layouts
    return w


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["do"] == "convert":
        return {"case": case, "w": torch.randn((case["N"], case["K"]), generator=gen, device="cuda", dtype=torch.float32) * 0.02}
    shapes = LAYER * case["layers"] if case["layers"] else [(case["K"], (case["N"],) * case["n_w"])]
    nodes = []
    for i, (K, rows) in enumerate(shapes):
        weights = [make_weight(case, K, N, seed * 1000 + 10 * i + j) for j, N in enumerate(rows)]
        x = activations(case["x"], case["M"], K, gen)
        outs = ws = None
        if case["kept"]:
            outs = [torch.empty((case["M"], N), device="cuda", dtype=torch.float32) for N in rows]
            ws = rq.new_workspace(K, case["M"])
        nodes.append((weights, x, outs, ws))
    state = {"case": case, "nodes": nodes, "graph": None}
    if case["graph"]:
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            run_nodes(state)        # first launches, before the capture
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                run_nodes(state)
        torch.cuda.current_stream().wait_stream(stream)
        state["graph"] = graph
    return state


def run_nodes(state):
    group = state["case"]["group"]
    return [rq.mul_mat(weights, x, out=outs, act_group=group, workspace=ws) for weights, x, outs, ws in state["nodes"]]


def run(state):
    case = state["case"]
    if case["do"] == "convert":
        return rq.quantize_weights(state["w"], rq.TYPE_W4A4H if case["had"] else rq.TYPE_W4A4, case["wgroup"], case["rot_blocks"])
    if state["graph"] is not None:
        state["graph"].replay()
        return [outs for _, _, outs, _ in state["nodes"]]
    return run_nodes(state)


def rotation_ops(case, K):
    """fp32 additions per input of the online rotation: log2(m) butterflies and p Paley terms."""
    if not case["had"]:
        return 0
    p, m = rq.hadamard_factor(K // case["rot_blocks"])
    return int(math.log2(m)) + (p if p > 1 else 0)


def work(case):
    if case["do"] == "convert":
        K, N = case["K"], case["N"]
        # rows in, blocks out; thirteen candidate scales per weight, each a division, a rounding, a product and a squared error
        return {"bytes": 4 * N * K + N * (K // 256) * 144, "flops": N * K * (13 * 6 + rotation_ops(case, K))}
    shapes = LAYER * case["layers"] if case["layers"] else [(case["K"], (case["N"],) * case["n_w"])]
    M, nbytes, flops = case["M"], 0, 0
    for K, rows in shapes:
        nbytes += 4 * M * K + sum(N * (K // 256) * 144 + 4 * M * N for N in rows)
        flops += M * K * rotation_ops(case, K) + sum(2 * M * K * N for N in rows)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # integer sums, and fp32 operations whose order is part of the format: every correct implementation gives the same bits
    return "exact"
