"""The work that users of this library have it do, as cases that can be timed and checked: radius graphs, PaiNN and l<=2
message layers (inference in FP32 and on the BF16 tensor-core path, and training), whole denoiser steps, and proximity
attention. Sizes are those of the benchmark workloads, the configurations and the tests, or smaller and larger systems of
the same density.

A case is a dict of plain values. `prepare` makes what a program holds before the call (inputs, weights, edge list),
`run` is one pass through the public entry points, `exact` the same outputs from plain torch in 64 bits."""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "learned-dynamics_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from ld_b200 import bee, painn  # noqa: E402
from ld_b200.graph import RadiusGraphBuilder  # noqa: E402
from ld_b200.graph_layers import Graph  # noqa: E402
from ld_b200.proxattn import proxattn, proxattn_periodic  # noqa: E402

DEV = "cuda"
V_ORDER = ("011", "101", "121", "211", "111")
D_ORDER = ("022", "202", "112", "222", "212")
BEE_DIMS = {"wide": (128, 64, 32, 128), "narrow": (64, 32, 32, 64)}   # dim_a, dim_v, dim_d, product channels


def listed():
    return [
        # the neighbour list of a few short open polymers: the smallest call, latency and launches count
        {"name": "graph_open_small", "kind": "graph", "systems": 8, "nodes": 64, "box": 0.0, "cutoff": 3.0, "shift": False},
        # the neighbour list of a batch of dense periodic boxes, with lattice shifts (benchmark config 1)
        {"name": "graph_periodic", "kind": "graph", "systems": 32, "nodes": 4096, "box": 16.0, "cutoff": 2.5, "shift": True},
        # one message layer of the dense periodic rollout on the tensor-core path
        {"name": "painn_layer_bf16", "kind": "painn_layer", "precision": "bf16", "systems": 4, "nodes": 2048, "density": 1.024,
         "cutoff": 4.0, "n": 128, "n_rbf": 8, "radial": "gaussian"},
        # the same layer at the default precision, one smaller box
        {"name": "painn_layer_fp32", "kind": "painn_layer", "precision": "fp32", "systems": 1, "nodes": 2048, "density": 1.024,
         "cutoff": 4.0, "n": 128, "n_rbf": 8, "radial": "gaussian"},
        # one evaluation of the reference's denoiser (2 + 5 blocks, bonds, default precision) on short polymers
        {"name": "painn_step_fp32", "kind": "painn_step", "precision": "fp32", "systems": 8, "nodes": 64, "cutoff": 3.0, "n": 64},
        # one training pass of a PaiNN block (messages, update), gradients of inputs and weights
        {"name": "painn_block_train", "kind": "painn_train", "systems": 16, "nodes": 128, "cutoff": 3.0, "n": 64},
        # one l<=2 layer (messages, node-local products) of the polymer denoiser on the tensor-core path (benchmark config 2)
        {"name": "bee_layer_bf16", "kind": "bee_layer", "precision": "bf16", "systems": 64, "nodes": 512, "cutoff": 5.0, "dims": "wide"},
        # the same layer at the default precision, fewer systems
        {"name": "bee_layer_fp32", "kind": "bee_layer", "precision": "fp32", "systems": 4, "nodes": 512, "cutoff": 5.0, "dims": "wide"},
        # one evaluation of the 6-layer l<=2 denoiser for the polymers of config 4, a small batch of them
        {"name": "bee_step_bf16", "kind": "bee_step", "precision": "bf16", "systems": 16, "nodes": 256, "cutoff": 5.0, "depth": 6,
         "dims": "wide"},
        # one training pass of an l<=2 message layer, gradients of inputs and weights
        {"name": "bee_messages_train", "kind": "bee_train", "systems": 4, "nodes": 128, "cutoff": 5.0, "dims": "wide"},
        # dense proximity attention, inference on the tensor cores
        {"name": "proxattn_tf32", "kind": "proxattn", "precision": "tf32", "Z": 32, "N": 4096, "dim": 64, "heads": 4, "box": 0.0,
         "grad": False},
        # proximity attention in a periodic box as a training pass, default precision, a size that fills no tile
        {"name": "proxattn_train", "kind": "proxattn", "precision": "fp32", "Z": 16, "N": 1000, "dim": 32, "heads": 4, "box": 12.0,
         "grad": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("graph", "painn_layer", "painn_step", "painn_train", "bee_layer", "bee_step", "bee_train", "proxattn"))
    if kind == "graph":
        nodes = _log_int(rng, 40, 4096)
        systems = max(1, min(32, _log_int(rng, 300, 131072) // nodes))
        cutoff = round(rng.uniform(2.0, 3.5), 2)
        box = 0.0
        if rng.random() < 0.6:   # a periodic box holds at least three cutoffs
            box = round(max((nodes / rng.uniform(0.3, 1.0)) ** (1 / 3), 3.1 * cutoff), 2)
        return {"kind": kind, "systems": systems, "nodes": nodes, "box": box, "cutoff": cutoff, "shift": rng.random() < 0.5}
    if kind == "painn_layer":
        precision = rng.choice(("bf16", "fp32"))
        nodes = _log_int(rng, 150, 2048)
        systems = max(1, _log_int(rng, 150, 8192 if precision == "bf16" else 2048) // nodes)
        radial = rng.choice(("gaussian", "painn"))
        n = rng.choice((32, 64, 128))
        return {"kind": kind, "precision": precision, "systems": systems, "nodes": nodes, "density": round(rng.uniform(0.4, 1.02), 3),
                "cutoff": round(rng.uniform(2.0, 4.0) if nodes >= 1900 else rng.uniform(1.7, (nodes ** (1 / 3)) / 3.2), 2), "n": n,
                "n_rbf": rng.choice((8, 16, 20)) if radial == "gaussian" else rng.choice((16, n)), "radial": radial}
    if kind == "painn_step":
        nodes = _log_int(rng, 20, 128)
        return {"kind": kind, "precision": rng.choice(("fp32", "bf16")), "systems": _log_int(rng, 1, max(1, 600 // nodes)), "nodes": nodes,
                "cutoff": round(rng.uniform(2.5, 3.0), 2), "n": rng.choice((32, 64))}
    if kind == "painn_train":
        nodes = _log_int(rng, 30, 300)
        return {"kind": kind, "systems": max(1, _log_int(rng, 60, 2048) // nodes), "nodes": nodes, "cutoff": round(rng.uniform(2.0, 3.0), 2),
                "n": rng.choice((32, 64))}
    if kind == "bee_layer":
        precision = rng.choice(("bf16", "fp32"))
        nodes = _log_int(rng, 30, 512)
        systems = max(1, _log_int(rng, 100, 32768 if precision == "bf16" else 2048) // nodes)
        return {"kind": kind, "precision": precision, "systems": systems, "nodes": nodes, "cutoff": round(rng.uniform(3.0, 5.0), 2),
                "dims": rng.choice(("wide", "wide", "narrow"))}
    if kind == "bee_step":
        nodes = _log_int(rng, 30, 300)
        return {"kind": kind, "precision": "bf16", "systems": max(1, _log_int(rng, 60, 4096) // nodes), "nodes": nodes,
                "cutoff": round(rng.uniform(3.0, 5.0), 2), "depth": rng.choice((2, 4, 6)), "dims": rng.choice(("wide", "narrow"))}
    if kind == "bee_train":
        nodes = _log_int(rng, 30, 300)
        return {"kind": kind, "systems": max(1, _log_int(rng, 60, 512) // nodes), "nodes": nodes, "cutoff": round(rng.uniform(3.0, 5.0), 2),
                "dims": rng.choice(("wide", "narrow"))}
    grad = rng.random() < 0.5
    heads = rng.choice((1, 2, 4))
    box = 0.0 if rng.random() < 0.5 else round(rng.uniform(8.0, 20.0), 2)
    if grad:
        return {"kind": kind, "precision": "fp32", "Z": heads * rng.randint(1, 16 // heads), "N": _log_int(rng, 60, 1000),
                "dim": rng.choice((16, 32)), "heads": heads, "box": box, "grad": True}
    return {"kind": kind, "precision": rng.choice(("tf32", "fp32")), "Z": heads * rng.randint(1, 16 // heads), "N": _log_int(rng, 100, 2500),
            "dim": rng.choice((16, 32, 64)), "heads": heads, "box": box, "grad": False}


# ---- inputs ------------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 + int(seed))


def _polymers(systems, nodes, g):
    """open chains with unit bond length (1/sqrt(3) per axis)"""
    return torch.cumsum(torch.randn(systems, nodes, 3, generator=g, device=DEV) / 3 ** 0.5, dim=1)


def _edges(pos, box, cutoff):
    """all ordered pairs of a system within the cutoff, sorted by source: flat int64 src, dst, and the displacements in the
    precision of pos"""
    B, N, _ = pos.shape
    src, dst, rij = [], [], []
    for b in range(B):
        d = pos[b][None, :, :] - pos[b][:, None, :]
        if box:
            d = d - box * torch.round(d / box)
        near = (d.double() ** 2).sum(-1) <= cutoff * cutoff
        near.fill_diagonal_(False)
        i, j = near.nonzero(as_tuple=True)
        src.append(i + b * N)
        dst.append(j + b * N)
        rij.append(d[i, j])
    return torch.cat(src), torch.cat(dst), torch.cat(rij)


class _Weights:
    """named weights in the order they are asked for, with torch's default distributions"""

    def __init__(self, g):
        self.g, self.d = g, {}

    def uniform(self, name, shape, bound):
        self.d[name] = (torch.rand(*shape, generator=self.g, device=DEV) * 2 - 1) * bound

    def normal(self, name, shape, std):
        self.d[name] = torch.randn(*shape, generator=self.g, device=DEV) * std

    def const(self, name, shape, value):
        self.d[name] = torch.full(shape, float(value), device=DEV)

    def linear(self, name, dim_in, dim_out, bias=True):
        self.uniform(name + ".weight", (dim_out, dim_in), dim_in ** -0.5)
        if bias:
            self.uniform(name + ".bias", (dim_out,), dim_in ** -0.5)

    def tens(self, name, dim_in, dim_out):
        self.normal(name + ".W", (dim_out, dim_in), dim_in ** -0.5)

    def mlp(self, name, dim_in, dim_out):
        for k, d in ((0, dim_in), (2, dim_out), (4, dim_out)):
            self.linear(f"{name}.layers.{k}", d, dim_out)

    def painn_message(self, p, n, n_rbf):
        self.mlp(p + "mlp_dist", n_rbf, 4 * n)
        self.mlp(p + "mlp_actv", n, 4 * n)

    def painn_block(self, p, n, n_rbf):
        self.painn_message(p + "message.", n, n_rbf)
        self.painn_message(p + "message_bond.", n, n_rbf)
        for k in ("lin_l", "lin_r", "lin_v"):
            self.tens(p + "update." + k, n, n)
        self.mlp(p + "update.mlp", 2 * n, 3 * n)
        self.const(p + "update.gn.gamma", (n,), 1)
        self.const(p + "update.gn.beta", (n,), 0)

    def bee_y(self, p, a, v, d, chan):
        for names, width in ((("000", "110", "220"), a), (V_ORDER, v), (D_ORDER, d)):
            for k in names:
                self.tens(p + "Y_" + k, chan, width)

    def bee_messages(self, p, a, v, d, chan):
        for k, width in (("L0", a), ("L1", v), ("L2", d)):
            self.tens(p + k, width, chan)
        self.bee_y(p, a, v, d, chan)
        self.linear(p + "lin_enc", 8, chan)
        self.linear(p + "mlp_a.lin_direct", a, a, bias=False)
        for k, i, o in ((0, a, 2 * a), (2, 2 * a, 2 * a), (4, 2 * a, a)):
            self.linear(f"{p}mlp_a.layers.{k}", i, o)

    def bee_block(self, p, a, v, d, chan):
        self.bee_messages(p + "messages.", a, v, d, chan)
        for side in ("L", "R"):
            for k, width in (("0", a), ("1", v), ("2", d)):
                self.tens(p + "prods." + side + k, width, chan)
        self.bee_y(p + "prods.", a, v, d, chan)
        for k, (name, width) in enumerate((("a", a), ("v", v), ("d", d))):
            self.const(f"{p}prods.gn_{name}.gamma", (width,) + (1,) * k, 1)


def _rbf(c):
    return c.get("n_rbf") or c["n"]


def _inputs(c, seed):
    """everything that prepare and exact share: tensors made from the seed"""
    g, kind, s = _gen(seed), c["kind"], {}
    w = _Weights(g)
    if kind == "proxattn":
        Z, N, D = c["Z"], c["N"], c["dim"]
        for k in ("Q", "K", "V"):
            s[k] = torch.randn(Z, N, D, generator=g, device=DEV)
        pos = torch.rand(Z, N, 3, generator=g, device=DEV) * (c["box"] or 12.0)
        s["X"], s["Y"] = pos, pos + 0.1 * torch.randn(Z, N, 3, generator=g, device=DEV)
        s["r0sq"] = 1.0 + 3.0 * torch.rand(c["heads"], generator=g, device=DEV)
        s["dO"] = torch.randn(Z, N, D, generator=g, device=DEV)
        return s
    B, N = c["systems"], c["nodes"]
    box = 0.0
    if kind == "graph":
        box = c["box"]
    elif kind == "painn_layer":
        box = (N / c["density"]) ** (1 / 3)
    pos = torch.rand(B, N, 3, generator=g, device=DEV) * box if box else _polymers(B, N, g)
    s.update(pos=pos, box=box)
    if kind == "graph":
        return s
    if kind.endswith("step"):
        s["noise"] = torch.randn(B, N, 3, generator=g, device=DEV)
        s["start"] = 0.4 * torch.rand(B, generator=g, device=DEV)
        s["end"] = s["start"] + 0.1 + 0.4 * torch.rand(B, generator=g, device=DEV)
        s["types"] = torch.randint(0, 20, (N,), generator=g, device=DEV)
    else:
        s["src"], s["dst"], s["rij"] = _edges(pos, box, c["cutoff"])
    if kind.startswith("painn"):
        n, r = c["n"], _rbf(c)
        if kind == "painn_step":
            w.normal("atom_embeddings", (N, n), 1.0)
            w.linear("t_embed.lin1", 128, n)
            w.mlp("mlp_embed", n, n)
            w.mlp("mlp_denoise", n, n)
            w.tens("pos_emb.lin_v", 1, n)
            for name, blocks in (("cpainn_0", 2), ("cpainn_1", 5)):
                w.normal(name + ".atom_embed.weight", (20, n), 1.0)
                for k in range(blocks):
                    w.painn_block(f"{name}.blocks.{k}.", n, r)
            w.tens("v_readin", 1, n)
            w.tens("readout", n, 1)
        elif kind == "painn_layer":
            w.painn_message("", n, r)
        else:
            w.painn_block("", n, r)
        if kind != "painn_step":
            s["x_a"] = torch.randn(B, N, n, generator=g, device=DEV)
            s["x_v"] = torch.randn(B, N, n, 3, generator=g, device=DEV)
        widths = [("a", (n,)), ("v", (n, 3))]
    else:
        a, v, d, chan = BEE_DIMS[c["dims"]]
        if kind == "bee_step":
            w.normal("type_embed.weight", (20, a), 1.0)
            w.tens("v_readin", 1, v)
            for k in range(c["depth"]):
                w.bee_block(f"blocks.{k}.", a, v, d, chan)
            w.tens("readout", v, 1)
        elif kind == "bee_layer":
            w.bee_block("", a, v, d, chan)
        else:
            w.bee_messages("", a, v, d, chan)
        if kind != "bee_step":
            s["x_a"] = torch.randn(B, N, a, generator=g, device=DEV)
            s["x_v"] = torch.randn(B, N, v, 3, generator=g, device=DEV)
            s["x_d"] = torch.randn(B, N, d, 3, 3, generator=g, device=DEV)
        widths = [("a", (a,)), ("v", (v, 3)), ("d", (d, 3, 3))]
    if kind.endswith("train"):   # the gradient that arrives from the layers above
        for k, shape in widths:
            s["g_" + k] = torch.randn(B, N, *shape, generator=g, device=DEV)
    s["w"] = w.d
    return s


def prepare(case, seed):
    c, s = case, _inputs(case, seed)
    s["case"], kind = c, c["kind"]
    if kind == "proxattn":
        if c["grad"]:
            for k in ("Q", "K", "V", "X", "Y"):
                s[k].requires_grad_(True)
        return s
    B, N = c["systems"], c["nodes"]
    if kind == "graph":
        # the rollout's form: buffers of a fixed capacity that every step reuses
        s["builder"] = RadiusGraphBuilder(B, N, c["cutoff"], (s["box"],) * 3 if s["box"] else None, device=DEV)
        cap = int(min(B * N * (N - 1), 2 * B * N * _degree(c) + 1024))
        s["src"], s["dst"] = (torch.zeros(cap, dtype=torch.int32, device=DEV) for _ in range(2))
        s["shift"] = torch.zeros(cap, dtype=torch.int32, device=DEV) if c["shift"] else None
        s["rij_out"] = torch.zeros(cap, 3, device=DEV)
        return s
    if kind == "painn_layer":
        m = painn.Message(c["cutoff"], c["n"], c["n_rbf"], c["radial"])
    elif kind == "painn_step":
        m = painn.SE3ITO(c["cutoff"], c["n"], N, ntypes=20)
    elif kind == "painn_train":
        m = painn.Block(c["cutoff"], c["n"])
    elif kind == "bee_layer":
        m = bee.BeeBlock(c["cutoff"], *BEE_DIMS[c["dims"]])
    elif kind == "bee_step":
        m = bee.BeeDenoiser(c["cutoff"], *BEE_DIMS[c["dims"]], ntypes=20, depth=c["depth"])
    else:
        m = bee.Messages(c["cutoff"], *BEE_DIMS[c["dims"]])
    m = m.to(DEV)
    m.load_state_dict(s.pop("w"))
    (painn if kind.startswith("painn") else bee).set_precision(m, c.get("precision", "fp32"))
    s["model"] = m
    if kind == "painn_step":
        s["bonds"] = painn.chain_bond_graph(B, N, DEV)
    elif kind != "bee_step":
        s["graph"] = Graph(s.pop("src"), s.pop("dst"), None, B, N)
        s["graph"].row_ptr
    if kind == "painn_train":
        s["bonds"] = painn.chain_bond_graph(B, N, DEV)
        flat = s["pos"].reshape(-1, 3)
        s["rij_bond"] = flat[s["bonds"].dst] - flat[s["bonds"].src]
    if kind.endswith("train"):
        for k in ("x_a", "x_v", "x_d"):
            if k in s:
                s[k].requires_grad_(True)
    return s


def _grads(outs, grads, s, keys):
    """outputs, then the gradients of the inputs `keys` and of the weights"""
    leaves = [s[k] for k in keys] + list(s["model"].parameters())
    return list(outs) + list(torch.autograd.grad(outs, leaves, grads))


def run(state):
    s = state
    c, kind = s["case"], s["case"]["kind"]
    if kind == "graph":
        b = s["builder"]
        b.build_fixed(s["pos"], s["src"].numel(), s["src"], s["dst"], s["shift"], s["rij_out"])
        return [b.row_ptr, b.edge_counts, s["src"], s["dst"], s["rij_out"]] + ([s["shift"]] if c["shift"] else [])
    if kind == "proxattn":
        qkv = (s["Q"], s["K"], s["V"], s["X"], s["Y"])
        call = (lambda: proxattn_periodic(*qkv, s["r0sq"], (c["box"],) * 3, precision=c["precision"])) if c["box"] else \
            (lambda: proxattn(*qkv, s["r0sq"], precision=c["precision"]))
        if not c["grad"]:
            with torch.no_grad():
                return call()
        out = call()
        return [out.detach()] + list(torch.autograd.grad(out, qkv, s["dO"]))
    if kind == "painn_train":
        pos = s["pos"]
        out = s["model"]((pos, s["graph"], s["rij"], s["bonds"], s["rij_bond"], s["x_a"], s["x_v"], None))
        return _grads((out[5], out[6]), (s["g_a"], s["g_v"]), s, ("x_a", "x_v"))
    if kind == "bee_train":
        outs = s["model"](s["graph"], s["rij"], s["x_a"], s["x_v"], s["x_d"])
        return _grads(outs, (s["g_a"], s["g_v"], s["g_d"]), s, ("x_a", "x_v", "x_d"))
    with torch.no_grad():
        if kind == "painn_layer":
            return list(s["model"](s["graph"], s["x_a"], s["x_v"], s["rij"]))
        if kind == "bee_layer":
            return list(s["model"](s["graph"], s["rij"], s["x_a"], s["x_v"], s["x_d"]))
        if kind == "bee_step":
            return s["model"](s["pos"], s["pos"] + 0.05 * s["noise"], None, s["types"])
        return s["model"]((s["start"], s["end"]), s["pos"], s["pos"] + 0.05 * s["noise"], None, s["types"], s["bonds"])


# ---- work and tolerances -----------------------------------------------------------------------------------------------

def _degree(c):
    """expected neighbours of a node: uniform density in a box; for chains with bond steps N(0, 1/3) per axis, the sum of
    P(|r| < cutoff) over the separations along the chain"""
    N, rc = c["nodes"], c["cutoff"]
    if c["kind"] == "painn_layer":
        return min(N - 1, c["density"] * 4 / 3 * math.pi * rc ** 3)
    if c.get("box"):
        return min(N - 1, N / c["box"] ** 3 * 4 / 3 * math.pi * rc ** 3)
    t = 0.0
    for k in range(1, N):
        x = rc / (2 * k / 3) ** 0.5   # radius over sqrt(2) standard deviations
        t += 2 * (1 - k / N) * (math.erf(x) - 2 / math.pi ** 0.5 * x * math.exp(-x * x))
    return t


def work(case):
    """bytes: inputs once and outputs once; flops: those of the factored form of each layer (node-level mixings once per node,
    what is linear in the edges' products once per node, the rest per edge)"""
    c, kind = case, case["kind"]
    if kind == "proxattn":
        Z, N, D = c["Z"], c["N"], c["dim"]
        tensors, products = (4, 2) if not c["grad"] else (8, 7)   # forward; with gradients also dO, dQ, dK, dV
        return {"bytes": 4 * Z * N * (tensors * D + 6 * (2 if c["grad"] else 1)), "flops": Z * N * N * (2 * D * products + 12)}
    Nt = c["systems"] * c["nodes"]
    E = Nt * _degree(c)
    if kind == "graph":
        return {"bytes": 16 * Nt + E * (20 + (4 if c["shift"] else 0)), "flops": 8 * E}
    if kind.startswith("painn"):
        n, r = c["n"], _rbf(c)
        edge = 2 * (r * 4 * n + 32 * n * n) + 30 * n
        node = 2 * (4 * n * n + 32 * n * n)
        update = 2 * (9 * n * n + 6 * n * n + 18 * n * n)
        rows = 4 * n * 4 * Nt   # x_a and x_v once
        weights = 4 * (r * 4 * n + 68 * n * n)
        if kind == "painn_layer":
            return {"bytes": 16 * E + 2 * rows + weights, "flops": E * edge + Nt * node}
        Eb = 2 * c["systems"] * (c["nodes"] - 1)
        block = (E + Eb) * edge + Nt * (2 * node + update)
        if kind == "painn_train":
            return {"bytes": 16 * (E + Eb) + 4 * rows + 2 * (2 * weights + 4 * 33 * n * n), "flops": 3 * block}
        return {"bytes": 7 * (2 * weights + 4 * 33 * n * n) + 12 * Nt * 3, "flops": 7 * block}
    a, v, d, C = BEE_DIMS[c["dims"]]
    feats = a + 3 * v + 9 * d
    y = 3 * C * a + 15 * C * v + 45 * C * d
    edge = 2 * (8 * C + 3 * C * a + 9 * a * a) + 120 * C
    left = C * feats
    msg_w = 4 * ((a + v + d) * C + 3 * C * a + 5 * C * (v + d) + 9 * a * a)
    prod_w = 4 * (2 * (a + v + d) * C + 3 * C * a + 5 * C * (v + d))
    messages = E * edge + Nt * 2 * (left + y - 3 * C * a)
    products = Nt * (2 * (2 * left + y) + 300 * C)
    if kind == "bee_train":
        return {"bytes": 16 * E + 4 * feats * 4 * Nt + 2 * msg_w, "flops": 3 * messages}
    if kind == "bee_layer":
        return {"bytes": 16 * E + 2 * feats * 4 * Nt + msg_w + prod_w, "flops": messages + products}
    return {"bytes": c["depth"] * (msg_w + prod_w) + 12 * Nt * 3, "flops": c["depth"] * (messages + products)}


def tolerance(case):
    c, kind = case, case["kind"]
    if kind == "graph":
        return "exact"
    return dict(TOLERANCE[kind if kind.endswith("train") else kind + "_" + c["precision"]])


# about four times the distance from the 64-bit result, seen over the listed and some forty drawn cases (bee_train: the weight
# gradients of the scalar products, where an activation's kink falls between two roundings)
TOLERANCE = {
    "painn_layer_bf16": {"rel": 0.02, "max": 0.8},
    "painn_layer_fp32": {"rel": 4e-6},
    "painn_step_fp32": {"rel": 2.5e-5},
    "painn_step_bf16": {"rel": 0.03, "max": 0.8},
    "painn_train": {"rel": 1e-5},
    "bee_layer_bf16": {"rel": 0.0125, "max": 0.5},
    "bee_layer_fp32": {"rel": 4e-6},
    "bee_step_bf16": {"rel": 0.025, "max": 0.8},
    "bee_train": {"rel": 1.5e-4},
    "proxattn_tf32": {"rel": 2.5e-3, "max": 0.1},
    "proxattn_fp32": {"rel": 4e-6},
}


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------------------

def _tens(W, x, inds):
    """channel mixing of (..., chan, (3,)*inds)"""
    if inds == 0:
        return x @ W.t()
    y = torch.tensordot(x, W, dims=([x.dim() - 1 - inds], [1]))   # the mixed axis comes last
    return y.movedim(-1, x.dim() - 1 - inds)


def _mlp(w, p, x, act):
    for k in (0, 2, 4):
        x = torch.nn.functional.linear(x, w[f"{p}.layers.{k}.weight"], w[f"{p}.layers.{k}.bias"])
        x = act(x) if k < 4 else x
    return x


def _painn_radial(c, rij):
    n, rc, dist = _rbf(c), c["cutoff"], rij.norm(dim=-1, keepdim=True)
    if c.get("radial") == "gaussian":
        width = rc / (n - 1)
        mu = torch.arange(n, dtype=rij.dtype, device=DEV) * width
        env = torch.where(dist < rc, 0.5 * (torch.cos(math.pi * dist / rc) + 1), torch.zeros_like(dist))
        return torch.exp(-0.5 * ((dist - mu) / width) ** 2) * env
    half = (n + 1) // 2
    phase = (math.pi / rc) * (1 + torch.arange(half, device=DEV) // 2) * dist
    return torch.cat([torch.cos(phase), torch.sin(phase[..., :n - half])], dim=-1)


def _pieces(E, width):
    step = max(1, int(1.5e8 / width))
    return [(k, min(E, k + step)) for k in range(0, E, step)]


def _painn_message(c, w, p, src, dst, rij, x_a, x_v):
    """messages summed per node, on flat node rows"""
    n, silu = c["n"], torch.nn.functional.silu
    actv = _mlp(w, p + "mlp_actv", x_a, silu)
    d_a, d_v = torch.zeros_like(x_a), torch.zeros_like(x_v)
    for lo, hi in _pieces(len(src), 16 * n):
        i, j, r = src[lo:hi], dst[lo:hi], rij[lo:hi]
        P = _mlp(w, p + "mlp_dist", _painn_radial(c, r), silu) * actv[j]
        u = (r / torch.sqrt(0.1 + (r ** 2).sum(-1, keepdim=True)))[:, None, :]
        xe = x_v[j]
        m = xe * P[:, :n, None] + torch.linalg.cross(xe, u.expand_as(xe)) * P[:, n:2 * n, None] + u * P[:, 2 * n:3 * n, None]
        d_v = d_v.index_add(0, i, m)
        d_a = d_a.index_add(0, i, P[:, 3 * n:])
    return d_a, d_v


def _painn_block(c, w, p, B, edges, bonds, x_a, x_v):
    n = c["n"]
    for name, graph in (("message_bond.", bonds), ("message.", edges)):
        d_a, d_v = _painn_message(c, w, p + name, *graph, x_a, x_v)
        x_a, x_v = x_a + d_a, x_v + d_v
    q = p + "update."
    left, right = _tens(w[q + "lin_l.W"], x_v, 1), _tens(w[q + "lin_r.W"], x_v, 1)
    y = _mlp(w, q + "mlp", torch.cat([x_a, right.norm(dim=-1)], dim=-1), torch.nn.functional.silu)
    d_v = _tens(w[q + "lin_v.W"], x_v, 1) * y[:, :n, None]
    h = ((left * right).sum(-1) * y[:, n:2 * n]).reshape(B, -1, 4, n // 4)
    h = h - h.mean([1, 3], keepdim=True)
    h = (h / torch.sqrt(1.0 + (h ** 2).mean([1, 3], keepdim=True))).reshape(-1, n)
    d_a = w[q + "gn.beta"] + w[q + "gn.gamma"] * h + y[:, 2 * n:]
    return x_a + d_a, x_v + d_v / torch.sqrt(1 + (d_v ** 2).sum(-1, keepdim=True))


def _jacobi(z):
    """shifted Jacobi(1, 0) polynomials of degrees 0..7 on [0, 1]"""
    out = []
    for n in range(8):
        t = torch.zeros_like(z)
        for k in range(n + 1):
            t = t + math.comb(n + 1, n - k) * math.comb(n, k) * (z - 1) ** k * z ** (n - k)
        out.append(t)
    return torch.cat(out, dim=-1)


def _bee_products(l, r):
    """the 13 products, grouped by the rank of the result"""
    l0, l1, l2 = l
    r0, r1, r2 = r
    e = torch.einsum
    a = {"000": l0 * r0, "110": (l1 * r1).sum(-1), "220": (l2 * r2).sum((-1, -2))}
    v = {"011": l0[..., None] * r1, "101": l1 * r0[..., None], "121": e("ncx,ncyx->ncy", l1, r2), "211": e("ncxy,ncy->ncx", l2, r1),
         "111": torch.linalg.cross(l1, r1)}
    d = {"022": l0[..., None, None] * r2, "202": l2 * r0[..., None, None], "112": l1[..., :, None] * r1[..., None, :],
         "222": e("ncxy,nczy->ncxz", l2, r2), "212": torch.linalg.cross(l2, r1[..., None, :].expand_as(l2))}
    return a, v, d


def _bee_mix(w, p, products):
    return [sum(_tens(w[p + "Y_" + k + ".W"], y, rank) for k, y in group.items()) for rank, group in enumerate(products)]


def _bee_messages(c, w, p, src, dst, rij, x):
    left = [_tens(w[f"{p}L{k}.W"], x[k], k) for k in range(3)]
    out = [torch.zeros_like(t) for t in x]
    leaky = lambda t: torch.nn.functional.leaky_relu(t, 0.1)  # noqa: E731
    for lo, hi in _pieces(len(src), 100 * BEE_DIMS[c["dims"]][3]):
        i, j, r = src[lo:hi], dst[lo:hi], rij[lo:hi]
        z = r.norm(dim=-1, keepdim=True) / c["cutoff"]
        phi = torch.nn.functional.linear(_jacobi(z) * torch.relu(1 - z), w[p + "lin_enc.weight"], w[p + "lin_enc.bias"])
        u = r * (7.0 / c["cutoff"])
        u = (u / torch.sqrt(1 + (u ** 2).sum(-1, keepdim=True)))[:, None, :]
        pv = phi[..., None] * u
        psi = _bee_mix(w, p, _bee_products([t[j] for t in left], (phi, pv, pv[..., :, None] * u[..., None, :])))
        psi[0] = psi[0] + psi[0] @ w[p + "mlp_a.lin_direct.weight"].t() + _mlp(w, p + "mlp_a", psi[0], leaky)
        out = [o.index_add(0, i, 0.1 * m) for o, m in zip(out, psi)]
    return out


def _bee_block(c, w, p, B, edges, x):
    x = [t + m for t, m in zip(x, _bee_messages(c, w, p + "messages.", *edges, x))]
    q = p + "prods."
    ys = [[] for _ in range(3)]
    for lo, hi in _pieces(len(x[0]), 100 * BEE_DIMS[c["dims"]][3]):
        sides = [[_tens(w[f"{q}{s}{k}.W"], x[k][lo:hi], k) for k in range(3)] for s in "LR"]
        for y, t in zip(ys, _bee_mix(w, q, _bee_products(*sides))):
            y.append(t)
    out = []
    for k, (name, y) in enumerate(zip("avd", ys)):
        y = torch.cat(y)
        g = y.reshape(B, -1, 8, y.shape[1] // 8, 3 ** k)
        g = g / torch.sqrt(1e-5 + (g ** 2).sum(-1, keepdim=True).mean([1, 3], keepdim=True))
        out.append(x[k] + w[f"{q}gn_{name}.gamma"] * g.reshape(y.shape))
    return out


def _proxattn(c, s):
    outs = []
    box = c["box"]
    for z in range(c["Z"]):
        t = [s[k][z].double().requires_grad_(c["grad"]) for k in ("Q", "K", "V", "X", "Y")]
        R = t[3][:, None, :] - t[4][None, :, :]
        d2 = (R ** 2).sum(-1) if not box else ((1 - torch.cos(2 * math.pi * R / box)) * (box ** 2 / (2 * math.pi ** 2))).sum(-1)
        del R
        r0 = s["r0sq"][z % c["heads"]].double()
        out = (r0 / (r0 + d2) * (t[0] @ t[1].t())) @ t[2]
        outs.append([out.detach()] + (list(torch.autograd.grad(out, t, s["dO"][z].double())) if c["grad"] else []))
    return [torch.stack(o) for o in zip(*outs)]


def _chain(B, N):
    i = torch.arange(N - 1, device=DEV)
    src, dst = torch.cat([i, i + 1]), torch.cat([i + 1, i])
    offs = N * torch.arange(B, device=DEV)[:, None]
    return (src[None] + offs).reshape(-1), (dst[None] + offs).reshape(-1)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "graph":
        return None   # whole numbers, and differences of inputs in a given order: compared bit by bit
    s = _inputs(c, seed)
    if kind == "proxattn":
        out = _proxattn(c, s)
        return out if c["grad"] else out[0]
    B, N, Nt = c["systems"], c["nodes"], c["systems"] * c["nodes"]
    w = {k: t.double() for k, t in s["w"].items()}
    train = kind.endswith("train")
    with torch.enable_grad() if train else torch.no_grad():
        if not kind.endswith("step"):
            edges = (s["src"], s["dst"], s["rij"].double())
            x = [s[k].double().reshape(Nt, *s[k].shape[2:]).requires_grad_(train) for k in ("x_a", "x_v", "x_d") if k in s]
            if train:
                for t in w.values():
                    t.requires_grad_(True)
        shaped = lambda t: t.reshape(B, N, *t.shape[1:])  # noqa: E731
        if kind == "painn_layer":
            return [shaped(t) for t in _painn_message(c, w, "", *edges, *x)]
        if kind == "bee_layer":
            return [shaped(t) for t in _bee_block(c, w, "", B, edges, x)]
        if train:
            if kind == "painn_train":
                bonds, flat = _chain(B, N), s["pos"].reshape(-1, 3)
                outs = _painn_block(c, w, "", B, edges, (*bonds, (flat[bonds[1]] - flat[bonds[0]]).double()), *x)
            else:
                outs = _bee_messages(c, w, "", *edges, x)
            got = torch.autograd.grad(outs, x + list(w.values()), [s["g_" + k].double().reshape(o.shape) for k, o in zip("avd", outs)])
            nodes = [shaped(t) for t in list(outs) + list(got[:len(x)])]
            return [t.detach() for t in nodes + list(got[len(x):])]
        z = s["pos"] + 0.05 * s["noise"]
        z64, pos64 = z.double(), s["pos"].double()
        if kind == "bee_step":
            src, dst, _ = _edges(z, 0.0, c["cutoff"])
            flat = z64.reshape(-1, 3)
            x_v = _tens(w["v_readin.W"], (z64 - pos64).reshape(Nt, 1, 3), 1)
            x = [w["type_embed.weight"][s["types"]].repeat(B, 1), x_v, torch.zeros(Nt, BEE_DIMS[c["dims"]][2], 3, 3, device=DEV).double()]
            for k in range(c["depth"]):
                x = _bee_block(c, w, f"blocks.{k}.", B, (src, dst, flat[dst] - flat[src]), x)
            return shaped(_tens(w["readout.W"], x[1], 1)[:, 0])
        silu = torch.nn.functional.silu
        x_a = _mlp(w, "mlp_embed", w["atom_embeddings"], silu).repeat(B, 1)
        x_v = _tens(w["v_readin.W"], (z64 - pos64).reshape(Nt, 1, 3), 1)
        bonds = _chain(B, N)
        for name, blocks, p in (("cpainn_0", 2, s["pos"]), ("cpainn_1", 5, z)):
            flat = p.double().reshape(-1, 3)
            src, dst, _ = _edges(p, 0.0, c["cutoff"])
            x_a = x_a + w[name + ".atom_embed.weight"][s["types"]].repeat(B, 1)
            for k in range(blocks):
                x_a, x_v = _painn_block(c, w, f"{name}.blocks.{k}.", B, (src, dst, flat[dst] - flat[src]),
                                        (*bonds, flat[bonds[1]] - flat[bonds[0]]), x_a, x_v)
            if name == "cpainn_0":
                freqs = torch.exp(-torch.arange(32, device=DEV, dtype=torch.float64) / 31)
                end, length = s["end"].double()[:, None], (s["end"].double() - s["start"].double())[:, None]
                phase = torch.cat([end * freqs, length * freqs], dim=1)
                t = torch.nn.functional.linear(torch.cat([torch.sin(phase), torch.cos(phase)], dim=1), w["t_embed.lin1.weight"],
                                               w["t_embed.lin1.bias"]).repeat_interleave(N, dim=0)
                x_a = _mlp(w, "mlp_denoise", x_a + t, silu)
                x_v = x_v + _tens(w["pos_emb.lin_v.W"], 0.1 * (z64 - pos64).reshape(Nt, 1, 3), 1)
        return (1 - length)[:, :, None] * shaped(_tens(w["readout.W"], x_v, 1)[:, 0])
