"""Timing cases: the work a user of this package has it do, through its public entry points.

A case is a dict of plain values.  ``kind`` names the entry point:

    forces     ``E = block(...)`` and dE/dpos with frozen parameters and embeddings: one step of
               molecular dynamics or relaxation
    infer      node output and energy under ``torch.no_grad()``: screening, evaluation
    train      ``block.node_output`` and its VJP w.r.t. embeddings, positions and all parameters,
               the upstream gradient given: the block as one layer of a network in training
    sweep      ``block.node_output_vjp``: the same in one pass over destination chunks, for batches
               and graphs of any size
    resident   ``EdgeConvRunner``: the edge convolution forward and backward on arrays that stay on
               the device, no autograd
    replay     ``CapturedStep``: the training step from pinned host arrays to pinned host results,
               recorded once and replayed
    neighbors  ``neighbor_list`` and ``EdgeGraph.build``: the periodic neighbour list and the sorted
               edge order, redone whenever atoms have moved

The other values: ``structures`` periodic cubes of ``atoms`` atoms at ``density`` atoms per cubic
Angstrom, edges within ``cutoff`` (per destination the nearest ``neighbors``, 0 = all of them), the
block's ``lmax``, ``mmax``, ``channels``, ``hidden``, ``edge_channels``, ``basis`` and operand
``precision``; ``graph``: the caller has the sorted edges in hand (a neighbour list is kept for many
steps) instead of having each call sort them; ``crystal``: the atoms are a thermally displaced fcc
crystal instead of uniform in the cube.
"""

from __future__ import annotations

import math

import torch

from zippel_b200.blocks.eso2 import BlockConfig, ESO2Block
from zippel_b200.blocks.wigner import gamma_harmonics
from zippel_b200.captured import CapturedStep
from zippel_b200.fixtures import bulk_supercell
from zippel_b200.graph import EdgeGraph, neighbor_list
from zippel_b200.runner import EdgeConvRunner

DEVICE = "cuda"
MAX_ELEMENT = 30
FCC_CELL, FCC_DISPLACEMENT = 3.615, 0.03        # shells at 5.72 and 6.26 A on either side of 6 A

# the block of the package's benchmark, and the smaller one of its reference fixtures
_WIDE = dict(lmax=4, mmax=2, channels=128, hidden=128, edge_channels=128, basis=64, cutoff=6.0,
             density=0.1, neighbors=30, structures=1, precision="fp32", graph=False,
             crystal=False)
_L2 = dict(_WIDE, lmax=2, density=0.05, neighbors=0)


def listed() -> list[dict]:
    return [
        # a molecule-sized cell in an MD loop: latency and launches, nothing else
        dict(_L2, name="forces_64", kind="forces", atoms=64, channels=32, hidden=32,
             edge_channels=32, basis=32, cutoff=5.0, density=0.064),
        # screening one small structure at a time
        dict(_WIDE, name="infer_200_bf16", kind="infer", atoms=200, precision="bf16"),
        # fine-tuning on small crystals, one structure per step, a new edge list every step
        dict(_L2, name="train_216", kind="train", atoms=216),
        # a training loop over structures of one size, recorded as a graph
        dict(_WIDE, name="replay_500", kind="replay", atoms=500),
        # widths and degrees off the beaten track, in the widest operand format
        dict(_WIDE, name="train_777_ragged", kind="train", atoms=777, lmax=3, mmax=3, channels=72,
             hidden=40, edge_channels=36, basis=50, neighbors=23, precision="fp32_bf16x3"),
        # the benchmark's structure: evaluation, training, and the kernels alone
        dict(_WIDE, name="infer_2000", kind="infer", atoms=2000, graph=True),
        dict(_WIDE, name="train_2000", kind="train", atoms=2000),
        dict(_WIDE, name="resident_2000", kind="resident", atoms=2000, graph=True),
        # a bulk crystal in an MD loop, the neighbour list kept between rebuilds
        dict(_L2, name="forces_5832", kind="forces", atoms=5832, graph=True),
        # a batch of independent structures in reduced precision
        dict(_WIDE, name="sweep_64x200_bf16", kind="sweep", atoms=200, structures=64,
             precision="bf16", graph=True),
        # one large graph at the highest degree
        dict(_WIDE, name="sweep_8000_lmax6", kind="sweep", atoms=8000, lmax=6, graph=True),
        # the neighbour list of a large cell
        dict(_WIDE, name="neighbors_100000", kind="neighbors", atoms=100000),
    ]


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the ranges the listed ones stand for."""
    ceiling = {}
    for c in listed():
        side = c["kind"] == "neighbors"
        cost, most = work(c), ceiling.setdefault(side, {"bytes": 0.0, "flops": 0.0})
        for k in most:
            most[k] = max(most[k], cost[k])
    while True:
        kind = rng.choice(["forces", "forces", "infer", "infer", "train", "train", "sweep",
                           "resident", "replay", "neighbors"])
        c = dict(_WIDE, kind=kind, lmax=rng.choice([1, 2, 2, 3, 4, 4, 4, 5, 6]),
                 density=round(rng.uniform(0.04, 0.11), 3))
        # high degrees are used with low orders
        c["mmax"] = min(c["lmax"], rng.choice([1, 2, 2, 2, 2, 3, 4]), {5: 3, 6: 2}.get(c["lmax"], 4))
        # mostly powers of two, the rest any width the kernels take
        for key, step in (("channels", 8), ("hidden", 8), ("edge_channels", 4)):
            c[key] = (rng.choice([32, 64, 128, 128, 128]) if rng.random() < 0.7
                      else step * rng.randint(16 // step, 160 // step))
        c["basis"] = rng.choice([32, 64, 64, rng.randint(8, 100)])
        c["neighbors"] = rng.choice([30, 30, 0, rng.randint(8, 48)])
        c["cutoff"] = rng.choice([5.0, 6.0, 6.0])
        c["precision"] = rng.choice(["fp32", "fp32", "fp32", "bf16", "bf16", "fp32_bf16x3"])
        c["graph"] = kind in ("resident", "sweep") or (kind in ("forces", "infer", "train")
                                                       and rng.random() < 0.5)
        c["atoms"] = _log_uniform(rng, 48, {"neighbors": 1e5, "replay": 2000}.get(kind, 2e4))
        if kind in ("infer", "train", "sweep") and rng.random() < 0.3:
            c["structures"] = _log_uniform(rng, 2, 64)
            c["atoms"] = _log_uniform(rng, 24, 400)
        if kind in ("neighbors", "resident"):
            # their outputs list the edges: structures whose edge count does not hang on the seed
            c.update(cutoff=6.0, density=0.1, neighbors=rng.choice([30, 30, 0, rng.randint(8, 40)]))
            if not c["neighbors"]:
                reps = max(2, round((c["atoms"] / 4) ** (1 / 3)))
                c.update(crystal=True, atoms=4 * reps ** 3, density=round(4 / FCC_CELL ** 3, 6))
        if kind == "neighbors":
            c.update(precision="fp32", lmax=4, mmax=2, channels=128, hidden=128, edge_channels=128,
                     basis=64)
        cost = work(c)
        if all(cost[k] <= most for k, most in ceiling[kind == "neighbors"].items()):
            return c


# ---------------------------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------------------------


def _n_nodes(c: dict) -> int:
    return c["atoms"] * c["structures"]


def _n_edges(c: dict) -> float:
    """Expected directed edges of uniformly placed atoms."""
    degree = c["density"] * 4.0 / 3.0 * math.pi * c["cutoff"] ** 3
    return _n_nodes(c) * (min(degree, c["neighbors"]) if c["neighbors"] else degree)


def _macs_per_edge(c: dict) -> dict:
    """Multiply-adds of one edge's forward: SO(2) products, radial layers, rotations in and out."""
    L, M, C, H, EC = c["lmax"], c["mmax"], c["channels"], c["hidden"], c["edge_channels"]
    so2 = (L + 1) * 2 * C * H * (2 * L + 1) + (L + 1) * H * C * (L + 1)
    rad = (c["basis"] + 2 * EC) * EC + EC * EC
    width = 0
    for m in range(M + 1):
        km = L + 1 - m
        width += 2 * C * km
        if m:
            so2 += (2 * km * 2 * C) * (2 * km * H) + (2 * km * H) * (2 * km * C)
    nnz = sum((2 * min(l, M) + 1) * (2 * l + 1) for l in range(L + 1))
    return {"so2": so2, "rad": rad, "last_rad": EC * width, "rotate": 3 * C * nnz, "width": width}


def work(c: dict) -> dict:
    """Bytes and operations one pass cannot do without: each input read once, each output written
    once; every product counted once, whatever the operand format."""
    n, e, kind = _n_nodes(c), _n_edges(c), c["kind"]
    if kind == "neighbors":
        degree = c["density"] * 4.0 / 3.0 * math.pi * c["cutoff"] ** 3
        # positions in; pairs, shifts, two orders of the edges and their offsets out
        return {"bytes": 24.0 * n + e * (16 + 24 + 16) + 12.0 * n, "flops": 10.0 * n * degree}
    L, C, H, EC = c["lmax"], c["channels"], c["hidden"], c["edge_channels"]
    per = _macs_per_edge(c)
    node = 4.0 * n * (L + 1) ** 2 * C
    edge_in = 16 + 12 + 8 * (L + 1)
    so2_params = 4.0 * sum(p for p in _so2_sizes(c))
    rad_params = 4.0 * ((c["basis"] + 3 * EC) * EC + EC * per["width"])
    if kind == "resident":
        macs = 3 * e * (per["so2"] + per["rotate"])
        rows = 12 + 4 * per["width"] + 4                 # edge vectors, radial features, envelope
        nbytes = 4 * node + e * (2 * rows + 16 + 8 * (L + 1)) + 2 * so2_params
        return {"bytes": nbytes, "flops": 2.0 * macs}
    macs = e * (per["so2"] + per["rotate"] + per["rad"] + per["last_rad"])
    params = so2_params + rad_params
    if kind == "infer":
        return {"bytes": 2 * node + 12.0 * n + e * edge_in + params, "flops": 2.0 * macs}
    if kind == "forces":
        return {"bytes": node + 24.0 * n + e * edge_in + params, "flops": 4.0 * macs}
    return {"bytes": 4 * node + 24.0 * n + e * edge_in + 2 * params, "flops": 6.0 * macs}


def _so2_sizes(c: dict) -> list[int]:
    L, C, H = c["lmax"], c["channels"], c["hidden"]
    out = [(L + 1) * 2 * C * H * (2 * L + 1), (L + 1) * H * C * (L + 1)]
    for m in range(1, c["mmax"] + 1):
        km = L + 1 - m
        out += [km * 2 * C * 2 * H * km, km * H * 2 * C * km]
    return out


def tolerance(c: dict):
    """The neighbour list and the sorted order are the same to the last bit; fp32 formats carry 22
    to 24 bits per operand, bf16 eight."""
    if c["kind"] == "neighbors":
        return "exact"
    return {"rel": 1e-2} if c["precision"] == "bf16" else {"rel": 1e-5}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------


def _structures(c: dict, gen: torch.Generator):
    """Atoms in periodic cubes and their edges, block-diagonal over the structures."""
    box = (c["atoms"] / c["density"]) ** (1.0 / 3.0)
    pos, edges, shifts = [], [], []
    for s in range(c["structures"]):
        if c["crystal"]:
            reps = round((c["atoms"] / 4) ** (1 / 3))
            box = reps * FCC_CELL
            p = torch.from_numpy(bulk_supercell("fcc", FCC_CELL, reps, gen.initial_seed(),
                                                FCC_DISPLACEMENT)[0]).to(DEVICE)
            drift = torch.rand(3, generator=gen, device=DEVICE, dtype=torch.float64) * box
            p = torch.remainder(p + drift, box)
        else:
            p = torch.rand(c["atoms"], 3, generator=gen, device=DEVICE, dtype=torch.float64) * box
        pos.append(p)
        if c["kind"] != "neighbors":
            ei, sh, _ = neighbor_list(p, box, c["cutoff"], c["neighbors"] or None)
            edges.append(ei + s * c["atoms"])
            shifts.append(sh)
    if c["kind"] == "neighbors":
        return pos[0], None, None, box
    return torch.cat(pos), torch.cat(edges, dim=1), torch.cat(shifts), box


def _block(c: dict, gen: torch.Generator) -> ESO2Block:
    """Xavier-uniform weights; small biases, as after some training."""
    cfg = BlockConfig(lmax=c["lmax"], mmax=c["mmax"], sphere_channels=c["channels"],
                      hidden_channels=c["hidden"], edge_channels=c["edge_channels"],
                      num_distance_basis=c["basis"], cutoff=c["cutoff"])
    with torch.device(DEVICE):
        block = ESO2Block(cfg, precision=c["precision"])
    with torch.no_grad():
        for name, p in block.named_parameters():
            u = torch.rand(p.shape, generator=gen, device=DEVICE) * 2 - 1
            if name.startswith("elem_emb"):
                p.copy_(u)
            elif p.dim() == 2:
                p.copy_(u * math.sqrt(6.0 / (p.shape[0] + p.shape[1])))
                if name.startswith(("c1_m.", "c2_m.")):
                    p.mul_(2 ** -0.5)
            else:
                p.copy_(u * 0.1 + (1.0 if name in ("rad_func.1.weight", "rad_func.4.weight") else 0.0))
    return block


def prepare(c: dict, seed: int) -> dict:
    gen = torch.Generator(DEVICE).manual_seed(seed)
    pos, edge_index, shifts, box = _structures(c, gen)
    if c["kind"] == "neighbors":
        return {"case": c, "pos": pos, "box": box}
    n, e, k = pos.shape[0], edge_index.shape[1], (c["lmax"] + 1) ** 2
    gamma = torch.rand(e, generator=gen, device=DEVICE, dtype=torch.float64) * 2 * math.pi
    cos_g, sin_g = gamma_harmonics(gamma, c["lmax"])
    randn = lambda *shape: torch.randn(*shape, generator=gen, device=DEVICE)         # noqa: E731
    s = {"case": c, "block": _block(c, gen), "pos": pos.float(),
         "z": torch.randint(1, MAX_ELEMENT, (n,), generator=gen, device=DEVICE),
         "x": randn(n, k, c["channels"]), "edge_index": edge_index, "shifts": shifts.float(),
         "cos": cos_g.float(), "sin": sin_g.float(), "graph": None}
    if c["kind"] not in ("infer", "forces"):
        s["upstream"] = randn(n, k, c["channels"])
    if c["graph"]:
        s["graph"] = EdgeGraph.build(edge_index, n)
    if c["kind"] == "forces":
        s["block"].requires_grad_(False)
    if c["kind"] == "replay":
        batch = {"pos": s["pos"], "x_node": s["x"], "edge_index": edge_index, "shifts": s["shifts"],
                 "cos_gamma_k": s["cos"], "sin_gamma_k": s["sin"], "atomic_numbers": s["z"],
                 "upstream": s["upstream"]}
        s["step"] = CapturedStep(s["block"], {key: v.cpu() for key, v in batch.items()}, DEVICE)
    if c["kind"] == "resident":
        s["runner"] = _runner(c, s, randn)
    return s


def _runner(c: dict, s: dict, randn) -> EdgeConvRunner:
    block, graph = s["block"], s["graph"]
    perm, src, dst = graph.perm64, graph.src.long(), graph.dst.long()
    vec = (s["pos"][dst] - s["pos"][src] + s["shifts"][perm]).contiguous()
    with torch.no_grad():
        env = block.envelope(vec.norm(dim=1) / c["cutoff"]).contiguous()
    # radial features as the last layer of the radial MLP leaves them: order one, both signs
    radial = randn(graph.n_edges, block.num_channels_rad)
    runner = EdgeConvRunner(block.plan(DEVICE), graph, with_backward=True)
    w = lambda p: p.detach()                                                         # noqa: E731
    runner.bind(s["x"], vec, s["cos"][perm].contiguous(), s["sin"][perm].contiguous(), radial, env,
                w(block.c1_m0.weight), w(block.c1_m0.bias), [w(l.weight) for l in block.c1_m],
                w(block.c2_m0.weight), w(block.c2_m0.bias), [w(l.weight) for l in block.c2_m])
    return runner


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------


def run(s: dict):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "neighbors":
        edge_index, shifts, row_ptr = neighbor_list(s["pos"], s["box"], c["cutoff"],
                                                    c["neighbors"] or None)
        g = EdgeGraph.build(edge_index, s["pos"].shape[0])
        return [edge_index, shifts, row_ptr, g.perm, g.src, g.dst, g.row_ptr, g.perm_src,
                g.row_ptr_src]
    if kind == "resident":
        runner = s["runner"]
        out = runner.forward()
        gx, gvec, grad, genv, gw = runner.backward(s["upstream"])
        return [out, gx, gvec, grad, genv, list(gw[:2]), list(gw[2]), list(gw[3:5]), list(gw[5])]
    if kind == "replay":
        step = s["step"]
        step.run()
        return [step.loss_host, step.grad_pos_host, step.node_out, step.grads["x_node"],
                list(step.grads["params"].values())]
    block = s["block"]
    edges = (s["edge_index"], s["shifts"], s["cos"], s["sin"])
    if kind == "infer":
        with torch.no_grad():
            out = block.node_output(s["pos"], s["z"], s["x"], *edges, graph=s["graph"])
            return [block.energy(out), out]
    if kind == "sweep":
        out, gx, gpos, gparams = block.node_output_vjp(s["pos"], s["z"], s["x"], *edges,
                                                       s["upstream"], graph=s["graph"])
        return [out, gx, gpos, gparams]
    pos = s["pos"].detach().requires_grad_(True)
    if kind == "forces":
        energy = block(pos, s["z"], s["x"], *edges, graph=s["graph"])
        (grad,) = torch.autograd.grad(energy, pos)
        return [energy.detach(), grad]
    x = s["x"].detach().requires_grad_(True)
    out = block.node_output(pos, s["z"], x, *edges, graph=s["graph"])
    grads = torch.autograd.grad(out, [x, pos, *block.parameters()], s["upstream"],
                                allow_unused=True)
    return [out.detach(), *grads]
