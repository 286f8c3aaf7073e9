"""The whole-block calls (zp_block_forward / zp_block_backward behind ``ESO2Block.node_output``) and
the checked edge sort, at the sizes where their dispatch turns: widths that are and are not
multiples of 8 (operand format of a layer, zero padding), frozen parameter groups, no edges."""

from __future__ import annotations

import pytest
import torch

from oracle import eso2_oracle as orc
from tests.helpers import (check_against, gpu_node_out_and_vjp, make_block, oracle_node_out_and_vjp,
                           random_case, rel_l2)
from zippel_b200.graph import EdgeGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("fp32_bf16x3", 1e-5), ("bf16", 2e-2)])
@pytest.mark.parametrize("ec,nb", [(12, 5), (8, 6), (20, 8), (132, 64)])
def test_radial_layer_widths(ec, nb, precision, tol, jd64):
    cfg = dict(lmax=2, mmax=1, sphere_channels=16, hidden_channels=8, edge_channels=ec,
               num_distance_basis=nb, cutoff=5.0)
    params = orc.init_params(cfg, seed=ec)
    case = random_case(cfg, 17, 131, seed=nb)
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    block = make_block(cfg, params, precision=precision)
    check_against(*gpu_node_out_and_vjp(block, case, case["upstream"]), *want, tol=tol)
    assert block.plan("cuda").device_status() == 0


@pytest.mark.parametrize("frozen", [("elem_emb",), ("rad_func",), ("c1_", "c2_"), ("elem_emb", "rad_func")])
def test_frozen_groups_leave_the_other_gradients_alone(frozen):
    cfg = dict(lmax=3, mmax=2, sphere_channels=16, hidden_channels=16, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1))
    case = {k: v.cuda().float() if v.is_floating_point() else v.cuda()
            for k, v in random_case(cfg, 20, 150, seed=2).items()}

    def grads():
        pos, x = case["pos"].clone().requires_grad_(True), case["x_node"].clone().requires_grad_(True)
        out = block.node_output(pos, case["atomic_numbers"], x, case["edge_index"], case["shifts"],
                                case["cos_gamma_k"], case["sin_gamma_k"])
        names = ["pos", "x"] + [n for n, p in block.named_parameters() if p.requires_grad]
        wrt = [pos, x] + [p for p in block.parameters() if p.requires_grad]
        return dict(zip(names, torch.autograd.grad(out, wrt, case["upstream"], allow_unused=True)))

    full = grads()
    for n, p in block.named_parameters():
        p.requires_grad_(not n.startswith(frozen))
    part = grads()
    assert set(full) - set(part) == {n for n in full if n.startswith(frozen)}
    for n, g in part.items():
        assert (g is None) == (full[n] is None) and (g is None or rel_l2(g, full[n]) < 1e-6), n


@pytest.mark.parametrize("precision,tol", [("fp32", 1.5e-5), ("fp32_bf16x3", 1.5e-5), ("bf16", 1e-4)])
@pytest.mark.parametrize("edges", [6000, 60000, 120000])
def test_every_choice_of_wanted_gradients(edges, precision, tol):
    """With side streams (from 4 096 edges on) and on both sides of the line up to which products share a launch,
    every choice of what wants a gradient forks and joins another way; each gradient is that of the call in which
    all are wanted, but for other splits of the sums over the edges: an accumulator adds 2 048 of them in 128 steps,
    each off by up to 2^-23 of the sum, 1.5e-5 at most.  (In bf16 such a difference may turn the rounding of an
    operand: 2^-9 of one value in a thousand.)"""
    cfg = dict(lmax=1, mmax=1, sphere_channels=16, hidden_channels=16, edge_channels=64,
               num_distance_basis=16, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1), precision=precision)
    case = {k: v.cuda().float() if v.is_floating_point() else v.cuda()
            for k, v in random_case(cfg, edges // 20, edges, seed=2).items()}
    groups = {"emb": ("elem_emb",), "rad": ("rad_func",), "so2": ("c1_", "c2_")}

    def grads(wanted):
        pos, x = (case[k].clone().requires_grad_(w in wanted) for k, w in (("pos", "pos"), ("x_node", "x")))
        for n, p in block.named_parameters():
            p.requires_grad_(any(n.startswith(groups[w]) for w in wanted if w in groups))
        wrt = {"pos": pos, "x": x, **dict(block.named_parameters())}
        wrt = {n: t for n, t in wrt.items() if t.requires_grad}
        out = block.node_output(pos, case["atomic_numbers"], x, case["edge_index"], case["shifts"],
                                case["cos_gamma_k"], case["sin_gamma_k"])
        return dict(zip(wrt, torch.autograd.grad(out, list(wrt.values()), case["upstream"])))

    everything = ("pos", "x", "emb", "rad", "so2")
    full = grads(everything)
    for choice in range(1, 31):
        wanted = [w for i, w in enumerate(everything) if choice >> i & 1]
        for n, g in grads(wanted).items():
            assert rel_l2(g, full[n]) < tol, (wanted, n)


@pytest.mark.parametrize("n,degree", [(3, 31), (3, 33), (2, 64), (2, 65), (16385, 2), (40000, 3)])
def test_sort_at_its_bucket_and_scan_edges(n, degree):
    import numpy as np
    from zippel_b200.graph import EdgeGraph, csr_reference
    g = torch.Generator("cpu").manual_seed(n + degree)
    ei = torch.stack([torch.randint(0, n, (n * degree,), generator=g),
                      torch.arange(n).repeat_interleave(degree)])[:, torch.randperm(n * degree, generator=g)]
    want = csr_reference(ei.numpy(), n)
    got, check = EdgeGraph.build_checked(ei.cuda(), torch.zeros(n, dtype=torch.int64, device="cuda"), 5)
    check()
    for key, val in want.items():
        assert np.array_equal(getattr(got, key).cpu().numpy(), val), key


def test_left_out_slots_are_edges_into_no_node():
    """A slot that an unvalidated sort has left out reads as an edge 0 -> 0 that counts for source 0 alone: an edge
    from a node at the same place with the same embedding.  (Sums in another order: 1e-5.)"""
    cfg = dict(lmax=3, mmax=2, sphere_channels=16, hidden_channels=16, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1))
    n, e = 12, 90
    case = {k: v.cuda().float() if v.is_floating_point() else v.cuda()
            for k, v in random_case(cfg, n + 1, e, seed=2).items()}
    case["edge_index"] %= n
    for k in ("pos", "x_node", "atomic_numbers"):
        case[k][n] = case[k][0]
    case["shifts"][0] = 0.5                    # the slots take those of edge 0
    bad = torch.tensor([7, 31, 32, 60], device="cuda")

    def grad_x(nodes, edge_index, edges):
        x = case["x_node"][:nodes].clone().requires_grad_(True)
        graph = EdgeGraph.build(edge_index, nodes, validate=False)
        out = block.node_output(case["pos"][:nodes], case["atomic_numbers"][:nodes], x, edge_index,
                                *[case[k][edges] for k in ("shifts", "cos_gamma_k", "sin_gamma_k")], graph=graph)
        return torch.autograd.grad(out, x, case["upstream"][:nodes])[0]

    broken = case["edge_index"].clone()
    broken[1, bad] = n + 5
    every = torch.arange(e, device="cuda")
    valid = every[~torch.isin(every, bad)]
    alone = grad_x(n, case["edge_index"][:, valid], valid)
    twin = grad_x(n + 1, torch.cat([case["edge_index"][:, valid], torch.tensor([[n], [0]], device="cuda").repeat(1, len(bad))], 1),
                  torch.cat([valid, torch.zeros_like(bad)]))
    want = alone.clone()
    want[0] += twin[n]
    assert rel_l2(grad_x(n, broken, every), want) < 1e-5


@pytest.mark.parametrize("what", ["edge", "element"])
def test_bad_input_raises(what):
    cfg = dict(lmax=1, mmax=1, sphere_channels=8, hidden_channels=8, edge_channels=8,
               num_distance_basis=4, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1))
    case = random_case(cfg, 6, 20, seed=2)
    if what == "edge":
        case["edge_index"][0, 3] = 6
    else:
        case["atomic_numbers"][5] = block.cfg.max_num_elements
    with pytest.raises(IndexError):
        gpu_node_out_and_vjp(block, case, case["upstream"])


@pytest.mark.parametrize("lmax,mmax,c,h", [(6, 3, 8, 8), (6, 6, 16, 8), (5, 4, 40, 8), (1, 0, 136, 8),
                                           (4, 4, 256, 8)])
def test_rotations_over_degrees_orders_and_widths(lmax, mmax, c, h, jd64):
    """Row walks, packed sums and torques of the rotate kernels from two degrees to seven, orders up to the
    degree, and widths that leave a warp partly idle (by edge) or a worker's lanes (by node)."""
    cfg = dict(lmax=lmax, mmax=mmax, sphere_channels=c, hidden_channels=h, edge_channels=8,
               num_distance_basis=6, cutoff=5.0)
    params = orc.init_params(cfg, seed=lmax)
    case = random_case(cfg, 7, 45, seed=mmax)
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    check_against(*gpu_node_out_and_vjp(make_block(cfg, params), case, case["upstream"]), *want)


@pytest.mark.parametrize("lmax,mmax,c,precision", [(2, 2, 16, "fp32"), (3, 1, 24, "fp32_bf16x3"), (4, 2, 136, "fp32"),
                                                   (5, 2, 72, "fp32")])
def test_nodes_of_many_edges_are_cut(lmax, mmax, c, precision, jd64):
    """A node with most of the edges, each way, among nodes of two: its edges are several blocks', whose sums are
    added at the end."""
    cfg = dict(lmax=lmax, mmax=mmax, sphere_channels=c, hidden_channels=8, edge_channels=8,
               num_distance_basis=6, cutoff=5.0)
    params = orc.init_params(cfg, seed=lmax)
    n, e = 300, 2100
    case = random_case(cfg, n, e, seed=mmax)
    hub = 211
    case["edge_index"][0, 600:1300] = hub
    case["edge_index"][1, 1300:] = hub
    case["shifts"] += 0.25                     # no edge of a node with itself has length zero
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    block = make_block(cfg, params, precision=precision)
    got = gpu_node_out_and_vjp(block, case, case["upstream"])
    check_against(*got, *want)
    again = gpu_node_out_and_vjp(block, case, case["upstream"])
    assert torch.equal(got[1], again[1])       # added in one order whoever comes last


@pytest.mark.parametrize("n,e", [(200, 199), (200, 200), (200, 599), (200, 600), (9, 160)])
@pytest.mark.parametrize("lmax,c", [(2, 64), (4, 16), (5, 32)])
def test_nodes_of_few_edges_whole_and_in_pieces(n, e, lmax, c, jd64, monkeypatch):
    """On either side of the lines between kernels by edge and by node, and with a piece's edges at few of the rows."""
    cfg = dict(lmax=lmax, mmax=2, sphere_channels=c, hidden_channels=8, edge_channels=8,
               num_distance_basis=6, cutoff=5.0)
    params = orc.init_params(cfg, seed=lmax)
    case = random_case(cfg, n, e, seed=n + e)
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    block = make_block(cfg, params)
    check_against(*gpu_node_out_and_vjp(block, case, case["upstream"]), *want)
    monkeypatch.setattr("zippel_b200.blocks.eso2.MAX_EDGES_PER_CALL", 64)
    dev = {k: v.cuda().float() if v.is_floating_point() else v.cuda() for k, v in case.items()}
    out, gx, gpos, gparams = block.node_output_vjp(
        *[dev[k] for k in ("pos", "atomic_numbers", "x_node", "edge_index", "shifts", "cos_gamma_k", "sin_gamma_k",
                           "upstream")])
    names = [name for name, _ in block.named_parameters()]
    check_against(out, gx, gpos, dict(zip(names, gparams)), *want)


def test_edges_along_the_polar_axis(jd64):
    """An edge whose direction is the polar axis has no proper rotation; its gradient follows the
    construction of the matrices (clamped, large) and must not disturb the other edges."""
    cfg = dict(lmax=3, mmax=2, sphere_channels=16, hidden_channels=8, edge_channels=8,
               num_distance_basis=6, cutoff=8.0)
    params = orc.init_params(cfg, seed=5)
    case = random_case(cfg, 12, 60, seed=6)
    case["pos"] = case["pos"].float().double()
    case["shifts"] = torch.zeros_like(case["shifts"])
    for e, sign in ((0, 1.0), (31, -1.0), (40, 1.0)):      # atoms that only these edges touch
        i, j = 2 * (e % 3), 2 * (e % 3) + 1
        case["edge_index"][:, e] = torch.tensor([i, j])
        case["pos"][j] = case["pos"][i] + torch.tensor([0.0, sign * 1.5, 0.0])
    for k in range(60):
        if k not in (0, 31, 40):
            case["edge_index"][:, k] = 6 + case["edge_index"][:, k] % 6
            if case["edge_index"][0, k] == case["edge_index"][1, k]:
                case["edge_index"][0, k] = 6 + (case["edge_index"][0, k] - 5) % 6
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    got = gpu_node_out_and_vjp(make_block(cfg, params), case, case["upstream"])
    assert rel_l2(got[0], want[0]) < 1e-5
    assert rel_l2(got[2][6:], want[2][6:]) < 1e-5 and rel_l2(got[2][:6], want[2][:6]) < 1e-3


@pytest.mark.parametrize("e", [63, 64, 65, 2049, 24000, 24001])
def test_products_together_and_apart(e):
    """Around the edge counts where the products of a step stop sharing one launch, where a split of
    the contraction over the edges has a remainder, and where it needs a second accumulation chunk:
    the same gradients as the three-plane format, whose kernel and tiles differ."""
    cfg = dict(lmax=1, mmax=1, sphere_channels=16, hidden_channels=24, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    params = orc.init_params(cfg, seed=e)
    case = random_case(cfg, 50, e, seed=e)
    a = gpu_node_out_and_vjp(make_block(cfg, params), case, case["upstream"])
    b = gpu_node_out_and_vjp(make_block(cfg, params, precision="fp32_bf16x3"), case, case["upstream"])
    check_against(*a, *b)


@pytest.mark.parametrize("e,ec,nb", [(37887, 12, 64), (37888, 12, 5), (37889, 12, 33), (37895, 132, 64),
                                     (37896, 260, 70), (40001, 128, 130)])
def test_front_end_of_many_edges(e, ec, nb, jd64):
    """From 37 888 edges on a warp of the front end takes eight: the last warp full and not, basis
    widths that end inside a quad of columns, that leave lanes over and that take several turns;
    LayerNorm rows of up to 128, 256 and 512 columns, more than its blocks hold at a time."""
    cfg = dict(lmax=1, mmax=1, sphere_channels=8, hidden_channels=8, edge_channels=ec,
               num_distance_basis=nb, cutoff=5.0)
    params = orc.init_params(cfg, seed=ec)
    case = random_case(cfg, 400, e, seed=nb)
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    block = make_block(cfg, params)
    check_against(*gpu_node_out_and_vjp(block, case, case["upstream"]), *want, tol=1e-5)


@pytest.mark.parametrize("how", ["checkpoint", "offload", "chunks"])
def test_gradients_when_saved_tensors_come_back_elsewhere(how, monkeypatch):
    """Checkpointed or with its saved tensors on the host, as one layer of a network whose embeddings are
    an intermediate; and in chunks, which checkpoint by themselves, with inputs that every chunk
    converts: the same gradients as the plain call, to the last bit where the sums are the same."""
    from torch.autograd.graph import save_on_cpu
    from torch.utils.checkpoint import checkpoint
    from zippel_b200.blocks import eso2

    cfg = dict(lmax=3, mmax=2, sphere_channels=32, hidden_channels=16, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=3))
    case = {k: v.cuda() for k, v in random_case(cfg, 60, 6000, seed=4).items()}
    f = {k: v.float() if v.is_floating_point() and k != "x_node" else v for k, v in case.items()}
    z = f["atomic_numbers"].int()

    def gradients(how):
        pos, a = f["pos"].clone().requires_grad_(True), f["x_node"].clone().requires_grad_(True)

        def layer(pos, a):
            return block.node_output(pos, z, torch.tanh(a), f["edge_index"], f["shifts"],
                                     f["cos_gamma_k"], f["sin_gamma_k"])

        if how == "offload":
            with save_on_cpu():
                out = layer(pos, a)
        elif how == "checkpoint":
            out = checkpoint(layer, pos, a, use_reentrant=False)
        else:
            out = layer(pos, a)
        junk = [torch.full_like(a, 1e3) for _ in range(40)]       # over whatever has been given back
        grads = torch.autograd.grad(out, [pos, a, *block.parameters()], f["upstream"].to(out.dtype),
                                    allow_unused=True)
        del junk
        return [out, *grads]

    want = gradients("plain")
    if how == "chunks":
        monkeypatch.setattr(eso2, "MAX_EDGES_PER_CALL", 4096)
    for got, ref in zip(gradients(how), want):
        if ref is not None:
            assert torch.equal(got, ref) if how != "chunks" else rel_l2(got, ref) < 2e-6


@pytest.mark.parametrize("frozen", [False, True])
def test_checkpointed_energy(frozen):
    from torch.utils.checkpoint import checkpoint
    cfg = dict(lmax=2, mmax=1, sphere_channels=16, hidden_channels=16, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1)).requires_grad_(not frozen)
    case = {k: v.cuda().float() if v.is_floating_point() else v.cuda()
            for k, v in random_case(cfg, 20, 150, seed=2).items()}

    def energy(pos):
        return block(pos, case["atomic_numbers"], case["x_node"], case["edge_index"], case["shifts"],
                     case["cos_gamma_k"], case["sin_gamma_k"])

    pos = case["pos"].clone().requires_grad_(True)
    wrt = [pos] if frozen else [pos, *block.parameters()]
    want = torch.autograd.grad(energy(pos), wrt)
    got = torch.autograd.grad(checkpoint(energy, pos, use_reentrant=False), wrt)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("what", ["eps", "deeper", "pruned", "parametrized"])
def test_blocks_with_layers_of_their_own(what, jd64, monkeypatch):
    """Two LayerNorms of different eps and a radial MLP of another depth run layer by layer; pruned and
    parametrized layers run in one call with the weights they form."""
    import torch.nn.utils.parametrize
    import torch.nn.utils.prune
    cfg = dict(lmax=2, mmax=1, sphere_channels=16, hidden_channels=8, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    params = orc.init_params(cfg, seed=9)
    case = random_case(cfg, 17, 131, seed=8)
    block = make_block(cfg, params)
    used, eps = {k: v.double() for k, v in params.items()}, [1e-5, 1e-5]
    deeper = None
    if what == "eps":
        eps[1] = block.rad_func[4].eps = 0.3
    elif what == "deeper":
        torch.manual_seed(3)
        deeper = torch.nn.Linear(16, 16).cuda()
        block.rad_func.insert(6, deeper)
    elif what == "pruned":
        torch.nn.utils.prune.l1_unstructured(block.rad_func[3], "weight", 0.4)
        torch.nn.utils.prune.l1_unstructured(block.c1_m[0], "weight", 0.4)
        used["rad_func.3.weight"] = block.rad_func[3].weight.detach().cpu().double()
        used["c1_m.0.weight"] = block.c1_m[0].weight.detach().cpu().double()
    else:
        class Twice(torch.nn.Module):
            def forward(self, w):
                return 2 * w
        torch.nn.utils.parametrize.register_parametrization(block.c2_m0, "weight", Twice())
        used["c2_m0.weight"] = 2 * used["c2_m0.weight"]

    def radial_mlp(p, h):
        f = torch.nn.functional
        for lin, ln, e in ((0, 1, eps[0]), (3, 4, eps[1])):
            h = f.linear(h, p[f"rad_func.{lin}.weight"], p[f"rad_func.{lin}.bias"])
            h = f.silu(f.layer_norm(h, h.shape[-1:], p[f"rad_func.{ln}.weight"], p[f"rad_func.{ln}.bias"], e))
        if deeper is not None:
            h = f.linear(h, deeper.weight.detach().cpu().double(), deeper.bias.detach().cpu().double())
        return f.linear(h, p["rad_func.6.weight"], p["rad_func.6.bias"])

    monkeypatch.setattr(orc, "radial_mlp", radial_mlp)
    want = oracle_node_out_and_vjp(cfg, used, case, case["upstream"], jd64)
    out, gx, gpos, pg = gpu_node_out_and_vjp(block, case, case["upstream"])
    assert rel_l2(out, want[0]) < 1e-5 and rel_l2(gx, want[1]) < 1e-5 and rel_l2(gpos, want[2]) < 1e-5
    for name, ref in want[3].items():
        if name in pg and ref is not None and ref.abs().max() > 0 and not (deeper is not None and name.startswith("rad_func.6")):
            assert rel_l2(pg[name], ref) < 1e-5, name
    if deeper is not None:
        assert rel_l2(pg["rad_func.7.weight"], want[3]["rad_func.6.weight"]) < 1e-5


@pytest.mark.parametrize("entry", ["node_output", "energy", "vjp", "edge_conv"])
def test_out_of_memory_in_one_piece_goes_on_in_chunks(entry, monkeypatch):
    """The first allocation of a workspace fails: the call is made in chunks, with the same results."""
    from zippel_b200.blocks import eso2
    from zippel_b200.graph import EdgeGraph

    cfg = dict(lmax=2, mmax=1, sphere_channels=16, hidden_channels=16, edge_channels=16,
               num_distance_basis=8, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=3))
    case = {k: v.cuda().float() if v.is_floating_point() else v.cuda()
            for k, v in random_case(cfg, 60, 6000, seed=4).items()}
    graph = EdgeGraph.build(case["edge_index"], 60)
    args = [case[k] for k in ("atomic_numbers", "x_node", "edge_index", "shifts", "cos_gamma_k", "sin_gamma_k")]
    plan, params = block.plan("cuda"), [p for n, p in block.named_parameters() if not n.startswith("readout")]

    def run():
        pos = case["pos"].clone().requires_grad_(True)
        if entry == "node_output":
            out = block.node_output(pos, *args, graph=graph)
            return [out, *torch.autograd.grad(out, [pos, *params], case["upstream"])]
        if entry == "energy":
            out = block(pos, *args, graph=graph)
            return [out, *torch.autograd.grad(out, [pos, *params])]
        if entry == "vjp":
            out, gx, gpos, gp = block.node_output_vjp(case["pos"], *args, case["upstream"], graph=graph)
            return [out, gx, gpos, *[g for g in gp if g is not None]]
        return [block._edges_to_nodes_in_parts(plan, graph, graph.perm, pos, *args[:2], *args[3:], None)]

    want = run()
    failed = []

    def failing(inner, nth):
        def call(*a, **k):
            if not failed:
                failed.append(nth)
                raise torch.cuda.OutOfMemoryError("for the test")
            return inner(*a, **k)
        return call

    monkeypatch.setattr(eso2, "_edge_budget", lambda *a: 4096)
    if entry == "edge_conv":
        monkeypatch.setattr(plan, "workspace", failing(plan.workspace, 1))
    else:
        monkeypatch.setattr(eso2, "_block", failing(eso2._block, 1))
    calls = []
    run_call = eso2._abi_forward if entry == "edge_conv" else eso2._block_vjp
    monkeypatch.setattr(eso2, run_call.__name__, lambda *a, **k: (calls.append(1), run_call(*a, **k))[1])
    got = run()
    assert failed and len(calls) == (2 if entry == "edge_conv" else 3)
    for a, b in zip(got, want):
        assert rel_l2(a, b) < 2e-6


@pytest.mark.parametrize("lmax,mmax,e", [(2, 1, 130), (3, 3, 300), (4, 2, 129), (6, 6, 140), (6, 1, 60)])
@pytest.mark.parametrize("what", ["bf16", "some", "unused", "scaled"])
def test_roll_angle_harmonics_are_taken_as_they_are(what, lmax, mmax, e, jd64):
    """Harmonics that are not cos(k g), sin(k g) of one angle (rounded to 16 bits, or a few edges' not of
    one angle at all, or scaled), and orders above mmax that the forward never reads: the gradient is
    that of the forward with the arrays as given."""
    cfg = dict(lmax=lmax, mmax=mmax, sphere_channels=40, hidden_channels=8, edge_channels=8,
               num_distance_basis=6, cutoff=8.0)
    params = orc.init_params(cfg, seed=lmax)
    case = random_case(cfg, 11, e, seed=mmax)
    for key in ("cos_gamma_k", "sin_gamma_k"):
        g = torch.Generator("cpu").manual_seed(len(key))
        h = case[key]
        if what == "bf16":
            h = h.bfloat16().double()
        elif what == "some":
            h[::7, 1:] = torch.randn(h[::7, 1:].shape, generator=g).float().double()
        elif what == "unused":
            h[:, mmax + 1:] = 0.0
        else:
            h[:, 1:] *= 1.01
        case[key] = h.float().double()
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    check_against(*gpu_node_out_and_vjp(make_block(cfg, params), case, case["upstream"]), *want)


@pytest.mark.parametrize("lmax,mmax", [(6, 6), (2, 2)])
def test_whole_blocks_of_polar_edges(lmax, mmax, jd64):
    """More edges along the polar axis than a block forms the entries of at a time, next to others."""
    cfg = dict(lmax=lmax, mmax=mmax, sphere_channels=16, hidden_channels=8, edge_channels=8,
               num_distance_basis=6, cutoff=8.0)
    params = orc.init_params(cfg, seed=5)
    n = 60
    case = random_case(cfg, n, 200, seed=6)
    case["pos"], case["shifts"] = case["pos"].float().double(), torch.zeros_like(case["shifts"])
    for e in range(90):                                   # pairs of atoms that only these edges touch
        i = e % 15 * 2
        case["edge_index"][:, e] = torch.tensor([i, i + 1])
        case["pos"][i + 1] = case["pos"][i] + torch.tensor([0.0, 1.0 + 0.03125 * i, 0.0])
    for e in range(90, 200):
        i, j = case["edge_index"][:, e].tolist()
        i, j = 30 + i % 30, 30 + j % 30
        case["edge_index"][:, e] = torch.tensor([i, j if j != i else 30 + (i - 29) % 30])
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    got = gpu_node_out_and_vjp(make_block(cfg, params), case, case["upstream"])
    assert rel_l2(got[0], want[0]) < 1e-5
    assert rel_l2(got[2][30:], want[2][30:]) < 1e-5 and rel_l2(got[2][:30], want[2][:30]) < 1e-3


def test_element_numbers_on_the_host_raise():
    from zippel_b200.graph import EdgeGraph
    with pytest.raises(RuntimeError):
        EdgeGraph.build_checked(torch.zeros(2, 3, dtype=torch.int64, device="cuda"),
                                torch.zeros(4, dtype=torch.int64), 5)


def test_element_numbers_as_a_column():
    cfg = dict(lmax=1, mmax=1, sphere_channels=8, hidden_channels=8, edge_channels=8,
               num_distance_basis=4, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1))
    case = random_case(cfg, 6, 20, seed=2)
    want = gpu_node_out_and_vjp(block, case, case["upstream"])
    column = dict(case, atomic_numbers=case["atomic_numbers"][:, None])
    got = gpu_node_out_and_vjp(block, column, case["upstream"])
    for a, b in zip((*got[:3], *got[3].values()), (*want[:3], *want[3].values())):
        assert (a is None and b is None) or torch.equal(a, b)
    column["atomic_numbers"] = column["atomic_numbers"].clone()
    column["atomic_numbers"][2, 0] = block.cfg.max_num_elements
    with pytest.raises(IndexError):
        gpu_node_out_and_vjp(block, column, case["upstream"])


def test_weights_of_the_edge_convolution_by_size():
    """Another arrangement of as many values is taken as it lies in memory; another size is refused."""
    from zippel_b200.blocks import eso2
    from zippel_b200.graph import EdgeGraph
    cfg = dict(lmax=1, mmax=1, sphere_channels=8, hidden_channels=8, edge_channels=8,
               num_distance_basis=4, cutoff=5.0)
    block = make_block(cfg, orc.init_params(cfg, seed=1))
    plan, g = block.plan("cuda"), torch.Generator("cuda").manual_seed(0)
    graph = EdgeGraph.build(torch.randint(0, 6, (2, 20), device="cuda", generator=g), 6)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)            # noqa: E731
    gamma = torch.rand(20, 1, device="cuda", generator=g) * torch.arange(2, device="cuda")
    ins = (rand(6, 4, 8), rand(20, 3), gamma.cos(), gamma.sin(), rand(20, plan.sizes.R), rand(20), None, None)
    w = [block.c1_m0.weight, block.c1_m0.bias, block.c2_m0.weight, block.c2_m0.bias, block.c1_m[0].weight,
         block.c2_m[0].weight]
    with torch.no_grad():
        want = eso2.EdgeConvFunction.apply(plan, graph, *ins, *w)
        flat = [w[0], w[1].reshape(-1, 8), w[2].flatten(), w[3].reshape(2, -1), *w[4:]]
        assert torch.equal(want, eso2.EdgeConvFunction.apply(plan, graph, *ins, *flat))
        with pytest.raises(AssertionError):
            eso2.EdgeConvFunction.apply(plan, graph, *ins, w[0][:-1], *w[1:])


@pytest.mark.parametrize("n,e", [(128, 4096), (129, 4096), (128, 4097), (3, 400), (1, 300), (2, 4096), (100, 7)])
@pytest.mark.parametrize("order", ["any", "rising", "sorted"])
def test_sort_by_one_block(n, e, order):
    """At the line between the sort of one block and the general one, and buckets beyond what registers hold."""
    import numpy as np

    from zippel_b200.graph import EdgeGraph, csr_reference
    g = torch.Generator("cpu").manual_seed(n + e)
    ei = torch.randint(0, n, (2, e), generator=g)
    if order == "sorted":
        ei = ei[:, torch.argsort(ei[0], stable=True)]
    if order != "any":
        ei = ei[:, torch.argsort(ei[1], stable=True)]
    want = csr_reference(ei.numpy(), n)
    got = EdgeGraph.build(ei.cuda(), n)
    for key in ("perm", "src", "dst", "row_ptr", "perm_src", "row_ptr_src"):
        assert np.array_equal(getattr(got, key).cpu().numpy(), want[key]), key
    ei[0, e // 2] = n
    with pytest.raises(IndexError):
        EdgeGraph.build(ei.cuda(), n)


@pytest.mark.parametrize("lmax,mmax,c,precision", [(4, 2, 128, "fp32"), (2, 2, 16, "fp32_bf16x3"), (3, 1, 40, "fp32"),
                                                   (1, 1, 72, "fp32"), (4, 4, 160, "fp32"), (5, 2, 136, "fp32"),
                                                   (6, 2, 24, "fp32_bf16x3"), (2, 0, 256, "fp32"), (1, 0, 8, "fp32")])
def test_rotations_by_node_of_uneven_degrees(lmax, mmax, c, precision, jd64):
    """Nodes of no edge, of one, of fewer than a block has workers, and a hub each way; with and without a
    gradient of x_node."""
    cfg = dict(lmax=lmax, mmax=mmax, sphere_channels=c, hidden_channels=16, edge_channels=8,
               num_distance_basis=6, cutoff=5.0)
    params = orc.init_params(cfg, seed=71)
    case = random_case(cfg, 30, 260, seed=72)
    ei = case["edge_index"]
    ei[1, :90] = 4                                     # into one
    ei[0, 90:150] = 7                                  # out of one
    ei[:, 150:] = torch.where((ei[:, 150:] == 9) | (ei[:, 150:] == 0), 11, ei[:, 150:])
    ei[0] = torch.where(ei[0] == ei[1], (ei[0] + 1) % 29 + 1, ei[0])
    want = oracle_node_out_and_vjp(cfg, params, case, case["upstream"], jd64)
    block = make_block(cfg, params, precision=precision)
    got = gpu_node_out_and_vjp(block, case, case["upstream"])
    check_against(*got, *want)
    block.requires_grad_(False)
    pos = case["pos"].cuda().float().requires_grad_(True)
    out = block.node_output(pos, case["atomic_numbers"].cuda(), case["x_node"].cuda().float(), ei.cuda(),
                            *(case[k].cuda().float() for k in ("shifts", "cos_gamma_k", "sin_gamma_k")))
    (gpos,) = torch.autograd.grad(out, pos, case["upstream"].cuda().float())
    assert rel_l2(gpos, want[2]) < 1e-5
