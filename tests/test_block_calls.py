"""What the whole-block autograd functions hand to the library, without a GPU: the library call is
replaced by one that looks at its arguments."""

from __future__ import annotations

import types

import pytest
import torch
import torch.nn.utils.parametrizations
import torch.nn.utils.parametrize
import torch.nn.utils.prune
from torch.autograd.graph import saved_tensors_hooks
from torch.utils.checkpoint import checkpoint

from tests.helpers import random_case
from zippel_b200 import _lib
from zippel_b200.blocks import eso2
from zippel_b200.graph import EdgeGraph, csr_reference

CFG = dict(lmax=2, mmax=1, sphere_channels=8, hidden_channels=8, edge_channels=8,
           num_distance_basis=6, cutoff=5.0)


class FakeLibrary:
    """Stands in for ``_lib``: keeps the arguments of every call, writes nothing."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return getattr(_lib, name)

    def load(self):
        return types.SimpleNamespace(zp_block_workspace_bytes=lambda *a: 4096,
                                     zp_readout_work_bytes=lambda *a: 4096)

    def run(self, device, name, *args):
        self.calls.append((name, args))


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(eso2, "_lib", lib)
    monkeypatch.setattr(eso2, "_need_cuda", lambda *tensors: None)
    block = eso2.ESO2Block(eso2.BlockConfig(**CFG))
    k = (CFG["lmax"] + 1) ** 2
    plan = types.SimpleNamespace(handle=None, c=8, h=8, lmax=CFG["lmax"], mmax=CFG["mmax"],
                                 sizes=types.SimpleNamespace(K=k), precision=2,
                                 device=torch.device("cpu"), bytes_per_edge=1.0, total_memory=1 << 40, foreign=0)
    monkeypatch.setattr(block, "plan", lambda device: plan)
    case = {key: v.float() if v.is_floating_point() else v for key, v in random_case(CFG, 9, 40, seed=1).items()}
    csr = csr_reference(case["edge_index"].numpy(), 9)
    graph = EdgeGraph(9, 40, **{key: torch.from_numpy(v) for key, v in csr.items()})
    return lib, block, case, graph


def node_output(block, case, graph, pos, x, z=None):
    return block.node_output(pos, case["atomic_numbers"] if z is None else z, x, case["edge_index"],
                             case["shifts"], case["cos_gamma_k"], case["sin_gamma_k"], graph=graph)


def backward_addresses(lib):
    """Addresses of x_node, atomic_numbers, Gaussian offsets and LayerNorm parameters, and the workspace."""
    (args,) = [a for name, a in lib.calls if name == "zp_block_backward"]
    call, params = args[2], args[3]
    return {call.x_node, call.atomic_numbers, params.gauss_offsets, *params.ln_gamma, *params.ln_beta, args[8]}


@pytest.mark.parametrize("what,entry", [("hooks", "node_output"), ("hooks", "energy"),
                                        ("checkpoint", "node_output"), ("checkpoint", "energy")])
def test_the_backward_reads_the_tensors_that_were_brought_back(fake, what, entry, monkeypatch):
    lib, block, case, graph = fake
    alive = []

    def unpack(t):
        alive.append(t.clone())
        return alive[-1]

    def layer(a):
        # an intermediate, and copies that only the call itself makes
        x, z = torch.tanh(a).double(), case["atomic_numbers"].int()
        args = (case["pos"], z, x, case["edge_index"], case["shifts"], case["cos_gamma_k"], case["sin_gamma_k"])
        return block.node_output(*args, graph=graph) if entry == "node_output" else block(*args, graph=graph)

    a = case["x_node"].requires_grad_(True)
    if what == "hooks":
        with saved_tensors_hooks(lambda t: t.clone(), unpack):
            out = layer(a)
        out.sum().backward()
    else:
        vjp = eso2._block_vjp
        monkeypatch.setattr(eso2, "_block_vjp",
                            lambda ctx, saved, *rest: (alive.extend(saved), vjp(ctx, saved, *rest))[1])
        checkpoint(layer, a, use_reentrant=False).sum().backward()
    assert backward_addresses(lib) <= {t.data_ptr() for t in alive}


def test_parameters_are_listed_in_registration_order():
    for lmax, mmax in ((0, 0), (2, 0), (3, 3), (6, 2)):
        block = eso2.ESO2Block(eso2.BlockConfig(**{**CFG, "lmax": lmax, "mmax": mmax, "hidden_channels": 16}))
        listed = block._call_params(True)
        assert [id(p) for p in listed] == [id(p) for p in block.parameters()]
        assert [id(p) for p in block._call_params(False)] == [id(p) for p in listed[:-4]]


@pytest.mark.parametrize("what", ["pruned", "weight_norm", "parametrized", "more parameters"])
def test_layers_that_form_their_weights_are_asked_for_them(fake, what):
    """The addresses the library gets are those of the weights the layers form, in their places."""
    lib, block, case, graph = fake
    torch.manual_seed(0)
    if what == "pruned":
        torch.nn.utils.prune.l1_unstructured(block.rad_func[0], "weight", 0.5)
        torch.nn.utils.prune.l1_unstructured(block.c1_m0, "weight", 0.5)
    elif what == "weight_norm":
        torch.nn.utils.parametrizations.weight_norm(block.rad_func[3])
        torch.nn.utils.parametrizations.weight_norm(block.c2_m[0])
    elif what == "parametrized":
        class Twice(torch.nn.Module):
            def forward(self, w):
                return 2 * w
        torch.nn.utils.parametrize.register_parametrization(block.elem_emb, "weight", Twice())
        torch.nn.utils.parametrize.register_parametrization(block.c2_m0, "bias", Twice())
    else:
        block.scale = torch.nn.Parameter(torch.ones(3))
        block.head2 = torch.nn.Linear(4, 4)
    want = [block.elem_emb.weight, *[t for i in (0, 1, 3, 4, 6) for t in (block.rad_func[i].weight, block.rad_func[i].bias)],
            block.c1_m0.weight, block.c1_m0.bias, block.c1_m[0].weight,
            block.c2_m0.weight, block.c2_m0.bias, block.c2_m[0].weight]
    got = []
    apply = eso2._block
    eso2._block = lambda *args: (got.extend(args[-1]), apply(*args))[1]
    try:
        node_output(block, case, graph, case["pos"].requires_grad_(True), case["x_node"]).sum().backward()
    finally:
        eso2._block = apply
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert a.shape == b.shape and torch.equal(a, b)
    named = dict(block.named_parameters())
    for name, p in named.items():
        unused = name.startswith(("readout", "scale", "head2"))
        assert (p.grad is None) == unused, name
        assert unused or p.grad.shape == p.shape


@pytest.mark.parametrize("what", ["eps", "bias", "layers"])
def test_radial_mlps_that_the_one_call_does_not_run(fake, what, monkeypatch):
    lib, block, case, graph = fake
    if what == "eps":
        block.rad_func[4].eps = 1e-3
    elif what == "bias":
        block.rad_func[3].bias = None
    else:
        block.rad_func = torch.nn.Sequential(block.rad_func[0], *block.rad_func[1:3], block.rad_func[6])
    taken = []
    monkeypatch.setattr(eso2, "_edge_budget", lambda *args: 1 << 20)
    monkeypatch.setattr(block, "_edges_to_nodes_in_parts", lambda *args: taken.append(args) or case["x_node"])
    node_output(block, case, graph, case["pos"], case["x_node"])
    assert len(taken) == 1 and not lib.calls


@pytest.mark.parametrize("entry", ["node_output", "energy"])
def test_tangents_of_frozen_parameters_are_refused(fake, entry):
    """There is no forward mode: as on a tensor argument, a tangent on a parameter raises and is not lost."""
    import torch.autograd.forward_ad as fwad
    lib, block, case, graph = fake
    block.requires_grad_(False)
    args = (case["pos"], case["atomic_numbers"], case["x_node"], case["edge_index"], case["shifts"],
            case["cos_gamma_k"], case["sin_gamma_k"])
    call = block.node_output if entry == "node_output" else block
    with fwad.dual_level():
        w = fwad.make_dual(block.c1_m0.weight.detach(), torch.ones_like(block.c1_m0.weight))
        del block.c1_m0._parameters["weight"]
        block.c1_m0.weight = w
        with pytest.raises(RuntimeError, match="forward"):
            call(*args, graph=graph)


@pytest.mark.parametrize("what", ["nothing", "energy", "node_output", "instance"])
def test_the_energy_goes_through_overridden_methods(fake, what, monkeypatch):
    lib, block, case, graph = fake
    seen = []

    def energy(self, out):
        seen.append("energy")
        return out.sum()

    def node_output(self, *args):
        seen.append("node_output")
        return eso2.ESO2Block.node_output(self, *args)

    monkeypatch.setattr(eso2, "Readout", types.SimpleNamespace(apply=lambda plan, out, *params: out.sum()))
    if what == "instance":
        block.energy = lambda out: energy(block, out)
    elif what != "nothing":
        block.__class__ = type("Own", (eso2.ESO2Block,), {what: {"energy": energy, "node_output": node_output}[what]})
    with torch.no_grad():
        block(case["pos"], case["atomic_numbers"], case["x_node"], case["edge_index"], case["shifts"],
              case["cos_gamma_k"], case["sin_gamma_k"], graph=graph)
    assert seen == {"nothing": [], "instance": ["energy"]}.get(what, [what])


def test_when_a_call_is_made_in_one_piece(monkeypatch):
    gib = 1 << 30
    plan = types.SimpleNamespace(device=torch.device("cuda", 0), bytes_per_edge=2.0 ** 17, total_memory=160 * gib,
                                 foreign=8 * gib)
    held = [0]
    monkeypatch.setattr(eso2, "_allocated", lambda device: held[0])
    edges = lambda g: int(g * gib / plan.bytes_per_edge)                             # noqa: E731
    assert eso2._one_piece(plan, edges(10), True, 4) and eso2._one_piece(plan, edges(10), False, 4)
    assert not eso2._one_piece(plan, edges(10.1), True, 4) and not eso2._one_piece(plan, edges(10.1), False, 4)
    # layers that keep their activations stop short of filling the device, in the end layer by layer
    held[0] = 112 * gib
    assert eso2._one_piece(plan, edges(10), True, 4) and not eso2._one_piece(plan, edges(10) + 1, True, 4)
    held[0] = 113 * gib
    assert not eso2._one_piece(plan, edges(10), True, 4) and eso2._one_piece(plan, edges(10), True, 2)
    plan.foreign = 100 * gib
    assert not eso2._one_piece(plan, edges(10), True, 2) and eso2._one_piece(plan, edges(10), False, 2)
    monkeypatch.setattr(eso2, "MAX_EDGES_PER_CALL", 64)
    assert not eso2._one_piece(plan, 8, False, 4)


def test_the_flags_of_a_sort_are_waited_for_whatever_happens(fake, monkeypatch):
    lib, block, case, graph = fake
    checked = []
    monkeypatch.setattr(block, "_sorted_edges", lambda *args: (graph, lambda: checked.append(1)))
    for what in ("plan", "_call_params"):
        with monkeypatch.context() as m:
            m.setattr(block, what, lambda *args: 1 / 0)
            with pytest.raises(ZeroDivisionError):
                node_output(block, case, None, case["pos"], case["x_node"])
    assert len(checked) == 2


def test_host_tensors_are_refused_before_their_addresses_are_taken(monkeypatch):
    """Each argument in turn is the only one not on the device (here: the only one said not to be)."""
    block = eso2.ESO2Block(eso2.BlockConfig(**CFG))
    seen = []
    monkeypatch.setattr(eso2, "_need_cuda", lambda *tensors: seen.extend(tensors) or 1 / 0)
    case = {key: v.float() if v.is_floating_point() else v for key, v in random_case(CFG, 9, 40, seed=1).items()}
    csr = csr_reference(case["edge_index"].numpy(), 9)
    graph = EdgeGraph(9, 40, **{key: torch.from_numpy(v) for key, v in csr.items()})
    plan = types.SimpleNamespace(sizes=types.SimpleNamespace(K=9), c=8)
    ctx = types.SimpleNamespace(needs_input_grad=(False,))
    with pytest.raises(ZeroDivisionError):
        eso2._block(ctx, block, plan, graph, None, case["atomic_numbers"], case["shifts"], case["cos_gamma_k"],
                    case["sin_gamma_k"], None, case["pos"], case["x_node"], block._call_params(False))
    at = {t.data_ptr() for t in seen}
    assert {case[k].data_ptr() for k in ("pos", "x_node", "shifts", "atomic_numbers", "cos_gamma_k",
                                         "sin_gamma_k")} <= at
    assert block.gauss_offset.data_ptr() in at and {p.data_ptr() for p in block._call_params(False)} <= at


def test_element_numbers_as_a_column(fake):
    """[N, 1], and more entries than atoms: the kernels read the first N."""
    lib, block, case, graph = fake
    for z in (case["atomic_numbers"][:, None], torch.cat([case["atomic_numbers"]] * 2)):
        assert node_output(block, case, graph, case["pos"], case["x_node"], z).shape == case["x_node"].shape
        assert lib.calls[-1][1][2].atomic_numbers == z.data_ptr()
    with pytest.raises(AssertionError):
        node_output(block, case, graph, case["pos"], case["x_node"], case["atomic_numbers"][:-1])


@pytest.mark.parametrize("parts", [False, True])
@pytest.mark.parametrize("form", ["int64", "strided"])
def test_a_graph_whose_order_is_of_another_type(fake, form, parts, monkeypatch):
    """The order of a graph made by hand, as int64 or a column of a table: the library gets int32."""
    import ctypes
    lib, block, case, graph = fake
    monkeypatch.setattr(eso2, "_edge_budget", lambda *args: 1 << 20)
    want, got = graph.perm.tolist(), []
    graph.perm = graph.perm.long() if form == "int64" else torch.stack([graph.perm, graph.perm], 1)[:, 0]
    if parts:
        block.rad_func[1].eps = 1e-3
        monkeypatch.setattr(eso2, "EdgeFeatures",
                            types.SimpleNamespace(apply=lambda g, perm, *rest: got.extend(
                                (perm.dtype, perm.is_contiguous(), *perm.tolist())) or 1 / 0))
        with pytest.raises(ZeroDivisionError):
            node_output(block, case, graph, case["pos"], case["x_node"])
        assert got == [torch.int32, True, *want]
    else:
        monkeypatch.setattr(lib, "run", lambda device, name, *args: got.extend(
            (ctypes.c_int32 * 40).from_address(args[2].perm)))
        node_output(block, case, graph, case["pos"], case["x_node"])
        assert got == want


def test_no_atoms_have_zero_parameter_gradients(fake, monkeypatch):
    lib, block, case, graph = fake
    monkeypatch.setattr(torch, "empty",                              # what fresh memory may hold
                        lambda *a, **k: torch.zeros(*a, **k) + (7 if k.get("dtype") is torch.float32 else 0))
    i32 = lambda n: torch.zeros(n, dtype=torch.int32)                                # noqa: E731
    none = EdgeGraph(0, 0, i32(0), i32(0), i32(0), i32(1), i32(0), i32(1))
    case = {k: v[:0] for k, v in case.items()}
    x, pos = case["x_node"].requires_grad_(True), case["pos"].requires_grad_(True)
    out = node_output(block, case, none, pos, x)
    grads = torch.autograd.grad(out, [pos, x, *block._call_params(False)], torch.zeros_like(out))
    assert all(g.abs().sum() == 0 for g in grads)


def test_edge_conv_lists_the_weights_of_its_layers(fake, monkeypatch):
    _, block, case, graph = fake
    got = []
    monkeypatch.setattr(eso2, "EdgeConvFunction", types.SimpleNamespace(apply=lambda *args: got.extend(args)))
    rest = [object() for _ in range(8)]
    eso2.edge_conv(*rest, block.c1_m0, block.c1_m, block.c2_m0, block.c2_m)
    assert got[:8] == rest and got[8:10] == [None, None]
    assert [t.shape for t in got[10:]] == eso2._so2_shapes(2, 1, 8, 8)
    assert got[14] is block.c1_m[0].weight and got[15] is block.c2_m[0].weight


@pytest.mark.parametrize("which", [0, 1])
def test_a_readout_of_other_widths_is_refused(fake, which):
    lib, block, case, graph = fake
    eso2._readout(block.plan("cpu"), case["x_node"], block._call_params(True)[-4:])
    if which:
        block.readout[2] = torch.nn.Linear(8, 2)
    else:
        block.readout[0] = torch.nn.Linear(24, 4)
    head = [block.readout[0].weight, block.readout[0].bias, block.readout[2].weight, block.readout[2].bias]
    with pytest.raises(ValueError, match="readout"):
        eso2._readout(block.plan("cpu"), case["x_node"], head)
