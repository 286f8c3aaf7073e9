"""What the whole-block autograd functions hand to the library, without a GPU: the library call is
replaced by one that looks at its arguments."""

from __future__ import annotations

import types

import pytest
import torch
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
                                 device=torch.device("cpu"), bytes_per_edge=1.0, total_memory=1 << 40)
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
