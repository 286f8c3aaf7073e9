"""How the edges of nodes that have very many are dealt out to blocks (``NodeEdges``): every edge half to one block.
Device code that runs on the host as well, compiled and run without a GPU."""

from __future__ import annotations

import pathlib
import subprocess

import pytest

from zippel_b200.build import CSRC, NVCC_FLAGS, ROOT, nvcc


@pytest.fixture(scope="module")
def cuts(tmp_path_factory):
    exe = tmp_path_factory.mktemp("cuts") / "cuts"
    src = pathlib.Path(__file__).parent / "native" / "cuts.cu"
    subprocess.run([nvcc(), *NVCC_FLAGS, "-cudart", "shared", "-I", str(ROOT / "include"), "-I", str(CSRC),
                    str(src), "-o", str(exe)], check=True, capture_output=True)
    return lambda seed: subprocess.run([str(exe), str(seed), "600"], capture_output=True, text=True).stdout


@pytest.mark.parametrize("seed", range(3))
def test_every_edge_half_is_in_one_stretch(cuts, seed):
    assert cuts(seed) == "ok\n"
