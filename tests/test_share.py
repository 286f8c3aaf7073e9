"""How the tiles of a launch's products are shared out (``share_out``): every tile to one unit, and no unit with
more to do than when the tiles are handed out one by one, longest first.  Host code, run without a GPU."""

from __future__ import annotations

import pathlib
import subprocess

import pytest

from zippel_b200.build import CSRC, NVCC_FLAGS, ROOT, nvcc


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    exe = tmp_path_factory.mktemp("share") / "share"
    src = pathlib.Path(__file__).parent / "native" / "share.cu"
    subprocess.run([nvcc(), *NVCC_FLAGS, "-cudart", "shared", "-I", str(ROOT / "include"), "-I", str(CSRC),
                    str(src), "-o", str(exe)], check=True, capture_output=True)
    return lambda seed: subprocess.run([str(exe), str(seed), "2000"], capture_output=True, text=True).stdout


@pytest.mark.parametrize("seed", range(3))
def test_every_tile_once_and_loads_as_one_by_one(share, seed):
    assert share(seed) == "ok\n"
