"""The side streams of a call (``ZpLanes``): the caller's stream waits for all they were given, also
where the call ends with an error between fork and join.  Host code, compiled and run without a GPU."""

from __future__ import annotations

import pathlib
import subprocess

import pytest

from zippel_b200.build import CSRC, NVCC_FLAGS, ROOT, nvcc


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    exe = tmp_path_factory.mktemp("lanes") / "lanes"
    src = pathlib.Path(__file__).parent / "native" / "lanes.cu"
    subprocess.run([nvcc(), *NVCC_FLAGS, "-cudart", "shared", "-I", str(ROOT / "include"), "-I", str(CSRC),
                    str(src), "-o", str(exe)], check=True, capture_output=True)

    def run(edges, script, fail_at=-1):
        rc, unlocked, *log = subprocess.run([str(exe), str(edges), script, str(fail_at)], check=True,
                                            capture_output=True, text=True).stdout.split()
        assert unlocked == "1"
        return int(rc), log
    return run


FORK1, FORK2 = ["record7@1", "2waits7"], ["record7@1", "3waits7"]
FORK, JOIN1, JOIN2 = ["record7@1", "2waits7", "3waits7"], ["record8@2", "1waits8"], ["record9@3", "1waits9"]


@pytest.mark.parametrize("script,want", [
    ("f3j3", FORK + JOIN1 + JOIN2),                  # as before: nothing is added to a joined call
    ("f1f1j1f3j3", FORK1 + FORK1 + JOIN1 + FORK + JOIN1 + JOIN2),
    ("f3", FORK + JOIN1 + JOIN2),                    # the call ended after the fork
    ("f3j1", FORK + JOIN1 + JOIN2),
    ("f2", FORK2 + JOIN2),
    ("f3j3f1", FORK + JOIN1 + JOIN2 + FORK1 + JOIN1),
    ("", []),
])
def test_every_call_ends_joined(lanes, script, want):
    assert lanes(5000, script) == (0, want)


def test_small_calls_have_no_lanes(lanes):
    assert lanes(4096, "f3j3") == (0, [])


@pytest.mark.parametrize("fail_at", range(7))
def test_a_failing_event_call_leaves_the_other_lane_joined(lanes, fail_at):
    rc, log = lanes(5000, "f3j3", fail_at)
    assert rc != 0
    for stream, event in (("2", "8"), ("3", "9")):
        if f"{stream}waits7" in log:                 # it has been given work
            assert f"1waits{event}" in log
