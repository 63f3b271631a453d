"""The host loop over the rounds (csrc/round_loop.h) with a script in the GPU's place:
the launch shapes follow the live cells, and an error never leaves rounds running."""
import ctypes
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    so = tmp_path_factory.mktemp("rl") / "librl.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(ROOT / "pelelmex_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "round_loop_c.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def go(live, left, warp_cells=9472, graph=1, max_rounds=1000, fail_capture=-1, fail_launch=-1):
        log, running = ctypes.create_string_buffer(4096), ctypes.c_int()
        err = lib.round_loop(ctypes.c_longlong(live), ctypes.c_longlong(warp_cells), ctypes.c_longlong(max_rounds), graph,
                             (ctypes.c_longlong * max(len(left), 1))(*left), len(left), fail_capture, fail_launch, log,
                             ctypes.byref(running))
        assert not running.value  # whatever happened, nothing is left running
        return err, log.value.decode().split()
    return go


LEFT = [150000, 90000, 5000, 300, 0]


def test_shapes_follow_the_live_cells(run):
    assert run(200000, LEFT) == (0, "c0 l0 c1 w l0 w l1 c2 w l2 c3 w l3 w".split())
    assert run(1000, [3, 0]) == (0, "c3 l3 w l3 w".split())
    assert run(200000, [500, 0]) == (0, "c0 l0 c1 w c3 l3 w".split())
    assert run(200000, LEFT, graph=0) == (0, "l0 w l0 w l1 w l2 w l3 w".split())


def test_no_graph_of_a_shape_that_cannot_come(run):
    # no warp form (no generated code): class 2 is empty; one that reaches beyond
    # the cells of class 1 leaves that one empty
    assert run(200000, [90000, 3000, 300, 0], warp_cells=0) == (0, "c0 l0 c1 w l1 c3 w l1 w l3 w".split())
    assert run(200000, [90000, 3000, 300, 0], warp_cells=140000) == (0, "c0 l0 c2 w l2 c3 w l2 w l3 w".split())


def test_graph_made_ahead_that_fails_is_tried_again_when_needed(run):
    # class 2 fails beside the rounds of class 1, and again with nothing running
    assert run(200000, LEFT, fail_capture=2) == (-7, "c0 l0 c1 w l0 w l1 c2 w c2 w".split())
    # not needed: no error
    assert run(200000, [90000, 300, 0], fail_capture=2) == (0, "c0 l0 c1 w l1 c2 w c3 l3 w".split())


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("at", range(5))
def test_failing_launch_is_waited_for(run, graph, at):
    err, log = run(200000, LEFT, graph=graph, fail_launch=at)
    assert err == -8 and log[-1] == "w"


def test_failing_first_graph_and_the_limit_of_rounds(run):
    assert run(200000, LEFT, fail_capture=0) == (-7, ["c0", "w"])
    err, log = run(2000, [2000] * 10, max_rounds=12)
    assert err == -9 and log.count("l2") == 3
