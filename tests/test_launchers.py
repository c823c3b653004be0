"""The launchers that set kernel attributes, over a stand-in CUDA runtime
(fake_cudart.cpp): a call's own size is never left behind for other threads'
calls, every device gets its attributes, and a refused launch is reported as
not launched, with no error left, so that the caller takes the other route;
and the caller's memory that a kernel may write."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def said(tmp_path_factory):
    from ion_gym_gb300 import build as B
    if not os.path.exists(os.path.join(B.OUT_DIR, "ig_f64.o")):
        B.build(force=True)
    exe = str(tmp_path_factory.mktemp("launchers") / "launchers")
    include = os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", B.CSRC, "-I", include,
                    os.path.join(HERE, "fake_cudart.cpp"),
                    os.path.join(B.OUT_DIR, "ig_f64.o"), os.path.join(B.OUT_DIR, "ig_solvers.o"),
                    "-o", exe, "-lpthread"], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return dict(line.split(" ", 1) for line in out.splitlines())


TOOK, REFUSED = "took=1 launched=1 error=0", "took=0 launched=0 error=0"


def test_sor_attribute_is_not_a_calls_own(said):
    assert said["sor-large"] == said["sor-small"] == TOOK
    assert said["sor-attribute"] == "lowered=0"


def test_sor_on_a_second_device_and_refused(said):
    assert said["sor-second-device"] == TOOK
    assert said["sor-refused"] == REFUSED


@pytest.mark.parametrize("device", [0, 1])
def test_cluster_and_bottom_on_every_device(said, device):
    assert said[f"tail-device{device}"] == TOOK
    assert said[f"bottom-device{device}"] == TOOK


def test_cluster_and_bottom_refused(said):
    assert said["tail-refused"] == REFUSED
    assert said["bottom-refused"] == REFUSED


CAP = 1  # IG_NOT_CONVERGED: the stand-in's loop never meets its tolerance


@pytest.mark.parametrize("what,want", [
    ("alone", (CAP, 1, 0, 100)),
    ("alone-turns", (CAP, 3, 0, 600)),      # a turn of 65^3 is 258 pairs
    ("no-pairs", (CAP, 0, 0, 0)),
    ("beside-a-session", (0, 0, 1, 1)),
    ("small-beside-a-session", (0, 0, 1, 1)),
    ("session-on-the-other-device", (CAP, 1, 0, 100)),
    ("beside-three-solves", (CAP, 1, 0, 100)),
    ("beside-four-solves", (0, 0, 1, 1)),
    ("small-beside-four-solves", (CAP, 1, 0, 100)),
    ("alone-again", (CAP, 1, 0, 100)),
    ("refused", (0, 0, 1, 1)),
    ("refused-later", (0, 1, 1, 259)),
    ("no-memory", (0, 0, 1, 1))])
def test_who_gets_the_resident_loop(said, what, want):
    """solve3d's loop holds every SM: alone, or among few or small solves, and
    nowhere else; what it cannot do the launched sweeps take up."""
    assert said[what] == "status=%d loops=%d launched=%d sweeps=%d" % want


@pytest.mark.parametrize("what,direct", [
    ("whole", 1), ("inside", 1), ("past", 0), ("odd", 0), ("float", 1), ("odd-float", 0),
    ("host", 0), ("other-device", 0)])
def test_results_a_kernel_may_write(said, what, direct):
    assert said["range-" + what] == str(direct)
