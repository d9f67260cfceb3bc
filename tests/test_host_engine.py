"""The engine's host code on the CPU, over a CUDA runtime of host memory
(tests/host_engine): what it makes of calls that fail."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def _build(out, *flags):
    subprocess.run(["g++", "-std=c++17", "-w", "-g", *flags, "-I", os.path.join(HERE, "host_engine"), "-I",
                    os.path.join(ROOT, "include"), os.path.join(HERE, "host_engine", "cases.cpp"),
                    os.path.join(ROOT, "empanada_b200", "csrc", "ingest.cpp"), "-o", out, "-lz", "-lpthread"],
                   check=True)
    return out


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("host_engine") / "cases"))


@pytest.mark.parametrize("case", ["rebuilt_list_times_out", "graph_input_copy_fails", "thread_allocation_fails",
                                  "graphs_make_room", "sort_room_refused",
                                  "step_ends_early", "graph_keeps_the_device"])
def test_a_failing_call_is_a_status(program, case):
    p = subprocess.run([program, case], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, (p.returncode, p.stderr)


def test_graphs_from_other_threads(tmp_path):
    """Under the thread sanitizer where the compiler has one."""
    try:
        exe = _build(str(tmp_path / "cases"), "-O1", "-fsanitize=thread")
    except subprocess.CalledProcessError:
        exe = _build(str(tmp_path / "cases"))
    p = subprocess.run([exe, "graphs_from_threads"], capture_output=True, text=True, timeout=90)
    assert p.returncode == 0, (p.returncode, p.stderr[-3000:])
