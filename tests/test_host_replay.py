"""The host code of replayed one-shot calls, run on stand-ins for the CUDA
runtime and the kernels' launchers (tests/host): events that only another
thread or a failing call brings about, at the moment they matter."""
import os
import subprocess

import pytest

from cvmatch_gb300 import build as b

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host")


def compile_host(name, out):
    exe = os.path.join(str(out), name)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-Wall", "-I" + os.path.join(b.ROOT, "include"),
                    "-I" + b.CSRC, "-I" + os.path.join(b._cuda_home(), "include"), os.path.join(HERE, name + ".cpp"),
                    os.path.join(b.CSRC, "cvm_plan.cpp"), "-o", exe, "-lpthread"], check=True)
    return exe


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    return compile_host("replay", tmp_path_factory.mktemp("host"))


@pytest.mark.parametrize("event", ["autotune_off", "plan_published"])
def test_one_plan_for_the_size_and_the_launches(replay, event):
    r = subprocess.run([replay, event], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr


def test_an_error_return_has_waited_for_what_reads_the_callers_memory(replay):
    r = subprocess.run([replay, "errors"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("event", ["threads_share", "threads_bounded", "shapes_in_turn", "memory_given_back"])
def test_what_the_process_keeps_is_bounded_and_shared(replay, event):
    r = subprocess.run([replay, event], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


def test_large_templates_are_read_in_place_beside_large_frames(replay):
    r = subprocess.run([replay, "staged_templates"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
