"""Fleets' host logic on stand-ins for the CUDA runtime and the kernels'
launchers (tests/host)."""
import subprocess

import pytest

from test_host_replay import compile_host


@pytest.fixture(scope="module")
def fleet(tmp_path_factory):
    return compile_host("fleet", tmp_path_factory.mktemp("host"))


def _run(exe, what):
    r = subprocess.run([exe, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr


def test_plans_are_timed_once_for_either_source_of_den(fleet):
    _run(fleet, "tuned_once")


@pytest.mark.parametrize("what", ["the_choice_follows", "captured_first", "a_stream_follows"])
def test_the_source_of_den_follows_the_frames(fleet, what):
    _run(fleet, what)


def test_a_stream_keeps_the_spectra_that_its_graphs_use(fleet):
    _run(fleet, "a_streams_spectra")


def test_only_a_call_that_times_plans_waits_for_the_callers_stream(fleet):
    _run(fleet, "no_waiting")


def test_a_kernel_reads_only_frames_that_are_locked_whole(fleet):
    _run(fleet, "partly_locked")
