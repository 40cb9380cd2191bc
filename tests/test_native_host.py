"""CPU checks of the engine's host-side parts that make no CUDA call of their own: small programs built with g++ and run here."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "rwkv-rsv_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"


def _run(tmp_path, name, *flags):
    exe = tmp_path / name
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, *flags, os.path.join(ROOT, "tests", "native", name + ".cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout[-2000:]
    return run.stdout


def test_decode_launches_continue_after_one_that_failed(tmp_path):
    assert "sequence ok" in _run(tmp_path, "stream_sequence_check")


def test_logits_that_arrive_in_parts(tmp_path):
    assert "parts ok" in _run(tmp_path, "parts_to_host_check")


def test_rows_are_cut_into_no_more_turns_than_the_widest_tiles_need(tmp_path):
    assert "row tiles ok" in _run(tmp_path, "row_tiles_check")


@pytest.mark.skipif(not os.path.exists(CUDA_INCLUDE), reason="no CUDA headers")
def test_memory_of_freed_states_is_given_back(tmp_path):
    assert "device memory ok" in _run(tmp_path, "device_memory_check", "-I", CUDA_INCLUDE)


@pytest.mark.skipif(not os.path.exists(CUDA_INCLUDE), reason="no CUDA headers")
def test_scored_texts_take_shorter_passes_where_memory_is_short(tmp_path):
    assert "passes ok" in _run(tmp_path, "passes_check", "-I", CUDA_INCLUDE)
