"""The group form's step (csrc/fk_group.cuh) compiled for the host, one warp on 32
threads, and the statuses of a set of sources (group_step_host.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gemini_unified_b200", "csrc")


def _build(tmp_path, *flags):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    open(tmp_path / "cuda_runtime.h", "w").close()   # the harness declares what the headers need
    exe = str(tmp_path / "warp")
    cmd = ["g++", "-std=c++17", "-ffp-contract=off", "-w", "-I", str(tmp_path), "-I", CSRC, *flags,
           os.path.join(HERE, "group_step_host.cpp"), "-o", exe, "-pthread"]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    if "-ltsan" in r.stderr or "libtsan" in r.stderr:
        pytest.skip("no thread sanitizer")
    assert r.returncode == 0, r.stderr[-2000:]
    return exe


def test_shared_memory_is_ordered(tmp_path):
    """No access to the group's shared memory that only a vote separates from another lane's."""
    r = subprocess.run([_build(tmp_path, "-O1", "-g", "-fsanitize=thread"), "race"], capture_output=True, text=True, timeout=600)
    if "unexpected memory mapping" in r.stderr:
        pytest.skip("the sanitizer cannot map its memory here")
    assert "data race" not in r.stderr, r.stderr[:2000]
    assert r.returncode == 0, r.stderr[:2000]


def test_group_form_equals_thread_form(tmp_path):
    """Steps of every size, from one whose attempts agree to one whose attempts overflow: the
    group form makes more attempts than the thread form and may use no more of them."""
    r = subprocess.run([_build(tmp_path, "-O2"), "compare"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout


def test_status_of_a_set_of_sources(tmp_path):
    """An item takes the status of its first source that failed; the spheroidal spectra of the
    sources after it are cleared, the blocks before it and the toroidal spectra stay."""
    assert subprocess.run([_build(tmp_path, "-O1"), "status"], timeout=600).returncode == 0
