"""The library's host code (contexts, copies, commitments) over a runtime without a device, compiled for the host: what happens when a call
of the runtime fails, or a thread cannot be made."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_api") / "host_api_emul")
    csrc = os.path.join(ROOT, "intelligenceregulation_b200", "csrc")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++17", "-O2", f"-I{cuda}/include", f"-I{csrc}", "-x", "c++", os.path.join(ROOT, "tests", "host_emul", "host_api_emul.cpp"),
                           *[os.path.join(csrc, f) for f in ("api.cu", "host_copy.cu", "commit_api.cu")], "-o", exe, "-lpthread", "-ldl"])
    return exe


def _ok(*argv):
    r = subprocess.run(argv, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout[-2000:], r.stderr[-500:])


def test_a_failing_call_leaves_no_copy_behind(emul):
    """every fallible runtime call of the commitments and openings fails in turn: no memory is freed while a copy on another stream uses it,
    no copy uses the caller's memory after the call, nothing is lost, and the next call works"""
    _ok(emul, "failures")


def test_an_encoder_wait_that_runs_out_is_told_to_its_own_store(emul):
    _ok(emul, "timeouts")


def test_an_encoding_is_put_into_the_columns_order_once(emul):
    """where a call fails behind the launch the rows are in order all the same; few rows of scratch are enough"""
    _ok(emul, "reorder")


def test_rows_of_every_length_come_in_pieces(emul):
    _ok(emul, "pieces")


def test_copies_of_all_sizes(emul):
    """the limits between the forms of a copy, unaligned ends, and more small copies in a call than the bounce areas hold"""
    _ok(emul, "copies")


@pytest.mark.parametrize("threads", [0, 1, 3, 100])
def test_copies_where_few_threads_can_be_made(emul, threads):
    _ok(emul, "threads", str(threads))
