"""The ring that large uploads go through (stager.h), compiled against a stand-in for
the CUDA runtime: no GPU, and the stream and its errors are the test's."""
import subprocess
from pathlib import Path

import pytest

TESTS = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("stager") / "check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(TESTS / "fake_cuda"),
                    "-I", str(TESTS.parent / "tileink_b200" / "csrc"), str(TESTS / "stager_check.cpp"), "-o", str(out)],
                   check=True)
    return out


def check(program, mode):
    assert subprocess.run([str(program), mode], timeout=120).returncode == 0


def test_uploads_arrive_whole(program):
    check(program, "data")


def test_fillers_sleep_while_the_stream_is_busy(program):
    check(program, "busy")


def test_a_failed_copy_leaves_the_slots_in_flight_alone(program):
    check(program, "fail")


def test_a_context_takes_the_ring_where_it_pays_and_asks_once(program):
    check(program, "context")
