"""Host-side parts of the CUDA library that need no device, built with g++ against stand-ins for what they call."""
import os
import subprocess

from conftest import PKG_NAME, ROOT


def _run(tmp_path, name, *flags):
    exe = str(tmp_path / name)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-Wall", os.path.join(ROOT, "tests", "integration", name + ".cpp"), "-I", os.path.join(ROOT, PKG_NAME, "csrc"),
                           "-I", "/usr/local/cuda/include", *flags, "-o", exe])
    done = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr


def test_pool_keeps_what_a_recorded_graph_addresses(tmp_path):
    _run(tmp_path, "pool")


def test_threads_that_cannot_be_started_leave_their_share(tmp_path):
    _run(tmp_path, "host_threads", "-pthread")


def test_pages_that_are_asked_for_keep_what_they_hold(tmp_path):
    _run(tmp_path, "pages", "-pthread")


def test_programs_on_the_cpp_headers_compile():
    """What a separately compiled program may call through HEMMer.hpp, calls that the library does not make itself among them."""
    for name in ("hemmer_snippet", "operands_after_error", "evaluator_calls"):
        subprocess.check_call(["g++", "-fsyntax-only", "-std=c++17", "-Wall", os.path.join(ROOT, "tests", "integration", name + ".cpp"), "-I", os.path.join(ROOT, "include"),
                               "-I", os.path.join(ROOT, PKG_NAME, "csrc", "hellm")])


def test_shared_memory_of_the_conversions(tmp_path):
    _run(tmp_path, "conv_shared")


def test_twiddle_values(tmp_path):
    _run(tmp_path, "twiddles")


def test_rules_of_dispatch_take_what_was_measured_quicker(tmp_path):
    _run(tmp_path, "launch_rules")


def test_buffers_that_a_call_can_do_without(tmp_path):
    _run(tmp_path, "pool_spare")


def test_threads_that_ask_for_pages_stay_within_their_cap(tmp_path):
    _run(tmp_path, "page_threads", "-pthread")
