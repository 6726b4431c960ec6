"""The host layer's own code (staged copies, result memory) built with g++ against a stand-in for the CUDA runtime
(tests/cpu_checks/fake_cuda.hpp), whose calls can be made to fail."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKS = os.path.join(ROOT, "tests", "cpu_checks")
CSRC = os.path.join(ROOT, "comet_b200", "csrc")


def build(exe, check, *sources):
    # the entry points of other files are not called
    subprocess.check_call(["g++", "-O1", "-g", "-std=c++17", "-pthread", "-I/usr/local/cuda/include", "-x", "c++",
                           os.path.join(CHECKS, check)] + [os.path.join(CSRC, s) for s in sources] +
                          ["-no-pie", "-Wl,--unresolved-symbols=ignore-in-object-files", "-o", exe])
    return exe


@pytest.fixture(scope="module")
def download_errors(tmp_path_factory):
    return build(str(tmp_path_factory.mktemp("checks") / "download_errors"), "download_errors_check.cpp", "abi_host.cu",
                 "hostcopy.cu")


@pytest.mark.parametrize("memory,call,n", [("pinned", "copy", 2), ("pinned", "copy", 3), ("pageable", "copy", 2),
                                           ("pageable", "copy", 4), ("pageable", "copy", 6), ("pinned", "sync", 1),
                                           ("pageable", "sync", 1)])
def test_a_call_that_failed_no_longer_writes_to_its_results(download_errors, memory, call, n):
    out = subprocess.run([download_errors, memory, call, str(n)], stdout=subprocess.PIPE, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
    assert out.stdout == "returned 1\n"


def test_the_result_pool_never_makes_a_caller_wait(tmp_path):
    exe = build(str(tmp_path / "result_pool"), "result_pool_check.cpp", "hostmem.cu")
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert (out.returncode, out.stdout) == (0, "ok\n")


def test_without_threads_the_caller_copies_and_nothing_is_thrown(tmp_path):
    exe = build(str(tmp_path / "no_threads"), "no_threads_check.cpp", "hostcopy.cu", "hostmem.cu")
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert (out.returncode, out.stdout) == (0, "ok\n")


def test_operands_of_a_few_mb_are_copied_by_the_caller(tmp_path):
    exe = build(str(tmp_path / "copy_workers"), "copy_workers_check.cpp", "hostcopy.cu")
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert (out.returncode, out.stdout) == (0, "1 several\n")


@pytest.mark.parametrize("host", [[], ["-DNOT_X86"]])
def test_chunks_are_filled_on_any_host(tmp_path, host):
    exe = str(tmp_path / "streamcopy")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(CHECKS, "streamcopy_check.cpp")] + host)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert (out.returncode, out.stdout) == (0, "ok\n")


def test_no_source_needs_an_x86_host():
    """Intrinsics and their header stand behind the architecture's macro."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".cpp")):
            continue
        depth = 0
        with open(os.path.join(CSRC, name)) as f:
            for line in f:
                if line.startswith("#if"):
                    depth = depth + 1 if depth or "__x86_64__" in line else 0
                elif line.startswith("#endif"):
                    depth = max(depth - 1, 0)
                assert depth or not any(w in line for w in ("immintrin.h", "__m256", "_mm_", "_mm256_")), (name, line)
