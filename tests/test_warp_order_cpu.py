"""Kernels in which the lanes of a warp hand each other values through shared memory, with their own text compiled by g++ against
tests/cpu_checks/fake_warp.hpp and run under ThreadSanitizer: results are compared, and an access that no barrier orders is a failure."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKS = os.path.join(ROOT, "tests", "cpu_checks")
CSRC = os.path.join(ROOT, "comet_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def function(name, text):
    """The definition of a function, from its first line (a template's or its qualifiers') to its closing brace."""
    at = re.search(r"^[^\n;{}/]*\b%s\(" % name, text, re.M).start()
    start = max(text.rfind("\n\n", 0, at), text.rfind("\n}\n", 0, at) + 1)
    end = text.index("\n}\n", at) + 3
    return re.sub(r"extern __shared__", "extern", text[start:end]) + "\n"


def constant(name, text):
    return re.search(r"^static const [a-z0-9_]+ %s = .*?;" % name, text, re.M).group(0) + "\n"


def body(name, until=None):
    """A header without its includes, up to a line."""
    text = source(name)
    text = text[:text.index(until)] + "}\n" if until else text
    text = re.sub(r"^#(include|pragma).*$", "", text, flags=re.M).replace("extern __shared__", "extern").replace("static __global__", "__global__")
    return relaxed(text)


def relaxed(text):
    return re.sub(r"\*\(volatile [a-z ]+ \*\)(&[\w>-]+)", r"__atomic_load_n(\1, __ATOMIC_RELAXED)", text)


def same_zero(store, text):
    """Several lanes may store the same 0 to a word, which is a race in C++ and none on the device; what they read has to be ordered."""
    assert text.count(store + " = 0;") == 1
    return text.replace(store + " = 0;", "__atomic_store_n(&%s, 0u, __ATOMIC_RELAXED);" % store)


def run(tmp_path, check, code, *args):
    with open(str(tmp_path / "kernels.inc"), "w") as f:
        f.write(code)
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-pthread", "-Wno-unknown-pragmas", "-I" + str(tmp_path),
                           "-I" + CHECKS, "-I" + os.path.join(ROOT, "include"), os.path.join(CHECKS, check), "-o", exe])
    out = subprocess.run([exe] + list(args), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=600)
    assert "data race" not in out.stdout, out.stdout[:3000]
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout[:3000]


def test_short_rows_of_few_columns(tmp_path):
    text = source("spgemm.cu")
    kernel = same_zero("bits[cols[x] >> 5]", function("few_columns_kernel", text))
    run(tmp_path, "few_columns_check.cpp", constant("HASH_ROW_MAX", text) + constant("HASH_WARPS", text) + kernel)


@pytest.mark.parametrize("kernel", ["warp", "mid"])
@pytest.mark.parametrize("out", ["all", "pairs", "values"])
def test_sets_of_a_warp(tmp_path, kernel, out):
    run(tmp_path, "warp_sets_check.cpp", body("semiring.cuh") + body("pairs.cuh", "template <int THREADS, bool SEGMENTED, class Out>\nstatic int"),
        kernel, out)


@pytest.mark.parametrize("graph", ["skewed", "upper", "no room", "even", "regular", "ends in a hub", "unordered", "repeats", "one below"])
def test_triangles_in_another_order(tmp_path, graph):
    order = same_zero("bm[hub[s + q] >> 5]", body("order.cuh"))
    for wide, narrow in (("TRI_HUBS = 16384", "TRI_HUBS = 256"), ("TRI_BITMAP = 64", "TRI_BITMAP = 16")):
        assert order.count(wide) == 1
        order = order.replace(wide, narrow)
    run(tmp_path, "triangle_order_check.cpp", body("semiring.cuh") + body("pairs.cuh", "template <int THREADS, bool SEGMENTED, class Out>\nstatic int") +
        order, graph)


def test_mates_of_a_symmetric_pattern(tmp_path):
    text = relaxed(source("masked.cu"))
    struct = re.search(r"^struct MaskedStats \{.*?^\};\n", text, re.M | re.S).group(0)
    run(tmp_path, "masked_mates_check.cpp", struct + "".join(function(f, text) for f in ("masked_weight", "masked_stats_kernel", "masked_mates_kernel")))
