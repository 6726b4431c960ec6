"""What the host side allocates and launches, with the library's own objects linked to a stand-in for the CUDA runtime
(tests/cpu_checks/fake_launch.hpp)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKS = os.path.join(ROOT, "tests", "cpu_checks")


def link(tmp_path_factory, check, *objects):
    from comet_b200 import build
    build.build_library()
    exe = str(tmp_path_factory.mktemp("checks") / check[:-4])
    # functions of the files that are not linked are not called
    subprocess.check_call(["g++", "-O1", "-g", "-std=c++17", "-I/usr/local/cuda/include", os.path.join(CHECKS, check)] +
                          [os.path.join(build.OBJ, o) for o in objects] +
                          ["-no-pie", "-Wl,--unresolved-symbols=ignore-in-object-files", "-o", exe])
    return exe


def output(*command):
    out = subprocess.run([str(c) for c in command], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
    return out.stdout.strip()


@pytest.fixture(scope="module")
def hub_launch(tmp_path_factory):
    return link(tmp_path_factory, "hub_launch_check.cpp", "spgemm.o")


# two blocks an SM at most; below, one for every 4096 entries of the longer operand
@pytest.mark.parametrize("nrows,nnz_a,nnz_b,ncols,blocks", [(20000, 6000000, 2400, 200000, 296), (100000, 30000000, 3600, 150000, 296),
                                                            (20000, 400000, 2400, 200000, 98), (20000, 40000, 4000000, 200000, 296),
                                                            # few rows against a large B: 25 bytes of bitmaps per entry of B, 63 and 64
                                                            (3200, 640000, 8000000, 500000, 0), (4032, 640000, 4000032, 500000, 0),
                                                            (4032, 640000, 3937500, 500000, 296)])
def test_a_tall_operand_is_looked_over_by_the_whole_chip(hub_launch, nrows, nnz_a, nnz_b, ncols, blocks):
    assert int(output(hub_launch, nrows, nnz_a, nnz_b, ncols, 1000).split()[0]) == blocks


@pytest.mark.parametrize("stored", [1, 100000, 219000, 221000, 254061, 270000, 286069, 300000, 400000, 819200])
def test_columns_that_need_a_look_up_have_a_stage(hub_launch, stored):
    """Shared memory holds the bitmap, its ranks and a stage of 128 columns a warp at least, whatever the number of CTAs."""
    _, ctas, stage = map(int, output(hub_launch, 6000, 600000, 500000, 1000000, stored).split())
    assert ctas >= 1 and 128 <= stage <= 512
    dynamic = (stored + 31) // 32 * 8 + stage * 16 * 4
    assert ctas * (dynamic + 4176 + 1024) <= 228 * 1024 and dynamic + 4176 <= 227 * 1024


# bitmaps of 6000 * 6250 words; 62.5 and 87.5 % of the columns
@pytest.mark.parametrize("stored,products,staged", [(125000, 0, 1), (125001, 0, 0), (150000, 149999999, 0), (150000, 150000000, 1), (175000, 150000000, 1),
                                                    (175001, 150000000, 0)])
def test_columns_are_renumbered_where_it_pays(hub_launch, stored, products, staged):
    assert (int(output(hub_launch, 6000, 600000, 400000, 200000, stored, products).split()[2]) > 0) == staged


# 1.13 shares of the L2 a row with three CTAs on an SM, 1.5 with four
@pytest.mark.parametrize("nrows,teams", [(20, 1), (443, 1), (887, 1), (888, 0), (20000, 0)])
def test_few_rows_are_given_to_teams(hub_launch, nrows, teams):
    assert int(output(hub_launch, nrows, nrows * 100, 400000, 20000, 20000, "teams")) == teams


@pytest.mark.parametrize("n,nnz", [(500000, 8000000), (1600000, 20000000)])
def test_a_count_goes_on_without_memory_it_can_do_without(tmp_path_factory, n, nnz):
    assert output(link(tmp_path_factory, "triangle_memory_check.cpp", "tc.o"), n, nnz) == "ok"


def test_scratch_that_a_call_can_do_without(tmp_path):
    exe = str(tmp_path / "scratch")
    subprocess.check_call(["g++", "-O1", "-g", "-std=c++17", "-pthread", "-I/usr/local/cuda/include", "-x", "c++", os.path.join(CHECKS, "scratch_check.cpp"),
                           os.path.join(ROOT, "comet_b200", "csrc", "runtime.cu"), "-no-pie",
                           "-Wl,--unresolved-symbols=ignore-in-object-files", "-o", exe])
    assert output(exe) == "ok"
