"""A DRAM record is reported while the kernel sources it was taken from are unchanged: the list of those sources has to hold
every file that the kernels of the workload are written in."""
import os
import re

import pytest

import bench

CSRC = os.path.join(bench.ROOT, "comet_b200", "csrc")
HOST_ONLY = {"hostcopy.cuh", "masked.cuh"}            # included by spgemm.cu for paths that the workload does not take
KERNELS = {                                            # of one step, as the launch list shows them
    "spmm": ["spmm_plan_kernel", "spmm_stream_kernel", "spmm_short_rows_kernel", "spmm_pieces_kernel"],
    "sddmm": ["sddmm_plan_kernel", "sddmm_kernel"],
    "spgemm": ["bin_rows_kernel", "hash_rows_kernel", "mid_rows_kernel", "bitmap_symbolic_kernel", "scan_tile_sums",
               "short_rows_kernel", "team_items_kernel", "bitmap_numeric_kernel"],
    "triangles": ["tc_narrow_kernel", "scan_tile_sums", "tc_route_kernel", "tc_mid_kernel", "tc_warp_kernel"],
}


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


@pytest.mark.parametrize("workload", sorted(bench.KERNEL_SOURCES))
def test_the_sources_of_a_record_are_all_of_its_kernels(workload):
    listed = set(bench.KERNEL_SOURCES[workload])
    for name in listed:
        for header in re.findall(r'#include "([a-z_]+\.cuh)"', read(name)):
            assert header in listed | HOST_ONLY, (name, header)
    text = "".join(read(name) for name in listed)
    for kernel in KERNELS[workload]:
        assert re.search(r"__global__[^;{]*\b%s\(" % kernel, text), kernel
