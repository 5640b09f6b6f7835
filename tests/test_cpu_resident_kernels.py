"""The serving loop's resident kernels leave room on every SM for the kernels
that a job launches on its own stream (two CTAs of the consensus service and
one of the alignment service, the defaults), by the registers that the
assembler reported for this build: nothing a job does may wait until a
resident kernel drains."""
import re

import pytest

SUB_PARTITION_REGISTERS = 16384  # four sub-partitions an SM; a CTA's warps spread evenly over them

# kernel -> threads of its CTA
JOB_KERNELS = {
    "nw_encode_kernel": 256, "nw_breakpoints_kernel": 256, "nw_cigar_kernel": 256, "exclusive_scan_kernel": 256,
    "cigar_breakpoints_kernel": 128, "nw_distance_kernel": 128, "nw_level_kernel": 128,
    "nw_distance_team_kernelILi4": 128, "nw_level_team_kernelILi4": 128,
    "layer_candidates_kernel": 256, "revcomp_kernel": 256, "quality_check_kernel": 256, "scan_kernel": 256,
    "place_kernel": 256, "order_kernel": 256, "gather_kernel": 256,
}


@pytest.fixture(scope="module")
def registers(native_lib):
    from racon_b200 import build
    regs = {}
    for src in build.CU_SOURCES:
        name = None
        with open(build.usage_file(src)) as f:
            for line in f:
                m = re.search(r"Compiling entry function '(\w+)'", line)
                name = m.group(1) if m else name
                m = re.search(r"Used (\d+) registers", line)
                if m and name:
                    regs[name] = int(m.group(1))
                    name = None
    return regs


def _of(registers, kernel):
    # the mangled name holds the kernel's own, its length before it
    own = kernel.split("IL")[0]
    hits = [r for n, r in registers.items() if "%d%s" % (len(own), kernel) in n]
    assert len(hits) == 1, (kernel, hits)
    return hits[0]


def _taken(regs, threads):
    per_warp = (regs * 32 + 255) // 256 * 256
    return per_warp * (threads // 32) // 4


@pytest.mark.parametrize("kernel", sorted(JOB_KERNELS))
def test_fits_beside_the_services(registers, kernel):
    resident = 2 * _taken(_of(registers, "poa_service_kernel"), 128) + _taken(_of(registers, "nw_service_kernel"), 128)
    assert resident + _taken(_of(registers, kernel), JOB_KERNELS[kernel]) <= SUB_PARTITION_REGISTERS
