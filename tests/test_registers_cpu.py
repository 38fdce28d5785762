"""Register pressure of the forward kernel, from the assembler's report: a softmax thread holds a row of 128 scores, and whatever a
change of the prologue or of a role leaves alive across the kernel is spilled inside its block loop."""
import os
import re
import subprocess

import pytest

from torch_mlu_b200 import build

# Bytes of spill stores by (head_dim, dropout, bias), the same for both 16-bit types: what the softmax loop of each instance leaves over.
LIMITS = {(64, 0, 0): 0, (64, 0, 1): 0, (64, 1, 0): 0, (64, 1, 1): 8, (128, 0, 0): 28, (128, 0, 1): 92, (128, 1, 0): 60, (128, 1, 1): 100}


def test_forward_instances_spill_no_more_than_their_loops_need(tmp_path):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc here")
    cmd = [nvcc, *build.NVCC_FLAGS, "-Xptxas", "-v", "-I", build.INCLUDE, "-c", os.path.join(build.CSRC, "fwd_prefill_sm100.cu"),
           "-o", str(tmp_path / "fwd.o")]
    report = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    found = re.findall(r"fwd_prefill_kernelILi(\d+)ELb([01])ELb([01])ELb([01])E[^\n]*\n\s*\d+ bytes stack frame, (\d+) bytes spill stores", report)
    spills = {(int(d), int(f16), int(drop), int(bias)): int(n) for d, f16, drop, bias, n in found}
    assert len(spills) == 16
    for (d, f16, drop, bias), n in spills.items():
        assert n <= LIMITS[d, drop, bias], (d, f16, drop, bias, n)


# The same by how units are claimed as well: the instance that takes them from waiting CTAs, and the one with the counter.
ALL_LIMITS = {(64, 0, 0): 0, (64, 0, 1): 0, (64, 1, 0): 0, (64, 1, 1): 8, (128, 0, 0): 28, (128, 0, 1): 48, (128, 1, 0): 60, (128, 1, 1): 100}


def test_either_way_to_claim_units_spills_no_more_than_its_loop_needs(tmp_path):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc here")
    cmd = [nvcc, *build.NVCC_FLAGS, "-Xptxas", "-v", "-I", build.INCLUDE, "-c", os.path.join(build.CSRC, "fwd_prefill_sm100.cu"),
           "-o", str(tmp_path / "fwd.o")]
    report = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    found = re.findall(r"fwd_prefill_kernelILi(\d+)ELb([01])ELb([01])ELb([01])ELb([01])E[^\n]*\n\s*\d+ bytes stack frame, (\d+) bytes spill stores", report)
    spills = {tuple(int(x) for x in f[:5]): int(f[5]) for f in found}
    assert len(spills) == 32
    for (d, f16, drop, bias, waiting), n in spills.items():
        assert n <= ALL_LIMITS[d, drop, bias], (d, f16, drop, bias, waiting, n)
