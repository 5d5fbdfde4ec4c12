"""Register spills of the in-place steps, as the assembler reports them.

The steps are launched at five blocks of 256 threads per SM, 48 registers a
thread, and are bound by memory: spilled values are extra traffic.  A face
row's values are held across two passes of stores, so what form they are held
in decides what the whole kernel spills.  The wait for the previous launch is
an ordering point for the compiler: what stands before it stays live across it.
"""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

# Bytes (stored, loaded): half as much again as the steps spilled before their
# launches overlapped and the face rows' branches were merged.
BOUNDS = {
    "float": {"k_aa_odd": (48, 66), "k_aa_even": (54, 54)},
    "Half16SR": {"k_aa_odd": (156, 162), "k_aa_even": (84, 114)},
    "BF16SR": {"k_aa_odd": (138, 150), "k_aa_even": (84, 114)},
}


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
@pytest.mark.parametrize("storage", BOUNDS)
def test_inplace_step_spills(tmp_path, storage):
    from culbm_b200.build import ARCH, CSRC, INCLUDE, NVCC_FLAGS
    src = tmp_path / "steps.cu"
    src.write_text('#include "stream_kernels.cuh"\nusing namespace culbm;\n' + "".join(
        f"template __global__ void culbm::{k}<{storage}, float>(const __grid_constant__ StepArgs<{storage}, float>);\n"
        for k in BOUNDS[storage]))
    log = subprocess.run([NVCC, *ARCH, *NVCC_FLAGS, "-Xptxas=-v", "-I", INCLUDE, "-I", CSRC, "-cubin", "-o",
                          str(tmp_path / "steps.cubin"), str(src)], capture_output=True, text=True, check=True).stderr
    found = {}
    for part in log.split("Compiling entry function")[1:]:
        found[re.search(r"k_aa_(?:odd|even)", part).group()] = tuple(
            int(v) for v in re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", part).groups())
    assert found.keys() == BOUNDS[storage].keys(), log
    for kernel, (stores, loads) in found.items():
        most = BOUNDS[storage][kernel]
        assert stores <= most[0] and loads <= most[1], (kernel, stores, loads)
