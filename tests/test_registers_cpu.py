"""CPU: what the compiler says of kernels that were tuned to their register limit."""

from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

from tq_local_b200.build import CSRC, NVCC_FLAGS

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_dequantisation_of_16_bit_rows_stays_in_registers(tmp_path):
    """1024 threads hold 64 registers each; a value too many is stored in every unrolled step of a tile."""
    flags = [f for f in NVCC_FLAGS if f != "--shared"] + ["-Xptxas", "-v"]
    said = subprocess.run([NVCC, *flags, "-c", os.path.join(CSRC, "tq_dequant_tc.cu"), "-o", str(tmp_path / "out.o")],
                          check=True, capture_output=True, text=True)
    kernels = re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads",
                         said.stdout + said.stderr, re.S)
    narrow = {name: (int(stores), int(loads)) for name, stores, loads in kernels if "bfloat16" in name or "half" in name}
    assert len(narrow) == 12
    assert all(spills == (0, 0) for spills in narrow.values()), narrow
