"""Register caps of the mixed-radix z pass: the compiler's spill counts at the
lengths whose fused stage is of radix 4 (the most registers a thread)."""
from __future__ import annotations

import importlib.util
import os
import re
import subprocess

from conftest import PKG_DIR

LENGTHS = (28, 32, 36, 40)


def test_radix4_z_kernels_keep_their_values_in_registers(tmp_path):
    """At most four 16-byte values of a thread in local memory: twelve are the
    fused stage's and up to twelve a frequency's kernel values."""
    spec = importlib.util.spec_from_file_location("gila_build", os.path.join(PKG_DIR, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    src = tmp_path / "z.cu"
    src.write_text('#include "matvec_mx_impl.cuh"\nnamespace gila {\n' + "".join(
        f"template __global__ void k_z_mx<{c}, {P}>(const ZParams<{c}>);\n"
        for P in LENGTHS for c in ("double2", "float2")) + "}\n")
    r = subprocess.run([b._nvcc(), *b.NVCC_FLAGS, "-Xptxas", "-v", "-I", b.INCLUDE, "-I", b.CSRC, "-c", str(src),
                        "-o", str(tmp_path / "z.o")], check=True, capture_output=True, text=True)
    spills = re.findall(r"properties for \S*k_z_mx\S*\s+\d+ bytes stack frame, (\d+) bytes spill stores", r.stderr)
    assert len(spills) == 2 * len(LENGTHS)
    assert max(int(s) for s in spills) <= 64
