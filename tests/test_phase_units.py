"""Profiling builds: every translation unit that includes the kernels' common
header registers its phase counters with the reader (host code, compiled here)."""
import shutil
import subprocess
from pathlib import Path

import pytest

from sunny_gen_eigensolver_b200 import build

UNIT = '#include "geneig_common.cuh"\n__global__ void k%d() { sgeig::phase_mark(0); }\n'
MAIN = '#include <cstdio>\nint main() { std::printf("%zu", sgeig::phase_readers().size()); }\n'


def test_every_kernel_unit_registers_its_counters(tmp_path):
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    for i in range(3):
        (tmp_path / f"u{i}.cu").write_text(UNIT % i + (MAIN if i == 0 else ""))
    exe = tmp_path / "units"
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-DSGEIG_PHASE_TIMERS", f"-I{build.CSRC}", "-o", str(exe),
                    *(str(tmp_path / f"u{i}.cu") for i in range(3))], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "3"


def test_every_kernel_source_includes_the_header():
    def reaches(name, seen=()):
        text = (Path(build.CSRC) / name).read_text()
        return "geneig_common.cuh" in text or any(
            f'"{h}"' in text and h not in seen and reaches(h, (*seen, h)) for h in build.HEADERS)
    for src in build.SOURCES:
        if "__global__" in (Path(build.CSRC) / src).read_text() or src.startswith("geneig_cta_"):
            assert reaches(src), src
