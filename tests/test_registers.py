"""Kernels whose launch bounds were chosen so that nothing is spilled: the
compiler's own report for sm_100a."""
import re
import subprocess

import pytest

from fastdose_b200 import build


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    def of(unit):
        out = str(tmp_path_factory.mktemp("ptxas") / "unit.o")
        cmd = [build._nvcc(), "-c", f"{build.CSRC}/{unit}", "-o", out] + build.ARCH + build.NVCC_FLAGS + ["-Xptxas", "-v"]
        log = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
        found = re.findall(r"Function properties for (\S+)\s+\d+ bytes stack frame, (\d+) bytes spill stores, "
                           r"(\d+) bytes spill loads", log)
        return {name: (int(a), int(b)) for name, a, b in found}

    return of


def test_terma_does_not_spill(report):
    spills = {k: v for k, v in report("terma.cu").items() if "terma_kernel" in k}
    assert len(spills) == 4
    assert all(v == (0, 0) for v in spills.values()), spills
