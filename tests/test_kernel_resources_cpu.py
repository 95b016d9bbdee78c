"""What ptxas reports of the kernels that keep a whole row in registers (no GPU needed)."""
import os
import re
import subprocess

import pytest


@pytest.fixture(scope="module")
def simt_report(pkg, lib, tmp_path_factory):
    path = os.path.join(pkg.build.REPORTS, "kernels_simt.cu.ptxas")
    if os.path.exists(path) and "layernorm_rows_vec_kernel" in open(path).read():
        return open(path).read()
    out = tmp_path_factory.mktemp("ptxas") / "kernels_simt.o"
    return subprocess.run([pkg.build.NVCC] + pkg.build.FLAGS + ["-c", os.path.join(pkg.build.CSRC, "kernels_simt.cu"), "-o", str(out)],
                          capture_output=True, text=True, check=True).stderr


def test_row_kernels_keep_their_rows_in_registers(simt_report):
    """A lane holds 8 * NP values (32 * NP bytes): a stack frame of up to two words beside that is a loop constant, a larger
    one means that the row itself goes through local memory."""
    seen = 0
    for name, frame in re.findall(r"Function properties for (\S*(?:layernorm|softmax)_rows_vec_kernel\S*)\s+(\d+) bytes stack frame", simt_report):
        assert int(frame) <= 8, (name, frame)
        seen += 1
    assert seen >= 2 * 7 * 3
