"""The kernels that end a 2D stage keep their working set in registers: the
assembler's own report (-Xptxas -v) of the shipped source and flags.  A spill
there is traffic on the path that bounds the kernel.  Compiled for the
numbers of variables with kernels of their own (4 and 11) no spill is
allowed; the kernels for any number work through memory anyway, and may put
two values there.
"""
import os
import re
import shutil
import subprocess

import pytest

from piafs_b200 import build


@pytest.mark.skipif(not (os.path.exists(build._nvcc()) or shutil.which(build._nvcc())), reason="needs nvcc")
def test_no_spills(tmp_path):
    r = subprocess.run([build._nvcc()] + build.ARCH + build.FLAGS +
                       ["-Xptxas", "-v", "-c", os.path.join(build.CSRC, "stage2d.cu"), "-o", str(tmp_path / "s.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    # the mangled name carries the template arguments <scheme, y mode, mixed, NV, threads>
    found = re.findall(r"Compiling entry function '\S*k_stage2dILi(\d)ELi(\d)ELb(\d)ELi(\d+)ELi(\d+)E\S*'"
                       r"(?:.*\n)*?.*?(\d+) bytes spill stores, (\d+) bytes spill loads", r.stdout + r.stderr)
    assert len(found) >= 4 * 3 * 2 * 3      # schemes x y modes x precisions x numbers of variables
    bad = [f for f in found if int(f[5]) > (16 if f[3] == "0" else 0)]
    assert not bad, bad
