"""GPU: the forms of the LDPCA kernel against one another on the same codewords
(bits, rates, codes, BP iterations and the bound's bits, all exactly)."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("n,count", [(1584, 64), (6336, 24)])
def test_block_per_ladder_with_a_given_bound(gpu_ctx, n, count, tmp_path):
    """The bound given instead of summed: the ladder starts with no barrier but its
    own between the staged syndrome and the first code (tests/given_bound.cpp)."""
    from dvc_b200 import build, ldpca_bench as lb, native
    exe = str(tmp_path / "given_bound")
    cmd = ["g++", "-O1", "-std=c++17", "-w", "-I", "/usr/local/cuda/include", "-I", os.path.dirname(HERE) + "/include",
           "-I", build.CSRC, "-o", exe, os.path.join(HERE, "given_bound.cpp"), build.LIB,
           "-Wl,-rpath," + os.path.dirname(build.LIB), "-L/usr/local/cuda/lib64", "-lcudart_static", "-lpthread", "-ldl",
           "-lrt"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lr, acc, crc, x = lb.make_codewords(n, count, 17 + n)
    crc[-1] ^= 0x5A  # no code's bits match: the ladder ends at the full rate
    for name, a in (("lr", lr), ("acc", acc), ("crc", crc)):
        np.ascontiguousarray(a).tofile(tmp_path / name)
    r = subprocess.run([exe, native.DATA_DIR, native.TABLE_DIR, str(n), str(count)] +
                       [str(tmp_path / f) for f in ("lr", "acc", "crc")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-1000:])
