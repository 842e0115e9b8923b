"""Handles used from several threads: what the launchers share between them."""
import glob
import os
import re
import subprocess

import numpy as np
import pytest

from systemds_b200 import CompressedMatrixBlock, datagen, native
from tests.util import TOL, abs_dense_of, dense_of, rel_err

COL_MINS = 3  # CLA_AGG_COL_MINS
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "test_once_per_device.cpp")


def test_marks_per_device_under_the_thread_sanitizer(tmp_path):
    def run(source, exe):
        r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", source, "-o", exe], capture_output=True, text=True)
        return r if r.returncode else subprocess.run([exe], capture_output=True, text=True, timeout=120)

    plain = tmp_path / "plain.cpp"
    plain.write_text("int main() { return 0; }\n")
    if run(str(plain), str(tmp_path / "plain")).returncode:
        pytest.skip("no thread sanitizer here")
    r = run(SRC, str(tmp_path / "once"))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_launchers_keep_no_unguarded_marks():
    """A plain static flag per device, written by whichever handle comes first, is a data race between two handles; the
    memory pool's are read and written under its lock."""
    for path in glob.glob(os.path.join(ROOT, "systemds_b200", "csrc", "*.cu*")):
        found = re.findall(r"\bstatic\s+bool\s+(\w+)\s*\[", open(path).read())
        assert [f for f in found if f != "g_poolTried"] == [], path


@pytest.mark.gpu
def test_column_extrema_wait_for_a_product_in_flight():
    """Column extrema of a block with reference tuples go through decompressed rows in the handle's scratch, on a stream of its
    own; a self product enqueued on another stream just before them is still reading its own rows there."""
    import torch
    rng, nRows, nCols = np.random.default_rng(4), 100000, 161
    cmb = CompressedMatrixBlock(nRows, nCols, [datagen.random_group("ddcfor" if c % 2 else "sdcfor", [c], nRows, rng) for c in range(nCols)])
    X, A = dense_of(cmb), abs_dense_of(cmb)
    cmb.to_device()
    lib, h = native.lib(), cmb.handle()
    out, lo, stream = torch.empty((nCols, nCols), dtype=torch.float64, device="cuda"), np.empty(nCols), torch.cuda.Stream()
    want, scale = X.T @ X, A.T @ A
    for _ in range(20):
        out.zero_()
        torch.cuda.synchronize()
        native.check(lib.cla_tsmm_dev(h, out.data_ptr(), stream.cuda_stream))
        native.check(lib.cla_unary_agg(h, COL_MINS, native.ptr(lo)))
        stream.synchronize()
        assert rel_err(out.cpu().numpy(), want, scale) < TOL
        assert rel_err(lo, X.min(axis=0), A.max(axis=0)) < 1e-14
    cmb.free()
