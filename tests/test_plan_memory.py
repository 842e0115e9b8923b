"""Products of handles whose plans find no memory: every call takes the kernels that work on the registered arrays and
gives the same products, the first time and when repeated."""
import numpy as np
import pytest

from systemds_b200 import CompressedMatrixBlock, datagen, native
from systemds_b200.cmb import CLALibDecompress, CLALibTSMM
from systemds_b200.native import check
from tests.test_kernel_edges import _by_kind, _check, _ddc
from tests.util import TOL, dense_of, rel_err


def _cocoded(nRows):
    rng = np.random.default_rng(nRows)
    return CompressedMatrixBlock(nRows, 13, [datagen.random_group(k, c, nRows, rng) for k, c in (
        ("sdc", [0, 1]), ("rle", [2, 3]), ("sdcz", [4]), ("ddc", [5]), ("rle", [6]), ("sdcs", [7, 8]), ("unc", [9, 10, 11]),
        ("ddc_char", [12]))])


def _wide_dense(nRows):  # more uncompressed columns than a block has threads
    rng = np.random.default_rng(nRows)
    return CompressedMatrixBlock(nRows, 523, [datagen.random_group(k, c, nRows, rng) for k, c in (
        ("sdcz", [0]), ("unc", list(range(1, 521))), ("rle", [521, 522]))])


BLOCKS = {
    "short": lambda: datagen.random_cmb(5, 1027, datagen.KINDS + ("ddcfor", "ddc2", "ole", "rle", "sdc")),
    "every kind": lambda: datagen.random_cmb(6, 5003, datagen.KINDS + ("ddcfor", "ddc2", "ole", "rle", "sdc")),
    "next to byte maps": lambda: datagen.random_cmb(7, 5003, ("ddc",) * 20 + ("sdc", "rle", "unc", "ole", "const", "sdcs")),
    "cocoded": lambda: _cocoded(4161),
    "wide dense": lambda: _wide_dense(4127),
    "16-bit maps": lambda: _ddc(17001, [300, 1000, 5000, 257], 3, const=True),
    "mixed kinds side by side": lambda: datagen.random_cmb(9, 70001, ("ddc", "sdcz", "rle", "unc") * 16),
    "a kind per 32 columns": lambda: _by_kind(18817),  # decompress by columns
}


def _plan_bytes(cmb):
    st = native.cla_stats()
    check(native.lib().cla_stats_get(cmb.handle(), st))
    return st.device_bytes


def _use(cmb):
    X = dense_of(cmb)
    for _ in range(2):
        _check(cmb, ks=(1, 2, 5, 9, 65), qs=(1, 3, 9))
        got = np.array(CLALibDecompress.decompress(cmb))
        assert np.array_equal(got, X) or rel_err(got, X, np.abs(X) + 1e-300) < TOL
        got = CLALibTSMM.leftMultByTransposeSelf(cmb)
        assert rel_err(got, X.T @ X, np.abs(X).T @ np.abs(X) + 1e-300) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(BLOCKS))
def test_products_without_room_for_plans(kind):
    cmb = BLOCKS[kind]().to_device()
    before = _plan_bytes(cmb)
    _use(cmb)
    total = _plan_bytes(cmb) - before
    cmb.free()
    assert total > 0
    for limit in sorted({0, total // 8, total // 2, total - 1}):
        cmb = BLOCKS[kind]().to_device()
        check(native.lib().cla_set_plan_limit(cmb.handle(), limit))
        before = _plan_bytes(cmb)
        _use(cmb)
        # (what no kernel does without, a record per column, is not counted)
        assert _plan_bytes(cmb) - before <= limit + 64 * cmb.clen
        cmb.free()


def test_plan_limit_of_an_unknown_handle():
    assert native.lib().cla_set_plan_limit(123456789, 0) == -1
